// fe_coef_c8.cu -- the cooperative solves of 8-column tiles: on the
// coefficient side (fe_coef.cuh) and the plain FP64 loop (fe_plain.cuh).
#include "fe_coef.cuh"
#include "fe_plain.cuh"

namespace fe {
template const void* coef_kernel<8>(int, int);
template const void* plain_kernel<8>(int, int);
template size_t coef_smem_bytes<8>(int, int);
}  // namespace fe
