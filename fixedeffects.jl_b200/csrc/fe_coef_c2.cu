// fe_coef_c2.cu -- the cooperative solves of 2-column tiles: on the
// coefficient side (fe_coef.cuh) and the plain FP64 loop (fe_plain.cuh).
#include "fe_coef.cuh"
#include "fe_plain.cuh"

namespace fe {
template const void* coef_kernel<2>(int, int);
template const void* plain_kernel<2>(int, int);
template size_t coef_smem_bytes<2>(int, int);
}  // namespace fe
