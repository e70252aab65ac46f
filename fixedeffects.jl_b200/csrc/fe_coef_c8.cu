// fe_coef_c8.cu -- the coefficient-side solve of 8-column tiles.
#include "fe_coef.cuh"

namespace fe {
template const void* coef_kernel<8>(int, int);
template size_t coef_smem_bytes<8>(int, int);
}  // namespace fe
