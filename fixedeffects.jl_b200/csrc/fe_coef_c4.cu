// fe_coef_c4.cu -- the coefficient-side solve of 4-column tiles.
#include "fe_coef.cuh"

namespace fe {
template const void* coef_kernel<4>(int, int);
template size_t coef_smem_bytes<4>(int, int);
}  // namespace fe
