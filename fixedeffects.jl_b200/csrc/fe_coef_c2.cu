// fe_coef_c2.cu -- the coefficient-side solve of 2-column tiles.
#include "fe_coef.cuh"

namespace fe {
template const void* coef_kernel<2>(int, int);
template size_t coef_smem_bytes<2>(int, int);
}  // namespace fe
