// fe_coef_c1.cu -- the coefficient-side solve of 1-column tiles.
#include "fe_coef.cuh"

namespace fe {
template const void* coef_kernel<1>(int, int);
template size_t coef_smem_bytes<1>(int, int);
}  // namespace fe
