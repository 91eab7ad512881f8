// Float32 fused kernels for hidden widths up to 32.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(float, 32, MmaGeom, fused_mma_kernel)
}  // namespace qb
