// Float32 fused kernels for hidden widths up to 16.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(float, 16, MmaGeom, fused_mma_kernel)
}  // namespace qb
