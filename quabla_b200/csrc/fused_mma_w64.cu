// Float32 fused kernels for hidden widths up to 64.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(float, 64, MmaGeom, fused_mma_kernel)
}  // namespace qb
