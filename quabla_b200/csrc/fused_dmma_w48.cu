// Float64 fused kernels for hidden widths up to 48.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(double, 48, DmmaGeom, fused_dmma_kernel)
}  // namespace qb
