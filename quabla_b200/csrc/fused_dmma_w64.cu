// Float64 fused kernels for hidden widths up to 64.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(double, 64, DmmaGeom, fused_dmma_kernel)
}  // namespace qb
