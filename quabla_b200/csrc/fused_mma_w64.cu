// Split-operand fused kernels for hidden widths up to 64.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(64)
}  // namespace qb
