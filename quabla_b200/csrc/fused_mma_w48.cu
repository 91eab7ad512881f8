// Split-operand fused kernels for hidden widths up to 48.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(48)
}  // namespace qb
