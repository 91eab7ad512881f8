// Split-operand fused kernels for hidden widths up to 32.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(32)
}  // namespace qb
