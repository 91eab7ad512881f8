// Split-operand fused kernels for hidden widths up to 16.
#include "fused_mma_entries.cuh"

namespace qb {
QB_MMA_LOOKUP(16)
}  // namespace qb
