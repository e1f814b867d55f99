// The instantiations of the batched solver kernel for patterns of too many
// columns for shared memory (FP32 and FP64) in a translation unit of their
// own: batch.cu with NQG_BATCH_LARGE_UNIT defined, which keeps only its
// templates and these instantiations.
#define NQG_BATCH_LARGE_UNIT
#include "batch.cu"
