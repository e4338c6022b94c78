// Batch kernel, layout variant set 0 (see batch_body.cuh).
// Four limbs a loop body: the operations of a mixed batch run side by side on a
// multiprocessor and share its instruction cache.  A batch of 47,452 mixed
// operations takes 24.1 ms with 4, 25.4 with 8 and 25.9 with 16 (batches queued
// behind each other 19.3, 20.6 and 22.1), one of a single kind 5 to 10% more with
// 4 than with 16.
#define HG_SQ_UNROLL 4

#include "batch_body.cuh"

namespace hg {

HG_BATCH_VARIANT_ENTRY_POINTS(0)

}  // namespace hg
