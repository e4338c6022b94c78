// Batch kernel, layout variant set 0 (see batch_body.cuh).
// Four limbs a loop body: the operations of a mixed batch run side by side on a
// multiprocessor and share its instruction cache.  A batch of 47,452 mixed
// operations takes 24.0 ms with 4, 25.4 with 8 and 25.9 with 16 (batches queued
// behind each other 19.2, 20.6 and 22.2).  One of a single kind takes 5 to 13%
// more with 4 than with 16: of 2048 bits 40,000 encryptions 8.4 ms against 7.5,
// 20,000 decryptions 34.6 against 31.4, 40,000 scalar Muls 10.7 against 10.1.
#define HG_SQ_UNROLL 4

#include "batch_body.cuh"

namespace hg {

HG_BATCH_VARIANT_ENTRY_POINTS(0)

}  // namespace hg
