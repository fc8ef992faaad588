// batch_unaligned.cu -- the persistent batch kernel for values off a 16-byte
// boundary; a separate translation unit, so that it compiles in parallel with
// batch.cu.
#include "batch_impl.cuh"

namespace rmq {

cudaError_t batch_kernel_unaligned(uint32_t mode, bool build, const void **fn, int *per_sm) {
    return batch_kernel_t<false>(mode, build, fn, per_sm);
}

RMQ_VIOLATIONS_READER(violations_batch_unaligned)

}  // namespace rmq
