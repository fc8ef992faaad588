// query_lead.cu -- plain queries on an array of a batch that starts off a
// 128-byte boundary (its index is built from that boundary on); a separate
// translation unit, so that it compiles in parallel with query.cu.
#include "query_kernel.cuh"

namespace rmq {

cudaError_t launch_query_lead(const BuildPlan &p, const V1View &v, const QueryOut &o, int64_t q,
                              const DeviceInfo &dev, cudaStream_t s) {
    return p.aligned ? launch_query_m<true, true, false, true>(v, o, q, nullptr, dev, s)
                     : launch_query_m<false, true, false, true>(v, o, q, nullptr, dev, s);
}

RMQ_VIOLATIONS_READER(violations_query_lead)

}  // namespace rmq
