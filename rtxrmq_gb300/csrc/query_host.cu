// query_host.cu -- plain queries on a table index whose results go to host memory
// in place: every line of them is stored once and whole. A separate translation
// unit, so that it compiles in parallel with query.cu.
#include "query_kernel.cuh"

namespace rmq {

cudaError_t launch_query_host(const BuildPlan &p, const V1View &v, const QueryOut &o, int64_t q,
                              const DeviceInfo &dev, cudaStream_t s) {
    return p.aligned ? launch_query_m<true, true, false, false, true>(v, o, q, nullptr, dev, s)
                     : launch_query_m<false, true, false, false, true>(v, o, q, nullptr, dev, s);
}

RMQ_VIOLATIONS_READER(violations_query_host)

}  // namespace rmq
