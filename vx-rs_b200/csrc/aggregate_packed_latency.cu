// The packed across-lanes scan form (aggregate_packed.cuh), kind kPackedLatency.
#include "aggregate_packed.cuh"

namespace vxsgm {
namespace packed {

cudaError_t launch_latency(const ScanGeometry& g, int ctas, const PairDev* d_pairs, const JobDev* d_jobs, const UnitDev* d_units,
                           int num_units, unsigned* counter, cudaStream_t stream, bool compact,
                           bool chained, bool more) {
    return launch_kind<kPackedLatency>(g, ctas, d_pairs, d_jobs, d_units, num_units, counter, stream, compact, chained, more);
}

}  // namespace packed
}  // namespace vxsgm
