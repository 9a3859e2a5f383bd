// Rules of the edge rows' exchange in elastic shots on chip (fwi_cluster.cuh).
//
// Who takes part: the lanes of the grid's columns send, and only they wait.  A lane
// that waited without sending would hold nobody up: the barrier could pass two phases
// while it still asks for the first, and two phases look like none to it.
//
// When a block may leave.
// A block whose halo waits all succeeded holds every edge row that was sent to it.
// One that gave up does not: a late neighbour may send its last rows only then,
// and its own wait succeeds, as the block that gave up had sent before it waited.
// So whoever may have rows on the way, or may be sent some, stays 20 us, long past
// their arrival, before the cluster's last barrier: the thread that gave up, and
// every thread that sees the status word set after its last send.  A sender that
// reads it still clear sent before the word was set, and the block that set it
// stays 20 us from there on.
#pragma once

#ifdef __CUDACC__
#define HMC_HALO_HD __host__ __device__ __forceinline__
#else
#define HMC_HALO_HD inline
#endif

namespace hmc {
namespace fwi {

HMC_HALO_HD bool halo_sends(bool column) { return column; }
HMC_HALO_HD bool halo_awaits(bool column) { return column; }

constexpr unsigned long long HALO_DRAIN_NS = 20000;
// gave_up: a wait of this thread ran out; status: the word, read after its last send.
HMC_HALO_HD bool halo_must_drain(bool gave_up, int status) { return gave_up || status != 0; }

}  // namespace fwi
}  // namespace hmc
