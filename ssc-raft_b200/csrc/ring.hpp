// ring.hpp -- bookkeeping of a ring of N shared-memory buffers that bulk copies fill:
// stage s is use s / N of buffer s % N.  A buffer's barrier completes one phase per
// use, so use u is waited for with parity u & 1.  Plain C++, also compiled for the host.
#pragma once

#ifdef __CUDACC__
#define RAFT_HD __host__ __device__ __forceinline__
#else
#define RAFT_HD inline
#endif

namespace raft {

template <int N> struct Ring {
    static RAFT_HD int buffer(int s) { return s % N; }
    static RAFT_HD unsigned parity(int s) { return (unsigned)(s / N) & 1u; }
    // whether stage s uses a buffer again, and the stage that it must wait for then
    static RAFT_HD bool reused(int s) { return s >= N; }
    static RAFT_HD int before(int s) { return s - N; }
};

}  // namespace raft
