// flow_wait.h -- the shared-memory words of the bounded waits of rk4_flow.cuh and
// rk4_flow_cluster.cuh (plain C++ too: the host tests run it for every CTA size).
#pragma once

#ifdef __CUDACC__
#define CMD_HD __host__ __device__ __forceinline__
#else
#define CMD_HD inline
#endif

namespace cmd {

struct FlowWait {
    unsigned dead;               // set when a wait of this CTA gave up
    unsigned unused;
};

// Written by one thread, whatever the CTA's size (a lattice of up to 32 cells runs 32 threads); a barrier of the CTA
// follows before any wait.
CMD_HD void flow_wait_init(FlowWait* w, int tid) {
    if (tid == 0) {
        w->dead = 0;
        w->unused = 0;
    }
}

}  // namespace cmd
