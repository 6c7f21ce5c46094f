// flow_wait.h -- the shared-memory words of the bounded waits of rk4_flow.cuh and
// rk4_flow_cluster.cuh (plain C++ too: the host tests run it for every CTA size).
#pragma once

#ifdef __CUDACC__
#define CMD_HD __host__ __device__ __forceinline__
#else
#define CMD_HD inline
#endif

namespace cmd {

// Limit of a wait in nanoseconds, unless cmd_set_wait_limit gives another: about 10^6 stages.
constexpr long long kWaitLimitNs = 1LL << 30;

struct FlowWait {
    unsigned dead;               // set when a wait of this CTA gave up
    unsigned unused;
    unsigned long long ns;       // limit of a wait
};

// Written by one thread, whatever the CTA's size (a lattice of up to 32 cells runs 32 threads); a barrier of the CTA
// follows before any wait.
CMD_HD void flow_wait_init(FlowWait* w, int tid, unsigned long long ns) {
    if (tid == 0) {
        w->dead = 0;
        w->unused = 0;
        w->ns = ns;
    }
}

}  // namespace cmd
