// flow_wait.h -- the shared-memory words of the bounded waits of rk4_flow.cuh and
// rk4_flow_cluster.cuh (plain C++ too: the host tests run it for every CTA size).
#pragma once

#include <cstddef>

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
    unsigned long long ns;       // limit of a wait between warps that exchange spins or a row
    unsigned long long row_ns;   // limit of the helper warp's wait for the next row
};

// A row lies up to `steps` steps ahead, which the caller sets, and a step has at most kWaitsPerStep waits of its own,
// each bounded by ns: no healthy run's row takes longer than all of them together.
constexpr unsigned long long kWaitsPerStep = 8;
CMD_HD unsigned long long flow_row_ns(unsigned long long ns, unsigned long long steps) {
    const unsigned long long most = ~0ULL;
    if (ns == 0) return 0;
    if (steps >= most / kWaitsPerStep - 1) return most;
    const unsigned long long waits = kWaitsPerStep * (steps + 1);
    return waits > most / ns ? most : waits * ns;
}

// Written by one thread, whatever the CTA's size (a lattice of up to 32 cells runs 32 threads); a barrier of the CTA
// follows before any wait.
CMD_HD void flow_wait_init(FlowWait* w, int tid, unsigned long long ns, unsigned long long row_ns) {
    if (tid == 0) {
        w->dead = 0;
        w->unused = 0;
        w->ns = ns;
        w->row_ns = row_ns;
    }
}

}  // namespace cmd
