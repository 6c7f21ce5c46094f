// The wait words of the flow kernels (csrc/flow_wait.h), run as a CTA's threads would, on garbage.
#include "flow_wait.h"

#include <cstdio>
#include <cstring>

int main() {
    for (int threads = 32; threads <= 1024; threads += 32) {
        cmd::FlowWait w;
        std::memset(&w, 0xa5, sizeof(w));
        for (int tid = threads - 1; tid >= 0; --tid) cmd::flow_wait_init(&w, tid, 1000u + threads, 7u * threads);
        if (w.dead != 0 || w.ns != 1000u + threads || w.row_ns != 7u * threads) {
            std::printf("%d threads: dead = %u, ns = %llu\n", threads, w.dead, w.ns);
            return 1;
        }
    }
    // the limit of a row's wait: every wait of the steps before it may take its own limit, without overflow
    const unsigned long long some[] = {0, 1, 2, 3, 1000, 600000, 1ULL << 30, 1ULL << 40, 1ULL << 58, 1ULL << 61,
                                       (1ULL << 62) + 1, ~0ULL};
    for (unsigned long long ns : some)
        for (unsigned long long steps : some) {
            const unsigned __int128 need = (unsigned __int128)ns * steps * cmd::kWaitsPerStep;
            const unsigned long long got = cmd::flow_row_ns(ns, steps);
            const unsigned __int128 most = ~0ULL;
            if (got < (need < most ? need : most) || (ns == 0 && got != 0)) {
                std::printf("ns %llu steps %llu: %llu\n", ns, steps, got);
                return 1;
            }
        }
    std::printf("ok\n");
    return 0;
}
