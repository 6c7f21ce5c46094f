// The wait words of the flow kernels (csrc/flow_wait.h), run as a CTA's threads would, on garbage.
#include "flow_wait.h"

#include <cstdio>
#include <cstring>

int main() {
    for (int threads = 32; threads <= 1024; threads += 32) {
        cmd::FlowWait w;
        std::memset(&w, 0xa5, sizeof(w));
        for (int tid = threads - 1; tid >= 0; --tid) cmd::flow_wait_init(&w, tid, 1000u + threads);
        if (w.dead != 0 || w.ns != 1000u + threads) {
            std::printf("%d threads: dead = %u, ns = %llu\n", threads, w.dead, w.ns);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
