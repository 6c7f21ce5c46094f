// cmd::upload_once (csrc/cmd_internal.h) over a fake runtime whose first copy fails.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>

static int copies = 0, live = 0;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { ++live; *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { --live; std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (++copies == 1) return cudaErrorInvalidValue;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void**, size_t, unsigned) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

#include "cmd_internal.h"

int cmd::fail(int code, const std::string&) { return code; }

int main() {
    const int table[3] = {7, 8, 9};
    cmd::DevBuf d;
    if (cmd::upload_once(d, table, sizeof(table), "table") != CMD_ERR_CUDA || d.p || live != 0) return std::puts("a copy that failed left its buffer"), 1;
    if (cmd::upload_once(d, table, sizeof(table), "table") != CMD_OK || std::memcmp(d.p, table, sizeof(table))) return std::puts("not uploaded again"), 1;
    if (cmd::upload_once(d, table, sizeof(table), "table") != CMD_OK || copies != 2) return std::puts("uploaded twice"), 1;
    cmd::DevBuf none;
    if (cmd::upload_once(none, nullptr, 0, "empty") != CMD_OK || !none.p || copies != 2) return std::puts("empty table"), 1;
    std::puts("ok");
    return 0;
}
