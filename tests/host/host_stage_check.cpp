// Host check of the context's pinned stage (api.cpp) against a pinned
// allocator that can be made to fail: a failure leaves no pending CUDA error,
// a map read goes on through pageable memory, keeps the stage there was and
// does not ask again.  Prints "ok" on success.
#include <cstdio>
#include <cstdlib>

#include "common.h"

static bool g_fail = false;
static int g_asked = 0, g_live = 0;
static cudaError_t g_pending = cudaSuccess;

extern "C" {
cudaError_t cudaMallocHost(void** p, size_t bytes) {
    ++g_asked;
    if (g_fail) return g_pending = cudaErrorMemoryAllocation;
    ++g_live;
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    --g_live;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = g_pending;
    g_pending = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

#define NEED(c)                                                    \
    do {                                                           \
        if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } \
    } while (0)

int main() {
    using namespace vd;
    Ctx c;
    // docking's stage: a failed growth, then a good one
    NEED(ensure_host_stage(&c, 1000) == VD_OK && c.h_stage_bytes >= 1000 && g_live == 1);
    g_fail = true;
    NEED(ensure_host_stage(&c, 100000) == VD_ERR_CUDA);
    NEED(cudaGetLastError() == cudaSuccess);
    NEED(c.h_stage == nullptr && c.h_stage_bytes == 0 && g_live == 0);
    g_fail = false;
    NEED(ensure_host_stage(&c, 1000) == VD_OK && g_live == 1);
    // map reads: pageable, then one request for pinned memory, refused
    g_fail = true;
    g_asked = 0;
    for (int i = 0; i < 200; ++i) {
        char* const s = map_slab(c, 50000);
        NEED(s && s != c.h_stage);
        s[0] = s[49999] = 1;
        NEED(cudaGetLastError() == cudaSuccess);
        NEED(g_asked == (i < 40 ? 0 : 1));
    }
    NEED(c.h_stage && c.h_stage_bytes >= 1000 && g_live == 1);
    NEED(map_slab(c, 900) == c.h_stage);
    // granted
    Ctx d;
    g_fail = false;
    g_asked = 0;
    for (int i = 0; i < 60; ++i) NEED((map_slab(d, 50000) == d.h_stage) == (i >= 40));
    NEED(g_asked == 1 && g_live == 2);
    std::printf("ok\n");
    return 0;
}
