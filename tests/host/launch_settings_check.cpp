// Host check of the kernels' launch settings (set_launch, api.cpp) against a
// record of what the driver was told: whichever context launches next has its
// own carve-out, the most a block may ask for never shrinks, the driver is
// asked only for changes, a refused change is asked for again, and threads with
// a context each can set what they need.  Prints "ok" on success.
#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "common.h"

static std::mutex g_mu;
static std::map<const void*, int> g_max, g_carve;
static int g_asked = 0;
static bool g_fail = false;

extern "C" cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    std::lock_guard<std::mutex> lock(g_mu);
    ++g_asked;
    if (g_fail) return cudaErrorInvalidValue;
    (a == cudaFuncAttributeMaxDynamicSharedMemorySize ? g_max : g_carve)[f] = v;
    return cudaSuccess;
}

static void k1(int) {}
static void k2(int) {}

#define NEED(c)                                                             \
    do {                                                                    \
        if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } \
    } while (0)

int main() {
    using namespace vd;
    Ctx a, b;
    for (Ctx* c : {&a, &b}) {
        c->smem_sm = 228 * 1024;
        c->smem_reserved = 1024;
    }
    const void* const f1 = reinterpret_cast<const void*>(&k1);
    const void* const f2 = reinterpret_cast<const void*>(&k2);
    // two contexts in turn, with ligands of different sizes
    for (int turn = 0; turn < 3; ++turn) {
        NEED(set_launch(a, &k1, 6, 7 * 1024) == cudaSuccess);
        NEED(g_carve[f1] == (6 * 8 * 100 + 227) / 228 && g_max[f1] == 227 * 1024);
        NEED(set_launch(b, &k1, 6, 20 * 1024) == cudaSuccess);
        NEED(g_carve[f1] == (6 * 21 * 100 + 227) / 228 && g_max[f1] == 227 * 1024);
    }
    int asked = g_asked;
    for (int i = 0; i < 5; ++i) NEED(set_launch(b, &k1, 6, 20 * 1024) == cudaSuccess);
    NEED(g_asked == asked);
    // static shared memory, no carve-out of its own
    NEED(set_launch(a, &k2, 0, 0, 64) == cudaSuccess && g_max[f2] == 227 * 1024 - 64 && g_carve.count(f2) == 0);
    // refused, then granted
    g_fail = true;
    NEED(set_launch(a, &k1, 4, 7 * 1024) != cudaSuccess);
    g_fail = false;
    NEED(set_launch(a, &k1, 4, 7 * 1024) == cudaSuccess && g_carve[f1] == (4 * 8 * 100 + 227) / 228);
    // a context made after the device was reset sets everything again
    forget_launch_settings(0);
    g_max.clear();
    g_carve.clear();
    NEED(set_launch(a, &k1, 4, 7 * 1024) == cudaSuccess && g_max[f1] == 227 * 1024 && g_carve[f1] == (4 * 8 * 100 + 227) / 228);
    // another device has settings of its own
    b.device = 1;
    asked = g_asked;
    NEED(set_launch(b, &k1, 4, 7 * 1024) == cudaSuccess && g_asked == asked + 2);
    // threads
    std::vector<std::thread> pool;
    for (int t = 0; t < 8; ++t)
        pool.emplace_back([&, t] {
            Ctx c;
            c.smem_sm = 228 * 1024;
            c.device = t % 3;
            for (int i = 0; i < 2000; ++i) {
                set_launch(c, &k1, 1 + (i + t) % 6, 7 * 1024);
                set_launch(c, &k2, 1 + i % 4, 9 * 1024);
            }
        });
    for (auto& t : pool) t.join();
    std::printf("ok\n");
    return 0;
}
