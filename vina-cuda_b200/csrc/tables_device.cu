// Pair-potential tables built on the device (vd_set_scoring_device).
//
// Same tables and operation order as the host build (tables.cpp,
// precalculate.h:121-140, 255-283): one thread per (type pair, entry)
// evaluates the weighted XS energy at its own and its neighbouring sample
// distances in FP64 and writes
//   se[i], sd[i] = (e[i+1]-e[i-1]) / ((r[i+1]-r[i-1]) r[i]), fast[i] = (e[i]+e[i+1])/2
// in double plus the device copies the kernels read: fast in FP32 and FP64,
// smooth as {e_i, dor_i, e_i+1, dor_i+1}.  The largest pair force, which sets the
// fixed-point scale, is found here too; the double tables cross to the host
// only for vd_get_tables (7.5 MB: 1.6 of the 2.1 ms a weight set took).
// This file is compiled without FMA contraction so the arithmetic rounds like
// the host build; only exp() may differ from the host's, by an ulp.
#include <algorithm>
#include <cfloat>

#include "common.h"
#include "xs_terms.h"

namespace vd {
namespace {

struct TableParams {
    double w[6];
    double* fast;     // [kPairTypes][kN]
    double* se;
    double* sd;
    float* fast_f;    // [kPairTypes][kBins]; null: the doubles above only
    double* fast_d;   // [kPairTypes][kBins]
    float4* smooth;   // [kPairTypes][kBins]
};

__device__ __forceinline__ double sample_r(int k) { return sqrt(k / 32.0); }

__global__ void __launch_bounds__(256) tables_kernel(TableParams p) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= kPairTypes * kN) return;
    const int tp = gid / kN, i = gid - tp * kN;
    int t2 = 0;
    while ((t2 + 1) * (t2 + 2) / 2 <= tp) ++t2;  // tp = t1 + t2 (t2 + 1) / 2, t1 <= t2
    const int t1 = tp - t2 * (t2 + 1) / 2;
    auto energy = [&](int k) { return fmin(DBL_MAX, xs_weighted_energy(p.w, t1, t2, sample_r(k))); };
    auto dor = [&](int k, double em, double ep) {
        return (k == 0 || k == kN - 1) ? 0.0 : (ep - em) / ((sample_r(k + 1) - sample_r(k - 1)) * sample_r(k));
    };
    const double e_i = energy(i);
    const double e_m = i > 0 ? energy(i - 1) : 0.0;
    const double e_p = i + 1 < kN ? energy(i + 1) : 0.0;
    const double sd_i = dor(i, e_m, e_p);
    const double fast_i = (e_p + e_i) / 2;
    const size_t o = size_t(tp) * kN + i;
    p.se[o] = e_i;
    p.sd[o] = sd_i;
    p.fast[o] = fast_i;
    if (p.fast_f && i < kBins) {  // i + 2 <= kN - 1: the next entry's derivative is defined
        const double sd_p = dor(i + 1, e_i, energy(i + 2));
        const size_t ob = size_t(tp) * kBins + i;
        p.fast_f[ob] = float(fast_i);
        p.fast_d[ob] = fast_i;
        p.smooth[ob] = make_float4(float(e_i), float(sd_i), float(e_p), float(sd_p));
    }
}

// Largest |derivative| x r over the reachable bins (pair_force_bound): the
// doubles are not negative, so their bits order like them.
__global__ void __launch_bounds__(256) force_bound_kernel(const double* sd, unsigned long long* bound) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x, tp = gid / kBins, i = gid - tp * kBins;
    double v = 0;
    if (tp < kPairTypes && i + 1 < kBins) {
        const double* d = sd + size_t(tp) * kN + i;
        v = fmax(0.0, fmax(fabs(d[0]), fabs(d[1])) * sqrt((i + 1) / 32.0));  // a NaN counts as 0, as on the host
    }
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) atomicMax(bound, static_cast<unsigned long long>(__double_as_longlong(v)));
}

}  // namespace

// Tables of w: the doubles (fast, se, sd in turn) to `doubles`; the kernels' copies too, where device is true.
static vd_status run_tables(Ctx& c, const double* w, double* doubles, bool device) {
    const size_t n = size_t(kPairTypes) * kN;
    TableParams p{};
    for (int k = 0; k < 6; ++k) p.w[k] = w[k];
    p.fast = doubles;
    p.se = p.fast + n;
    p.sd = p.se + n;
    p.fast_f = device ? c.d_fast : nullptr;
    p.fast_d = c.d_fastd;
    p.smooth = c.d_smooth;
    tables_kernel<<<unsigned((n + 255) / 256), 256, 0, c.stream>>>(p);
    VD_CUDA(cudaGetLastError());
    return VD_OK;
}

vd_status build_tables_device(Ctx& c, const double w[6], double& force_bound) {
    const size_t n = size_t(kPairTypes) * kN, nb = size_t(kPairTypes) * kBins;
    vd_status st = VD_OK;
    if (!c.d_fast && (st = dev_alloc(c, &c.d_fast, nb * sizeof(float), "pair tables")) != VD_OK) return st;
    if (!c.d_smooth && (st = dev_alloc(c, &c.d_smooth, nb * sizeof(float4), "pair tables")) != VD_OK) return st;
    if (!c.d_fastd && (st = dev_alloc(c, &c.d_fastd, nb * sizeof(double), "pair tables")) != VD_OK) return st;
    if ((st = ensure_scratch(&c, 3 * n * sizeof(double))) != VD_OK) return st;
    if ((st = settle_device_calls(c)) != VD_OK) return st;
    double* const d = static_cast<double*>(c.d_scratch);
    if ((st = run_tables(c, w, d, true)) != VD_OK) return st;
    unsigned long long* const bound = reinterpret_cast<unsigned long long*>(c.d_counter + 16);
    VD_CUDA(cudaMemsetAsync(bound, 0, sizeof(*bound), c.stream));
    force_bound_kernel<<<unsigned((nb + 255) / 256), 256, 0, c.stream>>>(d + 2 * n, bound);
    VD_CUDA(cudaGetLastError());
    VD_CUDA(cudaMemcpyAsync(&force_bound, bound, sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    VD_CUDA(cudaStreamSynchronize(c.stream));
    return VD_OK;
}

// Builds the doubles again (the scratch has had other uses since) and leaves
// the kernels' copies alone.  Without room for 7.5 MB of scratch under the
// context's cap they go straight to host memory.
vd_status fetch_tables(Ctx& c, double* fast, double* se, double* sd) {
    const size_t n = size_t(kPairTypes) * kN;
    double* const out[3] = {fast, se, sd};
    vd_status st = ensure_scratch(&c, 3 * n * sizeof(double));
    if (st == VD_ERR_NOMEM) {
        void* host = nullptr;
        VD_CUDA(cudaHostAlloc(&host, 3 * n * sizeof(double), cudaHostAllocMapped));
        double* const h = static_cast<double*>(host);
        st = run_tables(c, c.weights, h, false);
        const cudaError_t e = cudaStreamSynchronize(c.stream);
        for (int k = 0; k < 3 && st == VD_OK && e == cudaSuccess; ++k)
            if (out[k]) std::copy(h + k * n, h + (k + 1) * n, out[k]);
        cudaFreeHost(host);
        VD_CUDA(e);
        return st;
    }
    if (st != VD_OK) return st;
    double* const d = static_cast<double*>(c.d_scratch);
    if ((st = run_tables(c, c.weights, d, false)) != VD_OK) return st;
    for (int k = 0; k < 3; ++k)
        if (out[k]) VD_CUDA(cudaMemcpyAsync(out[k], d + k * n, n * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    VD_CUDA(cudaStreamSynchronize(c.stream));
    return VD_OK;
}

}  // namespace vd
