// Post-processing of the chain results on the GPU, replacing the host tail
// of the reference (main_procedure_cu.cpp:896-926, main.cpp:423-489):
//   cluster : energy-sorted greedy selection of up to 20 poses whose
//             heavy-atom RMSD to every kept pose is >= min_rmsd
//             (add_to_output_container semantics, coords.cpp:47-62, applied
//             in energy order)
//   refine  : refine_structure (main.cpp:139-157): dense BFGS (bfgs.h:95-140)
//             on the direct-sum score (non_cache.cpp:82-128) with the slope
//             ramp 100*10^(2p), authentic caps (1000)
//   score   : eval_intramolecular of the best mode and eval_adjusted
//             (model.cpp:1375-1431) in double, remove_redundant, the
//             num_modes / energy_range cut and RMSD bounds to mode 1
// dock_pipeline runs the docking launch and these kernels; the batched form
// records the whole sequence, with its uploads and downloads, into one CUDA
// graph per call (updated in place for the next call of the same shape).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <functional>
#include <string>

#include "dock.h"
#include "launch.h"
#include "search.cuh"

namespace vd {
namespace {

// ------------------------------------------------------------ receptor view
struct RecView {
    const float4* rec;          // relevant receptor atoms {x,y,z,type}
    const double4* recd;        // same in double
    const int32_t* cell_start;  // [cells+1]
    const int32_t* cell_list;   // atom indices per cell
    double init[3], per[3];     // szv_grid cell geometry: origin, cells per A
    int32_t dim[3];
    double gb[3], ge[3];        // box (non_cache gd)
    float gbf[3], gef[3];       // the same in FP32
};

// szv_grid.cpp:92-107 (fl_to_sz), with the cells per A in place of a division:
// a point within rounding of a cell face may take the neighbour cell, whose
// list reaches a little further than the cutoff (ensure_receptor_cells) and so
// holds the same atoms in reach, in the same order.  Optimisers do reach poses
// that are not finite: the conversion saturates and takes a NaN to the lowest
// integer, so clamping gives those a cell too.
__device__ __forceinline__ int cell_of(const RecView& R, double x, double y, double z) {
    const double c[3] = {x, y, z};
    int idx[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) idx[d] = max(0, min(int((c[d] - R.init[d]) * R.per[d]), R.dim[d] - 1));
    return VD_DCLAMP(idx[0] + R.dim[0] * (idx[1] + R.dim[1] * idx[2]), 0, R.dim[0] * R.dim[1] * R.dim[2] - 1, kChkCell);
}

// ------------------------------------------------------------ cluster
struct ClusterParams {
    const float4* pool;
    const int64_t* lig_off;
    const int32_t* prefix;      // items of ligand i: [prefix[i], prefix[i+1])
    const float* conf;          // [items][stride]
    const float* e;
    int32_t stride;
    float min_rmsd;
    int32_t max_keep;
    int32_t* kept;              // [n_ligs][20] item indices, -1 padded
    int32_t sort_n;             // power of two >= chains per ligand
    int32_t warp_floats;
    int32_t warps;              // candidates placed at a time
};

__device__ __forceinline__ uint32_t ordered(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// One block per ligand.  Its serial part is the greedy pass: with one warp,
// each candidate cost a pose load, its kinematics and up to 20 RMSDs one
// after the other.  p.warps warps take the next candidates together, each
// tests its own against the poses kept so far, and then the first survivor
// is kept and the ones behind it test it, until none is left: the same poses
// as taking candidates one by one.  6,500 chains of a 31-atom ligand, B200:
// 382 us with 256 threads and one greedy warp, 101 us (half of it the sort).
constexpr int kClusterThreads = 1024;

__global__ void __launch_bounds__(kClusterThreads) cluster_kernel(ClusterParams p) {
    extern __shared__ float4 smem4[];
    __shared__ int s_open[2];  // first survivor (warp index), alternating
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem4);
    const int li = blockIdx.x;
    const int b0 = p.prefix[li], n = p.prefix[li + 1] - b0;
    for (int i = threadIdx.x; i < p.sort_n; i += blockDim.x) {
        unsigned long long k = ~0ull;
        if (i < n) {
            const float e = p.e[b0 + i];
            if (e == e && e < FLT_MAX) k = (static_cast<unsigned long long>(ordered(e)) << 32) | uint32_t(i);
        }
        keys[i] = k;
    }
    __syncthreads();
    for (int size = 2; size <= p.sort_n; size <<= 1)  // bitonic sort, ascending
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int j = threadIdx.x; j < p.sort_n / 2; j += blockDim.x) {
                const int i = 2 * j - (j & (stride - 1));  // lower index of the j-th exchange
                const bool up = (i & size) == 0;
                const unsigned long long a = keys[i], b = keys[i + stride];
                if ((a > b) == up) { keys[i] = b; keys[i + stride] = a; }
            }
            __syncthreads();
        }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const LigView L = lig_view(p.pool, p.lig_off[li]);
    float* wbase = reinterpret_cast<float*>(keys + p.sort_n);
    const WarpMem m = carve(wbase + size_t(min(wid, p.warps - 1)) * p.warp_floats, L.na, L.nn, L.np, L.nt);
    float* kc = wbase + size_t(p.warps) * p.warp_floats;  // kept coordinates [20][na][3]
    const int nc = 7 + L.nt;
    auto close_to = [&](int j) {
        const float* c = kc + size_t(j) * 3 * L.na;
        float acc = 0.f;
        for (int i = lane; i < L.na; i += 32) {
            const float dx = m.c[i].x - c[3 * i], dy = m.c[i].y - c[3 * i + 1], dz = m.c[i].z - c[3 * i + 2];
            acc += dx * dx + dy * dy + dz * dz;
        }
        acc = warp_sum(acc);
        return sqrtf(acc / float(L.na)) < p.min_rmsd;
    };
    int nk = 0;
    if (threadIdx.x < 2) s_open[threadIdx.x] = p.warps;
    __syncthreads();
    for (int r0 = 0, turn = 0; r0 < n && nk < p.max_keep; r0 += p.warps) {
        const int r = r0 + wid;
        const unsigned long long k = (wid < p.warps && r < n) ? keys[r] : ~0ull;
        bool open = k != ~0ull;  // finite energies sort first
        int item = 0;
        if (open) {
            item = b0 + VD_DCLAMP(int(uint32_t(k)), 0, n - 1, kChkClusterKept);
            for (int i = lane; i < nc; i += 32) m.x[i] = p.conf[size_t(item) * p.stride + i];
            __syncwarp();
            kinematics(L, m, lane);
            for (int j = 0; j < nk && open; ++j) open = !close_to(j);
        }
        while (nk < p.max_keep) {
            if (open && lane == 0) atomicMin(&s_open[turn], wid);
            __syncthreads();
            const int first = s_open[turn];
            turn ^= 1;
            if (first < p.warps && wid == first) {
                float* c = kc + size_t(nk) * 3 * L.na;
                for (int i = lane; i < L.na; i += 32) { c[3 * i] = m.c[i].x; c[3 * i + 1] = m.c[i].y; c[3 * i + 2] = m.c[i].z; }
                if (lane == 0) p.kept[li * VD_MAX_MODES + nk] = item;
                open = false;
            }
            __syncthreads();
            if (threadIdx.x == 0) s_open[turn ^ 1] = p.warps;  // read by all above, next used a turn later
            if (first >= p.warps) break;  // no survivor: next candidates
            ++nk;
            if (open) open = !close_to(nk - 1);
        }
    }
    for (int j = nk + threadIdx.x; j < VD_MAX_MODES; j += blockDim.x) p.kept[li * VD_MAX_MODES + j] = -1;
}

// ------------------------------------------------------------ refine
struct RefineParams {
    const float4* pool;
    const int64_t* lig_off;     // per ligand in batch
    const int32_t* pose_lig;    // [n_poses] ligand (batch index) of each pose
    float* poses;               // [n_poses][stride] in/out
    float* e_out;               // [n_poses]
    int32_t stride;
    int32_t n_poses;
    int32_t max_steps_default;
    const int32_t* max_steps;   // per ligand (may be null)
    RecView R;
    const float4* smooth;
    float fix, inv_fix;         // fixed-point scale of the pair forces (EvalParams::fix) and 1/fix
    unsigned long long* evals;
    int32_t skip_invalid;       // leave poses whose e_out is FLT_MAX untouched
};

// One block refines one pose, on 16 warps or fewer (refine_launch).  A
// dense-BFGS run is a serial chain of evaluations, and an evaluation on the
// direct-sum score is mostly receptor neighbours (tens to hundreds per atom,
// three dependent loads each) and intra pairs: with one warp a pose, one lane
// walked an atom's neighbours one after the other and a 20-pose call kept 5 SMs
// busy.  Warp 0 runs the
// optimiser; for each evaluation it places the atoms, then all warps compute
// the neighbour and pair terms in parallel into shared memory, and their sums
// are taken from there in the order a single lane would take them (a
// receptor cell's list order per atom, 32 segments of the pair list), so the
// refined poses do not depend on how the work was spread.
// 20 poses of 45 atoms / 12 torsions in an 8,000-atom receptor, B200:
// 12.79 ms with one warp a pose, 2.22 ms with sixteen (a single docked ligand's
// 20 modes, 31 atoms / 8 torsions: 1.95 -> 0.57 ms).  What is left is latency:
// ~1,900 cycles of body frames, ~5,000 of receptor terms (two thirds of them
// gathers from L2), ~1,200 of pairs, ~2,300 of optimiser per evaluation.
constexpr int kNb = 32;    // neighbours of an atom per tile (one per lane)
constexpr int kSlots = 4;  // atoms a warp takes at a time

// Per-warp tile of neighbour terms, one row of kNb neighbours per atom and
// component: [kSlots * 4] {x, y, z, energy}, then [kSlots] derivatives; rows
// of 36 floats keep the row-wise 128-bit reads free of bank conflicts.  Then
// the atoms' clamped positions and cell ranges.
constexpr int kRow = kNb + 4;
constexpr int kTileFloats = kSlots * 5 * kRow + kSlots * 4 + kSlots * 2;
static_assert(kTileFloats % 4 == 0, "tiles stay 16-byte aligned");

struct TeamMem {
    float* tile;        // this warp's
    float* eatom;       // [na] receptor terms
    float* pair;        // [4][np] force on the second atom, energy
    uint16_t* run;      // [runs + 1] first pair of each run of one second atom
    int* cmd;           // 0: leave, 1: evaluate
    float* slope;
    int* runs;
};

__host__ __device__ inline int team_floats(int warps, int na, int np) {
    return warps * kTileFloats + pad4(na) + 4 * np + pad4((np + 2) / 2) + 4;
}

// non_cache::eval_deriv terms (FP32, smooth table, curl v) of the atom
// groups `wid`, `wid` + warps, ..: gradients to m.fx/fy/fz, energies
// to eatom.  Lanes are neighbours, a tile of kNb per atom at a time; then
// lane 4 s + c adds up component c (x, y, z, energy) of atom s in list order.
template <int warps>
__device__ __forceinline__ void direct_terms(const LigView& L, const WarpMem& m, const RecView& R, const float4* smooth,
                                             float v, float slope, const TeamMem& tm, int wid, int lane) {
    float* const td = tm.tile + kSlots * 4 * kRow;
    float4* const at = reinterpret_cast<float4*>(td + kSlots * kRow);
    int2* const range = reinterpret_cast<int2*>(at + kSlots);
    const int groups = (L.na + kSlots - 1) / kSlots;
    for (int g = wid; g < groups; g += warps) {
        float a[3] = {0.f, 0.f, 0.f}, od[3] = {0.f, 0.f, 0.f}, oob = 0.f;
        int n = 0;
        if (lane < kSlots) {
            const int i = g * kSlots + lane;
            int2 q = make_int2(0, 0);
            int t1 = 0;
            if (i < L.na) {
                const float4 c = m.c[i];
                a[0] = c.x; a[1] = c.y; a[2] = c.z;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const float b = R.gbf[d], e = R.gef[d];
                    if (a[d] < b) { oob += fabsf(a[d] - b); a[d] = b; od[d] = -1.f; }
                    else if (a[d] > e) { oob += fabsf(a[d] - e); a[d] = e; od[d] = 1.f; }
                }
                const int cell = cell_of(R, a[0], a[1], a[2]);
                q = make_int2(__ldg(&R.cell_start[cell]), __ldg(&R.cell_start[cell + 1]));
                t1 = __float_as_int(__ldg(&L.atoms[i].w)) & 0xff;
            }
            n = q.y - q.x;
            at[lane] = make_float4(a[0], a[1], a[2], __int_as_float(t1));
            range[lane] = q;
        }
        n = __reduce_max_sync(0xffffffffu, n);
        __syncwarp();
        const int s = (lane >> 2) < kSlots ? lane >> 2 : 0, c = lane & 3;
        float acc = 0.f;
        int idx[kSlots];  // the tile's neighbours, loaded one tile ahead; -1: none
        auto load_idx = [&](int k0) {
#pragma unroll
            for (int j = 0; j < kSlots; ++j) {
                const int2 q = range[j];
                const int qi = q.x + k0 + lane;
                idx[j] = qi < q.y ? __ldg(&R.cell_list[qi]) : -1;
            }
        };
        load_idx(0);
        for (int k0 = 0; k0 < n; k0 += kNb) {
            // all slots' loads in flight per stage, no branches
            float4 nb[kSlots], tv[kSlots];
            float rem[kSlots];
            bool in[kSlots];
#pragma unroll
            for (int j = 0; j < kSlots; ++j) {
                in[j] = idx[j] >= 0;
                nb[j] = __ldg(&R.rec[max(idx[j], 0)]);  // entry 0 always exists
            }
            if (k0 + kNb < n) load_idx(k0 + kNb);
#pragma unroll
            for (int j = 0; j < kSlots; ++j) {
                const float4 p = at[j];
                const float rx = p.x - nb[j].x, ry = p.y - nb[j].y, rz = p.z - nb[j].z;
                const float r2 = rx * rx + ry * ry + rz * rz;
                const int t1 = __float_as_int(p.w), t2 = int(nb[j].w);
                const int tp = (t1 <= t2) ? t1 + t2 * (t2 + 1) / 2 : t2 + t1 * (t1 + 1) / 2;
                in[j] = in[j] && r2 < 64.f;
                const float rf = in[j] ? 32.f * r2 : 0.f;
                const int i1 = int(rf);
                rem[j] = rf - float(i1);
                nb[j] = make_float4(rx, ry, rz, 0.f);
                tv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in[j]) tv[j] = __ldg(smooth + size_t(tp) * kBins + i1);
            }
#pragma unroll
            for (int j = 0; j < kSlots; ++j) {  // out of reach: all terms zero
                const float e = tv[j].x + rem[j] * (tv[j].z - tv[j].x), dor = tv[j].y + rem[j] * (tv[j].w - tv[j].y);
                float* const row = tm.tile + 4 * j * kRow + lane;
                row[0] = in[j] ? nb[j].x : 0.f;
                row[kRow] = in[j] ? nb[j].y : 0.f;
                row[2 * kRow] = in[j] ? nb[j].z : 0.f;
                row[3 * kRow] = in[j] ? e : 0.f;
                td[j * kRow + lane] = in[j] ? dor : 0.f;
            }
            __syncwarp();
            const int m_here = min(kNb, n - k0);  // rounded up to eights: the rest are zero terms
            const float4* const xr = reinterpret_cast<const float4*>(tm.tile + (4 * s + c) * kRow);
            const float4* const fr = reinterpret_cast<const float4*>(td + s * kRow);
            auto add = [&](float f, float x) { acc = fmaf(c < 3 ? f : 1.f, x, acc); };  // energy: 1 * e; force: derivative * r
            for (int k = 0; k < m_here; k += 8) {
                const float4 x0 = xr[k / 4], x1 = xr[k / 4 + 1], f0 = fr[k / 4], f1 = fr[k / 4 + 1];
                add(f0.x, x0.x); add(f0.y, x0.y); add(f0.z, x0.z); add(f0.w, x0.w);
                add(f1.x, x1.x); add(f1.y, x1.y); add(f1.z, x1.z); add(f1.w, x1.w);
            }
            __syncwarp();
        }
        const float this_e = __shfl_sync(0xffffffffu, acc, lane | 3);
        if (this_e > 0.f) {
            const float tt = v / (v + this_e);
            acc = (c < 3) ? acc * (tt * tt) : acc * tt;
        }
        const float o0 = __shfl_sync(0xffffffffu, od[0], s), o1 = __shfl_sync(0xffffffffu, od[1], s),
                    o2 = __shfl_sync(0xffffffffu, od[2], s), o3 = __shfl_sync(0xffffffffu, oob, s);
        const int i = g * kSlots + s;
        if ((lane >> 2) < kSlots && i < L.na) {
            float* const dst = c == 0 ? m.fx : c == 1 ? m.fy : c == 2 ? m.fz : tm.eatom;
            dst[i] = acc + slope * (c == 0 ? o0 : c == 1 ? o1 : c == 2 ? o2 : o3);
        }
        __syncwarp();
    }
}

// Intra-pair terms of one evaluation, one pair per thread: the pair's capped
// energy and force to tm.pair, the force on the first atom into its
// fixed-point accumulator (integer sums: exact in any order).  Two pairs'
// loads are in flight per thread.
template <int warps>
__device__ __forceinline__ void pair_terms(const LigView& L, const WarpMem& m, const float4* smooth, float v, float fix,
                                           const TeamMem& tm, int tid) {
    constexpr int kStep = 32 * warps;
    int* const qx = reinterpret_cast<int*>(m.ns);
    int* const qy = qx + pad4(L.na);
    int* const qz = qy + pad4(L.na);
    for (int p0 = tid; p0 < L.np; p0 += 2 * kStep) {
        float4 r[2], t[2];
        int a[2];
        bool in[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int p = p0 + j * kStep;
            in[j] = p < L.np;
            const int2 q = in[j] ? __ldg(&L.pairs[p]) : make_int2(0, 0);
            a[j] = VD_DCLAMP(q.x & 0xffff, 0, L.na - 1, kChkPairAtom);
            const float4 ca = m.c[a[j]], cb = m.c[VD_DCLAMP(q.x >> 16, 0, L.na - 1, kChkPairAtom)];
            const float rx = cb.x - ca.x, ry = cb.y - ca.y, rz = cb.z - ca.z;
            const float d = rx * rx + ry * ry + rz * rz;
            const float rf = fminf(32.f * d, 2047.5f);
            const int i = VD_DCLAMP(int(rf), 0, kBins - 2, kChkTableBin);
            r[j] = make_float4(rx, ry, rz, rf - float(i));
            in[j] = in[j] && d < 64.f;
            t[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in[j]) t[j] = __ldg(smooth + size_t(VD_DCLAMP(q.y, 0, kPairTypes - 1, kChkPairType)) * kBins + i);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in[j]) {
                const float w = r[j].w;
                const float e = t[j].x + w * (t[j].z - t[j].x), g = t[j].y + w * (t[j].w - t[j].y);
                const float c = (e > 0.f) ? __fdividef(v, v + e) : 1.f;
                const float gc = g * c * c;
                out = make_float4(gc * r[j].x, gc * r[j].y, gc * r[j].z, e * c);
                atomicAdd(&qx[a[j]], to_fixed(-out.x, fix)); atomicAdd(&qy[a[j]], to_fixed(-out.y, fix));
                atomicAdd(&qz[a[j]], to_fixed(-out.z, fix));
            }
            const int p = p0 + j * kStep;
            if (p < L.np) {
                tm.pair[p] = out.x;
                tm.pair[L.np + p] = out.y;
                tm.pair[2 * L.np + p] = out.z;
                tm.pair[3 * L.np + p] = out.w;
            }
        }
    }
}

// The pair list (sorted by second atom) is 32 segments, one per lane of a
// single-warp evaluation; a run is a stretch of one segment with one second
// atom.  First pairs of the runs to tm.run (tm.run[runs] = pairs).
__device__ __forceinline__ int find_runs(const LigView& L, const TeamMem& tm, int lane) {
    int runs = 0;
    for (int p0 = 0; p0 < L.np; p0 += 32) {
        const int p = p0 + lane;
        bool first = false;
        if (p < L.np) {
            // p starts a segment: some l has l * np / 32 (rounded down) = p
            const int l = (p * 32 + L.np - 1) / L.np;
            first = p == 0 || ((l * L.np) >> 5) == p || (L.pairs[p].x >> 16) != (L.pairs[p - 1].x >> 16);
        }
        const unsigned b = __ballot_sync(0xffffffffu, first);
        if (first) tm.run[runs + __popc(b & ((1u << lane) - 1u))] = uint16_t(p);
        runs += __popc(b);
    }
    if (lane == 0) {
        tm.run[runs] = uint16_t(L.np);
        *tm.runs = runs;
    }
    __syncwarp();
    return runs;
}

// The second atoms' forces: one thread per run and component adds the run's
// forces in list order, then the run to its atom's accumulator.
__device__ __forceinline__ void run_terms(const LigView& L, const WarpMem& m, float fix, const TeamMem& tm, int tid,
                                          int threads) {
    const int n = 3 * *tm.runs;
    for (int j = tid; j < n; j += threads) {
        const int r = j / 3, c = j - 3 * r;
        const int p0 = tm.run[r], p1 = tm.run[r + 1];
        const float* f = tm.pair + c * L.np;
        float b = 0.f;
        for (int p = p0; p < p1; p += 8) {
            float v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = p + k < p1 ? f[p + k] : 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) b += v[k];
        }
        const int atom = VD_DCLAMP(L.pairs[p0].x >> 16, 0, L.na - 1, kChkPairAtom);
        atomicAdd(reinterpret_cast<int*>(m.ns) + c * pad4(L.na) + atom, to_fixed(b, fix));
    }
}

// The energy: lane l takes atoms l, l + 32, .. and segment l of the pair list,
// two pairs at a time.
__device__ __forceinline__ float sum_energy(const LigView& L, const TeamMem& tm, int lane) {
    float e = 0.f;
    for (int i = lane; i < L.na; i += 32) e += tm.eatom[i];
    const float* pe = tm.pair + 3 * L.np;
    const int p1 = ((lane + 1) * L.np) >> 5;
    for (int p = (lane * L.np) >> 5; p < p1; p += 8) {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = p + j < p1 ? pe[p + j] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; j += 2) e += f[j] + f[j + 1];
    }
    return warp_sum(e);
}

__device__ __forceinline__ bool m_out(float v, double b, double e) {
    return v < float(b - 1e-4) || v > float(e + 1e-4);
}

// Barriers of a refinement block: 1, the atoms are placed (or the pose is
// done); 3, all warps: the terms are in shared memory; 2, the second atoms'
// forces are added.  Warp 0 arrives at 1 and waits at 2, the others the other
// way round; every thread takes part in each once per evaluation, and in 1
// once more at the end.
template <int warps, int blocks>
__global__ void __launch_bounds__(32 * warps, blocks) refine_kernel(RefineParams p) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, pose = blockIdx.x;
    const int li = p.pose_lig ? p.pose_lig[pose] : 0;
    if (p.skip_invalid && !(p.e_out[pose] < FLT_MAX)) return;  // the whole block
    const LigView L = lig_view(p.pool, p.lig_off[li]);
    const int n = 6 + L.nt, nc = 7 + L.nt;
    float* base = reinterpret_cast<float*>(smem4);
    SearchMem s;
    s.m = carve(base, L.na, L.nn, L.np, L.nt);
    s.xp = base + warp_floats(L.na, L.nn, L.np, L.nt);
    s.xo = s.xp + pad4(nc);
    float* H = s.xo + pad4(nc);
    float* gc = H + pad4(n * n);
    float* pv = gc + pad4(n);
    float* yv = pv + pad4(n);
    float* mhy = yv + pad4(n);
    TeamMem tm;
    float* team = mhy + pad4(n);
    tm.tile = team + wid * kTileFloats;
    tm.eatom = team + warps * kTileFloats;
    tm.pair = tm.eatom + pad4(L.na);
    tm.run = reinterpret_cast<uint16_t*>(tm.pair + 4 * L.np);
    tm.cmd = reinterpret_cast<int*>(tm.eatom + pad4(L.na) + 4 * L.np + pad4((L.np + 2) / 2));
    tm.slope = reinterpret_cast<float*>(tm.cmd + 1);
    tm.runs = tm.cmd + 2;
    auto terms = [&](float slope) {
        direct_terms<warps>(L, s.m, p.R, p.smooth, 1000.f, slope, tm, wid, lane);
        pair_terms<warps>(L, s.m, p.smooth, 1000.f, p.fix, tm, threadIdx.x);
        __syncwarp();
        if (warps > 1) team_sync<warps>(3);
    };
    if (wid == 0) find_runs(L, tm, lane);
    __syncthreads();
    if (wid > 0) {
        for (;;) {
            team_sync<warps>(1);
            if (*tm.cmd == 0) break;
            terms(*tm.slope);
            run_terms(L, s.m, p.fix, tm, threadIdx.x - 32, 32 * (warps - 1));
            __syncwarp();
            team_arrive<warps>(2);
        }
        return;
    }
    int evals = 0;
    float* x = p.poses + size_t(pose) * p.stride;
    for (int i = lane; i < nc; i += 32) s.m.x[i] = x[i];
    __syncwarp();
    const int max_steps = p.max_steps ? p.max_steps[li] : p.max_steps_default;
    float e = FLT_MAX;
    bool inside = false;
    for (int ramp = 0; ramp < 5; ++ramp) {
        const float slope = 100.f * powf(10.f, 2.f * ramp);
        const auto eval = [&](const SkipArmijo& skip) {
            frames(L, s.m, lane);
            int* const q = reinterpret_cast<int*>(s.m.ns);  // pair-force accumulators start at zero
            const int a4 = pad4(L.na);
            for (int i = lane; i < L.na; i += 32) {
                s.m.c[i] = atom_position(L, s.m, __ldg(&L.atoms[i]));
                q[i] = 0; q[a4 + i] = 0; q[2 * a4 + i] = 0;
            }
            if (lane == 0) {
                *tm.cmd = 1;
                *tm.slope = slope;
            }
            __syncwarp();
            if (warps > 1) team_arrive<warps>(1);
            terms(slope);
            const float sum = sum_energy(L, tm, lane);
            if (warps == 1) run_terms(L, s.m, p.fix, tm, lane, 32);
            __syncwarp();
            if (warps > 1) team_sync<warps>(2);
            if (skip(sum)) return sum;
            adjoint_phases(L, s.m, p.inv_fix, lane);
            return sum;
        };
        e = dense_bfgs(L, s, H, gc, pv, yv, mhy, eval, max_steps, lane, evals);
        kinematics(L, s.m, lane);
        bool ok = true;  // non_cache::within, margin 1e-4
        for (int i = lane; i < L.na; i += 32) {
            if (m_out(s.m.c[i].x, p.R.gb[0], p.R.ge[0]) || m_out(s.m.c[i].y, p.R.gb[1], p.R.ge[1]) ||
                m_out(s.m.c[i].z, p.R.gb[2], p.R.ge[2]))
                ok = false;
        }
        inside = __all_sync(0xffffffffu, ok);
        if (inside) break;
    }
    if (!inside) e = FLT_MAX;
    for (int i = lane; i < nc; i += 32) x[i] = s.m.x[i];
    if (lane == 0) {
        p.e_out[pose] = e;
        if (evals) atomicAdd(p.evals, (unsigned long long)evals);
        *tm.cmd = 0;
    }
    __syncwarp();
    if (warps > 1) team_arrive<warps>(1);
}

// ------------------------------------------------------------ score (double)
struct ScoreParams {
    const float4* pool;
    const int64_t* lig_off;
    const float* poses;         // [n_ligs][20][stride] refined poses
    const float* e_ref;         // [n_ligs][20] refined energies (FLT_MAX = rejected)
    const int32_t* n_in;        // [n_ligs] poses per ligand
    int32_t stride;
    RecView R;
    const double* fastd;        // [153][kBins]
    double w_rot;               // 0.1 * (weights[5] + 1)
    int32_t num_modes;
    double energy_range;
    double min_rmsd;
    vd_dock_result* out;        // [n_ligs]
};

// Heavy-atom coordinates of a pose in double (same frame walk as kinematics).
__device__ void coords_d(const LigView& L, const float* pose, double* nd, double* c, int lane) {
    for (int k = lane; k < L.nn; k += 32) {
        double* a = nd + 8 * k;
        a[0] = 1; a[1] = a[2] = a[3] = 0;
        if (k > 0) {
            const double th = 0.5 * double(pose[7 + k - 1]);
            const double s = sin(th), co = cos(th);
            a[0] = co; a[1] = s * double(L.nodes[k].axis[0]); a[2] = s * double(L.nodes[k].axis[1]);
            a[3] = s * double(L.nodes[k].axis[2]);
        }
    }
    __syncwarp();
    double* fr = nd + 8 * L.nn;  // per node: q[4], o[3]
    const double qr[4] = {pose[3], pose[4], pose[5], pose[6]};
    for (int k = lane; k < L.nn; k += 32) {
        double P[4] = {1, 0, 0, 0}, w[3] = {0, 0, 0};
        if (k > 0) {
            for (int i = 0; i < 4; ++i) P[i] = nd[8 * k + i];
            for (int i = 0; i < 3; ++i) w[i] = L.nodes[k].rel_origin[i];
            int j = L.nodes[k].parent;
            while (j > 0) {
                const double* A = nd + 8 * j;
                // w = rel_origin_j + rot(A) w
                const double tx = A[2] * w[2] - A[3] * w[1] + A[0] * w[0];
                const double ty = A[3] * w[0] - A[1] * w[2] + A[0] * w[1];
                const double tz = A[1] * w[1] - A[2] * w[0] + A[0] * w[2];
                const double r0 = w[0] + 2 * (A[2] * tz - A[3] * ty), r1 = w[1] + 2 * (A[3] * tx - A[1] * tz),
                             r2 = w[2] + 2 * (A[1] * ty - A[2] * tx);
                w[0] = L.nodes[j].rel_origin[0] + r0;
                w[1] = L.nodes[j].rel_origin[1] + r1;
                w[2] = L.nodes[j].rel_origin[2] + r2;
                const double n0 = A[0] * P[0] - A[1] * P[1] - A[2] * P[2] - A[3] * P[3];
                const double n1 = A[0] * P[1] + A[1] * P[0] + A[2] * P[3] - A[3] * P[2];
                const double n2 = A[0] * P[2] - A[1] * P[3] + A[2] * P[0] + A[3] * P[1];
                const double n3 = A[0] * P[3] + A[1] * P[2] - A[2] * P[1] + A[3] * P[0];
                P[0] = n0; P[1] = n1; P[2] = n2; P[3] = n3;
                j = L.nodes[j].parent;
            }
        }
        double q[4] = {qr[0] * P[0] - qr[1] * P[1] - qr[2] * P[2] - qr[3] * P[3],
                       qr[0] * P[1] + qr[1] * P[0] + qr[2] * P[3] - qr[3] * P[2],
                       qr[0] * P[2] - qr[1] * P[3] + qr[2] * P[0] + qr[3] * P[1],
                       qr[0] * P[3] + qr[1] * P[2] - qr[2] * P[1] + qr[3] * P[0]};
        const double inv = 1.0 / sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
        for (int i = 0; i < 4; ++i) q[i] *= inv;
        const double tx = qr[2] * w[2] - qr[3] * w[1] + qr[0] * w[0];
        const double ty = qr[3] * w[0] - qr[1] * w[2] + qr[0] * w[1];
        const double tz = qr[1] * w[1] - qr[2] * w[0] + qr[0] * w[2];
        double* f = fr + 8 * k;
        for (int i = 0; i < 4; ++i) f[i] = q[i];
        f[4] = double(pose[0]) + w[0] + 2 * (qr[2] * tz - qr[3] * ty);
        f[5] = double(pose[1]) + w[1] + 2 * (qr[3] * tx - qr[1] * tz);
        f[6] = double(pose[2]) + w[2] + 2 * (qr[1] * ty - qr[2] * tx);
    }
    __syncwarp();
    for (int i = lane; i < L.na; i += 32) {
        const float4 a = L.atoms[i];
        const int k = (__float_as_int(a.w) >> 8) & 0xff;
        const double* f = fr + 8 * k;
        const double v[3] = {a.x, a.y, a.z};
        const double tx = f[2] * v[2] - f[3] * v[1] + f[0] * v[0];
        const double ty = f[3] * v[0] - f[1] * v[2] + f[0] * v[1];
        const double tz = f[1] * v[1] - f[2] * v[0] + f[0] * v[2];
        c[3 * i] = f[4] + v[0] + 2 * (f[2] * tz - f[3] * ty);
        c[3 * i + 1] = f[5] + v[1] + 2 * (f[3] * tx - f[1] * tz);
        c[3 * i + 2] = f[6] + v[2] + 2 * (f[1] * ty - f[2] * tx);
    }
    __syncwarp();
}

__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// model.cpp:1206-1219 (eval_interacting_pairs, eval_fast, curl 1000): this
// lane's share of the pairs tid, tid + step, ..
__device__ __forceinline__ double intra_fast(const LigView& L, const double* c, const double* fastd, int tid, int step) {
    double e = 0;
#pragma unroll 4
    for (int p = tid; p < L.np; p += step) {
        const int2 pr = __ldg(&L.pairs[p]);
        const int a = pr.x & 0xffff, b = pr.x >> 16;
        const double dx = c[3 * a] - c[3 * b], dy = c[3 * a + 1] - c[3 * b + 1], dz = c[3 * a + 2] - c[3 * b + 2];
        const double r2 = (dx * dx + dy * dy) + dz * dz;
        if (r2 < 64.0) {
            double t = __ldg(&fastd[size_t(pr.y) * kBins + int(32.0 * r2)]);
            if (t > 0) t *= 1000.0 / (1000.0 + t);
            e += t;
        }
    }
    return e;
}

// non_cache.cpp:20-55 (non_cache::eval, eval_fast, curl 1000, slope 1e6) of the
// atom groups g, g + step, ..: four atoms at a time, lanes over a cell's
// receptor atoms (a lane walking its own atom's list alone paid three dependent
// loads per neighbour).  Same value in every lane.
__device__ __forceinline__ double inter_fast(const LigView& L, const RecView& R, const double* c, const double* fastd,
                                             int g, int step, int lane) {
    double e = 0;
    for (int i0 = 4 * g; i0 < L.na; i0 += 4 * step) {
        double a[4][3], oob[4], sum[4];
        int t1[4], q0[4], q1[4], longest = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = min(i0 + j, L.na - 1);
            t1[j] = __float_as_int(__ldg(&L.atoms[i].w)) & 0xff;
            oob[j] = sum[j] = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                a[j][d] = c[3 * i + d];
                if (a[j][d] < R.gb[d]) { oob[j] += fabs(a[j][d] - R.gb[d]); a[j][d] = R.gb[d]; }
                else if (a[j][d] > R.ge[d]) { oob[j] += fabs(a[j][d] - R.ge[d]); a[j][d] = R.ge[d]; }
            }
            const int ce = cell_of(R, a[j][0], a[j][1], a[j][2]);
            q0[j] = __ldg(&R.cell_start[ce]);
            q1[j] = __ldg(&R.cell_start[ce + 1]);
            longest = max(longest, q1[j] - q0[j]);
        }
        for (int k = lane; k < longest; k += 32) {
            int idx[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) idx[j] = q0[j] + k < q1[j] ? __ldg(&R.cell_list[q0[j] + k]) : -1;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double4 b = R.recd[max(idx[j], 0)];  // entry 0 always exists
                const double rx = a[j][0] - b.x, ry = a[j][1] - b.y, rz = a[j][2] - b.z;
                const double r2 = (rx * rx + ry * ry) + rz * rz;
                if (idx[j] >= 0 && r2 < 64.0) {
                    const int t2 = int(b.w);
                    const int tp = (t1[j] <= t2) ? t1[j] + t2 * (t2 + 1) / 2 : t2 + t1[j] * (t1[j] + 1) / 2;
                    sum[j] += __ldg(&fastd[size_t(tp) * kBins + int(32.0 * r2)]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            double this_e = warp_sum_d(sum[j]);
            if (this_e > 0) this_e *= 1000.0 / (1000.0 + this_e);
            if (i0 + j < L.na) e += this_e + oob[j] * 1e6;
        }
    }
    return e;
}

// Kept chain results -> refinement buffer ([ligand][20] slots).
__global__ void gather_kernel(const int32_t* kept, const float* conf, const float* e, int stride, int n_slots,
                              float* rp, float* re) {
    const int slot = blockIdx.x;
    if (slot >= n_slots) return;
    const int item = kept[slot];
    for (int i = threadIdx.x; i < stride; i += blockDim.x)
        rp[size_t(slot) * stride + i] = item >= 0 ? conf[size_t(item) * stride + i] : 0.f;
    if (threadIdx.x == 0) re[slot] = item >= 0 ? e[item] : FLT_MAX;
}

// model.cpp:1485-1523: RMSD upper bound (each heavy atom to the same atom)
// and lower bound (each heavy atom to the nearest atom of the same element,
// the larger of the two directions) between heavy-atom coordinate sets a and
// b ([na][3], taken as floats); sums in double.  Same value in every lane.
template <class T>
__device__ void rmsd_bounds(const LigView& L, const T* pa, const T* pb, int lane, double& lb, double& ub) {
    const auto a = [pa](int k) { return float(pa[k]); };
    const auto b = [pb](int k) { return float(pb[k]); };
    double su = 0, s1 = 0, s2 = 0;
    for (int i = lane; i < L.na; i += 32) {
        const int ei = (__float_as_int(L.atoms[i].w) >> 16) & 0xff;
        double d2 = 0, m1 = DBL_MAX, m2 = DBL_MAX;
        for (int d = 0; d < 3; ++d) d2 += double(a(3 * i + d) - b(3 * i + d)) * double(a(3 * i + d) - b(3 * i + d));
        for (int q = 0; q < L.na; ++q) {
            if (((__float_as_int(L.atoms[q].w) >> 16) & 0xff) != ei) continue;
            double t1 = 0, t2 = 0;
            for (int d = 0; d < 3; ++d) {
                t1 += double(a(3 * i + d) - b(3 * q + d)) * double(a(3 * i + d) - b(3 * q + d));
                t2 += double(b(3 * i + d) - a(3 * q + d)) * double(b(3 * i + d) - a(3 * q + d));
            }
            m1 = fmin(m1, t1);
            m2 = fmin(m2, t2);
        }
        su += d2; s1 += m1; s2 += m2;
    }
    su = warp_sum_d(su); s1 = warp_sum_d(s1); s2 = warp_sum_d(s2);
    ub = sqrt(su / L.na);
    lb = fmax(sqrt(s1 / L.na), sqrt(s2 / L.na));
}

// Doubles one warp needs for a pose: body frames, then its coordinates.
__host__ __device__ inline int pose_doubles(int na, int nn) { return 16 * nn + 3 * na; }

// RMSD bounds of poses to pose 0 (vd_rmsd_bounds): heavy-atom coordinates in
// double, taken as floats as the output stage does.  A warp per pose, and one
// more per block for pose 0.  20 poses of 45 atoms, B200: 278 us with one
// warp for all poses, 20 us.
constexpr int kRmsdWarps = 4;
__global__ void __launch_bounds__(32 * (kRmsdWarps + 1)) rmsd_poses_kernel(const float4* pool, const int64_t* off,
                                                                           const float* poses, int n, int stride,
                                                                           double* out) {
    extern __shared__ double smemd[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const LigView L = lig_view(pool, off[0]);
    const int per = pose_doubles(L.na, L.nn);
    const int i = wid < kRmsdWarps ? int(blockIdx.x) * kRmsdWarps + wid : 0;
    double* nd = smemd + wid * per;
    if (i < n) coords_d(L, poses + size_t(i) * stride, nd, nd + 16 * L.nn, lane);
    __syncthreads();
    if (wid == kRmsdWarps || i >= n) return;
    double lb, ub;
    rmsd_bounds(L, nd + 16 * L.nn, smemd + kRmsdWarps * per + 16 * L.nn, lane, lb, ub);
    if (lane == 0) {
        out[2 * i] = lb;
        out[2 * i + 1] = ub;
    }
}

// Receptor-ligand and intramolecular energy of a pose (vd_score; the caller
// relates them to pose 0's).  A block per pose: warp 0 places the atoms, all
// warps share them and the pairs.  20 poses of 45 atoms, B200: 1,386 us with
// one warp for all poses, 24 us (a launch, a pose placement in FP64, one round of
// neighbours).
constexpr int kScoreWarps = 8;
__global__ void __launch_bounds__(32 * kScoreWarps) score_poses_kernel(const float4* pool, const int64_t* off,
                                                                       const float* poses, int stride, RecView R,
                                                                       const double* fastd, double* out) {
    extern __shared__ double smemd[];
    __shared__ double part[2][kScoreWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, i = blockIdx.x;
    const LigView L = lig_view(pool, off[0]);
    double* c = smemd + 16 * L.nn;
    if (wid == 0) coords_d(L, poses + size_t(i) * stride, smemd, c, lane);
    __syncthreads();
    const double inter = inter_fast(L, R, c, fastd, wid, kScoreWarps, lane);
    const double intra = warp_sum_d(intra_fast(L, c, fastd, threadIdx.x, 32 * kScoreWarps));
    if (lane == 0) {
        part[0][wid] = inter;
        part[1][wid] = intra;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double e = 0;
        for (int w = 0; w < kScoreWarps; ++w) e += part[threadIdx.x][w];
        out[2 * i + threadIdx.x] = e;
    }
}

// Final scores, order, redundancy and RMSD bounds of a ligand's refined poses:
// a block per ligand, a warp per pose, every pose's coordinates kept in shared
// memory.  One warp going through them took 938 us for a 31-atom ligand's 20
// poses, latency all of it; 88 us.
__global__ void __launch_bounds__(32 * VD_MAX_MODES) score_kernel(ScoreParams p) {
    extern __shared__ double smemd[];
    __shared__ int order[VD_MAX_MODES], kept[VD_MAX_MODES], s_nk;
    __shared__ double adj[VD_MAX_MODES], s_intra[VD_MAX_MODES];
    __shared__ unsigned near[VD_MAX_MODES];  // bit q: within min_rmsd of the pose q places up the order
    const int li = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const LigView L = lig_view(p.pool, p.lig_off[li]);
    const int per = pose_doubles(L.na, L.nn);
    const auto coords = [&](int i) { return smemd + size_t(i) * per + 16 * L.nn; };
    const int n = p.n_in[li];
    const float* poses = p.poses + size_t(li) * VD_MAX_MODES * p.stride;
    const float* er = p.e_ref + size_t(li) * VD_MAX_MODES;
    vd_dock_result* out = p.out + li;
    // the best refined pose: the first of a stable ascending sort, which no
    // pose passes a NaN in
    int best = 0;
    for (int i = 0; i < n; ++i) {
        if (!(er[i] == er[i])) break;
        if (er[i] < er[best]) best = i;
    }
    const bool valid = w < n && er[w] < FLT_MAX;
    double e = 0;
    if (valid || (w == best && n > 0)) {
        coords_d(L, poses + size_t(w) * p.stride, smemd + size_t(w) * per, coords(w), lane);
        const double intra = warp_sum_d(intra_fast(L, coords(w), p.fastd, lane, 32));
        if (lane == 0) s_intra[w] = intra;
        if (valid) e = inter_fast(L, p.R, coords(w), p.fastd, 0, 1, lane) + intra;
    }
    __syncthreads();
    if (w < n && lane == 0) {
        double v = DBL_MAX;
        if (valid) {
            const double x = e - s_intra[best], y = 1 + p.w_rot * double(L.num_tors) / 5.0;
            v = (fabs(x) < DBL_EPSILON) ? 0.0 : x / y;  // smooth_div, everything.cpp:232-236
        }
        adj[w] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < n; ++i) order[i] = i;
        for (int i = 1; i < n; ++i)  // stable insertion sort
            for (int j = i; j > 0 && adj[order[j]] < adj[order[j - 1]]; --j) {
                const int t = order[j]; order[j] = order[j - 1]; order[j - 1] = t;
            }
    }
    __syncthreads();
    if (w < n && adj[order[w]] < 0.1 * DBL_MAX) {
        const double* c = coords(order[w]);
        unsigned bits = 0;
        for (int j = 0; j < w; ++j) {
            if (!(adj[order[j]] < 0.1 * DBL_MAX)) continue;
            const double* k = coords(order[j]);
            double acc = 0;
            for (int a = lane; a < L.na; a += 32)
                for (int d = 0; d < 3; ++d) {
                    const double x = c[3 * a + d] - double(float(k[3 * a + d]));
                    acc += x * x;
                }
            acc = warp_sum_d(acc);
            if (sqrt(acc / L.na) < p.min_rmsd) bits |= 1u << j;
        }
        if (lane == 0) near[w] = bits;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int nk = 0;  // remove_redundant (main.cpp:172-178) then the mode cut
        unsigned taken = 0;
        for (int r = 0; r < n; ++r) {
            const int i = order[r];
            if (!(adj[i] < 0.1 * DBL_MAX)) break;
            if (nk >= p.num_modes) break;
            if (nk > 0 && adj[i] > adj[kept[0]] + p.energy_range) break;
            if (near[r] & taken) continue;
            taken |= 1u << r;
            kept[nk++] = i;
        }
        s_nk = nk;
        out->n_modes = nk;
        out->ntors = L.nt;
    }
    __syncthreads();
    // outputs with RMSD bounds to mode 1 (model.cpp:1485-1523)
    if (w < s_nk) {
        double lb, ub;
        rmsd_bounds(L, coords(kept[w]), coords(kept[0]), lane, lb, ub);
        const int i = kept[w];
        if (lane == 0) {
            out->energy[w] = float(adj[i]);
            out->rmsd_ub[w] = float(ub);
            out->rmsd_lb[w] = float(lb);
        }
        for (int q = lane; q < 7 + L.nt; q += 32) out->pose[w][q] = poses[size_t(i) * p.stride + q];
    }
}

}  // namespace
}  // namespace vd

namespace vd {

// szv_grid over the box (szv_grid.cpp:28-74, 120-131), uploaded once per
// receptor and box.
vd_status ensure_receptor_cells(Ctx* c) {
    if (c->rec_dev_ready) return VD_OK;
    VD_CHECK(c->has_box, VD_ERR_ARG, "no box set");
    const GridGeom& g = c->geom;
    double init[3], range[3], end[3];
    int dim[3];
    for (int d = 0; d < 3; ++d) {
        init[d] = g.begin[d];
        end[d] = g.end[d];
        const int n_int = int((g.end[d] - g.begin[d]) / 3);
        dim[d] = n_int < 1 ? 1 : n_int;
    }
    for (int d = 0; d < 3; ++d) range[d] = end[d] - init[d];
    auto brick = [](const double* b, const double* e, const double* v) {
        double d2 = 0;
        for (int i = 0; i < 3; ++i) {
            const double q = (v[i] <= b[i]) ? b[i] : ((v[i] >= e[i]) ? e[i] : v[i]);
            d2 += (q - v[i]) * (q - v[i]);
        }
        return d2;
    };
    std::vector<int> rel;
    const int n_rec = int(c->rec_xs.size());
    for (int i = 0; i < n_rec; ++i)
        if (c->rec_xs[i] >= 0 && brick(init, end, &c->rec_xyz[3 * size_t(i)]) < kCutoff2) rel.push_back(i);
    // A cell's list reaches a little further than the cutoff, so that a point
    // that rounding puts into the cell next to its own (cell_of) still finds
    // every atom within 8 A there.
    double far = 0;
    for (int d = 0; d < 3; ++d) far = std::max({far, std::fabs(init[d]), std::fabs(end[d])});
    const double margin = 1e-6 + 1e-12 * far, reach2 = (8.0 + margin) * (8.0 + margin);
    const int ncell = dim[0] * dim[1] * dim[2];
    std::vector<std::vector<int>> cells(ncell);
    auto coord = [&](int d, int i) { return init[d] + range[d] * i / dim[d]; };
    for (int r = 0; r < int(rel.size()); ++r) {
        const double* a = &c->rec_xyz[3 * size_t(rel[r])];
        int lo[3], hi[3];
        for (int d = 0; d < 3; ++d) {  // candidate cells within the cutoff, then the exact test
            lo[d] = std::max(0, int(std::floor((a[d] - 8.0 - margin - init[d]) * dim[d] / range[d])) - 1);
            hi[d] = std::min(dim[d] - 1, int(std::floor((a[d] + 8.0 + margin - init[d]) * dim[d] / range[d])) + 1);
        }
        for (int z = lo[2]; z <= hi[2]; ++z)
            for (int y = lo[1]; y <= hi[1]; ++y)
                for (int x = lo[0]; x <= hi[0]; ++x) {
                    const double b[3] = {coord(0, x), coord(1, y), coord(2, z)};
                    const double e[3] = {coord(0, x + 1), coord(1, y + 1), coord(2, z + 1)};
                    if (brick(b, e, a) < reach2) cells[x + dim[0] * (y + dim[1] * z)].push_back(r);
                }
    }
    std::vector<int32_t> start(ncell + 1, 0), list;
    for (int i = 0; i < ncell; ++i) {
        start[i + 1] = start[i] + int(cells[i].size());
        list.insert(list.end(), cells[i].begin(), cells[i].end());
    }
    std::vector<float4> rf(std::max<size_t>(1, rel.size()));
    std::vector<double4> rd(std::max<size_t>(1, rel.size()));
    for (size_t r = 0; r < rel.size(); ++r) {
        const double* a = &c->rec_xyz[3 * size_t(rel[r])];
        rf[r] = make_float4(float(a[0]), float(a[1]), float(a[2]), float(c->rec_xs[rel[r]]));
        rd[r] = make_double4(a[0], a[1], a[2], double(c->rec_xs[rel[r]]));
    }
    dev_release(*c, c->d_rec);
    dev_release(*c, c->d_recd);
    dev_release(*c, c->d_cell_start);
    dev_release(*c, c->d_cell_list);
    vd_status st = dev_alloc(*c, &c->d_rec, rf.size() * sizeof(float4), "receptor cells");
    if (st == VD_OK) st = dev_alloc(*c, &c->d_recd, rd.size() * sizeof(double4), "receptor cells");
    if (st == VD_OK) st = dev_alloc(*c, &c->d_cell_start, start.size() * sizeof(int32_t), "receptor cells");
    if (st == VD_OK)
        st = dev_alloc(*c, &c->d_cell_list, std::max<size_t>(1, list.size()) * sizeof(int32_t), "receptor cells");
    if (st != VD_OK) {
        dev_release(*c, c->d_rec);
        dev_release(*c, c->d_recd);
        dev_release(*c, c->d_cell_start);
        dev_release(*c, c->d_cell_list);
        return st;
    }
    VD_CUDA(cudaMemcpy(c->d_rec, rf.data(), rf.size() * sizeof(float4), cudaMemcpyHostToDevice));
    VD_CUDA(cudaMemcpy(c->d_recd, rd.data(), rd.size() * sizeof(double4), cudaMemcpyHostToDevice));
    VD_CUDA(cudaMemcpy(c->d_cell_start, start.data(), start.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    if (!list.empty())
        VD_CUDA(cudaMemcpy(c->d_cell_list, list.data(), list.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
    for (int d = 0; d < 3; ++d) {
        c->cell_dim[d] = dim[d];
        c->cell_init[d] = init[d];
        c->cell_range[d] = range[d];
    }
    c->n_rec_dev = int(rel.size());
    c->rec_dev_ready = true;
    return VD_OK;
}

namespace {

RecView rec_view(const Ctx& c) {
    RecView R;
    R.rec = c.d_rec;
    R.recd = c.d_recd;
    R.cell_start = c.d_cell_start;
    R.cell_list = c.d_cell_list;
    for (int d = 0; d < 3; ++d) {
        R.init[d] = c.cell_init[d];
        R.per[d] = c.cell_dim[d] / c.cell_range[d];
        R.dim[d] = c.cell_dim[d];
        R.gbf[d] = float(c.geom.begin[d]);
        R.gef[d] = float(c.geom.end[d]);
        R.gb[d] = c.geom.begin[d];
        R.ge[d] = c.geom.end[d];
    }
    return R;
}

// Shared-memory floats of one pose's refinement block, without its tiles.
int refine_floats(const HostLigand& L) {
    const int n = 6 + L.h.ntors, nc = 7 + L.h.ntors;
    return lig_warp_floats(L) + 2 * pad4(nc) + pad4(n * n) + 4 * pad4(n) + team_floats(0, L.h.n_atoms, L.h.n_pairs);
}

// Refinement of `poses` poses of `atoms` heavy atoms (on average): kernel,
// threads and shared memory.  Few poses take 16 warps each, for their latency;
// more share the SMs on 8 (3 blocks per SM), or 4 where an evaluation is short,
// and thousands of small ones run a warp each.  The poses do not depend on it.
// ms with 16 / 8 / 4 / 1 warps, in a 4,000-atom receptor, and as it was with a
// warp per pose and four poses per block:
//   10 atoms / 1 torsion: 148 poses 0.26 / 0.28 / 0.26 / 0.43 (0.65), 1,500 1.01 / 0.89 /
//     0.78 / 1.14 (1.43), 10,000 4.81 / 3.05 / 2.24 / 1.94 (2.47)
//   24 / 5: 600 0.97 / 0.99 / 1.27 / 2.76 (2.59), 1,500 1.52 / 1.19 / 1.34 / 2.57 (2.26),
//     5,000 3.97 / 2.63 / 2.72 / 3.41 (3.26), 10,000 7.19 / 4.34 / 4.20 / 3.78 (3.87)
//   45 / 12: 1,000 2.14 / 2.24 / 2.54 / 7.04 (6.23), 1,500 2.72 / 2.70 / 3.10 / 8.49 (7.63),
//     10,000 12.4 / 9.2 / 9.2 / 15.5 (14.1)
struct RefineLaunch {
    void (*kernel)(RefineParams) = nullptr;
    int threads = 0;
    size_t smem = 0;
};
vd_status refine_launch(Ctx& c, int poses, double atoms, int floats, RefineLaunch& r) {
    const double per_sm = double(poses) / c.sms;
    const int warps = atoms <= 16   ? (per_sm > 30 ? 1 : per_sm > 2 ? 4 : 16)
                      : atoms <= 28 ? (per_sm > 60 ? 1 : per_sm > 40 ? 4 : per_sm > 6 ? 8 : 16)
                                    : (per_sm > 10 ? 8 : 16);
    r.kernel = warps == 16 ? refine_kernel<16, 1> : warps == 8 ? refine_kernel<8, 3> : warps == 4 ? refine_kernel<4, 5> : refine_kernel<1, 16>;
    r.threads = 32 * warps;
    r.smem = size_t(floats + warps * kTileFloats) * 4;
    VD_CHECK(r.smem <= 227 * 1024, VD_ERR_CAPACITY, "refine kernel shared memory exceeds 227 KB");
    VD_CUDA(set_launch(c, r.kernel, 0, r.smem));
    return VD_OK;
}

inline size_t al256(size_t b) { return (b + 255) & ~size_t(255); }

// Host side of cluster -> gather -> refine -> score for the ligands of one
// dock launch: parameters, device layout in the dock's extra scratch
// (params: off | prefix | steps | pose ligand | n_in, then kept poses and
// results) and the kernel launches; no stream operation.
struct PostPlan {
    std::vector<unsigned char> h_params;
    void* d_params = nullptr;
    vd_dock_result* d_out = nullptr;
    int n = 0;
    std::function<cudaError_t(cudaStream_t)> launch;
};

vd_status prepare_post(Ctx& c, const std::vector<int>& ligs, const vd_search_params& sp, const DockBuffers& db,
                       PostPlan& pp) {
    vd_status st = ensure_receptor_cells(&c);
    if (st != VD_OK) return st;
    const int n = int(ligs.size());
    int max_chains = 0, max_wf = 0, max_rwf = 0, max_na = 0, max_nn = 0;
    std::vector<int64_t> off(n);
    std::vector<int32_t> steps(n), depth(n);
    for (int i = 0; i < n; ++i) {
        const HostLigand& L = c.ligs[ligs[i]];
        off[i] = L.pool_offset;
        search_defaults(L, sp, depth[i], steps[i]);
        max_chains = std::max(max_chains, db.prefix[i + 1] - db.prefix[i]);
        max_wf = std::max(max_wf, lig_warp_floats(L));
        max_rwf = std::max(max_rwf, refine_floats(L));
        max_na = std::max(max_na, L.h.n_atoms);
        max_nn = std::max(max_nn, L.h.n_nodes);
    }
    int sort_n = 2;  // >= 2: the warp's arrays after the 8-byte keys start 16-byte aligned
    while (sort_n < max_chains) sort_n <<= 1;
    VD_CHECK(sort_n <= 16384, VD_ERR_CAPACITY, "more than 16384 chains per ligand");
    const int max_kept = std::min(VD_MAX_MODES, max_chains);
    std::vector<int32_t> plig(size_t(n) * VD_MAX_MODES), nin(n, max_kept);
    for (int i = 0; i < n * VD_MAX_MODES; ++i) plig[i] = i / VD_MAX_MODES;
    // parameter arrays (host), mirrored at the start of the extra scratch
    size_t o = 0;
    const size_t b_par = al256(n * sizeof(int64_t)) + al256((n + 1) * sizeof(int32_t)) + al256(n * sizeof(int32_t)) +
                         al256(plig.size() * sizeof(int32_t)) + al256(n * sizeof(int32_t));
    pp.h_params.assign(b_par, 0);
    char* s = db.d_extra;
    pp.d_params = s;
    auto put = [&](const void* src, size_t bytes) {
        std::memcpy(pp.h_params.data() + o, src, bytes);
        char* d = s + o;
        o += al256(bytes);
        return d;
    };
    const int64_t* d_off = reinterpret_cast<const int64_t*>(put(off.data(), n * sizeof(int64_t)));
    const int32_t* d_pre = reinterpret_cast<const int32_t*>(put(db.prefix.data(), (n + 1) * sizeof(int32_t)));
    const int32_t* d_steps = reinterpret_cast<const int32_t*>(put(steps.data(), n * sizeof(int32_t)));
    const int32_t* d_plig = reinterpret_cast<const int32_t*>(put(plig.data(), plig.size() * sizeof(int32_t)));
    const int32_t* d_nin = reinterpret_cast<const int32_t*>(put(nin.data(), n * sizeof(int32_t)));
    s += b_par;
    int32_t* d_kept = reinterpret_cast<int32_t*>(s); s += al256(size_t(n) * VD_MAX_MODES * sizeof(int32_t));
    float* d_rp = reinterpret_cast<float*>(s); s += al256(size_t(n) * VD_MAX_MODES * db.stride * sizeof(float));
    float* d_re = reinterpret_cast<float*>(s); s += al256(size_t(n) * VD_MAX_MODES * sizeof(float));
    vd_dock_result* d_out = reinterpret_cast<vd_dock_result*>(s);
    pp.d_out = d_out;
    pp.n = n;
    // cluster
    ClusterParams cp{};
    cp.pool = c.d_pool;
    cp.lig_off = d_off;
    cp.prefix = d_pre;
    cp.conf = db.d_conf;
    cp.e = db.d_e;
    cp.stride = db.stride;
    cp.min_rmsd = float(sp.min_rmsd > 0 ? sp.min_rmsd : 1.0);
    cp.max_keep = VD_MAX_MODES;
    cp.kept = d_kept;
    cp.sort_n = sort_n;
    cp.warp_floats = max_wf;
    // as many candidates at a time as there are chains and the shared memory left holds
    const size_t smem_c1 = size_t(sort_n) * 8 + size_t(VD_MAX_MODES) * 3 * max_na * 4, b_wf = size_t(max_wf) * 4;
    VD_CHECK(smem_c1 + b_wf <= 227 * 1024, VD_ERR_CAPACITY, "cluster kernel shared memory exceeds 227 KB");
    cp.warps = int(std::min<size_t>(kClusterThreads / 32, (227 * 1024 - 64 - smem_c1) / b_wf));
    cp.warps = std::max(1, std::min(cp.warps, max_chains));
    const size_t smem_c = smem_c1 + cp.warps * b_wf;
    const int threads_c = std::max(32 * cp.warps, std::min(kClusterThreads, sort_n / 2));
    VD_CUDA(set_launch(c, cluster_kernel, 0, smem_c, 64));
    // refine
    const bool refine = sp.refine != 0;
    RefineParams rp{};
    RefineLaunch rl;
    if (refine) {
        rp.pool = c.d_pool;
        rp.lig_off = d_off;
        rp.pose_lig = d_plig;
        rp.poses = d_rp;
        rp.e_out = d_re;
        rp.stride = db.stride;
        rp.n_poses = n * VD_MAX_MODES;
        rp.max_steps = d_steps;
        rp.R = rec_view(c);
        rp.smooth = c.d_smooth;
        rp.fix = c.fix_scale;
        rp.inv_fix = 1.f / c.fix_scale;
        rp.evals = reinterpret_cast<unsigned long long*>(c.d_counter + 4);
        rp.skip_invalid = 1;
        int poses = 0;
        double atoms = 0;
        for (int i = 0; i < n; ++i) {
            const int kept = std::min(VD_MAX_MODES, db.prefix[i + 1] - db.prefix[i]);
            poses += kept;
            atoms += double(kept) * c.ligs[ligs[i]].h.n_atoms;
        }
        if ((st = refine_launch(c, poses, atoms / poses, max_rwf, rl)) != VD_OK) return st;
    }
    // score
    ScoreParams sc{};
    sc.pool = c.d_pool;
    sc.lig_off = d_off;
    sc.poses = d_rp;
    sc.e_ref = d_re;
    sc.n_in = d_nin;
    sc.stride = db.stride;
    sc.R = rec_view(c);
    sc.fastd = c.d_fastd;
    sc.w_rot = 0.1 * (c.weights[5] + 1);
    sc.num_modes = std::max(1, std::min(VD_MAX_MODES, sp.num_modes > 0 ? sp.num_modes : 9));
    sc.energy_range = sp.energy_range > 0 ? sp.energy_range : 3.0;
    sc.min_rmsd = 1.0;
    sc.out = d_out;
    const size_t smem_s = size_t(max_kept) * pose_doubles(max_na, max_nn) * 8;
    VD_CHECK(smem_s <= 226 * 1024, VD_ERR_CAPACITY, "score kernel shared memory exceeds 226 KB");
    VD_CUDA(set_launch(c, score_kernel, 0, smem_s, 1024));
    const int stride = db.stride;
    const float* conf = db.d_conf;
    const float* e = db.d_e;
    pp.launch = [=](cudaStream_t stream) {
        cluster_kernel<<<n, threads_c, smem_c, stream>>>(cp);
        // gather kept poses (missing slots get e = FLT_MAX)
        gather_kernel<<<n * VD_MAX_MODES, 64, 0, stream>>>(d_kept, conf, e, stride, n * VD_MAX_MODES, d_rp, d_re);
        if (refine) rl.kernel<<<n * VD_MAX_MODES, rl.threads, rl.smem, stream>>>(rp);
        score_kernel<<<n, 32 * max_kept, smem_s, stream>>>(sc);
        return cudaGetLastError();
    };
    return VD_OK;
}

// Stream side: parameter upload, the kernels (ending at c.ev2), the results
// to out (host, pinned for graph capture).
vd_status enqueue_post(Ctx& c, const PostPlan& pp, const void* params_src, vd_dock_result* out,
                       cudaStream_t stream) {
    VD_CUDA(cudaMemcpyAsync(pp.d_params, params_src, pp.h_params.size(), cudaMemcpyHostToDevice, stream));
    VD_CUDA(pp.launch(stream));
    VD_CUDA(record_event(c.ev2, stream));
    VD_CUDA(cudaMemcpyAsync(out, pp.d_out, pp.n * sizeof(vd_dock_result), cudaMemcpyDeviceToHost, stream));
    return VD_OK;
}

// Ends a stream capture left open by an early return.
struct CaptureGuard {
    cudaStream_t s;
    bool open;
    ~CaptureGuard() {
        if (open) {
            cudaGraph_t g = nullptr;
            cudaStreamEndCapture(s, &g);
            if (g) cudaGraphDestroy(g);
        }
    }
};

}  // namespace

size_t post_scratch_bytes(int n_ligs, int stride) {
    return al256(n_ligs * 8) + al256((n_ligs + 1) * 4) + 3 * al256(size_t(n_ligs) * VD_MAX_MODES * 4) +
           2 * al256(n_ligs * 4) + al256(size_t(n_ligs) * VD_MAX_MODES * stride * 4) +
           al256(size_t(n_ligs) * VD_MAX_MODES * 4) + al256(n_ligs * sizeof(vd_dock_result)) + 1024;
}

// Docking of a ligand list followed by the post-processing.  The batched
// (persistent) form records the whole sequence -- parameter uploads from a
// pinned stage, the docking kernel, cluster / gather / refine / score and
// the result download -- into one CUDA graph, updated in place when the
// next call records the same topology, and submits it with one launch; the
// plain form issues the same operations directly, one ligand per launch.
vd_status dock_pipeline(Ctx& c, const std::vector<int>& ligs, const vd_search_params& sp, bool persistent,
                        vd_dock_result* out) {
    VD_CUDA(cudaSetDevice(c.device));
    for (int l : ligs) VD_CHECK(l >= 0 && l < int(c.ligs.size()), VD_ERR_ARG, "bad ligand id");
    int max_nt = 0;
    for (int l : ligs) max_nt = std::max(max_nt, c.ligs[l].h.ntors);
    const int n = int(ligs.size());
    DockBuffers db;
    db.extra_bytes = post_scratch_bytes(n, 7 + max_nt);
    vd_status st = prepare_dock(c, ligs, sp, persistent, db);
    if (st != VD_OK) return st;
    PostPlan pp;
    st = prepare_post(c, ligs, sp, db, pp);
    if (st != VD_OK) return st;
    // stage: [dock params | post params | results | counters]; pinned for the
    // recorded form, which needs it, plain host memory for the direct one (a
    // few KB; allocating pinned memory took 4 ms of a context's first call)
    const size_t b_dp = al256(db.h_params.size()), b_pp = al256(pp.h_params.size());
    const size_t b_res = al256(n * sizeof(vd_dock_result)), b_cnt = al256((2 + n) * sizeof(unsigned long long));
    std::vector<unsigned char> local;
    if (persistent) {
        st = ensure_host_stage(&c, b_dp + b_pp + b_res + b_cnt);
        if (st != VD_OK) return st;
    } else {
        local.resize(b_dp + b_pp + b_res + b_cnt + 256);
    }
    unsigned char* hs = persistent ? static_cast<unsigned char*>(c.h_stage)
                                   : local.data() + (-reinterpret_cast<uintptr_t>(local.data()) & 255);
    std::memcpy(hs, db.h_params.data(), db.h_params.size());
    std::memcpy(hs + b_dp, pp.h_params.data(), pp.h_params.size());
    vd_dock_result* h_res = reinterpret_cast<vd_dock_result*>(hs + b_dp + b_pp);
    unsigned long long* h_cnt = reinterpret_cast<unsigned long long*>(hs + b_dp + b_pp + b_res);
    auto enqueue_all = [&](cudaStream_t s) -> vd_status {
        vd_status e = enqueue_dock(c, db, hs, s);
        if (e != VD_OK) return e;
        e = enqueue_post(c, pp, hs + b_dp, h_res, s);
        if (e != VD_OK) return e;
        VD_CUDA(cudaMemcpyAsync(h_cnt, c.d_counter + 2, 2 * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        VD_CUDA(cudaMemcpyAsync(h_cnt + 2, db.d_lig_evals, n * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                s));
        return VD_OK;
    };
    if (persistent) {
        CaptureGuard guard{c.stream, false};
        VD_CUDA(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal));
        guard.open = true;
        st = enqueue_all(c.stream);
        if (st != VD_OK) return st;
        cudaGraph_t graph = nullptr;
        guard.open = false;
        VD_CUDA(cudaStreamEndCapture(c.stream, &graph));
        bool updated = false;
        if (c.pipe_exec) {
            cudaGraphExecUpdateResultInfo info{};
            updated = cudaGraphExecUpdate(c.pipe_exec, graph, &info) == cudaSuccess;
            if (!updated) {
                cudaGetLastError();  // clear the update failure; a new executable replaces it
                cudaGraphExecDestroy(c.pipe_exec);
                c.pipe_exec = nullptr;
            }
        }
        cudaError_t e = cudaSuccess;
        if (!updated) {
            e = cudaGraphInstantiate(&c.pipe_exec, graph, 0);
            ++c.stats.graph_instantiations;
        }
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            c.pipe_exec = nullptr;
            set_error(std::string("CUDA graph instantiation failed: ") + cudaGetErrorString(e));
            return VD_ERR_CUDA;
        }
        VD_CUDA(cudaGraphLaunch(c.pipe_exec, c.stream));
        ++c.stats.graph_launches;
    } else {
        st = enqueue_all(c.stream);
        if (st != VD_OK) return st;
    }
    VD_CUDA(cudaStreamSynchronize(c.stream));
    if ((st = dock_take_checks("docking kernel")) != VD_OK) return st;
    if ((st = take_device_checks("post-processing kernels")) != VD_OK) return st;
    float dock_ms = 0, post_ms = 0;
    VD_CUDA(cudaEventElapsedTime(&dock_ms, c.ev0, c.ev1));
    VD_CUDA(cudaEventElapsedTime(&post_ms, c.ev1, c.ev2));
    std::memcpy(out, h_res, n * sizeof(vd_dock_result));
    c.stats.dock_ms = dock_ms;
    c.stats.post_ms = post_ms;
    c.stats.bfgs_evals += int64_t(h_cnt[0] + h_cnt[1]);
    dock_tune_report(c, db, dock_ms, h_cnt + 2);
    for (int i = 0; i < n; ++i) out[i].bfgs_evals = int64_t(h_cnt[2 + i]);  // search evaluations
    return VD_OK;
}

}  // namespace vd

using namespace vd;

extern "C" {

vd_status vd_dock_plain(vd_ctx* h, int32_t lig, const vd_search_params* sp, vd_dock_result* out) {
    VD_CHECK(h && sp && out, VD_ERR_ARG, "vd_dock_plain: NULL argument");
    return dock_pipeline(h->c, {lig}, *sp, false, out);
}

vd_status vd_dock_batched(vd_ctx* h, const int32_t* ligs, int32_t n, const vd_search_params* sp,
                          vd_dock_result* out) {
    VD_CHECK(h && ligs && sp && out && n > 0, VD_ERR_ARG, "vd_dock_batched: bad arguments");
    Ctx& c = h->c;
    for (int i = 0; i < n; ++i) VD_CHECK(ligs[i] >= 0 && ligs[i] < int(c.ligs.size()), VD_ERR_ARG, "bad ligand id");
    // The work queue hands out ligands in the order given; most expensive
    // chains first shortens the tail (a chain's result does not depend on
    // its position in the batch).  Cost = MC steps x BFGS steps x bytes
    // touched per evaluation.
    std::vector<int> order(n);
    std::vector<double> cost(n);
    for (int i = 0; i < n; ++i) {
        const HostLigand& L = c.ligs[ligs[i]];
        int depth = 0, steps = 0;
        search_defaults(L, *sp, depth, steps);
        order[i] = i;
        // depth 0 here means no MC step (a negative search_depth): one evaluation's bytes
        cost[i] = double(depth > 0 ? double(depth) * steps : 1.0) * (32.0 * L.h.n_atoms + 16.0 * L.h.n_pairs);
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    std::vector<int> v(n);
    for (int i = 0; i < n; ++i) v[i] = ligs[order[i]];
    std::vector<vd_dock_result> tmp(n);
    vd_status st = dock_pipeline(c, v, *sp, true, tmp.data());
    if (st != VD_OK) return st;
    for (int i = 0; i < n; ++i) out[order[i]] = tmp[i];
    return VD_OK;
}

vd_status vd_refine(vd_ctx* h, int32_t lig, int32_t n, float* poses, int32_t max_steps, float* e_out) {
    VD_CHECK(h && poses && e_out && n >= 0, VD_ERR_ARG, "vd_refine: bad arguments");
    Ctx& c = h->c;
    VD_CHECK(lig >= 0 && lig < int(c.ligs.size()), VD_ERR_ARG, "vd_refine: bad ligand id");
    if (n == 0) return VD_OK;
    VD_CUDA(cudaSetDevice(c.device));
    vd_status st = sync_pool(&c);
    if (st != VD_OK) return st;
    st = ensure_receptor_cells(&c);
    if (st != VD_OK) return st;
    const HostLigand& L = c.ligs[lig];
    const int nc = 7 + L.h.ntors;
    // poses, then the blob's offset and a count of evaluations that starts at
    // zero (one upload), then the energies (one download with the count)
    struct { int64_t off; unsigned long long evals; } head = {L.pool_offset, 0};
    st = ensure_scratch(&c, al256(size_t(n) * nc * 4) + sizeof(head) + size_t(n) * 4);
    if (st != VD_OK) return st;
    float* d_p = static_cast<float*>(c.d_scratch);
    char* d_head = static_cast<char*>(c.d_scratch) + al256(size_t(n) * nc * 4);
    int64_t* d_off = reinterpret_cast<int64_t*>(d_head);
    unsigned long long* d_evals = reinterpret_cast<unsigned long long*>(d_head + sizeof(int64_t));
    float* d_e = reinterpret_cast<float*>(d_head + sizeof(head));
    VD_CUDA(cudaMemcpyAsync(d_p, poses, size_t(n) * nc * 4, cudaMemcpyHostToDevice, c.stream));
    VD_CUDA(cudaMemcpyAsync(d_head, &head, sizeof(head), cudaMemcpyHostToDevice, c.stream));
    RefineParams rp{};
    rp.pool = c.d_pool;
    rp.lig_off = d_off;
    rp.pose_lig = nullptr;
    rp.poses = d_p;
    rp.e_out = d_e;
    rp.stride = nc;
    rp.n_poses = n;
    rp.max_steps_default = max_steps > 0 ? max_steps : (30 + L.n_all_atoms) / 3;
    rp.max_steps = nullptr;
    rp.R = rec_view(c);
    rp.smooth = c.d_smooth;
    rp.fix = c.fix_scale;
    rp.inv_fix = 1.f / c.fix_scale;
    rp.evals = d_evals;
    rp.skip_invalid = 0;
    RefineLaunch rl;
    if ((st = refine_launch(c, n, L.h.n_atoms, refine_floats(L), rl)) != VD_OK) return st;
    rl.kernel<<<n, rl.threads, rl.smem, c.stream>>>(rp);
    VD_CUDA(cudaGetLastError());
    VD_CUDA(cudaMemcpyAsync(poses, d_p, size_t(n) * nc * 4, cudaMemcpyDeviceToHost, c.stream));
    std::vector<char> tail(sizeof(head.evals) + size_t(n) * 4);
    VD_CUDA(cudaMemcpyAsync(tail.data(), d_evals, tail.size(), cudaMemcpyDeviceToHost, c.stream));
    VD_CUDA(cudaStreamSynchronize(c.stream));
    { const vd_status cs = take_device_checks("refinement kernel"); if (cs != VD_OK) return cs; }
    std::memcpy(&head.evals, tail.data(), sizeof(head.evals));
    std::memcpy(e_out, tail.data() + sizeof(head.evals), size_t(n) * 4);
    c.stats.bfgs_evals += int64_t(head.evals);
    return VD_OK;
}

vd_status vd_score(vd_ctx* h, int32_t lig, int32_t n, const float* poses, float* adjusted, float* intra) {
    VD_CHECK(h && poses && n >= 0 && n <= VD_MAX_MODES, VD_ERR_ARG, "vd_score: 0..20 poses");
    Ctx& c = h->c;
    VD_CHECK(lig >= 0 && lig < int(c.ligs.size()), VD_ERR_ARG, "vd_score: bad ligand id");
    if (n == 0) return VD_OK;
    VD_CUDA(cudaSetDevice(c.device));
    vd_status st = sync_pool(&c);
    if (st != VD_OK) return st;
    st = ensure_receptor_cells(&c);
    if (st != VD_OK) return st;
    const HostLigand& L = c.ligs[lig];
    const int nc = 7 + L.h.ntors;
    st = ensure_scratch(&c, al256(size_t(n) * nc * 4) + al256(size_t(n) * 16) + 512);
    if (st != VD_OK) return st;
    char* s = static_cast<char*>(c.d_scratch);
    float* d_p = reinterpret_cast<float*>(s); s += al256(size_t(n) * nc * 4);
    double* d_o = reinterpret_cast<double*>(s); s += al256(size_t(n) * 16);
    int64_t* d_off = reinterpret_cast<int64_t*>(s);
    VD_CUDA(cudaMemcpyAsync(d_p, poses, size_t(n) * nc * 4, cudaMemcpyHostToDevice, c.stream));
    const int64_t off = L.pool_offset;
    VD_CUDA(cudaMemcpyAsync(d_off, &off, 8, cudaMemcpyHostToDevice, c.stream));
    VD_CUDA(set_launch(c, score_poses_kernel, 0, size_t(pose_doubles(L.h.n_atoms, L.h.n_nodes)) * 8, 1024));
    score_poses_kernel<<<n, 32 * kScoreWarps, size_t(pose_doubles(L.h.n_atoms, L.h.n_nodes)) * 8, c.stream>>>(
        c.d_pool, d_off, d_p, nc, rec_view(c), c.d_fastd, d_o);
    VD_CUDA(cudaGetLastError());
    std::vector<double> o(size_t(n) * 2);
    VD_CUDA(cudaMemcpyAsync(o.data(), d_o, o.size() * 8, cudaMemcpyDeviceToHost, c.stream));
    VD_CUDA(cudaStreamSynchronize(c.stream));
    { const vd_status cs = take_device_checks("scoring kernel"); if (cs != VD_OK) return cs; }
    const double y = 1 + 0.1 * (c.weights[5] + 1) * double(L.h.num_tors) / 5.0;
    for (int i = 0; i < n; ++i) {
        const double x = o[2 * i] + o[2 * i + 1] - o[1];  // relative to pose 0's intramolecular energy
        if (adjusted) adjusted[i] = float(std::fabs(x) < DBL_EPSILON ? 0.0 : x / y);
        if (intra) intra[i] = float(o[2 * i + 1]);
    }
    return VD_OK;
}

vd_status vd_rmsd_bounds(vd_ctx* h, int32_t lig, int32_t n, const float* poses, float* lb_out, float* ub_out) {
    VD_CHECK(h && poses && lb_out && ub_out && n >= 0, VD_ERR_ARG, "vd_rmsd_bounds: bad arguments");
    Ctx& c = h->c;
    VD_CHECK(lig >= 0 && lig < int(c.ligs.size()), VD_ERR_ARG, "vd_rmsd_bounds: bad ligand id");
    if (n == 0) return VD_OK;
    VD_CUDA(cudaSetDevice(c.device));
    vd_status st = sync_pool(&c);
    if (st != VD_OK) return st;
    const HostLigand& L = c.ligs[lig];
    const int nc = 7 + L.h.ntors;
    st = ensure_scratch(&c, al256(size_t(n) * nc * 4) + al256(size_t(n) * 16) + 512);
    if (st != VD_OK) return st;
    char* s = static_cast<char*>(c.d_scratch);
    float* d_p = reinterpret_cast<float*>(s); s += al256(size_t(n) * nc * 4);
    double* d_o = reinterpret_cast<double*>(s); s += al256(size_t(n) * 16);
    int64_t* d_off = reinterpret_cast<int64_t*>(s);
    VD_CUDA(cudaMemcpyAsync(d_p, poses, size_t(n) * nc * 4, cudaMemcpyHostToDevice, c.stream));
    const int64_t off = L.pool_offset;
    VD_CUDA(cudaMemcpyAsync(d_off, &off, 8, cudaMemcpyHostToDevice, c.stream));
    const size_t smem = size_t(kRmsdWarps + 1) * pose_doubles(L.h.n_atoms, L.h.n_nodes) * 8;
    VD_CUDA(set_launch(c, rmsd_poses_kernel, 0, smem));
    rmsd_poses_kernel<<<(n + kRmsdWarps - 1) / kRmsdWarps, 32 * (kRmsdWarps + 1), smem, c.stream>>>(c.d_pool, d_off, d_p,
                                                                                                   n, nc, d_o);
    VD_CUDA(cudaGetLastError());
    std::vector<double> o(size_t(n) * 2);
    VD_CUDA(cudaMemcpyAsync(o.data(), d_o, o.size() * 8, cudaMemcpyDeviceToHost, c.stream));
    VD_CUDA(cudaStreamSynchronize(c.stream));
    { const vd_status cs = take_device_checks("RMSD kernel"); if (cs != VD_OK) return cs; }
    for (int i = 0; i < n; ++i) {
        lb_out[i] = float(o[2 * i]);
        ub_out[i] = float(o[2 * i + 1]);
    }
    return VD_OK;
}

}  // extern "C"
