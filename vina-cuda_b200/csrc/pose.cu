// Pose batches: forward energy kernel, adjoint kernel (energy + gradient,
// recomputing atom coordinates from the torsion tree), coordinates, and
// one RILC-BFGS local optimisation per pose.  Energies and gradients run as tiles
// of poses with one pose per lane (tile_kernel), those of a few poses as teams of
// warps (pose_team_kernel), what is between and coordinates on one warp per pose.
#include <cstring>

#include "launch.h"
#include "search.cuh"

namespace vd {
namespace {

constexpr int kPoseWarps = 4;

struct PoseParams {
    const float4* lig;  // the ligand's blob
    LigHeader h;        // and its header: a call has one ligand, so no block waits for it
    MapView G;
    const float4* smooth;
    EvalParams ep;
    const float* poses;
    int32_t n_poses;
    float* e_out;
    float* g_out;       // adjoint only
    float* xyz_out;     // coords only
    float* poses_out;   // local opt
    int32_t max_steps;
    int32_t* queue;     // local opt: next pose
    unsigned long long* evals;
    int32_t warp_floats;
};

// mode 0: energy, 1: energy+gradient, 2: coordinates.  Held to 64 registers
// (8 blocks of 4 warps per SM): they fit without spills, and the adjoint
// (mode 1) left free takes 72 and loses a block per SM.
constexpr int kPoseBlocks = 8;
template <int mode>
__global__ void __launch_bounds__(32 * kPoseWarps, kPoseBlocks) pose_kernel(PoseParams p) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* base = reinterpret_cast<float*>(smem4) + size_t(wid) * p.warp_floats;
    const LigView L = lig_view(p.lig, p.h);
    const WarpMem m = carve(base, L.na, L.nn, L.np, L.nt);
    const int nc = 7 + L.nt, n = 6 + L.nt;
    for (int pose = blockIdx.x * kPoseWarps + wid; pose < p.n_poses; pose += gridDim.x * kPoseWarps) {
        const float* src = p.poses + size_t(pose) * nc;
        for (int i = lane; i < nc; i += 32) m.x[i] = src[i];
        __syncwarp();
        if (mode != 2) {
            const GridInter gi{&p.G, p.ep.v_inter, p.ep.slope};
            const float e = eval_pose_t<mode == 1, false, true>(L, m, gi, p.smooth, p.ep.v_intra, p.ep.fix, p.ep.inv_fix, lane);
            if (lane == 0) p.e_out[pose] = e;
            if (mode == 1)
                for (int i = lane; i < n; i += 32) p.g_out[size_t(pose) * n + i] = m.g[i];
        } else {
            kinematics<true>(L, m, lane);
            float* dst = p.xyz_out + size_t(pose) * 3 * L.na;
            for (int i = lane; i < L.na; i += 32) {
                dst[3 * i] = m.c[i].x;
                dst[3 * i + 1] = m.c[i].y;
                dst[3 * i + 2] = m.c[i].z;
            }
        }
        __syncwarp();
    }
}

// Modes 0 and 1 for few poses of a small ligand: a team of four warps per pose
// (eval.cuh), one evaluation and out.  Latency is all of it: us per launch in a
// graph on B200, a warp per pose -> a team, 64 poses of 8 / 16 / 24 / 30 atoms:
// 4.1 / 4.6 / 5.8 / 7.5 -> 3.5 / 3.9 / 3.9 / 4.4; 1,036 poses: 4.8 / 5.1 / 6.5 /
// 8.2 -> 4.1 / 4.4 / 4.9 / 5.7.
constexpr int kPoseTeam = 4, kTeamPoses = 7;  // warps per pose, poses resident per SM
template <int mode>
__global__ void __launch_bounds__(32 * kPoseTeam, kTeamPoses) pose_team_kernel(PoseParams p) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, pose = blockIdx.x;
    float* base = reinterpret_cast<float*>(smem4);
    const LigView L = lig_view(p.lig, p.h);
    const WarpMem m = carve(base, L.na, L.nn, L.np, L.nt);
    const PairTeam tm = pair_team(base + p.warp_floats);
    if (wid > 0) {
        const auto view = [&](int, LigView& l, WarpMem& w) {
            l = L;
            w = m;
        };
        pair_team_helper<kPoseTeam>(view, p.smooth, p.ep.v_intra, p.ep.fix, wid, lane, tm, 1);
        return;
    }
    const int nc = 7 + L.nt, n = 6 + L.nt;
    if (lane == 0) *tm.work = 1;
    const float* src = p.poses + size_t(pose) * nc;
    for (int i = lane; i < nc; i += 32) m.x[i] = src[i];
    __syncwarp();
    const GridInter gi{&p.G, p.ep.v_inter, p.ep.slope};
    const float thr = mode == 0 ? -INFINITY : INFINITY;  // energy only: no adjoint
    const float e = eval_pose_team<kPoseTeam, true>(L, m, gi, p.ep.inv_fix, lane, tm, SkipAbove{thr});
    if (lane == 0) {
        p.e_out[pose] = e;
        *tm.work = 0;
    }
    __syncwarp();
    team_arrive<kPoseTeam>(1);
    if (mode == 1)
        for (int i = lane; i < n; i += 32) p.g_out[size_t(pose) * n + i] = m.g[i];
}

// ---------------------------------------------------------------- pose tiles
// A block evaluates a tile of PL poses: a lane is one pose (lane mod PL) in one
// of S slots (warps x 32 / PL), and bodies, atoms and pairs are dealt to the
// slots.  Arrays in shared memory are [row][PL], rows being components of
// bodies or atoms.  With a warp per pose (pose_kernel) a pair's atoms lie at
// random places of shared memory and the lanes past a ligand's bodies and
// atoms idle: 1,198 L1 wavefronts and 3,241 warp instructions per evaluation
// of 40 atoms / 595 pairs at 65,536 poses, 90 % of the L1 data pipe.  With
// lanes as poses the loads are conflict-free and the pair list is uniform: 605
// and 2,218 with 8 warps a tile, 621 and 2,206 with 16; what is left is the
// table gathers, about one wavefront per lane, and L1 (27 to 33 % hits) decides:
// tile_shape below.
template <int PL>
struct Tile {
    int p, slot, slots;
    __device__ __forceinline__ Tile() {
        const int lane = threadIdx.x & 31;
        p = lane % PL;
        slot = (threadIdx.x >> 5) * (32 / PL) + lane / PL;
        slots = (blockDim.x >> 5) * (32 / PL);
    }
};
// Rows of a tile: coordinates [3][na]; pair forces [3][na] after the poses'
// components [7 + nt] and the bodies' local rotations [nn][4]; per body its
// axis and origin [6], then its part of the gradient; a partial energy per warp.
__host__ __device__ constexpr int tile_rows(int mode, int na, int nn, int nt, int warps) {
    const int early = 7 + nt + 4 * nn;
    const int forces = mode == 1 && 3 * na > early ? 3 * na : early;
    return 3 * na + forces + (mode == 1 ? 6 * nn : 0) + warps;
}
// Before them: the pairs as 32-bit words, an even number.
__host__ __device__ constexpr int tile_words(int np) { return pad4(np); }
static_assert((tile_words(VD_MAX_PAIRS) + tile_rows(1, VD_MAX_ATOMS, VD_MAX_TORS + 1, VD_MAX_TORS, 16) * 32) * 4 <= 227 * 1024,
              "the largest ligand fits the widest tile");

template <int mode, int PL>
__global__ void __launch_bounds__(512, 2) tile_kernel(PoseParams p) {
    extern __shared__ float4 smem4[];
    const Tile<PL> T;
    const LigView L = lig_view(p.lig, p.h);
    const int nc = 7 + L.nt, na = L.na;
    uint32_t* const W = reinterpret_cast<uint32_t*>(smem4);      // pairs: a | b << 8 | type pair << 16
    float* const C = reinterpret_cast<float*>(W + tile_words(L.np));  // [3][na]
    float* const X = C + 3 * na * PL;                            // [nc], then
    float* const A = X + nc * PL;                                // [nn][4]
    int* const Q = reinterpret_cast<int*>(X);                    // [3][na], later
    float* const B = X + PL * (mode == 1 ? max(3 * na, nc + 4 * L.nn) : nc + 4 * L.nn);  // [nn][6]
    float* const E = B + (mode == 1 ? 6 * L.nn * PL : 0);        // [warps]
    const int first = blockIdx.x * PL, here = min(PL, p.n_poses - first);

    // poses, transposed; a short last tile repeats its last pose
    for (int i = threadIdx.x; i < PL * nc; i += blockDim.x) {
        const int q = i / nc, c = i - q * nc;
        X[c * PL + q] = p.poses[size_t(first + min(q, here - 1)) * nc + c];
    }
    for (int i = threadIdx.x; i < L.np; i += blockDim.x) {
        const int2 q = __ldg(&L.pairs[i]);
        W[i] = uint32_t(q.x & 0xff) | uint32_t(q.x >> 16) << 8 | uint32_t(q.y) << 16;
    }
    __syncthreads();
    // local rotations, frames and coordinates: the arithmetic of frames() and
    // atom_position(), a slot per body
    for (int k = T.slot; k < L.nn; k += T.slots) {
        float4 aa = make_float4(1.f, 0.f, 0.f, 0.f);
        if (k > 0) {
            float s, c;
            __sincosf(0.5f * X[(7 + k - 1) * PL + T.p], &s, &c);
            const float4 ax = node_word(L.nodes, k, 1);
            aa = make_float4(c, __fmul_rn(s, ax.x), __fmul_rn(s, ax.y), __fmul_rn(s, ax.z));
        }
        float* const d = A + 4 * k * PL + T.p;
        d[0] = aa.x; d[PL] = aa.y; d[2 * PL] = aa.z; d[3 * PL] = aa.w;
    }
    __syncthreads();
    auto rotation = [&](int k) {
        const float* d = A + 4 * k * PL + T.p;
        return make_float4(d[0], d[PL], d[2 * PL], d[3 * PL]);
    };
    for (int k = T.slot; k < L.nn; k += T.slots) {
        float4 P = make_float4(1.f, 0.f, 0.f, 0.f);
        float3 w = make_float3(0.f, 0.f, 0.f);
        if (k > 0) {
            P = rotation(k);
            const float4 ok = node_word(L.nodes, k, 0);
            w = make_float3(ok.x, ok.y, ok.z);
            int j = VD_DCLAMP(__float_as_int(ok.w), 0, k - 1, kChkParent);
            while (j > 0) {
                const float4 aj = rotation(j);
                const float4 oj = node_word(L.nodes, j, 0);
                const float3 r = body_qrot(aj, w);
                w = make_float3(__fadd_rn(oj.x, r.x), __fadd_rn(oj.y, r.y), __fadd_rn(oj.z, r.z));
                P = walk_qmul(aj, P);
                j = VD_DCLAMP(__float_as_int(oj.w), 0, j - 1, kChkParent);
            }
        }
        const float4 qr = make_float4(X[3 * PL + T.p], X[4 * PL + T.p], X[5 * PL + T.p], X[6 * PL + T.p]);
        const float3 ro = body_qrot(qr, w);
        const BodyFrame f(root_qmul(qr, P), make_float3(__fadd_rn(X[T.p], ro.x), __fadd_rn(X[PL + T.p], ro.y),
                                                        __fadd_rn(X[2 * PL + T.p], ro.z)));
        const float4 w1 = node_word(L.nodes, k, 1);
        const int i1 = __float_as_int(node_word(L.nodes, k, 2).x);
        for (int i = __float_as_int(w1.w); i < i1; ++i) {
            const float4 a = __ldg(&L.atoms[i]);
#pragma unroll
            for (int d = 0; d < 3; ++d) C[(d * na + i) * PL + T.p] = f.point(d, a);
        }
        if (mode == 1) {
            float* const b = B + 6 * k * PL + T.p;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                b[d * PL] = f.direction(d, w1.x, w1.y, w1.z);
                b[(3 + d) * PL] = f.o[d];
            }
        }
    }
    __syncthreads();
    if (mode == 1) {
        for (int i = threadIdx.x; i < 3 * na * PL; i += blockDim.x) Q[i] = 0;
        __syncthreads();
    }
    auto coords = [&](int i) {
        return make_float3(C[i * PL + T.p], C[(na + i) * PL + T.p], C[(2 * na + i) * PL + T.p]);
    };
    // intra pairs: a slot takes a stretch of the pair list (sorted by second
    // atom), the second atom's position and force in registers while it repeats
    float e = 0.f;
    {
        const int twos = (L.np + 1) >> 1;  // two pairs at a time
        const int q1 = min(L.np, 2 * int(uint32_t(T.slot + 1) * uint32_t(twos) / uint32_t(T.slots)));
        int cur = -1;
        float3 cb = make_float3(0.f, 0.f, 0.f);
        float bx = 0.f, by = 0.f, bz = 0.f;  // in fixed-point units: fix is a power of two
        auto add_to = [&](int i, float x, float y, float z) {
            int* const d = Q + i * PL + T.p;
            atomicAdd(d, __float2int_rn(x));
            atomicAdd(d + na * PL, __float2int_rn(y));
            atomicAdd(d + 2 * na * PL, __float2int_rn(z));
        };
        auto turn_to = [&](int b) {
            if (mode == 1 && cur >= 0) add_to(cur, bx, by, bz);
            cur = b;
            bx = by = bz = 0.f;
        };
        for (int q = 2 * int(uint32_t(T.slot) * uint32_t(twos) / uint32_t(T.slots)); q < q1; q += 2) {
            const bool two = q + 1 < q1;
            const uint2 w = *reinterpret_cast<const uint2*>(W + q);
            const uint32_t w1 = two ? w.y : w.x;
            const int a0 = VD_DCLAMP(int(w.x & 0xff), 0, na - 1, kChkPairAtom), b0 = VD_DCLAMP(int(w.x >> 8 & 0xff), 0, na - 1, kChkPairAtom);
            const int a1 = VD_DCLAMP(int(w1 & 0xff), 0, na - 1, kChkPairAtom), b1 = VD_DCLAMP(int(w1 >> 8 & 0xff), 0, na - 1, kChkPairAtom);
            if (b0 != cur) {
                turn_to(b0);
                cb = coords(b0);
            }
            float3 cb1 = cb;
            if (b1 != b0) cb1 = coords(b1);
            const float3 ca0 = coords(a0), ca1 = coords(a1);
            const float r0x = cb.x - ca0.x, r0y = cb.y - ca0.y, r0z = cb.z - ca0.z;
            const float r1x = cb1.x - ca1.x, r1y = cb1.y - ca1.y, r1z = cb1.z - ca1.z;
            const float d0 = r0x * r0x + r0y * r0y + r0z * r0z, d1 = r1x * r1x + r1y * r1y + r1z * r1z;
            const float rf0 = fminf(32.f * d0, 2047.5f), rf1 = fminf(32.f * d1, 2047.5f);
            const Trunc bin0 = trunc_pos(rf0), bin1 = trunc_pos(rf1);
            const bool in0 = d0 < 64.f, in1 = two && d1 < 64.f;
            float4 t0 = make_float4(0.f, 0.f, 0.f, 0.f), t1 = t0;
            if (in0) t0 = __ldg(table_row(p.smooth, VD_DCLAMP(int(w.x >> 16), 0, kPairTypes - 1, kChkPairType), VD_DCLAMP(bin0.i, 0, kBins - 2, kChkTableBin)));
            if (in1) t1 = __ldg(table_row(p.smooth, VD_DCLAMP(int(w1 >> 16), 0, kPairTypes - 1, kChkPairType), VD_DCLAMP(bin1.i, 0, kBins - 2, kChkTableBin)));
            const float m0 = rf0 - bin0.f, m1 = rf1 - bin1.f, v = p.ep.v_intra;
            const float e0 = t0.x + m0 * (t0.z - t0.x), g0 = t0.y + m0 * (t0.w - t0.y);
            const float e1 = t1.x + m1 * (t1.z - t1.x), g1 = t1.y + m1 * (t1.w - t1.y);
            const float c0 = (e0 > 0.f) ? __fdividef(v, v + e0) : 1.f, c1 = (e1 > 0.f) ? __fdividef(v, v + e1) : 1.f;
            e += e0 * c0 + e1 * c1;  // zero past the cutoff
            if (mode == 1) {
                if (in0) {
                    const float h = g0 * c0 * c0 * p.ep.fix, Fx = h * r0x, Fy = h * r0y, Fz = h * r0z;
                    add_to(a0, -Fx, -Fy, -Fz);
                    bx += Fx; by += Fy; bz += Fz;
                }
                if (b1 != b0) turn_to(b1);
                if (in1) {
                    const float h = g1 * c1 * c1 * p.ep.fix, Fx = h * r1x, Fy = h * r1y, Fz = h * r1z;
                    add_to(a1, -Fx, -Fy, -Fz);
                    bx += Fx; by += Fy; bz += Fz;
                }
            } else {
                cur = b1;
            }
            cb = cb1;
        }
        turn_to(-1);
    }
    if (mode == 1) __syncthreads();
    // grid terms; an atom's total force takes the place of its pair force.
    // Energies from here on are added in FP64, rounded once per warp and once at
    // the end: an FP32 chain lost small terms behind an out-of-box penalty
    // and was 1 to 2 % further from FP64 than a warp per pose.
    const GridInter inter{&p.G, p.ep.v_inter, p.ep.slope};
    double sum = double(e);
    for (int i = T.slot; i < na; i += T.slots) {
        const float3 c = coords(i);
        float g[3];
        sum += inter(__float_as_int(__ldg(&L.atoms[i].w)) & 0xff, c.x, c.y, c.z, g[0], g[1], g[2]);
        if (mode == 1)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                int* const f = Q + (d * na + i) * PL + T.p;
                *reinterpret_cast<float*>(f) = g[d] + from_fixed(*f, p.ep.inv_fix);
            }
    }
#pragma unroll
    for (int o = 16; o >= PL; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);  // the warp's slots
    if ((threadIdx.x & 31) < PL) E[(threadIdx.x >> 5) * PL + T.p] = float(sum);
    __syncthreads();
    if (threadIdx.x < here) {
        double total = 0;
        for (int s = 0; s < blockDim.x >> 5; ++s) total += E[s * PL + threadIdx.x];
        p.e_out[first + threadIdx.x] = float(total);
    }
    if constexpr (mode == 1) {
        // a body's force and torque about its origin: the atoms of its subtree
        for (int k = T.slot; k < L.nn; k += T.slots) {
            float* const b = B + 6 * k * PL + T.p;
            const float ox = b[3 * PL], oy = b[4 * PL], oz = b[5 * PL];
            const float* const F = reinterpret_cast<const float*>(Q) + T.p;
            float fx = 0.f, fy = 0.f, fz = 0.f, tx = 0.f, ty = 0.f, tz = 0.f;
            const int i1 = VD_DCLAMP(__float_as_int(node_word(L.nodes, k, 2).w), 0, na, kChkSubtree);
            int i = VD_DCLAMP(__float_as_int(node_word(L.nodes, k, 1).w), 0, na, kChkSubtree);
            while (i < i1) {  // sums of up to 8 atoms first: a long chain of additions loses digits
                float sx = 0.f, sy = 0.f, sz = 0.f, ux = 0.f, uy = 0.f, uz = 0.f;
                for (const int stop = min(i + 8, i1); i < stop; ++i) {
                    const float3 c = coords(i);
                    const float x = F[i * PL], y = F[(na + i) * PL], z = F[(2 * na + i) * PL];
                    const float dx = c.x - ox, dy = c.y - oy, dz = c.z - oz;
                    sx += x; sy += y; sz += z;
                    ux += dy * z - dz * y;
                    uy += dz * x - dx * z;
                    uz += dx * y - dy * x;
                }
                fx += sx; fy += sy; fz += sz;
                tx += ux; ty += uy; tz += uz;
            }
            if (k == 0) {
                b[0] = fx; b[PL] = fy; b[2 * PL] = fz; b[3 * PL] = tx; b[4 * PL] = ty; b[5 * PL] = tz;
            } else {
                b[0] = tx * b[0] + ty * b[PL] + tz * b[2 * PL];
            }
        }
        __syncthreads();
        const int n = 6 + L.nt;
        for (int i = threadIdx.x; i < here * n; i += blockDim.x) {
            const int q = i / n, c = i - q * n;
            p.g_out[size_t(first) * n + i] = B[(c < 6 ? c : 6 * (c - 5)) * PL + q];
        }
    }
}

// Which kernel, by measurement (us on B200, energy + gradient | energy,
// warp per pose -> tile):
//   24 atoms / 5 torsions (~200 pairs): 64 poses 8.8 -> 9.7, 1,000 8.5 -> 10.5,
//     3,000 10.6 -> 12.4, 10,000 22.8 -> 17.7 | 16.7 -> 14.6, 65,536 105 -> 60 | 66 -> 50
//   33 / 9: 10,007 poses 41.4 -> 31.0 | 29.9 -> 27.0
//   40 / 10 (595 pairs): 64 poses 13.6 -> 10.6, 300 14.6 -> 12.6, 1,000 14.7 -> 13.6,
//     4,096 22.9 -> 21.1, 65,536 256 -> 175 | 198 -> 139
//   90 / 32 (~3,500 pairs): 64 poses 47.6 -> 16.7, 500 49.5 -> 22.8, 3,001 78 -> 62 | 74 -> 55
// A small ligand's evaluation in one warp is as short as a tile's phases, so
// below kTilePairs pairs it takes 64 poses per SM (two tiles of 32) for the
// tiles to pay.
constexpr int kTilePairs = 400;

// The size of a tile: PL poses (as many as leave two tiles per SM) and 8 or 16
// warps, by where the SMs run out of tiles or of L1; us with 8 | 16 warps:
//   up to 4 poses, 1,500 pairs and more: 16 warps while two tiles per SM hold all
//     poses, 80 atoms / 6 torsions 1,036 poses 23 | 22, 1,600 27 | 39
//   8 poses become 16 on 16 warps from 24 poses per SM (four tiles of 8 per SM):
//     4,096 poses of 60 / 15 39 -> 35, of 90 / 32 86 -> 74, of 128 / 3 68 -> 62
//   16 poses: 16 warps where the tiles of 8 that fit would need a second wave,
//     90 / 32 6,000 poses 111 | 114, 7,500 177 | 140; 128 / 3 144 | 116
//   32 poses become 16 on 16 warps where an SM holds one tile (20,000 poses of 128 /
//     3 327 -> 248), or where two take more than 160 KB and leave little L1 for the
//     records of many bodies: of 80 / 6 (154 KB) 178 and 180, 100 / 12 (202 KB) 266 ->
//     247, 90 / 32 (222 KB) 414 -> 306; with few bodies 100 / 4 (176 KB) 9 % slower
// A warp per pose took 282 for those of 128 / 3 and 111 for 7,500 of them.
inline bool few_bodies(const HostLigand& L) { return L.h.n_atoms > 8 * L.h.n_nodes; }
struct TileShape {
    int poses, warps;
    size_t smem;
    int resident;  // tiles per SM
};
template <int mode>
TileShape tile_shape(const Ctx& c, const HostLigand& L, int n_poses) {
    const int np = L.h.n_pairs;
    auto shape = [&](int poses, int warps) {
        TileShape t{poses, warps, 0, 0};
        t.smem = (size_t(tile_words(np)) + size_t(tile_rows(mode, L.h.n_atoms, L.h.n_nodes, L.h.ntors, warps)) * poses) * sizeof(float);
        t.resident = std::max(1, std::min(int(227 * 1024 / (t.smem + 1024)), 32 / warps));  // 64 registers
        return t;
    };
    const double per_sm = double(n_poses) / (2.0 * c.sms);  // poses per tile for two tiles per SM
    auto tiles = [&](int poses) { return (n_poses + poses - 1) / poses; };
    if (per_sm >= 32) {
        const TileShape t = shape(32, np >= kTilePairs ? 16 : 8);
        return t.resident < 2 || (2 * (t.smem + 1024) > 160 * 1024 && !few_bodies(L)) ? shape(16, 16) : t;
    }
    if (per_sm >= 16) {
        const TileShape t = shape(16, 8);
        return tiles(16) > t.resident * c.sms ? shape(16, 16) : t;
    }
    if (per_sm >= 12) return shape(16, 16);
    if (per_sm >= 8) return shape(8, 8);
    const int poses = per_sm >= 1.5 ? 4 : 1;
    return shape(poses, np >= 1500 && tiles(poses) <= 2 * c.sms ? 16 : 8);
}

// Ligands of many pairs in middle-sized batches that a warp per pose evaluates
// faster than tiles: with more than 8 atoms per body a tile's slots idle while
// bodies are placed and summed.  us, warp per pose and tile:
//   50 atoms / 5 torsions: 1,036 poses 12.3 and 12.7, 1,600 12.9 and 14.4, 2,500
//     15.4 and 17.8, 4,096 21.6 and 22.0, 4,900 31.1 and 26.2
//   60 / 3: 2,500 17.1 and 20.3, 3,300 20.4 and 21.7; 80 / 2: 1,600 24.5 and 22.6,
//     2,500 27.0 and 30.8, 3,300 33.7 and 32.6; 128 / 3: 2,500 49.8 and 54.3, 3,300 56.4 and 56.4
inline bool warps_win(const Ctx& c, const HostLigand& L, int n_poses) {
    const double per_sm = double(n_poses) / c.sms;
    const int np = L.h.n_pairs;
    return few_bodies(L) && (per_sm >= 16 ? per_sm < (np < 1500 ? 28 : 18) : np < 1000 && per_sm >= 10);
}

template <int mode>
vd_status launch_tile(Ctx& c, const HostLigand& L, const PoseParams& p, cudaStream_t stream) {
    const TileShape t = tile_shape<mode>(c, L, p.n_poses);
    auto k = t.poses == 32 ? tile_kernel<mode, 32> : t.poses == 16 ? tile_kernel<mode, 16> : t.poses == 8 ? tile_kernel<mode, 8>
             : t.poses == 4 ? tile_kernel<mode, 4> : tile_kernel<mode, 1>;
    VD_CUDA(set_launch(c, k, t.resident, t.smem));
    k<<<(p.n_poses + t.poses - 1) / t.poses, 32 * t.warps, t.smem, stream>>>(p);
    VD_CUDA(cudaGetLastError());
    return VD_OK;
}

// Local optimisation, one RILC-BFGS run per pose; poses come from a queue
// (their numbers of evaluations differ several times over).  team > 1: a
// block takes one pose at a time, evaluated by a team of warps.
template <int blocks, int team>
__global__ void __launch_bounds__(32 * (team > 1 ? team : kPoseWarps), blocks) local_opt_kernel(PoseParams p) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* base = reinterpret_cast<float*>(smem4) + (team > 1 ? size_t(0) : size_t(wid) * p.warp_floats);
    const LigView L = lig_view(p.lig, p.h);
    SearchMem s;
    s.m = carve(base, L.na, L.nn, L.np, L.nt);
    const PairTeam tm = pair_team(base + p.warp_floats);
    if (team > 1 && wid > 0) {
        const auto view = [&](int, LigView& l, WarpMem& m) {
            l = L;
            m = s.m;
        };
        pair_team_helper<team>(view, p.smooth, p.ep.v_intra, p.ep.fix, wid, lane, tm, 1);
        return;
    }
    s.xp = base + warp_floats(L.na, L.nn, L.np, L.nt);
    s.xo = s.xp + pad4(7 + L.nt);
    const int nc = 7 + L.nt;
    if (team > 1 && lane == 0) *tm.work = 1;
    int evals = 0;
    const auto eval = [&](const SkipAbove& skip) {
        const GridInter gi{&p.G, p.ep.v_inter, p.ep.slope};
        if constexpr (team > 1)
            return eval_pose_team<team>(L, s.m, gi, p.ep.inv_fix, lane, tm, skip);
        else
            return eval_pose_t<true, true>(L, s.m, gi, p.smooth, p.ep.v_intra, p.ep.fix, p.ep.inv_fix, lane, skip);
    };
    for (;;) {
        int v = 0;
        if (lane == 0) v = atomicAdd(p.queue, 1);
        const int pose = __shfl_sync(0xffffffffu, v, 0);
        if (pose >= p.n_poses) break;
        const float* src = p.poses + size_t(pose) * nc;
        for (int i = lane; i < nc; i += 32) s.m.x[i] = src[i];
        __syncwarp();
        const float e = rilc_bfgs(L, s, eval, p.max_steps, lane, evals);
        if (lane == 0) p.e_out[pose] = e;
        for (int i = lane; i < nc; i += 32) p.poses_out[size_t(pose) * nc + i] = s.m.x[i];
        __syncwarp();
    }
    if (lane == 0 && evals) atomicAdd(p.evals, (unsigned long long)evals);
    if (team > 1) {
        if (lane == 0) *tm.work = 0;
        __syncwarp();
        team_arrive<team>(1);
    }
}

// Launch of local_opt_kernel by the number of poses: a team of four warps per
// pose while all poses are resident that way (7 blocks per SM, as in the
// docking kernel), else one warp per pose, at 128 registers (4 blocks) while
// all poses are resident, else at 80 (6 blocks).  31-atom ligand, at most 20
// steps, us a call on B200, before (one warp a pose at 140 registers, 3 blocks
// per SM, no queue) -> now: 50 poses 287 -> 205, 1,000 426 -> 340, 1,300 449 ->
// 426 (80 registers: 454), 2,000 593 -> 505 (531), 2,800 644 -> 480, 8,000 1,515
// -> 1,150; 44 atoms, 1,000 poses 669 -> 400, 1,300 758 -> 636, 2,300 1,127 -> 930.
vd_status launch_local_opt(Ctx& c, const HostLigand& L, const PoseParams& p, cudaStream_t stream) {
    constexpr int kTeam = kPoseTeam, kWide = 4, kNarrow = 6;
    const int sms = c.sms;
    const size_t smem_team = (size_t(p.warp_floats) + pair_team_floats(L.h.sp_iters)) * sizeof(float);
    const bool team = p.n_poses <= sms * kTeamPoses && smem_team <= 227 * 1024 / kTeamPoses;
    const bool wide = p.n_poses <= sms * kWide * kPoseWarps;
    const size_t smem = team ? smem_team : size_t(p.warp_floats) * kPoseWarps * sizeof(float);
    VD_CHECK(smem <= 227 * 1024, VD_ERR_CAPACITY, "ligand too large for the pose kernel");
    auto k = team ? local_opt_kernel<kTeamPoses, kTeam> : wide ? local_opt_kernel<kWide, 1> : local_opt_kernel<kNarrow, 1>;
    const int threads = 32 * (team ? kTeam : kPoseWarps), poses = team ? 1 : kPoseWarps;  // per block
    VD_CUDA(set_launch(c, k, team ? kTeamPoses : wide ? kWide : kNarrow, smem));
    int per_sm = 0;
    VD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem));
    const int blocks = std::min(sms * std::max(1, per_sm), (p.n_poses + poses - 1) / poses);
    k<<<blocks, threads, smem, stream>>>(p);
    VD_CUDA(cudaGetLastError());
    return VD_OK;
}

template <int mode>
vd_status run_pose_kernel(Ctx& c, int lig, int n_poses, const float* d_poses, const vd_eval_params* ep,
                          float* d_e, float* d_g, float* d_xyz, float* d_out, int max_steps,
                          cudaStream_t stream) {
    VD_CHECK(lig >= 0 && lig < int(c.ligs.size()), VD_ERR_ARG, "bad ligand id");
    VD_CHECK(n_poses >= 0, VD_ERR_ARG, "negative pose count");
    if (n_poses == 0) return VD_OK;
    vd_status st = sync_pool(&c);
    if (st != VD_OK) return st;
    PoseParams p{};
    if (mode != 2) {
        st = make_map_view(c, p.G);
        if (st != VD_OK) return st;
        st = check_ligand_maps(c, lig);
        if (st != VD_OK) return st;
    }
    const HostLigand& L = c.ligs[lig];
    p.lig = c.d_pool + L.pool_offset;
    p.h = L.h;
    p.smooth = c.d_smooth;
    const vd_eval_params def = {10.0, 10.0, 1e6};
    const vd_eval_params* e = ep ? ep : &def;
    // One evaluation's forces may use the bits that the context's scale keeps
    // for 128 partners of an atom where this ligand's atoms have fewer: a team or
    // a tile rounds a pair's force more often than a warp, and this leaves the
    // gradient's error below the warp's at the context's scale.  The optimisers
    // keep that scale: their runs are the docking search's.
    float fix = c.fix_scale;
    if (mode == 0 || mode == 1)
        for (int d = std::max(1, L.max_partners); 2 * d <= 128; d *= 2) fix *= 2.f;
    p.ep = {float(e->v_intra), float(e->v_inter), float(e->slope), fix, 1.f / fix};
    p.poses = d_poses;
    p.n_poses = n_poses;
    p.e_out = d_e;
    p.g_out = d_g;
    p.xyz_out = d_xyz;
    p.poses_out = d_out;
    p.max_steps = max_steps;
    p.evals = reinterpret_cast<unsigned long long*>(c.d_counter + 8);
    p.queue = c.d_counter + 10;
    p.warp_floats = lig_warp_floats(L) + (mode == 3 ? 2 * pad4(7 + L.h.ntors) : 0);
    if constexpr (mode == 3) {
        return launch_local_opt(c, L, p, stream);
    } else {
        if constexpr (mode != 2) {
            if ((L.h.n_pairs >= kTilePairs && !warps_win(c, L, n_poses)) || n_poses >= 64 * c.sms)
                return launch_tile<mode>(c, L, p, stream);
            if (n_poses <= kTeamPoses * c.sms) {
                const size_t smem = (size_t(p.warp_floats) + pair_team_floats(L.h.sp_iters)) * sizeof(float);
                VD_CUDA(set_launch(c, pose_team_kernel<mode>, kTeamPoses, smem));
                pose_team_kernel<mode><<<n_poses, 32 * kPoseTeam, smem, stream>>>(p);
                VD_CUDA(cudaGetLastError());
                return VD_OK;
            }
        }
        const size_t smem = size_t(p.warp_floats) * kPoseWarps * sizeof(float);
        VD_CHECK(smem <= 227 * 1024, VD_ERR_CAPACITY, "ligand too large for the pose kernel");
        auto kern = pose_kernel<mode>;
        VD_CUDA(set_launch(c, kern, kPoseBlocks, smem));
        const int blocks = std::min((n_poses + kPoseWarps - 1) / kPoseWarps, c.sms * 16);
        kern<<<blocks, 32 * kPoseWarps, smem, stream>>>(p);
        VD_CUDA(cudaGetLastError());
        return VD_OK;
    }
}

}  // namespace
}  // namespace vd

using namespace vd;

extern "C" {

vd_status vd_energy_grad_device(vd_ctx* h, int32_t lig, int32_t n, const float* poses, const vd_eval_params* ep,
                                float* e, float* g, void* stream) {
    VD_CHECK(h && poses && e && g, VD_ERR_ARG, "vd_energy_grad_device: NULL argument");
    Ctx& c = h->c;
    VD_CUDA(cudaSetDevice(c.device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);  // NULL: the CUDA default stream
    const vd_status st = run_pose_kernel<1>(c, lig, n, poses, ep, e, g, nullptr, nullptr, 0, s);
    c.device_calls |= st == VD_OK;
    return st;
}

vd_status vd_energy_device(vd_ctx* h, int32_t lig, int32_t n, const float* poses, const vd_eval_params* ep,
                           float* e, void* stream) {
    VD_CHECK(h && poses && e, VD_ERR_ARG, "vd_energy_device: NULL argument");
    Ctx& c = h->c;
    VD_CUDA(cudaSetDevice(c.device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);  // NULL: the CUDA default stream
    const vd_status st = run_pose_kernel<0>(c, lig, n, poses, ep, e, nullptr, nullptr, nullptr, 0, s);
    c.device_calls |= st == VD_OK;
    return st;
}

static vd_status pose_host(vd_ctx* h, int32_t lig, int32_t n, const float* poses, const vd_eval_params* ep,
                           float* e_out, float* g_out, float* xyz_out, int mode, int max_steps,
                           float* poses_out, int64_t* evals) {
    VD_CHECK(h && poses, VD_ERR_ARG, "pose call: NULL argument");
    Ctx& c = h->c;
    VD_CHECK(lig >= 0 && lig < int(c.ligs.size()), VD_ERR_ARG, "bad ligand id");
    if (n <= 0) return n == 0 ? VD_OK : VD_ERR_ARG;
    VD_CUDA(cudaSetDevice(c.device));
    const HostLigand& L = c.ligs[lig];
    const size_t nc = 7 + L.h.ntors, ng = 6 + L.h.ntors, na = L.h.n_atoms;
    const size_t b_pose = ((n * nc * 4 + 255) / 256) * 256, b_e = ((n * 4 + 255) / 256) * 256;
    const size_t b_g = ((n * ng * 4 + 255) / 256) * 256, b_x = ((n * na * 12 + 255) / 256) * 256;
    vd_status st = ensure_scratch(&c, 2 * b_pose + b_e + b_g + b_x);
    if (st != VD_OK) return st;
    char* s = static_cast<char*>(c.d_scratch);
    float* d_pose = reinterpret_cast<float*>(s);
    float* d_out = reinterpret_cast<float*>(s + b_pose);
    float* d_e = reinterpret_cast<float*>(s + 2 * b_pose);
    float* d_g = reinterpret_cast<float*>(s + 2 * b_pose + b_e);
    float* d_x = reinterpret_cast<float*>(s + 2 * b_pose + b_e + b_g);
    VD_CUDA(cudaMemcpyAsync(d_pose, poses, n * nc * 4, cudaMemcpyHostToDevice, c.stream));
    if (mode == 3) VD_CUDA(cudaMemsetAsync(c.d_counter + 8, 0, 12, c.stream));  // evaluations, queue
    switch (mode) {
        case 0: st = run_pose_kernel<0>(c, lig, n, d_pose, ep, d_e, nullptr, nullptr, nullptr, 0, c.stream); break;
        case 1: st = run_pose_kernel<1>(c, lig, n, d_pose, ep, d_e, d_g, nullptr, nullptr, 0, c.stream); break;
        case 2: st = run_pose_kernel<2>(c, lig, n, d_pose, ep, nullptr, nullptr, d_x, nullptr, 0, c.stream); break;
        default: st = run_pose_kernel<3>(c, lig, n, d_pose, ep, d_e, nullptr, nullptr, d_out, max_steps, c.stream);
    }
    if (st != VD_OK) return st;
    if (e_out) VD_CUDA(cudaMemcpyAsync(e_out, d_e, n * 4, cudaMemcpyDeviceToHost, c.stream));
    if (g_out) VD_CUDA(cudaMemcpyAsync(g_out, d_g, n * ng * 4, cudaMemcpyDeviceToHost, c.stream));
    if (xyz_out) VD_CUDA(cudaMemcpyAsync(xyz_out, d_x, n * na * 12, cudaMemcpyDeviceToHost, c.stream));
    if (poses_out) VD_CUDA(cudaMemcpyAsync(poses_out, d_out, n * nc * 4, cudaMemcpyDeviceToHost, c.stream));
    unsigned long long ev = 0;
    if (mode == 3) VD_CUDA(cudaMemcpyAsync(&ev, c.d_counter + 8, 8, cudaMemcpyDeviceToHost, c.stream));
    VD_CUDA(cudaStreamSynchronize(c.stream));
    { const vd_status cs = take_device_checks("pose kernel"); if (cs != VD_OK) return cs; }
    if (evals) *evals = int64_t(ev);
    c.stats.bfgs_evals += int64_t(ev) + (mode == 1 ? n : 0);
    return VD_OK;
}

vd_status vd_energy(vd_ctx* h, int32_t lig, int32_t n, const float* poses, const vd_eval_params* ep, float* e) {
    VD_CHECK(e, VD_ERR_ARG, "vd_energy: NULL output");
    return pose_host(h, lig, n, poses, ep, e, nullptr, nullptr, 0, 0, nullptr, nullptr);
}
vd_status vd_energy_grad(vd_ctx* h, int32_t lig, int32_t n, const float* poses, const vd_eval_params* ep,
                         float* e, float* g) {
    VD_CHECK(e && g, VD_ERR_ARG, "vd_energy_grad: NULL output");
    return pose_host(h, lig, n, poses, ep, e, g, nullptr, 1, 0, nullptr, nullptr);
}
vd_status vd_pose_coords(vd_ctx* h, int32_t lig, int32_t n, const float* poses, float* xyz) {
    VD_CHECK(xyz, VD_ERR_ARG, "vd_pose_coords: NULL output");
    return pose_host(h, lig, n, poses, nullptr, nullptr, nullptr, xyz, 2, 0, nullptr, nullptr);
}
vd_status vd_local_opt(vd_ctx* h, int32_t lig, int32_t n, float* poses, const vd_eval_params* ep,
                       int32_t max_steps, float* e, int64_t* evals) {
    VD_CHECK(e, VD_ERR_ARG, "vd_local_opt: NULL output");
    return pose_host(h, lig, n, poses, ep, e, nullptr, nullptr, 3, max_steps, poses, evals);
}

}  // extern "C"
