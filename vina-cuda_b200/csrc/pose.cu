// Pose batches: forward energy kernel, adjoint kernel (energy + gradient,
// recomputing atom coordinates from the torsion tree), coordinates, and
// one RILC-BFGS local optimisation per pose.  One warp per pose.
#include <cstring>

#include "launch.h"
#include "search.cuh"

namespace vd {
namespace {

constexpr int kPoseWarps = 4;

struct PoseParams {
    const float4* pool;
    int64_t lig_off;
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
    const LigView L = lig_view(p.pool, p.lig_off);
    const WarpMem m = carve(base, L.na, L.nn, L.np, L.nt);
    const int nc = 7 + L.nt, n = 6 + L.nt;
    for (int pose = blockIdx.x * kPoseWarps + wid; pose < p.n_poses; pose += gridDim.x * kPoseWarps) {
        const float* src = p.poses + size_t(pose) * nc;
        for (int i = lane; i < nc; i += 32) m.x[i] = src[i];
        __syncwarp();
        if (mode == 0) {
            const float e = eval_pose<false>(L, m, p.G, p.smooth, p.ep, lane);
            if (lane == 0) p.e_out[pose] = e;
        } else if (mode == 1) {
            const float e = eval_pose<true>(L, m, p.G, p.smooth, p.ep, lane);
            if (lane == 0) p.e_out[pose] = e;
            for (int i = lane; i < n; i += 32) p.g_out[size_t(pose) * n + i] = m.g[i];
        } else {
            kinematics(L, m, lane);
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

// Local optimisation, one RILC-BFGS run per pose; poses come from a queue
// (their numbers of evaluations differ several times over).  team > 1: a
// block takes one pose at a time, evaluated by a team of warps.
template <int blocks, int team>
__global__ void __launch_bounds__(32 * (team > 1 ? team : kPoseWarps), blocks) local_opt_kernel(PoseParams p) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* base = reinterpret_cast<float*>(smem4) + (team > 1 ? size_t(0) : size_t(wid) * p.warp_floats);
    const LigView L = lig_view(p.pool, p.lig_off);
    SearchMem s;
    s.m = carve(base, L.na, L.nn, L.np, L.nt);
    const PairTeam tm = pair_team(base + p.warp_floats);
    if (team > 1 && wid > 0) {
        const auto view = [&](int, LigView& l, WarpMem& m) {
            l = L;
            m = s.m;
        };
        pair_team_helper<team>(view, p.smooth, p.ep.v_intra, p.ep.fix, wid, lane, tm);
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
// per SM, no queue) -> now: 50 poses 287 -> 215, 1,000 426 -> 340, 1,300 449 ->
// 431 (80 registers: 454), 2,000 593 -> 510 (531), 2,800 644 -> 480, 8,000 1,515
// -> 1,150; 44 atoms, 1,000 poses 669 -> 415.
vd_status launch_local_opt(Ctx& c, const HostLigand& L, const PoseParams& p, cudaStream_t stream) {
    constexpr int kTeam = 4, kTeamPoses = 7, kWide = 4, kNarrow = 6;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    const size_t smem_team = (size_t(p.warp_floats) + pair_team_floats(L.h.sp_iters)) * sizeof(float);
    const bool team = p.n_poses <= sms * kTeamPoses && smem_team <= 227 * 1024 / kTeamPoses;
    const bool wide = p.n_poses <= sms * kWide * kPoseWarps;
    const size_t smem = team ? smem_team : size_t(p.warp_floats) * kPoseWarps * sizeof(float);
    VD_CHECK(smem <= 227 * 1024, VD_ERR_CAPACITY, "ligand too large for the pose kernel");
    auto k = team ? local_opt_kernel<kTeamPoses, kTeam> : wide ? local_opt_kernel<kWide, 1> : local_opt_kernel<kNarrow, 1>;
    const int threads = 32 * (team ? kTeam : kPoseWarps), poses = team ? 1 : kPoseWarps;  // per block
    VD_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    VD_CUDA(prefer_l1(k, c.device, team ? kTeamPoses : wide ? kWide : kNarrow, smem));
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
    p.pool = c.d_pool;
    p.lig_off = L.pool_offset;
    p.smooth = c.d_smooth;
    const vd_eval_params def = {10.0, 10.0, 1e6};
    const vd_eval_params* e = ep ? ep : &def;
    p.ep = {float(e->v_intra), float(e->v_inter), float(e->slope), c.fix_scale, 1.f / c.fix_scale};
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
        const size_t smem = size_t(p.warp_floats) * kPoseWarps * sizeof(float);
        VD_CHECK(smem <= 227 * 1024, VD_ERR_CAPACITY, "ligand too large for the pose kernel");
        auto kern = pose_kernel<mode>;
        VD_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        VD_CUDA(prefer_l1(kern, c.device, kPoseBlocks, smem));
        int dev_sms = 148;
        cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, c.device);
        const int blocks = std::min((n_poses + kPoseWarps - 1) / kPoseWarps, dev_sms * 16);
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
    return run_pose_kernel<1>(c, lig, n, poses, ep, e, g, nullptr, nullptr, 0, s);
}

vd_status vd_energy_device(vd_ctx* h, int32_t lig, int32_t n, const float* poses, const vd_eval_params* ep,
                           float* e, void* stream) {
    VD_CHECK(h && poses && e, VD_ERR_ARG, "vd_energy_device: NULL argument");
    Ctx& c = h->c;
    VD_CUDA(cudaSetDevice(c.device));
    cudaStream_t s = static_cast<cudaStream_t>(stream);  // NULL: the CUDA default stream
    return run_pose_kernel<0>(c, lig, n, poses, ep, e, nullptr, nullptr, nullptr, 0, s);
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
