// Grid-map precompute: replaces kernel_grid / kernel1 (kernel1.cu:93-249).
//
// Value of map t at grid point p (cache.cpp:148-208):
//   G_t(p) = sum over receptor atoms a with r^2 = |a - p|^2 <= 64 of
//            fast[pair(t_a, t)][int(32 r^2)]
// The bin index must match the reference's double computation bit for bit,
// so p = init + finv*i and r^2 = ((ax-px)^2 + (ay-py)^2) + (az-pz)^2 are
// evaluated in double with explicitly rounded operations (no FMA
// contraction); the table values are FP32 and the sums are FP32.
//
// Launch: one CTA per tile of 16(x) x 8(y) x TZ(z) points (TZ = 4, or 8 when
// pinned), 32*TZ threads, each thread owning 4 consecutive x points so
// every map store is one 128-bit store; one launch per group of up to 8 maps.  The CTA stages, in shared
// memory, the receptor atoms whose brick distance to the tile is below the
// cutoff, taken from per-type 4 A cell lists in deterministic (receptor type,
// cell, index) order.  The bin index floor(32 r^2) comes from a rounded-down
// FP64 add of 2^52 (no FP64->int conversion), every point within the cutoff
// then reads one 32-byte table row (predicated loads, so a thread's four
// issue together) and the accumulators are packed FP32 pairs added with
// add.rn.f32x2.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "checks.cuh"
#include "common.h"

namespace vd {
namespace {

constexpr int kTileX = 16, kTileY = 8;  // z tile TZ: 4, or 8 when pinned; threads = 32 * TZ
constexpr int kStageCap = 128;    // atoms staged per chunk (4 KB; a 70 A tile keeps ~60, larger counts loop)
constexpr double kCellSize = 4.0;
constexpr int kLutRows = kBins + 1;  // table rows per receptor type; the last (zero) row is padding

struct StagedAtom {
    double x, y, z;
    int32_t type;
    int32_t pad;
};

struct GridParams {
    double init[3], finv[3];
    int32_t n[3];
    int32_t pitch;
    size_t map_stride;
    float* maps;                  // first map of this type group
    const float* lut;             // this group's [receptor types present][kLutRows][NTG]
    int32_t n_out;                // maps written by this group (<= NTG)
    const StagedAtom* atoms;      // relevant receptor atoms sorted by (type, cell)
    const int32_t* cell_start;    // [n_rtypes][cells+1] per receptor type
    int32_t n_rtypes;             // receptor types present
    int32_t n_cells;
    double cell_org[3];
    int32_t cell_dim[3];
};

__device__ __forceinline__ double probe_coord(double init, double finv, int i) {
    return __dadd_rn(init, __dmul_rn(finv, double(i)));
}

constexpr int kMaxRows = 36;            // (cell rows in y) x (cell rows in z) per tile
constexpr int kMaxCombos = kTypes * kMaxRows;
// Block-wide exclusive scan of cnt[0..n) into off[0..n]; n <= kMaxCombos.
template <int kThreads>
__device__ __forceinline__ void block_scan(const int32_t* cnt, int32_t* off, int32_t* s_warp, int n) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int per = (n + kThreads - 1) / kThreads;
    const int j0 = min(n, t * per), j1 = min(n, j0 + per);
    int sum = 0;
    for (int j = j0; j < j1; ++j) sum += cnt[j];
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    int run = incl - sum;
    for (int w = 0; w < warp; ++w) run += s_warp[w];
    for (int j = j0; j < j1; ++j) {
        off[j] = run;
        run += cnt[j];
    }
    if (t == kThreads - 1) off[n] = run;
    __syncthreads();
}

// floor(32 * r2) for 0 <= r2 <= 64 on the FP64 pipe: 32 * r2 is exact, and
// adding 2^52 rounded toward -inf leaves the floor in the low mantissa word.
__device__ __forceinline__ int bin_of(double r2) {
    return __double2loint(__fma_rd(r2, 32.0, 4503599627370496.0));
}

// Two FP32 accumulators in one 64-bit register, added with one packed
// instruction (each lane rounds exactly like a scalar FP32 add).
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// acc[0..NTG/2) += table row v (NTG floats, 32- or 16-byte aligned).
template <int NTG>
__device__ __forceinline__ void add_row(unsigned long long (&acc)[NTG / 2], const float* v) {
    if constexpr (NTG == 8) {
        unsigned long long a0, a1, a2, a3;
        asm("ld.global.nc.v4.b64 {%0,%1,%2,%3}, [%4];" : "=l"(a0), "=l"(a1), "=l"(a2), "=l"(a3) : "l"(v));
        acc[0] = add2(acc[0], a0);
        acc[1] = add2(acc[1], a1);
        acc[2] = add2(acc[2], a2);
        acc[3] = add2(acc[3], a3);
    } else {
        unsigned long long a0, a1;
        asm("ld.global.nc.v2.b64 {%0,%1}, [%2];" : "=l"(a0), "=l"(a1) : "l"(v));
        acc[0] = add2(acc[0], a0);
        acc[1] = add2(acc[1], a1);
    }
}

// TZ = 8: 256 threads, 2 blocks per SM (120 registers); TZ = 4: 128 threads,
// 4 blocks per SM, twice the blocks for small boxes.
template <int NTG, int TZ>
__global__ void __launch_bounds__(32 * TZ, 16 / TZ) grid_build_kernel(GridParams p) {
    constexpr int kThreads = 32 * TZ, kTileZ = TZ;
    __shared__ StagedAtom s_atoms[kStageCap];
    __shared__ int32_t s_cnt[kMaxCombos];
    __shared__ int32_t s_b[kMaxCombos];
    __shared__ int32_t s_off[kMaxCombos + 1];
    __shared__ int32_t s_warp[kThreads / 32];
    __shared__ int32_t s_keep[kThreads / 32];

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int xq = t & 3, ly = (t >> 2) & 7, lz = t >> 5;
    const int x0 = blockIdx.x * kTileX + xq * 4;
    const int y = blockIdx.y * kTileY + ly;
    const int z = blockIdx.z * kTileZ + lz;

    // Tile bounding box (double) and the cell rows covering it +- 8 A.
    const int tx_lo = blockIdx.x * kTileX, ty_lo = blockIdx.y * kTileY, tz_lo = blockIdx.z * kTileZ;
    const int tx_hi = min(tx_lo + kTileX - 1, p.n[0] - 1);
    const int ty_hi = min(ty_lo + kTileY - 1, p.n[1] - 1);
    const int tz_hi = min(tz_lo + kTileZ - 1, p.n[2] - 1);
    const double lo[3] = {probe_coord(p.init[0], p.finv[0], tx_lo), probe_coord(p.init[1], p.finv[1], ty_lo),
                          probe_coord(p.init[2], p.finv[2], tz_lo)};
    const double hi[3] = {probe_coord(p.init[0], p.finv[0], tx_hi), probe_coord(p.init[1], p.finv[1], ty_hi),
                          probe_coord(p.init[2], p.finv[2], tz_hi)};
    int c_lo[3], c_hi[3];
    for (int d = 0; d < 3; ++d) {
        c_lo[d] = max(0, int(floor((lo[d] - 8.0 - p.cell_org[d]) / kCellSize)));
        c_hi[d] = min(p.cell_dim[d] - 1, int(floor((hi[d] + 8.0 - p.cell_org[d]) / kCellSize)));
    }
    const int ry = max(0, c_hi[1] - c_lo[1] + 1), rz = max(0, c_hi[2] - c_lo[2] + 1);
    // rows <= kMaxRows: the host checks the tile span against the cell size
    VD_DCHECK(c_lo[0] > c_hi[0] || ry * rz <= kMaxRows, kChkGridRows);
    const int n_rows = (c_lo[0] <= c_hi[0]) ? min(kMaxRows, ry * rz) : 0;
    const int n_combo = p.n_rtypes * n_rows;  // (receptor type, row), type-major

    // Candidate ranges per combo, then their exclusive prefix: candidates are
    // numbered in (type, cz, cy, cx, index) order.
    for (int j = t; j < n_combo; j += kThreads) {
        const int tr = j / n_rows, r = j - tr * n_rows;
        const int cy = c_lo[1] + r % ry, cz = c_lo[2] + r / ry;
        const int32_t* cs = p.cell_start + size_t(tr) * (p.n_cells + 1) + p.cell_dim[0] * (cy + p.cell_dim[1] * cz);
        const int b = __ldg(cs + c_lo[0]), e = __ldg(cs + c_hi[0] + 1);
        s_b[j] = b;
        s_cnt[j] = e - b;
    }
    __syncthreads();
    block_scan<kThreads>(s_cnt, s_off, s_warp, n_combo);
    const int n_cand = s_off[n_combo];

    const bool active = (x0 < p.n[0]) && (y < p.n[1]) && (z < p.n[2]);
    double px[4];
    for (int k = 0; k < 4; ++k) px[k] = probe_coord(p.init[0], p.finv[0], x0 + k);
    const double py = probe_coord(p.init[1], p.finv[1], y);
    const double pz = probe_coord(p.init[2], p.finv[2], z);

    unsigned long long acc[4][NTG / 2];  // maps (2j, 2j+1) of point k
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < NTG / 2; ++j) acc[k][j] = 0ull;

    for (int chunk = 0;; chunk += kStageCap) {
        // Stage the kept candidates with ranks [chunk, chunk + kStageCap),
        // in candidate order (a block-wide stream compaction).
        int kept = 0;
        for (int base = 0; base < n_cand; base += kThreads) {
            const int i = base + t;
            bool k = false;
            StagedAtom a;
            if (i < n_cand) {
                int lo_j = 0, hi_j = n_combo;  // last j with s_off[j] <= i
                while (hi_j - lo_j > 1) {
                    const int mid = (lo_j + hi_j) >> 1;
                    if (s_off[mid] <= i) lo_j = mid;
                    else hi_j = mid;
                }
                a = p.atoms[s_b[lo_j] + (i - s_off[lo_j])];
                double d2 = 0;
                const double c[3] = {a.x, a.y, a.z};
                for (int d = 0; d < 3; ++d) {
                    const double q = c[d] < lo[d] ? lo[d] - c[d] : (c[d] > hi[d] ? c[d] - hi[d] : 0.0);
                    d2 += q * q;
                }
                k = d2 < kCutoff2 + 1e-6;  // conservative: the per-point test below is exact
            }
            const unsigned m = __ballot_sync(0xffffffffu, k);
            if (lane == 0) s_keep[warp] = __popc(m);
            __syncthreads();
            int rank = kept + __popc(m & ((1u << lane) - 1u));
            int step = 0;
            for (int w = 0; w < kThreads / 32; ++w) {
                const int cw = s_keep[w];
                rank += (w < warp) ? cw : 0;
                step += cw;
            }
            const int slot = rank - chunk;
            if (k && slot >= 0 && slot < kStageCap) s_atoms[slot] = a;
            kept += step;
            __syncthreads();
        }
        const int n_here = min(kStageCap, kept - chunk);
        if (active) {
            for (int a = 0; a < n_here; ++a) {
                const StagedAtom at = s_atoms[a];
                const double dy = __dsub_rn(at.y, py), dz = __dsub_rn(at.z, pz);
                const double dy2 = __dmul_rn(dy, dy), dz2 = __dmul_rn(dz, dz);
                if (__dadd_rn(dy2, dz2) > kCutoff2) continue;  // exact: sums are monotone
                // Each point within the cutoff loads its row; the loads are
                // predicated per point (no branch), so those of a thread still
                // issue back to back, and points beyond the cutoff cost no L1
                // wavefront (the kernel's limit).
                const float* row_base = p.lut + VD_DCLAMP(at.type, 0, p.n_rtypes - 1, kChkGridType) * (kLutRows * NTG);
                int bin[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double dx = __dsub_rn(at.x, px[k]);
                    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), dy2), dz2);
                    bin[k] = r2 <= kCutoff2 ? bin_of(r2) : kBins;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (bin[k] < kBins) add_row<NTG>(acc[k], row_base + bin[k] * NTG);
            }
        }
        if (kept <= chunk + kStageCap) break;
        __syncthreads();
    }
    if (!active) return;
    const size_t off = (size_t(z) * p.n[1] + y) * p.pitch + x0;
#pragma unroll
    for (int j = 0; j < NTG; ++j) {
        if (j >= p.n_out) break;
        const int h = j & 1, q = j >> 1;
        auto f = [&](int k) { return __int_as_float(int(h ? acc[k][q] >> 32 : acc[k][q] & 0xffffffffull)); };
        *reinterpret_cast<float4*>(p.maps + size_t(j) * p.map_stride + off) = make_float4(f(0), f(1), f(2), f(3));
    }
}

// Table slices of a build, per group of up to 8 maps [receptor types present]
// [kLutRows][w] (w = 8, or 4 for a last group of at most 4 maps), gathered from
// the FP32 pair table on the device (4 us; building them on the host and
// copying them took ~0.3 ms).  One thread per row.
struct LutParams {
    const float* fast;      // [153][kBins]
    float* lut;
    int32_t n_present, n_maps;
    int32_t present[kTypes], needed[kTypes];
};
__global__ void __launch_bounds__(256) lut_kernel(LutParams p) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x, ti = r / kLutRows, i = r - ti * kLutRows;
    if (ti >= p.n_present) return;
    const int g0 = 8 * blockIdx.y, w = p.n_maps - g0 <= 4 ? 4 : 8;  // groups before this one are 8 wide
    float* row = p.lut + size_t(g0) * p.n_present * kLutRows + size_t(r) * w;
    const int t1 = p.present[ti];
    for (int j = 0; j < w; ++j) {
        float v = 0.f;
        if (i < kBins && g0 + j < p.n_maps) {
            const int t2 = p.needed[g0 + j], a = min(t1, t2), b = max(t1, t2);
            v = __ldg(&p.fast[size_t(a + b * (b + 1) / 2) * kBins + i]);
        }
        row[j] = v;
    }
}

// Corner cells for the evaluation kernels: cell (x, y, z) of map j holds the
// map values at its 8 corners (x fastest, then y, then z), 32 bytes, so a
// trilinear lookup reads one sector instead of eight scattered floats.
// Bound by the cells' write: one thread per column of kCellZ cells, which
// loads each of its planes once, with 32-bit indices and one 256-bit store per
// cell (consecutive threads write consecutive cells).  With a 64-bit division
// per cell and two 128-bit stores the 188^3 x 8 maps of a 70 A box took
// 505 us (3.7 TB/s); now 294 us (6.4 TB/s, 98 % of a plain copy's rate).
constexpr int kCellZ = 4;
__global__ void __launch_bounds__(256) corner_cells_kernel(const float* maps, size_t map_stride, float* cells,
                                                           size_t cell_stride, int nx, int ny, int nz, int pitch) {
    const uint32_t cx = nx - 1, cy = ny - 1, cz = nz - 1, plane = cx * cy;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= plane) return;
    const uint32_t y = i / cx, x = i - y * cx;
    const size_t map_plane = size_t(ny) * pitch;
    auto load = [&](const float* q) { return make_float4(__ldg(q), __ldg(q + 1), __ldg(q + pitch), __ldg(q + pitch + 1)); };
    auto pack = [](float lo, float hi) {
        return (static_cast<unsigned long long>(__float_as_uint(hi)) << 32) | __float_as_uint(lo);
    };
    for (uint32_t z0 = blockIdx.y * kCellZ; z0 < cz; z0 += gridDim.y * kCellZ) {
        const float* b = maps + size_t(blockIdx.z) * map_stride + (size_t(z0) * ny + y) * pitch + x;
        float* d = cells + size_t(blockIdx.z) * cell_stride + (size_t(z0) * plane + i) * 8;
        float4 v[kCellZ + 1];
#pragma unroll
        for (int k = 0; k <= kCellZ; ++k)
            if (z0 + k <= cz) v[k] = load(b + k * map_plane);
#pragma unroll
        for (int k = 0; k < kCellZ; ++k) {
            if (z0 + k >= cz) break;
            asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(d + size_t(k) * plane * 8),
                         "l"(pack(v[k].x, v[k].y)), "l"(pack(v[k].z, v[k].w)), "l"(pack(v[k + 1].x, v[k + 1].y)),
                         "l"(pack(v[k + 1].z, v[k + 1].w))
                         : "memory");
        }
    }
}

// Corner cells are built when all of them fit in this many bytes (a 150 A
// box of 17 maps is about 11 GB); larger boxes keep the plain maps only.
constexpr size_t kMaxCellBytes = size_t(16) << 30;

}  // namespace
}  // namespace vd

using namespace vd;

extern "C" {

vd_status vd_build_grids(vd_ctx* h, const int32_t* types, int32_t n_types) {
    VD_CHECK(h && types && n_types > 0 && n_types <= kTypes, VD_ERR_ARG, "vd_build_grids: bad type list");
    Ctx& c = h->c;
    VD_CHECK(c.has_box, VD_ERR_ARG, "vd_build_grids: call vd_set_box first");
    VD_CHECK(c.scoring, VD_ERR_ARG, "vd_build_grids: scoring not set");
    std::vector<int> needed;
    for (int i = 0; i < n_types; ++i) {
        VD_CHECK(types[i] >= 0 && types[i] < kTypes, VD_ERR_ARG, "vd_build_grids: XS type out of range");
        if (std::find(needed.begin(), needed.end(), types[i]) == needed.end()) needed.push_back(types[i]);
    }
    VD_CUDA(cudaSetDevice(c.device));
    const GridGeom& g = c.geom;
    const int nt = int(needed.size());

    // Relevant receptor atoms (szv_grid.cpp:28-42 rule) binned into 4 A cells
    // spanning the box grown by the cutoff.
    double org[3];
    int cd[3];
    for (int d = 0; d < 3; ++d) {
        org[d] = g.begin[d] - 8.0 - 1e-3;
        cd[d] = std::max(1, int(std::ceil((g.end[d] - g.begin[d] + 16.0 + 2e-3) / kCellSize)));
    }
    std::vector<StagedAtom> rel;
    std::vector<int> cell_of;
    const int n_rec = int(c.rec_xs.size());
    for (int i = 0; i < n_rec; ++i) {
        if (c.rec_xs[i] < 0) continue;
        const double* a = &c.rec_xyz[3 * size_t(i)];
        double d2 = 0;
        for (int d = 0; d < 3; ++d) {
            double q = (a[d] <= g.begin[d]) ? g.begin[d] : ((a[d] >= g.end[d]) ? g.end[d] : a[d]);
            d2 += (q - a[d]) * (q - a[d]);
        }
        if (!(d2 < kCutoff2)) continue;
        int ci[3];
        for (int d = 0; d < 3; ++d)
            ci[d] = std::min(cd[d] - 1, std::max(0, int(std::floor((a[d] - org[d]) / kCellSize))));
        rel.push_back({a[0], a[1], a[2], c.rec_xs[i], 0});
        cell_of.push_back(ci[0] + cd[0] * (ci[1] + cd[1] * ci[2]));
    }
    // per receptor type present: cell list over the same cells, atoms sorted
    // by (type, cell) so a tile stages them type by type: one counting sort
    const int n_cells = cd[0] * cd[1] * cd[2];
    bool has[kTypes] = {};
    for (const auto& a : rel) has[a.type] = true;
    std::vector<int> present;
    int row_of[kTypes] = {};  // table rows of the present types
    for (int tr = 0; tr < kTypes; ++tr)
        if (has[tr]) {
            row_of[tr] = int(present.size());
            present.push_back(tr);
        }
    if (present.empty()) present.push_back(0);
    std::vector<int32_t> start(present.size() * size_t(n_cells + 1), 0);
    std::vector<StagedAtom> sorted(rel.size());
    {
        // counts one place on, so that the running sums are each cell's start
        for (size_t i = 0; i < rel.size(); ++i) {
            rel[i].type = row_of[rel[i].type];
            ++start[size_t(rel[i].type) * (n_cells + 1) + cell_of[i] + 1];
        }
        int32_t run = 0;
        for (int32_t& s : start) s = run += s;
        std::vector<int32_t> fill(start);
        for (size_t i = 0; i < rel.size(); ++i)
            sorted[fill[size_t(rel[i].type) * (n_cells + 1) + cell_of[i]]++] = rel[i];
    }
    const size_t lut_floats = present.size() * kLutRows * size_t(nt % 8 == 0 ? nt : nt / 8 * 8 + (nt % 8 <= 4 ? 4 : 8));

    const size_t map_stride = size_t(g.pitch) * g.n[1] * g.n[2];
    const size_t bytes_maps = map_stride * nt * sizeof(float);
    const size_t n_cells_map = size_t(g.n[0] - 1) * (g.n[1] - 1) * (g.n[2] - 1);
    const size_t bytes_cells = n_cells_map * 8 * sizeof(float) * nt;
    const bool with_cells = bytes_cells <= kMaxCellBytes;
    const size_t bytes_atoms = (std::max<size_t>(1, sorted.size()) * sizeof(StagedAtom) + 255) & ~size_t(255);
    const size_t bytes_start = (start.size() * sizeof(int32_t) + 255) & ~size_t(255);
    const size_t bytes_lut = lut_floats * sizeof(float);
    c.n_maps = 0;
    for (int i = 0; i < kTypes; ++i) c.map_slot[i] = -1;
    // Maps and cells of the same size as the last build's stay allocated
    // (allocating and freeing 1.9 GB took ~3 of the 4.4 ms of a 70 A build); others are
    // all given back first.
    if (!dev_keeps(c, c.d_maps, bytes_maps)) dev_release(c, c.d_maps);
    if (!with_cells || !dev_keeps(c, c.d_cells, bytes_cells)) dev_release(c, c.d_cells);
    const bool kept = c.d_maps || c.d_cells;
    vd_status st = VD_OK;
    if (!c.d_maps && (st = dev_alloc(c, &c.d_maps, bytes_maps, "vd_build_grids: maps")) != VD_OK) return st;
    st = ensure_scratch(&c, bytes_atoms + bytes_start + bytes_lut);
    if (st != VD_OK) return st;
    // allocated before the events below, which time the kernels
    if (with_cells && !c.d_cells && (st = dev_alloc(c, &c.d_cells, bytes_cells, "vd_build_grids: corner cells")) != VD_OK)
        return st;
    // atoms and cell starts in one upload
    char* s = static_cast<char*>(c.d_scratch);
    StagedAtom* d_atoms = reinterpret_cast<StagedAtom*>(s);
    int32_t* d_start = reinterpret_cast<int32_t*>(s + bytes_atoms);
    float* d_lut = reinterpret_cast<float*>(s + bytes_atoms + bytes_start);
    std::vector<char> up(bytes_atoms + bytes_start);
    std::memcpy(up.data(), sorted.data(), sorted.size() * sizeof(StagedAtom));
    std::memcpy(up.data() + bytes_atoms, start.data(), start.size() * sizeof(int32_t));
    VD_CUDA(cudaMemcpyAsync(s, up.data(), up.size(), cudaMemcpyHostToDevice, c.stream));
    LutParams lp{};
    lp.fast = c.d_fast;
    lp.lut = d_lut;
    lp.n_present = int(present.size());
    lp.n_maps = nt;
    std::copy(present.begin(), present.end(), lp.present);
    std::copy(needed.begin(), needed.end(), lp.needed);
    lut_kernel<<<dim3((lp.n_present * kLutRows + 255) / 256, (nt + 7) / 8), 256, 0, c.stream>>>(lp);
    VD_CUDA(cudaGetLastError());

    GridParams p{};
    for (int d = 0; d < 3; ++d) {
        p.init[d] = g.init[d];
        p.finv[d] = g.finv[d];
        p.n[d] = g.n[d];
        p.cell_org[d] = org[d];
        p.cell_dim[d] = cd[d];
    }
    p.pitch = g.pitch;
    p.map_stride = map_stride;
    p.atoms = d_atoms;
    p.cell_start = d_start;
    p.n_rtypes = int(present.size());
    p.n_cells = n_cells;
    for (int d = 1; d < 3; ++d)  // cell rows a tile can touch in y and z: floor(span / cell) + 2 <= 6
        VD_CHECK(int(std::floor(((kTileY - 1) * g.finv[d] + 16.0) / kCellSize)) + 2 <= 6, VD_ERR_CAPACITY,
                 "vd_build_grids: grid spacing too large for the tile");
    // z tile: 4, unless the caller pinned 8 (bit-identical maps: a point sums its
    // atoms in global (type, cell, index) order whatever the tile).  us at 4
    // and 8 for boxes of 20 / 30 / 40 / 45 / 70 A: 22.6 / 26.6, 60 / 64, 106 /
    // 104, 152 / 154, 565 / 563; timing both on a box's first build cost more
    // than it could find.
    const int shape = c.grid_shape_fixed > 0 ? c.grid_shape_fixed - 1 : 1;
    const int tz = shape == 0 ? 8 : 4;
    // shared-memory carve-out for the blocks each tile keeps resident (2 of
    // 256 threads or 4 of 128), the rest of the SM's data memory as L1
    using GridFn = void (*)(GridParams);
    const GridFn wide = tz == 8 ? grid_build_kernel<8, 8> : grid_build_kernel<8, 4>;
    const GridFn narrow = tz == 8 ? grid_build_kernel<4, 8> : grid_build_kernel<4, 4>;
    auto carve = [&](GridFn kern) -> cudaError_t {
        cudaFuncAttributes fa{};
        const cudaError_t r = cudaFuncGetAttributes(&fa, kern);
        return r != cudaSuccess ? r : set_launch(c, kern, 16 / tz, 0, fa.sharedSizeBytes);
    };
    if (nt > 4) VD_CUDA(carve(wide));
    if (nt % 8 >= 1 && nt % 8 <= 4) VD_CUDA(carve(narrow));
    // calls on other streams may still read what was kept
    if (kept && (st = settle_device_calls(c)) != VD_OK) return st;
    const dim3 grid((g.n[0] + kTileX - 1) / kTileX, (g.n[1] + kTileY - 1) / kTileY, (g.n[2] + tz - 1) / tz);
    VD_CUDA(cudaEventRecord(c.ev0, c.stream));
    for (int g0 = 0; g0 < nt; g0 += 8) {
        p.maps = c.d_maps + size_t(g0) * map_stride;
        p.lut = d_lut + size_t(g0) * present.size() * kLutRows;
        p.n_out = std::min(8, nt - g0);
        (nt - g0 <= 4 ? narrow : wide)<<<grid, 32 * tz, 0, c.stream>>>(p);
        VD_CUDA(cudaGetLastError());
    }
    VD_CUDA(cudaEventRecord(c.ev1, c.stream));
    // corner cells of the new maps (cells_ms)
    if (with_cells) {
        c.cell_stride = n_cells_map * 8;
        const dim3 cells((size_t(g.n[0] - 1) * (g.n[1] - 1) + 255) / 256, std::min((g.n[2] - 1 + kCellZ - 1) / kCellZ, 65535), nt);
        corner_cells_kernel<<<cells, 256, 0, c.stream>>>(c.d_maps, map_stride, c.d_cells, c.cell_stride, g.n[0], g.n[1],
                                                         g.n[2], g.pitch);
        VD_CUDA(cudaGetLastError());
    }
    VD_CUDA(cudaEventRecord(c.ev2, c.stream));
    VD_CUDA(cudaEventSynchronize(c.ev2));
    if ((st = take_device_checks("grid kernel")) != VD_OK) return st;
    float grid_ms = 0, cells_ms = 0;
    VD_CUDA(cudaEventElapsedTime(&grid_ms, c.ev0, c.ev1));
    VD_CUDA(cudaEventElapsedTime(&cells_ms, c.ev1, c.ev2));
    c.stats.grid_shape = shape + 1;
    c.stats.grid_ms = grid_ms;
    c.stats.cells_ms = with_cells ? cells_ms : 0;
    c.map_stride = map_stride;
    c.n_maps = nt;
    for (int i = 0; i < kTypes; ++i) c.map_slot[i] = -1;
    for (int j = 0; j < nt; ++j) c.map_slot[needed[j]] = j;
    return VD_OK;
}

vd_status vd_set_grid_shape(vd_ctx* h, int32_t shape) {
    VD_CHECK(h && shape >= 0 && shape <= 2, VD_ERR_ARG, "vd_set_grid_shape: shape must be 0, 1 or 2");
    h->c.grid_shape_fixed = shape;
    return VD_OK;
}

vd_status vd_get_grid(vd_ctx* h, int32_t t, float* out) {
    VD_CHECK(h && out, VD_ERR_ARG, "vd_get_grid: NULL argument");
    Ctx& c = h->c;
    VD_CHECK(t >= 0 && t < kTypes && c.map_slot[t] >= 0, VD_ERR_ARG, "vd_get_grid: map not built");
    VD_CUDA(cudaSetDevice(c.device));
    const GridGeom& g = c.geom;
    const float* src = c.d_maps + size_t(c.map_slot[t]) * c.map_stride;
    // Slabs of padded rows come in one piece each into host memory that stays
    // with the context, and the rows are copied out from there: 220 us a call
    // for a 61 x 50 x 71 map, 120 us through pinned memory; a row-wise 2D copy
    // took ~800 us, one piece straight into memory that the caller has not
    // touched yet 240 us.  Pinned memory takes 4 ms to allocate, what it saves
    // on 40 such calls: a context asks for it once, when it has made that many.
    const size_t row = size_t(g.n[0]) * sizeof(float), pitch = size_t(g.pitch) * sizeof(float);
    const size_t rows = size_t(g.n[1]) * g.n[2], per = std::max<size_t>(1, std::min(rows, kMapSlab / pitch));
    char* const slab = map_slab(c, per * pitch);
    for (size_t r0 = 0; r0 < rows; r0 += per) {
        const size_t n = std::min(per, rows - r0);
        VD_CUDA(cudaMemcpyAsync(slab, src + r0 * g.pitch, n * pitch, cudaMemcpyDeviceToHost, c.stream));
        VD_CUDA(cudaStreamSynchronize(c.stream));
        for (size_t r = 0; r < n; ++r) std::memcpy(out + (r0 + r) * g.n[0], slab + r * pitch, row);
    }
    return VD_OK;
}

}  // extern "C"
