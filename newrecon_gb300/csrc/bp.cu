// bp.cu -- voxel-driven bilinear back projector (SBP), a deterministic gather.
//
// For every view of the range the voxel centre is projected from the source
// onto the detector plane, the detector is bilinearly interpolated with the
// reference's edge rules, the sample is weighted by Vsize_z * depth_weight and
// the per-view terms are summed in view order; the voxel's accumulator gets one
// add.  No atomics, so results are bit-reproducible run to run.  Restates the
// arithmetic of backprj_gpu_manyviews_SBP, Tomo_OSTR.cu:1553-1734.
//
// The detector is [view][i][j] here, j (along y) fastest, and the volume has x
// fastest.  A block takes 32 x 32 voxels of a plane with its lanes along y, so
// that the taps of a warp are consecutive floats of two detector columns (one
// sector per lane and tap with the lanes along x), and turns its sums in shared
// memory to write along x.  A view's column taps depend on (x, z) and its row
// taps on (y, z): a block works both out once per plane and view, 64 taps
// instead of 1024, and keeps its views (a double sincos each) over several
// planes.  One view of 1024 x 512 x 60: 189 us, from 505 us with a thread per
// voxel along x; five views of 701 x 353 x 45: 143 us from 380.  Bound by the
// latency of the taps and of the barriers between a plane's phases: 94 M warp
// instructions at 42 % issue-active, 31 warps per SM at 64 registers.
#include "common.cuh"

namespace nr {

constexpr int BP_VIEWS = 32;  // views in shared memory at a time
constexpr int BP_T = 32;      // tile edge

__device__ __forceinline__ void load_views(const nr_geom& g, ViewSrc* sv,
                                           const float* __restrict__ angles,
                                           const int32_t* __restrict__ index, int a0, int nv) {
    for (int t = threadIdx.x; t < nv; t += blockDim.x) {
        const int s = index ? index[a0 + t] : a0 + t;
        sv[t] = view_source(g, angles[s]);
    }
}

struct BpTap {
    float frac;
    int lb;
};

// Lower bin and fraction of the detector position q along one axis.
__device__ __forceinline__ BpTap bp_tap(float q, float d0, float bin) {
    const float m = __fdiv_rn(q - d0, bin);
    int lb = (int)floorf(m);
    if (m < (float)lb + 0.5f) lb -= 1;
    return {m - ((float)lb + 0.5f), lb};
}

// The two rows' column sums at the row fraction f.
__device__ __forceinline__ float bp_rows(float d1, float d2, float f) {
    return __fmaf_rn(1.f - f, d1, __fmul_rn(f, d2));
}

// One view's bilinear sample of [i][j] plane p where taps may lie off the
// detector (Tomo_OSTR.cu:1684-1715: each tap contributes only on it; no
// renormalisation).  SENS: also of a detector of ones (the OS-SART sensitivity,
// Tomo_OSTR.cu:1838-1882).
template <bool SENS>
__device__ __forceinline__ float bp_edge(const nr_geom& g, const BpTap& ti, const BpTap& tj,
                                         const float* __restrict__ p, float* sens) {
    const int ilb = ti.lb, jlb = tj.lb;
    const float fracI = ti.frac;
    auto at = [&](int i, int j) -> float { return __ldg(p + (int64_t)i * g.nby + j); };
    float d1 = 0.f, d2 = 0.f, s1 = 0.f, s2 = 0.f;
    const bool i0 = (ilb < g.nbx) && (ilb >= 0);
    const bool i1 = (ilb < g.nbx - 1) && (ilb >= -1);
    const bool j0 = (jlb < g.nby) && (jlb >= 0);
    const bool j1 = (jlb < g.nby - 1) && (jlb >= -1);
    if (i0 && j0) {
        d1 = __fmul_rn(1.f - fracI, at(ilb, jlb));
        s1 = 1.f - fracI;
    }
    if (i1 && j0) {
        d1 = __fmaf_rn(fracI, at(ilb + 1, jlb), d1);
        s1 = s1 + fracI;
    }
    if (i0 && j1) {
        d2 = __fmul_rn(1.f - fracI, at(ilb, jlb + 1));
        s2 = 1.f - fracI;
    }
    if (i1 && j1) {
        d2 = __fmaf_rn(fracI, at(ilb + 1, jlb + 1), d2);
        s2 = s2 + fracI;
    }
    if (SENS) *sens = bp_rows(s1, s2, tj.frac);
    return bp_rows(d1, d2, tj.frac);
}

// Adds a view's samples u and (SENS) sn at a distance (ddx, ddy, ddz) from its
// source to the voxel's sums.
template <bool SENS>
__device__ __forceinline__ void bp_add(const nr_geom& g, float s2, float ddx, float ddy, float ddz,
                                       float u, float sn, float& total, float& total_sens) {
    const float depth_weight = __fdiv_rn(
        s2, __fmaf_rn(ddz, ddz, __fmaf_rn(ddx, ddx, __fmul_rn(ddy, ddy))));  // Tomo_OSTR.cu:1634
    total = __fadd_rn(total, __fmul_rn(__fmul_rn(u, g.vz), depth_weight));
    if (SENS)
        total_sens = __fadd_rn(total_sens, __fmul_rn(__fmul_rn(sn, g.vz), depth_weight));
}

// Writes voxel v from its sums (OSSART: see bp_kernel).
template <bool OSSART>
__device__ __forceinline__ void bp_store(float* __restrict__ vol, const float* __restrict__ prior,
                                         int64_t v, float total, float total_sens, float lambda,
                                         float beta) {
    if (!OSSART) {
        vol[v] = vol[v] + total;
        return;
    }
    float u = 0.f, bt = 0.f;
    if (total_sens != 0.f) {
        u = __fdiv_rn(total, total_sens);
        if (prior) bt = __fdiv_rn(beta * prior[v], total_sens);
    }
    const float xn = vol[v] + lambda * (u + bt);
    vol[v] = xn < 0.f ? 0.f : xn;
}

// vol[v] += sum_{views} SBP term.  prj planes are consecutive per view
// (view a-a0 at prj + (a-a0)*B).  index == nullptr means identity order.
// Block: tile blockIdx.x of the plane, planes [zc blockIdx.y, + zc).
//
// OSSART: instead the update in place over the [view][i][j] difference:
// x += lambda (sum_u + beta prior) / sum_sens (both terms 0 where sum_sens = 0),
// then x = max(x, 0).  prior == nullptr is backprj_OSSART_gpu_manyviews
// (Tomo_OSTR.cu:1737-1936), otherwise backprj_OSSART_R_gpu_manyviews
// (:1938-2143).  Each voxel reads and writes only itself, so the update is safe
// in place.
template <bool OSSART, int THREADS>
__global__ void __launch_bounds__(THREADS) bp_kernel(
    const __grid_constant__ Geo G, float* __restrict__ vol, const float* __restrict__ prj,
    const float* __restrict__ prior, const float* __restrict__ angles,
    const int32_t* __restrict__ index, int a0, int nv, int zc, float lambda, float beta) {
    __shared__ ViewSrc sv[BP_VIEWS];
    __shared__ BpTap taps[BP_VIEWS][2 * BP_T];  // columns of the tile, then its rows
    __shared__ float sums[OSSART ? 2 : 1][BP_T][BP_T + 1];
    constexpr int NC = BP_T * 32 / THREADS;  // columns per thread
    const nr_geom& g = G.g;
    const int tiles_x = (g.nx + BP_T - 1) / BP_T;
    const int x0 = (int)(blockIdx.x % tiles_x) * BP_T, y0 = (int)(blockIdx.x / tiles_x) * BP_T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t B = (int64_t)g.nbx * g.nby;
    // positions past the volume's edge repeat its last row and column
    const float y1 = vox_y(g, min(y0 + lane, g.ny - 1));
    float x1[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) x1[c] = vox_x(g, min(x0 + warp * NC + c, g.nx - 1));
    const int z_end = min((int)(blockIdx.y + 1) * zc, g.nz);
    bool loaded = false;
    for (int iz = blockIdx.y * zc; iz < z_end; iz++) {
        const float z1 = vox_z(g, iz);
        float total[NC], total_sens[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) total[c] = total_sens[c] = 0.f;
        for (int c0 = 0; c0 < nv; c0 += BP_VIEWS) {
            const int cn = min(BP_VIEWS, nv - c0);
            __syncthreads();
            if (!loaded || nv > BP_VIEWS) {
                load_views(g, sv, angles, index, a0 + c0, cn);
                __syncthreads();
                loaded = true;
            }
            for (int e = threadIdx.x; e < cn * 2 * BP_T; e += THREADS) {
                const ViewSrc v = sv[e / (2 * BP_T)];
                const int q = e % (2 * BP_T);
                const float t = __fdiv_rn(-g.detectorR - v.z0, z1 - v.z0);
                if (q < BP_T) {
                    const float xq = vox_x(g, min(x0 + q, g.nx - 1));
                    (&taps[0][0])[e] = bp_tap(__fmaf_rn(xq - v.x0, t, v.x0), g.x_d0, g.bx);
                } else {
                    const float yq = vox_y(g, min(y0 + q - BP_T, g.ny - 1));
                    (&taps[0][0])[e] = bp_tap(__fmaf_rn(yq - v.y0, t, v.y0), g.y_d0, g.by);
                }
            }
            __syncthreads();
            for (int t = 0; t < cn; t++) {
                const ViewSrc v = sv[t];
                if (z1 == v.z0) continue;  // the term is 0
                const BpTap tj = taps[t][BP_T + lane];
                const float ddy = v.y0 - y1, ddz = v.z0 - z1;
                const float* p = prj + (int64_t)(c0 + t) * B;
                BpTap ti[NC];
                bool in = (unsigned)tj.lb < (unsigned)(g.nby - 1);
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    ti[c] = taps[t][warp * NC + c];
                    in = in && (unsigned)ti[c].lb < (unsigned)(g.nbx - 1);
                }
                auto add = [&](int c, float u, float sn) {
                    bp_add<OSSART>(g, v.s2, v.x0 - x1[c], ddy, ddz, u, sn, total[c], total_sens[c]);
                };
                if (__all_sync(0xffffffffu, in)) {
                    float val[NC][4];
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        const float* q = p + (int64_t)ti[c].lb * g.nby + tj.lb;
                        val[c][0] = __ldg(q);
                        val[c][1] = __ldg(q + 1);
                        val[c][2] = __ldg(q + g.nby);
                        val[c][3] = __ldg(q + g.nby + 1);
                    }
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        const float f = ti[c].frac, e = 1.f - f;
                        const float d1 = __fmaf_rn(f, val[c][2], __fmul_rn(e, val[c][0]));
                        const float d2 = __fmaf_rn(f, val[c][3], __fmul_rn(e, val[c][1]));
                        const float s = OSSART ? e + f : 0.f;
                        add(c, bp_rows(d1, d2, tj.frac), OSSART ? bp_rows(s, s, tj.frac) : 0.f);
                    }
                } else {
#pragma unroll 1
                    for (int c = 0; c < NC; c++) {
                        float sn = 0.f;
                        const float u = bp_edge<OSSART>(g, taps[t][warp * NC + c], tj, p, &sn);
#pragma unroll
                        for (int k = 0; k < NC; k++)
                            if (k == c) add(k, u, sn);
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NC; c++) {
            sums[0][lane][warp * NC + c] = total[c];
            if (OSSART) sums[OSSART ? 1 : 0][lane][warp * NC + c] = total_sens[c];
        }
        __syncthreads();
        const int ix = x0 + lane;
        for (int r = warp; r < BP_T && y0 + r < g.ny; r += THREADS / 32) {
            if (ix >= g.nx) break;
            const int64_t v = ((int64_t)iz * g.ny + y0 + r) * g.nx + ix;
            bp_store<OSSART>(vol, prior, v, sums[0][r][lane], sums[OSSART ? 1 : 0][r][lane], lambda,
                             beta);
        }
    }
}

// The same, a thread per voxel of the volume taken as one row: for volumes that
// tiles would leave mostly idle (launch_sbp).  What these calls take is the chain
// of one thread, and this one has neither the tables nor the turn.
template <bool OSSART>
__global__ void __launch_bounds__(128) bp_small_kernel(
    const __grid_constant__ Geo G, float* __restrict__ vol, const float* __restrict__ prj,
    const float* __restrict__ prior, const float* __restrict__ angles,
    const int32_t* __restrict__ index, int a0, int nv, float lambda, float beta) {
    __shared__ ViewSrc sv[2 * BP_VIEWS];
    const nr_geom& g = G.g;
    const unsigned n = (unsigned)g.nx * g.ny * g.nz;
    const unsigned at = blockIdx.x * 128 + threadIdx.x, v = min(at, n - 1);
    const unsigned row = v / (unsigned)g.nx, z = row / (unsigned)g.ny;
    const float x1 = vox_x(g, v - row * g.nx), y1 = vox_y(g, row - z * g.ny), z1 = vox_z(g, z);
    const int64_t B = (int64_t)g.nbx * g.nby;
    float total = 0.f, total_sens = 0.f;
    for (int c0 = 0; c0 < nv; c0 += 2 * BP_VIEWS) {
        const int cn = min(2 * BP_VIEWS, nv - c0);
        if (c0) __syncthreads();
        load_views(g, sv, angles, index, a0 + c0, cn);
        __syncthreads();
#pragma unroll 4
        for (int t = 0; t < cn; t++) {
            const ViewSrc s = sv[t];
            if (z1 == s.z0) continue;  // the term is 0
            const float r = __fdiv_rn(-g.detectorR - s.z0, z1 - s.z0);
            const BpTap ti = bp_tap(__fmaf_rn(x1 - s.x0, r, s.x0), g.x_d0, g.bx);
            const BpTap tj = bp_tap(__fmaf_rn(y1 - s.y0, r, s.y0), g.y_d0, g.by);
            float sn = 0.f;
            const float u = bp_edge<OSSART>(g, ti, tj, prj + (int64_t)(c0 + t) * B, &sn);
            bp_add<OSSART>(g, s.s2, s.x0 - x1, s.y0 - y1, s.z0 - z1, u, sn, total, total_sens);
        }
    }
    if (at < n) bp_store<OSSART>(vol, prior, v, total, total_sens, lambda, beta);
}

// The form by size; all give the same bits.
//  - A thread per voxel while that makes at most four blocks per SM, or where the
//    tiles would be filled to less than two fifths.  40 x 24 x 8, five views:
//    5.4 us against 6.5 by tiles; 1000 x 1 x 300: 14.9 against 98; 33 x 33 x 640 (a
//    fill of 0.27): 26 against 46; but 1000 x 33 x 33 (0.5): 43 against 29, and
//    96 x 96 x 32 (295 k voxels): 30 against 8.3.
//  - Tiles of one column per thread (1024 threads) while all planes' tiles leave SMs
//    idle: 64 x 64 x 38, five views: 6.8 us against 8.1; 140 x 100 x 30: 16.7
//    against 10.9.
//  - Tiles of four columns per thread, so that the views' and rows' values are read
//    once for four voxels.  Planes per block: as many as leave two rounds of
//    resident blocks, at most 8.
template <bool OSSART>
static nr_status launch_sbp(const nr_geom& g, float* vol, const float* prj, const float* prior,
                            const float* angles, const int32_t* index, int a0, int a1,
                            float lambda, float beta, cudaStream_t s) {
    const int64_t tiles = (int64_t)cdiv(g.nx, BP_T) * cdiv(g.ny, BP_T);
    const int sms = sm_count();
    const int64_t full = tiles * g.nz / (sms * 16);
    const int zc = (int)(full < 1 ? 1 : (full > 8 ? 8 : full));
    const dim3 grd((unsigned)tiles, cdiv(g.nz, zc));
    const int64_t voxels = (int64_t)g.nx * g.ny * g.nz;
    if (voxels <= sms * 4 * 128 || 5 * voxels < 2 * tiles * BP_T * BP_T * g.nz)
        bp_small_kernel<OSSART><<<cdiv(voxels, 128), 128, 0, s>>>(
            make_geo(g), vol, prj, prior, angles, index, a0, a1 - a0, lambda, beta);
    else if (tiles * g.nz <= sms)
        bp_kernel<OSSART, 1024><<<grd, 1024, 0, s>>>(make_geo(g), vol, prj, prior, angles, index,
                                                     a0, a1 - a0, zc, lambda, beta);
    else
        bp_kernel<OSSART, 256><<<grd, 256, 0, s>>>(make_geo(g), vol, prj, prior, angles, index, a0,
                                                   a1 - a0, zc, lambda, beta);
    return launch_status();
}

}  // namespace nr

using namespace nr;

NR_API nr_status nr_bp_sbp(const nr_geom* g, float* vol, const float* prj, const int32_t* index,
                           const float* angles, int32_t a0, int32_t a1, void* stream) {
    if (!geom_ok(g)) return NR_ERR_BAD_GEOMETRY;
    if (!vol || !prj || !index || !angles || a0 < 0 || a1 < a0) return NR_ERR_BAD_ARGUMENT;
    if (g->ny > 65535 || g->nz > 65535) return NR_ERR_BAD_GEOMETRY;
    if (a1 == a0) return NR_OK;
    return launch_sbp<false>(*g, vol, prj, nullptr, angles, index, a0, a1, 0.f, 0.f,
                             as_stream(stream));
}

NR_API nr_status nr_bp_ossart(const nr_geom* g, float* x, const float* diff, const float* prior,
                              const int32_t* index, const float* angles, int32_t a0, int32_t a1,
                              float lambda, float beta, void* stream) {
    if (!geom_ok(g)) return NR_ERR_BAD_GEOMETRY;
    if (!x || !diff || !index || !angles || a0 < 0 || a1 < a0) return NR_ERR_BAD_ARGUMENT;
    if (prior == x) return NR_ERR_BAD_ARGUMENT;
    if (g->ny > 65535 || g->nz > 65535) return NR_ERR_BAD_GEOMETRY;
    if (a1 == a0) return NR_OK;
    return launch_sbp<true>(*g, x, diff, prior, angles, index, a0, a1, lambda, beta,
                            as_stream(stream));
}
