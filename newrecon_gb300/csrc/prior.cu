// prior.cu -- 26-neighbour edge-preserving penalty and the fused OSTR update.
//
// For voxel j and each of its 26 neighbours k (t = x_j - x_k, neighbour
// weight w = 1/sqrt(dx^2 + dy^2 + (dz * z_xy_ratio)^2)):
//     RDD_j += w * omega(t),   RD_j += w * omega(t) * t
// with omega = 1 (Q2), 1/(1+|t|/delta) (Lange), 1/sqrt(1+(t/delta)^2)
// (hyperbola) or min(1, delta/|t|) (Huber).  A neighbour outside the volume
// is replaced by the voxel itself: t = 0, omega = 1, so its weight still adds
// to RDD (Tomo_OSTR.cu:118-255).
//
// The fused kernel computes, per voxel and in one pass,
//     capL = M * SBP(h over the subset views)          (Tomo_OSTR_gold.cpp:759-771)
//     RDD, RD as above from the current x              (:775)
//     x' = max(0, x - (capL + beta RD) / (d + 2 beta RDD))   (update_est :265-295)
// and writes x' to a second buffer (neighbours must see the old x).
#include "update.cuh"

namespace nr {

struct PriorW {
    float w[27];  // weight of neighbour (dx,dy,dz) at ((dz+1)*3+(dy+1))*3+(dx+1); centre 0
};

__host__ inline PriorW make_weights(float zxy) {
    PriorW p;
    for (int dz = -1; dz <= 1; dz++)
        for (int dy = -1; dy <= 1; dy++)
            for (int dx = -1; dx <= 1; dx++) {
                // distance as the reference forms it: float sqrt of a float sum,
                // then 1.0/distance in double, rounded once (Tomo_OSTR.cu:229).
                float dist = std::sqrt((float)(dx * dx + dy * dy) + (float)(dz * dz) * zxy * zxy);
                int k = ((dz + 1) * 3 + (dy + 1)) * 3 + (dx + 1);
                p.w[k] = (dist == 0.f) ? 0.f : (float)(1.0 / (double)dist);
            }
    return p;
}

// omega(t) with inv_delta = 1/delta.
template <int POT>
__device__ __forceinline__ float omega(float t, float delta, float inv_delta) {
    if (POT == NR_POT_Q2) return 1.f;
    if (POT == NR_POT_LANGE) return __fdividef(1.f, __fmaf_rn(fabsf(t), inv_delta, 1.f));
    if (POT == NR_POT_HYPERBOLA) {
        const float u = t * inv_delta;
        return rsqrtf(__fmaf_rn(u, u, 1.f));
    }
    const float a = fabsf(t);  // Huber
    return a <= delta ? 1.f : __fdividef(delta, a);
}

// RDD/RD sums over the 26 neighbours of (ix, iy, iz), read through L1.
template <int POT>
__device__ __forceinline__ void prior_sums(const nr_geom& g, const PriorW& W,
                                           const float* __restrict__ x, int ix, int iy, int iz,
                                           float xc, float delta, float inv_delta, float* rdd,
                                           float* rd) {
    float sdd = 0.f, sd = 0.f;
    const int64_t plane = (int64_t)g.nx * g.ny;
#pragma unroll
    for (int dz = -1; dz <= 1; dz++) {
#pragma unroll
        for (int dy = -1; dy <= 1; dy++) {
#pragma unroll
            for (int dx = -1; dx <= 1; dx++) {
                if (dx == 0 && dy == 0 && dz == 0) continue;
                const int kx = ix + dx, ky = iy + dy, kz = iz + dz;
                const bool in = (unsigned)kx < (unsigned)g.nx && (unsigned)ky < (unsigned)g.ny &&
                                (unsigned)kz < (unsigned)g.nz;
                float t = 0.f;
                if (in) t = xc - __ldg(x + (int64_t)kz * plane + (int64_t)ky * g.nx + kx);
                const float wo = W.w[((dz + 1) * 3 + (dy + 1)) * 3 + (dx + 1)] *
                                 omega<POT>(t, delta, inv_delta);
                sdd += wo;
                sd = __fmaf_rn(wo, t, sd);
            }
        }
    }
    *rdd = sdd;
    *rd = sd;
}

// Reference-shaped prior: RDD += ..., RD += ... (prior_GPU_OSTR / _Q2).
template <int POT>
__global__ void __launch_bounds__(128) prior_kernel(const __grid_constant__ Geo G,
                                                    const __grid_constant__ PriorW W,
                                                    float* __restrict__ RDD,
                                                    float* __restrict__ RD,
                                                    const float* __restrict__ x, float delta) {
    const nr_geom& g = G.g;
    const int ix = blockIdx.x * 32 + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    const int iz = blockIdx.z;
    if (ix >= g.nx || iy >= g.ny) return;
    const int64_t v = ((int64_t)iz * g.ny + iy) * g.nx + ix;
    float rdd, rd;
    prior_sums<POT>(g, W, x, ix, iy, iz, x[v], delta, 1.f / delta, &rdd, &rd);
    RDD[v] = RDD[v] + rdd;
    RD[v] = RD[v] + rd;
}

// The SART prior gradient: prior += sum_k t/sqrt(1+(t/delta)^2) / dist_k with
// plain neighbour distances (G_Huber_prior, Tomo_OSTR.cu:258-325; W built
// with z ratio 1).  The RDD sums of prior_sums are dead here and drop out.
__global__ void __launch_bounds__(128) prior_grad_kernel(const __grid_constant__ Geo G,
                                                         const __grid_constant__ PriorW W,
                                                         float* __restrict__ prior,
                                                         const float* __restrict__ x,
                                                         float delta) {
    const nr_geom& g = G.g;
    const int ix = blockIdx.x * 32 + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    const int iz = blockIdx.z;
    if (ix >= g.nx || iy >= g.ny) return;
    const int64_t v = ((int64_t)iz * g.ny + iy) * g.nx + ix;
    float rdd, rd;
    prior_sums<NR_POT_HYPERBOLA>(g, W, x, ix, iy, iz, x[v], delta, 1.f / delta, &rdd, &rd);
    prior[v] = prior[v] + rd;
}

template <int POT>
static nr_status launch_prior_t(const nr_geom& g, float* RDD, float* RD, const float* x,
                                float delta, float zxy, cudaStream_t st) {
    dim3 blk(32, 4), grd(cdiv(g.nx, 32), cdiv(g.ny, 4), g.nz);
    prior_kernel<POT><<<grd, blk, 0, st>>>(make_geo(g), make_weights(zxy), RDD, RD, x, delta);
    return launch_status();
}

nr_status launch_prior(const nr_geom& g, int pot, float* RDD, float* RD, const float* x,
                       float delta, float zxy, cudaStream_t st) {
    switch (pot) {
    case NR_POT_Q2: return launch_prior_t<NR_POT_Q2>(g, RDD, RD, x, delta, zxy, st);
    case NR_POT_LANGE: return launch_prior_t<NR_POT_LANGE>(g, RDD, RD, x, delta, zxy, st);
    case NR_POT_HYPERBOLA: return launch_prior_t<NR_POT_HYPERBOLA>(g, RDD, RD, x, delta, zxy, st);
    case NR_POT_HUBER: return launch_prior_t<NR_POT_HUBER>(g, RDD, RD, x, delta, zxy, st);
    default: return NR_ERR_BAD_ARGUMENT;
    }
}

// The separable back-projection tables of update.cuh for every view position
// a (subset order), plane and column / row: grid (.., nz, A).  EXACT: detector
// positions to twice FP32's precision, a plane's two lines formed in double by a
// thread each (1.8 M entries, those of 1000 x 1 x 300 and six views: 40 us, against
// 94 with the entries in double as well; FP64 runs at 1/64 of the FP32 rate).
template <bool EXACT>
__global__ void __launch_bounds__(128) bp_table_kernel(const __grid_constant__ Geo G,
                                                       const ProjView* __restrict__ views,
                                                       float4* __restrict__ tx,
                                                       float4* __restrict__ ty) {
    __shared__ BpLine lines[2];
    const nr_geom& g = G.g;
    const int a = blockIdx.z, z = blockIdx.y;
    const ProjView& V = views[a];
    const ViewSrc src = V.src;
    const float z1 = vox_z(g, z);
    const bool valid = z1 != src.z0;
    if (EXACT) {
        if (threadIdx.x < 2) {
            const bool y = threadIdx.x == 1;
            const double zd = ((double)z + 0.5) * g.vz + g.z_p0;
            const double t = zd != V.z0 ? (-(double)g.detectorR - V.z0) / (zd - V.z0) : 0.0;
            const double o = y ? (double)g.sourceY : V.x0, p0 = y ? g.y_p0 : g.x_p0;
            const double v = y ? g.vy : g.vx, d0 = y ? g.y_d0 : g.x_d0, r = 1.0 / (y ? g.by : g.bx);
            lines[threadIdx.x] =
                bp_line((o + (0.5 * v + p0 - o) * t - d0) * r - 0.5, v * t * r);
        }
        __syncthreads();
    }
    const float tt = bp_tt(g, src, z1);
    const float inv_bx = 1.f / g.bx, inv_by = 1.f / g.by;
    const float k = EXACT ? __fdiv_rn(1.f, g.vz * src.s2) : 1.f;
    const int64_t row = (int64_t)a * g.nz + z;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < g.nx + g.ny;
         q += gridDim.x * blockDim.x) {
        if (q < g.nx) {
            const float x1 = vox_x(g, q), ddx = src.x0 - x1;
            float4 e;
            if (EXACT) {
                e = bp_taps_on(lines[0], q, g.nbx, true);
            } else {
                const float x2 = src.x0 + (x1 - src.x0) * tt;
                e = bp_taps_at((x2 - g.x_d0) * inv_bx, g.nbx, true);
            }
            e.w = k * (ddx * ddx);
            tx[row * g.nx + q] = e;
        } else {
            const int j = q - g.nx;
            const float y1 = vox_y(g, j), ddy = src.y0 - y1, ddz = src.z0 - z1;
            float4 e;
            if (EXACT) {
                e = bp_taps_on(lines[1], j, g.nby, valid);
            } else {
                const float y2 = src.y0 + (y1 - src.y0) * tt;
                e = bp_taps_at((y2 - g.y_d0) * inv_by, g.nby, valid);
            }
            e.x = __int_as_float(__float_as_int(e.x) * g.nbx);
            e.w = k * (ddy * ddy + ddz * ddz);
            ty[row * g.ny + j] = e;
        }
    }
}

nr_status launch_bp_tables(const nr_geom& g, const ProjView* views, float4* tx, float4* ty,
                           bool exact, cudaStream_t st) {
    dim3 grd(cdiv((int64_t)g.nx + g.ny, 128), g.nz, g.n_angles);
    if (exact)
        bp_table_kernel<true><<<grd, 128, 0, st>>>(make_geo(g), views, tx, ty);
    else
        bp_table_kernel<false><<<grd, 128, 0, st>>>(make_geo(g), views, tx, ty);
    return launch_status();
}

// d = SBP(prj) over all views: prj [view][j][i] in original order, the tables'
// views in subset order, index[a] the original view of position a.  A thread
// takes four voxels of a column (iy .. iy + 3), which share the table's column
// entries; the loop over views carries nothing but the four sums.  96 M voxels,
// 25 views: 4.4 ms against 11.6 ms for the reference-shaped back projection
// (four divisions per voxel and view, the views' sources computed by every
// block of 128 voxels).  Bound by the taps' passes through L1 (about 40 per
// warp, view and four voxels).
constexpr int CV_ROWS = 4;
__global__ void __launch_bounds__(128) curvature_kernel(const __grid_constant__ Geo G,
                                                        float* __restrict__ d,
                                                        const float* __restrict__ prj,
                                                        const int32_t* __restrict__ index,
                                                        const __grid_constant__ BpTab T) {
    const nr_geom& g = G.g;
    const int ix = blockIdx.x * 32 + threadIdx.x;
    const int iy = (blockIdx.y * 4 + threadIdx.y) * CV_ROWS, z = blockIdx.z;
    if (ix >= g.nx || iy >= g.ny) return;
    const int last = g.ny - 1 - iy;   // rows beyond the volume repeat the last one
    const int64_t B = (int64_t)g.nbx * g.nby;
    f32x2 sum[2] = {pk2(0.f, 0.f), pk2(0.f, 0.f)};
    int tix = z * g.nx + ix, tiy = z * g.ny + iy;
    const int sx = g.nz * g.nx, sy = g.nz * g.ny;
#pragma unroll 2
    for (int a = 0; a < g.n_angles; a++, tix += sx, tiy += sy) {
        const float* p = prj + (int64_t)__ldg(index + a) * B;
        UpdView V[2];
        V[0].ex = V[1].ex = __ldg(T.x + tix);
#pragma unroll
        for (int k = 0; k < 2; k++) {
            V[k].ea = __ldg(T.y + (tiy + min(2 * k, last)));
            V[k].eb = __ldg(T.y + (tiy + min(2 * k + 1, last)));
        }
#pragma unroll
        for (int k = 0; k < 2; k++) V[k].taps(p, g.nbx);
#pragma unroll
        for (int k = 0; k < 2; k++) V[k].add(sum[k]);
    }
    float* o = d + ((int64_t)z * g.ny + iy) * g.nx + ix;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        float u, w;
        upk2(sum[k], u, w);
        if (2 * k <= last) o[(int64_t)(2 * k) * g.nx] = u;
        if (2 * k + 1 <= last) o[(int64_t)(2 * k + 1) * g.nx] = w;
    }
}

// The same sums, a thread per voxel of the volume taken as one row.
__global__ void __launch_bounds__(128) curvature_thin_kernel(const __grid_constant__ Geo G,
                                                             float* __restrict__ d,
                                                             const float* __restrict__ prj,
                                                             const int32_t* __restrict__ index,
                                                             const __grid_constant__ BpTab T) {
    const nr_geom& g = G.g;
    const unsigned n = (unsigned)g.nx * g.ny * g.nz, v = blockIdx.x * 128 + threadIdx.x;
    if (v >= n) return;
    const unsigned row = v / (unsigned)g.nx, z = row / (unsigned)g.ny;
    const float4* tx = T.x + (z * g.nx + (v - row * g.nx));
    const float4* ty = T.y + row;
    const int sx = g.nz * g.nx, sy = g.nz * g.ny;
    const int64_t B = (int64_t)g.nbx * g.nby;
    float sum = 0.f;
#pragma unroll 4
    for (int a = 0; a < g.n_angles; a++, tx += sx, ty += sy)
        bp_view(prj + (int64_t)__ldg(index + a) * B, __ldg(tx), __ldg(ty), g, sum);
    d[v] = sum;
}

// Blocks of 32 x 16 voxels unless the volume would fill them to less than two
// fifths (1000 x 1 x 300, six views: 13 us against 23).
nr_status launch_curvature(const nr_geom& g, float* d, const float* prj, const int32_t* index,
                           const BpTab& T, cudaStream_t st) {
    const int64_t voxels = (int64_t)g.nx * g.ny * g.nz;
    dim3 blk(32, 4), grd(cdiv(g.nx, 32), cdiv(g.ny, 4 * CV_ROWS), g.nz);
    if (5 * voxels < 2 * (int64_t)grd.x * 32 * grd.y * 4 * CV_ROWS * grd.z)
        curvature_thin_kernel<<<cdiv(voxels, 128), 128, 0, st>>>(make_geo(g), d, prj, index, T);
    else
        curvature_kernel<<<grd, blk, 0, st>>>(make_geo(g), d, prj, index, T);
    return launch_status();
}

template <int POT, int ZC>
static nr_status launch_update_t(const nr_geom& g, int tile, const float* x, float* x_out, const float* d,
                                 const float* h, const BpTab& T, int a0, int nv, float M, float beta,
                                 float delta, int* status, const CUtensorMap* map,
                                 cudaStream_t st) {
    dim3 grd(cdiv(g.nx, UTX), cdiv(g.ny, UTY), cdiv(g.nz, ZC));
    const Geo G = make_geo(g);
    const PriorW5 W = make_w5(g.vz / g.vx, delta);
    if (tile == NR_TILE_TMA && map) {
        dim3 blk(UTX, UTY);
        if (nv == 1)
            update_tma_kernel<POT, ZC, 1><<<grd, blk, 0, st>>>(G, W, *map, x_out, d, h, T, a0, nv, M,
                                                               beta, delta, status);
        else
            update_tma_kernel<POT, ZC, 0><<<grd, blk, 0, st>>>(G, W, *map, x_out, d, h, T, a0, nv, M,
                                                               beta, delta, status);
        return launch_status();
    }
    dim3 blk(UTX, UTY / 2);
    if (nv == 1)
        update_kernel<POT, ZC, 1><<<grd, blk, 0, st>>>(G, W, x, x_out, d, h, T, a0, nv, M, beta,
                                                       delta, status);
    else
        update_kernel<POT, ZC, 0><<<grd, blk, 0, st>>>(G, W, x, x_out, d, h, T, a0, nv, M, beta,
                                                       delta, status);
    return launch_status();
}

template <int POT>
static nr_status launch_update_z(const nr_geom& g, int zc, int tile, const float* x, float* x_out,
                                 const float* d, const float* h, const BpTab& T, int a0, int nv,
                                 float M, float beta, float delta, int* status,
                                 const CUtensorMap* map, cudaStream_t st) {
    switch (zc ? zc : upd_planes_auto(g)) {
    case 4:
        return launch_update_t<POT, 4>(g, tile, x, x_out, d, h, T, a0, nv, M, beta, delta, status,
                                       map, st);
    case 8:
        return launch_update_t<POT, 8>(g, tile, x, x_out, d, h, T, a0, nv, M, beta, delta, status,
                                       map, st);
    case 32:
        return launch_update_t<POT, 32>(g, tile, x, x_out, d, h, T, a0, nv, M, beta, delta, status,
                                        map, st);
    default:
        return launch_update_t<POT, 16>(g, tile, x, x_out, d, h, T, a0, nv, M, beta, delta, status,
                                        map, st);
    }
}

nr_status launch_update(const nr_geom& g, int pot, int zc, int tile, const float* x, float* x_out,
                        const float* d, const float* h, const BpTab& T, int a0, int nv, float M,
                        float beta, float delta, int* status, const CUtensorMap* map,
                        cudaStream_t st) {
    if (nv > UPD_MAX_VIEWS) return NR_ERR_BAD_ARGUMENT;
    switch (pot) {
    case NR_POT_Q2:
        return launch_update_z<NR_POT_Q2>(g, zc, tile, x, x_out, d, h, T, a0, nv, M, beta, delta,
                                          status, map, st);
    case NR_POT_LANGE:
        return launch_update_z<NR_POT_LANGE>(g, zc, tile, x, x_out, d, h, T, a0, nv, M, beta, delta,
                                             status, map, st);
    case NR_POT_HYPERBOLA:
        return launch_update_z<NR_POT_HYPERBOLA>(g, zc, tile, x, x_out, d, h, T, a0, nv, M, beta,
                                                 delta, status, map, st);
    case NR_POT_HUBER:
        return launch_update_z<NR_POT_HUBER>(g, zc, tile, x, x_out, d, h, T, a0, nv, M, beta, delta,
                                             status, map, st);
    default: return NR_ERR_BAD_ARGUMENT;
    }
}

}  // namespace nr

using namespace nr;

NR_API nr_status nr_prior(const nr_geom* g, float* RDD, float* RD, const float* x,
                          int32_t potential, float delta, float z_xy_ratio, void* stream) {
    if (!geom_ok(g)) return NR_ERR_BAD_GEOMETRY;
    if (!RDD || !RD || !x) return NR_ERR_BAD_ARGUMENT;
    if (potential != NR_POT_Q2 && !(delta > 0.f)) return NR_ERR_BAD_ARGUMENT;  // Tomo_OSTR.cu:2232
    if (g->nz > 65535) return NR_ERR_BAD_GEOMETRY;
    return launch_prior(*g, potential, RDD, RD, x, potential == NR_POT_Q2 ? 1.f : delta,
                        z_xy_ratio, as_stream(stream));
}

NR_API nr_status nr_prior_sart(const nr_geom* g, float* prior, const float* x, float delta,
                               void* stream) {
    if (!geom_ok(g)) return NR_ERR_BAD_GEOMETRY;
    if (!prior || !x || prior == x) return NR_ERR_BAD_ARGUMENT;
    if (delta == 0.f || !(delta == delta)) return NR_ERR_BAD_ARGUMENT;  // Tomo_OSTR.cu:2260-2263
    if (g->nz > 65535) return NR_ERR_BAD_GEOMETRY;
    dim3 blk(32, 4), grd(cdiv(g->nx, 32), cdiv(g->ny, 4), g->nz);
    prior_grad_kernel<<<grd, blk, 0, as_stream(stream)>>>(make_geo(*g), make_weights(1.f), prior,
                                                          x, delta);
    return launch_status();
}
