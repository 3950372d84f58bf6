// update.cuh -- the fused OSTR update of one tile (device code shared by the
// single-reconstruction kernel in prior.cu and the batched kernel in batch.cu).
//
// Per voxel and in one pass:
//     capL = M * SBP(h over the subset views)          (Tomo_OSTR_gold.cpp:759-771)
//     RDD, RD = 26-neighbour penalty sums of x         (:775, Tomo_OSTR.cu:118-325)
//     x' = max(0, x - (capL + beta RD) / (d + 2 beta RDD))   (update_est :265-295)
#pragma once

#include <cmath>
#include <type_traits>

#include "tma.cuh"
#include "walk.cuh"

namespace nr {

constexpr int UPD_MAX_VIEWS = 32;               // views per subset
constexpr int UTX = 32, UTY = 8, UZC = 16;      // tile: 32 x 8 columns, 16 planes per block
constexpr int UNT = UTX * UTY / 2;              // threads of a block: two voxels each
// Resident blocks per SM.  96 registers hold the walk without spills; per
// sub-iteration of the clinical workload 5 blocks took 0.236 ms, 6 blocks (80
// registers) 0.243, 4 blocks 0.246, 8 blocks (64 registers, 300 bytes of
// spills) 0.27: fewer instructions win over more warps.
constexpr int UPD_BLOCKS = 5;

// Planes per block when the caller leaves the choice open: 16, or fewer when
// that leaves SMs without their UPD_BLOCKS blocks (a 256 x 128 x 24 volume makes
// 256 blocks of 16 planes, 768 of 4).  blocks(zc): those of a launch.
template <class F>
__host__ inline int upd_planes_by(F blocks) {
    const int fill = sm_count() * UPD_BLOCKS;
    for (int zc = UZC; zc > 4; zc /= 2)
        if (blocks(zc) >= fill) return zc;
    return 4;
}
__host__ inline int64_t upd_blocks(const nr_geom& g, int zc) {
    return (int64_t)cdiv(g.nx, UTX) * cdiv(g.ny, UTY) * cdiv(g.nz, zc);
}
__host__ inline int upd_planes_auto(const nr_geom& g) {
    return upd_planes_by([&](int zc) { return upd_blocks(g, zc); });
}

// The five distinct neighbour weights 1/sqrt(dx^2+dy^2+(dz zr)^2) of the
// 26-neighbourhood (in-plane face, in-plane diagonal, z face, z edge, z
// corner), the same times delta (Huber), 1/delta and 1, each duplicated into
// both halves of a packed FP32 pair: the penalty works on neighbour pairs
// (nb_pair), and a pair operand read whole from the constant bank costs no
// instruction to assemble.
enum { W_FACE, W_DIAG, W_ZFACE, W_ZEDGE, W_ZCORNER, W_CLASSES };
struct alignas(8) PriorW5 {
    float2 w[W_CLASSES];   // weight of each class
    float2 wd[W_CLASSES];  // weight x delta
    float2 inv_delta;      // 1 / delta (hyperbola)
    float2 one;
};

__host__ inline PriorW5 make_w5(float zxy, float delta) {
    auto w = [&](int dx, int dy, int dz) {
        const float dist = std::sqrt((float)(dx * dx + dy * dy) + (float)(dz * dz) * zxy * zxy);
        return (float)(1.0 / (double)dist);
    };
    const float cls[W_CLASSES] = {w(1, 0, 0), w(1, 1, 0), w(0, 0, 1), w(1, 0, 1), w(1, 1, 1)};
    PriorW5 p;
    for (int k = 0; k < W_CLASSES; k++) {
        p.w[k] = make_float2(cls[k], cls[k]);
        p.wd[k] = make_float2(cls[k] * delta, cls[k] * delta);
    }
    const float idl = 1.f / delta;
    p.inv_delta = make_float2(idl, idl);
    p.one = make_float2(1.f, 1.f);
    return p;
}

// Approximate reciprocal / reciprocal square root (the MUFU unit, <= 1 ulp
// relative error; arguments here are >= 1 or >= delta, never denormal).
__device__ __forceinline__ float rcp_approx(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float v) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// omega(t) of two differences of one potential, divided by delta for Huber
// (min(1, delta/|t|) = delta / max(|t|, delta): the class factor carries the
// delta).  EDGE: a difference with an out-of-volume cell (NaN) counts as t = 0.
template <int POT, bool EDGE>
__device__ __forceinline__ f32x2 omega2(f32x2& t2, const PriorW5& W, float delta,
                                        float inv_delta) {
    float ta, tb;
    upk2(t2, ta, tb);
    if (EDGE) {
        ta = (ta == ta) ? ta : 0.f;
        tb = (tb == tb) ? tb : 0.f;
        t2 = pk2(ta, tb);
    }
    if (POT == NR_POT_Q2) return ld2(W.one);
    if (POT == NR_POT_LANGE)
        return pk2(rcp_approx(__fmaf_rn(fabsf(ta), inv_delta, 1.f)),
                   rcp_approx(__fmaf_rn(fabsf(tb), inv_delta, 1.f)));
    if (POT == NR_POT_HYPERBOLA) {
        const f32x2 u2 = mul2(t2, ld2(W.inv_delta));
        float qa, qb;
        upk2(fma2(u2, u2, ld2(W.one)), qa, qb);
        return pk2(rsqrt_approx(qa), rsqrt_approx(qb));
    }
    return pk2(rcp_approx(fmaxf(fabsf(ta), delta)), rcp_approx(fmaxf(fabsf(tb), delta)));
}

// The factor of weight class CLS on omega2's values.
template <int POT>
__device__ __forceinline__ const float2& class_factor(const PriorW5& W, int cls) {
    return POT == NR_POT_HUBER ? W.wd[cls] : W.w[cls];
}

// Two neighbour pairs na, nb of one weight class: each lane sums its two terms
// omega and omega t first and scales the sums once, sdd += w sum omega, sd +=
// w sum omega t (one multiplication less per class than scaling each term).
template <int POT, bool EDGE, int CLS>
__device__ __forceinline__ void nb_class2(f32x2 xc2, f32x2 na, f32x2 nb, const PriorW5& W,
                                          float delta, float inv_delta, f32x2& sdd, f32x2& sd) {
    f32x2 ta = sub2(xc2, na), tb = sub2(xc2, nb);
    const f32x2 oa = omega2<POT, EDGE>(ta, W, delta, inv_delta);
    const f32x2 ob = omega2<POT, EDGE>(tb, W, delta, inv_delta);
    const f32x2 f = ld2(class_factor<POT>(W, CLS));
    sdd = fma2(f, add2(oa, ob), sdd);
    sd = fma2(f, fma2(ob, tb, mul2(oa, ta)), sd);
}

// The z-face neighbours na, nb of two voxels (one each): lane `LANE` of each
// voxel's sums takes its term.
template <int POT, bool EDGE, int LANE>
__device__ __forceinline__ void nb_zface(f32x2 xc2, f32x2 n2, const PriorW5& W, float delta,
                                         float inv_delta, f32x2& sdda, f32x2& sda, f32x2& sddb,
                                         f32x2& sdb) {
    f32x2 t2 = sub2(xc2, n2);
    const f32x2 o2 = omega2<POT, EDGE>(t2, W, delta, inv_delta);
    float oa, ob, pa, pb, v[2];
    upk2(o2, oa, ob);
    upk2(mul2(o2, t2), pa, pb);
    const float f = class_factor<POT>(W, W_ZFACE).x;
    upk2(sdda, v[0], v[1]);
    v[LANE] = __fmaf_rn(f, oa, v[LANE]);
    sdda = pk2(v[0], v[1]);
    upk2(sda, v[0], v[1]);
    v[LANE] = __fmaf_rn(f, pa, v[LANE]);
    sda = pk2(v[0], v[1]);
    upk2(sddb, v[0], v[1]);
    v[LANE] = __fmaf_rn(f, ob, v[LANE]);
    sddb = pk2(v[0], v[1]);
    upk2(sdb, v[0], v[1]);
    v[LANE] = __fmaf_rn(f, pb, v[LANE]);
    sdb = pk2(v[0], v[1]);
}

// Kinds of fused update (template argument KIND of update_tile).
constexpr int UPD_OSTR = 0;     // OSTR step above
constexpr int UPD_SART = 1;     // OS-SART, backprj_OSSART_gpu_manyviews (Tomo_OSTR.cu:1737-1936)
constexpr int UPD_SART_R = 2;   // OS-SART with the hyperbola prior, backprj_OSSART_R (:1938-2143)

// The back projection of a voxel onto one view's detector is separable: on a
// plane z, the detector column (ilb, fracI) of a voxel depends only on its x
// and the row (jlb, fracJ) only on its y (the ray from the source through
// the voxel centre meets the detector plane at x0 + (x1 - x0) t(z), y0 +
// (y1 - y0) t(z)).  Neither depends on the volume, so they are tabulated once
// per reconstruction, per view (subset order), plane and column / row, as a tap
// pair and its weights:
//   x[(a nz + z) nx + i] = {c, w0, w1, k (x0 - x1)^2}
//   y[(a nz + z) ny + j] = {r * BINSx, v0, v1, k ((y0 - y1)^2 + (z0 - z1)^2)}
// with k = 1 / (Vsize_z |source|^2), so that the depth weight times Vsize_z is
// the reciprocal of the entries' sum (OS-SART: k = 1).
// The bilinear stencil's columns are ilb, ilb + 1 with weights 1 - fracI,
// fracI; a column off the detector gets weight 0 (the rules of
// Tomo_OSTR.cu:1684-1715), and c is ilb clamped to [0, BINSx - 2] with the
// weights moved to the columns they belong to, so both loads of a pair are
// in bounds and need no test.  Rows likewise (both weights 0 when the plane
// holds the source, :1643).  Interior taps compute exactly what the masked
// stencil did; an edge tap adds w * h + 0 * h' = w * h.  With a detector one
// bin wide (or high) the second load of a pair lands up to BINSx + 1 floats
// past the subset's views: the h sections carry that many zeros (bp_pad).
// Each update reads one entry of each per voxel and view (the x entries of a
// warp are consecutive, its y entry is one broadcast); the tables of a subset
// stay in L2.
struct BpTab {
    const float4* __restrict__ x;
    const float4* __restrict__ y;
};

__device__ __forceinline__ float bp_tt(const nr_geom& g, const ViewSrc& vs, float z1) {
    return z1 != vs.z0 ? __fdividef(-g.detectorR - vs.z0, z1 - vs.z0) : 0.f;
}

// The tables are indexed in 32 bits: true when both hold fewer than 2^31
// entries (the device-resident paths refuse a geometry otherwise).
__host__ inline bool bp_tables_fit(const nr_geom& g) {
    const int64_t n = (int64_t)g.n_angles * g.nz * (g.nx > g.ny ? g.nx : g.ny);
    return n < ((int64_t)1 << 31);
}

// Floats of zero padding after an h section (see the tables above).
__host__ __device__ inline int64_t bp_pad(const nr_geom& g) { return (int64_t)g.nbx + 1; }

// The tap pair (c, c + 1) of two taps at (lb, lb + 1) with weights (w0, w1)
// on a line of n detector bins, weights of off-detector taps already 0.
__device__ __forceinline__ void bp_pair(int lb, float w0, float w1, int n, int& c, float& p0,
                                        float& p1) {
    c = max(0, min(n - 2, lb));
    if (lb == c) {
        p0 = w0;
        p1 = w1;
    } else if (lb == c - 1) {  // lb = -1: only tap lb + 1 = c can be on the detector
        p0 = w1;
        p1 = 0.f;
    } else if (lb == c + 1) {  // lb = n - 1 (n >= 2): only tap lb = c + 1
        p0 = 0.f;
        p1 = w0;
    } else {                   // both taps off the detector (w0 = w1 = 0)
        p0 = 0.f;
        p1 = 0.f;
    }
}

// Taps (lb, lb + 1) on a line of n bins from lb and the fraction f, 0 <= f <= 1,
// past bin lb's centre: the pair and its weights.
__device__ __forceinline__ float4 bp_taps(int lb, float f, int n, bool valid) {
    const bool t0 = valid && (lb < n) && (lb >= 0);
    const bool t1 = valid && (lb < n - 1) && (lb >= -1);
    int c;
    float p0, p1;
    bp_pair(lb, t0 ? 1.f - f : 0.f, t1 ? f : 0.f, n, c, p0, p1);
    return make_float4(__int_as_float(c), p0, p1, 0.f);
}

// The same from a detector position in bins.
__device__ __forceinline__ float4 bp_taps_at(float mb, int n, bool valid) {
    int lb = (int)floorf(mb);
    if (mb < (float)lb + 0.5f) lb -= 1;
    return bp_taps(lb, mb - ((float)lb + 0.5f), n, valid);
}

// Detector positions along a row of voxels, A + q B bins less a half, in two
// floats each: the fraction is then rounded once (a float position of some
// thousand bins is 1e-4 bin off) without FP64 per entry.
struct BpLine {
    float ah, al, bh, bl;
};
__device__ __forceinline__ BpLine bp_line(double a, double b) {
    BpLine l;
    l.ah = (float)a;
    l.al = (float)(a - l.ah);
    l.bh = (float)b;
    l.bl = (float)(b - l.bh);
    return l;
}
__device__ __forceinline__ float4 bp_taps_on(const BpLine& l, int q, int n, bool valid) {
    const float x = (float)q;
    const float p = __fmul_rn(x, l.bh), pe = __fmaf_rn(x, l.bh, -p);
    const float s = __fadd_rn(l.ah, p), t = __fsub_rn(s, l.ah);
    const float se = __fadd_rn(__fsub_rn(l.ah, __fsub_rn(s, t)), __fsub_rn(p, t));
    const float lo = __fadd_rn(se, __fadd_rn(pe, __fmaf_rn(x, l.bl, l.al)));
    float f = floorf(s), r = __fadd_rn(__fsub_rn(s, f), lo);
    if (r >= 1.f || r < 0.f) {   // s and s + lo on two sides of an integer
        f += r < 0.f ? -1.f : 1.f;
        r = fmaxf(__fadd_rn(__fsub_rn(s, f), lo), 0.f);
    }
    return bp_taps((int)f, r, n, valid);
}

// One view's back-projection term of one voxel, added to capL, from its table
// entries ex, ey and the taps of its pair (c, c + 1) x rows (r, r + 1);
// off-detector taps are weighted 0 and their loads kept in bounds by the
// tables.
__device__ __forceinline__ void bp_view(const float* __restrict__ p, const float4 ex,
                                        const float4 ey, const nr_geom& g, float& capL) {
    const float* q0 = p + (__float_as_int(ey.x) + __float_as_int(ex.x));
    const float* q1 = q0 + g.nbx;
    const float dw = rcp_approx(ex.w + ey.w);
    const float d1 = __fmaf_rn(ex.z, __ldg(q0 + 1), __fmul_rn(ex.y, __ldg(q0)));
    const float d2 = __fmaf_rn(ex.z, __ldg(q1 + 1), __fmul_rn(ex.y, __ldg(q1)));
    capL = __fmaf_rn(__fmaf_rn(ey.z, d2, __fmul_rn(ey.y, d1)), dw, capL);
}

// The OS-SART kinds' term and its sensitivity (the same weights on ones), from
// tables with k = 1; s2 = |source|^2.
__device__ __forceinline__ void bp_sart(const float4& ex, const float4& ey, const float (&q)[4],
                                        float s2, const nr_geom& g, float& capL, float& sens) {
    const float dw = __fdividef(s2, ex.w + ey.w);
    float d1 = ex.y * q[0];
    d1 = d1 + ex.z * q[1];
    float d2 = ex.y * q[2];
    d2 = d2 + ex.z * q[3];
    capL = capL + (ey.y * d1 + ey.z * d2) * g.vz * dw;
    const float s1 = ex.y + ex.z;
    sens = sens + (ey.y * s1 + ey.z * s1) * g.vz * dw;
}

// The value of the OSTR step, xc - (M capL + beta rd) / (dv + 2 beta rdd).
__device__ __forceinline__ float ostr_step(float xc, float capL, float rd, float rdd, float dv,
                                           float M, float beta) {
    const float num = __fmaf_rn(-M, capL, __fmul_rn(-beta, rd));
    const float den = __fmaf_rn(2.f * beta, rdd, dv);
    return __fmaf_rn(num, rcp_approx(den), xc);
}

// The value of the OS-SART step (Tomo_OSTR.cu:2193-2205: u / sens and beta
// prior / sens, 0 without sensitivity); lambda in M.
template <int KIND>
__device__ __forceinline__ float sart_step(float xc, float capL, float sens, float rd, float M,
                                           float beta) {
    float ut = 0.f, bt = 0.f;
    if (sens != 0.f) {
        ut = __fdiv_rn(capL, sens);
        if (KIND == UPD_SART_R) bt = __fdiv_rn(beta * rd, sens);
    }
    return xc + M * (ut + bt);
}

__device__ __forceinline__ bool not_finite(float v) {
    return !(fabsf(v) < __int_as_float(0x7f800000));
}

// The OSTR update of one voxel from its sums, stored at out (non-finite values
// flagged in status).
__device__ __forceinline__ void upd_store(float xc, float capL, float rd, float rdd, float dv,
                                          float M, float beta, float* __restrict__ out,
                                          int* __restrict__ status) {
    const float xn = ostr_step(xc, capL, rd, rdd, dv, M, beta);
    if (not_finite(xn)) atomicOr(status, NR_FLAG_NONFINITE);
    *out = xn < 0.f ? 0.f : xn;
}

// One view's back projection onto the voxels A = (ix, iy) and B = (ix, iy + 1)
// of a thread, in the steps its loads come in: the table entries (the column
// entry serves both), then the four taps of each, then bp_view's sums, packed
// (lane 0: A, lane 1: B; each lane rounded as there).
struct UpdView {
    float4 ex, ea, eb;
    float qa[4], qb[4];
    __device__ __forceinline__ void entries(const BpTab& T, int tix, int tiy, int jb) {
        ex = __ldg(T.x + tix);
        ea = __ldg(T.y + tiy);
        eb = __ldg(T.y + (tiy + jb));
    }
    __device__ __forceinline__ void taps(const float* __restrict__ p, int nbx) {
        const float* a = p + (__float_as_int(ea.x) + __float_as_int(ex.x));
        const float* b = p + (__float_as_int(eb.x) + __float_as_int(ex.x));
        qa[0] = __ldg(a);
        qa[1] = __ldg(a + 1);
        qb[0] = __ldg(b);
        qb[1] = __ldg(b + 1);
        a += nbx;
        b += nbx;
        qa[2] = __ldg(a);
        qa[3] = __ldg(a + 1);
        qb[2] = __ldg(b);
        qb[3] = __ldg(b + 1);
    }
    __device__ __forceinline__ void add(f32x2& cap) const {
        const f32x2 dw = pk2(rcp_approx(ex.w + ea.w), rcp_approx(ex.w + eb.w));
        const f32x2 w0 = pk2(ex.y, ex.y), w1 = pk2(ex.z, ex.z);
        const f32x2 v0 = pk2(ea.y, eb.y), v1 = pk2(ea.z, eb.z);
        const f32x2 d1 = fma2(w1, pk2(qa[1], qb[1]), mul2(w0, pk2(qa[0], qb[0])));
        const f32x2 d2 = fma2(w1, pk2(qa[3], qb[3]), mul2(w0, pk2(qa[2], qb[2])));
        cap = fma2(fma2(v1, d2, mul2(v0, d1)), dw, cap);
    }
};

// The voxels a thread of the update reads of one plane, around its voxels A =
// (ix, iy) and B = (ix, iy + 1): rows iy - 1 .. iy + 2, per row the cells x -
// 1, x + 1 and x.  Each neighbour class of A or B is then two packed pairs --
// (x - 1, x + 1) of two rows, or of one row with the centre cells above and
// below -- and every value read serves both voxels.
struct UpdRows {
    float l[4], e[4], c[4];
    __device__ __forceinline__ f32x2 lr(int r) const { return pk2(l[r], e[r]); }
};

// Plane z's rows, `at` the offset of (ix, iy) in plane 0; a plane outside the
// volume reads as zeros.  EDGE: cells outside the volume in x or y read as NaN.
template <bool EDGE>
__device__ __forceinline__ void upd_rows(const nr_geom& g, const float* __restrict__ x, int z,
                                         int at, int ix, int iy, UpdRows& R) {
    const int v = z * (g.nx * g.ny) + at;
    const float qnan = __int_as_float(0x7fc00000);
    const bool zin = z >= 0 && z < g.nz;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const float* q = x + (v + (r - 1) * g.nx);
        R.c[r] = R.l[r] = R.e[r] = 0.f;
        if (EDGE) {
            const bool on = iy + r - 1 >= 0 && iy + r - 1 < g.ny;
            if (zin) {
                R.c[r] = on ? __ldg(q) : qnan;
                R.l[r] = on && ix > 0 ? __ldg(q - 1) : qnan;
                R.e[r] = on && ix + 1 < g.nx ? __ldg(q + 1) : qnan;
            }
        } else if (zin) {
            R.c[r] = __ldg(q);
            R.l[r] = __ldg(q - 1);
            R.e[r] = __ldg(q + 1);
        }
    }
}

// The penalty sums of voxels A and B, one packed accumulator pair each (the
// voxel's sum is the sum of the lanes).
struct UpdSums {
    f32x2 sdda, sda, sddb, sdb;
};

// The nine neighbours of both voxels (cells ca, cb) in the plane below (LANE
// 0) or above (LANE 1).
template <int POT, bool EDGE, int LANE>
__device__ __forceinline__ void upd_far_plane(const UpdRows& R, float ca, float cb,
                                              const PriorW5& W, float delta, float inv_delta,
                                              UpdSums& S) {
    const f32x2 a2 = pk2(ca, ca), b2 = pk2(cb, cb);
    nb_class2<POT, EDGE, W_ZCORNER>(a2, R.lr(0), R.lr(2), W, delta, inv_delta, S.sdda, S.sda);
    nb_class2<POT, EDGE, W_ZCORNER>(b2, R.lr(1), R.lr(3), W, delta, inv_delta, S.sddb, S.sdb);
    nb_class2<POT, EDGE, W_ZEDGE>(a2, R.lr(1), pk2(R.c[0], R.c[2]), W, delta, inv_delta, S.sdda,
                                  S.sda);
    nb_class2<POT, EDGE, W_ZEDGE>(b2, R.lr(2), pk2(R.c[1], R.c[3]), W, delta, inv_delta, S.sddb,
                                  S.sdb);
    nb_zface<POT, EDGE, LANE>(pk2(ca, cb), pk2(R.c[1], R.c[2]), W, delta, inv_delta, S.sdda, S.sda,
                              S.sddb, S.sdb);
}

// The eight in-plane neighbours of both voxels.
template <int POT, bool EDGE>
__device__ __forceinline__ void upd_own_plane(const UpdRows& R, const PriorW5& W, float delta,
                                              float inv_delta, UpdSums& S) {
    const f32x2 a2 = pk2(R.c[1], R.c[1]), b2 = pk2(R.c[2], R.c[2]);
    nb_class2<POT, EDGE, W_FACE>(a2, R.lr(1), pk2(R.c[0], R.c[2]), W, delta, inv_delta, S.sdda,
                                 S.sda);
    nb_class2<POT, EDGE, W_FACE>(b2, R.lr(2), pk2(R.c[1], R.c[3]), W, delta, inv_delta, S.sddb,
                                 S.sdb);
    nb_class2<POT, EDGE, W_DIAG>(a2, R.lr(0), R.lr(2), W, delta, inv_delta, S.sdda, S.sda);
    nb_class2<POT, EDGE, W_DIAG>(b2, R.lr(1), R.lr(3), W, delta, inv_delta, S.sddb, S.sdb);
}

// The OS-SART prior's gradient of voxels A and B, pair by pair as the sums of
// update_tile's first form were: the rows' (x - 1, x + 1) pairs plane by plane,
// then the centre cells' pairs, each term weighted by itself.  The order is
// kept because this step can amplify a last bit -- lambda beta RD / sens where
// few rays see a voxel -- until runs that round differently part ways.
template <bool EDGE, int CLS>
__device__ __forceinline__ void sart_pair(f32x2 c2, f32x2 n2, const PriorW5& W, f32x2& sd) {
    f32x2 t2 = sub2(c2, n2);
    const f32x2 o2 = omega2<NR_POT_HYPERBOLA, EDGE>(t2, W, 0.f, 0.f);
    sd = fma2(mul2(ld2(W.w[CLS]), o2), t2, sd);
}
// The three row pairs of a plane: classes SIDE, MID, SIDE.
template <bool EDGE, int SIDE, int MID>
__device__ __forceinline__ void sart_rows(const UpdRows& R, float ca, float cb, const PriorW5& W,
                                          UpdSums& S) {
    const f32x2 a2 = pk2(ca, ca), b2 = pk2(cb, cb);
    sart_pair<EDGE, SIDE>(a2, R.lr(0), W, S.sda);
    sart_pair<EDGE, SIDE>(b2, R.lr(1), W, S.sdb);
    sart_pair<EDGE, MID>(a2, R.lr(1), W, S.sda);
    sart_pair<EDGE, MID>(b2, R.lr(2), W, S.sdb);
    sart_pair<EDGE, SIDE>(a2, R.lr(2), W, S.sda);
    sart_pair<EDGE, SIDE>(b2, R.lr(3), W, S.sdb);
}
// The centre cells' pairs: cp the plane below, N the voxels' own, F the plane
// above; lo / hi: the planes are in the volume.
template <bool EDGE>
__device__ __forceinline__ void sart_centres(const float (&cp)[4], const UpdRows& N,
                                             const UpdRows& F, bool lo, bool hi, const PriorW5& W,
                                             UpdSums& S) {
    const float ca = N.c[1], cb = N.c[2];
    const float la = lo ? ca : 0.f, lb = lo ? cb : 0.f, ha = hi ? ca : 0.f, hb = hi ? cb : 0.f;
    sart_pair<EDGE, W_ZEDGE>(pk2(la, la), pk2(cp[0], cp[2]), W, S.sda);
    sart_pair<EDGE, W_ZEDGE>(pk2(lb, lb), pk2(cp[1], cp[3]), W, S.sdb);
    sart_pair<EDGE, W_ZEDGE>(pk2(ha, ha), pk2(F.c[0], F.c[2]), W, S.sda);
    sart_pair<EDGE, W_ZEDGE>(pk2(hb, hb), pk2(F.c[1], F.c[3]), W, S.sdb);
    sart_pair<EDGE, W_ZFACE>(pk2(la, ha), pk2(cp[1], F.c[1]), W, S.sda);
    sart_pair<EDGE, W_ZFACE>(pk2(lb, hb), pk2(cp[2], F.c[2]), W, S.sdb);
    sart_pair<EDGE, W_FACE>(pk2(ca, ca), pk2(N.c[0], N.c[2]), W, S.sda);
    sart_pair<EDGE, W_FACE>(pk2(cb, cb), pk2(N.c[1], N.c[3]), W, S.sdb);
}

// One sub-iteration's update, fused: SBP of h (subset views, [view][j][i]),
// the penalty, and the update_est step.  Each block owns a 32 x 8 tile of
// (x, y) columns and walks ZC planes in z; a thread owns two voxels of each
// plane, one above the other in y, and carries the plane's rows in registers:
// plane z - 1 and its voxels' unfinished sums (own plane and the one below)
// wait there until plane z arrives, whose rows finish them and start plane z's.
// There is no shared memory and no barrier, so warps run independently of
// each other; the rows come through L1, where the tile's threads share them,
// and are brought into L2 three planes ahead.  The order of a step gives each
// load some arithmetic to hide behind: the next plane's rows and the taps of h
// the own-plane neighbours, d and the table entries the nine below.  The back
// projection reads the separable tables (BpTab).  Writes x_out; flags
// non-finite values.
//
// The update is bound by instruction issue (DRAM traffic is at the algorithmic
// bytes).  The form before -- one voxel per thread, three planes with halo in
// a shared-memory ring, 26 shared loads and two barriers per voxel and plane --
// issued 251 instructions per voxel at 77 % issue-active, 0.262 ms per
// clinical sub-iteration; this one 188 at 64 %, 0.236 ms (full resolution
// 1.20 -> 1.08 ms).  Measured beside it: the rows through a cp.async ring of
// each warp's own (235 instructions, 0.250 ms at 74 %), the next plane's rows
// a whole step ahead (spills, 0.31 ms).
//
// KIND = UPD_SART / UPD_SART_R turn the same tile into the OS-SART update:
// h is the normalised projection difference of the subset, the back
// projection also sums the interpolation weights (the sensitivity), and
//     x' = max(0, x + lambda (sum_u + beta RD) / sum_sens)   (0 where sum_sens = 0)
// with lambda passed in M, RD the hyperbola gradient of x with unit
// neighbour distances (G_Huber_prior, Tomo_OSTR.cu:258-325; W built with
// z ratio 1) for UPD_SART_R, and d unused.
//
// NV > 0 fixes the subset's view count at compile time (nv is then NV): with
// one view per subset the per-view loop disappears.
template <int POT, int ZC = UZC, int KIND = UPD_OSTR, int NV = 0>
__device__ __forceinline__ void update_tile(
    const Geo& G, const PriorW5& W, const float* __restrict__ x, float* __restrict__ x_out,
    const float* __restrict__ d, const float* __restrict__ h, const BpTab& T, int a0, int nv,
    float M, float beta, float delta, int* __restrict__ status, int bx, int by, int bz,
    const ProjView* __restrict__ views = nullptr) {
    const nr_geom& g = G.g;
    const int x0t = bx * UTX, y0t = by * UTY;
    const int ix = x0t + threadIdx.x, iy = y0t + 2 * threadIdx.y;
    if (ix >= g.nx || iy >= g.ny) return;
    const bool has_b = iy + 1 < g.ny;   // voxel B is in the volume
    const int zb = bz * ZC, ze = min(zb + ZC, g.nz);
    // voxel and table indices in 32 bits: volumes hold fewer than 2^31 voxels
    // (geom_ok) and the tables fewer than 2^31 entries (bp_tables_fit)
    const int plane = g.nx * g.ny;
    const int at = iy * g.nx + ix;
    const int jb = has_b ? 1 : 0;       // B's offsets, kept in bounds
    const float inv_delta = 1.f / delta;
    const int64_t B = (int64_t)g.nbx * g.nby;
    UpdSums S = {0, 0, 0, 0};
    UpdView V;
    float dva = 0.f, dvb = 0.f;
    // d and the first view's table entries of plane z's voxels
    auto fetch = [&](int z) {
        const int v = z * plane + at;
        if (KIND == UPD_OSTR) {
            dva = __ldg(d + v);
            dvb = __ldg(d + (v + jb * g.nx));
        }
        V.entries(T, (a0 * g.nz + z) * g.nx + ix, (a0 * g.nz + z) * g.ny + iy, jb);
    };
    // The update of plane z's voxels ca, cb from their sums (d and the first
    // view's taps are loaded): upd_store's steps, packed for the OSTR kind.
    auto finish = [&](int z, float ca, float cb) {
        const int v = z * plane + at;
        f32x2 cap = pk2(0.f, 0.f);
        float capa = 0.f, capb = 0.f, sa = 0.f, sb = 0.f;
        auto add = [&](int t) {
            if (KIND == UPD_OSTR) {
                V.add(cap);
            } else {
                const float s2 = __ldg(&views[a0 + t].src.s2);
                bp_sart(V.ex, V.ea, V.qa, s2, g, capa, sa);
                bp_sart(V.ex, V.eb, V.qb, s2, g, capb, sb);
            }
        };
        add(0);
        if (NV != 1) {
            const float* p = h;
            int tix = (a0 * g.nz + z) * g.nx + ix;
            int tiy = (a0 * g.nz + z) * g.ny + iy;
            const int sx = g.nz * g.nx, sy = g.nz * g.ny;
            for (int t = 1; t < (NV ? NV : nv); t++) {
                p += B;
                tix += sx;
                tiy += sy;
                V.entries(T, tix, tiy, jb);
                V.taps(p, g.nbx);
                add(t);
            }
        }
        float u, w, rda, rdb, xa, xb;
        upk2(S.sda, u, w);
        rda = u + w;
        upk2(S.sdb, u, w);
        rdb = u + w;
        if (KIND == UPD_OSTR) {
            float rdda, rddb;
            upk2(S.sdda, u, w);
            rdda = u + w;
            upk2(S.sddb, u, w);
            rddb = u + w;
            const f32x2 num = fma2(pk2(-M, -M), cap, mul2(pk2(-beta, -beta), pk2(rda, rdb)));
            const f32x2 den =
                fma2(pk2(2.f * beta, 2.f * beta), pk2(rdda, rddb), pk2(dva, dvb));
            upk2(den, u, w);
            upk2(fma2(num, pk2(rcp_approx(u), rcp_approx(w)), pk2(ca, cb)), xa, xb);
        } else {
            xa = sart_step<KIND>(ca, capa, sa, rda, M, beta);
            xb = sart_step<KIND>(cb, capb, sb, rdb, M, beta);
        }
        if (not_finite(xa) || (has_b && not_finite(xb))) atomicOr(status, NR_FLAG_NONFINITE);
        x_out[v] = xa < 0.f ? 0.f : xa;
        if (has_b) x_out[v + g.nx] = xb < 0.f ? 0.f : xb;
    };
    if (KIND == UPD_SART) {
        fetch(zb);
        for (int z = zb; z < ze; z++) {
            const int v = z * plane + at;
            const float ca = __ldg(x + v), cb = __ldg(x + (v + jb * g.nx));
            V.taps(h, g.nbx);
            const UpdView U = V;
            if (z + 1 < ze) fetch(z + 1);   // the next plane's entries while the taps come
            const UpdView F = V;
            V = U;
            finish(z, ca, cb);
            V = F;
        }
        return;
    }
    // Lanes 0-7: one end of a row of the warp, of x (lanes 0-3) or d (4-7).
    const int pl = threadIdx.x & 7;
    const float* pf = (pl < 4 || KIND != UPD_OSTR ? x : d) +
                      ((iy + ((pl >> 1) & 1) * jb) * g.nx + min(x0t + (pl & 1) * (UTX - 1), g.nx - 1));
    auto prefetch = [&](int z) {
        if (threadIdx.x < 8 && z < g.nz)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(
                __cvta_generic_to_global(pf + (int64_t)z * plane)));
    };
    auto walk = [&](auto edge_c) {
        constexpr bool EDGE = decltype(edge_c)::value;
        // Starts plane z's voxels (rows N; P holds plane z - 1), then loads plane
        // z + 1 into P.
        float cp[4];   // OS-SART: the centre cells of the plane below
        auto start = [&](UpdRows& P, const UpdRows& N, int z) {
            fetch(z);
            S.sdda = S.sda = S.sddb = S.sdb = pk2(0.f, 0.f);
            // a plane outside the volume (zeros) against zeros: t = 0
            const float ca = z > 0 ? N.c[1] : 0.f, cb = z > 0 ? N.c[2] : 0.f;
            if (KIND == UPD_SART_R) {
                sart_rows<EDGE, W_ZCORNER, W_ZEDGE>(P, ca, cb, W, S);
#pragma unroll
                for (int r = 0; r < 4; r++) cp[r] = P.c[r];
            } else {
                upd_far_plane<POT, EDGE, 0>(P, ca, cb, W, delta, inv_delta, S);
            }
            upd_rows<EDGE>(g, x, z + 1, at, ix, iy, P);
            V.taps(h, g.nbx);
            prefetch(z + 3);
            if (KIND == UPD_SART_R)
                sart_rows<EDGE, W_DIAG, W_FACE>(N, N.c[1], N.c[2], W, S);
            else
                upd_own_plane<POT, EDGE>(N, W, delta, inv_delta, S);
        };
        // Plane z + 1 is in F: finishes plane z's voxels (rows N).
        auto end = [&](const UpdRows& F, const UpdRows& N, int z) {
            const bool in = z + 1 < g.nz;
            const float ca = in ? N.c[1] : 0.f, cb = in ? N.c[2] : 0.f;
            if (KIND == UPD_SART_R) {
                sart_rows<EDGE, W_ZCORNER, W_ZEDGE>(F, ca, cb, W, S);
                sart_centres<EDGE>(cp, N, F, z > 0, in, W, S);
            } else {
                upd_far_plane<POT, EDGE, 1>(F, ca, cb, W, delta, inv_delta, S);
            }
            finish(z, N.c[1], N.c[2]);
        };
        UpdRows A, C;
        prefetch(zb + 1);
        prefetch(zb + 2);
        upd_rows<EDGE>(g, x, zb - 1, at, ix, iy, A);
        upd_rows<EDGE>(g, x, zb, at, ix, iy, C);
        for (int z = zb;; z += 2) {
            start(A, C, z);
            end(A, C, z);
            if (z + 1 == ze) break;
            start(C, A, z + 1);
            end(C, A, z + 1);
            if (z + 2 == ze) break;
        }
    };
    if (x0t == 0 || x0t + UTX >= g.nx || y0t == 0 || y0t + UTY >= g.ny)
        walk(std::integral_constant<bool, true>());
    else
        walk(std::integral_constant<bool, false>());
}

// One block of 32 x 4 threads per (x, y) tile and chunk of ZC planes; NV as in
// update_tile.
template <int POT, int ZC, int NV>
__global__ void __launch_bounds__(UNT, UPD_BLOCKS) update_kernel(
    const __grid_constant__ Geo G, const __grid_constant__ PriorW5 W,
    const float* __restrict__ x, float* __restrict__ x_out, const float* __restrict__ d,
    const float* __restrict__ h, const __grid_constant__ BpTab T, int a0, int nv,
    float M, float beta, float delta, int* __restrict__ status) {
    update_tile<POT, ZC, UPD_OSTR, NV>(G, W, x, x_out, d, h, T, a0, nv, M, beta, delta, status,
                                       blockIdx.x, blockIdx.y, blockIdx.z);
}

// ---- TMA-fed ring -----------------------------------------------------------
// One voxel per thread, the planes streamed by TMA: lane 0 of warp 0 loads each plane of the tile with its
// halo (one cp.async.bulk.tensor.3d box of UTW x USH voxels starting 4 voxels
// left of the tile, so that the box's x coordinate is a multiple of 4 floats;
// out-of-volume voxels read as NaN, the ring's convention for "outside") into
// a ring of UT_SLOTS slots, each with a "full" mbarrier (the copy landed) and
// an "empty" one (all eight warps are done with the plane).  Each warp runs
// update_tile's arithmetic on its row of the tile, plane by plane, waiting
// only for the plane it needs next: there is no block-wide barrier per
// plane, so a warp held up by its back-projection loads does not hold the
// others up, and up to UT_SLOTS - 3 planes are in flight ahead of the
// slowest warp.  Warp 0 refills a slot once every warp is done with it.
// Results are bit-identical to update_tile's (same sums in the same order).
//
// Every wait is bounded.  A wait that gives up flags NR_FLAG_TIMEOUT, after
// which that thread waits no more (the tile's output is then not to be
// used; the host reads the flag as NR_ERR_TIMEOUT).  Once the issuing lane
// has given up it issues no further copy, so no slot whose readers are
// unaccounted for is refilled, and before it exits it waits (bounded) for
// every copy it issued, so none is in flight when the block's shared memory
// is released.  A first version with a ninth, producer-only warp held 7
// blocks per SM instead of 8 and ran 11 % slower on the clinical workload.
constexpr int UTW = UTX + 8;            // columns of a staged row: x0 - 4 .. x0 + 35
constexpr int USH = UTY + 2;            // rows of a staged plane
constexpr int UT_SLOT = 416;            // floats per slot: UTW x USH = 400, rounded to 128 B
constexpr int UT_SLOTS = 6;
constexpr uint32_t UT_BYTES = UTW * USH * 4;
constexpr int UT_WAIT = 1 << 22;        // polls before a wait gives up
static_assert(UTW * USH <= UT_SLOT && (UT_SLOT * 4) % 128 == 0, "slot size");

struct UpdSmemT {
    alignas(128) float ring[UT_SLOTS][UT_SLOT];
    alignas(8) uint64_t full[UT_SLOTS];
    uint64_t empty[UT_SLOTS];
};

// One z-face neighbour n of a voxel, as nb_zface forms it: lane LANE of the sums.
template <int POT, bool EDGE, int LANE>
__device__ __forceinline__ void nb_zface1(float xc, float n, const PriorW5& W, float delta,
                                          float inv_delta, f32x2& sdd, f32x2& sd) {
    f32x2 zdd = pk2(0.f, 0.f), zd = pk2(0.f, 0.f);
    nb_zface<POT, EDGE, LANE>(pk2(xc, xc), pk2(n, n), W, delta, inv_delta, sdd, sd, zdd, zd);
}

// The penalty sums of the voxel at `base` of the ring's planes below (pb), its
// own (pc) and above (pa): the terms of update_tile in its order and grouping.
template <int POT, bool EDGE>
__device__ __forceinline__ void prior_ring(const float* __restrict__ pb,
                                           const float* __restrict__ pc,
                                           const float* __restrict__ pa, int base, float xc,
                                           const PriorW5& W, float delta, float inv_delta,
                                           float* rdd, float* rd) {
    const f32x2 c2 = pk2(xc, xc);
    f32x2 sdd = pk2(0.f, 0.f), sd = pk2(0.f, 0.f);
    auto lr = [&](const float* p, int dy) {
        return pk2(p[base + dy * UTW - 1], p[base + dy * UTW + 1]);
    };
    auto ud = [&](const float* p) { return pk2(p[base - UTW], p[base + UTW]); };
    nb_class2<POT, EDGE, W_ZCORNER>(c2, lr(pb, -1), lr(pb, 1), W, delta, inv_delta, sdd, sd);
    nb_class2<POT, EDGE, W_ZEDGE>(c2, lr(pb, 0), ud(pb), W, delta, inv_delta, sdd, sd);
    nb_zface1<POT, EDGE, 0>(xc, pb[base], W, delta, inv_delta, sdd, sd);
    nb_class2<POT, EDGE, W_FACE>(c2, lr(pc, 0), ud(pc), W, delta, inv_delta, sdd, sd);
    nb_class2<POT, EDGE, W_DIAG>(c2, lr(pc, -1), lr(pc, 1), W, delta, inv_delta, sdd, sd);
    nb_class2<POT, EDGE, W_ZCORNER>(c2, lr(pa, -1), lr(pa, 1), W, delta, inv_delta, sdd, sd);
    nb_class2<POT, EDGE, W_ZEDGE>(c2, lr(pa, 0), ud(pa), W, delta, inv_delta, sdd, sd);
    nb_zface1<POT, EDGE, 1>(xc, pa[base], W, delta, inv_delta, sdd, sd);
    float u, w;
    upk2(sdd, u, w);
    *rdd = u + w;
    upk2(sd, u, w);
    *rd = u + w;
}

template <int POT, int ZC = UZC, int NV = 0>
__device__ __forceinline__ void update_tile_tma(
    const Geo& G, const PriorW5& W, const CUtensorMap* map, float* __restrict__ x_out,
    const float* __restrict__ d, const float* __restrict__ h, const BpTab& T, int a0, int nv,
    float M, float beta, float delta, int* __restrict__ status, int bx, int by, int bz,
    UpdSmemT& sm) {
    const nr_geom& g = G.g;
    const int warp = threadIdx.y, lane = threadIdx.x;
    const int tid = warp * UTX + lane;
    const int x0t = bx * UTX, y0t = by * UTY;
    const int zb = bz * ZC, ze = min(zb + ZC, g.nz);
    const int np = ze - zb + 2;  // planes zb - 1 .. ze; plane k is z = zb - 1 + k
    const bool issuer = tid == 0;
    bool issuing = true;         // the issuer: false once one of its waits gave up
    int issued = np;             // planes issued: all of them unless the issuer gave up
    auto issue = [&](int k, int s) {  // plane k into slot s = k % UT_SLOTS (its last reader done)
        tc::fence_async_smem();
        mbar_arrive_tx(&sm.full[s], UT_BYTES);
        tma_load_3d(&sm.ring[s][0], map, x0t - 4, y0t - 1, zb - 1 + k, &sm.full[s]);
    };
    if (issuer) {
        for (int s = 0; s < UT_SLOTS; s++) {
            tc::mbar_init(&sm.full[s], 1);
            tc::mbar_init(&sm.empty[s], UTY);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int k = 0; k < min(np, UT_SLOTS); k++) issue(k, k);
    }
    __syncthreads();
    bool live = true;  // false after a wait of this thread gave up: it waits no more
    // test hook: the workspace's second status word k + 1 > 0 makes the wait
    // for plane k report giving up once it has in fact succeeded
    const int force_at = status[1] - 1;
    auto wait_full = [&](int k, int s, uint32_t parity) {  // plane k, in slot s
        if (live && (!tc::mbar_wait(&sm.full[s], parity, UT_WAIT) || k == force_at)) {
            if (lane == 0) atomicOr(status, NR_FLAG_TIMEOUT);
            live = false;
        }
    };
    const int ix = x0t + lane, iy = y0t + warp;
    const bool active = ix < g.nx && iy < g.ny;
    const bool edge_xy = x0t == 0 || x0t + UTX >= g.nx || y0t == 0 || y0t + UTY >= g.ny;
    const float inv_delta = 1.f / delta;
    const int plane = g.nx * g.ny;
    const int64_t B = (int64_t)g.nbx * g.nby;
    const int base = (warp + 1) * UTW + lane + 4;
    // ring slot and barrier parity of planes k - 1, k and k + 1, carried from
    // plane to plane (slot p % UT_SLOTS, parity (p / UT_SLOTS) & 1 of plane p)
    int sb = 0, sc = 1, sa = 2;
    uint32_t qb = 0, qa = 0;
    static_assert(UT_SLOTS > 3, "planes 0..2 share the first pass of the ring");
    wait_full(0, 0, 0);
    wait_full(1, 1, 0);
    for (int z = zb; z < ze; z++) {
        const int k = z - zb + 1;  // the centre plane's ring index
        wait_full(k + 1, sa, qa);
        const float* pb = sm.ring[sb];
        const float* pc = sm.ring[sc];
        const float* pa = sm.ring[sa];
        if (active) {
            const int v = z * plane + iy * g.nx + ix;
            const float dv = __ldg(d + v);
            const float xc = pc[base];
            float capL = 0.f;
            const float* p = h;
            int tix = (a0 * g.nz + z) * g.nx + ix;
            int tiy = (a0 * g.nz + z) * g.ny + iy;
            const int sx = g.nz * g.nx, sy = g.nz * g.ny;
            for (int t = 0; t < (NV ? NV : nv); t++, p += B, tix += sx, tiy += sy)
                bp_view(p, __ldg(T.x + tix), __ldg(T.y + tiy), g, capL);
            float rdd = 0.f, rd = 0.f;
            if (edge_xy || z == 0 || z == g.nz - 1)
                prior_ring<POT, true>(pb, pc, pa, base, xc, W, delta, inv_delta, &rdd, &rd);
            else
                prior_ring<POT, false>(pb, pc, pa, base, xc, W, delta, inv_delta, &rdd, &rd);
            upd_store(xc, capL, rd, rdd, dv, M, beta, x_out + v, status);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.empty[sb]);
        // plane k - 1 + UT_SLOTS goes where plane k - 1 was, once every warp is done with it
        const int kn = k - 1 + UT_SLOTS;
        if (issuer && issuing && kn < np) {
            if (tc::mbar_wait(&sm.empty[sb], qb, UT_WAIT)) {
                issue(kn, sb);
            } else {
                atomicOr(status, NR_FLAG_TIMEOUT);
                issuing = false;
                issued = kn;
            }
        }
        // rotate: k - 1 <- k, k <- k + 1, k + 1 <- k + 2
        qb = (sc < sb) ? qb ^ 1u : qb;  // plane k's parity: plane k - 1's, flipped on a wrap
        sb = sc;
        sc = sa;
        if (++sa == UT_SLOTS) {
            sa = 0;
            qa ^= 1u;
        }
    }
    if (issuer) {
        // no copy may be in flight when the block exits
        for (int k = max(0, issued - UT_SLOTS); k < issued; k++) {
            const int s = k % UT_SLOTS;
            if (!tc::mbar_wait(&sm.full[s], (k / UT_SLOTS) & 1, UT_WAIT)) {
                atomicOr(status, NR_FLAG_TIMEOUT);
                tc::mbar_wait(&sm.full[s], (k / UT_SLOTS) & 1, UT_WAIT);
            }
        }
    }
}

// One block per (x, y) tile and chunk of ZC planes, 8 warps (one row each).
template <int POT, int ZC, int NV>
__global__ void __launch_bounds__(256, NV == 1 ? 6 : 0) update_tma_kernel(
    const __grid_constant__ Geo G, const __grid_constant__ PriorW5 W,
    const __grid_constant__ CUtensorMap map, float* __restrict__ x_out,
    const float* __restrict__ d, const float* __restrict__ h, const __grid_constant__ BpTab T,
    int a0, int nv, float M, float beta, float delta, int* __restrict__ status) {
    __shared__ UpdSmemT sm;
    update_tile_tma<POT, ZC, NV>(G, W, &map, x_out, d, h, T, a0, nv, M, beta, delta,
                                           status, blockIdx.x, blockIdx.y, blockIdx.z, sm);
}

}  // namespace nr
