// walk.cuh -- the line integral of a warp of rays that travel down through z
// (device code of the projectors).
//
// The rays of a view all run from its source to the detector plane, so with
// the depth w = (zmax - z) / Vsize_z as the parameter (in planes, 0 at the top
// of the volume) the position of a ray in voxels is x(w) = e + s w with e and s
// functions of its detector column alone, y(w) likewise of its row, and the z
// planes lie at the integers.  The lanes of a warp hold consecutive columns
// of one row: the sequence of (y, z) cells is the same for all of them.  The
// warp builds it once as a sorted list in shared memory -- per segment the
// depth where it ends and the offset of its volume row -- and each lane
// merges the list with its own x crossings: per segment one three-input min,
// a compare that tells whose crossing comes first, and either the next x
// crossing or the next list entry.
//
// Crossing k of an axis is at fma(k, step, first), as in siddon.cuh, and the
// entry point is formed from the view's constants in double, so positions are
// at least as accurate as the walk from each ray's own entry point.  A segment
// of zero length (two crossings at one depth) is not read.
//
// Bound: instruction issue.  The walk of siddon.cuh spends about 20
// instructions per segment (three axes, each with its own test, count and
// crossing), this one about 14; times at fp_h_kernel.
#pragma once

#include "siddon.cuh"

namespace nr {

constexpr int WALK_ROWS = 256;   // list entries of a warp (2 KB)
constexpr int WALK_PAD = 8;      // entries past the last that a round of gathers may step over
constexpr float WALK_CROSSINGS = 1e6f;   // crossings of an axis: exact in FP32
constexpr float WALK_RATE = 200.f;       // y crossings per plane: a plane's fit one list

// A view's rays as functions of the bin's position, in voxels and per plane of
// depth, one line for x and one for y.  down: every ray of the view
// travels down, at most 2 mm sideways per mm and WALK_RATE rows per plane
// (steeper views, where w resolves positions less well than the path length
// does, and rays that travel up take the walk of siddon.cuh).
struct WalkLine {
    float c0, c1, s0, s1;   // position c0 + c1 bin, slope s0 + s1 bin: rounded
    float c0l, c1l;         // what c0 and c1 leave out
    // The position at the top of the volume, rounded once (the products of the
    // rounded constants would each be half an ulp of some hundred voxels off).
    __device__ __forceinline__ float at(float b) const {
        const float p = __fmul_rn(b, c1), pe = __fmaf_rn(b, c1, -p);
        const float q = __fadd_rn(p, c0), t = __fsub_rn(q, p);
        const float qe = __fadd_rn(__fsub_rn(p, __fsub_rn(q, t)), __fsub_rn(c0, t));
        return __fadd_rn(q, __fadd_rn(qe, __fadd_rn(pe, __fmaf_rn(b, c1l, c0l))));
    }
    __device__ __forceinline__ float slope(float b) const { return __fmaf_rn(b, s1, s0); }
};
struct WalkView {
    WalkLine x, y;
    int down;
};

// Whether rows of a view take more than one list: the planes and the y
// crossings of the outermost row that meets the volume, seen from the source
// straight above (an estimate: either form of the walk takes any row).
__host__ inline bool walk_long(const nr_geom& g) {
    auto reach = [&](float a, float len) {
        return fmaxf(fabsf(a - g.sourceY), fabsf(a + len - g.sourceY));
    };
    const float top = g.sourceR - (g.z_p0 + (float)g.nz * g.vz);
    float slope = reach(g.y_d0, (float)g.nby * g.by) / (g.sourceR + g.detectorR);
    if (top > 0.f) slope = fminf(slope, reach(g.y_p0, (float)g.ny * g.vy) / top);
    const float cross = fminf((float)g.ny, slope * g.vz / g.vy * (float)g.nz);
    return (float)g.nz + cross > (float)(WALK_ROWS - WALK_PAD);
}

// What the projection of a view starts from.  The device-resident paths keep
// one per view in their workspace: computed by a thread of each block (sincos
// and divisions in double) it held the block's warps at the barrier for a fifth
// of the projection's time.
struct ProjView {
    ViewSrc src;
    WalkView w;
    double x0, z0;   // the source, not rounded (the back-projection tables)
};

__device__ __forceinline__ void proj_view(const Geo& G, float theta, ProjView& V) {
    const nr_geom& g = G.g;
    double sn, cs;
    sincos((double)theta, &sn, &cs);
    V.src = view_source(g, sn, cs);
    V.x0 = (double)g.sourceR * sn;
    V.z0 = (double)g.sourceR * cs;
    const double x0 = V.src.x0, y0 = V.src.y0, z0 = V.src.z0;
    const double dz = -(double)g.detectorR - z0, rz = 1.0 / dz;
    const double at = ((double)G.zmax - z0) * rz;   // of the way at the top plane
    const double da = -(double)g.vz * rz;           // per plane
    const double rx = 1.0 / g.vx, ry = g.vy == g.vx ? rx : 1.0 / g.vy;
    auto line = [&](WalkLine& l, double o, double p0, double r) {
        const double c1 = at * r, c0 = (o * (1.0 - at) - p0) * r;
        l.c1 = (float)c1;
        l.c0 = (float)c0;
        l.c1l = (float)(c1 - l.c1);
        l.c0l = (float)(c0 - l.c0);
        l.s1 = (float)(da * r);
        l.s0 = (float)(-o * da * r);
    };
    line(V.w.x, x0, g.x_p0, rx);
    line(V.w.y, y0, g.y_p0, ry);
    // the extreme bins bound every ray's slope, and with it the crossings counted
    const float fz = (float)dz;
    bool down = fz < 0.f;
    for (int c = 0; c < 2; c++) {
        const float x = bin_x(g, c ? g.nbx - 1 : 0), y = bin_y(g, c ? g.nby - 1 : 0);
        down = down && fabsf(x - V.src.x0) <= -2.f * fz && fabsf(y - V.src.y0) <= -2.f * fz;
        const float ex = fabsf(V.w.x.at(x)) + (float)g.nz * fabsf(V.w.x.slope(x));
        const float ey = fabsf(V.w.y.at(y)) + (float)g.nz * fabsf(V.w.y.slope(y));
        down = down && ex < WALK_CROSSINGS && ey < WALK_CROSSINGS &&
               fabsf(V.w.y.slope(y)) <= WALK_RATE;
    }
    V.w.down = down;
}

// One axis of a ray: crossing c (c >= 0) at fma(c, step, first), the cell
// before it i0 + dir c; rate = 1 / step.  dir = 0: no crossing (first = inf).
struct DepthAxis {
    float first, step, rate;
    int i0, dir;
};

__device__ __forceinline__ DepthAxis depth_axis(float e, float s) {
    DepthAxis a;
    const float f = floorf(e);
    a.i0 = (int)f;
    a.rate = fabsf(s);
    a.step = __fdiv_rn(1.f, a.rate);
    if (!(a.step < NR_FINF)) {
        a.dir = 0;
        a.rate = 0.f;
        a.step = a.first = NR_FINF;
        return a;
    }
    a.dir = s > 0.f ? 1 : -1;
    a.first = (s > 0.f ? (f + 1.f) - e : e - f) * a.step;
    return a;
}

__device__ __forceinline__ float depth_crossing(const DepthAxis& a, int c) {
    return a.dir == 0 ? NR_FINF : __fmaf_rn((float)c, a.step, a.first);
}

// The first crossing after depth w (AT: at or after it).
template <bool AT>
__device__ __forceinline__ int depth_first(const DepthAxis& a, float w) {
    if (a.dir == 0) return 0;
    int c = max(0, (int)((w - a.first) * a.rate));
    auto past = [&](int k) {
        const float t = depth_crossing(a, k);
        return AT ? t >= w : t > w;
    };
    while (c > 0 && past(c - 1)) c--;
    while (!past(c)) c++;
    return c;
}

// Depths [lo, hi) at which the axis lies inside [0, n] (e its cell at depth 0).
__device__ __forceinline__ void depth_range(const DepthAxis& a, float e, int n, float& lo,
                                            float& hi) {
    lo = -NR_FINF;
    hi = NR_FINF;
    if (a.dir == 0) {
        if (!(e > 0.f && e < (float)n)) hi = -NR_FINF;
    } else if (a.dir > 0) {
        if (e < 0.f) lo = depth_crossing(a, -(a.i0 + 1));
        hi = a.i0 < n ? depth_crossing(a, n - (a.i0 + 1)) : -NR_FINF;
    } else {
        if (e > (float)n) lo = depth_crossing(a, a.i0 - n);
        hi = a.i0 >= 0 ? depth_crossing(a, a.i0) : -NR_FINF;
    }
}

// The list of a stretch of a detector row: entries (end depth, offset of the
// volume row as int bits), n of them, from depth w0 to w1.  more: the row goes
// on below w1.
struct RowList {
    int n;
    float w0, w1;
    bool more;
};

// Built by a whole warp; y1: the row's bin centre, from: the end of the stretch
// before (0: none).  n = 0 when the row misses the volume in y.  WHOLE: only
// a row that one list holds (n = -1: more).
template <bool WHOLE>
__device__ __forceinline__ RowList row_list(const nr_geom& g, const WalkView& V, float y1,
                                            float from, float2* __restrict__ L) {
    RowList R;
    const float e = V.y.at(y1);
    const DepthAxis Y = depth_axis(e, V.y.slope(y1));
    depth_range(Y, e, g.ny, R.w0, R.w1);
    R.w0 = fmaxf(R.w0, from);
    R.w1 = fminf(R.w1, (float)g.nz);
    R.n = 0;
    R.more = false;
    if (!(R.w0 < R.w1)) return R;
    const int ca = depth_first<false>(Y, R.w0);   // y crossings inside: ca, ca + 1, ...
    const int ka = (int)R.w0 + 1;                 // z planes inside: ka, ka + 1, ...
    int ny = max(0, depth_first<true>(Y, R.w1) - ca);
    int nz = max(0, (int)ceilf(R.w1) - ka);
    if (ny + nz + 1 + WALK_PAD > WALK_ROWS) {
        if (WHOLE) {
            R.n = -1;
            return R;
        }
        // p planes hold at most p rate + 2 crossings and p - 1 planes inside
        const int p = max(1, (int)__fdividef((float)(WALK_ROWS - WALK_PAD - 4), 1.f + Y.rate));
        R.more = (float)(ka - 1 + p) < R.w1;
        R.w1 = fminf(R.w1, (float)(ka - 1 + p));
        ny = max(0, depth_first<true>(Y, R.w1) - ca);
        nz = max(0, (int)ceilf(R.w1) - ka);
        ny = min(ny, WALK_ROWS - WALK_PAD - 1 - nz);
    }
    R.n = ny + nz + 1;
    const int lane = threadIdx.x;
    auto put = [&](int at, float w, int planes, int rows) {
        const int z = g.nz - ka - planes;
        const int y = max(0, min(g.ny - 1, Y.i0 + Y.dir * (ca + rows)));
        L[at] = make_float2(w, __int_as_float((z * g.ny + y) * g.nx));
    };
    __syncwarp();   // the warp's earlier readers of L are done
    for (int t = lane; t < nz; t += 32) {
        const float w = (float)(ka + t);
        const int r = Y.dir == 0 ? 0 : min(ny, max(0, depth_first<true>(Y, w) - ca));
        put(t + r, w, t, r);
    }
    for (int t = lane; t < ny; t += 32) {
        const float w = depth_crossing(Y, ca + t);
        const int p = min(nz, max(0, (int)w - ka + 1));
        put(t + p, w, p, t);
    }
    for (int t = lane; t <= WALK_PAD; t += 32)
        put(ny + nz + t, t == 0 ? R.w1 : NR_FINF, nz, ny);
    __syncwarp();
    return R;
}

// Adds to *out the segments of one ray, its length in depth times the voxel it
// lies in each: the ray of column x1 through the row list R, L.  K steps per
// round of reads (K <= WALK_PAD), as in siddon.cuh.  False when the ray misses.
template <int K>
__device__ __forceinline__ bool depth_walk(const nr_geom& g, const WalkView& V, const RowList& R,
                                           const float2* __restrict__ L,
                                           const float* __restrict__ vol, float x1, float* out) {
    static_assert(K <= WALK_PAD, "list padding");
    const float e = V.x.at(x1);
    const DepthAxis X = depth_axis(e, V.x.slope(x1));
    float s, end;
    depth_range(X, e, g.nx, s, end);
    s = fmaxf(s, R.w0);
    end = fminf(end, R.w1);
    if (!(s < end)) return false;
    const int c = depth_first<false>(X, s);
    float cx = (float)c, tx = depth_crossing(X, c);
    int xi = X.i0 + X.dir * c;
    if (s > R.w0) {  // entry through a side: the first list entry that ends after s
        int lo = 0, hi = R.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (L[mid].x > s) hi = mid;
            else lo = mid + 1;
        }
        L += lo;
    }
    float2 ent = *L;
    float sum = *out;
    while (s < end) {
        float seg[K];
        int id[K];
        bool on[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            const float m = fmin3(tx, ent.x, end);
            on[k] = s < m;
            seg[k] = m - s;
            id[k] = __float_as_int(ent.y) + xi;
            s = m;
            if (tx < ent.x) {
                cx += 1.f;
                tx = __fmaf_rn(cx, X.step, X.first);
                xi += X.dir;
            } else {
                L++;
                ent = *L;
            }
        }
        float v[K];
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = on[k] ? __ldg(vol + id[k]) : 0.f;
#pragma unroll
        for (int k = 0; k < K; k++)
            if (on[k]) sum = __fmaf_rn(seg[k], v[k], sum);
    }
    *out = sum;
    return true;
}

// Path length (mm) per plane of depth of the ray to the bin at (x1, y1).
__device__ __forceinline__ float depth_mm(const nr_geom& g, const ViewSrc& S, float x1, float y1) {
    const float dx = x1 - S.x0, dy = y1 - S.y0, dz = -g.detectorR - S.z0;
    return __fdiv_rn(g.vz * sqrtf(dx * dx + dy * dy + dz * dz), fabsf(dz));
}

// line_integral for the rows that take several lists and for the views of the
// general walk: {value, 1 where the ray meets the volume}.
template <int K>
__device__ __forceinline__ float2 line_far(const Geo& G, const float* __restrict__ vol,
                                           const ProjView& V, float x1, float y1, bool on,
                                           float2* __restrict__ L) {
    const nr_geom& g = G.g;
    float sum = 0.f;
    bool hit = false;
    if (V.w.down) {
        RowList R;
        R.w1 = 0.f;
        do {
            R = row_list<false>(g, V.w, y1, R.w1, L);
            if (R.n > 0 && on) hit |= depth_walk<K>(g, V.w, R, L, vol, x1, &sum);
        } while (R.more);
        sum *= depth_mm(g, V.src, x1, y1);
    } else if (on) {
        hit = trace<0, K>(G, vol, V.src.x0, V.src.y0, V.src.z0, x1, y1, -g.detectorR, &sum);
    }
    return make_float2(sum, hit ? 1.f : 0.f);
}
template <int K>
__device__ __noinline__ float2 line_far_call(const Geo& G, const float* __restrict__ vol,
                                             const ProjView& V, float x1, float y1, bool on,
                                             float2* __restrict__ L) {
    return line_far<K>(G, vol, V, x1, y1, on, L);
}

// The line integral of the ray to (x1, y1), called by a whole warp with one y1
// (on: the lane has a ray).  False (out untouched) where the ray misses the
// volume.  L: the warp's list, WALK_ROWS entries of shared memory.  LONG: for
// volumes whose rows take several lists (walk_long); otherwise those are walked
// out of line, so that the common walk keeps its registers (FP_BLOCKS).  Gmem:
// G where it lies in memory, for that call (the address of a copy in registers
// would put the copy on the stack).
template <int K, bool LONG = false>
__device__ __forceinline__ bool line_integral(const Geo& G, const Geo& Gmem,
                                              const float* __restrict__ vol, const ProjView& V,
                                              float x1, float y1, bool on,
                                              float2* __restrict__ L, float* out) {
    const nr_geom& g = G.g;
    if (!LONG && V.w.down) {
        const RowList R = row_list<true>(g, V.w, y1, 0.f, L);
        if (R.n == 0) return false;
        if (R.n > 0) {
            float sum = 0.f;
            if (!on || !depth_walk<K>(g, V.w, R, L, vol, x1, &sum)) return false;
            *out = sum * depth_mm(g, V.src, x1, y1);
            return true;
        }
    }
    const float2 r = LONG ? line_far<K>(G, vol, V, x1, y1, on, L)
                          : line_far_call<K>(Gmem, vol, V, x1, y1, on, L);
    if (r.y != 0.f) *out = r.x;
    return r.y != 0.f;
}

}  // namespace nr
