// project.cuh -- the fused forward projection + OSTR gradient of one block of
// bins (device code shared by the single-reconstruction kernel in fp.cu and the
// batched kernel in batch.cu).
#pragma once

#include "reduce.cuh"
#include "walk.cuh"

namespace nr {

// Resident blocks (128 threads) per SM of the projections in the subset loops:
// the walk waits on its volume gathers, so residency pays (32 registers; 12
// blocks of 40 registers are 1.5 % slower on the clinical workload).
constexpr int FP_BLOCKS = 16;

// Detector offset of bin (i, j) of one view: JI -> [j][i] (i fastest, the
// layout of the fused path and of the scanner files); otherwise [i][j] (the
// reference's in-memory layout, Tomo_OSTR.cu:1365).
template <bool JI>
__device__ __forceinline__ int64_t bin_off(const nr_geom& g, int i, int j) {
    return JI ? (int64_t)j * g.nbx + i : (int64_t)i * g.nby + j;
}

// Fused forward projection + OSTR gradient h for the subset views of the
// device-resident path.  Detector arrays are [view][j][i] in subset order;
// y, b (and r) are indexed by the subset position a.  Rays that miss the
// volume have line = 0 (the reference zeroes the line buffer every subset,
// Tomo_OSTR_gold.cpp:843).  h = (y/(b e^-l + r) - 1) b e^-l,
// Tomo_OSTR_gold.cpp:245-260.
// One block of 32 x 4 bins (bx, by) of subset view bz, a warp per detector row.
// Every thread of the block must call it (with DATA it synchronises the block).
// views: the plan's views in subset order; rows: the warps' lists, LONG and Gmem
// as in line_integral (walk.cuh).
//
// DATA: also the subset's FP64 data term, sum over its bins of
// ybar + r - y log(ybar + r) with ybar = b exp(-l) -- the data term of the
// objective (objective.cu) restricted to these views, each bin's term formed
// exactly as there -- as this block's partial in red[block] (warp shuffles,
// then a fixed-order block sum).
template <int K = 4, bool DATA = false, bool LONG = false>
__device__ __forceinline__ void fp_h_tile(const Geo& G, const float* __restrict__ vol,
                                          float* __restrict__ h,
                                          const ProjView* __restrict__ views, int a0,
                                          const float* __restrict__ y, const float* __restrict__ b,
                                          const float* __restrict__ r, int bx, int by, int bz,
                                          float2 (*rows)[WALK_ROWS], const Geo& Gmem,
                                          double* __restrict__ red = nullptr) {
    const nr_geom& g = G.g;
    const int a = a0 + bz;
    const ProjView& view = views[a];
    const int i = bx * 32 + threadIdx.x;
    const int j = by * 4 + threadIdx.y;
    const bool on = i < g.nbx && j < g.nby;
    if (!DATA && j >= g.nby) return;
    double term = 0.0;
    float v, l = 0.f;
    if (line_integral<K, LONG>(G, Gmem, vol, view, bin_x(g, i), bin_y(g, j), on,
                               rows[threadIdx.y], &v))
        l = v * view.src.ct;
    if (on) {
        const int64_t B = (int64_t)g.nbx * g.nby;
        const int64_t o = (int64_t)a * B + bin_off<true>(g, i, j);
        const float yb = b[o] * expf(-l);
        const float rr = r ? r[o] : 0.f;
        const float den = yb + rr;
        h[(int64_t)bz * B + bin_off<true>(g, i, j)] = (__fdiv_rn(y[o], den) - 1.f) * yb;
        if (DATA) {
            const double ybd = (double)b[o] * exp(-(double)l);
            const double m = ybd + (double)rr;
            const double yy = (double)y[o];
            term = m - (yy > 0.0 ? yy * log(m) : 0.0);
        }
    }
    if (DATA)
        block_partial(term, red, ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x +
                                     blockIdx.x);
}

}  // namespace nr
