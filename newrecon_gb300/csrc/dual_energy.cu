// dual_energy.cu -- weighted dual-energy subtraction of two reconstructions.
//
// syncrecon.m (the reference's post-processing of a high- and a low-energy
// OSTR volume) forms, for every weight w of a list, d = he - le * w and writes
// d as float32; it prints the entropy of one slice of each d, and computes an
// Otsu threshold of he (graythresh) whose mask it applies in commented-out
// lines.  MATLAB reads the float32 files as double, so d is
//     float(double(he) - double(le) * w)        (two roundings in double)
// which the kernel reproduces bit for bit: in FP32 by error-free transforms
// where a bound on what they drop decides the rounding (de_fast2), and with
// separate double multiply and subtract (no contraction to an FMA) where it
// cannot -- GB300's FP64 pipe runs at about 1/64 of the FP32 rate.  The K
// outputs of one voxel are written from one read of he and le.
//
// Image-statistics helpers (the 8-bit conversion of MATLAB's entropy and
// graythresh): a value v maps to bin round(255 v) (half away from zero),
// saturated to [0, 255], NaN to 0.
#include <cmath>

#include "common.cuh"

namespace nr {

constexpr int DE_MAX_WEIGHTS = 16;
constexpr int DE_BLOCKS = 4;  // per SM, all resident

struct DeWeights {
    double w[DE_MAX_WEIGHTS];
    float w1[DE_MAX_WEIGHTS], w2[DE_MAX_WEIGHTS];  // w = w1 + w2 + (|.| <= 2^-47 |w|)
    unsigned fast;     // bit k: weight k takes the FP32 path (de_fast2)
    unsigned pow2;     // bit k: weight k is a power of two (a w exact in float)
    int k;
    int masked;        // 1: he and le multiplied by (he > level) first
    double level;
    float level_f;     // the largest float <= level: (double)h > level iff h > level_f
};

__device__ __forceinline__ int im8_bin(double v) {
    if (!(v == v)) return 0;
    const double r = round(255.0 * v);   // CUDA round(): half away from zero
    return r <= 0.0 ? 0 : (r >= 255.0 ? 255 : (int)r);
}

__device__ __forceinline__ double de_value(double h, double l, double w) {
    return __dadd_rn(h, -__dmul_rn(l, w));
}

// The FP32 evaluation of double(b) - double(a) * w, without the FP64 pipe.
//
// a w1 = p1 + e1 exactly (FMA), a w2 rounds once; two error-free sums give
// b - a w ~ hi + lo with hi = RN(hi + lo).  The terms dropped on the way (a
// w2's rounding and the w tail, under 2^-47 |p1|; the float sums of the
// small terms, under 2^-48 (2 |s| + 3 |p1|), s = RN(b - p1)) and both
// roundings of the double evaluation (under 2^-53 (|b| + 2 |p1|)) add up to
// less than 2^-45.2 |p1| + 2^-46.9 |b|; B = 2^-44 |p1| + 2^-46 |b| bounds
// them with a factor of 1.8 to spare.
// b - a w ~ hi + lo as above, with B bounding |the double value - (hi + lo)|;
// false for tiny, huge or non-finite products.
__device__ __forceinline__ bool de_sum(float b, float a, float w1, float w2, float& hi, float& lo,
                                       float& B) {
    const float p1 = __fmul_rn(a, w1);
    const float ap1 = fabsf(p1);
    if (!(ap1 >= 0x1p-100f && ap1 <= 0x1p100f)) return false;
    const float e1 = __fmaf_rn(a, w1, -p1);
    const float q = __fmul_rn(a, w2);
    const float s = __fsub_rn(b, p1);  // TwoSum(b, -p1)
    const float bp = __fsub_rn(s, b);
    const float ap = __fsub_rn(s, bp);
    const float serr = __fsub_rn(__fsub_rn(b, ap), __fadd_rn(p1, bp));
    const float t = __fsub_rn(__fsub_rn(serr, e1), q);
    hi = __fadd_rn(s, t);  // TwoSum(s, t)
    const float tp = __fsub_rn(hi, s);
    const float sp = __fsub_rn(hi, tp);
    lo = __fadd_rn(__fsub_rn(s, sp), __fsub_rn(t, tp));
    B = __fmaf_rn(fabsf(b), 0x1p-46f, __fmul_rn(ap1, 0x1p-44f));
    return true;
}

// float(double(b) - double(a) * w) for a weight of the fast class, and a bit
// for each of the two the FP32 evaluation did not decide.  As de_sum with a w2 + e1 in one FMA:
// b - a w = s + t + (dropped terms), and the double evaluation lies within B of
// s + t, B = 2^-43 |p1| + 2^-45 |b|.  The dropped terms and the double's own
// roundings are below 2^-45.2 |p1| + 2^-46.9 |b| as above (one rounding less),
// and rounding t + B and t - B, |t| <= 2^-24 (|b| + 3 |p1|), adds at most
// 2^-46.3 |p1| + 2^-47.9 |b|: a factor of 2 to spare.  Rounding is monotone: where
// s + (t + B) and s + (t - B) round to one float, so does the double value.
// Overflow gives an infinity less an infinity on the way, a NaN, which decides
// nothing.  |p1| >= min_p: 2^-100, where every error term is a normal number or
// exact; 0 for a voxel with a = 0 and b not -0, whose terms are all exact and
// whose zeros come out positive as in double.
//
// Two voxels at a time in packed pairs and without a branch: 16 instructions per
// output of 22 in scalar form (the kernel is bound by instruction issue).
__device__ __forceinline__ uint32_t de_fast2(f32x2 b, float bb0, float bb1, float a0, float a1,
                                             float min0, float min1, float w1, float w2, float& r0,
                                             float& r1) {
    const f32x2 neg = pk2(-1.f, -1.f), a = pk2(a0, a1);
    const float p0 = __fmul_rn(a0, -w1), p1 = __fmul_rn(a1, -w1);  // -p1 of each
    const f32x2 np = pk2(p0, p1);
    const f32x2 t1 = fma2(a, pk2(w2, w2), fma2(a, pk2(w1, w1), np));
    const f32x2 s = add2(b, np);  // TwoSum(b, -p1)
    const f32x2 bp = fma2(b, neg, s);
    const f32x2 ap = fma2(bp, neg, s);
    const f32x2 serr = add2(fma2(ap, neg, b), fma2(bp, neg, np));
    const f32x2 t = fma2(t1, neg, serr);
    const f32x2 B = pk2(__fmaf_rn(fabsf(p0), 0x1p-43f, bb0), __fmaf_rn(fabsf(p1), 0x1p-43f, bb1));
    float d0, d1;
    upk2(add2(s, add2(t, B)), r0, r1);
    upk2(add2(s, fma2(B, neg, t)), d0, d1);
    return (r0 == d0 && fabsf(p0) >= min0 ? 0u : 1u) | (r1 == d1 && fabsf(p1) >= min1 ? 0u : 2u);
}

// im8_bin of a double value v known as |v - (hi + lo)| <= B: round(255 v)
// half away from zero, saturated to [0, 255]; -1 when v lies too close to a
// bin edge (255 v = k + 1/2) for the float evaluation to tell.
__device__ __forceinline__ int de_bin(float hi, float lo, float B) {
    const float yh = __fmul_rn(255.f, hi);
    const float ye = __fmaf_rn(255.f, hi, -yh);  // exact
    const float y = __fadd_rn(yh, __fmaf_rn(255.f, lo, ye));
    const float err = __fmaf_rn(255.f, B, __fmaf_rn(fabsf(y), 0x1p-22f, 0x1p-40f));
    const float f = floorf(__fadd_rn(y, 0.5f));
    const float dist = __fsub_rn(0.5f, fabsf(__fsub_rn(y, f)));
    if (!(dist > err)) return -1;  // also NaN
    return f <= 0.f ? 0 : (f >= 255.f ? 255 : (int)f);
}

// The FP64 evaluation, out of line: inlined, ptxas predicates it and runs
// it for every output beside the FP32 one.
__device__ __noinline__ float de_slow(float b, float a, double w) {
    return __double2float_rn(de_value(b, a, w));
}

// A weight that is a power of two: a w is exact, and double(b) - a w needs more
// than 53 bits only when one operand is below 2^-29 of the other, where both
// roundings land on the float of b - a w (the nearest float midpoint is 2^-25
// away).
__device__ __forceinline__ bool de_pow2(float b, float a, float w1, float& r) {
    const float p = __fmul_rn(a, w1);
    r = __fsub_rn(b, p);
    return a == 0.f || (fabsf(p) >= 0x1p-100f && fabsf(p) <= 0x1p100f);
}

// d[k][i] = float(he[i] - le[i] * w_k), 128 voxels per warp and step.  VEC (n a
// multiple of 4, so that every output row d + k n stays 16-byte aligned): a
// lane's voxels are adjacent, with 16-byte loads and stores; otherwise they lie
// 32 apart.
//
// What FP32 leaves open is not rare where the weights are tenths: for one a in
// ten the exact product lies within 2^-53 of a float, and 2 to 3 % of the
// outputs are ties that the double product's own rounding decides.  One such
// lane holds its warp for the FP64 instructions' full time (evaluated in place,
// the FP64 pipe was 66 % busy and bound the kernel), so a warp writes its open
// outputs' numbers to a list and evaluates the list with all lanes.
//
// Bound by instruction issue (231 M warp instructions, 66 % issue): 280 us for
// nine weights of 1024 x 512 x 60 (its 1.38 GB take 204 us), from 790 us with
// FP64 in place; 350 us with scalar FP32.
constexpr int DE_TILE = 128;

template <bool VEC>
__global__ void __launch_bounds__(256, DE_BLOCKS) de_subtract_kernel(
    const float* he, const float* le, float* d, int64_t n,
    const __grid_constant__ DeWeights W) {
    __shared__ uint16_t list[8][DE_TILE * DE_MAX_WEIGHTS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint16_t* open = list[warp];
    const int64_t step = (int64_t)gridDim.x * 8 * DE_TILE;
    for (int64_t i0 = (blockIdx.x * 8 + warp) * (int64_t)DE_TILE; i0 < n; i0 += step) {
        const int64_t i = i0 + (VEC ? 4 * lane : lane);
        float h[4] = {0.f, 0.f, 0.f, 0.f}, l[4] = {0.f, 0.f, 0.f, 0.f}, hb[4], lm[4];
        if (VEC) {
            if (i < n) {
                // plain loads: d may lie over he or le, which rules out the
                // read-only path
                const float4 h4 = *reinterpret_cast<const float4*>(he + i);
                const float4 l4 = *reinterpret_cast<const float4*>(le + i);
                h[0] = h4.x; h[1] = h4.y; h[2] = h4.z; h[3] = h4.w;
                l[0] = l4.x; l[1] = l4.y; l[2] = l4.z; l[3] = l4.w;
            }
        } else {
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (i + 32 * t < n) {
                    h[t] = he[i + 32 * t];
                    l[t] = le[i + 32 * t];
                }
        }
#pragma unroll
        for (int t = 0; t < 4; t++) {
            if (W.masked && !(h[t] > W.level_f)) h[t] = l[t] = 0.f;
            hb[t] = __fmul_rn(fabsf(h[t]), 0x1p-45f);
            lm[t] = l[t] == 0.f && __float_as_uint(h[t]) != 0x80000000u ? 0.f : 0x1p-100f;
        }
        const int lim = (int)(n - i < DE_TILE ? n - i : DE_TILE);
        // nothing to subtract in the warp's voxels (air, a masked background)
        const bool air = __all_sync(0xffffffffu, lm[0] == 0.f && lm[1] == 0.f && lm[2] == 0.f &&
                                                     lm[3] == 0.f);
        uint64_t bad = 0;  // bit 4 k + t: weight k of voxel t is left to FP64
        float* row = d + i;
#pragma unroll 1
        for (int k = 0; k < W.k; k++, row += n) {
            float o[4];
            uint32_t m = 0;
            if ((W.pow2 >> k) & 1u) {
#pragma unroll
                for (int t = 0; t < 4; t++)
                    m |= de_pow2(h[t], l[t], W.w1[k], o[t]) ? 0u : 1u << t;
            } else if ((W.fast >> k) & 1u) {
                const float w1 = W.w1[k], w2 = W.w2[k];
                if (air) {
#pragma unroll
                    for (int t = 0; t < 4; t++) o[t] = __fsub_rn(h[t], __fmul_rn(l[t], w1));
                } else {
#pragma unroll
                    for (int t = 0; t < 4; t += 2)
                        m |= de_fast2(pk2(h[t], h[t + 1]), hb[t], hb[t + 1], l[t], l[t + 1], lm[t],
                                      lm[t + 1], w1, w2, o[t], o[t + 1]) << t;
                }
            } else {
#pragma unroll
                for (int t = 0; t < 4; t++) o[t] = de_slow(h[t], l[t], W.w[k]);
            }
            bad |= (uint64_t)m << (4 * k);
            if (VEC) {
                if (i < n)
                    __stcs(reinterpret_cast<float4*>(row), make_float4(o[0], o[1], o[2], o[3]));
            } else {
#pragma unroll
                for (int t = 0; t < 4; t++)
                    if (32 * t < lim) __stcs(row + 32 * t, o[t]);
            }
        }
        if (!__any_sync(0xffffffffu, bad != 0)) continue;
        const int cnt = __popcll(bad);
        int end = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += up;
        }
        const int total = __shfl_sync(0xffffffffu, end, 31);
        int pos = end - cnt;
        for (; bad; bad &= bad - 1) open[pos++] = (uint16_t)(((__ffsll(bad) - 1) << 5) | lane);
        __syncwarp();  // the list, and the stores above before those below
        // he and le from their lanes' registers: d may lie over them
        for (int j0 = 0; j0 < total; j0 += 32) {
            const bool on = j0 + lane < total;
            const int e = on ? open[j0 + lane] : 0, t = (e >> 5) & 3, k = e >> 7, from = e & 31;
            float b = 0.f, a = 0.f;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float bu = __shfl_sync(0xffffffffu, h[u], from);
                const float au = __shfl_sync(0xffffffffu, l[u], from);
                if (t == u) {
                    b = bu;
                    a = au;
                }
            }
            if (on)
                d[(int64_t)k * n + i0 + (VEC ? 4 * from + t : from + 32 * t)] =
                    __double2float_rn(de_value(b, a, W.w[k]));
        }
        __syncwarp();
    }
}

// hist[k][b] += voxels of [begin, begin + len) whose double d_k falls in bin
// b; the double value (before rounding to float) as MATLAB's entropy sees it.
__global__ void __launch_bounds__(256) de_hist_kernel(const float* __restrict__ he,
                                                      const float* __restrict__ le,
                                                      int64_t begin, int64_t len,
                                                      int* __restrict__ hist,
                                                      const __grid_constant__ DeWeights W) {
    __shared__ int sh[DE_MAX_WEIGHTS * 256];
    for (int t = threadIdx.x; t < W.k * 256; t += blockDim.x) sh[t] = 0;
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < len;
         i += (int64_t)gridDim.x * blockDim.x) {
        float h = he[begin + i], l = le[begin + i];
        if (W.masked && !(h > W.level_f)) h = l = 0.f;
        for (int k = 0; k < W.k; k++) {
            int bin = -1;
            if ((W.fast >> k) & 1u) {
                float hi = h, lo = 0.f, B = 0.f;  // a = 0: the double value is b
                if (l == 0.f || de_sum(h, l, W.w1[k], W.w2[k], hi, lo, B)) bin = de_bin(hi, lo, B);
            }
            if (bin < 0) bin = im8_bin(de_value(h, l, W.w[k]));
            atomicAdd(&sh[k * 256 + bin], 1);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < W.k * 256; t += blockDim.x)
        if (sh[t]) atomicAdd(&hist[t], sh[t]);
}

// hist[b] += voxels of x in bin b (graythresh's 8-bit histogram).
__global__ void __launch_bounds__(256) hist8_kernel(const float* __restrict__ x, int64_t n,
                                                    int* __restrict__ hist) {
    __shared__ int sh[256];
    sh[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&sh[im8_bin((double)x[i])], 1);
    __syncthreads();
    if (sh[threadIdx.x]) atomicAdd(&hist[threadIdx.x], sh[threadIdx.x]);
}

static unsigned de_blocks(int64_t work) {
    const int64_t b = (work + 255) / 256, most = 16 * sm_count();
    return (unsigned)(b > most ? most : (b < 1 ? 1 : b));
}

}  // namespace nr

using namespace nr;

NR_API nr_status nr_de_subtract(const float* he, const float* le, const double* weights,
                                int32_t n_weights, int64_t n, double mask_level, float* d,
                                int64_t hist_begin, int64_t hist_len, int32_t* hist,
                                void* stream) {
    if (!he || !le || !weights || !d || n < 0) return NR_ERR_BAD_ARGUMENT;
    if (n_weights < 1 || n_weights > DE_MAX_WEIGHTS) return NR_ERR_BAD_ARGUMENT;
    if (hist && (hist_begin < 0 || hist_len < 0 || hist_begin + hist_len > n))
        return NR_ERR_BAD_ARGUMENT;
    if (((uintptr_t)he | (uintptr_t)le | (uintptr_t)d) & 15) return NR_ERR_BAD_ARGUMENT;
    // float4 path: he, le, d 16-byte aligned (checked) and n % 4 == 0, so each
    // row d + k n is aligned too; q < n/4 keeps every access below n.
    DeWeights W;
    W.fast = 0u;
    W.pow2 = 0u;
    for (int k = 0; k < DE_MAX_WEIGHTS; k++) {
        const double w = k < n_weights ? weights[k] : 0.0;
        W.w[k] = w;
        // w = w1 + w2 + w3: both differences are exact in double
        const float w1 = (float)w;
        const float w2 = (float)(w - (double)w1);
        const double w3 = (w - (double)w1) - (double)w2;
        W.w1[k] = w1;
        W.w2[k] = w2;
        const double aw = std::fabs(w);
        if (k < n_weights && std::isfinite(w) && aw >= 0x1p-60 && aw <= 0x1p60 &&
            std::fabs(w3) <= std::ldexp(aw, -47))
            W.fast |= 1u << k;
        int ex = 0;
        if (k < n_weights && std::isfinite(w) && w != 0.0 && std::fabs(std::frexp(w, &ex)) == 0.5 &&
            ex > -90 && ex < 90)
            W.pow2 |= 1u << k;
    }
    W.k = n_weights;
    W.masked = mask_level >= 0.0;
    W.level = mask_level;
    float lf = (float)mask_level;
    if ((double)lf > mask_level) lf = std::nextafterf(lf, -INFINITY);
    W.level_f = lf;
    cudaStream_t s = as_stream(stream);
    // first, while he and le are as given: d may lie over them
    if (hist) {
        if (cudaMemsetAsync(hist, 0, (size_t)n_weights * 256 * sizeof(int32_t), s) != cudaSuccess)
            return NR_ERR_CUDA;
        if (hist_len > 0)
            de_hist_kernel<<<de_blocks(hist_len), 256, 0, s>>>(he, le, hist_begin, hist_len,
                                                               hist, W);
    }
    const int64_t steps = (n + 8 * DE_TILE - 1) / (8 * DE_TILE);
    const int64_t most = DE_BLOCKS * sm_count();
    const unsigned blocks = (unsigned)(steps > most ? most : steps);
    if (n > 0 && n % 4 == 0)
        de_subtract_kernel<true><<<blocks, 256, 0, s>>>(he, le, d, n, W);
    else if (n > 0)
        de_subtract_kernel<false><<<blocks, 256, 0, s>>>(he, le, d, n, W);
    return launch_status();
}

NR_API nr_status nr_hist8(const float* x, int64_t n, int32_t* hist, void* stream) {
    if (!x || !hist || n < 0) return NR_ERR_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    if (cudaMemsetAsync(hist, 0, 256 * sizeof(int32_t), s) != cudaSuccess) return NR_ERR_CUDA;
    if (n > 0) hist8_kernel<<<de_blocks(n), 256, 0, s>>>(x, n, hist);
    return launch_status();
}

// Host: Shannon entropy (bits) of a 256-bin histogram of `count` values,
// -sum p log2 p over the non-empty bins, p = hist / count.
NR_API nr_status nr_hist_entropy(const int32_t* hist, int64_t count, double* entropy) {
    if (!hist || !entropy || count <= 0) return NR_ERR_BAD_ARGUMENT;
    double e = 0.0;
    for (int b = 0; b < 256; b++) {
        if (hist[b] <= 0) continue;
        const double p = (double)hist[b] / (double)count;
        e -= p * std::log2(p);
    }
    *entropy = e;
    return NR_OK;
}

// Host: Otsu's threshold (Otsu 1979) of a 256-bin histogram: the bin k that
// maximises the between-class variance (mu_T w(k) - mu(k))^2 / (w(k)(1 - w(k))),
// w and mu the cumulative class probability and first moment; with several
// maxima the mean of their indices; returned as k / 255 (0 when the maximum is
// not finite, e.g. one occupied bin).
NR_API nr_status nr_otsu_level(const int32_t* hist, double* level) {
    if (!hist || !level) return NR_ERR_BAD_ARGUMENT;
    double total = 0.0;
    for (int b = 0; b < 256; b++) total += hist[b] > 0 ? (double)hist[b] : 0.0;
    if (!(total > 0.0)) return NR_ERR_BAD_ARGUMENT;
    double sb[256], w = 0.0, mu = 0.0, mu_t = 0.0;
    for (int b = 0; b < 256; b++) mu_t += (hist[b] > 0 ? hist[b] / total : 0.0) * (b + 1);
    double best = -1.0;
    for (int b = 0; b < 256; b++) {
        const double p = hist[b] > 0 ? hist[b] / total : 0.0;
        w += p;
        mu += p * (b + 1);
        const double num = mu_t * w - mu;
        sb[b] = num * num / (w * (1.0 - w));
        if (sb[b] > best) best = sb[b];   // NaN/inf never win: compared below
    }
    if (!(best >= 0.0) || !(best < INFINITY)) {
        *level = 0.0;
        return NR_OK;
    }
    double sum = 0.0;
    int cnt = 0;
    for (int b = 0; b < 256; b++)
        if (sb[b] == best) {
            sum += b + 1;
            cnt++;
        }
    *level = (sum / cnt - 1.0) / 255.0;
    return NR_OK;
}
