// cnn.cu -- the learned warm start: a 3D residual CNN (6 conv 3x3x3 layers,
// 32 channels, ReLU) in BF16 on the tensor cores (tcgen05, FP32 accumulate in
// TMEM), with its backward pass and Adam.
//
// Network, in scaled units u = s * x (s = in_scale):
//     a1 = relu(conv1(u)), a_l = relu(conv_l(a_{l-1})) l = 2..5, f = conv6(a5)
//     prediction  x_warm = x + f / s          (residual on the input volume)
// Activations are channels-last BF16 [voxel][32]; a batch of nb patches is
// stacked along z with zero padding at every patch boundary.
//
// Convolution = implicit GEMM.  An output tile is one run of 128 consecutive x
// of a (patch, z, y) row (M = 128), N = output channels, K = 27 taps x input
// channels.  For 32-channel inputs the tile reads, per (dz, dy), one strip of
// 130 input rows (x0-1 .. x0+128, zero outside the volume) into shared memory
// in the K-major core-matrix layout with rows 16 bytes apart; the three dx
// taps are the same strip read from row offsets 0, 1, 2 (descriptor start +
// 16 B).  The strips arrive by TMA (activations are stored in 8-channel planes
// so that a strip's K chunk is one contiguous block); a CTA walks along y and
// adds each staged input row into the accumulators of the three output rows
// that read it, and a producer warp, two MMA warps and groups of epilogue warps
// overlap staging, MMAs and stores (conv32_ys_kernel).  Weights of all 27 taps
// stay in shared memory.  1-channel inputs gather the 27 neighbours into one K = 32 row
// instead.  Weight gradients are GEMMs over voxels on the tensor cores
// (wgrad_tc_kernel), ending in a fixed-order reduction of per-CTA partials.
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <type_traits>

#include "common.cuh"
#include "tc.cuh"
#include "tma.cuh"

namespace nr {
namespace cnn {

constexpr int C = 32;                 // hidden channels
constexpr int TM = 128;               // output voxels per tile
constexpr int SROWS = TM + 2;         // strip rows incl. the x halo
constexpr int KCH = 4;                // 16-byte K chunks per 32-channel row
constexpr int WAIT_LIMIT = 1 << 24;   // polls before a wait gives up

enum { EPI_RELU = 0, EPI_MASK = 1 };

struct Dims {
    int nx, ny, nz, nb;
};

__host__ __device__ inline int64_t nvox(const Dims& d) { return (int64_t)d.nx * d.ny * d.nz * d.nb; }
__host__ __device__ inline int xtiles(const Dims& d) { return (d.nx + TM - 1) / TM; }
__host__ __device__ inline int64_t ntiles(const Dims& d) {
    return (int64_t)d.ny * d.nz * d.nb * xtiles(d);
}

// Packed BF16 B operand of one tap: N rows (output channels) x 32 K in core
// matrices [N/8][4][8 rows][16 B]: SBO = 512 B between row groups, LBO = 128 B.
__host__ __device__ inline int bpk_index(int n, int k) {
    return (n >> 3) * 256 + (k >> 3) * 64 + (n & 7) * 8 + (k & 7);
}

// Activations (and their gradients) are BF16 in planes of 8 channels: per
// row of nx voxels (one (patch, z, y) row), four planes [c / 8][x][c % 8], so
// that one K chunk (8 channels, 16 bytes) of a run of consecutive x is one
// contiguous block -- the unit the convolution's TMA boxes move.
__host__ __device__ inline int64_t act_off(int64_t v, int c, int nx) {
    const int64_t row = v / nx;
    const int x = (int)(v - row * nx);
    return (row * KCH + (c >> 3)) * (int64_t)nx * 8 + (int64_t)x * 8 + (c & 7);
}

// Row (patch b, z, y) of tile t and its first x.
__device__ __forceinline__ void tile_pos(const Dims& d, int64_t t, int& b, int& z, int& y, int& x0) {
    const int xt = xtiles(d);
    int64_t row = t / xt;
    x0 = (int)(t - row * xt) * TM;
    y = (int)(row % d.ny);
    row /= d.ny;
    z = (int)(row % d.nz);
    b = (int)(row / d.nz);
}

// ---- strip staging shared by the convolution and the weight gradient ------
// A strip is 130 input rows (x0 - 1 .. x0 + 128) of one (patch, z, y) row in
// four planes of 8 channels, each plane a K-major core-matrix column block
// (rows 16 bytes apart) for the MMAs.
constexpr int PLANE = 2176;                           // one K-chunk plane: 130 rows x 16 B, 128-B aligned
constexpr int TSTRIP = KCH * PLANE;                   // 8704 bytes per staged strip
constexpr uint32_t STRIP_TX = (uint32_t)KCH * SROWS * 16;  // bytes the four boxes deliver

// One strip (130 rows x 4 K-chunk planes, plane stride `pstride`) of row
// `row` from x0 - 1 by TMA.  The activation tensor is mapped as (2 nx 8-byte
// units, 4 K chunks, R rows), so one plane is one contiguous run; it is loaded
// as two boxes, rows 0-63 (map lo, 128 units) and rows 64-129 (map hi, 132
// units), both 128-byte aligned in shared memory.  Out-of-range units (x < 0,
// x >= nx, row < 0) arrive as zeros; 4 x 2080 bytes complete on `bar`.
__device__ __forceinline__ void load_strip(uint8_t* dst, int pstride, const CUtensorMap* lo,
                                           const CUtensorMap* hi, int x0, int row, uint64_t* bar) {
    const int u0 = 2 * (x0 - 1);
#pragma unroll
    for (int kc = 0; kc < KCH; kc++) {
        tma_load_3d(dst + kc * pstride, lo, u0, kc, row, bar);
        tma_load_3d(dst + kc * pstride + 1024, hi, u0 + 128, kc, row, bar);
    }
}

// A bounded wait that also gives up once the block has aborted.
__device__ __forceinline__ bool wait_live(uint64_t* bar, uint32_t parity, volatile int* abort) {
    for (int round = 0; round < WAIT_LIMIT / 1024; round++) {
        if (tc::mbar_wait(bar, parity, 1024)) return true;
        if (*abort) return false;
    }
    return false;
}

// ---- conv32: bulk copies + tcgen05, walking along y ----------------------------
// 32 -> 32 channels (hidden layers and their input gradients).  A work item is
// a run of up to L output rows y0 .. y0 + L - 1 of one column (patch b, planes
// z and z + 1, x tile of 128).  The item's input rows Y = y0 - 1 .. y0 + L come
// one after another as row-sets (the strips of row Y in planes z - 1 .. z + 2),
// and each row-set is used by one step only: the three dy taps are stacked
// along N, so that one MMA over a strip at row offset dx adds
//     D[x][(dy, o)] += sum_i a[x0 - 1 + x + dx][i] W[dz][dy][dx][o][i]
// to the accumulators of the three output rows that read row Y -- rows Y - 1
// (dy = 2), Y (dy = 1) and Y + 1 (dy = 0), 32 TMEM columns each, side by side:
// 18 MMAs of M = 128, N = 96, K = 16 per input row and output plane.
//
// Two output planes share two of their four strips, and each plane's MMAs are
// issued by a warp of its own: issued from a one-lane branch the MMAs followed
// each other 96 - 140 cycles apart whatever their size (N = 32 and N = 96
// alike: 48 cycles of math at N = 96), with warp-uniform descriptors about 65,
// with one warp per plane about 35 -- the operand fetch (7 KB of shared memory
// per N = 96 MMA, 56 cycles) is then the tensor side's limit and the strips'
// delivery (0.94 ms per clinical layer with the MMAs left out) the next.
// A hidden layer on 1024 x 512 x 60 voxels: 1.05 - 1.12 ms against 2.46 ms for
// the form before (dx stacked along N, shifted back in the epilogue by warp
// shuffles); steps: 2.35 ms with dy stacked, one plane per CTA and tensor-map
// copies; 1.42 with two planes and bulk copies; 1.18 with warp-wide issue.
//
// Accumulators: 8 slots of 32 columns per plane.  Step T (the CTA's steps
// counted through) works on the window of slots s, s + 1, s + 2, s = T % 6.
// For s > 0 the last of the three is fresh (its part of the step's first MMA
// is issued by itself, without accumulation); at s = 0 the window jumps back
// to slots 0 - 2 and all three are fresh, so that the two rows in the middle
// of their three steps have their sum in two slots, added by the epilogue.
// The row that step T starts is "row T" (rows outside the run are computed
// and not stored): complete after step T + 2, in slot T % 6 + 2 (T % 6 < 4),
// in slots 6 and 0 (4) or 7 and 1 (5); step T needs row T - 6 read.
//
// The dx shift is the strip's row offset (descriptor start + 16 B), so the
// accumulator rows are output voxels and the epilogue is one TMEM read, bias
// and ReLU (or mask) and the store.  Strips arrive as plain bulk copies, one
// contiguous run per 8-channel plane (a tensor-map copy of the same run as two
// boxes took about 90 cycles per 1 KB box, 2.0 ms per clinical layer by
// itself); rows outside the patch come from a block of zeros.
//   warp 4 Y_NG            producer (16 lanes): row-sets into a ring of Y_R slots;
//   warps 4 Y_NG + 1, + 2  MMA issuers of the two planes (one elected lane each);
//   groups of four warps   epilogues, group g: plane g & 1 of the rows T with
//                          T % Y_NT == g >> 1.
// One CTA per SM (the ring and all 27 taps' weights).  Every wait is bounded
// and also gives up once another role has aborted; a role that gives up flags
// NR_FLAG_TIMEOUT and aborts the block.  Before TMEM is released the issuer's
// MMAs are drained, and the producer waits for every copy it issued.
constexpr int W_SET = 3 * TSTRIP;                      // three strips (wgrad_walk_kernel)
constexpr int Y_SET = 4 * TSTRIP;                      // 34816 bytes
constexpr int Y_R = 4;                                 // row-set slots
constexpr int Y_NT = 2;                                // rows in the epilogue at once
constexpr int Y_NG = 2 * Y_NT;                         // epilogue groups
constexpr int Y_THREADS = 32 * (4 * Y_NG + 3);
constexpr int Y_ROWS = 8;                              // row barriers (six rows in use at most)
constexpr int Y_WBYTES = 27 * C * C * 2;

struct WalkPlan {
    int L, nchunk;
    int tw;  // outputs per tile along x
    int64_t nitems;
};

struct YCtl {
    uint64_t full[Y_R], empty[Y_R], accf[Y_ROWS], acce[Y_ROWS], drain;
    uint32_t tslot;
    int abort;
    float bias[C];
};

// The zeros that rows outside a patch are copied from.
static __device__ __align__(16) uint4 g_zero_rows[SROWS];

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(tc::smem_u32(dst)),
        "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(tc::smem_u32(bar))
        : "memory");
}

// K chunk kc of the strip of row `row` (-1: zeros) from x0 - 1, 130 rows of 16
// bytes: the part inside [0, nx) from the activations, the rest zeros.
// inner: only the rows inside [0, nx) (the others hold zeros already).
__device__ __forceinline__ void load_chunk(uint8_t* dst, const __nv_bfloat16* in, int nx, int x0,
                                           int64_t row, int kc, bool inner, uint64_t* bar) {
    const int lo = x0 == 0 ? 1 : 0, hi = min(x0 + SROWS - 1, nx) - x0 + 1;  // strip rows [lo, hi)
    if (row < 0 || inner) {
        const void* src = row < 0 ? (const void*)g_zero_rows
                                  : in + ((row * KCH + kc) * nx + x0 - 1 + lo) * 8;
        bulk_load(dst + (inner ? lo * 16 : 0), src, (uint32_t)(inner ? hi - lo : SROWS) * 16, bar);
        return;
    }
    if (lo) bulk_load(dst, g_zero_rows, 16, bar);
    bulk_load(dst + lo * 16, in + ((row * KCH + kc) * nx + x0 - 1 + lo) * 8, (uint32_t)(hi - lo) * 16,
              bar);
    if (hi < SROWS) bulk_load(dst + hi * 16, g_zero_rows, (uint32_t)(SROWS - hi) * 16, bar);
}

// Column (b, z, x0) and rows y0 .. y0 + ly - 1 of item it.
__device__ __forceinline__ void item_pos(const Dims& d, const WalkPlan& w, int64_t it, int& b,
                                         int& z, int& x0, int& y0, int& ly) {
    const int xt = (d.nx + w.tw - 1) / w.tw;
    int64_t col = it / w.nchunk;
    const int ch = (int)(it - col * w.nchunk);
    x0 = (int)(col % xt) * w.tw;
    col /= xt;
    z = (int)(col % d.nz);
    b = (int)(col / d.nz);
    y0 = ch * w.L;
    ly = min(w.L, d.ny - y0);
}

// Epilogue of output row `row` (one (patch, z, y) row), voxel x: bias and ReLU
// or the ReLU mask of the layer below, stored as BF16.  bias: C floats.
template <int EPI>
__device__ __forceinline__ void epilogue_rx(const uint32_t* acc, int64_t row, int x, int nx,
                                            const float* __restrict__ bias,
                                            __nv_bfloat16* __restrict__ out,
                                            const __nv_bfloat16* __restrict__ mask) {
    const int64_t o0 = row * KCH * (int64_t)nx * 8 + (int64_t)x * 8;  // chunk q at o0 + q nx 8
    __align__(16) __nv_bfloat16 o[C];
    if (EPI == EPI_RELU) {
        // the bias in FP32, then BF16 pairs and the ReLU on the pairs (rounding
        // is monotone, so max(round(v), 0) = round(max(v, 0)) up to a zero's sign)
        const __nv_bfloat162 zero2 = __float2bfloat162_rn(0.f);
#pragma unroll
        for (int c = 0; c < C; c += 2)
            ((__nv_bfloat162*)o)[c / 2] =
                __hmax2(__floats2bfloat162_rn(__uint_as_float(acc[c]) + bias[c],
                                              __uint_as_float(acc[c + 1]) + bias[c + 1]),
                        zero2);
    } else {
        __align__(16) __nv_bfloat16 m[C];
#pragma unroll
        for (int q = 0; q < KCH; q++)
            ((uint4*)m)[q] = __ldg((const uint4*)(mask + o0 + (int64_t)q * nx * 8));
#pragma unroll
        for (int c = 0; c < C; c++)
            o[c] = __bfloat162float(m[c]) > 0.f ? __float2bfloat16(__uint_as_float(acc[c]))
                                                : __float2bfloat16(0.f);
    }
#pragma unroll
    for (int q = 0; q < KCH; q++)
        *(uint4*)(out + o0 + (int64_t)q * nx * 8) = ((const uint4*)o)[q];
}

// Column (b, z, x0) and rows y0 .. y0 + ly - 1 of item it: z the first of two planes.
__device__ __forceinline__ void item_pos2(const Dims& d, const WalkPlan& w, int64_t it, int& b,
                                          int& z, int& x0, int& y0, int& ly) {
    item_pos(Dims{d.nx, d.ny, (d.nz + 1) / 2, d.nb}, w, it, b, z, x0, y0, ly);
    z *= 2;
}

template <int EPI>
__global__ void __launch_bounds__(Y_THREADS, 1) conv32_ys_kernel(
    Dims d, WalkPlan wp, const __nv_bfloat16* __restrict__ in,
    const __nv_bfloat16* __restrict__ wpk, const float* __restrict__ bias,
    __nv_bfloat16* __restrict__ out, const __nv_bfloat16* __restrict__ mask, int* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* ring = smem;
    uint8_t* sW = smem + Y_R * Y_SET;
    YCtl* K = (YCtl*)(sW + Y_WBYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int k = tid; k < Y_WBYTES / 16; k += Y_THREADS)
        ((uint4*)sW)[k] = __ldg((const uint4*)wpk + k);
    if (EPI == EPI_RELU && tid < C) K->bias[tid] = bias[tid];
    // a row of one tile: the strips' rows outside it are zeros once and for all,
    // one copy per chunk instead of three (bulk copies of 16 bytes cost as much
    // as a row's): 34 us per launch instead of 40 at 126 x 32 x 16 x 8
    const bool one = d.nx <= TM;
    if (one)
        for (int k = tid; k < Y_R * Y_SET / 16; k += Y_THREADS)
            ((uint4*)ring)[k] = make_uint4(0, 0, 0, 0);
    if (tid == 0) {
        for (int s = 0; s < Y_R; s++) {
            tc::mbar_init(&K->full[s], 1);
            tc::mbar_init(&K->empty[s], 2);
        }
        for (int a = 0; a < Y_ROWS; a++) {
            tc::mbar_init(&K->accf[a], 2);
            tc::mbar_init(&K->acce[a], 8);
        }
        tc::mbar_init(&K->drain, 2);
        K->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(&K->tslot, 512);
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = K->tslot;
    volatile int* abort = &K->abort;
    auto fail = [&]() {
        if (!*abort) atomicOr(status, NR_FLAG_TIMEOUT);
        *abort = 1;
        __threadfence_block();
    };
    if (warp == 4 * Y_NG) {
        // producer: lane = (strip, K chunk)
        const int sp = lane >> 2, kc = lane & 3;
        int T = 0;
        bool stop = false;
        for (int64_t it = blockIdx.x; it < wp.nitems && !stop; it += gridDim.x) {
            int b, z, x0, y0, ly;
            item_pos2(d, wp, it, b, z, x0, y0, ly);
            const int zz = z - 1 + sp;
            for (int j = 0; j < ly + 2; j++, T++) {
                const int s = T % Y_R;
                bool go = !*abort;
                if (go && T >= Y_R) go = wait_live(&K->empty[s], (uint32_t)((T / Y_R - 1) & 1), abort);
                if (!__all_sync(0xffffffffu, go)) {
                    if (lane == 0) fail();
                    stop = true;
                    break;
                }
                if (lane == 0)
                    mbar_arrive_tx(&K->full[s], 4 * KCH * 16 * (uint32_t)(one ? d.nx : SROWS));
                __syncwarp();
                const int Y = y0 - 1 + j;
                const bool ok = zz >= 0 && zz < d.nz && Y >= 0 && Y < d.ny;
                if (lane < 4 * KCH)
                    load_chunk(ring + s * Y_SET + sp * TSTRIP + kc * PLANE, in, d.nx, x0,
                               ok ? ((int64_t)b * d.nz + zz) * d.ny + Y : -1, kc, one, &K->full[s]);
            }
        }
        // no copy may be in flight when the block exits (T row-sets were issued)
        if (lane == 0)
            for (int k = T > Y_R ? T - Y_R : 0; k < T; k++) {
                uint64_t* bar = &K->full[k % Y_R];
                if (!tc::mbar_wait(bar, (uint32_t)((k / Y_R) & 1), WAIT_LIMIT))
                    tc::mbar_wait(bar, (uint32_t)((k / Y_R) & 1), WAIT_LIMIT);
            }
    } else if (warp > 4 * Y_NG) {
        // MMA issuer of plane p: the whole warp runs the loop, one elected lane issues
        const int p = warp - (4 * Y_NG + 1);
        const uint64_t ad0 = tc::sdesc(tc::smem_u32(ring), PLANE, 128);
        const uint64_t bd0 = tc::sdesc(tc::smem_u32(sW), 128, 512);
        const uint32_t ahi = (uint32_t)(ad0 >> 32), bhi = (uint32_t)(bd0 >> 32);
        // K step m = (dz, dx, j): N = 32 n accumulator columns from window row k
        // on (row 0 = output row Y - 1, whose weights come first in the packed
        // block of (dz, dx))
        auto mma = [&](uint32_t alo, uint32_t win, int m, int k, int n, uint32_t acc) {
            const int dz = m / 6, dx = (m / 2) % 3, j = m & 1;
            tc::mma_bf16_warp(
                win + (uint32_t)(k * 32),
                alo + (uint32_t)((dz * TSTRIP + dx * 16 + j * 2 * PLANE) >> 4), ahi,
                (uint32_t)bd0 + (uint32_t)((((dz * 3 + dx) * 3 + k) * C * C * 2 + j * 256) >> 4),
                bhi, tc::idesc_bf16(TM, 32 * n), acc);
        };
        // the second plane of patches one plane deep has nothing to issue (one
        // 128 x 64 plane, forward: 55 us against 61); decided per item it would cost
        // the others 1 %
        auto steps = [&](auto live_c) {
            int T = 0, w = 0;  // step, T % 6
            bool stop = false;
            for (int64_t it = blockIdx.x; it < wp.nitems && !stop; it += gridDim.x) {
                int b, z, x0, y0, ly;
                item_pos2(d, wp, it, b, z, x0, y0, ly);
                for (int i = 0; i < ly + 2; i++, T++) {
                    const int s = T % Y_R;
                    const bool go =
                        (T < 6 || wait_live(&K->acce[(T - 6) % Y_ROWS],
                                            (uint32_t)(((T - 6) / Y_ROWS) & 1), abort)) &&
                        wait_live(&K->full[s], (uint32_t)((T / Y_R) & 1), abort);
                    if (!__all_sync(0xffffffffu, go)) {
                        if (lane == 0) fail();
                        stop = true;
                        break;
                    }
                    tc::fence_after();
                    const uint32_t alo = (uint32_t)ad0 + (uint32_t)((s * Y_SET + p * TSTRIP) >> 4);
                    const uint32_t win = tmem + (uint32_t)(p * 256 + w * 32);
                    if (decltype(live_c)::value) {
                        if (w == 0) {
                            mma(alo, win, 0, 0, 3, 0u);
                        } else {
                            mma(alo, win, 0, 0, 2, 1u);
                            mma(alo, win, 0, 2, 1, 0u);
                        }
#pragma unroll
                        for (int m = 1; m < 18; m++) mma(alo, win, m, 0, 3, 1u);
                    }
                    tc::commit_warp(&K->empty[s]);
                    if (T >= 2) tc::commit_warp(&K->accf[(T - 2) % Y_ROWS]);
                    if (++w == 6) w = 0;
                }
            }
            // the last two rows lie outside the last run: nothing more is added
            if (!stop)
                for (int r = max(T - 2, 0); r < T; r++) tc::commit_warp(&K->accf[r % Y_ROWS]);
        };
        if (p < d.nz)
            steps(std::integral_constant<bool, true>());
        else
            steps(std::integral_constant<bool, false>());
        __syncwarp();
    } else {
        // epilogue: TMEM lanes 32 (warp % 4) .. + 31.  Test hook: the workspace's
        // second status word k + 1 > 0 makes the wait for this CTA's row k report
        // giving up once it has in fact succeeded.
        const int p = (warp >> 2) & 1, tset = warp >> 3, wq = warp & 3;
        const int force_at = status[1] - 1;
        const int64_t qs = (int64_t)d.nx * 8, rs = KCH * qs;  // elements per chunk and per row
        const uint32_t l0 = (uint32_t)(wq * 32);
        int T = 0, w = 0;
        bool stop = false;
        for (int64_t it = blockIdx.x; it < wp.nitems && !stop; it += gridDim.x) {
            int b, z, x0, y0, ly;
            item_pos2(d, wp, it, b, z, x0, y0, ly);
            const int x = x0 + wq * 32 + lane;
            const bool in_vol = x < d.nx && z + p < d.nz;
            const int64_t o00 =
                (((int64_t)b * d.nz + z + p) * d.ny + y0) * rs + (int64_t)x * 8;  // chunk q: + q qs
            for (int i = 0; i < ly + 2; i++, T++) {
                const int wt = w;
                if (++w == 6) w = 0;
                if (T % Y_NT != tset) continue;
                const bool on = in_vol && i < ly;
                const int64_t o0 = o00 + i * rs;
                __align__(16) uint4 m4[EPI == EPI_MASK ? KCH : 1];
                if (EPI == EPI_MASK && on) {
#pragma unroll
                    for (int q = 0; q < KCH; q++) m4[q] = __ldg((const uint4*)(mask + o0 + q * qs));
                }
                bool got = wait_live(&K->accf[T % Y_ROWS], (uint32_t)((T / Y_ROWS) & 1), abort);
                if (T == force_at) got = false;
                if (!__all_sync(0xffffffffu, got)) {
                    if (lane == 0) fail();
                    stop = true;
                    break;
                }
                if (i < ly) {
                    tc::fence_after();
                    uint32_t acc[32];
                    tc::ld32(tmem, l0, (uint32_t)(p * 256 + (wt + 2) * 32), acc);
                    if (wt >= 4) {
                        uint32_t a2[32];
                        tc::ld32(tmem, l0, (uint32_t)(p * 256 + (wt - 4) * 32), a2);
#pragma unroll
                        for (int c = 0; c < C; c++)
                            acc[c] = __float_as_uint(__uint_as_float(acc[c]) + __uint_as_float(a2[c]));
                    }
                    tc::fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&K->acce[T % Y_ROWS]);
                    if (on) {
                        __align__(16) __nv_bfloat162 o[C / 2];
                        if (EPI == EPI_RELU) {
                            // the bias in FP32, then BF16 pairs and the ReLU on the pairs
                            // (rounding is monotone, so max(round(v), 0) =
                            // round(max(v, 0)) up to a zero's sign)
                            const __nv_bfloat162 zero2 = __float2bfloat162_rn(0.f);
#pragma unroll
                            for (int c = 0; c < C; c += 4) {
                                const float4 b4 = *(const float4*)(K->bias + c);
                                o[c / 2] = __hmax2(
                                    __floats2bfloat162_rn(__uint_as_float(acc[c]) + b4.x,
                                                          __uint_as_float(acc[c + 1]) + b4.y),
                                    zero2);
                                o[c / 2 + 1] = __hmax2(
                                    __floats2bfloat162_rn(__uint_as_float(acc[c + 2]) + b4.z,
                                                          __uint_as_float(acc[c + 3]) + b4.w),
                                    zero2);
                            }
                        } else {
                            const __nv_bfloat16* m = (const __nv_bfloat16*)m4;
#pragma unroll
                            for (int c = 0; c < C; c += 2)
                                o[c / 2] = __floats2bfloat162_rn(
                                    __bfloat162float(m[c]) > 0.f ? __uint_as_float(acc[c]) : 0.f,
                                    __bfloat162float(m[c + 1]) > 0.f ? __uint_as_float(acc[c + 1])
                                                                     : 0.f);
                        }
#pragma unroll
                        for (int q = 0; q < KCH; q++)
                            *(uint4*)(out + o0 + q * qs) = ((const uint4*)o)[q];
                    }
                } else {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&K->acce[T % Y_ROWS]);
                }
            }
        }
    }
    // drain: every MMA issued has completed before TMEM is released
    __syncthreads();
    if (warp > 4 * Y_NG) tc::commit_warp(&K->drain);
    if (!tc::mbar_wait(&K->drain, 0, WAIT_LIMIT)) tc::mbar_wait(&K->drain, 0, WAIT_LIMIT);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// ---- the 32 -> 1 layer in two passes -----------------------------------------
// f[v] = b + sum over taps of W[tap] . a[v + off(tap)], regrouped by the tap's
// (dz, dy).  Pass 1 (last_rows_kernel), per input row u of the volume:
//     q[(dz, dy)][u] = sum_dx W[dz][dy][dx] . a[u + (dx - 1, 0, 0)]
// as three MMAs (one per dx: the row's strip at a 16-byte offset) of N = 16
// (rows (dz, dy), 9 used) and K = 32 per 128 voxels -- one strip per tile
// against the convolution's nine, and no walk.  Pass 2 (last_sum_kernel):
//     f[v] = b + sum_{(dz, dy)} q[(dz, dy)][v + (0, dy - 1, dz - 1)]
// (zero outside the patch), nine coalesced loads in a fixed order.  Pass 1:
// a producer lane loads the strips into a ring of LR_STAGE stages, an issuer
// warp runs the MMAs into one of two TMEM accumulators, four epilogue warps
// store the nine planes of q; waits bounded as in conv32_ys_kernel.
constexpr int LR_STAGE = 6;
constexpr int LR_THREADS = 192;

struct LastCtl {
    uint64_t full[LR_STAGE], empty[LR_STAGE], accf[2], acce[2], drain;
    uint32_t tslot;
    int abort;
};

__global__ void __launch_bounds__(LR_THREADS) last_rows_kernel(
    Dims d, const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap amap_hi,
    const __nv_bfloat16* __restrict__ wpk, float* __restrict__ q, int* status) {
    constexpr int WBYTES = 3 * 16 * C * 2;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* ring = smem;
    uint8_t* sW = smem + LR_STAGE * TSTRIP;
    LastCtl* K = (LastCtl*)(sW + WBYTES);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int k = tid; k < WBYTES / 16; k += LR_THREADS)
        ((uint4*)sW)[k] = __ldg((const uint4*)wpk + k);
    if (tid == 0) {
        for (int s = 0; s < LR_STAGE; s++) {
            tc::mbar_init(&K->full[s], 1);
            tc::mbar_init(&K->empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            tc::mbar_init(&K->accf[a], 1);
            tc::mbar_init(&K->acce[a], 4);
        }
        tc::mbar_init(&K->drain, 1);
        K->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(&K->tslot, 64);
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = K->tslot;
    const int64_t nt = ntiles(d);
    const int64_t V = nvox(d);
    volatile int* abort = &K->abort;
    auto fail = [&]() {
        if (!*abort) atomicOr(status, NR_FLAG_TIMEOUT);
        *abort = 1;
        __threadfence_block();
    };
    if (warp == 4) {
        if (lane == 0) {
            // producer
            int64_t lt = 0, issued = 0;
            for (int64_t t = blockIdx.x; t < nt && !*abort; t += gridDim.x, lt++) {
                const int s = (int)(lt % LR_STAGE);
                if (lt >= LR_STAGE &&
                    !wait_live(&K->empty[s], (uint32_t)((lt / LR_STAGE - 1) & 1), abort)) {
                    fail();
                    break;
                }
                int b, z, y, x0;
                tile_pos(d, t, b, z, y, x0);
                mbar_arrive_tx(&K->full[s], STRIP_TX);
                load_strip(ring + s * TSTRIP, PLANE, &amap, &amap_hi, x0, (b * d.nz + z) * d.ny + y,
                           &K->full[s]);
                issued = lt + 1;
            }
            for (int64_t k = issued > LR_STAGE ? issued - LR_STAGE : 0; k < issued; k++) {
                uint64_t* bar = &K->full[k % LR_STAGE];
                if (!tc::mbar_wait(bar, (uint32_t)((k / LR_STAGE) & 1), WAIT_LIMIT))
                    tc::mbar_wait(bar, (uint32_t)((k / LR_STAGE) & 1), WAIT_LIMIT);
            }
        }
    } else if (warp == 5) {
        // MMA issuer (the warp, one elected lane: issued by one lane of a diverged
        // warp an MMA takes 96 to 140 clocks): per dx, the strip at offset dx
        // rows against its 16 x 32 block
        constexpr uint32_t idesc = tc::idesc_bf16(TM, 16);
        const uint64_t ad0 = tc::sdesc(tc::smem_u32(ring), PLANE, 128);
        const uint64_t bd0 = tc::sdesc(tc::smem_u32(sW), 128, 512);
        int64_t lt = 0;
        for (int64_t t = blockIdx.x; t < nt; t += gridDim.x, lt++) {
            const int a = (int)(lt & 1), s = (int)(lt % LR_STAGE);
            const bool go =
                (lt < 2 || wait_live(&K->acce[a], (uint32_t)(((lt >> 1) - 1) & 1), abort)) &&
                wait_live(&K->full[s], (uint32_t)((lt / LR_STAGE) & 1), abort);
            if (!__all_sync(0xffffffffu, go)) {
                if (lane == 0) fail();
                break;
            }
            tc::fence_after();
            const uint32_t alo = (uint32_t)ad0 + (uint32_t)((s * TSTRIP) >> 4);
#pragma unroll
            for (int dx = 0; dx < 3; dx++)
#pragma unroll
                for (int j = 0; j < 2; j++)
                    tc::mma_bf16_warp(tmem + (uint32_t)(a * 32),
                                      alo + (uint32_t)((dx * 16 + j * 2 * PLANE) >> 4),
                                      (uint32_t)(ad0 >> 32),
                                      (uint32_t)bd0 + (uint32_t)((dx * 16 * C * 2 + j * 256) >> 4),
                                      (uint32_t)(bd0 >> 32), idesc, (dx | j) ? 1u : 0u);
            tc::commit_warp(&K->empty[s]);
            tc::commit_warp(&K->accf[a]);
        }
        __syncwarp();
    } else {
        // epilogue warps 0-3: row 32 warp + lane of each tile.  Test hook: the
        // workspace's second status word k + 1 > 0 makes the wait for this
        // CTA's tile k report giving up once it has in fact succeeded.
        const int force_at = status[1] - 1;
        int64_t lt = 0;
        for (int64_t t = blockIdx.x; t < nt; t += gridDim.x, lt++) {
            const int a = (int)(lt & 1);
            bool got = wait_live(&K->accf[a], (uint32_t)((lt >> 1) & 1), abort);
            if (lt == force_at) got = false;
            if (!got) {
                if (lane == 0) fail();
                break;
            }
            tc::fence_after();
            uint32_t acc[32];
            tc::ld32(tmem, (uint32_t)(warp * 32), (uint32_t)(a * 32), acc);
            tc::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&K->acce[a]);
            int b, z, y, x0;
            tile_pos(d, t, b, z, y, x0);
            const int x = x0 + warp * 32 + lane;
            if (x < d.nx) {
                const int64_t v = (((int64_t)b * d.nz + z) * d.ny + y) * d.nx + x;
#pragma unroll
                for (int n = 0; n < 9; n++) q[n * V + v] = __uint_as_float(acc[n]);
            }
        }
    }
    __syncthreads();
    if (warp == 5) tc::commit_warp(&K->drain);
    if (!tc::mbar_wait(&K->drain, 0, WAIT_LIMIT)) tc::mbar_wait(&K->drain, 0, WAIT_LIMIT);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 64);
}

// Pass 2: grid (row of the stacked volume, block of 256 x VEC); VEC = 4 when
// rows are 16-byte aligned (nx % 4 == 0): four x per thread in float4 loads.
// RESID: the network's output max(0, x_in + f / s) instead of f.  Bound by DRAM
// (36 bytes of q, 8 of x and the output per voxel): 213 us at 1024 x 512 x 60,
// where the sum alone took 195 us and a residual pass over f another 55 us.
template <int VEC, bool RESID>
__global__ void __launch_bounds__(256) last_sum_kernel(Dims d, const float* __restrict__ q,
                                                       const float* __restrict__ bias,
                                                       const float* __restrict__ x_in,
                                                       float inv_s, float* __restrict__ f) {
    auto out = [&](float v, float xi) { return RESID ? fmaxf(xi + v * inv_s, 0.f) : v; };
    const int64_t row = blockIdx.x;
    const int x = (blockIdx.y * 256 + threadIdx.x) * VEC;
    if (x >= d.nx) return;
    const int y = (int)(row % d.ny), z = (int)((row / d.ny) % d.nz);
    const int64_t b = row / ((int64_t)d.ny * d.nz);
    const int64_t V = nvox(d);
    if (VEC == 4) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int n = 0; n < 9; n++) {
            const int zz = z + n / 3 - 1, yy = y + n % 3 - 1;
            if (zz >= 0 && zz < d.nz && yy >= 0 && yy < d.ny) {
                const float4 v =
                    __ldg((const float4*)(q + n * V + ((b * d.nz + zz) * d.ny + yy) * d.nx + x));
                sum.x += v.x;
                sum.y += v.y;
                sum.z += v.z;
                sum.w += v.w;
            }
        }
        const float b0 = bias[0];
        const float4 xi = RESID ? __ldg((const float4*)(x_in + row * d.nx + x))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
        *(float4*)(f + row * d.nx + x) =
            make_float4(out(sum.x + b0, xi.x), out(sum.y + b0, xi.y), out(sum.z + b0, xi.z),
                        out(sum.w + b0, xi.w));
    } else {
        float sum = 0.f;
#pragma unroll
        for (int n = 0; n < 9; n++) {
            const int zz = z + n / 3 - 1, yy = y + n % 3 - 1;
            if (zz >= 0 && zz < d.nz && yy >= 0 && yy < d.ny)
                sum += __ldg(q + n * V + ((b * d.nz + zz) * d.ny + yy) * d.nx + x);
        }
        f[row * d.nx + x] = out(sum + bias[0], RESID ? __ldg(x_in + row * d.nx + x) : 0.f);
    }
}

// 1-channel input conv (the first layer, and the back projection of the last
// layer's gradient): each output row gathers its 27 neighbours (zero outside
// its patch) x scale into one K = 32 row.  Weights: one packed 32 x 32 tile.
template <int EPI>
__global__ void __launch_bounds__(128) conv1_kernel(Dims d, WalkPlan wp, const float* __restrict__ in,
                                                    float scale,
                                                    const __nv_bfloat16* __restrict__ wpk,
                                                    const float* __restrict__ bias,
                                                    __nv_bfloat16* __restrict__ out,
                                                    const __nv_bfloat16* __restrict__ mask,
                                                    int* status) {
    __shared__ __align__(1024) uint8_t sW[C * C * 2];
    __shared__ __align__(1024) uint8_t sA[KCH * TM * 16];
    __shared__ __align__(8) uint64_t bars[1];
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5;
    for (int k = tid; k < C * C * 2 / 16; k += 128) ((uint4*)sW)[k] = __ldg((const uint4*)wpk + k);
    if (tid == 0) tc::mbar_init(&bars[0], 1);
    if (warp == 0) tc::tmem_alloc(&tslot, 32);
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tslot;
    constexpr uint32_t idesc = tc::idesc_bf16(TM, C);
    int ntile = 0;
    int ncommit = 0;
    bool ok = true;
    const int force_at = status[1] - 1;  // test hook, as in conv32_ys_kernel
    // Tiles in runs of rows along y (the items of conv32_ys_kernel), so
    // that consecutive tiles of a CTA share six of their nine input rows.
    struct Pos {
        int64_t it;
        int i, b, z, y0, ly, x0;
    };
    auto first = [&](int64_t it, Pos& p) {
        p.it = it;
        p.i = 0;
        if (it < wp.nitems) item_pos(d, wp, it, p.b, p.z, p.x0, p.y0, p.ly);
    };
    auto advance = [&](Pos& p) {
        if (++p.i >= p.ly) first(p.it + gridDim.x, p);
    };
    // the 27 neighbours of this thread's voxel in a tile (zero outside the
    // patch), loaded one tile ahead so that their latency overlaps the
    // previous tile's MMAs and epilogue
    // The nine rows' bases and validity and the three x offsets' validity
    // are formed once per tile; each tap is then one predicated load.
    float nb[27];
    auto gather = [&](const Pos& p) {
        const int b = p.b, z = p.z, y = p.y0 + p.i;
        const int x = p.x0 + tid;
        const bool xv[3] = {x >= 1 && x - 1 < d.nx, x < d.nx, x + 1 < d.nx};
#pragma unroll
        for (int q = 0; q < 9; q++) {
            const int zz = z + q / 3 - 1, yy = y + q % 3 - 1;
            const bool rv = zz >= 0 && zz < d.nz && yy >= 0 && yy < d.ny;
            const float* row = in + (((int64_t)b * d.nz + (rv ? zz : z)) * d.ny + (rv ? yy : y)) * d.nx;
#pragma unroll
            for (int dx = 0; dx < 3; dx++)
                nb[3 * q + dx] = (rv && xv[dx]) ? __ldg(row + x + dx - 1) : 0.f;
        }
    };
    Pos cur, nxt;
    first(blockIdx.x, cur);
    if (cur.it < wp.nitems) gather(cur);
    for (; cur.it < wp.nitems; cur = nxt) {
        nxt = cur;
        advance(nxt);
        const int b = cur.b, z = cur.z, y = cur.y0 + cur.i, x0 = cur.x0;
        const int x = x0 + tid;
        __align__(16) __nv_bfloat162 row[16];
#pragma unroll
        for (int k = 0; k < 16; k++)
            row[k] = __floats2bfloat162_rn(2 * k < 27 ? nb[2 * k] * scale : 0.f,
                                           2 * k + 1 < 27 ? nb[2 * k + 1] * scale : 0.f);
        // previous tile's MMAs have completed (waited below), so sA is free
#pragma unroll
        for (int kc = 0; kc < KCH; kc++) *(uint4*)(sA + kc * TM * 16 + tid * 16) = ((uint4*)row)[kc];
        tc::fence_async_smem();
        ok = __syncthreads_and(ok) != 0;  // uniform: every thread counts the commits alike
        if (tid == 0 && ok) {
            tc::fence_after();
            const uint32_t sa = tc::smem_u32(sA), sw = tc::smem_u32(sW);
#pragma unroll
            for (int j = 0; j < 2; j++)
                tc::mma_bf16(tmem, tc::sdesc(sa + j * 2 * TM * 16, TM * 16, 128),
                             tc::sdesc(sw + j * 256, 128, 512), idesc, j != 0);
            tc::commit(&bars[0]);
        }
        if (nxt.it < wp.nitems) gather(nxt);
        if (ok) {
            ok = tc::mbar_wait(&bars[0], (uint32_t)(ncommit & 1), WAIT_LIMIT) && ntile != force_at;
            ncommit++;
        }
        ntile++;
        tc::fence_after();
        if (!__syncthreads_and(ok)) {
            if (tid == 0) atomicOr(status, NR_FLAG_TIMEOUT);
            break;
        }
        uint32_t acc[32];
        tc::ld32(tmem, (uint32_t)(warp * 32), 0, acc);
        if (x < d.nx) epilogue_rx<EPI>(acc, ((int64_t)b * d.nz + z) * d.ny + y, x, d.nx, bias, out, mask);
        tc::fence_before();
        __syncthreads();
    }
    if (tid == 0) tc::commit(&bars[0]);  // drain: every MMA issued completes before TMEM goes
    if (!tc::mbar_wait(&bars[0], (uint32_t)(ncommit & 1), WAIT_LIMIT))
        tc::mbar_wait(&bars[0], (uint32_t)(ncommit & 1), WAIT_LIMIT);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 32);
}

// ---------------------------------------------------------------------------
// Weight gradients on the tensor cores.  dW[tap][o][i] = sum_v g[v][o]
// in[v + off(tap)][i] over the stacked patches (zero outside each patch) and
// db[o] = sum_v g[v][o]: per layer one GEMM with the voxels as K, in K blocks
// of one tile (128 consecutive x of a (patch, z, y) row).
//
// The activations' plane layout makes staged strips operands as they land: a
// strip plane is [x][8 channels], i.e. MN-major core matrices (8 channels x 8
// consecutive x in 16-byte rows), and strips staged one after another sit at
// one uniform plane stride, so several strips form one operand whose rows are
// (strip, channel), and a shift along x is a 16-byte start offset.
// This kernel serves the 1-channel layers (the 32 -> 32 ones walk along y in
// wgrad_walk_kernel, below):
//   WG_LAST  (32 -> 1)   A = four input strips (rows (strip, i)) at the tap's
//                        x shift: blocks {0-3}, {4-7}, {5-8} (of the last only
//                        strip 8's rows are kept) x dx = 9 MMA blocks; B = the
//                        FP32 gradient of the one output split as hi + lo BF16
//                        (rows 0, 1 of an N = 16 K-major operand): dW = column
//                        0 + column 1.
//   WG_FIRST (1 -> 32)   A = the FP32 input u = s x at the 27 shifts split as
//                        hi (rows 0-26) + lo (rows 32-58) of a K-major M = 128
//                        operand; B = the gradient strip.
// The split keeps the FP32 operand to 2^-17 relative: hi = bf16(u), lo =
// bf16(u - hi), and the products of BF16 values are exact in the FP32
// accumulator.  The bias gradient is summed on the CUDA cores (FP32 per
// thread, then in a fixed order).
//
// Roles (6 warps): warp 0 lane 0 loads each K block's strips by TMA into one
// of two stages (a strip outside the patch in z or y is loaded from row -1,
// i.e. zero-filled); warp 1 (one elected lane) issues the MMAs and frees the stage by
// tcgen05.commit; warps 2-5 (x - x0 in 32 h .. 32 h + 31 for warp 2 + h) build
// the split operand from global data fetched one block ahead and sum the
// bias.  Every wait is bounded and gives up once another role has aborted; a
// role that gives up flags NR_FLAG_TIMEOUT and aborts the block.  Before TMEM
// is released the issuer's MMAs are drained and the producer waits for every
// copy it issued.  Each CTA writes one partial per weight (row blockIdx.x of
// partial[CTA][28 x weights per tap]); wgrad_reduce_kernel adds the rows in
// order.
enum { WG_LAST = 1, WG_FIRST = 2 };
constexpr int WG_MAXCTA = 256;  // partial slots per weight
constexpr int WG_GROUP = 2048;  // K-major built operand: bytes per 8-row group (16 K chunks)
constexpr int WG_PLANE = 2176;  // staged plane: 130 rows x 16 B, 128-B aligned
constexpr int WG_STRIP = KCH * WG_PLANE;
constexpr int WG_THREADS = 192;
constexpr int WG_WIN = 34;      // WG_FIRST: input window per builder warp and row

struct WgCtl {
    uint64_t tfull[2], bfull[2], empty[2], drain;
    uint32_t tslot;
    int abort;
    float bsum[4][C];
};

template <int MODE>
struct WgCfg {
    // one stage: [input strips 0..8 | gradient strip | built operand]
    static constexpr int NSTRIP = MODE == WG_FIRST ? 0 : 9;
    static constexpr int NCOPY = MODE == WG_FIRST ? 1 : 0;
    static constexpr int NLOAD = NCOPY;
    static constexpr int OFF_G = NSTRIP * WG_STRIP;
    static constexpr int OFF_X = OFF_G + NCOPY * WG_STRIP;
    static constexpr int XBYTES =
        MODE == WG_LAST ? 2 * WG_GROUP : (MODE == WG_FIRST ? 16 * WG_GROUP : 0);
    static constexpr int STAGE = OFF_X + XBYTES;
    static constexpr uint32_t TX = (uint32_t)(NSTRIP + NLOAD) * KCH * SROWS * 16;
    static constexpr int N = MODE == WG_LAST ? 16 : C;
    static constexpr uint32_t NCOL = MODE == WG_FIRST ? 32 : 512;
    // WG_FIRST: each builder warp's window of the input, 9 rows x WG_WIN x
    static constexpr int XS = MODE == WG_FIRST ? 4 * 9 * WG_WIN * 4 : 0;
    static constexpr int SMEM = 2 * STAGE + XS + (int)sizeof(WgCtl);
    // bit 15 / 16: A / B MN-major
    static constexpr uint32_t IDESC = tc::idesc_bf16(TM, N) |
                                      (MODE != WG_FIRST ? 1u << 15 : 0u) |
                                      (MODE != WG_LAST ? 1u << 16 : 0u);
    // arrivals that free a stage: the MMA commit, and the bias warps after
    // reading the gradient strip
    static constexpr int EMPTY_COUNT = MODE == WG_LAST ? 1 : 5;
};

// Stores the BF16 pair hi + lo of u at rows (mh, ml), K index k of a K-major
// built operand (8-row groups WG_GROUP apart, K chunks 128 B apart).
__device__ __forceinline__ void wg_split_store(uint8_t* op, int mh, int ml, int k, float u) {
    const __nv_bfloat16 hi = __float2bfloat16_rn(u);
    const __nv_bfloat16 lo = __float2bfloat16_rn(u - __bfloat162float(hi));
    const int kk = (k >> 3) * 128 + (k & 7) * 2;
    *(__nv_bfloat16*)(op + (mh >> 3) * WG_GROUP + kk + (mh & 7) * 16) = hi;
    *(__nv_bfloat16*)(op + (ml >> 3) * WG_GROUP + kk + (ml & 7) * 16) = lo;
}

// The global data one builder lane needs for the K block of tile t: WG_LAST
// the gradient at x = x0 + 32 h + lane; WG_FIRST its share of the warp's
// window u = s x at x0 - 1 + 32 h + j (j < WG_WIN) of the nine rows.
template <int MODE>
__device__ __forceinline__ void wg_fetch(const Dims& d, int64_t t, int h, int lane,
                                         const float* __restrict__ gvec,
                                         const float* __restrict__ xin, float s, float* r) {
    int b, z, y, x0;
    tile_pos(d, t, b, z, y, x0);
    if (MODE == WG_LAST) {
        const int x = x0 + 32 * h + lane;
        r[0] = x < d.nx ? __ldg(gvec + (((int64_t)b * d.nz + z) * d.ny + y) * d.nx + x) : 0.f;
    } else if (MODE == WG_FIRST) {
#pragma unroll
        for (int k = 0; k < (9 * WG_WIN + 31) / 32; k++) {
            const int e = lane + 32 * k;
            const int q = e / WG_WIN, j = e - q * WG_WIN;
            const int zz = z + q / 3 - 1, yy = y + q % 3 - 1;
            const int xx = x0 - 1 + 32 * h + j;
            r[k] = 0.f;
            if (e < 9 * WG_WIN && zz >= 0 && zz < d.nz && yy >= 0 && yy < d.ny && xx >= 0 &&
                xx < d.nx)
                r[k] = __ldg(xin + (((int64_t)b * d.nz + zz) * d.ny + yy) * d.nx + xx) * s;
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(WG_THREADS, 1) wgrad_tc_kernel(
    Dims d, const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap amap_hi,
    const __grid_constant__ CUtensorMap gmap, const __grid_constant__ CUtensorMap gmap_hi,
    const float* __restrict__ gvec, const float* __restrict__ xin, float s,
    float* __restrict__ partial, int* status) {
    using Cfg = WgCfg<MODE>;
    extern __shared__ __align__(1024) uint8_t smem[];
    WgCtl* K = (WgCtl*)(smem + 2 * Cfg::STAGE + Cfg::XS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // regions the copies and the builders never write stay zero
    constexpr int ZOFF = Cfg::OFF_X;
    constexpr int ZBYTES = Cfg::XBYTES;
    for (int k = tid; k < ZBYTES / 16; k += WG_THREADS) {
        ((uint4*)(smem + ZOFF))[k] = make_uint4(0, 0, 0, 0);
        ((uint4*)(smem + Cfg::STAGE + ZOFF))[k] = make_uint4(0, 0, 0, 0);
    }
    tc::fence_async_smem();
    if (tid == 0) {
        for (int k = 0; k < 2; k++) {
            tc::mbar_init(&K->tfull[k], 1);
            tc::mbar_init(&K->bfull[k], 4);
            tc::mbar_init(&K->empty[k], Cfg::EMPTY_COUNT);
        }
        tc::mbar_init(&K->drain, 1);
        K->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(&K->tslot, Cfg::NCOL);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = K->tslot;
    const int64_t nt = ntiles(d);
    volatile int* abort = &K->abort;
    auto fail = [&]() {
        if (!*abort) atomicOr(status, NR_FLAG_TIMEOUT);
        *abort = 1;
        __threadfence_block();
    };
    if (warp == 0) {
        if (lane == 0) {
            // producer
            int64_t kb = 0, issued = 0;
            for (int64_t t = blockIdx.x; t < nt && !*abort; t += gridDim.x, kb++) {
                const int sg = (int)(kb & 1);
                if (kb >= 2 &&
                    !wait_live(&K->empty[sg], (uint32_t)(((kb >> 1) - 1) & 1), abort)) {
                    fail();
                    break;
                }
                int b, z, y, x0;
                tile_pos(d, t, b, z, y, x0);
                uint8_t* st = smem + sg * Cfg::STAGE;
                mbar_arrive_tx(&K->tfull[sg], Cfg::TX);
                const int grow = (b * d.nz + z) * d.ny + y;
                // gradient copy c starts at x0 + 1 - c (HID) / x0 - 1 (FIRST)
                for (int c = 0; c < Cfg::NLOAD; c++)
                    load_strip(st + Cfg::OFF_G + c * WG_STRIP, WG_PLANE, &gmap, &gmap_hi,
                               x0, grow, &K->tfull[sg]);
                for (int q = 0; q < Cfg::NSTRIP; q++) {
                    const int zz = z + q / 3 - 1, yy = y + q % 3 - 1;
                    const int row = (zz >= 0 && zz < d.nz && yy >= 0 && yy < d.ny)
                                        ? (b * d.nz + zz) * d.ny + yy
                                        : -1;
                    load_strip(st + q * WG_STRIP, WG_PLANE, &amap, &amap_hi, x0, row,
                               &K->tfull[sg]);
                }
                issued = kb + 1;
            }
            // no copy may be in flight when the block exits
            for (int64_t k = issued > 2 ? issued - 2 : 0; k < issued; k++) {
                uint64_t* bar = &K->tfull[k & 1];
                if (!tc::mbar_wait(bar, (uint32_t)((k >> 1) & 1), WAIT_LIMIT))
                    tc::mbar_wait(bar, (uint32_t)((k >> 1) & 1), WAIT_LIMIT);
            }
        }
    } else if (warp == 1) {
        // MMA issuer (the warp, one elected lane).  Test hook: the workspace's
        // second status word k + 1 > 0 makes the wait for this CTA's K block k
        // report giving up once it has in fact succeeded.
        const int force_at = status[1] - 1;
        auto mma = [&](uint32_t dacc, uint64_t ad, uint64_t bd, uint32_t acc) {
            tc::mma_bf16_warp(dacc, (uint32_t)ad, (uint32_t)(ad >> 32), (uint32_t)bd,
                              (uint32_t)(bd >> 32), Cfg::IDESC, acc);
        };
        int64_t kb = 0;
        for (int64_t t = blockIdx.x; t < nt; t += gridDim.x, kb++) {
            const int sg = (int)(kb & 1);
            const uint32_t par = (uint32_t)((kb >> 1) & 1);
            bool got = !*abort && wait_live(&K->tfull[sg], par, abort);
            if (got) got = wait_live(&K->bfull[sg], par, abort);
            if (kb == force_at) got = false;
            if (!__all_sync(0xffffffffu, got)) {
                if (lane == 0) fail();
                break;
            }
            tc::fence_after();
            const uint32_t sb = tc::smem_u32(smem + sg * Cfg::STAGE);
            if (MODE == WG_FIRST) {
#pragma unroll
                for (int k = 0; k < TM / 16; k++)
                    mma(tmem, tc::sdesc(sb + Cfg::OFF_X + k * 256, 128, WG_GROUP),
                        tc::sdesc(sb + Cfg::OFF_G + 16 + k * 256, 128, WG_PLANE),
                        (kb > 0 || k > 0) ? 1u : 0u);
            } else {
                for (int gi = 0; gi < 3; gi++) {
                    const int g0 = gi == 0 ? 0 : (gi == 1 ? 4 : 5);
                    // the three dx accumulators in turn
#pragma unroll
                    for (int k = 0; k < TM / 16; k++)
#pragma unroll
                        for (int dx = 0; dx < 3; dx++)
                            mma(tmem + (uint32_t)((gi * 3 + dx) * 32),
                                tc::sdesc(sb + g0 * WG_STRIP + dx * 16 + k * 256, 128, WG_PLANE),
                                tc::sdesc(sb + Cfg::OFF_X + k * 256, 128, WG_GROUP),
                                (kb > 0 || k > 0) ? 1u : 0u);
                }
            }
            tc::commit_warp(&K->empty[sg]);
        }
        __syncwarp();
    } else {
        // warps 2-5: the built operand and the bias sum
        const int h = warp - 2;
        float* xs = (float*)(smem + 2 * Cfg::STAGE) + h * 9 * WG_WIN;  // WG_FIRST
        constexpr int NR = MODE == WG_FIRST ? (9 * WG_WIN + 31) / 32 : 1;
        float r[NR];  // the next block's global data, in flight
        float bacc = 0.f;
        int64_t t = blockIdx.x;
        if (t < nt) wg_fetch<MODE>(d, t, h, lane, gvec, xin, s, r);
        for (int64_t kb = 0; t < nt && !*abort; t += gridDim.x, kb++) {
            const int sg = (int)(kb & 1);
            uint8_t* st = smem + sg * Cfg::STAGE;
            {
                if (!__all_sync(0xffffffffu,
                                kb < 2 || wait_live(&K->empty[sg],
                                                    (uint32_t)(((kb >> 1) - 1) & 1), abort))) {
                    if (lane == 0) fail();
                    break;
                }
                float cur[NR];
#pragma unroll
                for (int k = 0; k < NR; k++) cur[k] = r[k];
                if (t + gridDim.x < nt) wg_fetch<MODE>(d, t + gridDim.x, h, lane, gvec, xin, s, r);
                const int k = 32 * h + lane;
                if (MODE == WG_LAST) {
                    bacc += cur[0];
                    wg_split_store(st + Cfg::OFF_X, 0, 1, k, cur[0]);
                } else {
                    __syncwarp();  // the previous block's reads of the window are done
#pragma unroll
                    for (int e = 0; e < NR; e++)
                        if (lane + 32 * e < 9 * WG_WIN) xs[lane + 32 * e] = cur[e];
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 9; q++)
#pragma unroll
                        for (int dx = 0; dx < 3; dx++)
                            wg_split_store(st + Cfg::OFF_X, 3 * q + dx, 32 + 3 * q + dx, k,
                                           xs[q * WG_WIN + lane + dx]);
                }
                tc::fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&K->bfull[sg]);
            }
            if (MODE != WG_LAST) {
                if (!__all_sync(0xffffffffu,
                                wait_live(&K->tfull[sg], (uint32_t)((kb >> 1) & 1), abort))) {
                    if (lane == 0) fail();
                    break;
                }
                // channel o = lane of x = 32 h .. 32 h + 31, in the gradient
                // copy staged from x0 - 1 (row x + 1)
                const uint8_t* gp = st + Cfg::OFF_G +
                                    (lane >> 3) * WG_PLANE + (lane & 7) * 2;
#pragma unroll 8
                for (int x = 32 * h; x < 32 * h + 32; x++)
                    bacc += __bfloat162float(*(const __nv_bfloat16*)(gp + (x + 1) * 16));
                __syncwarp();
                if (lane == 0) mbar_arrive(&K->empty[sg]);
            }
        }
        K->bsum[h][lane] = bacc;
    }
    // drain: every MMA issued has completed before TMEM is read or released
    __syncthreads();
    if (warp == 1) tc::commit_warp(&K->drain);
    if (!tc::mbar_wait(&K->drain, 0, WAIT_LIMIT)) tc::mbar_wait(&K->drain, 0, WAIT_LIMIT);
    tc::fence_after();
    const bool ok = *abort == 0;
    float* prow = partial + (int64_t)blockIdx.x * 28 * C;
    auto bias_of = [&](int o) {
        return ((K->bsum[0][o] + K->bsum[1][o]) + K->bsum[2][o]) + K->bsum[3][o];
    };
    if (MODE == WG_FIRST) {
        // rows 32 + tap (lo) of warp 1 meet rows tap (hi) of warp 0
        float* lo = (float*)smem;  // the stages are idle now
        uint32_t acc[32];
        if (ok && warp == 1) {
            tc::ld32(tmem, 32, 0, acc);
            for (int o = 0; o < C; o++) lo[lane * C + o] = __uint_as_float(acc[o]);
        }
        __syncthreads();
        if (ok && warp == 0) {
            tc::ld32(tmem, 0, 0, acc);
            if (lane < 27)
                for (int o = 0; o < C; o++)
                    prow[lane * C + o] = __uint_as_float(acc[o]) + lo[lane * C + o];
        }
        if (ok && warp == 2) prow[27 * C + lane] = bias_of(lane);
    } else if (ok && warp < 4) {
        // TMEM lane 32 w + i of block (gi, dx): strip g0 + w
        for (int gi = 0; gi < 3; gi++) {
            if (gi == 2 && warp < 3) continue;  // strips 5-7 again
            const int q = (gi == 0 ? 0 : (gi == 1 ? 4 : 5)) + warp;
            for (int dx = 0; dx < 3; dx++) {
                uint32_t acc[32];
                tc::ld32(tmem, (uint32_t)(warp * 32), (uint32_t)((gi * 3 + dx) * 32), acc);
                prow[(3 * q + dx) * C + lane] = __uint_as_float(acc[0]) + __uint_as_float(acc[1]);
            }
        }
        if (tid == 0) {
            float sacc = 0.f;
            for (int k = 0; k < 4 * C; k++) sacc += K->bsum[k >> 5][k & 31];
            prow[27 * C] = sacc;
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, Cfg::NCOL);
}

// ---- 32 -> 32 weight gradient walking along y --------------------------------
// dW of a 32 -> 32 layer: the tap's x shift moves onto the gradient (per row of
// the volume, sum_x g[x] a[x + dx - 1] = sum_x' g[x' + 1 - dx] a[x'], both zero
// outside the row), so that with K = x' the input strips are B unshifted (rows
// (strip, i)) and A (M = 128) is the gradient strip in three copies, copy c
// staged from x0 + 1 - c (rows (c, o); copy 3 is zeros): D[(dx, o)][(strip, i)].
// The staging is shared between neighbouring rows, as in conv32_ys_kernel: a CTA takes runs of L rows y of
// one (patch, z, x tile) column; the input strips come as row-sets (the strips
// of one input row in planes z - 1, z, z + 1) through a ring of GW_R slots, each
// row-set loaded once for the three K blocks (output rows) that read it.  Per
// K step three MMAs of N = 96, one per row-set (its three strips; the ring's
// slots are not contiguous), into TMEM columns 96 dy + 32 dz + i.  The
// gradient strip is loaded once per K block (from x0 - 1) and the builder
// warps derive the copies staged from x0 + 1 and x0 (rows shifted by 2 and 1)
// in shared memory; copy 3 stays zero.  About 5.5 strips are staged per K
// block instead of 12.  Roles as in wgrad_tc_kernel; every wait is bounded.
constexpr int GW_R = 5;
constexpr int GW_G = 4 * WG_STRIP;  // one gradient stage: copies 0..3
constexpr int GW_THREADS = 192;

struct GwCtl {
    uint64_t rfull[GW_R], rempty[GW_R], gfull[2], gbuilt[2], gempty[2], drain;
    uint32_t tslot;
    int abort;
    float bsum[4][C];
};

__global__ void __launch_bounds__(GW_THREADS, 1) wgrad_walk_kernel(
    Dims d, WalkPlan wp, const __grid_constant__ CUtensorMap amap,
    const __grid_constant__ CUtensorMap amap_hi, const __grid_constant__ CUtensorMap gmap,
    const __grid_constant__ CUtensorMap gmap_hi, float* __restrict__ partial, int* status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* ring = smem;
    uint8_t* gst = smem + GW_R * W_SET;
    GwCtl* K = (GwCtl*)(gst + 2 * GW_G);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int k = tid; k < WG_STRIP / 16; k += GW_THREADS) {  // copy 3 of both stages: zeros
        ((uint4*)(gst + 3 * WG_STRIP))[k] = make_uint4(0, 0, 0, 0);
        ((uint4*)(gst + GW_G + 3 * WG_STRIP))[k] = make_uint4(0, 0, 0, 0);
    }
    tc::fence_async_smem();
    if (tid == 0) {
        for (int s = 0; s < GW_R; s++) {
            tc::mbar_init(&K->rfull[s], 1);
            tc::mbar_init(&K->rempty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            tc::mbar_init(&K->gfull[s], 1);
            tc::mbar_init(&K->gbuilt[s], 4);
            tc::mbar_init(&K->gempty[s], 1);
        }
        tc::mbar_init(&K->drain, 1);
        K->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tc::tmem_alloc(&K->tslot, 512);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = K->tslot;
    volatile int* abort = &K->abort;
    auto fail = [&]() {
        if (!*abort) atomicOr(status, NR_FLAG_TIMEOUT);
        *abort = 1;
        __threadfence_block();
    };
    auto strip_ok = [&](int zz, int yy) { return zz >= 0 && zz < d.nz && yy >= 0 && yy < d.ny; };
    if (warp == 0) {
        if (lane == 0) {
            // producer: per item row-sets 0 and 1, then per K block i row-set
            // i + 2 and the gradient strip
            int64_t G = 0, kb = 0, rissued = 0, kissued = 0;
            bool stop = false;
            auto load_set = [&](int b, int z, int x0, int Y) {
                const int s = (int)(G % GW_R);
                if (G >= GW_R &&
                    !wait_live(&K->rempty[s], (uint32_t)((G / GW_R - 1) & 1), abort))
                    return false;
                mbar_arrive_tx(&K->rfull[s], 3 * STRIP_TX);
                for (int dz = 0; dz < 3; dz++)
                    load_strip(ring + s * W_SET + dz * TSTRIP, PLANE, &amap, &amap_hi, x0,
                               strip_ok(z + dz - 1, Y) ? (b * d.nz + z + dz - 1) * d.ny + Y : -1,
                               &K->rfull[s]);
                rissued = ++G;
                return true;
            };
            for (int64_t it = blockIdx.x; it < wp.nitems && !stop && !*abort; it += gridDim.x) {
                int b, z, x0, y0, ly;
                item_pos(d, wp, it, b, z, x0, y0, ly);
                if (!load_set(b, z, x0, y0 - 1) || !load_set(b, z, x0, y0)) {
                    fail();
                    break;
                }
                for (int i = 0; i < ly; i++, kb++) {
                    if (!load_set(b, z, x0, y0 + i + 1)) {
                        fail();
                        stop = true;
                        break;
                    }
                    const int gs = (int)(kb & 1);
                    if (kb >= 2 && !wait_live(&K->gempty[gs], (uint32_t)(((kb >> 1) - 1) & 1), abort)) {
                        fail();
                        stop = true;
                        break;
                    }
                    mbar_arrive_tx(&K->gfull[gs], STRIP_TX);
                    load_strip(gst + gs * GW_G + 2 * WG_STRIP, PLANE, &gmap, &gmap_hi, x0,
                               (b * d.nz + z) * d.ny + y0 + i, &K->gfull[gs]);
                    kissued = kb + 1;
                }
            }
            // no copy may be in flight when the block exits
            for (int64_t k = rissued > GW_R ? rissued - GW_R : 0; k < rissued; k++) {
                uint64_t* bar = &K->rfull[k % GW_R];
                if (!tc::mbar_wait(bar, (uint32_t)((k / GW_R) & 1), WAIT_LIMIT))
                    tc::mbar_wait(bar, (uint32_t)((k / GW_R) & 1), WAIT_LIMIT);
            }
            for (int64_t k = kissued > 2 ? kissued - 2 : 0; k < kissued; k++) {
                uint64_t* bar = &K->gfull[k & 1];
                if (!tc::mbar_wait(bar, (uint32_t)((k >> 1) & 1), WAIT_LIMIT))
                    tc::mbar_wait(bar, (uint32_t)((k >> 1) & 1), WAIT_LIMIT);
            }
        }
    } else if (warp == 1) {
        // MMA issuer (the warp, one elected lane).  Test hook: the workspace's
        // second status word k + 1 > 0 makes the wait for this CTA's K block k
        // report giving up once it has in fact succeeded.
        const int force_at = status[1] - 1;
        constexpr uint32_t idesc = tc::idesc_bf16(TM, 96) | (1u << 15) | (1u << 16);
        const uint64_t ad0 = tc::sdesc(tc::smem_u32(gst), 128, WG_PLANE);
        const uint64_t bd0 = tc::sdesc(tc::smem_u32(ring), 128, WG_PLANE);
        int64_t G = 0, kb = 0;
        bool stop = false;
        for (int64_t it = blockIdx.x; it < wp.nitems && !stop; it += gridDim.x) {
            int b, z, x0, y0, ly;
            item_pos(d, wp, it, b, z, x0, y0, ly);
            for (int i = 0; i < ly; i++, kb++) {
                const int gs = (int)(kb & 1);
                bool got = !*abort && wait_live(&K->gbuilt[gs], (uint32_t)((kb >> 1) & 1), abort);
                int slot[3];
#pragma unroll
                for (int dy = 0; dy < 3; dy++) {
                    const int64_t g2 = G + i + dy;
                    slot[dy] = (int)(g2 % GW_R);
                    if (got && (i == 0 || dy == 2))
                        got = wait_live(&K->rfull[slot[dy]], (uint32_t)((g2 / GW_R) & 1), abort);
                }
                if (kb == force_at) got = false;
                if (!__all_sync(0xffffffffu, got)) {
                    if (lane == 0) fail();
                    stop = true;
                    break;
                }
                tc::fence_after();
                const uint32_t alo = (uint32_t)ad0 + (uint32_t)((gs * GW_G) >> 4);
#pragma unroll
                for (int ks = 0; ks < TM / 16; ks++)
#pragma unroll
                    for (int dy = 0; dy < 3; dy++)
                        tc::mma_bf16_warp(
                            tmem + (uint32_t)(dy * 96), alo + (uint32_t)((ks * 256) >> 4),
                            (uint32_t)(ad0 >> 32),
                            (uint32_t)bd0 + (uint32_t)((slot[dy] * W_SET + 16 + ks * 256) >> 4),
                            (uint32_t)(bd0 >> 32), idesc, (kb > 0 || ks > 0) ? 1u : 0u);
                tc::commit_warp(&K->gempty[gs]);
                // row-set i is not read after this K block; the last one of
                // the item also frees row-sets ly and ly + 1
                tc::commit_warp(&K->rempty[slot[0]]);
                if (i == ly - 1) {
                    tc::commit_warp(&K->rempty[slot[1]]);
                    tc::commit_warp(&K->rempty[slot[2]]);
                }
            }
            G += ly + 2;
        }
        __syncwarp();
    } else {
        // warps 2-5: the shifted gradient copies and the bias sum
        const int h = warp - 2;
        float bacc = 0.f;
        int64_t kb = 0;
        bool stop = false;
        for (int64_t it = blockIdx.x; it < wp.nitems && !stop && !*abort; it += gridDim.x) {
            int b, z, x0, y0, ly;
            item_pos(d, wp, it, b, z, x0, y0, ly);
            for (int i = 0; i < ly; i++, kb++) {
                const int gs = (int)(kb & 1);
                if (!__all_sync(0xffffffffu,
                                wait_live(&K->gfull[gs], (uint32_t)((kb >> 1) & 1), abort))) {
                    if (lane == 0) fail();
                    stop = true;
                    break;
                }
                uint8_t* st = gst + gs * GW_G;
                // copy c (c = 0, 1) row r = copy 2 row r + 2 - c, r < 128: 8 planes
                // x 128 rows of 16 bytes over the 128 builder threads
                const int t = h * 32 + lane;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int u = k * 128 + t;  // 0 .. 1023
                    const int c = u >> 9, p = (u >> 7) & 3, r = u & 127;
                    const uint4 v = *(const uint4*)(st + 2 * WG_STRIP + p * WG_PLANE + (r + 2 - c) * 16);
                    *(uint4*)(st + c * WG_STRIP + p * WG_PLANE + r * 16) = v;
                }
                // channel o = lane of x = 32 h .. 32 h + 31 (copy 2, row x + 1)
                const uint8_t* gp = st + 2 * WG_STRIP + (lane >> 3) * WG_PLANE + (lane & 7) * 2;
#pragma unroll 8
                for (int x = 32 * h; x < 32 * h + 32; x++)
                    bacc += __bfloat162float(*(const __nv_bfloat16*)(gp + (x + 1) * 16));
                tc::fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(&K->gbuilt[gs]);
            }
        }
        K->bsum[h][lane] = bacc;
    }
    // drain: every MMA issued has completed before TMEM is read or released
    __syncthreads();
    if (warp == 1) tc::commit_warp(&K->drain);
    if (!tc::mbar_wait(&K->drain, 0, WAIT_LIMIT)) tc::mbar_wait(&K->drain, 0, WAIT_LIMIT);
    tc::fence_after();
    const bool ok = *abort == 0;
    float* prow = partial + (int64_t)blockIdx.x * 28 * C * C;
    // TMEM lane 32 dx + o, column 96 dy + 32 dz + i: dW[9 dz + 3 dy + dx][o][i]
    if (ok && warp < 3) {
        for (int dy = 0; dy < 3; dy++)
            for (int dz = 0; dz < 3; dz++) {
                uint32_t acc[32];
                tc::ld32(tmem, (uint32_t)(warp * 32), (uint32_t)(dy * 96 + dz * 32), acc);
                float4* dst = (float4*)(prow + ((dz * 9 + dy * 3 + warp) * C + lane) * C);
#pragma unroll
                for (int j = 0; j < 8; j++)
                    dst[j] = make_float4(__uint_as_float(acc[4 * j]), __uint_as_float(acc[4 * j + 1]),
                                         __uint_as_float(acc[4 * j + 2]),
                                         __uint_as_float(acc[4 * j + 3]));
            }
    }
    if (ok && warp == 3)
        prow[(27 * C + lane) * C] =
            ((K->bsum[0][lane] + K->bsum[1][lane]) + K->bsum[2][lane]) + K->bsum[3][lane];
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// grad[tap][o][i] (and grad_b[o] from tap 27, i = 0) = the sum of the CTAs'
// partials (partial[cta][e], e = tap nout + o ni + i).  A block of 8 warps
// takes 32 consecutive e: warp w adds, in CTA order, the CTAs of its eighth of
// the range for the lane's e (coalesced rows), and warp 0 adds the eight
// subtotals in warp order -- a fixed order for a given CTA count.
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float* __restrict__ partial,
                                                           int64_t nchunk, int nout, int ni,
                                                           float* __restrict__ gw,
                                                           float* __restrict__ gb) {
    __shared__ double sub[8][32];
    const int64_t n = 28LL * nout;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * 32 + lane;
    const int64_t c0 = nchunk * w / 8, c1 = nchunk * (w + 1) / 8;
    double s = 0.0;
    if (e < n) {
        int64_t c = c0;
        for (; c + 4 <= c1; c += 4) {
            const float a0 = partial[c * n + e], a1 = partial[(c + 1) * n + e];
            const float a2 = partial[(c + 2) * n + e], a3 = partial[(c + 3) * n + e];
            s += a0;
            s += a1;
            s += a2;
            s += a3;
        }
        for (; c < c1; c++) s += partial[c * n + e];
    }
    sub[w][lane] = s;
    __syncthreads();
    if (w == 0 && e < n) {
        double t = 0.0;
        for (int k = 0; k < 8; k++) t += sub[k][lane];
        const int tap = (int)(e / nout), oi = (int)(e % nout);
        if (tap < 27) gw[e] = (float)t;
        else if (oi % ni == 0) gb[oi / ni] = (float)t;
    }
}

// ---------------------------------------------------------------------------
// Packing FP32 master weights W[tap][o][i] into the BF16 B operands.
// mode 0: forward of a 32-input layer: tap t, row n = o (NOUT rows, o >= NO zero), k = i.
// mode 1: dgrad of a 32-output layer (input gradient has NO = 32 channels):
//         tap t' , row n = i, k = o, from W[26 - t'] (flipped).
// mode 2: forward of the 1-input layer: one tile, row n = o, k = tap.
// mode 3: dgrad of the 1-output layer as a 1-channel conv: row n = i, k = tap',
//         from W[26 - tap'][0][i].
// mode 4: forward of the 1-output layer in row passes: per dx one 16 x 32
//         block, row n = (dz, dy) = 3 dz + dy (n < 9), k = i, from
//         W[9 dz + 3 dy + dx][0][i].
// The 27 taps t = 9 dz + 3 dy + dx of modes 0 and 1 stand in the order of
// conv32_ys_kernel: per (dz, dx) the taps dy = 2, 1, 0 one after another.
__host__ __device__ inline int hid_tap(int t) {
    const int dz = t / 9, dy = (t / 3) % 3, dx = t % 3;
    return (dz * 3 + dx) * 3 + (2 - dy);
}

__global__ void pack_kernel(const float* __restrict__ w, int mode, int NI, int NO, int NOUT,
                            __nv_bfloat16* __restrict__ out) {
    const int per_tap = NOUT * C;
    const int total = (mode == 2 || mode == 3) ? C * C : (mode == 4 ? 3 * 16 * C : 27 * per_tap);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        float v = 0.f;
        int dst;
        if (mode == 0) {
            const int t = e / per_tap, r = e % per_tap, n = r / C, k = r % C;
            if (n < NO && k < NI) v = w[((int64_t)t * NO + n) * NI + k];
            dst = hid_tap(t) * per_tap + bpk_index(n, k);
        } else if (mode == 1) {
            const int t = e / per_tap, r = e % per_tap, n = r / C, k = r % C;
            if (n < NI && k < NO) v = w[((int64_t)(26 - t) * NO + k) * NI + n];
            dst = hid_tap(t) * per_tap + bpk_index(n, k);
        } else if (mode == 2) {
            const int n = e / C, k = e % C;
            if (k < 27 && n < NO) v = w[((int64_t)k * NO + n) * NI + 0];
            dst = bpk_index(n, k);
        } else if (mode == 3) {
            const int n = e / C, k = e % C;
            if (k < 27 && n < NI) v = w[((int64_t)(26 - k) * NO + 0) * NI + n];
            dst = bpk_index(n, k);
        } else {
            const int dx = e / (16 * C), r = e % (16 * C), n = r / C, k = r % C;
            if (n < 9) v = w[((int64_t)((n / 3) * 9 + (n % 3) * 3 + dx) * NO + 0) * NI + k];
            dst = dx * 16 * C + bpk_index(n, k);
        }
        out[dst] = __float2bfloat16(v);
    }
}

// Loss 1/V sum (f - r)^2 (per-block FP64 partials) and its gradient 2(f - r)/V.
__global__ void loss_kernel(const float* __restrict__ f, const float* __restrict__ r, int64_t V,
                            float* __restrict__ g, double* __restrict__ partial) {
    __shared__ double ws[8];
    double s = 0.0;
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V;
         v += (int64_t)gridDim.x * blockDim.x) {
        const float e = f[v] - r[v];
        g[v] = 2.f * e / (float)V;
        s += (double)e * e;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += ws[k];
        partial[blockIdx.x] = t;
    }
}

// One warp: lane l adds partials l, l + 32, ...; then a fixed shuffle tree.
__global__ void loss_final_kernel(const double* __restrict__ partial, int n, int64_t V,
                                  double* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    for (int k = lane; k < n; k += 32) t += partial[k];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) out[0] = t / (double)V;
}

// Adam (Kingma & Ba 2015) with bias correction, FP32 master parameters.
__global__ void adam_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                            const float* __restrict__ g, int64_t n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
         k += (int64_t)gridDim.x * blockDim.x) {
        const float gk = g[k];
        const float mk = b1 * m[k] + (1.f - b1) * gk;
        const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
        m[k] = mk;
        v[k] = vk;
        p[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
    }
}

}  // namespace cnn
}  // namespace nr

// ---------------------------------------------------------------------------
// Host side: parameter layout, workspace layout, forward / backward sequencing.
namespace nr {
namespace cnn {

struct Layer {
    int ni, no;
};
constexpr Layer LAYERS[6] = {{1, C}, {C, C}, {C, C}, {C, C}, {C, C}, {C, 1}};

// FP32 parameters: for each layer W[27][no][ni] then b[no].
static void param_offsets(int64_t* w, int64_t* b, int64_t* total) {
    int64_t o = 0;
    for (int l = 0; l < 6; l++) {
        w[l] = o;
        o += 27LL * LAYERS[l].no * LAYERS[l].ni;
        b[l] = o;
        o += LAYERS[l].no;
    }
    *total = o;
}

constexpr size_t PK_HID = 27 * C * C * 2;   // packed 32 -> 32 taps
constexpr size_t PK_LAST = 27 * 16 * C * 2; // packed 32 -> 1 (16 rows)
constexpr size_t PK_ONE = C * C * 2;        // packed 1-channel tile

struct WSL {
    size_t status, pk_fwd[6], pk_bwd[6], act[5], f, r, g6, dpre[2], part, grad, lpart, lout, total;
    int64_t nchunk, lblocks;
};

static size_t al(size_t v) { return (v + 255) & ~(size_t)255; }

static WSL layout(const Dims& d, bool training) {
    WSL L{};
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o = al(o + bytes);
        return at;
    };
    const int64_t V = nvox(d);
    int64_t wo[6], bo[6], P;
    param_offsets(wo, bo, &P);
    L.status = take(256);
    L.pk_fwd[0] = take(PK_ONE);
    for (int l = 1; l < 5; l++) L.pk_fwd[l] = take(PK_HID);
    L.pk_fwd[5] = take(PK_LAST);
    const int nact = training ? 5 : 2;
    for (int k = 0; k < nact; k++) L.act[k] = take((size_t)V * C * 2);
    L.nchunk = ntiles(d) < WG_MAXCTA ? ntiles(d) : WG_MAXCTA;  // CTAs of a weight gradient
    L.lblocks = 1024;
    if (training) {
        for (int l = 1; l < 5; l++) L.pk_bwd[l] = take(PK_HID);
        L.pk_bwd[5] = take(PK_ONE);
        L.f = take((size_t)V * 4);
        L.r = take((size_t)V * 4);
        L.g6 = take((size_t)V * 4);
        L.dpre[0] = take((size_t)V * C * 2);
        L.dpre[1] = take((size_t)V * C * 2);
        L.part = take((size_t)28 * C * C * L.nchunk * 4);
        L.grad = take((size_t)P * 4);
        L.lpart = take((size_t)L.lblocks * 8);
        L.lout = take(8);
    }
    L.total = o;
    return L;
}

}  // namespace cnn
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encode_fn();
namespace cnn {

// The TMA maps of an activation tensor (act_off's layout) seen as (2 nx
// 8-byte units, 4 K chunks, R rows): one K chunk of a row is one contiguous
// run; `lo` boxes are 128 units (strip rows 0-63), `hi` boxes 132 units (rows
// 64-129).  Zeros outside the tensor.
struct ActMaps {
    CUtensorMap lo, hi;
};
static bool act_maps(const Dims& d, const __nv_bfloat16* in, ActMaps* m) {
    auto enc = tensor_map_encode_fn();
    if (!enc || ((uintptr_t)in & 15) != 0) return false;
    const cuuint64_t rows = (cuuint64_t)d.ny * d.nz * d.nb;
    const cuuint64_t dims[3] = {(cuuint64_t)d.nx * 2, (cuuint64_t)KCH, rows};
    const cuuint64_t strides[2] = {(cuuint64_t)d.nx * 16, (cuuint64_t)d.nx * C * 2};
    const cuuint32_t estr[3] = {1, 1, 1};
    const cuuint32_t box_lo[3] = {128, 1, 1}, box_hi[3] = {132, 1, 1};
    auto one = [&](CUtensorMap* map, const cuuint32_t* box) {
        return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, (void*)in, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    return one(&m->lo, box_lo) && one(&m->hi, box_hi);
}

template <int EPI>
static nr_status launch_conv32(const Dims& d, const __nv_bfloat16* in, const __nv_bfloat16* wpk,
                               const float* bias, __nv_bfloat16* out, const __nv_bfloat16* mask,
                               int* status, cudaStream_t s) {
    // Runs of L rows, each L + 2 steps: the number of runs per column whose
    // busiest CTA has the fewest steps (few columns want short runs that fill
    // the GPU, many want long ones).
    const int64_t nsm = sm_count();
    const int64_t ncols = (int64_t)d.nb * ((d.nz + 1) / 2) * xtiles(d);
    WalkPlan wp;
    int64_t best = INT64_MAX;
    for (int nchunk = 1; nchunk <= d.ny && nchunk <= 64; nchunk++) {
        const int64_t L = (d.ny + nchunk - 1) / nchunk, n = (d.ny + L - 1) / L;
        const int64_t steps = (ncols * n + nsm - 1) / nsm * (L + 2);
        if (steps < best) {
            best = steps;
            wp.L = (int)L;
            wp.nchunk = (int)n;
        }
    }
    wp.tw = TM;
    wp.nitems = ncols * wp.nchunk;
    const size_t smem = (size_t)Y_R * Y_SET + Y_WBYTES + sizeof(YCtl);
    if (cudaFuncSetAttribute(conv32_ys_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
        return NR_ERR_CUDA;
    const int grid = (int)(wp.nitems < nsm ? wp.nitems : nsm);
    conv32_ys_kernel<EPI><<<grid, Y_THREADS, smem, s>>>(d, wp, in, wpk, bias, out, mask, status);
    return launch_status();
}

template <int EPI>
static nr_status launch_conv1(const Dims& d, const float* in, float scale,
                              const __nv_bfloat16* wpk, const float* bias, __nv_bfloat16* out,
                              const __nv_bfloat16* mask, int* status, cudaStream_t s) {
    // four CTAs per SM (nine, as many as fit, measured 2.7x slower on the
    // clinical volume), each walking runs of L rows: about eight runs per CTA
    const int nsm = sm_count();
    const int64_t ncols = (int64_t)d.nb * d.nz * xtiles(d);
    int64_t L = ((int64_t)d.ny * ncols + 32LL * nsm - 1) / (32LL * nsm);
    L = L < 1 ? 1 : (L > 32 ? 32 : L);
    if (L > d.ny) L = d.ny;
    WalkPlan wp;
    wp.L = (int)L;
    wp.nchunk = (int)((d.ny + L - 1) / L);
    wp.tw = TM;
    wp.nitems = ncols * wp.nchunk;
    const int grid = (int)(wp.nitems < (int64_t)nsm * 4 ? wp.nitems : (int64_t)nsm * 4);
    conv1_kernel<EPI><<<grid, 128, 0, s>>>(d, wp, in, scale, wpk, bias, out, mask, status);
    return launch_status();
}

// The 32 -> 1 layer (two passes); q: 9 V floats of scratch.  f: the layer's
// output, or with x_in the network's, max(0, x_in + inv_s f).
static nr_status launch_last(const Dims& d, const __nv_bfloat16* in, const __nv_bfloat16* wpk,
                             const float* bias, float* q, const float* x_in, float inv_s, float* f,
                             int* status, cudaStream_t s) {
    ActMaps map;
    if (!act_maps(d, in, &map)) return NR_ERR_CUDA;
    const size_t smem = (size_t)LR_STAGE * TSTRIP + 3 * 16 * C * 2 + sizeof(LastCtl);
    if (cudaFuncSetAttribute(last_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
        return NR_ERR_CUDA;
    const int64_t nt = ntiles(d);
    const int grid = (int)(nt < (int64_t)sm_count() * 4 ? nt : (int64_t)sm_count() * 4);
    last_rows_kernel<<<grid, LR_THREADS, smem, s>>>(d, map.lo, map.hi, wpk, q, status);
    // q planes start at multiples of V floats: with nx % 4 == 0 every row is 16-byte
    // aligned (the workspace is 256-byte aligned; x_in and f are the caller's)
    const bool vec = d.nx % 4 == 0 && (((uintptr_t)x_in | (uintptr_t)f) & 15) == 0;
    const dim3 g2((unsigned)((int64_t)d.nb * d.nz * d.ny),
                  (unsigned)(((vec ? d.nx / 4 : d.nx) + 255) / 256));
    if (vec && x_in)
        last_sum_kernel<4, true><<<g2, 256, 0, s>>>(d, q, bias, x_in, inv_s, f);
    else if (vec)
        last_sum_kernel<4, false><<<g2, 256, 0, s>>>(d, q, bias, nullptr, 0.f, f);
    else if (x_in)
        last_sum_kernel<1, true><<<g2, 256, 0, s>>>(d, q, bias, x_in, inv_s, f);
    else
        last_sum_kernel<1, false><<<g2, 256, 0, s>>>(d, q, bias, nullptr, 0.f, f);
    return launch_status();
}

static void pack(const float* w, int mode, int ni, int no, int nout, __nv_bfloat16* out,
                 cudaStream_t s) {
    pack_kernel<<<64, 256, 0, s>>>(w, mode, ni, no, nout, out);
}

// Forward through layer 6: f = conv6(a5) in the workspace's `f`, or with out
// given the network's output there; activations in `acts` (5 buffers when
// `keep`, else 2 ping-pong buffers).
static nr_status forward(const Dims& d, const float* params, const float* x, float s, float* out,
                         char* ws, const WSL& L, bool keep, cudaStream_t st) {
    int64_t wo[6], bo[6], P;
    param_offsets(wo, bo, &P);
    int* status = (int*)(ws + L.status);
    auto pkf = [&](int l) { return (__nv_bfloat16*)(ws + L.pk_fwd[l]); };
    pack(params + wo[0], 2, 1, C, C, pkf(0), st);
    for (int l = 1; l < 5; l++) pack(params + wo[l], 0, C, C, C, pkf(l), st);
    pack(params + wo[5], 4, C, 1, 16, pkf(5), st);
    auto act = [&](int l) {  // output of layer l (0-based, l < 5)
        return (__nv_bfloat16*)(ws + L.act[keep ? l : (l & 1)]);
    };
    nr_status e;
    if ((e = launch_conv1<EPI_RELU>(d, x, s, pkf(0), params + bo[0], act(0), nullptr, status, st)) != NR_OK)
        return e;
    for (int l = 1; l < 5; l++)
        if ((e = launch_conv32<EPI_RELU>(d, act(l - 1), pkf(l), params + bo[l], act(l), nullptr,
                                            status, st)) != NR_OK)
            return e;
    // q of the last layer: a buffer idle by now (the gradient buffer when the
    // activations are kept for training, else layer 4's ping-pong buffer)
    float* q = (float*)(ws + (keep ? L.dpre[0] : L.act[1]));
    return launch_last(d, act(4), pkf(5), params + bo[5], q, out ? x : nullptr, 1.f / s,
                       out ? out : (float*)(ws + L.f), status, st);
}

__global__ void target_kernel(const float* __restrict__ x, const float* __restrict__ t, float s,
                              int64_t V, float* __restrict__ r) {
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < V;
         v += (int64_t)gridDim.x * blockDim.x)
        r[v] = s * (t[v] - x[v]);
}

template <int MODE>
static nr_status launch_wgrad(const Dims& d, const ActMaps& am, const ActMaps& gm,
                              const float* gvec, const float* xin, float s, float* part,
                              int* status, int64_t nch, cudaStream_t st) {
    if (cudaFuncSetAttribute(wgrad_tc_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             WgCfg<MODE>::SMEM) != cudaSuccess)
        return NR_ERR_CUDA;
    wgrad_tc_kernel<MODE><<<(unsigned)nch, WG_THREADS, WgCfg<MODE>::SMEM, st>>>(
        d, am.lo, am.hi, gm.lo, gm.hi, gvec, xin, s, part, status);
    return launch_status();
}

// Weight and bias gradients of layer l (0-based) into grad: the tensor-core
// GEMM (one partial per CTA), then the fixed-order reduction.  Layer 0 reads
// the FP32 input volume (times s), layer 5 the FP32 gradient of the output.
static nr_status wgrad(const Dims& d, int l, const void* g, const void* in, float s, char* ws,
                       const WSL& L, float* grad, int* status, cudaStream_t st) {
    int64_t wo[6], bo[6], P;
    param_offsets(wo, bo, &P);
    float* part = (float*)(ws + L.part);
    const int64_t nt = ntiles(d);
    int64_t nch = nt < (int64_t)sm_count() ? nt : (int64_t)sm_count();
    if (nch > L.nchunk) nch = L.nchunk;
    ActMaps am{}, gm{};  // a map a mode does not read stays zero
    if (l > 0 && !act_maps(d, (const __nv_bfloat16*)in, &am)) return NR_ERR_CUDA;
    if (l < 5 && !act_maps(d, (const __nv_bfloat16*)g, &gm)) return NR_ERR_CUDA;
    nr_status e;
    int nout = C, ni = C;
    if (l == 0) {
        e = launch_wgrad<WG_FIRST>(d, am, gm, nullptr, (const float*)in, s, part, status, nch, st);
        ni = 1;
    } else if (l == 5) {
        e = launch_wgrad<WG_LAST>(d, am, gm, (const float*)g, nullptr, 1.f, part, status, nch, st);
    } else {
        // runs of L rows along y: about eight per CTA
        int64_t L = ((int64_t)d.ny * d.nb * d.nz * xtiles(d) + 8 * nch - 1) / (8 * nch);
        L = L < 4 ? 4 : (L > 32 ? 32 : L);
        if (L > d.ny) L = d.ny;
        WalkPlan wp;
        wp.L = (int)L;
        wp.nchunk = (int)((d.ny + L - 1) / L);
        wp.tw = TM;
        wp.nitems = (int64_t)d.nb * d.nz * xtiles(d) * wp.nchunk;
        if (wp.nitems < nch) nch = wp.nitems;
        const size_t smem = (size_t)GW_R * W_SET + 2 * GW_G + sizeof(GwCtl);
        if (cudaFuncSetAttribute(wgrad_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem) != cudaSuccess)
            return NR_ERR_CUDA;
        wgrad_walk_kernel<<<(unsigned)nch, GW_THREADS, smem, st>>>(d, wp, am.lo, am.hi, gm.lo,
                                                                   gm.hi, part, status);
        e = launch_status();
        nout = C * C;
    }
    if (e != NR_OK) return e;
    wgrad_reduce_kernel<<<(28 * nout + 31) / 32, 256, 0, st>>>(part, nch, nout, ni, grad + wo[l],
                                                               grad + bo[l]);
    return launch_status();
}

static nr_status loss_grad(const Dims& d, const float* params, const float* x, const float* target,
                           float s, float* grad, char* ws, const WSL& L, cudaStream_t st) {
    const int64_t V = nvox(d);
    int64_t wo[6], bo[6], P;
    param_offsets(wo, bo, &P);
    int* status = (int*)(ws + L.status);
    nr_status e;
    if ((e = forward(d, params, x, s, nullptr, ws, L, true, st)) != NR_OK) return e;
    float* r = (float*)(ws + L.r);
    float* g6 = (float*)(ws + L.g6);
    target_kernel<<<1024, 256, 0, st>>>(x, target, s, V, r);
    loss_kernel<<<(unsigned)L.lblocks, 256, 0, st>>>((const float*)(ws + L.f), r, V, g6,
                                                      (double*)(ws + L.lpart));
    loss_final_kernel<<<1, 32, 0, st>>>((const double*)(ws + L.lpart), (int)L.lblocks, V,
                                        (double*)(ws + L.lout));
    auto act = [&](int l) { return (const __nv_bfloat16*)(ws + L.act[l]); };
    auto dpre = [&](int k) { return (__nv_bfloat16*)(ws + L.dpre[k & 1]); };
    auto pkb = [&](int l) { return (__nv_bfloat16*)(ws + L.pk_bwd[l]); };
    for (int l = 1; l < 5; l++) pack(params + wo[l], 1, C, C, C, pkb(l), st);
    pack(params + wo[5], 3, C, 1, C, pkb(5), st);
    // layer 6: weight gradient and the masked input gradient dpre5
    if ((e = wgrad(d, 5, g6, act(4), 1.f, ws, L, grad, status, st)) != NR_OK) return e;
    if ((e = launch_conv1<EPI_MASK>(d, g6, 1.f, pkb(5), nullptr, dpre(4), act(4), status, st)) !=
        NR_OK)
        return e;
    // layers 5..2: dpre_l lives in dpre(l-1)
    for (int l = 4; l >= 1; l--) {
        if ((e = wgrad(d, l, dpre(l), act(l - 1), 1.f, ws, L, grad, status, st)) != NR_OK) return e;
        if ((e = launch_conv32<EPI_MASK>(d, dpre(l), pkb(l), nullptr, dpre(l - 1), act(l - 1),
                                            status, st)) != NR_OK)
            return e;
    }
    return wgrad(d, 0, dpre(0), x, s, ws, L, grad, status, st);
}

}  // namespace cnn
}  // namespace nr

using namespace nr;
using namespace nr::cnn;

static bool dims_ok(const nr_cnn_dims* d) {
    return d && d->nx > 0 && d->ny > 0 && d->nz > 0 && d->nb > 0 &&
           (int64_t)d->nx * d->ny * d->nz * d->nb < ((int64_t)1 << 31);
}

static Dims to_dims(const nr_cnn_dims* d) { return Dims{d->nx, d->ny, d->nz, d->nb}; }

NR_API nr_status nr_cnn_param_count(int64_t* n) {
    if (!n) return NR_ERR_BAD_ARGUMENT;
    int64_t wo[6], bo[6];
    param_offsets(wo, bo, n);
    return NR_OK;
}

NR_API nr_status nr_cnn_workspace_size(const nr_cnn_dims* d, int32_t training, size_t* bytes) {
    if (!dims_ok(d) || !bytes) return NR_ERR_BAD_ARGUMENT;
    *bytes = layout(to_dims(d), training != 0).total;
    return NR_OK;
}

NR_API nr_status nr_cnn_forward(const nr_cnn_dims* d, const float* params, const float* x,
                                float in_scale, float* x_out, void* ws, size_t ws_bytes,
                                void* stream) {
    if (!dims_ok(d) || !params || !x || !x_out || !(in_scale > 0.f)) return NR_ERR_BAD_ARGUMENT;
    const Dims D = to_dims(d);
    const WSL L = layout(D, false);
    if (!ws || ws_bytes < L.total || ((uintptr_t)ws & 255)) return NR_ERR_WORKSPACE;
    cudaStream_t st = as_stream(stream);
    return forward(D, params, x, in_scale, x_out, (char*)ws, L, false, st);
}

NR_API nr_status nr_cnn_loss_grad(const nr_cnn_dims* d, const float* params, const float* x,
                                  const float* target, float in_scale, float* grad, double* loss,
                                  void* ws, size_t ws_bytes, void* stream) {
    if (!dims_ok(d) || !params || !x || !target || !(in_scale > 0.f)) return NR_ERR_BAD_ARGUMENT;
    const Dims D = to_dims(d);
    const WSL L = layout(D, true);
    if (!ws || ws_bytes < L.total || ((uintptr_t)ws & 255)) return NR_ERR_WORKSPACE;
    cudaStream_t st = as_stream(stream);
    char* w = (char*)ws;
    float* g = grad ? grad : (float*)(w + L.grad);
    nr_status e = loss_grad(D, params, x, target, in_scale, g, w, L, st);
    if (e != NR_OK) return e;
    if (loss &&
        cudaMemcpyAsync(loss, w + L.lout, 8, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return NR_ERR_CUDA;
    return NR_OK;
}

NR_API nr_status nr_cnn_adam(float* params, float* m, float* v, const float* grad, int64_t n,
                             int32_t step, float lr, void* stream) {
    if (!params || !m || !v || !grad || n <= 0 || step < 1 || !(lr > 0.f)) return NR_ERR_BAD_ARGUMENT;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    adam_kernel<<<256, 256, 0, as_stream(stream)>>>(params, m, v, grad, n, lr, b1, b2, 1e-8f, c1,
                                                    c2);
    return launch_status();
}

NR_API nr_status nr_cnn_train_step(const nr_cnn_dims* d, float* params, float* adam_m,
                                   float* adam_v, int32_t step, float lr, const float* x,
                                   const float* target, float in_scale, double* loss, void* ws,
                                   size_t ws_bytes, void* stream) {
    nr_status e = nr_cnn_loss_grad(d, params, x, target, in_scale, nullptr, loss, ws, ws_bytes,
                                   stream);
    if (e != NR_OK) return e;
    const WSL L = layout(to_dims(d), true);
    int64_t P;
    nr_cnn_param_count(&P);
    return nr_cnn_adam(params, adam_m, adam_v, (const float*)((char*)ws + L.grad), P, step, lr,
                       stream);
}

NR_API nr_status nr_cnn_check(void* ws, int32_t* flags, void* stream) {
    if (!ws || !flags) return NR_ERR_BAD_ARGUMENT;
    cudaStream_t s = as_stream(stream);
    int v = 0;
    if (cudaMemcpyAsync(&v, ws, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return NR_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return NR_ERR_CUDA;
    *flags = v;
    if (v) cudaMemsetAsync(ws, 0, sizeof(int), s);
    return (v & NR_FLAG_TIMEOUT) ? NR_ERR_TIMEOUT : NR_OK;
}
