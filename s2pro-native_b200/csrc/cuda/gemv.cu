/* Stand-alone GEMV entry points of the C ABI (include/s2p_b200_abi.h):
 * s2p_int8_gemv, s2p_intq_gemv, s2p_int4p_gemv — the reference's
 * src/sched/int8_gemv.cu:964-986, :773-799, :836-902.
 *
 * One row, and two of a matrix of few rows, run k_gemv_row; up to 16 rows run
 * k_gemv_batch, where codes are widened once per tile for up to eight rows.  Every
 * row of x is an independent product with one summation order (the reference's
 * batched GEMV computes rows independently too, int8_gemv.cu:77-91).  The stage
 * kernel of gemv.cuh (k_gemv_stage) serves the fused per-stage frame only.
 */
#include <stdio.h>
#include "gemv.cuh"
#include "ops.h"
#include "packed.cuh"
#include "s2p_b200_abi.h"

namespace s2p {

int device_sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

template <int WK, int PRO, int EPI>
__global__ void __launch_bounds__(GEMV_THREADS, 1) k_gemv_stage(GemvStage g) {
    extern __shared__ __align__(16) unsigned char smem[];
    int row0, cnt;
    gemv_cta_rows<EPI>(g, blockIdx.x, gridDim.x, row0, cnt);
    gemv_stage_cta<WK, PRO, EPI>(g, row0, cnt, smem);
}

/* Rows per pass that keep the CTA's shared memory within `limit` bytes. */
int gemv_rows_per_pass(int wk, int rows_per_cta, int K, int gshift, int swiglu, size_t limit) {
    int r = rows_per_cta;
    while (r > 8 && gemv_smem_bytes(wk, r * (swiglu ? 2 : 1), K, gshift) > limit) r = (r + 1) / 2;
    return r < 1 ? 1 : r;
}

constexpr size_t GEMV_SMEM_LIMIT = 200 * 1024;

/* Opt the kernel in to large dynamic shared memory, once per device. */
template <int WK, int PRO, int EPI>
cudaError_t gemv_stage_setup() {
    static int done_mask = 0; /* bit per device ordinal */
    int dev = 0;
    cudaGetDevice(&dev);
    if (done_mask & (1 << (dev & 31))) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(k_gemv_stage<WK, PRO, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)GEMV_SMEM_LIMIT);
    if (e == cudaSuccess) done_mask |= 1 << (dev & 31);
    return e;
}

template <int WK, int PRO, int EPI>
cudaError_t launch_gemv_stage(GemvStage g, cudaStream_t stream) {
    const size_t limit = GEMV_SMEM_LIMIT;
    {
        const cudaError_t e = gemv_stage_setup<WK, PRO, EPI>();
        if (e != cudaSuccess) return e;
    }
    const int units = (EPI == EPI_SWIGLU) ? (g.N >> 1) : g.N;
    int grid = device_sm_count();
    if (grid > units) grid = units;
    const int rows_per_cta = (units + grid - 1) / grid;
    g.rows_per_pass = gemv_rows_per_pass(WK, rows_per_cta, g.K, g.gshift, EPI == EPI_SWIGLU, limit);
    const size_t smem = gemv_smem_bytes(WK, g.rows_per_pass * (EPI == EPI_SWIGLU ? 2 : 1), g.K, g.gshift);
    return launch_after(k_gemv_stage<WK, PRO, EPI>, dim3((unsigned)grid), GEMV_THREADS, smem, stream, g);
}

/* instantiations used by the tick live here so that every kernel is compiled once */
#define S2P_INST(WK)                                                                         \
    template cudaError_t launch_gemv_stage<WK, PRO_NORM, EPI_STORE>(GemvStage, cudaStream_t); \
    template cudaError_t launch_gemv_stage<WK, PRO_VEC, EPI_RESID>(GemvStage, cudaStream_t);  \
    template cudaError_t launch_gemv_stage<WK, PRO_NORM, EPI_SWIGLU>(GemvStage, cudaStream_t);\
    template cudaError_t launch_gemv_stage<WK, PRO_NORM, EPI_ARGMAX>(GemvStage, cudaStream_t);
S2P_INST(WK_INT8_CH)
S2P_INST(WK_INT8_GRP)
S2P_INST(WK_INT4_PACK)
#undef S2P_INST

/* Attribute set-up for every instantiation, to be called once before any stream
 * capture (function attributes are not stream operations). */
extern "C" cudaError_t gemv_setup_all(void) {
    cudaError_t e = cudaSuccess;
#define S2P_SETUP(WK, PRO, EPI) if (e == cudaSuccess) e = gemv_stage_setup<WK, PRO, EPI>();
#define S2P_SETUP_WK(WK)               \
    S2P_SETUP(WK, PRO_NORM, EPI_STORE) \
    S2P_SETUP(WK, PRO_VEC, EPI_RESID)  \
    S2P_SETUP(WK, PRO_NORM, EPI_SWIGLU) \
    S2P_SETUP(WK, PRO_NORM, EPI_ARGMAX)
    S2P_SETUP_WK(WK_INT8_CH)
    S2P_SETUP_WK(WK_INT8_GRP)
    S2P_SETUP_WK(WK_INT4_PACK)
#undef S2P_SETUP_WK
#undef S2P_SETUP
    return e;
}

/* ---- exact-order small batch (2 <= M <= 16) -------------------------------
 * Lane l owns k = 512 i + 16 l .. +15 of every tile i, as for M == 1; a warp carries four weight rows and MM activation
 * rows, 4 x MM independent chains.
 *
 * What bounds it: fp32 fma and what surrounds one.  Two activation rows share a register pair, so a chain step is packed
 * (fma.rn.f32x2: two independent roundings, the same bits as fmaf on either half); an activation becomes f32 with one
 * instruction, a code (a byte planted in the mantissa of 2^23 twice and one packed subtraction, exact) once per MM activation rows.
 * The chains of a k advance side by side, because each waits for its own previous step.  Weights go from DRAM to registers a tile
 * ahead; the activations of a tile are shared by the SM's warps through L1.
 *
 * A matrix of few rows does not fill the GPU with warps of four rows, and a lone warp per scheduler waits on its own
 * latencies.  There NS = 4 warps share four rows and take tiles in turn; the tiles' chain results meet in shared memory and each warp
 * folds a quarter of the activation rows, tiles ascending.
 * Measured, us for one layer's four matrices (N x K 6144 x 2560, 2560 x 4096, 19456 x 2560, 2560 x 9728), before (scalar fma, one
 * weight row per warp for INT8; mixed bf16 fma, one to four for INT4) and now, at 2 / 4 / 8 / 16 rows:
 *   INT8  52 / 84 / 148 / 258 -> 44 / 56 / 81 / 135      INT4  46 / 70 / 103 / 180 -> 46 / 56 / 85 / 146
 * (2 rows now share the one-row kernel where rows are few: 38 and 39).
 * An odd row's chain is scalar: padded to a pair it held the fma pipe for two (3 rows INT4 58 -> 53, 5 rows 74 -> 68, 9 rows 119 -> 108).
 * 16 rows of 19456 x 2560 INT4 run at 11.4 T fma/s; the pipe's rate is 36 T.  Counters there: issue slots 59 %, fma pipe 51 %, integer
 * pipe 44 % busy, 11 of 64 warps resident (168 registers), 5 % of DRAM. */
/* A SwiGLU over stacked [gate | up] rows (SW): half of a warp's rows are of either half, so gate and up of an output meet in
 * the warp; both round to bf16 first, as where a kernel of its own follows the linear. */
template <bool SW, int R> __device__ __forceinline__ int gemv_row_of(int n0, int r, int F) {
    return SW ? min(n0 + r % (R / 2), F - 1) + r / (R / 2) * F : min(n0 + r, F - 1);
}
__device__ __forceinline__ float gemv_swiglu(float gate, float up_) {
    const float g = bf16_round(gate), up = bf16_round(up_);
    const float sig = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-g)));
    return __fmul_rn(bf16_round(__fmul_rn(g, sig)), up);
}
template <int WK> struct BatchCodes;
template <> struct BatchCodes<WK_INT8_CH> {
    static __device__ __forceinline__ f32x2 twice(uint32_t u, uint32_t sel, float minus) {
        const float f = __uint_as_float(__byte_perm(u, 0x4B000000u, sel));
        return fadd2(pack2(f, f), pack2(minus, minus));
    }
    /* codes k = 8 h + 0..7 of two rows as f32 pairs (row a, row b) */
    static __device__ __forceinline__ f32x2 both(uint32_t a, uint32_t b, uint32_t sel, float minus) {
        return fadd2(pack2(__uint_as_float(__byte_perm(a, 0x4B000000u, sel)), __uint_as_float(__byte_perm(b, 0x4B000000u, sel))), pack2(minus, minus));
    }
    static __device__ __forceinline__ void widen8(const uint4& a, const uint4& b, int h, f32x2 (&w)[8]) {
        const uint32_t ua[2] = {s8x4_bias(h ? a.z : a.x), s8x4_bias(h ? a.w : a.y)}, ub[2] = {s8x4_bias(h ? b.z : b.x), s8x4_bias(h ? b.w : b.y)};
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = both(ua[j >> 2], ub[j >> 2], 0x7440u + (j & 3), -8388736.0f);
    }
    /* codes k = 8 h + 0..7 of a lane as f32 pairs of equals */
    static __device__ __forceinline__ void widen8(const uint4& a, int h, f32x2 (&w)[8]) {
        const uint32_t u[2] = {s8x4_bias(h ? a.z : a.x), s8x4_bias(h ? a.w : a.y)};
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = twice(u[j >> 2], 0x7440u + (j & 3), -8388736.0f);
    }
};
template <> struct BatchCodes<WK_INT8_GRP> : BatchCodes<WK_INT8_CH> {};
template <> struct BatchCodes<WK_INT4_PACK> {
    static __device__ __forceinline__ void widen8(const uint2& a, const uint2& b, int h, f32x2 (&w)[8]) {
        const uint32_t ua = h ? a.y : a.x, ub = h ? b.y : b.x;
        const uint32_t ea = (ua & 0x0F0F0F0Fu) ^ 0x08080808u, oa = ((ua >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
        const uint32_t eb = (ub & 0x0F0F0F0Fu) ^ 0x08080808u, ob = ((ub >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
#pragma unroll
        for (int j = 0; j < 8; j++)
            w[j] = BatchCodes<WK_INT8_CH>::both(j & 1 ? oa : ea, j & 1 ? ob : eb, 0x7440u + (j >> 1), -8388616.0f);
    }
    static __device__ __forceinline__ void widen8(const uint2& a, int h, f32x2 (&w)[8]) {
        const uint32_t u = h ? a.y : a.x; /* two's complement nibble -> code + 8, even and odd k apart */
        const uint32_t e = (u & 0x0F0F0F0Fu) ^ 0x08080808u, o = ((u >> 4) & 0x0F0F0F0Fu) ^ 0x08080808u;
#pragma unroll
        for (int j = 0; j < 8; j++) w[j] = BatchCodes<WK_INT8_CH>::twice(j & 1 ? o : e, 0x7440u + (j >> 1), -8388616.0f);
    }
};

template <int WK, int MM, int NS, bool SW>
__global__ void __launch_bounds__(128, 3) k_gemv_batch(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x,
                                                       const void* __restrict__ w, const void* __restrict__ scales,
                                                       int M, int N, int K, int gshift) {
    typedef typename LaneTile<WK>::type tile_t;
    constexpr int R = 4, P = MM / 2; /* weight rows of a warp, pairs of activation rows; an odd last one has scalar chains */
    constexpr bool ODD = MM % 2 != 0;
    constexpr int PD = WK == WK_INT4_PACK && MM <= 4 ? 2 : 1; /* tiles of weights under way */
    constexpr int FM = NS == 1 ? MM : (MM + NS - 1) / NS; /* activation rows whose sums this warp keeps */
    __shared__ float part[NS == 1 ? 1 : 2 * NS * (MM + 1) * R * 32]; /* [round parity][tile of the round][m, then the scales][row][lane] */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int F = SW ? N >> 1 : N; /* outputs */
    const int n0 = (blockIdx.x * (4 / NS) + warp / NS) * (SW ? R / 2 : R), ns = warp % NS;
    if (n0 >= F) return; /* NS > 1: uniform over the CTA */
    const size_t row_bytes = (WK == WK_INT4_PACK) ? (size_t)(K >> 1) : (size_t)K;
    const int T = K >> 9, spr = K >> gshift;
    /* the grid's y dimension walks groups of MM activation rows */
    x += (size_t)blockIdx.y * MM * K + lane * 16;
    y += (size_t)blockIdx.y * MM * F;
    M = min(MM, M - (int)blockIdx.y * MM);
    const unsigned char* wrow[R];
    const __half* srow[R];
#pragma unroll
    for (int r = 0; r < R; r++) { /* rows beyond the last repeat it and are not stored */
        const int n = gemv_row_of<SW, R>(n0, r, F);
        wrow[r] = static_cast<const unsigned char*>(w) + (size_t)n * row_bytes + (size_t)lane * sizeof(tile_t);
        srow[r] = static_cast<const __half*>(scales) + (size_t)n * spr;
    }
    float acc[FM][R];
#pragma unroll
    for (int m = 0; m < FM; m++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[m][r] = 0.f;
    tile_t nxt[PD][R];
    __half gnx[PD][R];
    auto fetch = [&](int d, int i) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            nxt[d][r] = *reinterpret_cast<const tile_t*>(wrow[r] + (size_t)i * 32 * sizeof(tile_t));
            gnx[d][r] = WK != WK_INT8_CH ? srow[r][(i * 512 + lane * 16) >> gshift] : __half(0.f);
        }
    };
#pragma unroll
    for (int d = 0; d < PD; d++) fetch(d, min(d * NS + ns, T - 1));
    grid_wait();
    grid_release();
    const int rounds = (T + NS - 1) / NS;
    for (int rnd0 = 0; rnd0 < rounds; rnd0 += PD)
#pragma unroll
    for (int d = 0; d < PD; d++) {
        const int rnd = rnd0 + d, i = rnd * NS + ns;
        if (PD > 1 && rnd >= rounds) break;
        tile_t cur[R];
        float gs[R];
#pragma unroll
        for (int r = 0; r < R; r++) { cur[r] = nxt[d][r]; gs[r] = __half2float(gnx[d][r]); }
        if (i + PD * NS < T) fetch(d, i + PD * NS);
        if (NS == 1 || i < T) {
            f32x2 s[R][P];
            float so[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                so[r] = 0.f;
#pragma unroll
                for (int p = 0; p < P; p++) s[r][p] = 0ull;
            }
#pragma unroll
            for (int h = 0; h < 2; h++) { /* eight k of the lane's sixteen */
                uint4 xv[MM];
#pragma unroll
                for (int m = 0; m < MM; m++) xv[m] = *reinterpret_cast<const uint4*>(x + (size_t)min(m, M - 1) * K + i * 512 + h * 8);
                f32x2 wf[R][8];
#pragma unroll
                for (int r = 0; r < R; r++) BatchCodes<WK>::widen8(cur[r], h, wf[r]);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    auto word = [&](const uint4& v) { return (j >> 1) == 0 ? v.x : (j >> 1) == 1 ? v.y : (j >> 1) == 2 ? v.z : v.w; };
                    auto value = [&](int m) { return j & 1 ? bf_hi(word(xv[m])) : bf_lo(word(xv[m])); };
                    f32x2 xx[P];
#pragma unroll
                    for (int p = 0; p < P; p++) xx[p] = pack2(value(2 * p), value(2 * p + 1));
#pragma unroll
                    for (int r = 0; r < R; r++) {
#pragma unroll
                        for (int p = 0; p < P; p++) ffma2(s[r][p], wf[r][j], xx[p]);
                        if (ODD) {
                            float w0, w1;
                            unpack2(wf[r][j], w0, w1);
                            so[r] = __fmaf_rn(w0, value(MM - 1), so[r]);
                        }
                    }
                }
            }
            auto sum_of = [&](int r, int m) {
                if (ODD && m == MM - 1) return so[r];
                float lo, hi;
                unpack2(s[r][m >> 1], lo, hi);
                return m & 1 ? hi : lo;
            };
            if (NS == 1) {
#pragma unroll
                for (int r = 0; r < R; r++)
#pragma unroll
                    for (int m = 0; m < MM; m++)
                        acc[m][r] = WK == WK_INT8_CH ? acc[m][r] + sum_of(r, m) : __fmaf_rn(sum_of(r, m), gs[r], acc[m][r]);
            } else {
                float* at = part + ((rnd & 1) * NS + ns) * ((MM + 1) * R * 32) + lane;
#pragma unroll
                for (int r = 0; r < R; r++) {
#pragma unroll
                    for (int m = 0; m < MM; m++) at[(m * R + r) * 32] = sum_of(r, m);
                    if (WK != WK_INT8_CH) at[(MM * R + r) * 32] = gs[r];
                }
            }
        }
        if (NS > 1) { /* the round's tiles in ascending order, for this warp's activation rows */
            __syncthreads();
            const int live = min(NS, T - rnd * NS);
            for (int t = 0; t < live; t++) {
                const float* at = part + ((rnd & 1) * NS + t) * ((MM + 1) * R * 32) + lane;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float g = WK != WK_INT8_CH ? at[(MM * R + r) * 32] : 1.f;
#pragma unroll
                    for (int m = 0; m < FM; m++) {
                        const int mm = ns * FM + m;
                        if (FM * NS > MM && mm >= MM) continue;
                        const float v = at[(mm * R + r) * 32];
                        acc[m][r] = WK == WK_INT8_CH ? acc[m][r] + v : __fmaf_rn(v, g, acc[m][r]);
                    }
                }
            }
        }
    }
    /* the four rows' lane trees packed into one: lane 8 r ends with row r's sum */
    const int r = lane >> 3, n = n0 + r;
    const float rs = WK == WK_INT8_CH ? static_cast<const float*>(scales)[gemv_row_of<SW, R>(n0, r, F)] : 1.f;
#pragma unroll
    for (int m = 0; m < FM; m++) {
        const int mm = NS == 1 ? m : ns * FM + m;
        float a = warp_tree4<false>(acc[m][0], acc[m][1], acc[m][2], acc[m][3], lane);
        if (WK == WK_INT8_CH) a = __fmul_rn(a, rs);
        if (SW) a = gemv_swiglu(a, __shfl_down_sync(S2P_FULL_MASK, a, 16));
        if ((lane & 7) == 0 && mm < M && n < F && r < (SW ? R / 2 : R)) y[(size_t)mm * F + n] = f2bf(a);
    }
}

template <int WK, int MM, int NS, bool SW>
static cudaError_t run_gemv_batch(void* y, const void* x, const void* w, const void* scales, int M, int N, int K, int gshift, int early, cudaStream_t stream) {
    constexpr int rows = 4 * (4 / NS); /* weight rows of a CTA */
    return launch_early(early, k_gemv_batch<WK, MM, NS, SW>, dim3((unsigned)((N + rows - 1) / rows), (unsigned)((M + MM - 1) / MM)), 128, 0, stream,
                       (__nv_bfloat16*)y, (const __nv_bfloat16*)x, w, scales, M, N, K, gshift);
}
template <int WK, bool SW>
cudaError_t launch_gemv_batch(void* y, const void* x, const void* w, const void* scales, int M, int N, int K,
                              int gshift, int early, cudaStream_t stream) {
    /* As few groups of activation rows as eight a group allow (each converts every code once), of one size.  Four warps share
     * four rows where one warp each would leave a scheduler with less than 2.5, which do not hide each other's latencies, provided
     * that three quarters of the rounds' turns have a tile (a CTA waits for its slowest warp: at K = 2560, five tiles
     * in eight turns, sharing loses), or where less than every second scheduler would get a warp at all.  (A SwiGLU's pairs of rows
     * meet in a warp, which the tiles' sums of a shared row do not; the layers that have one have rows enough.) */
    const int groups = (M + 7) / 8;
    /* Seven rows of packed INT4 take the kernel of eight: the seventh row's scalar chains spill there (86.8 us for a layer's four
     * matrices, 85.4 padded).  Two groups of seven have two warps to a scheduler and are faster as they are (13 rows 142.4, padded
     * 145.3), and so is INT8 (7 rows 79.2, padded 80.7). */
    const int mm = WK == WK_INT4_PACK && M == 7 ? 8 : (M + groups - 1) / groups;
    const long long warps = (long long)((N + 3) / 4) * groups, sched = 4ll * device_sm_count();
    const int T = K >> 9, turns = (T + 3) / 4 * 4;
    const bool shared = !SW && (2 * warps < sched || (2 * warps < 5 * sched && 4 * T >= 3 * turns));
#define S2P_GB(MM)                                                                                            \
    do {                                                                                                      \
        if (shared) return run_gemv_batch<WK, MM, SW ? 1 : 4, SW>(y, x, w, scales, M, N, K, gshift, early, stream); \
        return run_gemv_batch<WK, MM, 1, SW>(y, x, w, scales, M, N, K, gshift, early, stream);                \
    } while (0)
    if (mm == 2) S2P_GB(2);
    if (mm == 3) S2P_GB(3);
    if (mm == 4) S2P_GB(4);
    if constexpr (!SW) {
        if (mm == 5) S2P_GB(5);
        if (mm == 6) S2P_GB(6);
        if (mm == 7) S2P_GB(7);
        S2P_GB(8);
    }
    return cudaErrorInvalidValue;
#undef S2P_GB
}

/* ---- one row, or two of a matrix of few rows ---------------------------------
 * The linear alone, as callers' own layers and one-row frames of a model on one GPU use it.
 *
 * What bounds it: instruction issue inside a wave of CTAs too short to be steady (19456 x 2560 INT4: issue slots 63 %, integer pipe
 * 57 %, fma pipe 43 % busy over the launch, DRAM 22 %).  So a few thousand warps have their weights under way at once.  A warp carries four rows (or six) as
 * packed chains (a register pair holds the same k of two rows), PD tiles at a time side by side, since every tile starts a chain of its
 * own; the next PD tiles' weights are in registers meanwhile.  Where there are too few rows for that NS = 4 warps share
 * four rows as in k_gemv_batch.
 * Measured, us (before: a CTA per SM with the tiles' sums in shared memory): INT4 6144 x 2560 10.2 -> 6.4, 2560 x 4096 8.2 -> 4.6,
 * 19456 x 2560 25.3 -> 12.9, 2560 x 9728 14.9 -> 9.7; INT8 8.5 -> 6.2, 6.8 -> 4.8, 18.9 -> 11.2, 10.7 -> 8.6. */
template <int WK, int MM, int R, int PD, int NS, bool SW>
__global__ void __launch_bounds__(128, MM == 2 ? 4 : R == 6 ? 6 : PD == 1 ? 8 : 4) k_gemv_row(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* __restrict__ x,
                                                     const void* __restrict__ w, const void* __restrict__ scales, int N, int K, int gshift) {
    typedef typename LaneTile<WK>::type tile_t;
    constexpr int P = R / 2;
    __shared__ float part[NS == 1 ? 1 : 2 * PD * NS * (MM + 1) * R * 32]; /* [round parity][tile of the round][sums, then scales][row][lane] */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int F = SW ? N >> 1 : N; /* outputs */
    const int n0 = (blockIdx.x * (4 / NS) + warp / NS) * (SW ? R / 2 : R), ns = warp % NS;
    if (n0 >= F) return; /* NS > 1: uniform over the CTA */
    const size_t row_bytes = (WK == WK_INT4_PACK) ? (size_t)(K >> 1) : (size_t)K;
    const int T = K >> 9, spr = K >> gshift;
    const unsigned char* wrow[R];
    const __half* srow[R];
#pragma unroll
    for (int r = 0; r < R; r++) { /* rows beyond the last repeat it and are not stored */
        const int n = gemv_row_of<SW, R>(n0, r, F);
        wrow[r] = static_cast<const unsigned char*>(w) + (size_t)n * row_bytes + (size_t)lane * sizeof(tile_t);
        srow[r] = static_cast<const __half*>(scales) + (size_t)n * spr;
    }
    tile_t nxt[PD][R];
    __half gnx[PD][R];
    auto tile_of = [&](int rnd, int d) { return (rnd * NS + ns) * PD + d; };
    auto fetch = [&](int rnd) {
#pragma unroll
        for (int d = 0; d < PD; d++) {
            const int i = min(tile_of(rnd, d), T - 1);
#pragma unroll
            for (int r = 0; r < R; r++) {
                nxt[d][r] = __ldcs(reinterpret_cast<const tile_t*>(wrow[r] + (size_t)i * 32 * sizeof(tile_t)));
                gnx[d][r] = WK != WK_INT8_CH ? srow[r][(i * 512 + lane * 16) >> gshift] : __half(0.f);
            }
        }
    };
    fetch(0);
    grid_wait();
    grid_release();
    float acc[MM][R];
#pragma unroll
    for (int m = 0; m < MM; m++)
#pragma unroll
        for (int r = 0; r < R; r++) acc[m][r] = 0.f;
    const int rounds = (T + NS * PD - 1) / (NS * PD);
    for (int rnd = 0; rnd < rounds; rnd++) {
        uint4 xv[PD][2][MM];
#pragma unroll
        for (int d = 0; d < PD; d++)
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int m = 0; m < MM; m++) xv[d][h][m] = *reinterpret_cast<const uint4*>(x + (size_t)m * K + min(tile_of(rnd, d), T - 1) * 512 + lane * 16 + h * 8);
        tile_t cur[PD][R];
        float gs[PD][R];
#pragma unroll
        for (int d = 0; d < PD; d++)
#pragma unroll
            for (int r = 0; r < R; r++) { cur[d][r] = nxt[d][r]; gs[d][r] = __half2float(gnx[d][r]); }
        if (rnd + 1 < rounds) fetch(rnd + 1);
        f32x2 s[PD][MM][P];
#pragma unroll
        for (int d = 0; d < PD; d++)
#pragma unroll
            for (int m = 0; m < MM; m++)
#pragma unroll
                for (int q = 0; q < P; q++) s[d][m][q] = 0ull;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            f32x2 wf[PD][P][8];
#pragma unroll
            for (int d = 0; d < PD; d++)
#pragma unroll
                for (int q = 0; q < P; q++) BatchCodes<WK>::widen8(cur[d][2 * q], cur[d][2 * q + 1], h, wf[d][q]);
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int d = 0; d < PD; d++) {
#pragma unroll
                    for (int m = 0; m < MM; m++) {
                        const uint4& v = xv[d][h][m];
                        const uint32_t u = (j >> 1) == 0 ? v.x : (j >> 1) == 1 ? v.y : (j >> 1) == 2 ? v.z : v.w;
                        const float xf = j & 1 ? bf_hi(u) : bf_lo(u);
                        const f32x2 xx = pack2(xf, xf);
#pragma unroll
                        for (int q = 0; q < P; q++) ffma2(s[d][m][q], wf[d][q][j], xx);
                    }
                }
        }
        auto fold = [&](int m, int r, float v, float g) { acc[m][r] = WK == WK_INT8_CH ? acc[m][r] + v : __fmaf_rn(v, g, acc[m][r]); };
#pragma unroll
        for (int d = 0; d < PD; d++) {
            if (tile_of(rnd, d) >= T) continue;
            float* at = part + (((rnd & 1) * NS + ns) * PD + d) * ((MM + 1) * R * 32) + lane;
#pragma unroll
            for (int m = 0; m < MM; m++) {
                float v[R];
#pragma unroll
                for (int q = 0; q < P; q++) unpack2(s[d][m][q], v[2 * q], v[2 * q + 1]);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (NS == 1) fold(m, r, v[r], gs[d][r]);
                    else at[(m * R + r) * 32] = v[r];
                }
            }
#pragma unroll
            for (int r = 0; r < R; r++)
                if (NS > 1) at[(MM * R + r) * 32] = gs[d][r];
        }
        if (NS > 1) { /* the round's tiles in ascending order; warp ns keeps row ns */
            __syncthreads();
            const int live = min(NS * PD, T - rnd * NS * PD);
            const float* at = part + (rnd & 1) * NS * PD * ((MM + 1) * R * 32) + ns * 32 + lane;
            for (int t = 0; t < live; t++, at += (MM + 1) * R * 32)
#pragma unroll
                for (int m = 0; m < MM; m++) fold(m, 0, at[m * R * 32], at[MM * R * 32]);
        }
    }
#pragma unroll
    for (int m = 0; m < MM; m++, y += F) {
    if (R != 4) { /* every lane has every sum */
#pragma unroll
        for (int r = 0; r < R; r++) {
            acc[m][r] = warp_tree_sum(acc[m][r]);
            if (WK == WK_INT8_CH) acc[m][r] = __fmul_rn(acc[m][r], static_cast<const float*>(scales)[gemv_row_of<SW, R>(n0, r, F)]);
        }
#pragma unroll
        for (int r = 0; r < (SW ? P : R); r++) {
            const float a = SW ? gemv_swiglu(acc[m][r], acc[m][r + (SW ? P : 0)]) : acc[m][r];
            if (lane == r && n0 + r < F) y[n0 + r] = f2bf(a);
        }
    } else if (NS == 1) {
        /* the four rows' lane trees packed into one: lane 8 r ends with row r's sum */
        const int r = lane >> 3, n = n0 + r;
        float a = warp_tree4<false>(acc[m][0], acc[m][1], acc[m][2], acc[m][3], lane);
        if (WK == WK_INT8_CH) a = __fmul_rn(a, static_cast<const float*>(scales)[gemv_row_of<SW, R>(n0, r, F)]);
        if (SW) a = gemv_swiglu(a, __shfl_down_sync(S2P_FULL_MASK, a, 16));
        if ((lane & 7) == 0 && n < F && r < (SW ? R / 2 : R)) y[n] = f2bf(a);
    } else {
        float a = warp_tree_sum(acc[m][0]);
        if (n0 + ns < N && lane == 0) {
            if (WK == WK_INT8_CH) a = __fmul_rn(a, static_cast<const float*>(scales)[n0 + ns]);
            y[n0 + ns] = f2bf(a);
        }
    }
    }
}

/* Four warps share four rows where one each would give a scheduler less than 1.5, if most of their turns have a tile
 * (2560 x 9728: 14.0 -> 9.7 us, 6144 x 2560 the other way round 6.4 -> 7.7). */
static bool gemv_row_shared(int N, int K) { return 2 * ((N + 3) / 4) < 3 * 4 * device_sm_count() && K > 4 * 512; }
template <int WK, bool SW>
static cudaError_t launch_gemv_row(void* y, const void* x, const void* w, const void* scales, int M, int N, int K, int gshift, int early, cudaStream_t stream) {
    /* From six warps per scheduler on a tile at a time with twice the warps resident hides more than two tiles side by side (19456
     * rows INT8 12.5 -> 11.2 us).  There packed INT4, whose tiles are half the loads, takes six rows a warp where the warps of four do
     * not fit the GPU at once (8 CTAs of 4 x 4 rows to an SM; of six 6 CTAs, so 144 rows instead of 128).  K = 2560, us with six /
     * four rows: one wave of either 14208 rows 12.2 / 10.9, 18944 13.3 / 11.6; beyond it 21312 13.3 / 13.9, 24576 13.9 / 15.0,
     * 28416 17.0 / 16.7, 38912 20.3 / 21.5, 155776 70.5 / 73.1.  (19456 rows: 13.4 / 13.1 in a chain of early launches, 12.9 / 13.5
     * launched the ordinary way.) */
    const int sms = device_sm_count();
    const bool shared = !SW && gemv_row_shared(N, K), many = (N + 3) / 4 >= 6 * 4 * sms;
    const bool six = WK == WK_INT4_PACK && N > 8 * 4 * 4 * sms;
    void (*kernel)(__nv_bfloat16*, const __nv_bfloat16*, const void*, const void*, int, int, int) =
        many ? k_gemv_row<WK, 1, 4, 1, 1, SW> : k_gemv_row<WK, 1, 4, 2, 1, SW>;
    if constexpr (WK == WK_INT4_PACK) {
        if (six) kernel = k_gemv_row<WK, 1, 6, 1, 1, SW>;
    }
    if constexpr (!SW) {
        if (shared) kernel = M == 2 ? k_gemv_row<WK, 2, 4, 2, 4, false> : k_gemv_row<WK, 1, 4, 2, 4, false>;
    }
    const int per_warp = six ? 6 : 4, warps = (N + per_warp - 1) / per_warp;
    return launch_early(early, kernel, dim3((unsigned)(shared ? warps : (warps + 3) / 4)), 128, 0, stream,
                       (__nv_bfloat16*)y, (const __nv_bfloat16*)x, w, scales, N, K, gshift);
}

int gshift_of(int G) {
    if (G < 16 || (G & (G - 1))) return -1;
    int s = 0;
    while ((1 << s) < G) s++;
    return s;
}

template <int WK, bool SW = false>
s2p_status gemv_entry(const char* what, void* y, const void* x, const void* w, const void* scales, int M, int N,
                      int K, int gshift, int early, cudaStream_t stream) {
    /* 16-byte loads of activations and weight tiles */
    if (((uintptr_t)x | (uintptr_t)w) & 15) return S2P_ERR_INVALID;
    cudaError_t ce;
    if (M == 1 || (M == 2 && !SW && gemv_row_shared(N, K))) { /* two rows where rows are few: 2560 x 4096 INT4 7.6 -> 5.9 us, x 9728 16.0 -> 13.1 */
        ce = launch_gemv_row<WK, SW>(y, x, w, scales, M, N, K, gshift, early, stream);
    } else {
        ce = launch_gemv_batch<WK, SW>(y, x, w, scales, M, N, K, gshift, early, stream);
    }
    if (ce != cudaSuccess) {
        fprintf(stderr, "[s2pro] %s launch (M=%d,N=%d,K=%d): %s\n", what, M, N, K, cudaGetErrorString(ce));
        return S2P_ERR_CUDA;
    }
    return S2P_OK;
}

}  // namespace s2p

using namespace s2p;

template <bool SW>
static s2p_status gemv_rows_of(const LinRef* lin, const void* x, void* y, int M, int early, cudaStream_t stream) {
    if (!lin || !lin->w || !lin->scales || !x || !y || M <= 0 || M > S2P_INT8_GEMV_MAX_M || lin->N <= 0 || lin->K <= 0 || lin->K % 512 ||
        (lin->kind != WK_INT8_CH && lin->K % (1 << lin->gshift)) || (SW && (lin->N % 2 || M > GEMV_SWIGLU_ROWS)))
        return S2P_ERR_INVALID;
    switch (lin->kind) {
    case WK_INT8_CH: return gemv_entry<WK_INT8_CH, SW>("int8 gemv", y, x, lin->w, lin->scales, M, lin->N, lin->K, 0, early, stream);
    case WK_INT8_GRP: return gemv_entry<WK_INT8_GRP, SW>("intq gemv", y, x, lin->w, lin->scales, M, lin->N, lin->K, lin->gshift, early, stream);
    case WK_INT4_PACK: return gemv_entry<WK_INT4_PACK, SW>("int4p gemv", y, x, lin->w, lin->scales, M, lin->N, lin->K, lin->gshift, early, stream);
    }
    return S2P_ERR_INVALID;
}
extern "C" int gemv_rows(const LinRef* lin, const void* x, void* y, int M, int early, cudaStream_t stream) { return gemv_rows_of<false>(lin, x, y, M, early, stream); }
extern "C" int gemv_rows_swiglu(const LinRef* lin, const void* x, void* h, int M, cudaStream_t stream) { return gemv_rows_of<true>(lin, x, h, M, 1, stream); }

extern "C" s2p_status s2p_int8_gemv(void* y_bf16, const void* x_bf16, const void* w_i8, const float* scales, int M,
                                    int N, int K, cudaStream_t stream) {
    if (!y_bf16 || !x_bf16 || !w_i8 || !scales || M <= 0 || N <= 0 || K <= 0) return S2P_ERR_INVALID;
    if (M > S2P_INT8_GEMV_MAX_M || K % 512 != 0) return S2P_ERR_INVALID;
    return gemv_entry<WK_INT8_CH>("int8 gemv", y_bf16, x_bf16, w_i8, scales, M, N, K, 0, 0, stream);
}

extern "C" s2p_status s2p_intq_gemv(void* y_bf16, const void* x_bf16, const void* w_i8, const void* scales_f16,
                                    int M, int N, int K, int G, cudaStream_t stream) {
    if (!y_bf16 || !x_bf16 || !w_i8 || !scales_f16 || M <= 0 || N <= 0 || K <= 0) return S2P_ERR_INVALID;
    const int gs = gshift_of(G);
    if (M > S2P_INT8_GEMV_MAX_M || K % 512 != 0 || gs < 0 || K % G != 0) return S2P_ERR_INVALID;
    return gemv_entry<WK_INT8_GRP>("intq gemv", y_bf16, x_bf16, w_i8, scales_f16, M, N, K, gs, 0, stream);
}

extern "C" s2p_status s2p_int4p_gemv(void* y_bf16, const void* x_bf16, const void* w_pack, const void* scales_f16,
                                     int M, int N, int K, int G, cudaStream_t stream) {
    if (!y_bf16 || !x_bf16 || !w_pack || !scales_f16 || M <= 0 || N <= 0 || K <= 0) return S2P_ERR_INVALID;
    const int gs = gshift_of(G);
    if (M > S2P_INT8_GEMV_MAX_M || K % 512 != 0 || gs < 0 || K % G != 0) return S2P_ERR_INVALID;
    return gemv_entry<WK_INT4_PACK>("int4p gemv", y_bf16, x_bf16, w_pack, scales_f16, M, N, K, gs, 0, stream);
}
