/* Stand-alone GEMV entry points of the C ABI (include/s2p_b200_abi.h):
 * s2p_int8_gemv, s2p_intq_gemv, s2p_int4p_gemv — the reference's
 * src/sched/int8_gemv.cu:964-986, :773-799, :836-902.
 *
 * Up to 16 rows run k_gemv_batch, where codes are widened once per tile for up to eight rows, or up to four
 * k_gemv_row where that is faster (gemv_row_grid), which also takes the norm in front.  Every
 * row of x is an independent product with one summation order (the reference's
 * batched GEMV computes rows independently too, int8_gemv.cu:77-91).  The stage
 * kernel of gemv.cuh (k_gemv_stage) serves the fused per-stage frame only.
 */
#include <stdio.h>
#include <type_traits>
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

template <int WK> cudaError_t gemv_row_setup_kind();

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
    if (e == cudaSuccess) e = gemv_row_setup_kind<WK_INT8_CH>();
    if (e == cudaSuccess) e = gemv_row_setup_kind<WK_INT8_GRP>();
    if (e == cudaSuccess) e = gemv_row_setup_kind<WK_INT4_PACK>();
    return e;
}

/* ---- exact-order small batch (1 <= M <= 16) -------------------------------
 * Lane l owns k = 512 i + 16 l .. +15 of every tile i; a warp carries four weight rows and MM activation
 * rows, 4 x MM independent chains.
 *
 * What bounds it: issue.  A chain step is one mixed fma (bf16 x bf16 + f32: the bits of fmaf), which costs 1.33 cycles of a scheduler because
 * its three operands come through two register ports; an activation needs no conversion, a code one per MM activation rows.  The
 * chains of a k advance side by side, because each waits for its own previous step, those of one activation one after another, so that its
 * register is read once for four of them.  Weights go from DRAM to registers a tile ahead; the activations of a tile are shared by the
 * SM's warps through L1.
 *
 * A matrix of few rows does not fill the GPU with warps of four rows, and a lone warp per scheduler waits on its own
 * latencies.  There NS = 4 warps share four rows and take tiles in turn; the tiles' chain results meet in shared memory and each warp
 * folds one of the weight rows for all activation rows, tiles ascending.  (Where a warp folded four weight rows for a share of the activation rows,
 * three of the four had nothing to do for one row and less than their share for five to seven: 2560 x 4096 INT8, us, 1 / 5 / 8 rows 5.6 / 7.9 / 8.6, so
 * 4.6 / 7.0 / 8.5.)
 * Measured, ticks of the full model, ms, before (two activation rows to a packed fma, each widened to f32; 168 registers) and now: 3 rows INT4
 * 4.25 -> 4.06, 8 rows INT4 8.12 -> 6.55, 16 rows INT8 12.80 -> 10.81.  CTAs to an SM: of the shared form 5 (8 rows 7.23 with 4); of the other 4,
 * where up to four rows are slower by 1 % than with 3.  16 rows of 19456 x 2560 INT4 take 46 us, 17 T fma/s of the 28 that a loop of mixed fma
 * alone reaches. */
/* A SwiGLU over stacked [gate | up] rows (SW): half of a warp's rows are of either half, so gate and up of an output meet in
 * the warp; both round to bf16 first, as where a kernel of its own follows the linear. */
template <bool SW, int R> __device__ __forceinline__ int gemv_row_of(int n0, int r, int F) {
    return SW ? min(n0 + r % (R / 2), F - 1) + r / (R / 2) * F : min(n0 + r, F - 1);
}
__device__ __forceinline__ float gemv_swiglu(float gate, float up_) {
    return swiglu_f32(bf16_round(gate), bf16_round(up_));
}
/* Codes of a lane as operands of the mixed fma (fma.rn.f32.bf16: bf16 x bf16 + f32, one rounding, the same bits as fmaf on the widened
 * values).  STEP codes are converted together; get(w, j) is the j-th of them.  An activation needs no conversion at all: the fma
 * takes either half of a register. */
__device__ __forceinline__ unsigned short half_of(uint32_t v, bool high) {
    unsigned short lo, hi;
    asm("mov.b32 {%0, %1}, %2;" : "=h"(lo), "=h"(hi) : "r"(v));
    return high ? hi : lo;
}
template <int WK> struct Codes;
template <> struct Codes<WK_INT8_CH> {
    static constexpr int STEP = 2, WORDS = 2;
    /* two bytes planted in the mantissa of 2^23, one packed subtraction: an f32 whose upper half is the code as bf16 */
    static __device__ __forceinline__ void widen(const uint4& a, int k, uint32_t (&w)[WORDS]) {
        const uint32_t u = s8x4_bias(k < 4 ? a.x : k < 8 ? a.y : k < 12 ? a.z : a.w);
        float lo, hi;
        unpack2(fadd2(pack2(__uint_as_float(prmt(u, 0x4B000000u, 0x7440u + (k & 3))), __uint_as_float(prmt(u, 0x4B000000u, 0x7441u + (k & 3)))),
                      pack2(-8388736.0f, -8388736.0f)), lo, hi);
        w[0] = __float_as_uint(lo); w[1] = __float_as_uint(hi);
    }
    static __device__ __forceinline__ unsigned short get(const uint32_t (&w)[WORDS], int j) { return half_of(w[j], true); }
};
template <> struct Codes<WK_INT8_GRP> : Codes<WK_INT8_CH> {};
/* INT8 where registers count: two codes to a register.  0x43bb with the byte's sign in the exponent's last bit: 128 + low seven bits
 * less 128 or 256 */
struct CodesInt8Packed {
    static constexpr int STEP = 4, WORDS = 2;
    static __device__ __forceinline__ void widen(const uint4& a, int k, uint32_t (&w)[WORDS]) {
        const uint32_t u = k < 4 ? a.x : k < 8 ? a.y : k < 12 ? a.z : a.w;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t t = prmt(u, 0x43434343u, j ? 0x4342u : 0x4140u);
            asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(w[j]) : "r"(lop3<0xC0>(t, 0x437F437Fu, 0u)), "r"(lop3<0xC0>(t, 0x43804380u, 0u)));
        }
    }
    static __device__ __forceinline__ unsigned short get(const uint32_t (&w)[WORDS], int j) { return half_of(w[j >> 1], j & 1); }
};
template <> struct Codes<WK_INT4_PACK> {
    static constexpr int STEP = 8, WORDS = 4;
    /* nibbles j and j + 4 as bf16 128 + 8 + code, one packed subtraction of 136 */
    static __device__ __forceinline__ void widen(const uint2& a, int k, uint32_t (&w)[WORDS]) {
        const uint32_t u = k < 8 ? a.x : a.y;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t v = lop3<LOP_AND_XOR>(u >> (4 * j), 0x000F000Fu, 0x43084308u);
            asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(w[j]) : "r"(v), "r"(0x43084308u));
        }
    }
    static __device__ __forceinline__ unsigned short get(const uint32_t (&w)[WORDS], int j) { return half_of(w[j & 3], j >= 4); }
};
/* the first step of a chain, which starts at zero */
__device__ __forceinline__ float fma_bf16_first(unsigned short w, unsigned short x) {
    float s;
    asm("fma.rn.f32.bf16 %0, %1, %2, 0f00000000;" : "=f"(s) : "h"(w), "h"(x));
    return s;
}
/* sixteen steps of the chains of R weight rows against MM activation rows: s[m][r] */
template <int WK> struct BatchCodes : Codes<WK> {};
template <> struct BatchCodes<WK_INT8_CH> : CodesInt8Packed {};
template <> struct BatchCodes<WK_INT8_GRP> : CodesInt8Packed {};
template <class C, int MM, int R, class T, class X>
__device__ __forceinline__ void lane_chains(const T (&t)[R], X x_word, float (&s)[MM][R]) {
#pragma unroll
    for (int k = 0; k < 16; k += C::STEP) {
        uint32_t w[R][C::WORDS];
#pragma unroll
        for (int r = 0; r < R; r++) C::widen(t[r], k, w[r]);
#pragma unroll
        for (int j = 0; j < C::STEP; j++)
#pragma unroll
            for (int m = 0; m < MM; m++) {
                const unsigned short xv = half_of(x_word(m, (k + j) >> 1), j & 1);
#pragma unroll
                for (int r = 0; r < R; r++) s[m][r] = k + j == 0 ? fma_bf16_first(C::get(w[r], j), xv) : fma_bf16(C::get(w[r], j), xv, s[m][r]);
            }
    }
}

/* Tiles of weights under way in a warp, CTAs to an SM.  One and two rows have registers for more of either; which hides more was measured for
 * each, us.  Alone: INT8 6144 x 2560 and 19456 x 2560, one row 6.0 and 11.3 (6 CTAs, a tile: 5.5 and 11.8; 8: 5.9 and 12.8), grouped INT8 6.1 and 12.3 (two
 * tiles 6.7 and 11.6), two rows 6.7 and 14.0 (5: 7.4 and 13.3; 8: 7.3 and 15.1); packed INT4 155776 x 2560, one row 53 (6 CTAs 61, two tiles 70).
 * Shared: 2560 x 4096 in a tick, one row INT8 3.5, INT4 2.6 (6 CTAs, a tile 4.3, 3.0; 4 CTAs 3.4, 4.1); two rows 4.6 (4 CTAs, two tiles 6.1; 7: 4.9). */
template <int WK, int MM, int NS> struct BatchPlan {
    static constexpr int CTAS = NS > 1 ? (MM == 2 ? 6 : 5) : MM == 1 ? (WK == WK_INT4_PACK ? 8 : WK == WK_INT8_CH ? 5 : 6) : MM == 2 ? 6 : MM <= 4 ? 3 : 4;
    static constexpr int PD = (MM == 1 && (NS > 1 || WK == WK_INT8_CH)) || (NS == 1 && MM > 2 && MM <= 4 && WK == WK_INT4_PACK) ? 2 : 1;
};
template <int WK, int MM, int NS, bool SW>
__global__ void __launch_bounds__(128, (BatchPlan<WK, MM, NS>::CTAS)) k_gemv_batch(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* x,
                                                       const void* __restrict__ w, const void* __restrict__ scales,
                                                       int M, int N, int K, int gshift, int settled) {
    typedef typename LaneTile<WK>::type tile_t;
    constexpr int R = 4; /* weight rows of a warp */
    constexpr int PD = BatchPlan<WK, MM, NS>::PD;
    constexpr int KEPT = NS == 1 ? R : 1; /* weight rows whose sums this warp keeps: all four, or the one of its number */
    static_assert(NS == 1 || NS == R, "a weight row each");
    typedef typename std::conditional<(MM <= 2), Codes<WK>, BatchCodes<WK>>::type C; /* few chains to a code leave registers for the cheaper conversion */
    __shared__ float part[NS == 1 ? 1 : 2 * NS * (MM + 1) * R * 32]; /* [round parity][tile of the round][m, then the scales][row][lane] */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int F = SW ? N >> 1 : N; /* outputs */
    const int n0 = (blockIdx.x * (4 / NS) + warp / NS) * (SW ? R / 2 : R), ns = warp % NS;
    if (n0 >= F) return; /* NS > 1: uniform over the CTA */
    if (!settled) grid_wait_for(w, scales); /* a caller's: see run_gemv_batch */
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
    float acc[MM][KEPT];
#pragma unroll
    for (int m = 0; m < MM; m++)
#pragma unroll
        for (int r = 0; r < KEPT; r++) acc[m][r] = 0.f;
    tile_t nxt[PD][R];
    __half gnx[PD][R];
    auto fetch = [&](int d, int i) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            const tile_t* at = reinterpret_cast<const tile_t*>(wrow[r] + (size_t)i * 32 * sizeof(tile_t));
            nxt[d][r] = MM <= 2 ? __ldcs(at) : *at;
            gnx[d][r] = WK != WK_INT8_CH ? srow[r][(i * 512 + lane * 16) >> gshift] : __half(0.f);
        }
    };
#pragma unroll
    for (int d = 0; d < PD; d++) fetch(d, min(d * NS + ns, T - 1));
    grid_wait();
    grid_release();
    unsigned x_row[MM];
#pragma unroll
    for (int m = 0; m < MM; m++) {
        x_row[m] = (unsigned)min(m, M - 1) * (unsigned)K;
        if (MM > 4) asm("" : "+r"(x_row[m])); /* stays in a register: left to the compiler, it is recomputed for every load (tick of 8 rows 6.70 -> 6.55 ms) */
    }
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
            float s[MM][R];
            uint4 xv[MM];
            const __nv_bfloat16* xt = x + i * 512;
            lane_chains<C, MM, R>(cur, [&](int m, int i2) {
                if ((i2 & 3) == 0) xv[m] = *reinterpret_cast<const uint4*>(xt + x_row[m] + i2 * 2);
                const uint4& v = xv[m];
                return (i2 & 3) == 0 ? v.x : (i2 & 3) == 1 ? v.y : (i2 & 3) == 2 ? v.z : v.w;
            }, s);
            if (NS == 1) {
#pragma unroll
                for (int r = 0; r < KEPT; r++)
#pragma unroll
                    for (int m = 0; m < MM; m++)
                        acc[m][r] = WK == WK_INT8_CH ? acc[m][r] + s[m][r] : __fmaf_rn(s[m][r], gs[r], acc[m][r]);
            } else {
                float* at = part + ((rnd & 1) * NS + ns) * ((MM + 1) * R * 32) + lane;
#pragma unroll
                for (int r = 0; r < R; r++) {
#pragma unroll
                    for (int m = 0; m < MM; m++) at[(m * R + r) * 32] = s[m][r];
                    if (WK != WK_INT8_CH) at[(MM * R + r) * 32] = gs[r];
                }
            }
        }
        if (NS > 1) { /* the round's tiles in ascending order, for this warp's weight row */
            __syncthreads();
            const int live = min(NS, T - rnd * NS);
            const float* at = part + (rnd & 1) * NS * ((MM + 1) * R * 32) + ns * 32 + lane;
#pragma unroll
            for (int t = 0; t < NS; t++, at += (MM + 1) * R * 32) {
                if (t >= live) break;
                const float g = WK != WK_INT8_CH ? at[MM * R * 32] : 1.f;
#pragma unroll
                for (int m = 0; m < MM; m++) acc[m][0] = WK == WK_INT8_CH ? acc[m][0] + at[m * R * 32] : __fmaf_rn(at[m * R * 32], g, acc[m][0]);
            }
        }
    }
    if (NS > 1) { /* the lane trees of four activation rows packed into one: lane 8 j ends with the sum of row m + j */
        const int n = n0 + ns;
        const float rs = WK == WK_INT8_CH ? static_cast<const float*>(scales)[min(n, N - 1)] : 1.f;
        auto of = [&](int m) { return m < MM ? acc[m < MM ? m : 0][0] : 0.f; };
#pragma unroll
        for (int m = 0; m < MM; m += 4) {
            float a = MM == 1 ? warp_tree_sum(of(m)) : warp_tree4<false>(of(m), of(m + 1), of(m + 2), of(m + 3), lane);
            if (WK == WK_INT8_CH) a = __fmul_rn(a, rs);
            const int mm = m + (lane >> 3);
            if ((lane & 7) == 0 && mm < M && n < N) y[(size_t)mm * N + n] = f2bf(a);
        }
        return;
    }
    /* the four rows' lane trees packed into one: lane 8 r ends with row r's sum */
    const int r = lane >> 3, n = n0 + r;
    const float rs = WK == WK_INT8_CH ? static_cast<const float*>(scales)[gemv_row_of<SW, R>(n0, r, F)] : 1.f;
#pragma unroll
    for (int m = 0; m < MM; m++) {
        float a = warp_tree4<false>(acc[m][0], acc[m][KEPT > 1 ? 1 : 0], acc[m][KEPT > 1 ? 2 : 0], acc[m][KEPT > 1 ? 3 : 0], lane);
        if (WK == WK_INT8_CH) a = __fmul_rn(a, rs);
        if (SW) a = gemv_swiglu(a, __shfl_down_sync(S2P_FULL_MASK, a, 16));
        if ((lane & 7) == 0 && m < M && n < F && r < (SW ? R / 2 : R)) y[(size_t)m * F + n] = f2bf(a);
    }
}

/* Launched to start while the kernel in front finishes, inside a tick and for callers alike (launch.cuh).  Inside a tick (`early`) the
 * weights are settled and asked for before the wait; a caller may have written them just before, so there the wait comes first and only
 * the launch itself overlaps: calls one after another of one row, INT4 19456 x 2560, 12.4 -> 10.4 us.  A lone call has nothing to overlap (24.5 us host to
 * host, 27 with the kernel before). */
template <int WK, int MM, int NS, bool SW>
static cudaError_t run_gemv_batch(void* y, const void* x, const void* w, const void* scales, int M, int N, int K, int gshift, int early, cudaStream_t stream) {
    constexpr int rows = 4 * (4 / NS); /* weight rows of a CTA */
    return launch_after(k_gemv_batch<WK, MM, NS, SW>, dim3((unsigned)((N + rows - 1) / rows), (unsigned)((M + MM - 1) / MM)), 128, 0, stream,
                       (__nv_bfloat16*)y, (const __nv_bfloat16*)x, w, scales, M, N, K, gshift, early);
}
/* Where four warps share four rows (a SwiGLU's pairs of rows meet in a warp, which the tiles' sums of a shared row do not; the layers that have one
 * have rows enough).  us, each warp its own rows / shared:
 *  - where the CTAs of the shared form all fit the GPU at once, up to 2960 rows of weights, 3552 for two rows (3552 x 2560 INT8, one row 4.6 / 5.4, two 5.7 / 4.4,
 *    three 5.2 / 6.8), but for one and two rows of a single tile (2560 x 512 1.9 / 2.2);
 *  - not where K has a tile or two, of which most of a CTA's warps get none: 4096 x 1024 INT8 one row 2.5 / 3.8, eight 4.6 / 5.7;
 *  - where one warp each would leave a scheduler with less than 2.5, which do not hide each other's latencies, provided that three quarters of the rounds'
 *    turns have a tile (a CTA waits for its slowest warp);
 *  - five to eight rows where the other form puts a third CTA on some SMs and the shared one takes two waves at most: 4864 x 2560 eight rows INT8 13.3 / 10.6, INT4
 *    12.9 / 10.1; 6144 x 2560, above, 13.4 / 13.5;
 *  - two and five to eight rows of a long K, up to what was measured: 6144 x 9728 INT8 two 20.7 / 17.2, eight 43.0 / 37.7, 9728 x 9728 grouped eight 70 / 51; 19456 x 9728
 *    two INT8 52 / 56. */
static bool gemv_batch_fits_shared(int M, int N) { return (long long)((N + 3) / 4) * ((M + 7) / 8) <= (M == 2 ? 6ll : 5ll) * device_sm_count(); }
static bool gemv_short(int M, int N, int K) { return gemv_batch_fits_shared(M, N) ? K == 512 && M <= 2 : K <= 2 * 512; }
static bool gemv_batch_shared(int M, int N, int K) {
    if (gemv_short(M, N, K)) return false;
    if (gemv_batch_fits_shared(M, N)) return true;
    const long long quads = (N + 3) / 4, warps = quads * ((M + 7) / 8), sms = device_sm_count();
    const int T = K >> 9, turns = (T + 3) / 4 * 4;
    if (warps < 10 * sms && 4 * T >= 3 * turns) return true;
    if (M > 4 && M <= 8 && T >= 5 && quads > 8 * sms && quads <= 10 * sms) return true;
    return (M == 2 || (M > 4 && M <= 8)) && T >= 8 && quads <= 17 * sms;
}
template <int WK, bool SW>
cudaError_t launch_gemv_batch(void* y, const void* x, const void* w, const void* scales, int M, int N, int K,
                              int gshift, int early, cudaStream_t stream) {
    /* as few groups of activation rows as eight a group allow (each converts every code once), of one size */
    const int groups = (M + 7) / 8;
    const int mm = (M + groups - 1) / groups;
    const bool shared = !SW && gemv_batch_shared(M, N, K);
#define S2P_GB(MM)                                                                                            \
    do {                                                                                                      \
        if (shared) return run_gemv_batch<WK, MM, SW ? 1 : 4, SW>(y, x, w, scales, M, N, K, gshift, early, stream); \
        return run_gemv_batch<WK, MM, 1, SW>(y, x, w, scales, M, N, K, gshift, early, stream);                \
    } while (0)
    if (mm == 1) S2P_GB(1);
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

/* ---- one and two rows; up to four of a matrix of middling size ---------------------
 * The linear alone or with the add and norm in front of it, as small ticks of a model on one GPU and callers' own layers use it.
 *
 * A CTA per SM owns a contiguous block of rows.  Its work is cut into units of four rows x one K tile, tile-major, and a warp takes a
 * contiguous run of units: its activations stay in registers, its weights have no order to wait for (all units are independent chains),
 * so D units of them are under way, the first before the kernel in front has ended.  Lane sums go to shared memory, [tile][unit][row][lane];
 * after one CTA barrier a warp folds four rows, tiles ascending, with scales that came to shared memory meanwhile.  So a matrix of 2560
 * rows occupies every warp whatever its K, and no warp of a large one has more than its share.
 *
 * What bounds it: about 3 us of fixed cost per launch (the wait, the first activations, barrier, fold), then the issue of conversions and
 * chains: 3.3 cycles per weight and scheduler for INT4, 4.1 for INT8 in a loop of nothing else, which is 4.5 us for 19456 x 2560 INT4
 * (its bytes take 4.3).  The mixed fma runs at the rate of fmaf and reads either half of its registers, so an activation costs nothing and
 * an INT4 pair one logic operation, one shift and one subtraction; packed f32 chains needed a conversion of either side.
 * Measured, us, launches of one matrix back to back in a graph (more of its copies than L2 holds), before (k packed over two rows of weights, warps of
 * four rows, four warps to a row's tiles where rows are few) and now; * is k_gemv_batch's now, see gemv_batch_faster:
 *                   6144 x 2560    2560 x 4096     19456 x 2560     2560 x 9728
 *   tick    INT4 1   7.4 -> 4.0     3.4 -> 2.6 *   13.1 -> 9.3      8.7 -> 5.4 *
 *           INT4 2   7.3 -> 5.8     4.8 -> 4.6 *   15.5 -> 13.4    11.9 -> 8.0
 *           INT8 1   6.4 -> 5.0     3.8 -> 3.5 *   10.4 -> 11.5     8.7 -> 7.0
 *           INT8 2   8.1 -> 6.8     5.5 -> 4.7 *   14.1 -> 15.1    12.5 -> 9.0
 *   caller  INT4 1   6.2 -> 5.0     4.8 -> 3.5 *   12.8 -> 10.6     9.9 -> 6.4 *
 *           INT4 2   6.9 -> 6.2 *   6.0 -> 5.3 *   15.7 -> 12.9 *  13.2 -> 9.0
 *           INT8 1   6.2 -> 6.0 *   4.8 -> 4.7 *   11.4 -> 11.5 *   8.7 -> 8.3
 *           INT8 2   7.1 -> 6.7 *   6.5 -> 5.3 *   14.7 -> 13.9 *  12.2 -> 10.2
 * (In a tick the two wide matrices carry the norm, which the launch that it saves pays for; 19456 x 2560 INT8 alone is the one entry that lost.
 * 155776 x 2560, a caller's one row: INT8 61.7 -> 63.2, INT4 72 -> 53.)
 * At 64 registers, two CTAs to an SM, the frame took 3.67 ms instead of 2.68; 24 warps of 80 registers and other depths were within 1 %.
 *
 * NORM: the residual add and the norm in front of the linear, taken by every CTA while its first weights are on their way, instead of a
 * launch of k_norm_row: frame of one row 2.67 -> 2.52 ms INT4, 2.97 -> 2.79 INT8. */
template <int WK, int MM> struct RowPlan {
    static constexpr int WARPS = 16, R = 4;
    static constexpr int D = WK == WK_INT4_PACK ? 4 : MM <= 2 ? 3 : 2; /* units of weights under way in a warp */
    static constexpr bool XN = MM <= 2;                                  /* the next tile's activations too */
    static constexpr size_t LIMIT = 200 * 1024;
    static constexpr int NORM_K = 8 * WARPS * 32; /* longest activation whose norm the kernel takes itself: a vector of eight per thread */
    static size_t norm_smem(int K) { return (size_t)MM * (K * 2 + 257 * sizeof(float)); }
    static size_t smem(int outputs, int K, int gshift, bool sw) {
        const int rows_a = sw ? 2 : 4, units = (outputs + rows_a - 1) / rows_a, T = K / 512;
        return (size_t)MM * units * R * T * 32 * sizeof(float) + (WK == WK_INT8_CH ? 0 : ((size_t)units * R * (K >> gshift) * 2 + 15) & ~(size_t)15);
    }
    /* CTAs, one per SM; 0 where the sums do not fit its shared memory (in several turns 155776 x 2560 took 68 us for one row of INT4 and
     * 106 for two, k_gemv_batch 53 and 77), or offsets would not fit 32 bits */
    static int grid(int F, int K, int gshift, bool sw, int sms) {
        const int g = sms < F ? sms : F;
        return smem((F + g - 1) / g, K, gshift, sw) > LIMIT || (size_t)F * (sw ? 2 : 1) * K > 0xF0000000ull ? 0 : g;
    }
};
template <int WK, int MM, bool SW, bool NORM>
__global__ void __launch_bounds__(RowPlan<WK, MM>::WARPS * 32, 1) k_gemv_row(__nv_bfloat16* __restrict__ y, const __nv_bfloat16* x, NormIn nm,
                                                                            const void* __restrict__ w, const void* __restrict__ scales, int N, int K, int gshift, int settled) {
    typedef typename LaneTile<WK>::type tile_t;
    constexpr int R = 4, RA = SW ? 2 : 4, W = RowPlan<WK, MM>::WARPS, D = RowPlan<WK, MM>::D; /* RA: rows of a unit that follow one another */
    constexpr bool XN = RowPlan<WK, MM>::XN;
    extern __shared__ __align__(16) unsigned char smem[];
    if (!settled) grid_wait_for(w, scales); /* see run_gemv_batch */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int T = K >> 9, spr = K >> gshift;
    const unsigned row_bytes = WK == WK_INT4_PACK ? (unsigned)(K >> 1) : (unsigned)K;
    const int F = SW ? N >> 1 : N; /* outputs */
    const int o0 = (int)((long long)F * blockIdx.x / gridDim.x), outs = (int)((long long)F * (blockIdx.x + 1) / gridDim.x) - o0;
    const int per_tile = (outs + RA - 1) / RA, units = per_tile * T;
    float* sums = reinterpret_cast<float*>(smem);                          /* [m][tile][unit of the tile][row][lane] */
    __half* ssc = reinterpret_cast<__half*>(sums + (size_t)MM * units * R * 32); /* [row (SW: gates, then ups)][spr] */
    if (WK != WK_INT8_CH) {
#pragma unroll
        for (int part = 0; part < R / RA; part++) {
            const __half* src = static_cast<const __half*>(scales) + (size_t)(o0 + part * F) * spr;
            __half* dst = ssc + part * per_tile * RA * spr;
            const int n = outs * spr;
            if ((((uintptr_t)src | (uintptr_t)dst | (unsigned)(n * 2)) & 15) == 0) {
                for (int c = threadIdx.x * 8; c < n; c += W * 32 * 8)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + c)), "l"(src + c) : "memory");
            } else {
                for (int c = threadIdx.x; c < n; c += W * 32) dst[c] = src[c];
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int u0 = (int)((long long)units * warp / W);
    const int n_units = (int)((long long)units * (warp + 1) / W) - u0;
    int t = u0 / per_tile, ru = u0 - t * per_tile;
    /* 32-bit offsets from the block's first row */
    const unsigned char* wb = static_cast<const unsigned char*>(w) + (size_t)o0 * row_bytes;
    constexpr unsigned TILE = 32 * sizeof(tile_t);
    unsigned at_row[R];
#pragma unroll
    for (int r = 0; r < R; r++) at_row[r] = (r % RA) * row_bytes + (r / RA) * F * row_bytes;
    int lu = ru, left = n_units; /* where the loads are */
    unsigned at_tile = t * TILE + lane * (unsigned)sizeof(tile_t), at = at_tile + ru * RA * row_bytes;
    tile_t q[D][R];
    auto load = [&](int d) {
        if (left <= 0) return;
        left--;
        if ((lu + 1) * RA <= outs) {
#pragma unroll
            for (int r = 0; r < R; r++) q[d][r] = __ldcs(reinterpret_cast<const tile_t*>(wb + (at + at_row[r])));
        } else { /* rows beyond the last repeat it and are not stored */
            const int last = outs - 1 - lu * RA;
#pragma unroll
            for (int r = 0; r < R; r++)
                q[d][r] = __ldcs(reinterpret_cast<const tile_t*>(wb + (at + min(r % RA, last) * row_bytes + (r / RA) * F * row_bytes)));
        }
        at += RA * row_bytes;
        if (++lu == per_tile) { lu = 0; at = at_tile += TILE; }
    };
#pragma unroll
    for (int d = 0; d < D; d++) load(d);
    __nv_bfloat16* xs = reinterpret_cast<__nv_bfloat16*>(smem + nm.at); /* NORM: the normalised rows */
    uint4 gain = make_uint4(0, 0, 0, 0);
    const int v = threadIdx.x, nv = K >> 3;
    if (NORM && v < nv) gain = reinterpret_cast<const uint4*>(nm.gain)[v];
    grid_wait();
    grid_release();
    if (NORM) { /* k_norm_row's pairs and roundings (prims.cu), in every CTA; the first one keeps the sum */
        static_assert(!NORM || MM <= 2, "256 threads a row");
        float* red = reinterpret_cast<float*>(xs + MM * K);
        uint4 q[MM];
#pragma unroll
        for (int m = 0; m < MM; m++) {
            if (v >= nv) continue;
            q[m] = reinterpret_cast<const uint4*>(nm.src + (size_t)m * K)[v];
            const uint4 a = reinterpret_cast<const uint4*>(nm.add + (size_t)m * K)[v];
            q[m] = make_uint4(add_bf16x2(q[m].x, a.x), add_bf16x2(q[m].y, a.y), add_bf16x2(q[m].z, a.z), add_bf16x2(q[m].w, a.w));
            reinterpret_cast<uint4*>(xs + (size_t)m * K)[v] = q[m];
            if (blockIdx.x == 0) reinterpret_cast<uint4*>(nm.x_out + (size_t)m * K)[v] = q[m];
        }
        __syncthreads();
        const int mine = threadIdx.x >> 8, i0 = threadIdx.x & 255;
        float* r = red + mine * 257;
        if (mine < MM) {
            float ss = 0.f;
            for (int i = i0; i < K; i += 256) {
                const float e = bf2f(xs[(size_t)mine * K + i]);
                ss = __fmaf_rn(e, e, ss);
            }
            r[i0] = ss;
        }
        __syncthreads();
        if (mine < MM && i0 < 32) {
            const float tot = tree256_of(r, i0);
            if (i0 == 0) r[256] = tot;
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < MM; m++)
            if (v < nv) reinterpret_cast<uint4*>(xs + (size_t)m * K)[v] = norm_vec8(q[m], gain, rsqrtf(__fdiv_rn(red[m * 257 + 256], (float)K) + nm.eps));
        __syncthreads();
    }
    uint4 xv[MM][2], xn[MM][2];
    const __nv_bfloat16* xp = (NORM ? xs : x) + (size_t)min(t, T - 1) * 512 + lane * 16;
    auto load_x = [&](uint4 (&v)[MM][2]) {
#pragma unroll
        for (int m = 0; m < MM; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) v[m][h] = *reinterpret_cast<const uint4*>(xp + (size_t)m * K + h * 8);
    };
    load_x(xv);
    if (XN) {
        if (t + 1 < T) xp += 512;
        load_x(xn);
    }
    float* sp = sums + u0 * (R * 32) + lane;
    const int plane = units * R * 32;
#pragma unroll 1
    for (int n = n_units; n > 0; n -= D)
#pragma unroll
        for (int d = 0; d < D; d++) {
            if (d && d >= n) break;
            float s[MM][R];
            lane_chains<Codes<WK>, MM, R>(q[d], [&](int m, int i2) {
                const uint4& v = xv[m][i2 >> 2];
                return (i2 & 3) == 0 ? v.x : (i2 & 3) == 1 ? v.y : (i2 & 3) == 2 ? v.z : v.w;
            }, s);
            load(d);
#pragma unroll
            for (int m = 0; m < MM; m++)
#pragma unroll
                for (int r = 0; r < R; r++) sp[m * plane + r * 32] = s[m][r];
            sp += R * 32;
            if (++ru == per_tile) {
                ru = 0; t++;
                if (XN) {
#pragma unroll
                    for (int m = 0; m < MM; m++) { xv[m][0] = xn[m][0]; xv[m][1] = xn[m][1]; }
                }
                if (t + (XN ? 1 : 0) < T) {
                    xp += 512;
                    if (XN) load_x(xn); else load_x(xv);
                }
            }
        }
    if (WK != WK_INT8_CH) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int g = warp; g < per_tile * MM; g += W) {
        const int m = MM == 1 ? 0 : g / per_tile, u = MM == 1 ? g : g - m * per_tile;
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0.f;
        const float* at = sums + (size_t)(m * units + u) * (R * 32) + lane;
#pragma unroll 2
        for (int i = 0; i < T; i++, at += per_tile * (R * 32)) {
            const __half* sc = ssc + u * RA * spr + ((i * 512 + lane * 16) >> gshift); /* a group may be longer than a tile */
#pragma unroll
            for (int r = 0; r < R; r++) {
                const float v = at[r * 32];
                acc[r] = WK == WK_INT8_CH ? acc[r] + v : __fmaf_rn(v, __half2float(sc[(r % RA) * spr + r / RA * per_tile * RA * spr]), acc[r]);
            }
        }
        /* the four rows' lane trees packed into one: lane 8 r ends with row r's sum */
        const int r = lane >> 3, o = u * RA + r % RA;
        float a = warp_tree4<false>(acc[0], acc[1], acc[2], acc[3], lane);
        if (WK == WK_INT8_CH) a = __fmul_rn(a, static_cast<const float*>(scales)[o0 + min(o, outs - 1) + r / RA * F]);
        if (SW) a = gemv_swiglu(a, __shfl_down_sync(S2P_FULL_MASK, a, 16));
        if ((lane & 7) == 0 && r < RA && o < outs) y[(size_t)m * F + o0 + o] = f2bf(a);
    }
}
template <int WK, int MM, bool SW, bool NORM>
static cudaError_t gemv_row_setup() {
    static int done_mask = 0; /* bit per device ordinal */
    int dev = 0;
    cudaGetDevice(&dev);
    if (done_mask & (1 << (dev & 31))) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(k_gemv_row<WK, MM, SW, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(RowPlan<WK, MM>::LIMIT + (NORM ? RowPlan<WK, MM>::norm_smem(RowPlan<WK, MM>::NORM_K) : 0)));
    if (e == cudaSuccess) done_mask |= 1 << (dev & 31);
    return e;
}
template <int WK> cudaError_t gemv_row_setup_kind() {
    const cudaError_t e[] = {gemv_row_setup<WK, 1, false, false>(), gemv_row_setup<WK, 2, false, false>(), gemv_row_setup<WK, 3, false, false>(),
                             gemv_row_setup<WK, 4, false, false>(), gemv_row_setup<WK, 1, true, false>(), gemv_row_setup<WK, 2, true, false>(),
                             gemv_row_setup<WK, 3, true, false>(), gemv_row_setup<WK, 4, true, false>(), gemv_row_setup<WK, 1, false, true>(),
                             gemv_row_setup<WK, 2, false, true>(), gemv_row_setup<WK, 1, true, true>(), gemv_row_setup<WK, 2, true, true>()};
    for (cudaError_t c : e)
        if (c != cudaSuccess) return c;
    return cudaSuccess;
}
template <int WK, int MM, bool SW, bool NORM = false>
static cudaError_t run_gemv_row(int grid, void* y, const void* x, const NormIn* norm, const void* w, const void* scales, int N, int K, int gshift, int early, cudaStream_t stream) {
    typedef RowPlan<WK, MM> Plan;
    const cudaError_t e = gemv_row_setup<WK, MM, SW, NORM>();
    if (e != cudaSuccess) return e;
    const int F = SW ? N >> 1 : N;
    size_t smem = Plan::smem((F + grid - 1) / grid, K, gshift, SW);
    NormIn nm = {};
    if (NORM) {
        nm = *norm;
        nm.at = (unsigned)smem;
        smem += Plan::norm_smem(K);
    }
    return launch_after(k_gemv_row<WK, MM, SW, NORM>, dim3((unsigned)grid), Plan::WARPS * 32, smem, stream,
                        (__nv_bfloat16*)y, (const __nv_bfloat16*)x, nm, w, scales, N, K, gshift, early);
}
/* the CTAs of k_gemv_row for M rows, 0 where it cannot take them */
template <int WK, bool SW> static int gemv_row_grid(int M, int N, int K, int gshift) {
    const int F = SW ? N >> 1 : N, sms = device_sm_count();
    switch (M) {
    case 1: return RowPlan<WK, 1>::grid(F, K, gshift, SW, sms);
    case 2: return RowPlan<WK, 2>::grid(F, K, gshift, SW, sms);
    case 3: return RowPlan<WK, 3>::grid(F, K, gshift, SW, sms);
    case 4: return RowPlan<WK, 4>::grid(F, K, gshift, SW, sms);
    }
    return 0;
}
/* Whether k_gemv_batch is the faster of the two for a linear without the norm.  Both sides in us, k_gemv_row first; callers' calls, a tick's in brackets:
 *  - few rows of weights, shared by a CTA's warps: 2560 x 4096, one row INT8 5.6 / 4.7 (4.4 / 3.5), grouped 5.6 / 4.8 (4.4 / 3.5), INT4 4.5 / 3.5 (3.7 / 2.6),
 *    two 6.9 / 5.3, 6.8 / 5.5, 5.7 / 5.3, four INT4 7.6 / 5.5.  But each further round of a CTA's tiles costs two barriers, which few chains do not make
 *    up for: one row INT8 x 6144 6.4 / 5.9 (5.2 / 5.3), x 9728 8.3 / 8.1 (7.0 / 7.5); two rows x 9728 INT4 9.0 / 10.2, four INT8 13.1 / 13.6.  One, three and four
 *    rows of INT4 and four of grouped INT8 keep the gain at any length (x 9728 7.0 / 6.4, 10.8 / 9.4, 15.4 / 11.3; 16.7 / 13.7);
 *  - from two warps of four rows to a scheduler, three and four rows (4097 x 2560, three rows INT4 5.9 / 6.3 (5.1 / 5.8); 6144 x 2560 7.4 / 6.5).  One and two rows only
 *    outside a tick: a caller's weights are not asked for before the wait, and more, smaller CTAs have more of them under way then (6144 x 2560 INT8 two
 *    rows 8.1 / 6.7 (7.0 / 6.4), 19456 x 2560 one row 13.1 / 11.5 (11.5 / 11.0), two 16.7 / 13.9 (15.3 / 13.7)).  One row of packed INT4 has too few
 *    instructions for that to matter (5.0 / 5.3, 10.6 / 10.5).  A long K turns both: one row is back with k_gemv_row while an SM has few enough rows
 *    (6144 x 9728 INT8 13.7 / 17.1, grouped 14.1 / 18.2), two rows INT8 are with the shared form in a tick too (6144 x 6144 12.1 / 11.3);
 *  - where some SMs get a fourth CTA of two rows and most do not, from 7104 to 9472 rows of weights: 7168 x 2560 INT4 7.6 / 8.6, 8192 8.0 / 9.1, grouped 8.7 / 9.2 and 9.1 / 9.6
 *    (INT8 per channel 8.4 / 8.3, 9.0 / 9.2);
 *  - a tile or two of K, whatever the rows: nothing to spread over an SM's warps (4096 x 512 INT8 two rows 3.1 / 2.0, 4096 x 1024 one row 3.3 / 2.5);
 *  - three rows of INT8 per channel, whose chains the batch kernel holds with the fewest registers (4096 x 2560 6.7 / 5.4 (5.6 / 5.1), 4096 x 4096 9.0 / 7.4). */
template <int WK, bool SW> static bool gemv_batch_faster(int M, int N, int K, int early) {
    if (M > 4 || (!SW && gemv_short(M, N, K))) return true;
    if (!SW && gemv_batch_fits_shared(M, N)) return K <= 12 * 512 || (WK == WK_INT4_PACK ? M != 2 : WK == WK_INT8_GRP && M == 4);
    if (!SW && WK == WK_INT8_CH && M == 3 && K <= 12 * 512) return true;
    const int quads = (N + 3) / 4, sms = device_sm_count();
    const bool many = quads >= 2 * 4 * sms, deep = !SW && K >= 8 * 512;
    if (!many || M > 2) return many;
    if (deep && M == 1 && quads <= 12 * sms) return false;
    if (!SW && !deep && M == 2 && WK != WK_INT8_CH && quads > 12 * sms && quads <= 16 * sms) return false;
    return early ? deep && M == 2 && WK != WK_INT4_PACK : M == 2 || WK != WK_INT4_PACK;
}
template <int WK, bool SW>
static cudaError_t launch_gemv_row(int grid, void* y, const void* x, const void* w, const void* scales, int M, int N, int K, int gshift, int early, cudaStream_t stream) {
    switch (M) {
    case 1: return run_gemv_row<WK, 1, SW>(grid, y, x, nullptr, w, scales, N, K, gshift, early, stream);
    case 2: return run_gemv_row<WK, 2, SW>(grid, y, x, nullptr, w, scales, N, K, gshift, early, stream);
    case 3: return run_gemv_row<WK, 3, SW>(grid, y, x, nullptr, w, scales, N, K, gshift, early, stream);
    case 4: return run_gemv_row<WK, 4, SW>(grid, y, x, nullptr, w, scales, N, K, gshift, early, stream);
    }
    return cudaErrorInvalidValue;
}

int gshift_of(int G) {
    if (G < 16 || (G & (G - 1))) return -1;
    int s = 0;
    while ((1 << s) < G) s++;
    return s;
}

/* the same with the add and the norm in front of it in the kernel, one or two rows */
template <int WK, bool SW> static cudaError_t launch_gemv_row_norm(const LinRef* lin, const NormIn* norm, void* y, int M, cudaStream_t stream) {
    const int grid = gemv_row_grid<WK, SW>(M, lin->N, lin->K, lin->gshift);
    if (!grid || M > 2 || lin->K > RowPlan<WK, 1>::NORM_K) return cudaErrorInvalidValue;
    return M == 1 ? run_gemv_row<WK, 1, SW, true>(grid, y, nullptr, norm, lin->w, lin->scales, lin->N, lin->K, lin->gshift, 1, stream)
                  : run_gemv_row<WK, 2, SW, true>(grid, y, nullptr, norm, lin->w, lin->scales, lin->N, lin->K, lin->gshift, 1, stream);
}

template <int WK, bool SW = false>
s2p_status gemv_entry(const char* what, void* y, const void* x, const void* w, const void* scales, int M, int N,
                      int K, int gshift, int early, cudaStream_t stream) {
    /* 16-byte loads of activations and weight tiles */
    if (((uintptr_t)x | (uintptr_t)w) & 15) return S2P_ERR_INVALID;
    cudaError_t ce;
    const int grid = gemv_batch_faster<WK, SW>(M, N, K, early) ? 0 : gemv_row_grid<WK, SW>(M, N, K, gshift);
    if (grid) {
        ce = launch_gemv_row<WK, SW>(grid, y, x, w, scales, M, N, K, gshift, early, stream);
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
extern "C" int gemv_norm_serves(const LinRef* lin, int swiglu, int M) {
    if (!lin || M < 1 || M > 2 || lin->K % 512 || lin->K > RowPlan<WK_INT8_CH, 1>::NORM_K) return 0;
    switch (lin->kind) {
    case WK_INT8_CH: return (swiglu ? gemv_row_grid<WK_INT8_CH, true>(M, lin->N, lin->K, 0) : gemv_row_grid<WK_INT8_CH, false>(M, lin->N, lin->K, 0)) != 0;
    case WK_INT8_GRP: return (swiglu ? gemv_row_grid<WK_INT8_GRP, true>(M, lin->N, lin->K, lin->gshift) : gemv_row_grid<WK_INT8_GRP, false>(M, lin->N, lin->K, lin->gshift)) != 0;
    case WK_INT4_PACK: return (swiglu ? gemv_row_grid<WK_INT4_PACK, true>(M, lin->N, lin->K, lin->gshift) : gemv_row_grid<WK_INT4_PACK, false>(M, lin->N, lin->K, lin->gshift)) != 0;
    }
    return 0;
}
extern "C" cudaError_t gemv_rows_norm(const LinRef* lin, const NormIn* norm, void* y, int swiglu, int M, cudaStream_t stream) {
    if (!gemv_norm_serves(lin, swiglu, M) || !norm || norm->src == norm->x_out) return cudaErrorInvalidValue;
    switch (lin->kind) {
    case WK_INT8_CH: return swiglu ? launch_gemv_row_norm<WK_INT8_CH, true>(lin, norm, y, M, stream) : launch_gemv_row_norm<WK_INT8_CH, false>(lin, norm, y, M, stream);
    case WK_INT8_GRP: return swiglu ? launch_gemv_row_norm<WK_INT8_GRP, true>(lin, norm, y, M, stream) : launch_gemv_row_norm<WK_INT8_GRP, false>(lin, norm, y, M, stream);
    default: return swiglu ? launch_gemv_row_norm<WK_INT4_PACK, true>(lin, norm, y, M, stream) : launch_gemv_row_norm<WK_INT4_PACK, false>(lin, norm, y, M, stream);
    }
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
