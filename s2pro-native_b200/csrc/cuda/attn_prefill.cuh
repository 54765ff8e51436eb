/* Single-pass causal attention for a prompt slice: 4 x QT consecutive query rows of ONE session per CTA.
 *
 * Arithmetic per (row, head): that of the single-row kernel in prims.cu (the reference's k_attention /
 * k_attention8, src/slowar/kernels.cu:234-309 and :625-728) - tiles of 128 cached positions, per position one
 * 128-term fma chain against the pre-scaled query (INT8 cache: four 32-term chains folded with the f16 group scale),
 * tile max and sum by 128-wide halving trees, l = fma(l, corr, tile_sum), acc *= corr, then one fma per position in
 * ascending order - so the outputs are the same bits.
 *
 * What bounds it: fp32 fma issue (the chains are fp32 by contract, 256 fma per (row, head, position)).  So the two
 * products are laid out as register-tiled fp32 matrix products.  The queries of a CTA are its rows x the four heads of
 * one kv head, 2 QT NW of them; consumer warp w owns queries 2 QT w .. +2 QT - 1 in BOTH phases, a thread QT of them times
 * eight positions (score phase) or eight dimensions (value phase).  Keys and values of a tile are widened to f32 once per CTA
 * into shared memory, keys transposed, and every chain advances on the packed fma (fma.rn.f32x2, two independent
 * roundings; it holds the fma pipe for two cycles, so shared reads and the broadcast of the query or weight operand issue
 * beside it).  A warp sees all 128 positions of its queries, so max, sum and weights never leave it (the sum tree's pairs: 64
 * in the thread, 32..4 over four lane bits, 2 and 1 in the thread).  Four producer warps widen the tiles ahead of the
 * consumers, which therefore meet no CTA barrier.
 *
 * Measured (INT8 cache, 2048 rows after 6052 positions, 119 G fma): 12.6 ms with four rows per 512-thread CTA, keys converted
 * by every reader and trees over shared memory; 10.6 ms register-tiled 2 x 8; 6.5 ms 4 x 8; 5.7 ms with 12 warps instead of
 * 8; 5.4 ms = 22 T fma/s with the producers, 0.6 of the fp32 peak.  Counters of that launch: fma pipe 77 % of its cycles
 * busy (the value phase pays one multiplication per weight and group scale beside its fma), issue slots 59 %, the shared-memory
 * data path 59 %.  77 rows after 1024 positions (104 CTAs, nine tiles in sequence): 50 %, 47 % and 50 %.  8 x 8 tiles measured
 * the same per row with worse waves; 2 queries x 16 dimensions per thread in the value phase slower (more shared reads).
 */
#pragma once
#include <math.h>
#include "common.cuh"
#include "headops.cuh"
#include "ops.h"
#include "pipe.cuh"
#include "packed.cuh"
#include "launch.cuh"

namespace s2p {

constexpr int ATTN_PREFILL_PRODUCERS = 128; /* threads that widen the tiles */

template <bool KV8, int QT, int NW, bool APART> struct AttnPrefillSmem {
    static constexpr int M = 2 * QT * NW, RB = M / 4;   /* queries and rows of a CTA */
    alignas(16) float q[128][M];                        /* pre-scaled queries, dimension-major */
    alignas(16) float k[128][128];                      /* key tile, dimension-major */
    /* value tile; the 16-byte chunk c of a row (dimensions 4c..) at slot (c & 1) * 16 + (c >> 1), which makes a thread's
     * eight dimensions two conflict-free reads */
    alignas(16) float v[128][128];
    /* soft-max weights, private to a warp: [half of its queries][query][position], the second half with position bit 4
     * flipped so that the two halves of a warp read different banks */
    alignas(16) float p[NW][2][QT][128];
    alignas(16) __half ksc[KV8 ? 4 : 1][128], vsc[KV8 ? 4 : 1][128]; /* group scales of the tile */
    alignas(16) float corr[APART ? NW : 1][2][QT], l[APART ? NW : 1][2][QT]; /* APART, beside p: the factor of the sums so far, the weights' total */
    int last[RB];                                       /* positions a row sees, 0 beyond the slice */
    alignas(8) uint64_t kfull, kempty, vfull, vempty, pfull[NW], pempty[NW]; /* the last two: APART */
};

/* 16 payload bytes, from an address that may be aligned to 4 bytes only; an ordinary load, because the kernel in front writes the slice's own */
__device__ __forceinline__ uint4 attn_prefill_load16(const unsigned char* src, int wide) {
    if (wide) return *reinterpret_cast<const uint4*>(src);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
    return make_uint4(w[0], w[1], w[2], w[3]);
}
/* 16 bytes of a key, chunk c of position r, to f32: dimension-major, so with a thread per position the stores are conflict-free */
template <bool KV8>
__device__ __forceinline__ void attn_prefill_key(float (*k)[128], int c, int r, const uint4& x) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    float(*d)[128] = k + c * (KV8 ? 16 : 8);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (KV8) {
            const uint32_t b = s8x4_bias(w[j]);
            d[4 * j][r] = s8_biased_to_f32<0>(b);
            d[4 * j + 1][r] = s8_biased_to_f32<1>(b);
            d[4 * j + 2][r] = s8_biased_to_f32<2>(b);
            d[4 * j + 3][r] = s8_biased_to_f32<3>(b);
        } else {
            d[2 * j][r] = bf_lo(w[j]);
            d[2 * j + 1][r] = bf_hi(w[j]);
        }
    }
}
/* 16 bytes of a value, chunk c of position r, to f32 in the slot order of AttnPrefillSmem::v */
template <bool KV8>
__device__ __forceinline__ void attn_prefill_value(float (*v)[128], int c, int r, const uint4& x) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    float4* d = reinterpret_cast<float4*>(v[r]);
    if (KV8) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t b = s8x4_bias(w[j]);
            d[(j & 1) * 16 + c * 2 + (j >> 1)] = make_float4(s8_biased_to_f32<0>(b), s8_biased_to_f32<1>(b), s8_biased_to_f32<2>(b), s8_biased_to_f32<3>(b));
        }
    } else {
        d[c] = make_float4(bf_lo(w[0]), bf_hi(w[0]), bf_lo(w[1]), bf_hi(w[1]));
        d[16 + c] = make_float4(bf_lo(w[2]), bf_hi(w[2]), bf_lo(w[3]), bf_hi(w[3]));
    }
}
/* What a producer thread brings of a key or value tile: a position's whole key, or one chunk of every PRODUCERS / NCH-th
 * value.  AHEAD: all of it is asked for before the thread waits for the buffer to come free, so that the memory's latency passes
 * meanwhile (a small block's consumers are done with a tile sooner than four round trips take: 8 rows, 10.1 -> 9.4 us per
 * tile).  Otherwise two requests at a time, for the producers that have given their registers away. */
template <bool KV8, bool AHEAD, bool KEYS> struct AttnPrefillFeed {
    static constexpr int NCH = KV8 ? 8 : 16; /* 16-byte chunks of a cached vector */
    uint4 x[AHEAD ? NCH : 1];
    unsigned short sc[AHEAD ? 4 : 1];
    const unsigned char* src;
    const unsigned short* scales;
    int pt, wide, lim;

    __device__ __forceinline__ uint4 fetch(int i) const {
        const int r = KEYS ? pt : pt / NCH + i * (ATTN_PREFILL_PRODUCERS / NCH), c = KEYS ? i : pt % NCH;
        return r < lim ? attn_prefill_load16(src + (size_t)r * (NCH * 16) + c * 16, wide) : make_uint4(0, 0, 0, 0);
    }
    /* rows past `lim` become zero */
    __device__ __forceinline__ void ask(const unsigned char* tile, const __half* tile_scales, int positions) {
        src = tile; scales = reinterpret_cast<const unsigned short*>(tile_scales) + (size_t)pt * 4; lim = positions;
        if (AHEAD) {
#pragma unroll
            for (int i = 0; i < NCH; i++) x[i] = fetch(i);
            if (KV8)
#pragma unroll
                for (int g = 0; g < 4; g++) sc[g] = scale(g);
        }
    }
    __device__ __forceinline__ unsigned short scale(int g) const { return pt < lim ? scales[g] : (unsigned short)0; }
    __device__ __forceinline__ void put(float (*to)[128], __half (*to_scales)[128]) const {
        auto one = [&](int i, const uint4& v) {
            if (KEYS) attn_prefill_key<KV8>(to, i, pt, v);
            else attn_prefill_value<KV8>(to, pt % NCH, pt / NCH + i * (ATTN_PREFILL_PRODUCERS / NCH), v);
        };
        if (AHEAD) {
#pragma unroll
            for (int i = 0; i < NCH; i++) one(i, x[i]);
        } else {
#pragma unroll 1
            for (int i = 0; i < NCH; i += 2) {
                const uint4 a = fetch(i), b = fetch(i + 1);
                one(i, a);
                one(i + 1, b);
            }
        }
        if (KV8)
#pragma unroll
            for (int g = 0; g < 4; g++) to_scales[g][pt] = __ushort_as_half(AHEAD ? sc[AHEAD ? g : 0] : scale(g));
    }
};
__device__ __forceinline__ f32x2 half2_to_f32x2(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return pack2(f.x, f.y);
}

/* one dimension of the score phase: QT queries x eight positions */
template <int QT>
__device__ __forceinline__ void attn_prefill_dim(const float* krow, const float* qrow, int tx, f32x2 (&s)[QT][4]) {
    const ulonglong2 ka = *reinterpret_cast<const ulonglong2*>(krow + tx * 4), kb = *reinterpret_cast<const ulonglong2*>(krow + 64 + tx * 4);
    float qv[QT];
    if (QT >= 4) {
#pragma unroll
        for (int i = 0; i < QT; i += 4) *reinterpret_cast<float4*>(qv + i) = *reinterpret_cast<const float4*>(qrow + i);
    } else {
#pragma unroll
        for (int i = 0; i < QT; i += 2) *reinterpret_cast<float2*>(qv + i) = *reinterpret_cast<const float2*>(qrow + i);
    }
#pragma unroll
    for (int i = 0; i < QT; i++) {
        const f32x2 qq = pack2(qv[i], qv[i]);
        ffma2(s[i][0], qq, ka.x);
        ffma2(s[i][1], qq, ka.y);
        ffma2(s[i][2], qq, kb.x);
        ffma2(s[i][3], qq, kb.y);
    }
}

/* NW consumer warps and four producer warps.  The producers widen key tile t + 1 while the consumers are in the value
 * phase of tile t, and value tile t + 1 under score phase t + 1; the four mbarriers let every consumer warp run at its own
 * pace inside that window, so one warp's soft-max overlaps another's fma.  SPLIT_REGS: 512 threads at 128 registers, of
 * which the producers give theirs up (12 x 32 x 160 + 4 x 32 x 32 = 65536 = what the block was launched with).
 *
 * APART: 2 NW consumer warps, of which warp w forms the weights of its queries (they need nothing from the value sums) and warp
 * NW + w adds the values up, a tile behind.  A small block has one or two warps per scheduler, whose chains wait on themselves;
 * apart, both products of neighbouring tiles run at once.  Per tile (INT8): 4 rows 7.0 -> 5.8 us; 8 rows 9.4 -> 9.0, and 8.7 with twice as many
 * warps of half the queries, which load the schedulers evenly. */
template <bool KV8, int QT, int NW, bool APART>
__global__ void __launch_bounds__((APART ? 64 : 32) * NW + ATTN_PREFILL_PRODUCERS, 1) k_attn_prefill(AttnArgs a, int rows, int wide, int* status) {
    extern __shared__ __align__(16) unsigned char attn_prefill_smem[];
    typedef AttnPrefillSmem<KV8, QT, NW, APART> Smem;
    Smem& sm = *reinterpret_cast<Smem*>(attn_prefill_smem);
    constexpr int M = Smem::M, RB = Smem::RB, NC = (APART ? 64 : 32) * NW, VB = KV8 ? 128 : 256;
    constexpr int DIMS = APART ? 8 : 4, FOURS = APART ? 2 : 1; /* unrolling; small blocks have the registers (2 % faster), 16 and 24 rows are slower with more */
    constexpr bool SPLIT_REGS = !APART && NW == 12, AHEAD = NC + ATTN_PREFILL_PRODUCERS <= (KV8 ? 512 : 384) && !SPLIT_REGS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    /* the last rows of the slice look furthest back: their blocks start first, of all heads (x varies fastest), the short ones fill in behind
     * them (one head after another, 512 rows of a new prompt took 109 us instead of 76, 2048 912 instead of 806) */
    const int r0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * RB, kvh = blockIdx.x;
    const int rb = min(RB, rows - r0);
    const int len0 = a.pos0 + r0 + 1;   /* positions row r0 attends over; row r0 + i: len0 + i */
    const int len_max = len0 + rb - 1;
    if (tid == 0) {
        mbar_init(&sm.kfull, ATTN_PREFILL_PRODUCERS);
        mbar_init(&sm.vfull, ATTN_PREFILL_PRODUCERS);
        mbar_init(&sm.kempty, NW);
        mbar_init(&sm.vempty, NW);
        for (int w = 0; w < NW; w++) { mbar_init(&sm.pfull[w], 1); mbar_init(&sm.pempty[w], 1); }
        mbar_init_fence();
    }
    grid_wait();
    grid_release();
    const float scale = rsqrtf((float)a.head_dim); /* run-time value on purpose, see AttnArgs */
    for (int i = tid; i < M * 16; i += NC + ATTN_PREFILL_PRODUCERS) { /* 16 bytes of one query's vector each, neighbouring lanes neighbouring queries */
        const int qi = i % M, c = i / M, row = qi >> 2;
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        if (row < rb) {
            const __nv_bfloat16* src = a.q + ((size_t)(r0 + row) * a.q_heads + kvh * 4 + (qi & 3)) * 128 + c * 8;
            if (wide) {
                const uint4 x = *reinterpret_cast<const uint4*>(src);
                w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    w[j] = (uint32_t)__bfloat16_as_ushort(src[2 * j]) | ((uint32_t)__bfloat16_as_ushort(src[2 * j + 1]) << 16);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            sm.q[c * 8 + 2 * j][qi] = __fmul_rn(bf_lo(w[j]), scale);
            sm.q[c * 8 + 2 * j + 1][qi] = __fmul_rn(bf_hi(w[j]), scale);
        }
    }
    if (tid < RB) sm.last[tid] = tid < rb ? len0 + tid : 0;
    __syncthreads();

    if (tid >= NC) { /* ---- producers ---- */
        if (SPLIT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        const size_t plane = (size_t)kvh * a.max_seq;
        const unsigned char* kc = kv_payload(a.kv, r0) + a.kv.k_off + plane * VB; /* one cache for all rows of the block */
        const unsigned char* vc = kv_payload(a.kv, r0) + a.kv.v_off + plane * VB;
        const __half* ks = KV8 ? reinterpret_cast<const __half*>(kv_scales(a.kv, r0) + a.kv.ks_off) + plane * 4 : nullptr;
        const __half* vs = KV8 ? reinterpret_cast<const __half*>(kv_scales(a.kv, r0) + a.kv.vs_off) + plane * 4 : nullptr;
        AttnPrefillFeed<KV8, AHEAD, true> keys;
        AttnPrefillFeed<KV8, AHEAD, false> values;
        keys.pt = values.pt = tid - NC;
        keys.wide = values.wide = wide;
        unsigned phase = 1; /* the buffers start empty: the first waits pass at once */
        keys.ask(kc, ks, min(128, len_max));
        for (int t0 = 0; t0 < len_max; t0 += 128, phase ^= 1) {
            values.ask(vc + (size_t)t0 * VB, vs + (size_t)t0 * 4, min(128, len_max - t0));
            if (!mbar_wait_bounded(&sm.kempty, phase, status)) return;
            keys.put(sm.k, sm.ksc);
            mbar_arrive(&sm.kfull);
            const int t1 = t0 + 128;
            if (t1 < len_max) keys.ask(kc + (size_t)t1 * VB, ks + (size_t)t1 * 4, min(128, len_max - t1));
            if (!mbar_wait_bounded(&sm.vempty, phase, status)) return;
            values.put(sm.v, sm.vsc);
            mbar_arrive(&sm.vfull);
        }
        return;
    }
    if (SPLIT_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");

    /* ---- consumers ---- */
    const int w = APART && warp >= NW ? warp - NW : warp;
    const int tx = lane >> 1, qg = lane & 1; /* neighbouring lanes read the same key / value: 16-byte shared reads merge pairs */
    const int q0 = (w * 2 + qg) * QT;        /* this thread's queries q0 .. q0 + QT - 1; query = 4 * (row in block) + head */
    float* const pw = &sm.p[w][qg][0][0];
    const int flip = qg << 4;
    unsigned phase = 0;
    float m[QT], l[QT], corr[QT];
    f32x2 acc[QT][4];
#pragma unroll
    for (int i = 0; i < QT; i++) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4; c++) acc[i][c] = 0ull;
    }
    auto weights = [&](int t0) -> bool {
        if (!mbar_wait_bounded(&sm.kfull, phase, status)) return false;
        /* ---- scores of QT queries x positions {4 tx .. +3, 64 + 4 tx .. +3}, two positions per packed fma ---- */
        f32x2 d[QT][4];
#pragma unroll
        for (int i = 0; i < QT; i++)
#pragma unroll
            for (int c = 0; c < 4; c++) d[i][c] = 0ull;
        if (KV8) {
#pragma unroll 1
            for (int gi = 0; gi < 4; gi++) {
                f32x2 pp[QT][4];
#pragma unroll
                for (int i = 0; i < QT; i++)
#pragma unroll
                    for (int c = 0; c < 4; c++) pp[i][c] = 0ull;
#pragma unroll DIMS
                for (int e = gi * 32; e < gi * 32 + 32; e++) attn_prefill_dim<QT>(sm.k[e], sm.q[e] + q0, tx, pp);
                const uint2 ha = *reinterpret_cast<const uint2*>(&sm.ksc[gi][tx * 4]), hb = *reinterpret_cast<const uint2*>(&sm.ksc[gi][64 + tx * 4]);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const f32x2 f = half2_to_f32x2(c == 0 ? ha.x : c == 1 ? ha.y : c == 2 ? hb.x : hb.y);
#pragma unroll
                    for (int i = 0; i < QT; i++) d[i][c] = ffma2_of(pp[i][c], f, d[i][c]);
                }
            }
        } else {
#pragma unroll DIMS
            for (int e = 0; e < 128; e++) attn_prefill_dim<QT>(sm.k[e], sm.q[e] + q0, tx, d);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.kempty);

        if (APART && !mbar_wait_bounded(&sm.pempty[w], phase ^ 1, status)) return false;

        /* soft-max of the tile, one query after another; its eight weights of this thread go to shared memory */
#pragma unroll
        for (int i = 0; i < QT; i++) {
            const int row = (q0 + i) >> 2;
            const int see = row < rb ? len0 + row - t0 : 0; /* positions of the tile this query sees (may be <= 0 or > 128) */
            float s[8];
#pragma unroll
            for (int c = 0; c < 4; c++) unpack2(d[i][c], s[2 * c], s[2 * c + 1]);
            float mx = -INFINITY;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const int pos = (c >> 2) * 64 + tx * 4 + (c & 3);
                if (pos >= see) s[c] = -INFINITY;
                mx = fmaxf(mx, s[c]);
            }
#pragma unroll
            for (int off = 16; off > 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(S2P_FULL_MASK, mx, off));
            const float mn = fmaxf(m[i], mx);
            corr[i] = (m[i] == -INFINITY) ? 0.f : expf(m[i] - mn);
#pragma unroll
            for (int c = 0; c < 8; c++) s[c] = (s[c] == -INFINITY) ? 0.f : expf(s[c] - mn);
            *reinterpret_cast<float4*>(pw + i * 128 + ((tx * 4) ^ flip)) = make_float4(s[0], s[1], s[2], s[3]);
            *reinterpret_cast<float4*>(pw + i * 128 + 64 + ((tx * 4) ^ flip)) = make_float4(s[4], s[5], s[6], s[7]);
            /* the 128-wide halving tree: 64 in the thread; 32 (lane bit 3) and 16 (bit 2) while handing half of the
             * four sums away each time; 8 and 4 (bits 1, 0); the last two levels pair what those lanes kept */
            const float u0 = s[0] + s[4], u1 = s[1] + s[5], u2 = s[2] + s[6], u3 = s[3] + s[7];
            const bool b3 = (tx & 8) != 0, b2 = (tx & 4) != 0;
            const float g0 = __shfl_xor_sync(S2P_FULL_MASK, b3 ? u0 : u2, 16), g1 = __shfl_xor_sync(S2P_FULL_MASK, b3 ? u1 : u3, 16);
            const float k0 = (b3 ? u2 : u0) + g0, k1 = (b3 ? u3 : u1) + g1;   /* sums 0,1 or 2,3 */
            const float g2 = __shfl_xor_sync(S2P_FULL_MASK, b2 ? k0 : k1, 8);
            float k = (b2 ? k1 : k0) + g2;                                    /* sum (b3, b2) */
            k += __shfl_xor_sync(S2P_FULL_MASK, k, 4);
            k += __shfl_xor_sync(S2P_FULL_MASK, k, 2);
            k += __shfl_xor_sync(S2P_FULL_MASK, k, 16);                       /* level 2: sums 0 + 2, 1 + 3 */
            k += __shfl_xor_sync(S2P_FULL_MASK, k, 8);                        /* level 1 */
            if (see > 0) { /* the query reaches into this tile */
                l[i] = __fmaf_rn(l[i], corr[i], k);
                m[i] = mn;
            } else {
                corr[i] = 1.f;
            }
            if (APART && tx == 0) { sm.corr[w][qg][i] = corr[i]; sm.l[w][qg][i] = l[i]; }
        }
        __syncwarp();
        if (APART && lane == 0) mbar_arrive(&sm.pfull[w]);
        return true;
    };
    auto values = [&](int t0) -> bool {
        if (APART) {
            if (!mbar_wait_bounded(&sm.pfull[w], phase, status)) return false;
#pragma unroll
            for (int i = 0; i < QT; i++) { corr[i] = sm.corr[w][qg][i]; l[i] = sm.l[w][qg][i]; }
        }
#pragma unroll
        for (int i = 0; i < QT; i++) {
            const f32x2 cc = pack2(corr[i], corr[i]);
#pragma unroll
            for (int c = 0; c < 4; c++) acc[i][c] = fmul2(acc[i][c], cc);
        }

        /* ---- value sums of QT queries x dimensions 8 tx .. +7 (one scale group), two dimensions per packed fma: in fours as
         * far as every query of the CTA sees, then one by one up to the last position of this thread's (they are of one row). A
         * weight of 0 times what lies behind it would be NaN where that is infinite.
         * The row's limit is read from shared memory and the INT8 form branches around the rest, because the loop of fours has no
         * register to spare: with the limits in registers 2048 rows after 6052 positions take 5.51 ms, so 5.39, as without any. ---- */
        static_assert(QT == 2 || QT == 4, "a thread's queries are heads of one row");
        const int all_see = min(128, KV8 ? len0 - t0 : max(len0 - t0, 0)) & ~3; /* < 0: behind the first row's last tile */
        if (!mbar_wait_bounded(&sm.vfull, phase, status)) return false;
#pragma unroll FOURS
        for (int j = 0; j < all_see; j += 4) {
            f32x2 w01[QT], w23[QT];
#pragma unroll
            for (int i = 0; i < QT; i++) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(pw + i * 128 + (j ^ flip));
                w01[i] = w.x; w23[i] = w.y;
            }
            if (KV8) {
                const uint2 h = *reinterpret_cast<const uint2*>(&sm.vsc[tx >> 2][j]);
                const f32x2 f01 = half2_to_f32x2(h.x), f23 = half2_to_f32x2(h.y);
#pragma unroll
                for (int i = 0; i < QT; i++) { w01[i] = fmul2(w01[i], f01); w23[i] = fmul2(w23[i], f23); }
            }
#pragma unroll
            for (int jj = 0; jj < 4; jj++) {
                const ulonglong2 va = *reinterpret_cast<const ulonglong2*>(&sm.v[j + jj][tx * 4]);
                const ulonglong2 vb = *reinterpret_cast<const ulonglong2*>(&sm.v[j + jj][64 + tx * 4]);
#pragma unroll
                for (int i = 0; i < QT; i++) {
                    float lo, hi;
                    unpack2(jj < 2 ? w01[i] : w23[i], lo, hi);
                    const float w = jj & 1 ? hi : lo;
                    const f32x2 ww = pack2(w, w);
                    ffma2(acc[i][0], ww, va.x);
                    ffma2(acc[i][1], ww, va.y);
                    ffma2(acc[i][2], ww, vb.x);
                    ffma2(acc[i][3], ww, vb.y);
                }
            }
        }
        if (!KV8 || t0 + 128 > len0) {
            const int see = min(128, *reinterpret_cast<volatile int*>(&sm.last[q0 >> 2]) - t0);
#pragma unroll 1
            for (int j = max(all_see, 0); j < see; j++) {
                const float f = KV8 ? __half2float(sm.vsc[tx >> 2][j]) : 1.f;
                const ulonglong2 va = *reinterpret_cast<const ulonglong2*>(&sm.v[j][tx * 4]), vb = *reinterpret_cast<const ulonglong2*>(&sm.v[j][64 + tx * 4]);
#pragma unroll
                for (int i = 0; i < QT; i++) {
                    const float p = pw[i * 128 + (j ^ flip)], w = KV8 ? __fmul_rn(p, f) : p;
                    const f32x2 ww = pack2(w, w);
                    ffma2(acc[i][0], ww, va.x);
                    ffma2(acc[i][1], ww, va.y);
                    ffma2(acc[i][2], ww, vb.x);
                    ffma2(acc[i][3], ww, vb.y);
                }
            }
        }
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&sm.vempty);
            if (APART) mbar_arrive(&sm.pempty[w]);
        }
        return true;
    };
    if (APART) {
        if (warp < NW) {
            for (int t0 = 0; t0 < len_max; t0 += 128, phase ^= 1)
                if (!weights(t0)) return;
            return;
        }
        for (int t0 = 0; t0 < len_max; t0 += 128, phase ^= 1)
            if (!values(t0)) return;
    } else {
        for (int t0 = 0; t0 < len_max; t0 += 128, phase ^= 1)
            if (!weights(t0) || !values(t0)) return;
    }
#pragma unroll
    for (int i = 0; i < QT; i++) {
        const int qi = q0 + i, row = qi >> 2;
        if (row >= rb) continue;
        uint32_t o[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            float lo, hi;
            unpack2(acc[i][c], lo, hi);
            o[c] = (uint32_t)__bfloat16_as_ushort(f2bf(__fdiv_rn(lo, l[i]))) | ((uint32_t)__bfloat16_as_ushort(f2bf(__fdiv_rn(hi, l[i]))) << 16);
        }
        __nv_bfloat16* dst = a.out + ((size_t)(r0 + row) * a.q_heads + kvh * 4 + (qi & 3)) * 128 + tx * 8;
        if (wide) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int c = 0; c < 8; c++) dst[c] = __ushort_as_bfloat16((unsigned short)(c & 1 ? o[c >> 1] >> 16 : o[c >> 1] & 0xffffu));
        }
    }
}

}  // namespace s2p
