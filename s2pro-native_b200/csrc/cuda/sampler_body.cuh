/* Device body of the semantic sampler (see sampler.cu for the algorithm), for a
 * CTA of NT threads: the stand-alone kernel runs it with 256, the persistent tick
 * kernel with its 512.  The top-30 selection is a total order, so the thread
 * count does not change the result. */
#pragma once
#include <math.h>
#include "common.cuh"
#include "ops.h"
#include "s2p_b200_abi.h"

namespace s2p {

constexpr int SMP_N_SEM = 4096;
constexpr int SMP_N_CAND = 4097;
constexpr int SMP_TOPK = 30;

template <int NT> struct SamplerSmem {
    float cand[SMP_N_CAND];
    int wtop[(NT / 32) * SMP_TOPK];      /* every warp's own top-30, best first */
    float tv[SMP_TOPK];
    int ti[SMP_TOPK];
    float sh_temp, sh_topp;
    int64_t hist[64];   /* the history window, read once */
    int64_t fin_tok;    /* the sampled token */
    int fin_mode;       /* 0 EOS (state untouched), 1 append at `count`, 2 shift the full window */
};

__device__ __forceinline__ uint64_t rotl64(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }
static __device__ __forceinline__ uint64_t xoshiro_next(uint64_t* s) {
    const uint64_t result = rotl64(s[1] * 5, 7) * 9;
    const uint64_t t = s[1] << 17;
    s[2] ^= s[0]; s[3] ^= s[1]; s[1] ^= s[2]; s[0] ^= s[3];
    s[2] ^= t;
    s[3] = rotl64(s[3], 45);
    return result;
}

/* (value descending, index ascending) as integers: larger key first, then lower index.  -0 counts as +0, NaN is never chosen (key 0). */
__device__ __forceinline__ uint32_t sampler_key(float v) {
    if (v != v) return 0u;
    uint32_t u = __float_as_uint(v);
    if (u == 0x80000000u) u = 0u;
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
/* the best of a warp's (key, index) pairs; index SMP_N_CAND where nothing is left */
__device__ __forceinline__ int sampler_best(uint32_t key, int idx) {
    const uint32_t top = __reduce_max_sync(S2P_FULL_MASK, key);
    const int i = (int)__reduce_min_sync(S2P_FULL_MASK, key == top ? (unsigned)idx : (unsigned)SMP_N_CAND);
    return top ? i : SMP_N_CAND;
}

/* logits: 4096 semantic logits of the row; eos_logit: its EOS logit; sp: its state;
 * outputs are the row's own slots. */
template <int NT>
__device__ void sampler_cta(const __nv_bfloat16* lrow, const __nv_bfloat16* eos_logit, SamplerState* sp,
                            int64_t* out_tok, int32_t* out_sem, int32_t* out_code0, uint8_t* out_eos,
                            SamplerSmem<NT>& sm) {
    constexpr int SMP_THREADS = NT;
    constexpr int SMP_PER_THREAD = (SMP_N_CAND + NT - 1) / NT;
    float* cand = sm.cand;
    float* tv = sm.tv;
    int* ti = sm.ti;
    float& sh_temp = sm.sh_temp;
    float& sh_topp = sm.sh_topp;
    const int tid = threadIdx.x;
    for (int i = tid; i < SMP_N_SEM; i += SMP_THREADS) cand[i] = bf_bits_to_f32(__ldcg(reinterpret_cast<const unsigned short*>(lrow + i)));
    if (tid == 0) cand[SMP_N_SEM] = bf_bits_to_f32(__ldcg(reinterpret_cast<const unsigned short*>(eos_logit)));
    int64_t* hist = sm.hist;
    if (tid < 64) hist[tid] = sp->prev[tid];
    const uint64_t count0 = sp->count;
    const int window = sp->window;
    S2P_CTA_SYNC();

    const bool greedy = sp->temperature == 0.0f;
    const int capped = count0 < (uint64_t)window ? (int)count0 : window;
    float pen = 0.f;
    int pen_at = -1; /* the history's tokens side by side: all read the original values, equal tokens write equal ones */
    if (tid < capped) {
        const int64_t tok = hist[tid];
        if (tok >= S2P_TOK_SEMANTIC_START && tok <= S2P_TOK_SEMANTIC_END) pen_at = (int)(tok - S2P_TOK_SEMANTIC_START);
        else if (tok == S2P_TOK_EOS) pen_at = SMP_N_SEM;
        if (pen_at >= 0) {
            const float v = cand[pen_at], rep_penalty = sp->rep_penalty;
            pen = v < 0.f ? __fmul_rn(v, rep_penalty) : __fdiv_rn(v, rep_penalty);
        }
    }
    if (tid == 0) {
        bool ras = false;
        if (!greedy && capped >= 4) {
            int64_t last4[4];
            for (int r = 0; r < 4; r++) {
                int idx = capped - (4 - r);
                last4[r] = hist[idx < 0 ? 0 : idx];
            }
            for (int x = 0; x < 4; x++)
                for (int y = x + 1; y < 4; y++) ras |= (last4[x] == last4[y]);
        }
        sh_temp = ras ? 1.0f : sp->temperature;
        sh_topp = ras ? 0.9f : sp->top_p;
    }
    S2P_CTA_SYNC();
    if (pen_at >= 0) cand[pen_at] = pen;
    S2P_CTA_SYNC();

    /* top-30 in two warp-level passes without block-wide rounds: every warp selects the 30 best of its own candidates
     * (i = tid + NT j, keys in registers), two integer reductions a choice, after which only the owner looks through its
     * candidates again; warp 0 then merges the warps' sorted lists, a list per lane.  (value desc, index asc) is a total order, so the
     * result is the block-wide top-30 in order. */
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int NW = SMP_THREADS / 32;
    int* wt = sm.wtop;
    {
        uint32_t mine[SMP_PER_THREAD], key = 0u;
        int idx = SMP_N_CAND;
        auto look = [&] {
            key = 0u; idx = SMP_N_CAND;
#pragma unroll
            for (int j = 0; j < SMP_PER_THREAD; j++)
                if (mine[j] > key) { key = mine[j]; idx = tid + j * SMP_THREADS; }
        };
#pragma unroll
        for (int j = 0; j < SMP_PER_THREAD; j++) {
            const int i = tid + j * SMP_THREADS;
            mine[j] = i < SMP_N_CAND ? sampler_key(cand[i]) : 0u;
        }
        look();
        for (int k = 0; k < SMP_TOPK; k++) {
            const int best = sampler_best(key, idx);
            if (lane == 0) wt[warp * SMP_TOPK + k] = best;
            if (best < SMP_N_CAND && best == idx) { /* the owner retires the winner */
#pragma unroll
                for (int j = 0; j < SMP_PER_THREAD; j++)
                    if (tid + j * SMP_THREADS == best) mine[j] = 0u;
                look();
            }
        }
    }
    S2P_CTA_SYNC();
    if (warp == 0) {
        int at = 0;
        int idx = lane < NW ? wt[lane * SMP_TOPK] : SMP_N_CAND;
        uint32_t key = idx < SMP_N_CAND ? sampler_key(cand[idx]) : 0u;
        for (int k = 0; k < SMP_TOPK; k++) {
            const int best = sampler_best(key, idx);
            if (lane == 0) { tv[k] = best < SMP_N_CAND ? cand[best] : -INFINITY; ti[k] = min(best, SMP_N_SEM); } /* nothing left: EOS, a row of NaN ends its stream */
            if (best < SMP_N_CAND && best == idx) {
                at++;
                idx = at < SMP_TOPK ? wt[lane * SMP_TOPK + at] : SMP_N_CAND;
                key = idx < SMP_N_CAND ? sampler_key(cand[idx]) : 0u;
            }
        }
        __syncwarp();
        int choice = 0;
        if (!greedy) {
            /* a rank per lane; the sums are the reference's, rank after rank */
            const bool rank = lane < SMP_TOPK;
            const float v = tv[rank ? lane : 0], m = tv[0];
            auto sum_of = [](float x) {
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < SMP_TOPK; j++) s = __fadd_rn(s, __shfl_sync(S2P_FULL_MASK, x, j));
                return s;
            };
            const float e = expf(v - m);
            const float share = __fdiv_rn(e, sum_of(e));
            float cum = 0.f, upto = 0.f;
#pragma unroll
            for (int j = 0; j < SMP_TOPK; j++) {
                cum = __fadd_rn(cum, __shfl_sync(S2P_FULL_MASK, share, j));
                if (j == lane) upto = cum;
            }
            const bool masked = lane > 0 && upto > sh_topp;
            const float t = sh_temp < 1e-5f ? 1e-5f : sh_temp;
            const float m2 = __fdiv_rn(m, t);
            float p2 = masked ? 0.f : expf(__fsub_rn(__fdiv_rn(v, t), m2));
            p2 = __fdiv_rn(p2, sum_of(p2));

            if (sp->seeded) {
                const uint64_t step_seed = ((uint64_t)sp->seed31 * 19349663ULL) ^ (count0 * 73856093ULL);
                const uint64_t hashed = (step_seed * 8589934591ULL) ^ ((uint64_t)lane * 479001599ULL);
                float u = __fdiv_rn((float)(uint32_t)(hashed & 0xFFFFFFULL), 16777216.0f);
                if (u < 1e-10f) u = 1e-10f;
                const float g = -logf(-logf(u));
                const float pert = __fadd_rn(logf(__fadd_rn(p2, 1e-10f)), g);
                /* the first largest; what does not exceed -inf is never chosen, and rank 0 stands where nothing is */
                const uint32_t key = rank && pert > -INFINITY ? sampler_key(pert) : 0u;
                const uint32_t top = __reduce_max_sync(S2P_FULL_MASK, key);
                choice = top ? __ffs(__ballot_sync(S2P_FULL_MASK, key == top)) - 1 : 0;
            } else {
                double r = 0.0;
                if (lane == 0) r = (double)(xoshiro_next(sp->rng) >> 11) * 0x1.0p-53;
                double cum2 = 0.0;
                int lastnz = 0;
                choice = -1;
                for (int j = 0; j < SMP_TOPK; j++) { /* lane 0's result counts */
                    const float p = __shfl_sync(S2P_FULL_MASK, p2, j);
                    if (p <= 0.f) continue;
                    lastnz = j;
                    cum2 += (double)p;
                    if (choice < 0 && r < cum2) choice = j;
                }
                if (choice < 0) choice = lastnz;
            }
        }
        if (tid == 0) {
            const int ci = ti[choice];
            if (ci == SMP_N_SEM) { /* EOS: semantic code forced to 0, sampler state untouched */
                *out_tok = S2P_TOK_EOS;
                *out_sem = 0;
                *out_code0 = 0;
                *out_eos = 1;
                sm.fin_mode = 0;
            } else {
                const int64_t tok = (int64_t)S2P_TOK_SEMANTIC_START + ci;
                *out_tok = tok;
                *out_sem = ci;
                *out_code0 = ci;
                *out_eos = 0;
                sm.fin_tok = tok;
                sm.fin_mode = count0 < (uint64_t)window ? 1 : 2;
                sp->count = count0 + 1;
            }
        }
    }
    S2P_CTA_SYNC();
    /* history update, the shift done by the threads side by side from the staged window */
    if (sm.fin_mode == 1) {
        if (tid == 0) sp->prev[count0] = sm.fin_tok;
    } else if (sm.fin_mode == 2) {
        if (tid < window - 1) sp->prev[tid] = hist[tid + 1];
        else if (tid == window - 1) sp->prev[tid] = sm.fin_tok;
    }
}

}  // namespace s2p
