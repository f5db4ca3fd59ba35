// Device functions shared by the router kernels and the single-launch decode step: the canonical logit of an
// expert row staged in shared memory, the warp-parallel top-k + softmax, and the grouping of a small block's routes.
#pragma once

#include "tf_common.cuh"

namespace tf {

// Top-k of a row of scores (highest first, ties to the lower expert index) and the softmax over the selected scores
// times the per-expert gain, rounded to fp16: the first k entries of the order (score desc, index asc), which is the
// result of the reference's insertion scan (Metal/MoE/moe.metal:152-184). Every lane holds its experts' scores as
// order-preserving integer keys, sorted; a round is one warp-wide integer maximum over the lanes' greatest keys (lanes that tie
// compare indices), and the winner's lane moves on to its next key. When nothing above -inf is left (fewer comparable candidates
// than top_k), the remaining ranks repeat the lowest expert that is selected or at -inf, expert 0 if there is none. NaN scores never
// win. The per-expert gains travel during the rounds; the exponentials are taken by top_k lanes at once and summed in rank
// order. `scores` is only read. (With two reductions and a scan of the lane's keys per round and the gains loaded at the end, 3300
// to 6000 clocks for 8 of 128 in a step; 2700 to 3600 with this.)
__device__ __forceinline__ uint32_t topk_score_key(float v) {
    if (v != v) return 0u;
    const uint32_t b = __float_as_uint(v + 0.0f);             // -0 and +0 compare equal: one key for both
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);       // -inf maps to 0x007FFFFF, above the NaN key
}
__device__ __forceinline__ float topk_key_score(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
template <int kPerLane>        // experts per lane: num_experts <= 32 * kPerLane
__device__ __forceinline__ void warp_select_topk_held(const float* scores /*shared*/, uint32_t num_experts, uint32_t top_k,
                                                      const uint16_t* __restrict__ per_expert_scale,
                                                      uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w, int lane) {
    constexpr uint32_t kNegInfKey = 0x007FFFFFu;
    uint32_t key[kPerLane], idx[kPerLane];
    uint16_t gain[kPerLane];
    uint32_t low = 0xFFFFFFFFu;                  // this lane's lowest expert that is selected or at -inf
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const uint32_t e = lane + j * kWarp;
        idx[j] = e;
        key[j] = e < num_experts ? topk_score_key(scores[e]) : 0u;
        gain[j] = e < num_experts ? __ldg(per_expert_scale + e) : (uint16_t)0;
        if (key[j] == kNegInfKey) low = min(low, e);
    }
    // descending by key; equal keys keep their order, which is ascending by expert
#pragma unroll
    for (int i = 1; i < kPerLane; ++i) {
#pragma unroll
        for (int j = i; j > 0; --j) {
            const bool swap = key[j] > key[j - 1];
            const uint32_t k0 = swap ? key[j] : key[j - 1], k1 = swap ? key[j - 1] : key[j];
            const uint32_t i0 = swap ? idx[j] : idx[j - 1], i1 = swap ? idx[j - 1] : idx[j];
            key[j - 1] = k0; key[j] = k1; idx[j - 1] = i0; idx[j] = i1;
        }
    }
    float my_score = 0.0f, max_s = 0.0f;
    uint32_t my_idx = 0, r = 0;
    for (; r < top_k; ++r) {
        const uint32_t top = __reduce_max_sync(kFullMask, key[0]);
        if (top <= kNegInfKey) break;
        const uint32_t holders = __ballot_sync(kFullMask, key[0] == top);
        uint32_t winner;
        if (holders & (holders - 1u)) winner = __reduce_min_sync(kFullMask, key[0] == top ? idx[0] : 0xFFFFFFFFu);
        else winner = __shfl_sync(kFullMask, idx[0], __ffs((int)holders) - 1);
        const float top_score = topk_key_score(top);
        if (r == 0) max_s = top_score;
        if ((uint32_t)lane == r) { my_score = top_score; my_idx = winner; }
        if (key[0] == top && idx[0] == winner) {
            low = min(low, winner);
#pragma unroll
            for (int j = 1; j < kPerLane; ++j) { key[j - 1] = key[j]; idx[j - 1] = idx[j]; }
            key[kPerLane - 1] = 0u;
        }
    }
    if (r < top_k) {
        const uint32_t lowest = __reduce_min_sync(kFullMask, low), winner = lowest == 0xFFFFFFFFu ? 0u : lowest;
        if (r == 0) max_s = -INFINITY;
        if ((uint32_t)lane >= r) { my_score = -INFINITY; my_idx = winner; }
    }
    uint32_t my_gain = 0;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const uint32_t v = __shfl_sync(kFullMask, (uint32_t)gain[j], (int)(my_idx % kWarp));
        if (my_idx / kWarp == (uint32_t)j) my_gain = v;
    }
    const float ex = (uint32_t)lane < top_k ? expf(my_score - max_s) : 0.0f;
    float sum_exp = 0.0f;
#pragma unroll 4
    for (uint32_t k = 0; k < top_k; ++k) sum_exp += __shfl_sync(kFullMask, ex, (int)k);
    if ((uint32_t)lane < top_k) {
        const float w = ex / sum_exp * bf16_bits_to_float((uint16_t)my_gain);
        out_idx[lane] = my_idx;
        out_w[lane] = __half_as_ushort(__float2half_rn(w));
    }
}

// Half of the comparisons of every round for up to 128 experts.
__device__ __forceinline__ void warp_select_topk(const float* scores /*shared*/, uint32_t num_experts, uint32_t top_k,
                                                 const uint16_t* __restrict__ per_expert_scale,
                                                 uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w, int lane) {
    static_assert(TF_MAX_ROUTER_EXPERTS == 8 * kWarp, "eight experts per lane at the most");
    if (num_experts <= 4u * kWarp) warp_select_topk_held<4>(scores, num_experts, top_k, per_expert_scale, out_idx, out_w, lane);
    else warp_select_topk_held<8>(scores, num_experts, top_k, per_expert_scale, out_idx, out_w, lane);
}

// Canonical logit of one expert row whose bytes, scales and biases sit in shared memory
// (same arithmetic and order as router_row_logit; only the operand source differs).
__device__ __forceinline__ float router_row_logit_smem(const uint8_t* Wrow, const uint16_t* s_row, const uint16_t* b_row,
                                                       const float* xf, uint32_t groups, int lane) {
    float acc = 0.0f;
#pragma unroll 4
    for (uint32_t g = 0; g < groups; ++g) {
        const uint32_t i0 = g * kGroup + lane * 2;
        const uint32_t w = *reinterpret_cast<const uint16_t*>(Wrow + i0);
        const float q0 = (float)(w & 0xFFu), q1 = (float)(w >> 8);
        const float2 xv = *reinterpret_cast<const float2*>(xf + i0);
        const float s = bf16_bits_to_float(s_row[g]);
        const float b = bf16_bits_to_float(b_row[g]);
        const float p = __fmaf_rn(q1, xv.y, __fmul_rn(q0, xv.x));
        acc = __fmaf_rn(s, p, acc);
        acc = __fmaf_rn(b, __fadd_rn(xv.x, xv.y), acc);
    }
    return warp_sum(acc);
}

// Grouping of a small block's routes inside the router launch (the work of group_routes_kernel for a few
// hundred rows): the block that finishes the last row sorts the (token, rank) pairs by expert, stably in
// token-major order, and writes offsets, counts, groups and the 8-token chunk table. A pair's place is its expert's
// offset plus the number of earlier pairs of that expert, counted on a per-expert bitmap over the pairs.
struct RouterGroupOut {
    tf_pair* sorted_pairs;          // nullptr: no grouping
    uint32_t* per_expert_offsets;
    uint32_t* per_expert_counts;
    tf_group* groups;
    uint32_t* chunk_group;
    uint32_t* chunk_start;
    uint32_t* counters;
};

__host__ __device__ inline size_t router_group_smem_bytes(uint32_t n_pairs, uint32_t num_experts, bool counted) {
    const uint32_t nw = (n_pairs + 31) / 32;
    // mask, its prefix counts, hist + offs, expert ids, warp totals (3 x 32), weights
    return (size_t)num_experts * nw * 4 + (counted ? (size_t)((num_experts * nw + 1) / 2) * 4 : 0) + (size_t)num_experts * 2 * 4 + (size_t)n_pairs * 4 + 96 * 4 + (size_t)((n_pairs + 1) / 2) * 4;
}

// COUNTED (the few-row router): the counts before every bitmap word are taken first, a thread per expert (a thread
// per pair that adds up the words before its own took 20 us for 1600 pairs). Otherwise (one block per row) the words before a
// pair's own are added up on the spot.
template <bool COUNTED>
__device__ __forceinline__ void group_routes_in_block(const uint32_t* __restrict__ idx, const uint16_t* __restrict__ w, uint32_t T, uint32_t K,
                                      uint32_t E, const RouterGroupOut& out, uint8_t* smem) {
    const uint32_t n = T * K, nw = (n + 31) / 32;
    uint32_t* mask = reinterpret_cast<uint32_t*>(smem);          // [E][nw]
    uint32_t* hist = mask + (size_t)E * nw;                      // [E]
    uint32_t* offs = hist + E;                                   // [E]
    uint32_t* exs = offs + E;                                    // [n]
    uint32_t* wtot = exs + n;                                    // [3][32]: per-warp totals of the scan
    uint16_t* wts = reinterpret_cast<uint16_t*>(wtot + 96);      // [n]
    uint16_t* pre = wts + ((n + 1u) & ~1u);                      // [E][nw]: pairs of the expert in the words before this one
    const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp, nwarps = blockDim.x / kWarp;
    // ids and weights (written by other blocks of this launch) travel while the bitmaps are cleared
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        uint32_t ex = __ldcg(idx + i);
        if (ex != 0xFFFFFFFFu && ex >= E) ex = E - 1;            // min(id, E-1): Runtime/Inference/RealForwardRunner.swift:955
        exs[i] = ex;
        wts[i] = __ldcg(w + i);
    }
    for (uint32_t i = threadIdx.x; i < E * nw + E; i += blockDim.x) mask[i] = 0;      // mask and hist are adjacent
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t ex = exs[i];
        if (ex != 0xFFFFFFFFu) {
            atomicAdd(&hist[ex], 1u);
            atomicOr(&mask[(size_t)ex * nw + i / 32], 1u << (i % 32));
        }
    }
    __syncthreads();
    if constexpr (COUNTED) {
        // a thread per expert walks its words (1600 pairs: 50 words; a warp per expert with a scan took 11 700 clocks for 128 experts)
        for (uint32_t ex = threadIdx.x; ex < E; ex += blockDim.x) {
            const uint32_t* m = mask + (size_t)ex * nw;
            uint16_t* p = pre + (size_t)ex * nw;
            uint32_t run = 0;
#pragma unroll 4
            for (uint32_t q = 0; q < nw; ++q) {
                p[q] = (uint16_t)run;
                run += __popc(m[q]);
            }
        }
        __syncthreads();
    }
    // exclusive scans over the experts (pairs, non-empty groups, chunks): every warp scans 32 experts, the warps'
    // totals meet in shared memory, and rounds of nwarps * 32 experts carry the running totals.
    uint32_t off = 0, gi = 0, ch = 0;
    for (uint32_t base = 0; base < E; base += nwarps * kWarp) {
        const uint32_t e = base + warp * kWarp + lane;
        const uint32_t cnt = e < E ? hist[e] : 0u;
        const uint32_t nch = (cnt + (uint32_t)kChunkTokens - 1) / (uint32_t)kChunkTokens;
        uint32_t i_off = cnt, i_g = cnt ? 1u : 0u, i_ch = nch;
#pragma unroll
        for (int o = 1; o < kWarp; o <<= 1) {
            const uint32_t a = __shfl_up_sync(kFullMask, i_off, o), b2 = __shfl_up_sync(kFullMask, i_g, o),
                           c = __shfl_up_sync(kFullMask, i_ch, o);
            if ((int)lane >= o) { i_off += a; i_g += b2; i_ch += c; }
        }
        if (lane == kWarp - 1) { wtot[warp] = i_off; wtot[32 + warp] = i_g; wtot[64 + warp] = i_ch; }
        __syncthreads();
        uint32_t p_off = off, p_g = gi, p_ch = ch;
        for (uint32_t v = 0; v < nwarps; ++v) {
            const uint32_t a = wtot[v], b2 = wtot[32 + v], c = wtot[64 + v];
            if (v < warp) { p_off += a; p_g += b2; p_ch += c; }
            off += a; gi += b2; ch += c;
        }
        const uint32_t my_off = p_off + i_off - cnt, my_g = p_g + i_g - (cnt ? 1u : 0u), my_ch = p_ch + i_ch - nch;
        if (e < E) {
            offs[e] = my_off;
            out.per_expert_counts[e] = cnt;
            out.per_expert_offsets[e] = cnt ? my_off : 0xFFFFFFFFu;
            if (cnt) {
                out.groups[my_g] = tf_group{e, my_off, cnt};
                out.chunk_start[my_g] = my_ch;
                for (uint32_t j = 0; j < nch; ++j) out.chunk_group[my_ch + j] = my_g;
            }
        }
        __syncthreads();                                          // wtot is reused by the next round; offs is read below
    }
    if (threadIdx.x == 0) {
        out.counters[0] = gi;
        out.counters[1] = ch;
        out.counters[2] = n;
        out.counters[3] = off;
    }
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t ex = exs[i];
        if (ex == 0xFFFFFFFFu) continue;
        const uint32_t* m = mask + (size_t)ex * nw;
        uint32_t pos = offs[ex] + __popc(m[i / 32] & ((1u << (i % 32)) - 1u));
        if constexpr (COUNTED) {
            pos += pre[(size_t)ex * nw + i / 32];
        } else {
            for (uint32_t q = 0; q < i / 32; ++q) pos += __popc(m[q]);
        }
        out.sorted_pairs[pos] = tf_pair{i / K, ex, i % K, (uint32_t)wts[i]};
    }
}

// The tables of one token: a pair's place is the number of selected experts with a smaller id; every group holds one pair and one
// chunk. That needs distinct experts: a row with fewer than top_k selectable logits (NaN, -inf) repeats an expert, and then the general
// grouping merges the repeats into one group. All threads of the block, after a barrier behind the writes of out_idx and out_w.
__device__ __forceinline__ void group_one_token(const uint32_t* out_idx, const uint16_t* out_w, uint32_t top_k, uint32_t num_experts,
                                                const RouterGroupOut& grp, uint8_t* smem) {
    int repeated = 0;
    if (threadIdx.x < top_k) {
        uint32_t mine = out_idx[threadIdx.x];
        if (mine >= num_experts) mine = num_experts - 1;
        for (uint32_t r = 0; r < top_k; ++r) {
            uint32_t other = out_idx[r];
            if (other >= num_experts) other = num_experts - 1;
            repeated |= (r != threadIdx.x && other == mine) ? 1 : 0;
        }
    }
    if (__syncthreads_or(repeated)) {
        group_routes_in_block<false>(out_idx, out_w, 1, top_k, num_experts, grp, smem);
        return;
    }
    for (uint32_t e = threadIdx.x; e < num_experts; e += blockDim.x) {
        grp.per_expert_counts[e] = 0u;
        grp.per_expert_offsets[e] = 0xFFFFFFFFu;
    }
    __syncthreads();
    if (threadIdx.x < top_k) {
        uint32_t mine = out_idx[threadIdx.x];
        if (mine >= num_experts) mine = num_experts - 1;
        uint32_t pos = 0;
        for (uint32_t r = 0; r < top_k; ++r) {
            uint32_t other = out_idx[r];
            if (other >= num_experts) other = num_experts - 1;
            pos += other < mine ? 1u : 0u;
        }
        grp.sorted_pairs[pos] = tf_pair{0u, mine, threadIdx.x, (uint32_t)out_w[threadIdx.x]};
        grp.per_expert_counts[mine] = 1u;
        grp.per_expert_offsets[mine] = pos;
        grp.groups[pos] = tf_group{mine, pos, 1u};
        grp.chunk_start[pos] = pos;
        grp.chunk_group[pos] = pos;
    }
    if (threadIdx.x == 0) {
        grp.counters[0] = top_k;
        grp.counters[1] = top_k;
        grp.counters[2] = top_k;
        grp.counters[3] = top_k;
    }
}

}  // namespace tf
