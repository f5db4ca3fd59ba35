// Router: 8-bit affine GEMV + top-k + softmax in ONE launch, ids stay on the device.
// Replaces router_gemv_gemma4_r4 + router_topk_select_k8 (Metal/MoE/moe.metal:78-185)
// and prefill_router_gemma4_block (Metal/Prefill/prefill.metal:478-573).
//
// Logit arithmetic is canonical so that a CPU emulation reproduces every bit
// (top-k indices must match exactly):
//   xf[i]  = fmul(float(hidden[i]), float(effective_scale[i]))
//   lane l, group g: i0 = 64 g + 2 l
//     p   = fma(q1, xf[i0+1], fmul(q0, xf[i0]))
//     acc = fma(s, p, acc);  acc = fma(b, fadd(xf[i0], xf[i0+1]), acc)
//   logit = xor-butterfly sum over the 32 lanes (offsets 16, 8, 4, 2, 1)
// which is the reference kernel's per-lane element assignment with the
// contraction and reduction order fixed.
#include <algorithm>

#include "router.cuh"
#include "router_tensor.cuh"

namespace tf {

constexpr int kSplitExpertsPerBlock = 4;
constexpr int kSplitThreads = kSplitExpertsPerBlock * kWarp;
constexpr int kBlockRouterThreads = 256;

template <bool X_BF16>
__device__ __forceinline__ void stage_router_x(const uint16_t* hidden, const uint16_t* __restrict__ eff,
                                               float* xf, uint32_t d) {
    for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) {
        const float h = X_BF16 ? bf16_bits_to_float(hidden[i]) : f16_bits_to_float(hidden[i]);
        xf[i] = __fmul_rn(h, bf16_bits_to_float(eff[i]));
    }
    __syncthreads();
}

__device__ __forceinline__ float router_row_logit(const uint8_t* __restrict__ Wrow, const uint16_t* __restrict__ s_row,
                                                  const uint16_t* __restrict__ b_row, const float* xf,
                                                  uint32_t groups, int lane, bool a2) {
    float acc = 0.0f;
    for (uint32_t g = 0; g < groups; ++g) {
        const uint32_t i0 = g * kGroup + lane * 2;
        uint32_t w;
        if (a2) w = *reinterpret_cast<const uint16_t*>(Wrow + i0);
        else w = (uint32_t)Wrow[i0] | ((uint32_t)Wrow[i0 + 1] << 8);
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

// Few rows (decode): grid (rows, experts/4); the block first copies its four expert rows into
// shared memory with coalesced loads (the per-lane access pattern of the canonical order would
// otherwise be a chain of 2-byte global loads); the last block to finish a row (self-resetting
// ticket) runs the selection, so one launch does everything.
template <bool X_BF16>
__global__ void __launch_bounds__(kSplitThreads)
router_split_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                    const uint16_t* hidden, uint32_t hidden_stride,
                    const uint16_t* __restrict__ eff, const uint16_t* __restrict__ per_expert_scale,
                    const float* __restrict__ logit_bias,
                    uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w, float* __restrict__ out_logits,
                    float* scratch_logits, unsigned int* tickets, const RouterGroupOut grp,
                    uint32_t num_experts, uint32_t d, uint32_t top_k, bool a2) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* xf = reinterpret_cast<float*>(smem);                                   // [d]
    uint8_t* wrows = smem + (size_t)d * 4;                                        // [4][d]
    const uint32_t groups = d / kGroup;
    uint16_t* srows = reinterpret_cast<uint16_t*>(wrows + (size_t)kSplitExpertsPerBlock * d);   // [4][groups]
    uint16_t* brows = srows + kSplitExpertsPerBlock * groups;
    __shared__ float scores[TF_MAX_ROUTER_EXPERTS];
    __shared__ bool is_last;
    const uint32_t row = blockIdx.x;
    const uint32_t e0 = blockIdx.y * kSplitExpertsPerBlock;
    const uint32_t ne = num_experts - e0 < (uint32_t)kSplitExpertsPerBlock ? num_experts - e0 : (uint32_t)kSplitExpertsPerBlock;
    // the four rows are contiguous in every plane
    const uint8_t* wsrc = W + (size_t)e0 * d;
    const uint16_t* hrow = hidden + (size_t)row * hidden_stride;
    const bool a16 = (reinterpret_cast<uintptr_t>(wsrc) & 15) == 0 && (d & 15) == 0;
    const bool x16 = (reinterpret_cast<uintptr_t>(hrow) & 15) == 0 && (reinterpret_cast<uintptr_t>(eff) & 15) == 0 && (d & 7) == 0;
    const bool late = grp.sorted_pairs != nullptr;        // see below
    if (!late) pdl_launch_dependents();
    if (a16 && x16 && ne * d <= kSplitThreads * 16 * 6 && d <= kSplitThreads * 8 * 3) {
        // latency path: every load of the block is issued before the first one is consumed
        uint4 wv[6], hv[3], ev[3];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const uint32_t i = threadIdx.x + j * kSplitThreads;
            wv[j] = i < ne * d / 16 ? ldg_nc_u4(wsrc + (size_t)i * 16) : make_uint4(0u, 0u, 0u, 0u);
        }
        pdl_wait();          // the weights above do not depend on the previous kernel; the hidden row does
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const uint32_t i = threadIdx.x + j * kSplitThreads;
            const bool ok = i < d / 8;
            hv[j] = ok ? reinterpret_cast<const uint4*>(hrow)[i] : make_uint4(0u, 0u, 0u, 0u);
            ev[j] = ok ? __ldg(reinterpret_cast<const uint4*>(eff) + i) : make_uint4(0u, 0u, 0u, 0u);
        }
        for (uint32_t i = threadIdx.x; i < ne * groups; i += blockDim.x) {
            srows[i] = S[(size_t)e0 * groups + i];
            brows[i] = B[(size_t)e0 * groups + i];
        }
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const uint32_t i = threadIdx.x + j * kSplitThreads;
            if (i < ne * d / 16) reinterpret_cast<uint4*>(wrows)[i] = wv[j];
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const uint32_t i = threadIdx.x + j * kSplitThreads;
            if (i < d / 8) {
                const uint32_t hw[4] = {hv[j].x, hv[j].y, hv[j].z, hv[j].w}, ew[4] = {ev[j].x, ev[j].y, ev[j].z, ev[j].w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint16_t h0 = (uint16_t)(hw[q] & 0xFFFFu), h1 = (uint16_t)(hw[q] >> 16);
                    const float f0 = X_BF16 ? bf16_bits_to_float(h0) : f16_bits_to_float(h0);
                    const float f1 = X_BF16 ? bf16_bits_to_float(h1) : f16_bits_to_float(h1);
                    xf[i * 8 + 2 * q] = __fmul_rn(f0, bf16_bits_to_float((uint16_t)(ew[q] & 0xFFFFu)));
                    xf[i * 8 + 2 * q + 1] = __fmul_rn(f1, bf16_bits_to_float((uint16_t)(ew[q] >> 16)));
                }
            }
        }
        __syncthreads();
    } else {
        if (a16) {
            for (uint32_t i = threadIdx.x; i < ne * d / 16; i += blockDim.x)
                reinterpret_cast<uint4*>(wrows)[i] = ldg_nc_u4(wsrc + (size_t)i * 16);
        } else if (a2) {
            for (uint32_t i = threadIdx.x; i < ne * d / 2; i += blockDim.x)
                reinterpret_cast<uint16_t*>(wrows)[i] = reinterpret_cast<const uint16_t*>(wsrc)[i];
        } else {
            for (uint32_t i = threadIdx.x; i < ne * d; i += blockDim.x) wrows[i] = wsrc[i];
        }
        for (uint32_t i = threadIdx.x; i < ne * groups; i += blockDim.x) {
            srows[i] = S[(size_t)e0 * groups + i];
            brows[i] = B[(size_t)e0 * groups + i];
        }
        pdl_wait();
        stage_router_x<X_BF16>(hrow, eff, xf, d);     // ends with a barrier
    }

    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t e = e0 + warp;
    if (e < num_experts) {
        float logit = router_row_logit_smem(wrows + (size_t)warp * d, srows + warp * groups, brows + warp * groups, xf, groups, lane);
        if (logit_bias) logit = __fadd_rn(logit, logit_bias[e]);
        if (lane == 0) scratch_logits[(size_t)row * TF_MAX_ROUTER_EXPERTS + e] = logit;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int tk = atomicAdd(&tickets[row], 1u);
        is_last = (tk == gridDim.y - 1);
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (uint32_t i = threadIdx.x; i < num_experts; i += blockDim.x) {
        const float v = __ldcg(&scratch_logits[(size_t)row * TF_MAX_ROUTER_EXPERTS + i]);
        scores[i] = v;
        if (out_logits) out_logits[(size_t)row * num_experts + i] = v;
    }
    if (threadIdx.x == 0) tickets[row] = 0;   // ready for the next launch on this stream
    __syncthreads();
    if (warp == 0)
        warp_select_topk(scores, num_experts, top_k, per_expert_scale, out_idx + (size_t)row * top_k,
                         out_w + (size_t)row * top_k, lane);
    // With grouping (a block forward) the next launch is let in only now, while warp 0 selects: the routed gate/up launch would otherwise
    // sit on the SMs, waiting, from the first microsecond on, and keep both launches of the shared expert, which run beside this
    // kernel, until it has ended. One token, 30 layers: released at the start 994 us, after the logits 860.
    if (!late) return;
    pdl_launch_dependents();
    if (gridDim.x == 1) {
        __syncthreads();                       // warp 0 has written the row's indices and weights
        group_one_token(out_idx, out_w, top_k, num_experts, grp, smem);
        return;
    }
    // the block that completes the last row groups all rows (second ticket, after the row tickets)
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int tk = atomicAdd(&tickets[kRouterSplitRows], 1u);
        is_last = (tk == gridDim.x - 1);
        if (is_last) tickets[kRouterSplitRows] = 0;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    group_routes_in_block<false>(out_idx, out_w, gridDim.x, top_k, num_experts, grp, smem);
}

// A handful of rows (batched decode, 2...kRouterSplitRows): grid (rows / R, experts / 8). A block stages R activation
// rows (as fp32 x * effective_scale) and its eight expert rows in shared memory; warp w then computes the logits of
// expert e0 + w for all R rows at once, so the codes, scales and biases of a group are decoded once per R rows. The
// arithmetic and its order per (row, expert) are those of router_row_logit_smem. The last block of a row group
// (ticket) selects the top-k of its R rows, one warp per row; the block that completes the last row group builds the
// grouping tables.
constexpr int kRowsThreads = 256;
constexpr uint32_t kRowsLateRows = 52;
constexpr int kRowsExpertsPerBlock = kRowsThreads / kWarp;
template <bool X_BF16, int R>
__global__ void __launch_bounds__(kRowsThreads)
router_rows_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                   const uint16_t* hidden, uint32_t hidden_stride,
                   const uint16_t* __restrict__ eff, const uint16_t* __restrict__ per_expert_scale,
                   const float* __restrict__ logit_bias,
                   uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w, float* __restrict__ out_logits,
                   float* scratch_logits, unsigned int* tickets, const RouterGroupOut grp,
                   uint32_t rows, uint32_t num_experts, uint32_t d, uint32_t top_k, bool resident) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t groups = d / kGroup;
    float* xf = reinterpret_cast<float*>(smem);                                        // [R][d]
    uint8_t* wrows = smem + (size_t)R * d * 4;                                         // [8][d]
    uint16_t* srows = reinterpret_cast<uint16_t*>(wrows + (size_t)kRowsExpertsPerBlock * d);   // [8][groups]
    uint16_t* brows = srows + kRowsExpertsPerBlock * groups;
    __shared__ float scores[R][TF_MAX_ROUTER_EXPERTS];
    __shared__ bool is_last;
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t row0 = blockIdx.x * R;
    const uint32_t e0 = blockIdx.y * kRowsExpertsPerBlock;
    const uint32_t ne = num_experts - e0 < (uint32_t)kRowsExpertsPerBlock ? num_experts - e0 : (uint32_t)kRowsExpertsPerBlock;
    // As in router_split_kernel the routed launch is let in late, by the block that groups, before it does: released at the start, the
    // routed blocks take every SM that a router block leaves and wait there, ahead of the shared expert. Blocks that are not
    // all resident let it in late by themselves, when the last of them starts; what is left then are the microseconds of selection
    // and grouping, and with many rows those let the shared expert's down projection in before the routed blocks, too, which
    // must not be. us a layer, at the start and late. All resident: 128 experts of 2816, 40 rows 119.9 and 110.7; 16 experts of
    // 2816, 64 rows 73.2 and 64.8; 64 experts of 1024, 64 rows 56.1 and 51.1. Not all: 256 experts of 2816, 32 rows 138.8 and 135.2, 52
    // rows 176.3 and 174.1, 64 rows 189.7 and 190.5; 128 experts, 56 rows 123.8 and 125.4, 64 rows 129.3 and 132.2. A call without
    // grouping has no such launch behind it.
    const bool late = gridDim.x <= kRowsLateRows || resident;
    if (!late || grp.sorted_pairs == nullptr) pdl_launch_dependents();
    // expert rows (contiguous in every plane; d is a multiple of 64 and the planes are 16-byte aligned by contract)
    {
        const uint8_t* wsrc = W + (size_t)e0 * d;
        for (uint32_t i = threadIdx.x; i < ne * d / 16; i += kRowsThreads)
            reinterpret_cast<uint4*>(wrows)[i] = ldg_nc_u4(wsrc + (size_t)i * 16);
        for (uint32_t i = threadIdx.x; i < ne * groups; i += kRowsThreads) {
            srows[i] = S[(size_t)e0 * groups + i];
            brows[i] = B[(size_t)e0 * groups + i];
        }
    }
    pdl_wait();          // the weights above do not depend on the previous kernel; the hidden rows do
    for (uint32_t i = threadIdx.x; i < d / 8; i += kRowsThreads) {
        const uint4 ev = __ldg(reinterpret_cast<const uint4*>(eff) + i);
        const uint32_t ew[4] = {ev.x, ev.y, ev.z, ev.w};
        uint4 hv[R];
#pragma unroll
        for (int r = 0; r < R; ++r)
            hv[r] = row0 + r < rows ? reinterpret_cast<const uint4*>(hidden + (size_t)(row0 + r) * hidden_stride)[i]
                                    : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t hw[4] = {hv[r].x, hv[r].y, hv[r].z, hv[r].w};
            float o[8];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint16_t h0 = (uint16_t)(hw[q] & 0xFFFFu), h1 = (uint16_t)(hw[q] >> 16);
                const float f0 = X_BF16 ? bf16_bits_to_float(h0) : f16_bits_to_float(h0);
                const float f1 = X_BF16 ? bf16_bits_to_float(h1) : f16_bits_to_float(h1);
                o[2 * q] = __fmul_rn(f0, bf16_bits_to_float((uint16_t)(ew[q] & 0xFFFFu)));
                o[2 * q + 1] = __fmul_rn(f1, bf16_bits_to_float((uint16_t)(ew[q] >> 16)));
            }
            float4* dst = reinterpret_cast<float4*>(xf + (size_t)r * d + i * 8);
            dst[0] = make_float4(o[0], o[1], o[2], o[3]);
            dst[1] = make_float4(o[4], o[5], o[6], o[7]);
        }
    }
    __syncthreads();

    if ((uint32_t)warp < ne) {
        const uint8_t* wr = wrows + (size_t)warp * d;
        const uint16_t* sr = srows + warp * groups;
        const uint16_t* br = brows + warp * groups;
        float acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = 0.0f;
#pragma unroll 2
        for (uint32_t g = 0; g < groups; ++g) {
            const uint32_t i0 = g * kGroup + lane * 2;
            const uint32_t w = *reinterpret_cast<const uint16_t*>(wr + i0);
            // byte -> float through the 2^23 mantissa trick (exact for 0...255)
            const float q0 = __uint_as_float(0x4B000000u | (w & 0xFFu)) - 8388608.0f;
            const float q1 = __uint_as_float(0x4B000000u | (w >> 8)) - 8388608.0f;
            const float sc = bf16_bits_to_float(sr[g]);
            const float bi = bf16_bits_to_float(br[g]);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 xv = *reinterpret_cast<const float2*>(xf + (size_t)r * d + i0);
                const float p = __fmaf_rn(q1, xv.y, __fmul_rn(q0, xv.x));
                acc[r] = __fmaf_rn(sc, p, acc[r]);
                acc[r] = __fmaf_rn(bi, __fadd_rn(xv.x, xv.y), acc[r]);
            }
        }
        const uint32_t e = e0 + warp;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float logit = warp_sum(acc[r]);
            if (logit_bias) logit = __fadd_rn(logit, logit_bias[e]);
            if (lane == 0 && row0 + r < rows) scratch_logits[(size_t)(row0 + r) * TF_MAX_ROUTER_EXPERTS + e] = logit;
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int tk = atomicAdd(&tickets[blockIdx.x], 1u);
        is_last = (tk == gridDim.y - 1);
        if (is_last) tickets[blockIdx.x] = 0;            // ready for the next launch on this stream
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (uint32_t i = threadIdx.x; i < R * num_experts; i += kRowsThreads) {
        const uint32_t r = i / num_experts, e = i % num_experts;
        if (row0 + r < rows) {
            const float v = __ldcg(&scratch_logits[(size_t)(row0 + r) * TF_MAX_ROUTER_EXPERTS + e]);
            scores[r][e] = v;
            if (out_logits) out_logits[(size_t)(row0 + r) * num_experts + e] = v;
        }
    }
    __syncthreads();
    if (warp < R && row0 + warp < rows)
        warp_select_topk(scores[warp], num_experts, top_k, per_expert_scale, out_idx + (size_t)(row0 + warp) * top_k,
                         out_w + (size_t)(row0 + warp) * top_k, lane);
    if (grp.sorted_pairs == nullptr) return;
    // the block that completes the last row group groups all rows (second ticket, after the row tickets)
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int tk = atomicAdd(&tickets[kRouterSplitRows], 1u);
        is_last = (tk == gridDim.x - 1);
        if (is_last) tickets[kRouterSplitRows] = 0;
    }
    __syncthreads();
    if (!is_last) return;
    if (late) pdl_launch_dependents();
    __threadfence();
    group_routes_in_block<true>(out_idx, out_w, rows, top_k, num_experts, grp, smem);
}

// Many rows (batched decode, prefill): one block per row.
template <bool X_BF16>
__global__ void __launch_bounds__(kBlockRouterThreads)
router_block_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                    const uint16_t* hidden, uint32_t hidden_stride,
                    const uint16_t* __restrict__ eff, const uint16_t* __restrict__ per_expert_scale,
                    const float* __restrict__ logit_bias,
                    uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w, float* __restrict__ out_logits,
                    uint32_t num_experts, uint32_t d, uint32_t top_k, bool a2) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* xf = reinterpret_cast<float*>(smem);
    __shared__ float scores[TF_MAX_ROUTER_EXPERTS];
    const uint32_t row = blockIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    stage_router_x<X_BF16>(hidden + (size_t)row * hidden_stride, eff, xf, d);
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t groups = d / kGroup;
    for (uint32_t e = warp; e < num_experts; e += kBlockRouterThreads / kWarp) {
        float logit = router_row_logit(W + (size_t)e * d, S + (size_t)e * groups, B + (size_t)e * groups, xf, groups, lane, a2);
        if (logit_bias) logit = __fadd_rn(logit, logit_bias[e]);
        if (lane == 0) {
            scores[e] = logit;
            if (out_logits) out_logits[(size_t)row * num_experts + e] = logit;
        }
    }
    __syncthreads();
    // the form for any number of experts: with the choice between two of them this kernel is 0.4 us slower (200 rows of 256: 21.4, 20.9)
    if (warp == 0)
        warp_select_topk_held<TF_MAX_ROUTER_EXPERTS / kWarp>(scores, num_experts, top_k, per_expert_scale, out_idx + (size_t)row * top_k,
                                                             out_w + (size_t)row * top_k, lane);
}

// Prefill-sized batches: one block per R token rows (R = 6, 7 or 8, picked by the host so that the row tiles fill whole
// rounds of the resident blocks). Same canonical arithmetic per (row, expert) as router_row_logit, but an expert's codes,
// scale and bias are decoded once per group for R rows, and a group's activations are read from shared memory once for
// four experts: the rows' scaled activations sit in shared memory as fp32 and every lane carries 4 R accumulators.
constexpr int kTileRouterRows = 8;          // most rows per block (sizes the shared memory)
constexpr int kTileExperts = 4;             // experts per warp iteration
template <bool X_BF16, int R>
__global__ void __launch_bounds__(kBlockRouterThreads, 2)
router_tile_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                   const uint16_t* hidden, uint32_t hidden_stride,
                   const uint16_t* __restrict__ eff, const uint16_t* __restrict__ per_expert_scale,
                   const float* __restrict__ logit_bias,
                   uint32_t* __restrict__ out_idx, uint16_t* __restrict__ out_w, float* __restrict__ out_logits,
                   uint32_t rows, uint32_t num_experts, uint32_t d, uint32_t top_k) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* xf = reinterpret_cast<float*>(smem);                                   // [R][d]
    float* scores = xf + (size_t)R * d;                                           // [R][num_experts]
    const uint32_t row0 = blockIdx.x * R;
    const uint32_t nrows = rows - row0 < (uint32_t)R ? rows - row0 : (uint32_t)R;
    pdl_launch_dependents();
    pdl_wait();
    for (uint32_t c = threadIdx.x; c < d; c += blockDim.x) {
        const float es = bf16_bits_to_float(eff[c]);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float v = 0.0f;
            if ((uint32_t)r < nrows) {
                const uint16_t hb = hidden[(size_t)(row0 + r) * hidden_stride + c];
                v = __fmul_rn(X_BF16 ? bf16_bits_to_float(hb) : f16_bits_to_float(hb), es);
            }
            xf[(size_t)r * d + c] = v;
        }
    }
    __syncthreads();
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t groups = d / kGroup;
    constexpr uint32_t kWarps = kBlockRouterThreads / kWarp;
    // A warp takes four experts at a time (e, e + 8, e + 16, e + 24); experts past the end repeat the first one and
    // are not stored. The next group's codes, scales and biases are on their way while the current group is multiplied.
    for (uint32_t e0 = warp; e0 < num_experts; e0 += kTileExperts * kWarps) {
        uint32_t ex[kTileExperts];
        const uint8_t* Wp[kTileExperts];
        const uint16_t* sp[kTileExperts];
        const uint16_t* bp[kTileExperts];
#pragma unroll
        for (int j = 0; j < kTileExperts; ++j) {
            const uint32_t e = e0 + j * kWarps;
            ex[j] = e < num_experts ? e : e0;
            Wp[j] = W + (size_t)ex[j] * d + lane * 2;
            sp[j] = S + (size_t)ex[j] * groups;
            bp[j] = B + (size_t)ex[j] * groups;
        }
        float acc[kTileExperts][R];
        uint32_t wn[kTileExperts];
        uint16_t sn[kTileExperts], bn[kTileExperts];
#pragma unroll
        for (int j = 0; j < kTileExperts; ++j) {
#pragma unroll
            for (int r = 0; r < R; ++r) acc[j][r] = 0.0f;
            wn[j] = *reinterpret_cast<const uint16_t*>(Wp[j]);          // d % 64 == 0, 2-byte aligned rows
            sn[j] = sp[j][0]; bn[j] = bp[j][0];
        }
        for (uint32_t g = 0; g < groups; ++g) {
            float q0[kTileExperts], q1[kTileExperts], sc[kTileExperts], bi[kTileExperts];
#pragma unroll
            for (int j = 0; j < kTileExperts; ++j) {
                // byte -> float through the 2^23 mantissa trick (exact for 0...255)
                q0[j] = __uint_as_float(0x4B000000u | (wn[j] & 0xFFu)) - 8388608.0f;
                q1[j] = __uint_as_float(0x4B000000u | (wn[j] >> 8)) - 8388608.0f;
                sc[j] = bf16_bits_to_float(sn[j]);
                bi[j] = bf16_bits_to_float(bn[j]);
            }
            if (g + 1 < groups) {
#pragma unroll
                for (int j = 0; j < kTileExperts; ++j) {
                    wn[j] = *reinterpret_cast<const uint16_t*>(Wp[j] + (g + 1) * kGroup);
                    sn[j] = sp[j][g + 1]; bn[j] = bp[j][g + 1];
                }
            }
            const float* xg = xf + g * kGroup + lane * 2;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 xv = *reinterpret_cast<const float2*>(xg + (size_t)r * d);
                const float xs = __fadd_rn(xv.x, xv.y);
#pragma unroll
                for (int j = 0; j < kTileExperts; ++j) {
                    const float p = __fmaf_rn(q1[j], xv.y, __fmul_rn(q0[j], xv.x));
                    acc[j][r] = __fmaf_rn(sc[j], p, acc[j][r]);
                    acc[j][r] = __fmaf_rn(bi[j], xs, acc[j][r]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kTileExperts; ++j) {
            const bool live = e0 + j * kWarps < num_experts;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float l = warp_sum(acc[j][r]);
                if (logit_bias) l = __fadd_rn(l, logit_bias[ex[j]]);
                if (lane == 0 && live && (uint32_t)r < nrows) {
                    scores[r * num_experts + ex[j]] = l;
                    if (out_logits) out_logits[(size_t)(row0 + r) * num_experts + ex[j]] = l;
                }
            }
        }
    }
    __syncthreads();
    if ((uint32_t)warp < nrows)          // eight warps, at most eight rows
        warp_select_topk(scores + warp * num_experts, num_experts, top_k, per_expert_scale, out_idx + (size_t)(row0 + warp) * top_k,
                         out_w + (size_t)(row0 + warp) * top_k, lane);
}

// Rows per block of router_tile_kernel: the R in 6...8 whose tiles leave the fewest idle block slots in the last round
// (rounds x R is the time in units of one row's work).
static int tile_router_rows(uint32_t rows, uint32_t slots) {
    int best = kTileRouterRows;
    uint64_t best_cost = ~0ull;
    for (int r = kTileRouterRows; r >= 6; --r) {
        const uint32_t tiles = (rows + r - 1) / r;
        const uint64_t cost = (uint64_t)((tiles + slots - 1) / slots) * r;
        if (cost < best_cost) { best_cost = cost; best = r; }
    }
    return best;
}

// Scratch of the two-launch router: `parts` planes of (approximate logit, magnitude) per (row, expert), owned by the context and grown
// on demand, to twice its size at least. A buffer that was outgrown stays (see router_approx_replaced): more rows do not always take more
// scratch, since the number of parts falls, so a call of fewer rows than a captured one may be what outgrows it. Growing allocates, which a stream
// that is being captured must not do. There, and where memory runs out, the parts are as many as the buffer holds; false if that is
// none (the caller then takes the one-launch kernel).
static bool router_scratch(tf_context* ctx, cudaStream_t st, uint32_t rows, uint32_t num_experts, uint32_t& parts) {
    const size_t plane = (size_t)rows * num_experts * sizeof(float2), need = plane * parts;
    if (need <= ctx->router_approx_bytes) return true;
    const uint32_t held = (uint32_t)(ctx->router_approx_bytes / plane);       // planes, fewer than `parts`
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        for (uint32_t want : {parts, 1u}) {                   // one plane where there is no memory for all
            if (want <= held) break;
            const size_t bytes = std::max(plane * want, 2 * ctx->router_approx_bytes);
            void* grown = nullptr;
            if (cudaMalloc(&grown, bytes) != cudaSuccess) { cudaGetLastError(); continue; }
            if (ctx->router_approx) ctx->router_approx_replaced[ctx->router_approx_replaced_count++] = ctx->router_approx;
            ctx->router_approx = grown;
            ctx->router_approx_bytes = bytes;
            parts = want;
            return true;
        }
    }
    cudaGetLastError();
    parts = held;
    return held > 0;
}

static RouterGroupOut router_group_out(const tf_device_routes* routes) {
    return RouterGroupOut{static_cast<tf_pair*>(routes->sorted_pairs), static_cast<uint32_t*>(routes->per_expert_offsets),
                          static_cast<uint32_t*>(routes->per_expert_counts), static_cast<tf_group*>(routes->groups),
                          static_cast<uint32_t*>(routes->chunk_group), static_cast<uint32_t*>(routes->chunk_start),
                          static_cast<uint32_t*>(routes->counters)};
}

// See as_used in launch_router.
constexpr uint32_t kRecheckAsUsedRows = 112, kRecheckAsUsedCodes = 262144;

// Scratch of the two-launch router that belongs to the caller's workspace: nothing of the context is shared, so such calls may
// overlap on several streams (the one-launch kernel for more than kRouterSplitRows rows shares nothing either).
struct RouterScratch {
    float2* approx;             // [parts][rows, num_experts]
    size_t bytes;
    unsigned int* ticket;       // zero between calls
};

// routes: the tables of the grouping, when it is wanted; *grouped (may be NULL) tells whether a launch of this call fills
// them (always for at most kRouterSplitRows rows, and with own scratch). own: take the two-launch form whatever the row count.
static tf_status launch_router(tf_context* ctx, void* stream, const uint8_t* W, const uint8_t* S, const uint8_t* B,
                               const uint8_t* hidden, tf_dtype hidden_dtype, const uint8_t* eff, const uint8_t* pes,
                               const float* logit_bias, uint32_t* out_idx, uint8_t* out_w, float* out_logits,
                               uint32_t rows, uint32_t num_experts, uint32_t d, uint32_t top_k, uint32_t stride,
                               const char* name, const tf_device_routes* routes = nullptr, bool* grouped = nullptr, const RouterScratch* own = nullptr) {
    if (grouped) *grouped = routes != nullptr && rows <= (uint32_t)kRouterSplitRows;
    TF_REQUIRE(ctx, aligned(S, 2) && aligned(B, 2) && aligned(hidden, 2) && aligned(eff, 2) && aligned(pes, 2) &&
                        aligned(out_w, 2) && aligned(out_idx, 4),
               TF_ERR_ALIGNMENT, "%s: 16-bit planes must be 2-byte aligned, indices 4-byte aligned", name);
    const bool a2 = aligned(W, 2);
    const size_t smem = (size_t)d * sizeof(float);
    TF_REQUIRE(ctx, smem <= 160 * 1024, TF_ERR_UNSUPPORTED, "%s: D=%u too large", name, d);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool bf = hidden_dtype == TF_BF16;
    auto Sp = reinterpret_cast<const uint16_t*>(S);
    auto Bp = reinterpret_cast<const uint16_t*>(B);
    auto hp = reinterpret_cast<const uint16_t*>(hidden);
    auto ep = reinterpret_cast<const uint16_t*>(eff);
    auto pp = reinterpret_cast<const uint16_t*>(pes);
    auto wp = reinterpret_cast<uint16_t*>(out_w);
    const bool vec16 = aligned(W, 16) && aligned(hp, 16) && aligned(ep, 16) && d % 16 == 0 && stride % 8 == 0;
    // Parts of the approximate logits: a chunk of columns each while two rounds of two blocks per SM hold them all, three chunks, whose loads
    // overlap, beyond that. One chunk, three, all eleven (us): 333 rows 7.5, 17.9, 37.9; 512 rows 14.9, 18.0, 39.0; 800 rows 14.9, 16.9, 38.8;
    // 1500 rows 23.7, 22.4, 45.6; 4096 rows 47.8, 41.0, 48.5 (and adding the planes takes the re-check 9 us less with three).
    const uint32_t apx_blocks = (rows + kApxTokens - 1) / kApxTokens * ((num_experts + kApxExperts - 1) / kApxExperts) * (d / kApxChunk);
    // Few rows: blocks of 8 tokens x 32 experts with all of their operands in flight at once, while they make one round of the SMs: 200 rows,
    // 100 blocks, 9.8 us. Two rounds (333 rows, 168 blocks) take 16.6, the parts of the other kernel 7.5. (Those take 6.2 us at 200 rows. Steps of
    // 30 layers, us, here and with those: 80 tokens 4232, 4253; 100: 4839, 4933; 110: 5517, 5640; 120: 5693, 5463; 150: 6118, 5999; 200: 7001, 6932;
    // 255: 8139, 8111; prefills of 256 5513, 5453, of 290 the same.)
    const size_t smem_few = router_approx_few_smem_bytes(d);
    const dim3 grid_few((rows + kFewTokens - 1) / kFewTokens, (num_experts + kFewExperts - 1) / kFewExperts);
    const bool few = smem_few <= 224 * 1024 && grid_few.x * grid_few.y <= (uint32_t)ctx->sm_count;
    uint32_t parts = few ? 1u : apx_blocks <= 4u * (uint32_t)ctx->sm_count ? d / kApxChunk : (d / kApxChunk + 2) / 3;
    if (rows >= 2 && rows <= (uint32_t)kRouterSplitRows && vec16) {
        constexpr int R = 1;          // latency bound: a 64-token step took 4.35 ms with four rows per block, 4.28 with two, 4.16 with one
        auto k = bf ? router_rows_kernel<true, R> : router_rows_kernel<false, R>;
        size_t smem_rows = (size_t)R * d * 4 + (size_t)kRowsExpertsPerBlock * d + (size_t)kRowsExpertsPerBlock * (d / kGroup) * 4;
        RouterGroupOut grp{};
        if (routes) {
            grp = router_group_out(routes);
            const size_t need = router_group_smem_bytes(rows * top_k, num_experts, true);
            if (need > smem_rows) smem_rows = need;
        }
        TF_REQUIRE(ctx, smem_rows <= 200 * 1024, TF_ERR_UNSUPPORTED, "%s: D=%u too large", name, d);
        static DeviceSmemCache configured_rows[2];
        if (tf_status s2 = ensure_dynamic_smem(ctx, k, configured_rows[bf ? 1 : 0], smem_rows)) return s2;
        dim3 grid((rows + R - 1) / R, (num_experts + kRowsExpertsPerBlock - 1) / kRowsExpertsPerBlock);
        // While all blocks are resident (five per SM at the production width: up to 46 rows of 128 experts), and up to kRowsLateRows rows in
        // any case, the next launch is let in late, see the kernel.
        static ResidentBlocksCache held[2];
        const bool resident = grid.x * grid.y <= resident_blocks(ctx, k, held[bf ? 1 : 0], kRowsThreads, smem_rows);
        launch_pdl(k, grid, dim3(kRowsThreads), smem_rows, st, W, Sp, Bp, hp, stride, ep, pp, logit_bias, out_idx, wp, out_logits,
                   ctx->router_logits, ctx->router_tickets, grp, rows, num_experts, d, top_k, resident);
        return check_launch(ctx, name);
    }
    if (rows <= (uint32_t)kRouterSplitRows) {
        dim3 grid(rows, (num_experts + kSplitExpertsPerBlock - 1) / kSplitExpertsPerBlock);
        auto k = bf ? router_split_kernel<true> : router_split_kernel<false>;
        size_t smem_split = (size_t)d * 4 + (size_t)kSplitExpertsPerBlock * d + (size_t)kSplitExpertsPerBlock * (d / kGroup) * 4;
        RouterGroupOut grp{};
        if (routes) {
            grp = router_group_out(routes);
            const size_t need = router_group_smem_bytes(rows * top_k, num_experts, false);
            if (need > smem_split) smem_split = need;
        }
        TF_REQUIRE(ctx, smem_split <= 200 * 1024, TF_ERR_UNSUPPORTED, "%s: D=%u too large", name, d);
        if (smem_split > 40 * 1024) TF_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_split));
        launch_pdl(k, grid, dim3(kSplitThreads), smem_split, st, W, Sp, Bp, hp, stride, ep, pp, logit_bias, out_idx, wp, out_logits,
                   ctx->router_logits, ctx->router_tickets, grp, num_experts, d, top_k, a2);
        return check_launch(ctx, name);
    } else if ((own || rows >= ctx->router_tensorcore_min_rows) && !out_logits && vec16 && d % kApxChunk == 0 && aligned(S, 8) && aligned(B, 8) &&
               num_experts <= TF_MAX_ROUTER_EXPERTS && top_k <= (uint32_t)kWarp && top_k <= num_experts &&
               router_recheck_smem_bytes(d, num_experts, kRecheckWarps) <= 205 * 1024 && (own || router_scratch(ctx, st, rows, num_experts, parts))) {
        // logits on the tensor cores, then the canonical logits of the few experts that can reach the top k
        float2* approx = own ? own->approx : static_cast<float2*>(ctx->router_approx);
        const uint32_t sms = (uint32_t)ctx->sm_count;
        if (few) {
            auto ka = bf ? router_approx_few_kernel<true> : router_approx_few_kernel<false>;
            static DeviceSmemCache configured_few[2];
            if (tf_status s = ensure_dynamic_smem(ctx, ka, configured_few[bf ? 1 : 0], smem_few)) return s;
            launch_pdl(ka, grid_few, dim3(kFewThreads), smem_few, st, W, Sp, Bp, hp, stride, ep, approx, rows, num_experts, d);
        } else {
            if (own) parts = std::max(1u, std::min(parts, (uint32_t)(own->bytes / ((size_t)rows * num_experts * sizeof(float2)))));
            const uint32_t chunks = (d / kApxChunk + parts - 1) / parts;
            parts = (d / kApxChunk + chunks - 1) / chunks;
            auto ka = bf ? router_approx_kernel<true> : router_approx_kernel<false>;
            static DeviceSmemCache configured_approx[2];
            if (tf_status s = ensure_dynamic_smem(ctx, ka, configured_approx[bf ? 1 : 0], router_approx_smem_bytes(2))) return s;
            launch_pdl(ka, dim3((rows + kApxTokens - 1) / kApxTokens, (num_experts + kApxExperts - 1) / kApxExperts, parts), dim3(kApxThreads),
                       router_approx_smem_bytes(chunks), st, W, Sp, Bp, hp, stride, ep, approx, rows, num_experts, d, chunks);
        }
        if (tf_status s = check_launch(ctx, name)) return s;
        constexpr int kProductionGroups = 2816 / kGroup;          // the recheck keeps an expert's 44 code words in registers
        const bool fixed = d / kGroup == (uint32_t)kProductionGroups;
        // Warps per token: as many as leave the rows in one round of two blocks per SM. A warp that takes all of a token's
        // candidates one after the other needs about 30 us however few rows there are.
        // (Only the form with a token per block can group.)
        const int which = rows <= 2 * sms || (own && routes) ? 3 : rows <= 4 * sms ? 2 : rows <= 8 * sms ? 1 : 0;
        // Blocks of few rows and many experts read the approximate logits where they are used: a re-check that requests them ahead ends earlier, and
        // the routed gate/up launch that it lets in then takes the SMs on which the shared expert's down launch would run beside it. Steps of
        // 30 layers of 128 experts x 2816, us, as used and ahead: 75 tokens 4129, 4129; 90: 4525, 4566; 98: 4820, 4992; 105: 5443, 5650; 112: 5545,
        // 5654; 115: 5655, 5636; 120: 5691, 5657; 150: 6258, 6135. Blocks of 128 x 1024, 90 to 110 tokens: 67 to 69, 63 to 66; of 64 x 2816 the same.
        const bool as_used = own && routes && parts == 1 && rows <= kRecheckAsUsedRows && num_experts * d > kRecheckAsUsedCodes;
        void (*kr)(const uint8_t*, const uint16_t*, const uint16_t*, const uint16_t*, uint32_t, const uint16_t*, const uint16_t*, const float*,
                   const float2*, uint32_t, uint32_t*, uint16_t*, unsigned int*, RouterGroupOut, uint32_t, uint32_t, uint32_t, uint32_t);
#define TF_RECHECK(WPT) kr = fixed ? (bf ? router_recheck_kernel<true, kProductionGroups, WPT> : router_recheck_kernel<false, kProductionGroups, WPT>) \
                                   : (bf ? router_recheck_kernel<true, 0, WPT> : router_recheck_kernel<false, 0, WPT>)
        if (as_used)
            kr = fixed ? (bf ? router_recheck_kernel<true, kProductionGroups, 8, false> : router_recheck_kernel<false, kProductionGroups, 8, false>)
                       : (bf ? router_recheck_kernel<true, 0, 8, false> : router_recheck_kernel<false, 0, 8, false>);
        else if (which == 3) TF_RECHECK(8);
        else if (which == 2) TF_RECHECK(4);
        else if (which == 1) TF_RECHECK(2);
        else TF_RECHECK(1);
#undef TF_RECHECK
        const uint32_t per_block = (uint32_t)kRecheckWarps >> which;
        size_t smem_r = router_recheck_smem_bytes(d, num_experts, per_block) + (fixed && which > 0 ? router_recheck_code_bytes(d) : 0);
        RouterGroupOut grp{};
        if (own && routes) {
            grp = router_group_out(routes);
            const size_t need = router_group_rows_smem_bytes(rows * top_k, num_experts);
            if (need > smem_r) smem_r = need;
        }
        static DeviceSmemCache configured_recheck[5][4];
        if (tf_status s = ensure_dynamic_smem(ctx, kr, configured_recheck[as_used ? 4 : which][(bf ? 1 : 0) + (fixed ? 2 : 0)], smem_r)) return s;
        launch_pdl(kr, dim3((rows + per_block - 1) / per_block), dim3(kRecheckWarps * kWarp), smem_r, st, W, Sp, Bp, hp, stride,
                   ep, pp, logit_bias, static_cast<const float2*>(approx), parts, out_idx, wp, own ? own->ticket : nullptr, grp, rows, num_experts, d, top_k);
        if (grouped) *grouped = own && routes;
    } else if (rows >= 256 && a2 && (size_t)kTileRouterRows * (d + num_experts) * 4 <= 100 * 1024) {
        const int R = tile_router_rows(rows, (uint32_t)ctx->sm_count * 2u);
        void (*k)(const uint8_t*, const uint16_t*, const uint16_t*, const uint16_t*, uint32_t, const uint16_t*, const uint16_t*, const float*,
                  uint32_t*, uint16_t*, float*, uint32_t, uint32_t, uint32_t, uint32_t);
        if (R == 6) k = bf ? router_tile_kernel<true, 6> : router_tile_kernel<false, 6>;
        else if (R == 7) k = bf ? router_tile_kernel<true, 7> : router_tile_kernel<false, 7>;
        else k = bf ? router_tile_kernel<true, 8> : router_tile_kernel<false, 8>;
        const size_t smem_tile = (size_t)R * (d + num_experts) * 4;
        static DeviceSmemCache configured[2][3];
        if (tf_status s = ensure_dynamic_smem(ctx, k, configured[bf ? 1 : 0][R - 6], smem_tile)) return s;
        launch_pdl(k, dim3((rows + R - 1) / R), dim3(kBlockRouterThreads), smem_tile, st, W, Sp, Bp, hp, stride,
                   ep, pp, logit_bias, out_idx, wp, out_logits, rows, num_experts, d, top_k);
    } else {
        auto k = bf ? router_block_kernel<true> : router_block_kernel<false>;
        if (smem > 40 * 1024) TF_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        launch_pdl(k, dim3(rows), dim3(kBlockRouterThreads), smem, st, W, Sp, Bp, hp, stride, ep, pp, logit_bias, out_idx, wp, out_logits,
                   num_experts, d, top_k, a2);
    }
    return check_launch(ctx, name);
}

// tf_router_gemma4_block_grouped; approx_scratch ([query_count, num_experts] pairs of floats) and ticket (a zero word), when
// given, belong to the caller's workspace: blocks of 65 to kRouterFusedGroupRows rows then route in two launches, the second of
// which groups them (the block that finishes the last row does it). One block per row computes every canonical logit there
// otherwise: 168 us and a grouping launch against 10 + 27 for 200 rows. Larger blocks group with launches of their own, which many SMs share; nothing between the two was measured.
// The one launch grows with experts * D and the two hardly do. Blocks of 65, 130 and 255 tokens gain from two by, in us: 16 x 256 -13,
// -16, -17; 32 x 1024 -1, -3, -6; 64 x 768 6, 5, 0; 128 x 512 0, -3, -5; 64 x 1024 13, 11, 8; 32 x 2816 20, 20, 18; 128 x 1024 43, 43, 41.
constexpr uint32_t kRouterTwoLaunchCodes = 65536;
tf_status router_block_grouped(tf_context* ctx, void* stream, const void* weights, uint64_t weights_off,
                               const void* scales, uint64_t scales_off, const void* biases, uint64_t biases_off,
                               const void* hidden, uint64_t hidden_off, tf_dtype hidden_dtype,
                               const void* effective_scale, uint64_t effective_scale_off,
                               const void* per_expert_scale, uint64_t per_expert_scale_off,
                               const float* logit_bias, uint32_t* out_indices, void* out_weights,
                               uint32_t query_count, uint32_t num_experts, uint32_t d, uint32_t top_k,
                               uint32_t hidden_stride_elements, const tf_device_routes* routes, void* approx_scratch, size_t approx_bytes, uint32_t* ticket) {
    const char* name = "tf_router_gemma4_block_grouped";
    TF_REQUIRE(ctx, weights && scales && biases && hidden && effective_scale && per_expert_scale && out_indices && out_weights,
               TF_ERR_INVALID_ARGUMENT, "%s: NULL buffer", name);
    TF_REQUIRE(ctx, query_count > 0, TF_ERR_INVALID_ARGUMENT, "%s: queryCount must be positive", name);
    TF_REQUIRE(ctx, num_experts > 0 && num_experts <= TF_MAX_ROUTER_EXPERTS, TF_ERR_INVALID_ARGUMENT,
               "%s: numExperts > 256 is not supported", name);
    TF_REQUIRE(ctx, top_k > 0 && top_k <= TF_MAX_TOP_K && num_experts >= top_k, TF_ERR_INVALID_ARGUMENT,
               "%s: topK must be in 1...%d and at most numExperts, got %u", name, TF_MAX_TOP_K, top_k);
    TF_REQUIRE(ctx, d > 0 && d % tf::kGroup == 0 && hidden_stride_elements >= d, TF_ERR_INVALID_ARGUMENT,
               "%s: D must be a multiple of 64 and the stride at least D", name);
    TF_REQUIRE(ctx, hidden_dtype == TF_FP16 || hidden_dtype == TF_BF16, TF_ERR_INVALID_ARGUMENT, "%s: bad hidden dtype", name);
    const RouterScratch own{static_cast<float2*>(approx_scratch), approx_bytes, ticket};
    const bool use_own = approx_scratch && ticket && query_count > (uint32_t)kRouterSplitRows && query_count <= kRouterFusedGroupRows &&
                         (ctx->router_block_min_rows ? query_count >= ctx->router_block_min_rows : num_experts * d > kRouterTwoLaunchCodes);
    bool grouped = false;
    tf_status s = launch_router(ctx, stream, byte_ptr(weights, weights_off), byte_ptr(scales, scales_off),
                                byte_ptr(biases, biases_off), byte_ptr(hidden, hidden_off), hidden_dtype,
                                byte_ptr(effective_scale, effective_scale_off),
                                byte_ptr(per_expert_scale, per_expert_scale_off), logit_bias, out_indices,
                                static_cast<uint8_t*>(out_weights), nullptr, query_count, num_experts, d, top_k,
                                hidden_stride_elements, name, routes, &grouped, use_own ? &own : nullptr);
    if (s || grouped) return s;
    return tf_group_routes_device(ctx, stream, out_indices, out_weights, query_count, top_k, num_experts, routes);
}

}  // namespace tf

extern "C" {

tf_status tf_router_gemma4(tf_context* ctx, void* stream, const void* weights, uint64_t weights_off,
                           const void* scales, uint64_t scales_off, const void* biases, uint64_t biases_off,
                           const void* hidden, const void* effective_scale, uint64_t effective_scale_off,
                           const void* per_expert_scale, uint64_t per_expert_scale_off,
                           uint32_t* out_indices, void* out_weights, float* out_logits,
                           uint32_t num_experts, uint32_t d, uint32_t top_k) {
    const char* name = "tf_router_gemma4";
    TF_REQUIRE(ctx, ctx != nullptr, TF_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", name);
    TF_REQUIRE(ctx, weights && scales && biases && hidden && effective_scale && per_expert_scale && out_indices && out_weights,
               TF_ERR_INVALID_ARGUMENT, "%s: NULL buffer", name);
    TF_REQUIRE(ctx, d > 0 && d % tf::kGroup == 0, TF_ERR_INVALID_ARGUMENT, "%s: D=%u must be a multiple of 64", name, d);
    TF_REQUIRE(ctx, num_experts > 0 && num_experts <= TF_MAX_ROUTER_EXPERTS, TF_ERR_INVALID_ARGUMENT,
               "%s: numExperts=%u must be in 1...256", name, num_experts);
    TF_REQUIRE(ctx, top_k == TF_MAX_TOP_K, TF_ERR_INVALID_ARGUMENT, "%s: topK must be 8, got %u", name, top_k);
    TF_REQUIRE(ctx, num_experts >= top_k, TF_ERR_INVALID_ARGUMENT, "%s: numExperts < topK", name);
    return tf::launch_router(ctx, stream, tf::byte_ptr(weights, weights_off), tf::byte_ptr(scales, scales_off),
                             tf::byte_ptr(biases, biases_off), static_cast<const uint8_t*>(hidden), TF_FP16,
                             tf::byte_ptr(effective_scale, effective_scale_off),
                             tf::byte_ptr(per_expert_scale, per_expert_scale_off), nullptr, out_indices,
                             static_cast<uint8_t*>(out_weights), out_logits, 1, num_experts, d, top_k, d, name);
}

tf_status tf_router_gemma4_block(tf_context* ctx, void* stream, const void* weights, uint64_t weights_off,
                                 const void* scales, uint64_t scales_off, const void* biases, uint64_t biases_off,
                                 const void* hidden, uint64_t hidden_off, tf_dtype hidden_dtype,
                                 const void* effective_scale, uint64_t effective_scale_off,
                                 const void* per_expert_scale, uint64_t per_expert_scale_off,
                                 const float* logit_bias,
                                 uint32_t* out_indices, uint64_t out_indices_off,
                                 void* out_weights, uint64_t out_weights_off, float* out_logits,
                                 uint32_t query_count, uint32_t num_experts, uint32_t d,
                                 uint32_t top_k, uint32_t hidden_stride_elements) {
    const char* name = "tf_router_gemma4_block";
    TF_REQUIRE(ctx, ctx != nullptr, TF_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", name);
    TF_REQUIRE(ctx, weights && scales && biases && hidden && effective_scale && per_expert_scale && out_indices && out_weights,
               TF_ERR_INVALID_ARGUMENT, "%s: NULL buffer", name);
    TF_REQUIRE(ctx, query_count > 0, TF_ERR_INVALID_ARGUMENT, "%s: queryCount must be positive", name);
    TF_REQUIRE(ctx, num_experts > 0 && num_experts <= TF_MAX_ROUTER_EXPERTS, TF_ERR_INVALID_ARGUMENT,
               "%s: numExperts > 256 is not supported", name);
    TF_REQUIRE(ctx, top_k > 0 && top_k <= TF_MAX_TOP_K, TF_ERR_INVALID_ARGUMENT,
               "%s: topK must be in 1...%d, got %u", name, TF_MAX_TOP_K, top_k);
    TF_REQUIRE(ctx, num_experts >= top_k, TF_ERR_INVALID_ARGUMENT, "%s: numExperts < topK", name);
    TF_REQUIRE(ctx, d > 0 && d % tf::kGroup == 0, TF_ERR_INVALID_ARGUMENT, "%s: D must be a multiple of 64", name);
    TF_REQUIRE(ctx, hidden_stride_elements >= d, TF_ERR_INVALID_ARGUMENT, "%s: hidden stride is too small", name);
    TF_REQUIRE(ctx, hidden_dtype == TF_FP16 || hidden_dtype == TF_BF16, TF_ERR_INVALID_ARGUMENT, "%s: bad hidden dtype", name);
    return tf::launch_router(ctx, stream, tf::byte_ptr(weights, weights_off), tf::byte_ptr(scales, scales_off),
                             tf::byte_ptr(biases, biases_off), tf::byte_ptr(hidden, hidden_off), hidden_dtype,
                             tf::byte_ptr(effective_scale, effective_scale_off),
                             tf::byte_ptr(per_expert_scale, per_expert_scale_off), logit_bias,
                             reinterpret_cast<uint32_t*>(tf::byte_ptr(static_cast<void*>(out_indices), out_indices_off)),
                             tf::byte_ptr(out_weights, out_weights_off), out_logits, query_count, num_experts, d, top_k,
                             hidden_stride_elements, name);
}

tf_status tf_router_gemma4_block_grouped(tf_context* ctx, void* stream, const void* weights, uint64_t weights_off,
                                         const void* scales, uint64_t scales_off, const void* biases, uint64_t biases_off,
                                         const void* hidden, uint64_t hidden_off, tf_dtype hidden_dtype,
                                         const void* effective_scale, uint64_t effective_scale_off,
                                         const void* per_expert_scale, uint64_t per_expert_scale_off,
                                         const float* logit_bias, uint32_t* out_indices, void* out_weights,
                                         uint32_t query_count, uint32_t num_experts, uint32_t d, uint32_t top_k,
                                         uint32_t hidden_stride_elements, const tf_device_routes* routes) {
    const char* name = "tf_router_gemma4_block_grouped";
    TF_REQUIRE(ctx, ctx != nullptr, TF_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", name);
    TF_REQUIRE(ctx, routes && routes->sorted_pairs && routes->per_expert_offsets && routes->per_expert_counts && routes->groups &&
                        routes->chunk_group && routes->chunk_start && routes->counters,
               TF_ERR_INVALID_ARGUMENT, "%s: NULL routes buffer", name);
    return tf::router_block_grouped(ctx, stream, weights, weights_off, scales, scales_off, biases, biases_off, hidden, hidden_off, hidden_dtype,
                                    effective_scale, effective_scale_off, per_expert_scale, per_expert_scale_off, logit_bias, out_indices,
                                    out_weights, query_count, num_experts, d, top_k, hidden_stride_elements, routes, nullptr, 0, nullptr);
}

}  // extern "C"
