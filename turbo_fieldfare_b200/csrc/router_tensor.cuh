// Router of prefill-sized batches in two launches, with the same indices and weights as the canonical fp32 router
// (Metal/MoE/moe.metal:135-185 fixes a per-logit order of fp32 operations; router_row_logit restates it).
//
//   1. router_approx_kernel: all logits on the tensor cores (mma.sync.m16n8k16, fp32 accumulation). The 8-bit codes
//      enter the A operand as exact fp16 integers; an activation x is split into two fp16 numbers hi + lo of
//      x * 2^10, so the operands carry the inputs (nearly) exactly and the only differences from the canonical value
//      are rounding errors of the sums. Beside each logit the kernel accumulates a MAGNITUDE
//      sum_g (255 |s_g| + |b_g|) * (sum_{i in g} |x_i|), an upper bound of the sum of |terms| of either evaluation.
//   2. router_recheck_kernel: per token, eps_e = kRelError * magnitude_e bounds |approximate - canonical| (derivation
//      below). With lower_e = v_e - eps_e and upper_e = v_e + eps_e, the top_k-th largest lower value LB is reached by
//      top_k canonical logits, so an expert with upper_e < LB cannot be among the canonical top_k, whatever the ties.
//      All other experts (typically top_k plus one or two) get their canonical logit computed in the canonical
//      order, and the usual top-k + softmax runs over those. Rows with a non-finite value anywhere re-check every expert.
//
// Error budget behind kRelError = 2^-13 (relative to the magnitude, which over-estimates sum |terms| by about 1.5):
//   canonical order: a term passes at most 2 + 2 * groups + 5 fp32 roundings, 95 * 2^-24 = 5.7e-6 at 44 groups;
//   tensor cores: products of fp16 numbers are exact in fp32; a k = 16 step adds 16 products and the accumulator with
//     aligned, truncated addends, at most 18 * 2^-23 of the step's magnitude; 8 steps per group: 1.7e-5;
//   the group epilogue and the 88 accumulations behind it: 5.3e-6; the group sums of x: 1e-6;
//   the fp16 split: |x * 2^10 - hi - lo| <= 2^-22 |x * 2^10| + 2^-25, the absolute part is added to the group's |x| sum.
//   Sum 2.9e-5, kRelError = 1.2e-4 leaves a factor four.
#pragma once

#include <cuda_fp16.h>

#include "router.cuh"

namespace tf {

constexpr int kApxTokens = 16;                     // tokens per block of router_approx_kernel (two n = 8 tiles)
constexpr int kApxExperts = 128;                   // experts per block: eight warps, one 16-row MMA tile each
constexpr int kApxChunk = 256;                     // columns staged at a time (four groups)
constexpr int kApxWPitch = kApxChunk + 64;         // bytes per staged weight row: the rows of a quarter-warp load fill all banks
constexpr int kApxXPitch = kApxChunk * 2 + 16;     // bytes per staged activation row (fp16): the same for the B fragments
constexpr int kApxThreads = 256;
constexpr float kApxPrescale = 1024.0f;            // activations are split as x * 2^10 = hi + lo
constexpr float kApxRelError = 1.220703125e-04f;   // 2^-13
constexpr int kRecheckWarps = 8;                   // warps per block of router_recheck_kernel

__host__ __device__ inline size_t router_approx_smem_bytes(uint32_t chunks) {        // one weight buffer for parts of one chunk
    return (chunks > 1 ? 2 : 1) * (size_t)kApxExperts * kApxWPitch + 2 * (size_t)kApxTokens * kApxXPitch + 2 * 4 * kApxTokens * sizeof(float);
}
__host__ __device__ inline size_t router_recheck_smem_bytes(uint32_t d, uint32_t num_experts, uint32_t tokens_per_block) {
    return ((size_t)tokens_per_block * (((size_t)d + num_experts) * sizeof(float) + num_experts * sizeof(uint16_t)) + 15) & ~(size_t)15;
}
// Two expert rows per warp, where the re-check stages them (see router_logit_staged).
__host__ __device__ inline size_t router_recheck_code_bytes(uint32_t d) { return (size_t)kRecheckWarps * 2 * d; }

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* global_src) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(global_src) : "memory");
}

__device__ __forceinline__ void mma_f16_f32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Two bytes of `word` (selected by `sel`) as two exact fp16 integers: the bytes become the low mantissa bits of
// 1024 + byte (0x6400 | byte), then 1024 is subtracted.
__device__ __forceinline__ uint32_t bytes_to_half2(uint32_t word, uint32_t sel) {
    const uint32_t biased = __byte_perm(word, 0x64646464u, sel);
    const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&biased), __half2half2(__ushort_as_half((unsigned short)0x6400)));
    return *reinterpret_cast<const uint32_t*>(&v);
}

// out[token][expert] = (approximate logit without the logit bias, magnitude), both in units of x (not x * 2^10).
// Grid: (ceil(rows / 16), ceil(num_experts / 128), parts); a part sums `chunks` chunks of 256 columns into its own plane of out, and the
// re-check adds the planes. A chunk alone is a chain of latencies (rows, conversion, MMAs, store), eleven in a row took 41 us at 512 rows
// with 32 blocks; see launch_router for the split. The weights, scales and biases are requested before the previous kernel has ended. Column k of an MMA step is mapped to the matrix column
// 16 t + 4 step + {0, 1} (k = 2 t + {0, 1}) and 16 t + 4 step + {2, 3} (k = 2 t + 8 + {0, 1}) of the group, for both
// operands, so a thread's 16 weight bytes and 16 activation values of a group are contiguous.
template <bool X_BF16>
__global__ void __launch_bounds__(kApxThreads, 2)
router_approx_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                     const uint16_t* hidden, uint32_t hidden_stride, const uint16_t* __restrict__ eff,
                     float2* __restrict__ out, uint32_t rows, uint32_t num_experts, uint32_t d, uint32_t chunks) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint8_t* Wc0 = smem;                                                   // [2 or 1][128][kApxWPitch]
    uint8_t* Hi = Wc0 + (chunks > 1 ? 2 : 1) * (size_t)kApxExperts * kApxWPitch;             // [16][kApxXPitch]
    uint8_t* Lo = Hi + (size_t)kApxTokens * kApxXPitch;
    float* XS = reinterpret_cast<float*>(Lo + (size_t)kApxTokens * kApxXPitch);   // [4 groups][16 tokens]: sum of x * 2^10
    float* XA = XS + 4 * kApxTokens;                                       // the same of |x * 2^10| (+ the split's absolute part)
    const int tid = threadIdx.x, warp = tid / kWarp, lane = tid % kWarp, g = lane >> 2, t = lane & 3;
    const uint32_t tok0 = blockIdx.x * kApxTokens, e0 = blockIdx.y * kApxExperts;
    const uint32_t groups = d / kGroup;
    const uint32_t last = num_experts - 1;
    const uint32_t e_lo = min(e0 + warp * 16 + g, last), e_hi = min(e0 + warp * 16 + g + 8, last);   // rows past the end repeat the last one
    const uint32_t c_first = blockIdx.z * chunks * kApxChunk, c_end = min(c_first + chunks * kApxChunk, d);
    out += (size_t)blockIdx.z * rows * num_experts;
    pdl_launch_dependents();
    float acc[2][4] = {}, mag[2][4] = {};
    // The next chunk's weight codes (cp.async into the other buffer) and activation rows (registers) are requested
    // before the current chunk is multiplied.
    auto request_weights = [&](uint32_t c0, uint8_t* dst) {
#pragma unroll
        for (int i = 0; i < (kApxExperts * kApxChunk / 16) / kApxThreads; ++i) {
            const uint32_t idx = tid + kApxThreads * i, row = idx >> 4, seg = idx & 15;
            const uint32_t e = min(e0 + row, last);
            cp_async_16(dst + (size_t)row * kApxWPitch + seg * 16, W + (size_t)e * d + c0 + seg * 16);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    uint4 hreg[2], ereg;
    auto request_rows = [&](uint32_t c0) {
        ereg = *reinterpret_cast<const uint4*>(eff + c0 + lane * 8);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t tok = tok0 + warp + 8 * h;
            hreg[h] = tok < rows ? *reinterpret_cast<const uint4*>(hidden + (size_t)tok * hidden_stride + c0 + lane * 8) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    // scales and biases of a chunk's four groups for this thread's two expert rows (8-byte aligned: groups % 4 == 0)
    uint2 s_lo, s_hi, b_lo, b_hi;
    auto request_scales = [&](uint32_t c0) {
        const uint32_t gq = c0 / kGroup;
        s_lo = __ldg(reinterpret_cast<const uint2*>(S + (size_t)e_lo * groups + gq));
        s_hi = __ldg(reinterpret_cast<const uint2*>(S + (size_t)e_hi * groups + gq));
        b_lo = __ldg(reinterpret_cast<const uint2*>(B + (size_t)e_lo * groups + gq));
        b_hi = __ldg(reinterpret_cast<const uint2*>(B + (size_t)e_hi * groups + gq));
    };
    request_weights(c_first, Wc0);
    request_scales(c_first);
    pdl_wait();                                  // the activations
    request_rows(c_first);
    uint32_t ci = 0;
    for (uint32_t c0 = c_first; c0 < c_end; c0 += kApxChunk, ++ci) {
        uint8_t* Wc = Wc0 + (size_t)(ci & 1u) * kApxExperts * kApxWPitch;
        __syncthreads();                         // the previous chunk's fragments have been read
        // activations: a warp stages the 256 columns of tokens `warp` and `warp + 8`, eight columns per lane (zero bits
        // are +0 in fp16 and bf16: rows past the end contribute nothing)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t tl = warp + 8 * h;
            float y[8];
            const uint32_t hw[4] = {hreg[h].x, hreg[h].y, hreg[h].z, hreg[h].w}, ew[4] = {ereg.x, ereg.y, ereg.z, ereg.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint16_t h0 = (uint16_t)(hw[j] & 0xFFFFu), h1 = (uint16_t)(hw[j] >> 16);
                const float x0 = __fmul_rn(X_BF16 ? bf16_bits_to_float(h0) : f16_bits_to_float(h0), bf16_bits_to_float((uint16_t)(ew[j] & 0xFFFFu)));
                const float x1 = __fmul_rn(X_BF16 ? bf16_bits_to_float(h1) : f16_bits_to_float(h1), bf16_bits_to_float((uint16_t)(ew[j] >> 16)));
                y[2 * j] = x0 * kApxPrescale;
                y[2 * j + 1] = x1 * kApxPrescale;
            }
            uint32_t hiw[4], low[4];
            float sum = 0.0f, asum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 hh = __floats2half2_rn(y[2 * j], y[2 * j + 1]);
                const float2 hf = __half22float2(hh);
                const __half2 ll = __floats2half2_rn(y[2 * j] - hf.x, y[2 * j + 1] - hf.y);
                hiw[j] = *reinterpret_cast<const uint32_t*>(&hh);
                low[j] = *reinterpret_cast<const uint32_t*>(&ll);
                sum += y[2 * j] + y[2 * j + 1];
                asum += fabsf(y[2 * j]) + fabsf(y[2 * j + 1]);
            }
            *reinterpret_cast<uint4*>(Hi + (size_t)tl * kApxXPitch + lane * 16) = make_uint4(hiw[0], hiw[1], hiw[2], hiw[3]);
            *reinterpret_cast<uint4*>(Lo + (size_t)tl * kApxXPitch + lane * 16) = make_uint4(low[0], low[1], low[2], low[3]);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                sum += __shfl_xor_sync(kFullMask, sum, o);
                asum += __shfl_xor_sync(kFullMask, asum, o);
            }
            if ((lane & 7) == 0) {
                XS[(lane >> 3) * kApxTokens + tl] = sum;
                XA[(lane >> 3) * kApxTokens + tl] = asum + 0.015625f;     // 64 x 2^-25 / kApxRelError, rounded up
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (c0 + kApxChunk < c_end) {
            request_weights(c0 + kApxChunk, Wc0 + (size_t)((ci + 1u) & 1u) * kApxExperts * kApxWPitch);
            request_rows(c0 + kApxChunk);
        }
        const uint2 sc_lo = s_lo, sc_hi = s_hi, bc_lo = b_lo, bc_hi = b_hi;
        if (c0 + kApxChunk < c_end) request_scales(c0 + kApxChunk);
#pragma unroll 1
        for (int gi = 0; gi < 4; ++gi) {
            const uint4 a_lo = *reinterpret_cast<const uint4*>(Wc + (size_t)(warp * 16 + g) * kApxWPitch + gi * 64 + t * 16);
            const uint4 a_hi = *reinterpret_cast<const uint4*>(Wc + (size_t)(warp * 16 + g + 8) * kApxWPitch + gi * 64 + t * 16);
            const uint32_t alw[4] = {a_lo.x, a_lo.y, a_lo.z, a_lo.w}, ahw[4] = {a_hi.x, a_hi.y, a_hi.z, a_hi.w};
            uint32_t af[4][4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                af[s][0] = bytes_to_half2(alw[s], 0x5140u); af[s][1] = bytes_to_half2(ahw[s], 0x5140u);
                af[s][2] = bytes_to_half2(alw[s], 0x7362u); af[s][3] = bytes_to_half2(ahw[s], 0x7362u);
            }
            const uint32_t sh = (gi & 1) * 16;
            const float sl = bf16_bits_to_float((uint16_t)((gi < 2 ? sc_lo.x : sc_lo.y) >> sh)), sH = bf16_bits_to_float((uint16_t)((gi < 2 ? sc_hi.x : sc_hi.y) >> sh));
            const float bL = bf16_bits_to_float((uint16_t)((gi < 2 ? bc_lo.x : bc_lo.y) >> sh)), bH = bf16_bits_to_float((uint16_t)((gi < 2 ? bc_hi.x : bc_hi.y) >> sh));
            const float ml = fmaf(255.0f, fabsf(sl), fabsf(bL)), mh = fmaf(255.0f, fabsf(sH), fabsf(bH));
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                float P[4] = {};
                const size_t off = (size_t)(nt * 8 + g) * kApxXPitch + (size_t)(gi * 64 + t * 16) * 2;
                const uint4 h0 = *reinterpret_cast<const uint4*>(Hi + off), h1 = *reinterpret_cast<const uint4*>(Hi + off + 16);
                const uint4 l0 = *reinterpret_cast<const uint4*>(Lo + off), l1 = *reinterpret_cast<const uint4*>(Lo + off + 16);
                const uint32_t bh[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                const uint32_t bl[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    mma_f16_f32(P, af[s][0], af[s][1], af[s][2], af[s][3], bh[2 * s], bh[2 * s + 1]);
                    mma_f16_f32(P, af[s][0], af[s][1], af[s][2], af[s][3], bl[2 * s], bl[2 * s + 1]);
                }
                const float2 xs = *reinterpret_cast<const float2*>(XS + gi * kApxTokens + nt * 8 + 2 * t);
                const float2 xa = *reinterpret_cast<const float2*>(XA + gi * kApxTokens + nt * 8 + 2 * t);
                acc[nt][0] = fmaf(sl, P[0], fmaf(bL, xs.x, acc[nt][0]));
                acc[nt][1] = fmaf(sl, P[1], fmaf(bL, xs.y, acc[nt][1]));
                acc[nt][2] = fmaf(sH, P[2], fmaf(bH, xs.x, acc[nt][2]));
                acc[nt][3] = fmaf(sH, P[3], fmaf(bH, xs.y, acc[nt][3]));
                mag[nt][0] = fmaf(ml, xa.x, mag[nt][0]);
                mag[nt][1] = fmaf(ml, xa.y, mag[nt][1]);
                mag[nt][2] = fmaf(mh, xa.x, mag[nt][2]);
                mag[nt][3] = fmaf(mh, xa.y, mag[nt][3]);
            }
        }
    }
    const float unscale = 1.0f / kApxPrescale;
    const uint32_t er_lo = e0 + warp * 16 + g, er_hi = er_lo + 8;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint32_t tok = tok0 + nt * 8 + 2 * t + c;
            if (tok >= rows) continue;
            if (er_lo < num_experts) out[(size_t)tok * num_experts + er_lo] = make_float2(acc[nt][c] * unscale, mag[nt][c] * unscale);
            if (er_hi < num_experts) out[(size_t)tok * num_experts + er_hi] = make_float2(acc[nt][2 + c] * unscale, mag[nt][2 + c] * unscale);
        }
    }
}

// The same for few rows: a block of 8 tokens x 32 experts holds the whole rows of both operands in shared memory, so one
// round of loads is on its way at once (the weights before the previous kernel has ended) instead of eleven in a row; warp w
// multiplies expert tile w % 2 over a quarter of the groups (w / 2), and the quarters are added in shared memory. At 200
// rows the 16 x 128 blocks made 13 blocks that ran 25 us; the sums differ in order only, within the same error bound.
constexpr int kFewTokens = 8, kFewExperts = 32, kFewThreads = 256, kFewParts = 4;
__host__ __device__ inline size_t router_approx_few_smem_bytes(uint32_t d) {
    const size_t groups = d / kGroup;
    return (size_t)kFewExperts * (d + 64) + 2 * (size_t)kFewTokens * (2 * d + 16) + 2 * groups * kFewTokens * sizeof(float);
}
template <bool X_BF16>
__global__ void __launch_bounds__(kFewThreads, 1)
router_approx_few_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                         const uint16_t* hidden, uint32_t hidden_stride, const uint16_t* __restrict__ eff,
                         float2* __restrict__ out, uint32_t rows, uint32_t num_experts, uint32_t d) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t w_pitch = d + 64, x_pitch = 2 * d + 16;                 // bank-conflict free, as kApxWPitch and kApxXPitch
    const uint32_t groups = d / kGroup;
    uint8_t* Ws = smem;                                                    // [32][w_pitch]
    uint8_t* Hi = Ws + (size_t)kFewExperts * w_pitch;                      // [8][x_pitch]
    uint8_t* Lo = Hi + (size_t)kFewTokens * x_pitch;
    float* XS = reinterpret_cast<float*>(Lo + (size_t)kFewTokens * x_pitch);   // [groups][8]: sum of x * 2^10
    float* XA = XS + groups * kFewTokens;                                  // of |x * 2^10| (+ the split's absolute part)
    const int tid = threadIdx.x, warp = tid / kWarp, lane = tid % kWarp, g = lane >> 2, t = lane & 3;
    const uint32_t tok0 = blockIdx.x * kFewTokens, e0 = blockIdx.y * kFewExperts, last = num_experts - 1;
    pdl_launch_dependents();
    const uint32_t segs = d / 16;
    for (uint32_t row = warp; row < (uint32_t)kFewExperts; row += kFewThreads / kWarp) {        // rows past the end repeat the last expert
        const uint8_t* src = W + (size_t)min(e0 + row, last) * d;
        for (uint32_t i = lane; i < segs; i += kWarp) cp_async_16(Ws + (size_t)row * w_pitch + i * 16, src + i * 16);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    pdl_wait();
    {
        // a warp stages one token, eight columns per lane and step (rows past the end are zeros)
        const uint32_t tok = tok0 + warp;
        const uint16_t* hrow = hidden + (size_t)min(tok, rows - 1) * hidden_stride;
#pragma unroll 4
        for (uint32_t c = lane * 8; c < d; c += 8 * kWarp) {               // d is a multiple of 256: whole warps
            const uint4 ev = *reinterpret_cast<const uint4*>(eff + c);
            uint4 hv = *reinterpret_cast<const uint4*>(hrow + c);
            if (tok >= rows) hv = make_uint4(0u, 0u, 0u, 0u);
            const uint32_t hw[4] = {hv.x, hv.y, hv.z, hv.w}, ew[4] = {ev.x, ev.y, ev.z, ev.w};
            uint32_t hiw[4], low[4];
            float sum = 0.0f, asum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint16_t h0 = (uint16_t)(hw[j] & 0xFFFFu), h1 = (uint16_t)(hw[j] >> 16);
                const float y0 = __fmul_rn(X_BF16 ? bf16_bits_to_float(h0) : f16_bits_to_float(h0), bf16_bits_to_float((uint16_t)(ew[j] & 0xFFFFu))) * kApxPrescale;
                const float y1 = __fmul_rn(X_BF16 ? bf16_bits_to_float(h1) : f16_bits_to_float(h1), bf16_bits_to_float((uint16_t)(ew[j] >> 16))) * kApxPrescale;
                const __half2 hh = __floats2half2_rn(y0, y1);
                const float2 hf = __half22float2(hh);
                const __half2 ll = __floats2half2_rn(y0 - hf.x, y1 - hf.y);
                hiw[j] = *reinterpret_cast<const uint32_t*>(&hh);
                low[j] = *reinterpret_cast<const uint32_t*>(&ll);
                sum += y0 + y1;
                asum += fabsf(y0) + fabsf(y1);
            }
            *reinterpret_cast<uint4*>(Hi + (size_t)warp * x_pitch + c * 2) = make_uint4(hiw[0], hiw[1], hiw[2], hiw[3]);
            *reinterpret_cast<uint4*>(Lo + (size_t)warp * x_pitch + c * 2) = make_uint4(low[0], low[1], low[2], low[3]);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                sum += __shfl_xor_sync(kFullMask, sum, o);
                asum += __shfl_xor_sync(kFullMask, asum, o);
            }
            if ((lane & 7) == 0) {
                XS[(c / kGroup) * kFewTokens + warp] = sum;
                XA[(c / kGroup) * kFewTokens + warp] = asum + 0.015625f;   // 64 x 2^-25 / kApxRelError, rounded up
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int tile = warp & 1, part = warp >> 1;
    const uint32_t e_lo = min(e0 + tile * 16 + g, last), e_hi = min(e0 + tile * 16 + g + 8, last);
    const uint32_t per = (groups + kFewParts - 1) / kFewParts, g_begin = part * per, g_end = min(g_begin + per, groups);
    float acc[4] = {}, mag[4] = {};
#pragma unroll 2
    for (uint32_t gi = g_begin; gi < g_end; ++gi) {
        const uint4 a_lo = *reinterpret_cast<const uint4*>(Ws + (size_t)(tile * 16 + g) * w_pitch + gi * 64 + t * 16);
        const uint4 a_hi = *reinterpret_cast<const uint4*>(Ws + (size_t)(tile * 16 + g + 8) * w_pitch + gi * 64 + t * 16);
        const float sl = bf16_bits_to_float(__ldg(S + (size_t)e_lo * groups + gi)), sH = bf16_bits_to_float(__ldg(S + (size_t)e_hi * groups + gi));
        const float bL = bf16_bits_to_float(__ldg(B + (size_t)e_lo * groups + gi)), bH = bf16_bits_to_float(__ldg(B + (size_t)e_hi * groups + gi));
        const size_t off = (size_t)g * x_pitch + (size_t)(gi * 64 + t * 16) * 2;
        const uint4 h0 = *reinterpret_cast<const uint4*>(Hi + off), h1 = *reinterpret_cast<const uint4*>(Hi + off + 16);
        const uint4 l0 = *reinterpret_cast<const uint4*>(Lo + off), l1 = *reinterpret_cast<const uint4*>(Lo + off + 16);
        const uint32_t alw[4] = {a_lo.x, a_lo.y, a_lo.z, a_lo.w}, ahw[4] = {a_hi.x, a_hi.y, a_hi.z, a_hi.w};
        const uint32_t bh[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
        const uint32_t bl[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
        float P[4] = {};
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint32_t a0 = bytes_to_half2(alw[s], 0x5140u), a1 = bytes_to_half2(ahw[s], 0x5140u);
            const uint32_t a2 = bytes_to_half2(alw[s], 0x7362u), a3 = bytes_to_half2(ahw[s], 0x7362u);
            mma_f16_f32(P, a0, a1, a2, a3, bh[2 * s], bh[2 * s + 1]);
            mma_f16_f32(P, a0, a1, a2, a3, bl[2 * s], bl[2 * s + 1]);
        }
        const float ml = fmaf(255.0f, fabsf(sl), fabsf(bL)), mh = fmaf(255.0f, fabsf(sH), fabsf(bH));
        const float2 xs = *reinterpret_cast<const float2*>(XS + gi * kFewTokens + 2 * t);
        const float2 xa = *reinterpret_cast<const float2*>(XA + gi * kFewTokens + 2 * t);
        acc[0] = fmaf(sl, P[0], fmaf(bL, xs.x, acc[0]));
        acc[1] = fmaf(sl, P[1], fmaf(bL, xs.y, acc[1]));
        acc[2] = fmaf(sH, P[2], fmaf(bH, xs.x, acc[2]));
        acc[3] = fmaf(sH, P[3], fmaf(bH, xs.y, acc[3]));
        mag[0] = fmaf(ml, xa.x, mag[0]);
        mag[1] = fmaf(ml, xa.y, mag[1]);
        mag[2] = fmaf(mh, xa.x, mag[2]);
        mag[3] = fmaf(mh, xa.y, mag[3]);
    }
    __syncthreads();                                  // every fragment has been read: the activations' space holds the partial sums
    float4* red = reinterpret_cast<float4*>(Hi);      // [warp][lane] x (acc, mag)
    red[(warp * kWarp + lane) * 2] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    red[(warp * kWarp + lane) * 2 + 1] = make_float4(mag[0], mag[1], mag[2], mag[3]);
    __syncthreads();
    if (part != 0) return;
#pragma unroll
    for (int p = 1; p < kFewParts; ++p) {
        const float4 a = red[((warp + 2 * p) * kWarp + lane) * 2], m = red[((warp + 2 * p) * kWarp + lane) * 2 + 1];
        acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
        mag[0] += m.x; mag[1] += m.y; mag[2] += m.z; mag[3] += m.w;
    }
    const float unscale = 1.0f / kApxPrescale;
    const uint32_t er_lo = e0 + tile * 16 + g, er_hi = er_lo + 8;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const uint32_t tok = tok0 + 2 * t + c;
        if (tok >= rows) continue;
        if (er_lo < num_experts) out[(size_t)tok * num_experts + er_lo] = make_float2(acc[c] * unscale, mag[c] * unscale);
        if (er_hi < num_experts) out[(size_t)tok * num_experts + er_hi] = make_float2(acc[2 + c] * unscale, mag[2 + c] * unscale);
    }
}

// Canonical logits with the expert's codes, scales and biases read from global memory and the row's scaled activations
// from shared memory (the arithmetic and order of router_row_logit), kLogitChunk groups at a time: the loads of a chunk
// are issued together, one chunk ahead of the arithmetic (across experts too); lane i holds the scale and bias of the
// chunk's group i.
constexpr int kLogitChunk = 16;
__device__ __forceinline__ void router_logit_load(const uint8_t* __restrict__ Wrow, const uint16_t* __restrict__ s_row,
                                                  const uint16_t* __restrict__ b_row, uint32_t g0, uint32_t groups, int lane,
                                                  uint32_t (&w)[kLogitChunk], uint32_t& sb) {
#pragma unroll
    for (int i = 0; i < kLogitChunk; ++i)
        w[i] = g0 + i < groups ? (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(Wrow + (size_t)(g0 + i) * kGroup + lane * 2)) : 0u;
    sb = 0u;
    if (lane < kLogitChunk && g0 + lane < groups) sb = (uint32_t)__ldg(s_row + g0 + lane) | ((uint32_t)__ldg(b_row + g0 + lane) << 16);
}
__device__ __forceinline__ float router_logit_chunk(float acc, const uint32_t (&wv)[kLogitChunk], uint32_t sb, const float* xf,
                                                    uint32_t g0, uint32_t groups, int lane) {
#pragma unroll
    for (int i = 0; i < kLogitChunk; ++i) {
        const uint32_t sbv = __shfl_sync(kFullMask, sb, i);
        if (g0 + i < groups) {                                                          // the same for the whole warp
            const uint32_t w = wv[i];
            const float q0 = __uint_as_float(0x4B000000u | (w & 0xFFu)) - 8388608.0f;      // exact for 0...255
            const float q1 = __uint_as_float(0x4B000000u | (w >> 8)) - 8388608.0f;
            const float2 xv = *reinterpret_cast<const float2*>(xf + (size_t)(g0 + i) * kGroup + lane * 2);
            const float s = bf16_bits_to_float((uint16_t)(sbv & 0xFFFFu));
            const float b = bf16_bits_to_float((uint16_t)(sbv >> 16));
            const float p = __fmaf_rn(q1, xv.y, __fmul_rn(q0, xv.x));
            acc = __fmaf_rn(s, p, acc);
            acc = __fmaf_rn(b, __fadd_rn(xv.x, xv.y), acc);
        }
    }
    return acc;
}
// The same for a group count known at compile time (the production width): all of an expert's codes are requested at
// once, lane l holds the scale and bias of groups l and l + 32, and nothing in the loop is guarded.
template <int GROUPS>
struct LogitOperands {
    uint32_t w[GROUPS];
    uint32_t sb0, sb1;
};
template <int GROUPS>
__device__ __forceinline__ void router_logit_load_all(const uint8_t* __restrict__ Wrow, const uint16_t* __restrict__ s_row,
                                                      const uint16_t* __restrict__ b_row, int lane, LogitOperands<GROUPS>& r) {
    static_assert(GROUPS <= 2 * kWarp, "two scale words per lane");
    const uint8_t* wl = Wrow + lane * 2;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) r.w[g] = (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(wl + g * kGroup));
    r.sb0 = lane < GROUPS ? (uint32_t)__ldg(s_row + lane) | ((uint32_t)__ldg(b_row + lane) << 16) : 0u;
    r.sb1 = lane + kWarp < GROUPS ? (uint32_t)__ldg(s_row + lane + kWarp) | ((uint32_t)__ldg(b_row + lane + kWarp) << 16) : 0u;
}
template <int GROUPS>
__device__ __forceinline__ float router_logit_all(const LogitOperands<GROUPS>& r, const float* xf, int lane) {
    const float* xl = xf + lane * 2;
    float acc = 0.0f;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) {
        const uint32_t sbv = __shfl_sync(kFullMask, g < kWarp ? r.sb0 : r.sb1, g % kWarp);
        const uint32_t w = r.w[g];
        const float q0 = __uint_as_float(0x4B000000u | (w & 0xFFu)) - 8388608.0f;      // exact for 0...255
        const float q1 = __uint_as_float(0x4B000000u | (w >> 8)) - 8388608.0f;
        const float2 xv = *reinterpret_cast<const float2*>(xl + g * kGroup);
        const float s = __uint_as_float(sbv << 16);
        const float b = __uint_as_float(sbv & 0xFFFF0000u);
        const float p = __fmaf_rn(q1, xv.y, __fmul_rn(q0, xv.x));
        acc = __fmaf_rn(s, p, acc);
        acc = __fmaf_rn(b, __fadd_rn(xv.x, xv.y), acc);
    }
    return warp_sum(acc);
}

// The same for two experts whose rows are staged in shared memory, in a loop of a few dozen instructions; activations and their sums
// are shared. For the forms with several warps per token, whose warps have one to three candidates: with the unrolled form above,
// some ten KB of instructions executed once or twice, that phase took 35 900 clocks at 333 rows, 20 500 with this one (10 200
// since the candidates are a list). With a warp per token and 16 warps per SM the unrolled form stays ahead (4096 rows, 30
// layers: 22.1 ms against 22.5 with two warps per token and this form).
template <int GROUPS>
__device__ __forceinline__ float2 router_logits_staged(const uint8_t* codes_a, const uint8_t* codes_b, uint32_t a0, uint32_t a1, uint32_t b0,
                                                       uint32_t b1, const float* xf, int lane) {
    static_assert(GROUPS <= 2 * kWarp, "two scale words per lane");
    const uint8_t *wa = codes_a + lane * 2, *wb = codes_b + lane * 2;
    const float* xl = xf + lane * 2;
    float acc_a = 0.0f, acc_b = 0.0f;
#pragma unroll 4
    for (int g = 0; g < GROUPS; ++g) {
        const uint32_t va = __shfl_sync(kFullMask, g < kWarp ? a0 : a1, g % kWarp), vb = __shfl_sync(kFullMask, g < kWarp ? b0 : b1, g % kWarp);
        const uint32_t qa = *reinterpret_cast<const uint16_t*>(wa + g * kGroup), qb = *reinterpret_cast<const uint16_t*>(wb + g * kGroup);
        const float2 xv = *reinterpret_cast<const float2*>(xl + g * kGroup);
        const float sum = __fadd_rn(xv.x, xv.y);
        // byte -> float through the 2^23 mantissa trick (exact for 0...255)
        const float pa = __fmaf_rn(__uint_as_float(0x4B000000u | (qa >> 8)) - 8388608.0f, xv.y,
                                   __fmul_rn(__uint_as_float(0x4B000000u | (qa & 0xFFu)) - 8388608.0f, xv.x));
        const float pb = __fmaf_rn(__uint_as_float(0x4B000000u | (qb >> 8)) - 8388608.0f, xv.y,
                                   __fmul_rn(__uint_as_float(0x4B000000u | (qb & 0xFFu)) - 8388608.0f, xv.x));
        acc_a = __fmaf_rn(__uint_as_float(va << 16), pa, acc_a);
        acc_b = __fmaf_rn(__uint_as_float(vb << 16), pb, acc_b);
        acc_a = __fmaf_rn(__uint_as_float(va & 0xFFFF0000u), sum, acc_a);
        acc_b = __fmaf_rn(__uint_as_float(vb & 0xFFFF0000u), sum, acc_b);
    }
    return make_float2(warp_sum(acc_a), warp_sum(acc_b));
}

// The experts that can reach the top k, in list (ascending), and their number: those whose upper bound is not below the top_k-th
// largest lower bound. N: experts per lane. (A list: warps that took their candidates off bit masks, each skipping those of the token's
// other warps, spent up to 20 000 clocks on that at eight warps per token.)
template <int N, bool AHEAD>
__device__ __forceinline__ uint32_t router_candidates(const float2* approx_row, uint32_t parts, size_t part_stride, const float* __restrict__ logit_bias,
                                                      uint32_t num_experts, uint32_t top_k, int lane, uint16_t* list /* shared */) {
    float upper[N];
    uint32_t key[N];
    bool bad = false;
    float2 sum[N];
    if constexpr (AHEAD) {
#pragma unroll
        for (int j = 0; j < N; ++j) sum[j] = (uint32_t)(lane + j * kWarp) < num_experts ? approx_row[lane + j * kWarp] : make_float2(0.0f, 0.0f);
        if (parts > 1) {
#pragma unroll 5
            for (uint32_t p = 1; p < parts; ++p) {
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    if ((uint32_t)(lane + j * kWarp) < num_experts) {
                        const float2 more = approx_row[p * part_stride + lane + j * kWarp];
                        sum[j].x += more.x; sum[j].y += more.y;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t e = lane + j * kWarp;
        upper[j] = -INFINITY;
        key[j] = 0u;
        if (e < num_experts) {
            const float2 am = AHEAD ? sum[j] : approx_row[e];
            float v = am.x;
            if (!isfinite(am.x) || !isfinite(am.y)) bad = true;
            if (logit_bias) v = __fadd_rn(v, logit_bias[e]);
            if (v == -INFINITY) {
                key[j] = topk_score_key(-INFINITY);             // a -inf bias: the canonical logit is -inf as well
            } else if (!isfinite(v)) {
                bad = true;
            } else {
                const float eps = fmaf(kApxRelError, am.y, fabsf(v) * 2.384185791015625e-07f);    // + 2^-22 |v|: the bias add
                upper[j] = v + eps;
                key[j] = topk_score_key(v - eps);
            }
        }
    }
    // the top_k-th largest lower bound
    uint32_t lb_key = 0u;
#pragma unroll 1
    for (uint32_t r = 0; r < top_k; ++r) {
        uint32_t best = 0u;
#pragma unroll
        for (int j = 0; j < N; ++j) best = max(best, key[j]);
        lb_key = __reduce_max_sync(kFullMask, best);
        const uint32_t who = __reduce_min_sync(kFullMask, (best == lb_key && lb_key != 0u) ? (uint32_t)lane : 32u);
        if ((uint32_t)lane == who) {
            bool done = false;
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (!done && key[j] == lb_key) { key[j] = 0u; done = true; }
        }
    }
    if (lb_key == 0u) bad = true;                 // fewer than top_k comparable experts
    bad = __any_sync(kFullMask, bad);
    const float lb = bad ? -INFINITY : topk_key_score(lb_key);
    uint32_t count = 0;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t e = lane + j * kWarp;
        const bool cand = e < num_experts && (bad || upper[j] >= lb);
        const uint32_t mask = __ballot_sync(kFullMask, cand);
        if (cand) list[count + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)e;
        count += __popc(mask);
    }
    return count;
}

// The grouping of the re-check's last block, up to a few thousand pairs: a warp takes consecutive pairs, 32 to a round, whose lanes find their
// rank among the round's pairs of the same expert with match.any; the first of them adds their number to the warp's count of the expert. A
// thread per expert then turns the counts into starts. Latency bounds it. (group_routes_in_block, whose bitmaps have rows of 64 words at 255
// tokens of top 8, all in one bank: 255 rows 42 -> 30 us for the launch, 200 rows 31 -> 27, 70 rows 19 -> 16.5; steps of 30 layers, 255
// tokens 8446 -> 8139, 200 tokens 7076 -> 7001, 130 tokens 5869 -> 5810, up to 120 tokens the same. The few-row router stays with those: up to 11
// tokens it took 1 to 3 % longer with this.)
constexpr uint32_t kGroupRowsWarps = kRecheckWarps;
__host__ __device__ inline size_t router_group_rows_smem_bytes(uint32_t n_pairs, uint32_t num_experts) {
    return (size_t)num_experts * (kGroupRowsWarps + 1) * 4 + (size_t)n_pairs * 4 + 3 * kGroupRowsWarps * 4 + (size_t)((n_pairs + 1) / 2) * 4;
}
__device__ __forceinline__ void group_rows_in_block(const uint32_t* __restrict__ idx, const uint16_t* __restrict__ w, uint32_t T, uint32_t K,
                                                    uint32_t E, const RouterGroupOut& out, uint8_t* smem) {
    constexpr uint32_t kAtOnce = 8;                              // rounds whose ids are requested together
    const uint32_t n = T * K, rounds = (n + kGroupRowsWarps * kWarp - 1) / (kGroupRowsWarps * kWarp);
    uint32_t* counts = reinterpret_cast<uint32_t*>(smem);        // [warp][E]: the warp's pairs of the expert, then where they start
    uint32_t* offs = counts + (size_t)kGroupRowsWarps * E;       // [E]
    uint32_t* exs = offs + E;                                    // [n]: expert | rank among the warp's pairs of it << 16
    uint32_t* wtot = exs + n;                                    // [3][warps]
    uint16_t* wts = reinterpret_cast<uint16_t*>(wtot + 3 * kGroupRowsWarps);      // [n]
    const uint32_t lane = threadIdx.x % kWarp, warp = threadIdx.x / kWarp, first = warp * rounds * kWarp + lane;
    uint32_t* mine = counts + (size_t)warp * E;
    for (uint32_t i = lane; i < E; i += kWarp) mine[i] = 0;
    __syncwarp();
    for (uint32_t r0 = 0; r0 < rounds; r0 += kAtOnce) {
        uint32_t ids[kAtOnce], wt[kAtOnce];
#pragma unroll
        for (uint32_t j = 0; j < kAtOnce; ++j) {                 // written by other blocks of this launch
            const uint32_t i = first + (r0 + j) * kWarp;
            const bool in = r0 + j < rounds && i < n;
            ids[j] = in ? __ldcg(idx + i) : 0xFFFFFFFFu;
            wt[j] = in ? (uint32_t)__ldcg(w + i) : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < kAtOnce; ++j) {
            if (r0 + j < rounds) {
                const uint32_t i = first + (r0 + j) * kWarp;
                uint32_t ex = ids[j];
                if (ex != 0xFFFFFFFFu && ex >= E) ex = E - 1;    // min(id, E-1): Runtime/Inference/RealForwardRunner.swift:955
                const uint32_t peers = __match_any_sync(kFullMask, ex);
                const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
                uint32_t before = 0;
                if (ex != 0xFFFFFFFFu && rank == 0) {
                    before = mine[ex];
                    mine[ex] = before + __popc(peers);
                }
                before = __shfl_sync(kFullMask, before, __ffs(peers) - 1);
                if (i < n) {
                    exs[i] = ex == 0xFFFFFFFFu ? ex : ex | (before + rank) << 16;
                    wts[i] = (uint16_t)wt[j];
                }
                __syncwarp();
            }
        }
    }
    __syncthreads();
    // a thread per expert: the warps' counts to starts, exclusive scans over the experts (pairs, non-empty groups, chunks) of 32 to a warp
    static_assert(TF_MAX_ROUTER_EXPERTS <= kGroupRowsWarps * kWarp, "a thread per expert");
    const uint32_t e = threadIdx.x;
    uint32_t cnt = 0;
    if (e < E) {
        uint32_t c[kGroupRowsWarps];
#pragma unroll
        for (uint32_t v = 0; v < kGroupRowsWarps; ++v) c[v] = counts[(size_t)v * E + e];
#pragma unroll
        for (uint32_t v = 0; v < kGroupRowsWarps; ++v) {
            counts[(size_t)v * E + e] = cnt;
            cnt += c[v];
        }
    }
    const uint32_t nch = (cnt + (uint32_t)kChunkTokens - 1) / (uint32_t)kChunkTokens;
    uint32_t i_off = cnt, i_g = cnt ? 1u : 0u, i_ch = nch;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const uint32_t a = __shfl_up_sync(kFullMask, i_off, o), b2 = __shfl_up_sync(kFullMask, i_g, o), c = __shfl_up_sync(kFullMask, i_ch, o);
        if ((int)lane >= o) { i_off += a; i_g += b2; i_ch += c; }
    }
    if (lane == kWarp - 1) { wtot[warp] = i_off; wtot[kGroupRowsWarps + warp] = i_g; wtot[2 * kGroupRowsWarps + warp] = i_ch; }
    __syncthreads();
    uint32_t off = i_off - cnt, gi = i_g - (cnt ? 1u : 0u), ch = i_ch - nch;
#pragma unroll
    for (uint32_t v = 0; v < kGroupRowsWarps; ++v)
        if (v < warp) { off += wtot[v]; gi += wtot[kGroupRowsWarps + v]; ch += wtot[2 * kGroupRowsWarps + v]; }
    if (e < E) {
        offs[e] = off;
        out.per_expert_counts[e] = cnt;
        out.per_expert_offsets[e] = cnt ? off : 0xFFFFFFFFu;
        if (cnt) {
            out.groups[gi] = tf_group{e, off, cnt};
            out.chunk_start[gi] = ch;
            for (uint32_t j = 0; j < nch; ++j) out.chunk_group[ch + j] = gi;
        }
    }
    if (e == E - 1) {
        out.counters[0] = gi + (cnt ? 1u : 0u);
        out.counters[1] = ch + nch;
        out.counters[2] = n;
        out.counters[3] = off + cnt;
    }
    __syncthreads();
    for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t i = first + r * kWarp;
        if (i >= n) break;
        const uint32_t v = exs[i], ex = v & 0xFFFFu;
        if (v == 0xFFFFFFFFu) continue;
        out.sorted_pairs[offs[ex] + mine[ex] + (v >> 16)] = tf_pair{i / K, ex, i % K, (uint32_t)wts[i]};
    }
}

// WPT warps per token: candidates from the approximate logits and their bounds (every warp of the token finds them), canonical
// logits of the candidates (dealt out to the warps), top-k and softmax as in every other router kernel (one warp). A
// canonical logit is one long dependent chain, so with few rows a token's eight or nine must not follow one another: one
// warp per token took 30 us at 333 rows; four take 15. With grp.sorted_pairs the block that finishes the last row groups all of them.
// AHEAD: the planes' values are requested before the first is looked at; otherwise (one plane) each where it is used, see launch_router.
template <bool X_BF16, int GROUPS, int WPT, bool AHEAD = true>          // GROUPS: d / 64 when known at compile time, 0 for any width
__global__ void __launch_bounds__(kRecheckWarps * kWarp, 2)
router_recheck_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                      const uint16_t* hidden, uint32_t hidden_stride, const uint16_t* __restrict__ eff,
                      const uint16_t* __restrict__ per_expert_scale, const float* __restrict__ logit_bias,
                      const float2* approx, uint32_t parts, uint32_t* out_idx, uint16_t* out_w, unsigned int* ticket, const RouterGroupOut grp,
                      uint32_t rows, uint32_t num_experts, uint32_t d, uint32_t top_k) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kTokens = kRecheckWarps / WPT;                    // tokens per block
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const int slot = warp / WPT, part = warp % WPT;                 // token within the block, warp within the token
    float* xf = reinterpret_cast<float*>(smem) + (size_t)slot * d;
    float* scores = reinterpret_cast<float*>(smem) + (size_t)kTokens * d + (size_t)slot * num_experts;
    const uint32_t groups = d / kGroup;
    // tokens past the end repeat the last one (the same values are written twice)
    const uint32_t row = min(blockIdx.x * kTokens + slot, rows - 1);
    // With grouping the routed gate/up launch comes next and is let in only before the grouping, as in router_rows_kernel: let in at the
    // start it takes the SMs that the shared expert's gate/up, which no longer fits beside a block of this kernel since that holds
    // staged rows, could use meanwhile. 30 layers, us, at the start and late: 65 tokens 4819 and 4112, 100 tokens 5623 and 4952, 128
    // tokens 6583 and 6088, 150 tokens 6998 and 6190, 175 tokens 7427 and 6634, 190 to 255 tokens the same.
    const bool late = WPT == kRecheckWarps && grp.sorted_pairs != nullptr;
    if (!late) pdl_launch_dependents();
    pdl_wait();
    const uint16_t* hrow = hidden + (size_t)row * hidden_stride;
    for (uint32_t e = part * kWarp + lane; e < num_experts; e += WPT * kWarp) scores[e] = -INFINITY;
    for (uint32_t c0 = (part * kWarp + lane) * 2; c0 < d; c0 += 8 * 2 * kWarp * WPT) {          // eight independent pairs of loads at a time
        uint32_t hv[8], ev[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t c = c0 + u * 2 * kWarp * WPT;
            hv[u] = c < d ? *reinterpret_cast<const uint32_t*>(hrow + c) : 0u;
            ev[u] = c < d ? *reinterpret_cast<const uint32_t*>(eff + c) : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t c = c0 + u * 2 * kWarp * WPT;
            const uint16_t h0 = (uint16_t)(hv[u] & 0xFFFFu), h1 = (uint16_t)(hv[u] >> 16);
            const float x0 = __fmul_rn(X_BF16 ? bf16_bits_to_float(h0) : f16_bits_to_float(h0), bf16_bits_to_float((uint16_t)(ev[u] & 0xFFFFu)));
            const float x1 = __fmul_rn(X_BF16 ? bf16_bits_to_float(h1) : f16_bits_to_float(h1), bf16_bits_to_float((uint16_t)(ev[u] >> 16)));
            if (c < d) *reinterpret_cast<float2*>(xf + c) = make_float2(x0, x1);
        }
    }
    // (every warp of a token writes the same list)
    uint16_t* list = reinterpret_cast<uint16_t*>(reinterpret_cast<float*>(smem) + (size_t)kTokens * (d + num_experts)) + (size_t)slot * num_experts;
    const float2* approx_row = approx + (size_t)row * num_experts;
    const uint32_t candidates = num_experts <= 4u * kWarp ? router_candidates<4, AHEAD>(approx_row, parts, (size_t)rows * num_experts, logit_bias, num_experts, top_k, lane, list)
                                                          : router_candidates<TF_MAX_ROUTER_EXPERTS / kWarp, AHEAD>(approx_row, parts, (size_t)rows * num_experts, logit_bias, num_experts, top_k, lane, list);
    if (WPT == 1) __syncwarp(); else __syncthreads();             // the row's activations and the cleared scores
    // this warp's candidates: every WPT-th one
    uint32_t next = part;
    auto next_candidate = [&]() {
        const uint32_t e = next < candidates ? (uint32_t)list[next] : 0xFFFFFFFFu;
        next += WPT;
        // The shuffle tells the compiler that the warp has one expert, and its guards in the chunked loop one outcome: 1200 rows of 128
        // experts x 2048, 87 -> 82 us, 4096 rows x 4096 312 -> 297. (Nothing is guarded in the other loops.)
        return GROUPS > 0 ? e : __shfl_sync(kFullMask, e, 0);
    };
    // (expert, chunk) pairs in one software pipeline: the next pair's loads are issued before the current pair is multiplied
    uint32_t ld_e = next_candidate(), ld_g = 0u;
    if constexpr (GROUPS > 0 && WPT > 1) {
        // two candidates at a time (a last one alone is computed twice)
        uint8_t* codes = smem + router_recheck_smem_bytes(d, num_experts, kTokens) + (size_t)warp * 2 * d;
        auto request = [&](uint32_t e, uint8_t* dst, uint32_t& s0, uint32_t& s1) {
            const uint8_t* src = W + (size_t)e * d;
            for (uint32_t i = lane; i < d / 16; i += kWarp) cp_async_16(dst + i * 16, src + i * 16);
            const uint16_t *sr = S + (size_t)e * GROUPS, *br = B + (size_t)e * GROUPS;
            s0 = lane < GROUPS ? (uint32_t)__ldg(sr + lane) | ((uint32_t)__ldg(br + lane) << 16) : 0u;
            s1 = lane + kWarp < GROUPS ? (uint32_t)__ldg(sr + lane + kWarp) | ((uint32_t)__ldg(br + lane + kWarp) << 16) : 0u;
        };
#pragma unroll 1
        for (uint32_t ea = ld_e; ea != 0xFFFFFFFFu; ea = next_candidate()) {
            const uint32_t eb = next_candidate();
            uint32_t a0, a1, b0, b1;
            request(ea, codes, a0, a1);
            if (eb != 0xFFFFFFFFu) request(eb, codes + d, b0, b1);
            else { b0 = a0; b1 = a1; }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            const float2 l = router_logits_staged<GROUPS>(codes, eb != 0xFFFFFFFFu ? codes + d : codes, a0, a1, b0, b1, xf, lane);
            if (lane == 0) {
                scores[ea] = logit_bias ? __fadd_rn(l.x, logit_bias[ea]) : l.x;
                if (eb != 0xFFFFFFFFu) scores[eb] = logit_bias ? __fadd_rn(l.y, logit_bias[eb]) : l.y;
            }
            __syncwarp();                                         // the rows have been read
        }
    } else if constexpr (GROUPS > 0) {
        // two operand sets used in turns: the next candidate's loads are in flight while the current one is multiplied
        LogitOperands<GROUPS> ra, rb;
        auto finish = [&](uint32_t e, float l) {
            if (logit_bias) l = __fadd_rn(l, logit_bias[e]);
            if (lane == 0) scores[e] = l;
        };
        uint32_t ea = ld_e;
        if (ea != 0xFFFFFFFFu) router_logit_load_all<GROUPS>(W + (size_t)ea * d, S + (size_t)ea * GROUPS, B + (size_t)ea * GROUPS, lane, ra);
        while (ea != 0xFFFFFFFFu) {
            const uint32_t eb = next_candidate();
            if (eb != 0xFFFFFFFFu) router_logit_load_all<GROUPS>(W + (size_t)eb * d, S + (size_t)eb * GROUPS, B + (size_t)eb * GROUPS, lane, rb);
            finish(ea, router_logit_all<GROUPS>(ra, xf, lane));
            if (eb == 0xFFFFFFFFu) break;
            ea = next_candidate();
            if (ea != 0xFFFFFFFFu) router_logit_load_all<GROUPS>(W + (size_t)ea * d, S + (size_t)ea * GROUPS, B + (size_t)ea * GROUPS, lane, ra);
            finish(eb, router_logit_all<GROUPS>(rb, xf, lane));
        }
    } else if (ld_e != 0xFFFFFFFFu) {
        uint32_t wa[kLogitChunk], wb[kLogitChunk], sba, sbb = 0u;          // two chunk buffers, used in turns
        uint32_t cur_e = ld_e, cur_g = 0u;
        float acc = 0.0f;
        auto advance = [&]() {
            ld_g += kLogitChunk;
            if (ld_g >= groups) { ld_e = next_candidate(); ld_g = 0u; }
        };
        // multiplies the chunk in (wc, sbc) after requesting the next one into (wn, sbn); true when it was the last one
        auto step = [&](const uint32_t (&wc)[kLogitChunk], uint32_t sbc, uint32_t (&wn)[kLogitChunk], uint32_t& sbn) -> bool {
            const uint32_t nxt_e = ld_e, nxt_g = ld_g;
            if (nxt_e != 0xFFFFFFFFu) {
                router_logit_load(W + (size_t)nxt_e * d, S + (size_t)nxt_e * groups, B + (size_t)nxt_e * groups, nxt_g, groups, lane, wn, sbn);
                advance();
            }
            acc = router_logit_chunk(acc, wc, sbc, xf, cur_g, groups, lane);
            if (cur_g + kLogitChunk >= groups) {
                float l = warp_sum(acc);
                if (logit_bias) l = __fadd_rn(l, logit_bias[cur_e]);
                if (lane == 0) scores[cur_e] = l;
                acc = 0.0f;
            }
            cur_e = nxt_e; cur_g = nxt_g;
            return nxt_e == 0xFFFFFFFFu;
        };
        router_logit_load(W + (size_t)ld_e * d, S + (size_t)ld_e * groups, B + (size_t)ld_e * groups, 0u, groups, lane, wa, sba);
        advance();
        while (true) {
            if (step(wa, sba, wb, sbb)) break;
            if (step(wb, sbb, wa, sba)) break;
        }
    }
    if (WPT == 1) __syncwarp(); else __syncthreads();
    if (part == 0)
        warp_select_topk(scores, num_experts, top_k, per_expert_scale, out_idx + (size_t)row * top_k, out_w + (size_t)row * top_k, lane);
    if constexpr (WPT == kRecheckWarps) {                      // the form of the few rows that are grouped here
        if (grp.sorted_pairs == nullptr) return;
        __shared__ bool is_last;
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
            if (is_last) *ticket = 0;                          // ready for the next launch
        }
        __syncthreads();
        if (!is_last) return;
        pdl_launch_dependents();
        __threadfence();
        group_rows_in_block(out_idx, out_w, rows, top_k, num_experts, grp, smem);
    }
}

}  // namespace tf
