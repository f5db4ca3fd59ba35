// One activation vector against 16 weight rows per block, the columns split over the block's warps: the kernels for one
// token, which are bound by latency. The warp-per-row kernels walk a row with one 16-byte load per lane in flight and then
// extract and convert every nibble; here a warp requests all the codes that it will need (8 bytes per lane for rows g and
// g + 8 of each 64-column group) before it uses the first, and four mma.sync.m16n8k16 per group do the products (mma_gemv.cuh).
//
// Columns are taken in parts of four groups; a part's sum is
//     sum over its groups, in order, of  s * (q . x) + b * sum(x)        (Metal/Quant/dequant_int4.metal:132-170)
// and the parts are added in order by one thread per row, so the result does not depend on how many warps share the work.
#pragma once

#include "mma_gemv.cuh"

namespace tf {

constexpr int kTileRows16 = 16;
constexpr int kTilePart = 4;               // groups per part

// x as B fragments ([groups][4 lanes t][8 words]) and group sums scaled by 2^-24 (the codes enter the MMA as q * 2^-24).
// Called by whole warps; `count` vectors of `ng` groups, x_stride elements apart, 16-byte aligned.
__device__ __forceinline__ void tile_stage_x(const uint16_t* x, uint32_t x_stride, uint32_t count, uint32_t ng,
                                             uint32_t* frag, float* xsum) {
    const uint32_t items = count * ng * 4;
    for (uint32_t idx = threadIdx.x; idx < ((items + 31u) & ~31u); idx += blockDim.x) {
        const bool ok = idx < items;
        const uint32_t vg = idx >> 2, t = idx & 3;                   // (vector, group) and quarter of the group
        uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
        if (ok) {
            const uint4* p = reinterpret_cast<const uint4*>(x + (size_t)(vg / ng) * x_stride + (vg % ng) * kGroup + t * 16);
            lo = p[0]; hi = p[1];
        }
        const uint32_t r[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        float sum = 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&r[q]));
            sum += v.x + v.y;
        }
        sum += __shfl_xor_sync(kFullMask, sum, 1);
        sum += __shfl_xor_sync(kFullMask, sum, 2);
        if (!ok) continue;
        if (t == 0) xsum[vg] = sum * 5.9604644775390625e-08f;
        // MMA j of the group takes (x0,x4),(x2,x6) | (x1,x5),(x3,x7) | the same of x8..x15. The activations stay as they are
        // (gm_make_frag scales the odd ones by 1/16, which costs small ones their last bits): the odd codes are shifted instead.
        uint4* dst = reinterpret_cast<uint4*>(frag + (size_t)idx * 8);
#pragma unroll
        for (int h = 0; h < 2; ++h)
            dst[h] = make_uint4(gm_prmt(r[4 * h], r[4 * h + 2], 0x5410), gm_prmt(r[4 * h + 1], r[4 * h + 3], 0x5410),
                                gm_prmt(r[4 * h], r[4 * h + 2], 0x7632), gm_prmt(r[4 * h + 1], r[4 * h + 3], 0x7632));
    }
}
__host__ __device__ inline size_t tile_x_bytes(uint32_t vectors, uint32_t ng) { return (size_t)vectors * ng * (128 + 4) + 16; }

// The operands of N parts of a 16-row tile: part p = first + i * step, i < N.
template <int N>
struct TileOperands {
    uint2 wa[N][kTilePart], wb[N][kTilePart];        // codes of rows g and g + 8
    uint32_t sb[N][kTilePart];                       // lane t: scale (t even) or bias (t odd) of row g (t < 2) or g + 8
};
template <int N>
__device__ __forceinline__ void tile_load(TileOperands<N>& o, const uint8_t* W, const uint16_t* S, const uint16_t* B, uint32_t row0,
                                          uint32_t rows, uint32_t ng, uint32_t first, uint32_t step) {
    const int lane = threadIdx.x % kWarp, g = lane >> 2, t = lane & 3;
    // rows past the matrix read its last row; their sums are not stored
    const uint32_t r0 = min(row0 + g, rows - 1), r1 = min(row0 + g + 8, rows - 1);
    const uint8_t* w0 = W + (size_t)r0 * (ng * 32) + t * 8;
    const uint8_t* w1 = W + (size_t)r1 * (ng * 32) + t * 8;
    const uint16_t* sp = ((t & 1) ? B : S) + (size_t)(t < 2 ? r0 : r1) * ng;
#pragma unroll
    for (int n = 0; n < N; ++n) {
#pragma unroll
        for (int i = 0; i < kTilePart; ++i) {
            const uint32_t G = (first + n * step) * kTilePart + i;
            const bool ok = G < ng;
            o.wa[n][i] = ok ? gm_ldg64(w0 + G * 32) : make_uint2(0u, 0u);
            o.wb[n][i] = ok ? gm_ldg64(w1 + G * 32) : make_uint2(0u, 0u);
            o.sb[n][i] = ok ? (uint32_t)__ldg(sp + G) : 0u;
        }
    }
}
// Sum of part n for rows g (x) and g + 8 (y), valid in the lanes with t == 0.
template <bool SB_FP16, int N>
__device__ __forceinline__ float2 tile_part(const TileOperands<N>& o, int n, const uint32_t* frag, const float* xsum, uint32_t ng, uint32_t part) {
    const int lane = threadIdx.x % kWarp, g = lane >> 2, t = lane & 3;
    float c[kTilePart][4];
#pragma unroll
    for (int i = 0; i < kTilePart; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < kTilePart; ++i) {
            const uint32_t G = part * kTilePart + i;
            uint2 bf = make_uint2(0u, 0u);                             // x is column 0 of the B operand: lanes with g == 0
            if (g == 0 && G < ng) bf = *reinterpret_cast<const uint2*>(frag + (size_t)(G * 4 + t) * 8 + j * 2);
            const uint32_t wx = j < 2 ? o.wa[n][i].x : o.wa[n][i].y, wy = j < 2 ? o.wb[n][i].x : o.wb[n][i].y;
            const int sh = (j & 1) * 4;
            constexpr uint32_t mask = 0x000F000Fu;
            gm_mma(c[i], (wx >> sh) & mask, (wy >> sh) & mask, (wx >> (8 + sh)) & mask, (wy >> (8 + sh)) & mask, bf.x, bf.y, c[i]);
        }
    }
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < kTilePart; ++i) {
        const uint32_t G = part * kTilePart + i;
        const uint32_t v = o.sb[n][i];
        const uint32_t vb0 = __shfl_down_sync(kFullMask, v, 1), vs1 = __shfl_down_sync(kFullMask, v, 2), vb1 = __shfl_down_sync(kFullMask, v, 3);
        const float xs = G < ng ? xsum[G] : 0.0f;
        acc.x = fmaf(sb_to_float<SB_FP16>((uint16_t)v), c[i][0], fmaf(sb_to_float<SB_FP16>((uint16_t)vb0), xs, acc.x));
        acc.y = fmaf(sb_to_float<SB_FP16>((uint16_t)vs1), c[i][2], fmaf(sb_to_float<SB_FP16>((uint16_t)vb1), xs, acc.y));
    }
    return make_float2(acc.x * 16777216.0f, acc.y * 16777216.0f);
}

// tile_gemv.cu
bool tile_gemv_eligible(const void* W, const void* x, uint32_t n);
tf_status launch_tile_gemv(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B, const uint16_t* x,
                           void* y, bool out_f32, uint32_t m, uint32_t n, bool sb_fp16, const char* name);
bool tile_gate_up_eligible(tf_context* ctx, uint32_t d, uint32_t f, uint32_t top_k, const void* x);
bool tile_down_eligible(uint32_t f, const void* acts);
tf_status launch_tile_gate_up(tf_context* ctx, void* stream, const void* const* blobs, const tf_expert_offsets* offsets, const void* x,
                              void* acts, uint32_t d, uint32_t f, uint32_t top_k, const uint32_t* slot_map, uint32_t slots, const char* name);
tf_status launch_tile_down(tf_context* ctx, void* stream, const void* const* blobs, const tf_expert_offsets* offsets, const void* acts,
                           const void* routing_w, const void* residual, void* y, uint32_t d, uint32_t f, uint32_t top_k, const char* name);

}  // namespace tf
