// One-token kernels over 16-row tiles (tile_gemv.cuh): the int4 GEMV of matrices too small for the streaming kernel, and the
// routed experts' gate/up and down phases of a single token. One layer's operators for one token as
// a host calls them one by one: 80 -> 59 us, 44 with the wrappers' cheaper look-up of the stream.
#include "tile_gemv.cuh"

namespace tf {

constexpr int kTileWarps = 8, kTileThreads = kTileWarps * kWarp;

// y[m] = deq4(W[m, n]) . x[n]: a block per 16 rows; part p of the columns belongs to warp p % WARPS, two of its parts in flight.
template <bool SB_FP16, bool OUT_F32, int WARPS>
__global__ void __launch_bounds__(WARPS * kWarp, 16 / WARPS)
tile_gemv_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                 const uint16_t* x, void* __restrict__ y, uint32_t m, uint32_t ng) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t parts = (ng + kTilePart - 1) / kTilePart;
    uint32_t* frag = reinterpret_cast<uint32_t*>(smem);
    float* xsum = reinterpret_cast<float*>(smem + (size_t)ng * 128);
    float* sums = xsum + ((ng + 3u) & ~3u);                             // [parts][16]
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t row0 = blockIdx.x * kTileRows16;
    pdl_launch_dependents();
    pdl_wait();
    TileOperands<2> o;
    tile_load<2>(o, W, S, B, row0, m, ng, warp, WARPS);
    tile_stage_x(x, 0, 1, ng, frag, xsum);
    __syncthreads();
    for (uint32_t p0 = warp; p0 < parts; p0 += 2 * WARPS) {
        if (p0 != (uint32_t)warp) tile_load<2>(o, W, S, B, row0, m, ng, p0, WARPS);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const uint32_t p = p0 + n * WARPS;
            if (p < parts) {
                const float2 a = tile_part<SB_FP16, 2>(o, n, frag, xsum, ng, p);
                if ((lane & 3) == 0) { sums[p * 16 + (lane >> 2)] = a.x; sums[p * 16 + (lane >> 2) + 8] = a.y; }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < kTileRows16 && row0 + threadIdx.x < m) {
        float acc = 0.0f;
        for (uint32_t p = 0; p < parts; ++p) acc += sums[p * 16 + threadIdx.x];
        if constexpr (OUT_F32) static_cast<float*>(y)[row0 + threadIdx.x] = acc;
        else static_cast<uint16_t*>(y)[row0 + threadIdx.x] = __half_as_ushort(__float2half_rn(acc));
    }
}

// acts[slot][row] = half(gelu(gate) * up): grid (F / 16, slots). Warp w takes matrix w % 2 and the parts w / 2, w / 2 + 4, ...,
// three of them in flight (the production width has eleven parts).
__global__ void __launch_bounds__(kTileThreads, 2)
tile_gate_up_kernel(const uint8_t* const* blobs, const tf_expert_offsets off, const uint16_t* x, uint16_t* __restrict__ acts,
                    uint32_t ng, uint32_t f, uint32_t top_k, const uint32_t* slot_map) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t parts = (ng + kTilePart - 1) / kTilePart;
    uint32_t* frag = reinterpret_cast<uint32_t*>(smem);
    float* xsum = reinterpret_cast<float*>(smem + (size_t)ng * 128);
    float* sums = xsum + ((ng + 3u) & ~3u);                             // [2][parts][16]
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t row0 = blockIdx.x * kTileRows16, mat = warp & 1;
    pdl_launch_dependents();
    pdl_wait();
    uint32_t slot = blockIdx.y;
    if (slot_map) {
        slot = slot_map[blockIdx.y];
        if (slot >= top_k) return;                                      // moe.metal:399 (the whole block leaves)
    }
    const uint8_t* blob = blobs[slot];
    const uint8_t* W = blob + (mat ? off.up_w_off : off.gate_w_off);
    const uint16_t* S = reinterpret_cast<const uint16_t*>(blob + (mat ? off.up_s_off : off.gate_s_off));
    const uint16_t* B = reinterpret_cast<const uint16_t*>(blob + (mat ? off.up_b_off : off.gate_b_off));
    constexpr int kInFlight = 3, kStep = kTileWarps / 2;
    const uint32_t kq = warp >> 1;
    TileOperands<kInFlight> o;
    tile_load<kInFlight>(o, W, S, B, row0, f, ng, kq, kStep);
    tile_stage_x(x, 0, 1, ng, frag, xsum);
    __syncthreads();
    for (uint32_t p0 = kq; p0 < parts; p0 += kInFlight * kStep) {
        if (p0 != kq) tile_load<kInFlight>(o, W, S, B, row0, f, ng, p0, kStep);
#pragma unroll
        for (int n = 0; n < kInFlight; ++n) {
            const uint32_t p = p0 + n * kStep;
            if (p < parts) {
                const float2 a = tile_part<false, kInFlight>(o, n, frag, xsum, ng, p);
                float* dst = sums + ((size_t)mat * parts + p) * 16 + (lane >> 2);
                if ((lane & 3) == 0) { dst[0] = a.x; dst[8] = a.y; }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < kTileRows16 && row0 + threadIdx.x < f) {
        float gt = 0.0f, up = 0.0f;
        for (uint32_t p = 0; p < parts; ++p) { gt += sums[p * 16 + threadIdx.x]; up += sums[(parts + p) * 16 + threadIdx.x]; }
        acts[(size_t)slot * f + row0 + threadIdx.x] = __half_as_ushort(__float2half_rn(gelu_tanh(gt) * up));
    }
}

// The down projection of every slot for 16 output rows: a warp per slot, three parts in flight (all of the production width).
// y = half(residual + sum over the slots, in order, of w_s * sum_s) (moe.metal:473-480).
__global__ void __launch_bounds__(kTileThreads, 2)
tile_down_kernel(const uint8_t* const* blobs, const tf_expert_offsets off, const uint16_t* acts, const uint16_t* routing_w,
                 const uint16_t* residual, uint16_t* __restrict__ y, uint32_t d, uint32_t ng, uint32_t top_k) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t* frag = reinterpret_cast<uint32_t*>(smem);                 // [top_k][ng] groups
    float* xsum = reinterpret_cast<float*>(smem + (size_t)top_k * ng * 128);
    __shared__ float slot_sum[TF_MAX_TOP_K][kTileRows16];
    static_assert(TF_MAX_TOP_K <= kTileWarps, "a warp per slot");
    const uint32_t warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const uint32_t row0 = blockIdx.x * kTileRows16;
    const uint32_t parts = (ng + kTilePart - 1) / kTilePart;
    pdl_launch_dependents();
    pdl_wait();
    constexpr int kInFlight = 3;
    TileOperands<kInFlight> o;
    const uint8_t* blob = warp < top_k ? blobs[warp] : nullptr;
    const uint8_t* W = blob + off.down_w_off;
    const uint16_t* S = reinterpret_cast<const uint16_t*>(blob + off.down_s_off);
    const uint16_t* B = reinterpret_cast<const uint16_t*>(blob + off.down_b_off);
    if (warp < top_k) tile_load<kInFlight>(o, W, S, B, row0, d, ng, 0, 1);
    tile_stage_x(acts, ng * kGroup, top_k, ng, frag, xsum);
    __syncthreads();
    if (warp < top_k) {
        float2 acc = make_float2(0.0f, 0.0f);
        for (uint32_t p0 = 0; p0 < parts; p0 += kInFlight) {
            if (p0 != 0) tile_load<kInFlight>(o, W, S, B, row0, d, ng, p0, 1);
#pragma unroll
            for (int n = 0; n < kInFlight; ++n) {
                if (p0 + n < parts) {
                    const float2 a = tile_part<false, kInFlight>(o, n, frag + (size_t)warp * ng * 32, xsum + warp * ng, ng, p0 + n);
                    acc.x += a.x; acc.y += a.y;
                }
            }
        }
        if ((lane & 3) == 0) { slot_sum[warp][lane >> 2] = acc.x; slot_sum[warp][(lane >> 2) + 8] = acc.y; }
    }
    __syncthreads();
    if (threadIdx.x < kTileRows16 && row0 + threadIdx.x < d) {
        const uint32_t row = row0 + threadIdx.x;
        float acc = residual ? f16_bits_to_float(residual[row]) : 0.0f;
        for (uint32_t s = 0; s < top_k; ++s) acc += f16_bits_to_float(routing_w[s]) * slot_sum[s][threadIdx.x];
        y[row] = __half_as_ushort(__float2half_rn(acc));
    }
}

// ---- host ----

static size_t tile_gemv_smem(uint32_t ng, uint32_t mats) {
    return tile_x_bytes(1, ng) + (size_t)mats * ((ng + kTilePart - 1) / kTilePart) * 16 * 4;
}
// Aligned planes of any row count; vectors up to 16384 columns (shared memory).
bool tile_gemv_eligible(const void* W, const void* x, uint32_t n) { return aligned(W, 16) && aligned(x, 16) && n % kGroup == 0 && n <= 16384; }

// Two blocks of eight warps fit an SM. Rows of more than 4096 columns take several rounds of loads per warp, one memory latency
// each; where every block has an SM to itself, sixteen warps halve the rounds (704 x 16384: 22.8 -> 13.2 us a call, 1000 x 8192:
// 12.6 -> 7.2; the warp-per-row kernel takes 20.5 and 12.3).
template <int WARPS>
static tf_status launch_tile_gemv_warps(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B, const uint16_t* x,
                                        void* y, bool out_f32, uint32_t m, uint32_t ng, bool sb_fp16, const char* name) {
    const size_t smem = tile_gemv_smem(ng, 1);
    auto k = sb_fp16 ? (out_f32 ? tile_gemv_kernel<true, true, WARPS> : tile_gemv_kernel<true, false, WARPS>)
                     : (out_f32 ? tile_gemv_kernel<false, true, WARPS> : tile_gemv_kernel<false, false, WARPS>);
    static DeviceSmemCache configured[4];
    if (smem > 48 * 1024)
        if (tf_status s = ensure_dynamic_smem(ctx, k, configured[(sb_fp16 ? 2 : 0) + (out_f32 ? 1 : 0)], smem)) return s;
    launch_pdl(k, dim3((m + kTileRows16 - 1) / kTileRows16), dim3(WARPS * kWarp), smem, static_cast<cudaStream_t>(stream), W, S, B, x, y, m, ng);
    return check_launch(ctx, name);
}

tf_status launch_tile_gemv(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B, const uint16_t* x,
                           void* y, bool out_f32, uint32_t m, uint32_t n, bool sb_fp16, const char* name) {
    const bool alone = (m + kTileRows16 - 1) / kTileRows16 <= (uint32_t)ctx->sm_count;
    return n > 4096 && alone ? launch_tile_gemv_warps<16>(ctx, stream, W, S, B, x, y, out_f32, m, n / kGroup, sb_fp16, name)
                             : launch_tile_gemv_warps<8>(ctx, stream, W, S, B, x, y, out_f32, m, n / kGroup, sb_fp16, name);
}

// Blobs and packed sub-tensor offsets must be 16-byte aligned (checked by the callers).
// Up to 3072 columns a warp has all of its codes in flight at once; beyond, the tiles win while the blocks of all slots are at most
// two and a half rounds of one per SM (8 experts, row kernel / tiles: 4096 x 704 19.2 / 18.7 us, 6144 x 704 27.8 / 22.1, 4096 x
// 1408 28.5 / 29.5, 8192 x 4096 120 / 146). The number of active slots doesn't count: a split call has the bits of a whole one.
bool tile_gate_up_eligible(tf_context* ctx, uint32_t d, uint32_t f, uint32_t top_k, const void* x) {
    const uint64_t blocks = (uint64_t)((f + kTileRows16 - 1) / kTileRows16) * top_k;
    return d % kGroup == 0 && d <= 16384 && aligned(x, 16) && (d <= 3072 || 2 * blocks <= 5ull * (uint32_t)ctx->sm_count);
}
bool tile_down_eligible(uint32_t f, const void* acts) { return f % kGroup == 0 && f <= 8192 && aligned(acts, 16); }

tf_status launch_tile_gate_up(tf_context* ctx, void* stream, const void* const* blobs, const tf_expert_offsets* offsets, const void* x,
                              void* acts, uint32_t d, uint32_t f, uint32_t top_k, const uint32_t* slot_map, uint32_t slots, const char* name) {
    const uint32_t ng = d / kGroup;
    const size_t smem = tile_gemv_smem(ng, 2);
    static DeviceSmemCache configured;
    if (smem > 48 * 1024)
        if (tf_status s = ensure_dynamic_smem(ctx, tile_gate_up_kernel, configured, smem)) return s;
    launch_pdl(tile_gate_up_kernel, dim3((f + kTileRows16 - 1) / kTileRows16, slots), dim3(kTileThreads), smem, static_cast<cudaStream_t>(stream),
               reinterpret_cast<const uint8_t* const*>(blobs), *offsets, static_cast<const uint16_t*>(x), static_cast<uint16_t*>(acts), ng, f, top_k,
               slot_map);
    return check_launch(ctx, name);
}

tf_status launch_tile_down(tf_context* ctx, void* stream, const void* const* blobs, const tf_expert_offsets* offsets, const void* acts,
                           const void* routing_w, const void* residual, void* y, uint32_t d, uint32_t f, uint32_t top_k, const char* name) {
    const uint32_t ng = f / kGroup;
    const size_t smem = tile_x_bytes(top_k, ng);
    static DeviceSmemCache configured;
    // whatever the size: the 48 KB that a launch may use unasked include the kernel's static array
    if (tf_status s = ensure_dynamic_smem(ctx, tile_down_kernel, configured, smem)) return s;
    launch_pdl(tile_down_kernel, dim3((d + kTileRows16 - 1) / kTileRows16), dim3(kTileThreads), smem, static_cast<cudaStream_t>(stream),
               reinterpret_cast<const uint8_t* const*>(blobs), *offsets, static_cast<const uint16_t*>(acts), static_cast<const uint16_t*>(routing_w),
               static_cast<const uint16_t*>(residual), static_cast<uint16_t*>(y), d, ng, top_k);
    return check_launch(ctx, name);
}

}  // namespace tf
