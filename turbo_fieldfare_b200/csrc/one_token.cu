// One token through a MoE block: the decode step of a single sequence (Runtime/Inference/RealForwardRunner.swift:1449-1693).
//
// What bounds it is latency: 37 MB of weights are 6 us of the HBM rate, and a layer is a chain of products that need each other's
// results. So a layer of a stack is three launches, each of which requests all of its weights at once:
//   front     norm of the hidden row (in every block) -> router logits | shared gate/up
//   gate/up   top-k of the logits (in every block) -> routed gate/up; one block writes ids, weights and routing tables
//   down      shared and routed down projections of 16 to 20 rows per block -> weighted sum -> residual add
// No sum crosses a block, so nothing waits on a ticket or an atomic. Weights that no kernel writes are requested before the wait
// for the previous launch; the down launch even knows its experts before that (see rank_experts), and has a place on every SM beside
// the gate/up launch. A 30-layer step: 855 us with the layered launches (router with selection and grouping, two of the shared
// expert, gate/up, down, combine with norm; 28.5 us a layer), 620 us here (20 to 21: front 4, gate/up 10 of which 3 are the wait for the first
// tile and 3 the stream, down 5). A block forward: 30.4 and 25.0 us.
//
// All sums have the bits of the layered kernels: parts of four 64-column groups, added in order (grouped.cu), and the norm's
// sum of squares in the order of residual_rmsnorm_kernel.
//
// A block forward alone takes six launches, the parts of the above: router | shared gate/up, routed gate/up, shared down, routed
// down, combine.
#include "async_copy.cuh"
#include "block.cuh"
#include "router.cuh"
#include "mma_gemv.cuh"

namespace tf {

constexpr int kTileRows16 = 16, kTilePart = 4;       // rows of an MMA tile, groups whose sum a warp forms
constexpr int kOneWarps = 11;                       // a warp per part of the production width (2816 columns)
constexpr int kOneThreads = kOneWarps * kWarp;
constexpr int kOneDownWarps = 15, kOneDownThreads = kOneDownWarps * kWarp;      // two rounds of the production width's 30 units
constexpr int kOneRouterExperts = 8;                // per block, a warp each
constexpr uint32_t kOneMaxGroups = 48;              // 3072 columns, as the layered kernels
constexpr uint32_t kOneSlots = 4;                   // gate/up tiles in flight per block, 25.5 KB each at the production width
// Shared memory is also what keeps blocks of one launch apart: two gate/up blocks that met on an SM, because others were still taken when they
// started, ended 3 us after the rest. A gate/up block takes more than half of an SM's 228 KB, a front block more than half of what
// a down block leaves.
constexpr uint32_t kOneAloneBytes = 114 * 1024, kOneFrontBytes = 61 * 1024;
constexpr uint32_t kOneDownBytes = 108 * 1024;      // a block of the down launch beside a gate/up block
constexpr uint32_t kOneBlockDownBytes = 160 * 1024, kOneBlockMinD = 1024, kOneBlockMaxF = 2048;      // see one_token_size
constexpr uint32_t kErrTimeoutOneToken = 0x7F000041u;
static_assert(TF_MAX_ROUTER_EXPERTS <= kOneThreads, "a thread per expert");

struct OnePlanes {
    const uint8_t* W;
    const uint16_t* S;
    const uint16_t* B;
};

struct OneTokenArgs {
    uint32_t d, f, fs, experts, top_k;
    // front
    const uint16_t* x;             // the row, or with norm the hidden row
    const uint16_t* norm_w;
    uint16_t* x_out;               // with norm: the normed row
    float eps;
    uint32_t router_blocks;        // the first blocks of the front launch
    uint32_t behind_router;        // front launch of the shared expert alone, right behind the one of the router alone
    OnePlanes router;
    const uint16_t* eff;
    const float* logit_bias;
    float* logits;
    OnePlanes shared[3];           // gate, up, down
    uint16_t* shared_act;
    // routed experts
    const uint8_t* pool;
    uint64_t stride;
    tf_expert_offsets off;
    const uint16_t* per_expert_scale;
    uint32_t* indices;
    uint16_t* weights;
    RouterGroupOut routes;
    uint16_t* acts;
    // down
    uint16_t* shared_y;            // fp16 [d] (shared part alone)
    float* partials;               // fp32 [top_k, d] (routed part alone)
    uint16_t* hidden;              // updated in place (both)
    uint32_t* error;
};

// Sixteen activations of a row, 64 G + 16 t ...: the B fragments of (G, t) and, in the lane with t == 0, the group's sum at 2^-24.
// Whole warps.
__device__ __forceinline__ void one_stage_frag(const uint32_t (&r)[8], bool ok, uint32_t item, uint32_t* frag, float* xsum) {
    float sum = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&r[q]));
        sum += v.x + v.y;
    }
    sum += __shfl_xor_sync(kFullMask, sum, 1);
    sum += __shfl_xor_sync(kFullMask, sum, 2);
    if (!ok) return;
    if ((item & 3) == 0) xsum[item >> 2] = sum * 5.9604644775390625e-08f;
    uint32_t f[8];
    gm_make_frag(r, f);
    uint4* dst = reinterpret_cast<uint4*>(frag + (size_t)item * 8);
    dst[0] = make_uint4(f[0], f[1], f[2], f[3]);
    dst[1] = make_uint4(f[4], f[5], f[6], f[7]);
}

// A warp's sum over the four groups of a part for MMA rows g (x) and g + 8 (y), in every lane: the arithmetic and order of
// grouped_ksplit_kernel, with x in all eight columns of the B operand. codes0, codes1: this lane's 8 bytes of the two rows in the part's first
// group; scales, biases: of row g; row8: from there to those of row g + 8. A part that reaches past the last group (left < 4) reads codes
// that follow (its activations are zero there) and takes its scales as zero. FOURS: ng % 4 == 0, a row's scales of a part are one 8-byte word. COLUMNS:
// frag and xsum may differ from one g to the next; column g then holds the x of lanes g, and the lanes with t == g / 2 have column g, an
// odd one if `odd`. What takes the time is a chain of latencies: loads, four MMAs, eight FMAs (without the scales' loads 0.75 of it, without MMAs
// 0.83, without masks 0.94); as a loop of two groups each it took 5 % longer, with the weights in registers before the activations as long.
template <bool FOURS, bool COLUMNS>
__device__ __forceinline__ float2 one_part(const uint8_t* codes0, const uint8_t* codes1, const uint16_t* scales, const uint16_t* biases, uint32_t row8,
                                           const uint32_t* frag, const float* xsum, uint32_t left, bool odd) {
    const uint4* f4 = reinterpret_cast<const uint4*>(frag) + (threadIdx.x & 3) * 2;
    uint2 wa[kTilePart], wb[kTilePart];
    float c[kTilePart][4], zero[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) asm volatile("mov.f32 %0, 0f00000000;" : "=f"(zero[j]));
#pragma unroll
    for (int i = 0; i < kTilePart; ++i) {
        wa[i] = *reinterpret_cast<const uint2*>(codes0 + i * 32);
        wb[i] = *reinterpret_cast<const uint2*>(codes1 + i * 32);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint4 f[kTilePart];
#pragma unroll
        for (int i = 0; i < kTilePart; ++i) f[i] = f4[i * 8 + h];
#pragma unroll
        for (int i = 0; i < kTilePart; ++i) {
            const uint32_t wx = h ? wa[i].y : wa[i].x, wy = h ? wb[i].y : wb[i].x;
            if (h == 0) gm_mma(c[i], wx & 0x000F000Fu, wy & 0x000F000Fu, (wx >> 8) & 0x000F000Fu, (wy >> 8) & 0x000F000Fu, f[i].x, f[i].y, zero);
            else gm_mma(c[i], wx & 0x000F000Fu, wy & 0x000F000Fu, (wx >> 8) & 0x000F000Fu, (wy >> 8) & 0x000F000Fu, f[i].x, f[i].y, c[i]);
        }
#pragma unroll
        for (int i = 0; i < kTilePart; ++i) {
            const uint32_t wx = h ? wa[i].y : wa[i].x, wy = h ? wb[i].y : wb[i].x;
            gm_mma(c[i], wx & 0x00F000F0u, wy & 0x00F000F0u, (wx >> 8) & 0x00F000F0u, (wy >> 8) & 0x00F000F0u, f[i].z, f[i].w, c[i]);
        }
    }
    const float4 xs = *reinterpret_cast<const float4*>(xsum);
    float2 acc = make_float2(0.0f, 0.0f);
    uint2 s0, s1, b0, b1;
    if constexpr (FOURS) {
        s0 = *reinterpret_cast<const uint2*>(scales); s1 = *reinterpret_cast<const uint2*>(scales + row8);
        b0 = *reinterpret_cast<const uint2*>(biases); b1 = *reinterpret_cast<const uint2*>(biases + row8);
    }
#pragma unroll
    for (int i = 0; i < kTilePart; ++i) {
        float sa, sb, ba, bb;
        if constexpr (FOURS) {
            const uint32_t w0 = i < 2 ? s0.x : s0.y, w1 = i < 2 ? s1.x : s1.y, w2 = i < 2 ? b0.x : b0.y, w3 = i < 2 ? b1.x : b1.y;
            sa = __uint_as_float((i & 1) ? w0 & 0xFFFF0000u : w0 << 16); sb = __uint_as_float((i & 1) ? w1 & 0xFFFF0000u : w1 << 16);
            ba = __uint_as_float((i & 1) ? w2 & 0xFFFF0000u : w2 << 16); bb = __uint_as_float((i & 1) ? w3 & 0xFFFF0000u : w3 << 16);
        } else {
            const bool in = (uint32_t)i < left;
            sa = in ? bf16_bits_to_float(scales[i]) : 0.0f; sb = in ? bf16_bits_to_float(scales[row8 + i]) : 0.0f;
            ba = in ? bf16_bits_to_float(biases[i]) : 0.0f; bb = in ? bf16_bits_to_float(biases[row8 + i]) : 0.0f;
        }
        const float x = i == 0 ? xs.x : i == 1 ? xs.y : i == 2 ? xs.z : xs.w;
        acc.x = fmaf(sa, COLUMNS && odd ? c[i][1] : c[i][0], fmaf(ba, x, acc.x));
        acc.y = fmaf(sb, COLUMNS && odd ? c[i][3] : c[i][2], fmaf(bb, x, acc.y));
    }
    return make_float2(acc.x * 16777216.0f, acc.y * 16777216.0f);
}

__host__ __device__ inline uint32_t one_parts(uint32_t ng) { return (ng + kTilePart - 1) / kTilePart; }

// The parts' sums of a row, added in order; all loads before the first addition.
__device__ __forceinline__ float one_add_parts(const float* sums, uint32_t stride, uint32_t parts) {
    constexpr uint32_t kMax = kOneMaxGroups / kTilePart;
    float v[kMax];
#pragma unroll
    for (uint32_t p = 0; p < kMax; ++p) v[p] = p < parts ? sums[p * stride] : 0.0f;
    float acc = v[0];
#pragma unroll
    for (uint32_t p = 1; p < kMax; ++p)
        if (p < parts) acc += v[p];
    return acc;
}

// Gate/up tiles: eight gate rows and the eight up rows of the same index, in shared memory. Codes come as four copies of four rows
// (gate 0-3, gate 4-7, up 0-3, up 4-7), 32 bytes of padding behind each: MMA row m is row m / 4 of copy m % 4, so the four rows that a
// half warp reads at once lie 32 bytes apart in the banks (a row is a multiple of 32 bytes, four rows one of 128).
// Straight loads into the MMA's registers, 8 bytes a lane, took 20 us for the 17.8 MB of a layer's gate/up launch: a lane's scales are
// 2 bytes of a sector each.
struct OneTiles {
    uint32_t ng, slots, tiles;                 // tiles: the most that a block has
    __host__ __device__ uint32_t copy() const { return ng * 32 * 4 + 32; }
    __host__ __device__ uint32_t plane() const { return ng * 2 * 8; }
    __host__ __device__ uint32_t bytes() const { return 4 * copy() + 4 * plane(); }
    __host__ __device__ uint32_t off_frag() const { return slots * bytes(); }
    __host__ __device__ uint32_t off_xsum() const { return off_frag() + one_parts(ng) * kTilePart * 128; }          // whole parts
    __host__ __device__ uint32_t off_sums() const { return off_xsum() + one_parts(ng) * kTilePart * 4; }
    __host__ __device__ uint32_t off_bars() const { return off_sums() + tiles * one_parts(ng) * 64; }                // landed | free
    __host__ __device__ size_t total() const { return off_bars() + slots * 16; }
};
// Router blocks: [d] fp32 activations, the experts' codes, scales and biases, a barrier.
struct OneRouterSmem {
    uint32_t ng;
    __host__ __device__ uint32_t off_codes() const { return ng * kGroup * 4; }
    __host__ __device__ uint32_t off_scales() const { return off_codes() + kOneRouterExperts * ng * kGroup; }
    __host__ __device__ uint32_t off_biases() const { return off_scales() + kOneRouterExperts * ng * 2; }
    __host__ __device__ uint32_t off_bar() const { return off_biases() + kOneRouterExperts * ng * 2 + 16; }
    __host__ __device__ size_t total() const { return off_bar() + 8; }
};

struct OneGateUp {
    const uint8_t* w[2];
    const uint16_t* s[2];
    const uint16_t* b[2];
    uint16_t* out;
};
// Lanes 0-7 of a warp request a tile: four copies of codes, four planes.
__device__ __forceinline__ void one_request_tile(const OneTiles& lay, uint32_t smem, uint32_t bar, const OneGateUp& p, uint32_t row0) {
    const uint32_t lane = threadIdx.x % kWarp;
    if (lane == 0) mbar_arrive_expect_tx(bar, 16 * lay.ng * 32 + 4 * lay.plane());
    __syncwarp();
    const uint32_t m = (lane >> 1) & 1, k = lane & 1;
    if (lane < 4)
        bulk_copy_g2s(smem + lane * lay.copy(), (m ? p.w[1] : p.w[0]) + (size_t)(row0 + k * 4) * (lay.ng * 32), 4 * lay.ng * 32, bar);
    else if (lane < 8)
        bulk_copy_g2s(smem + 4 * lay.copy() + (lane - 4) * lay.plane(), (m ? (k ? p.b[1] : p.s[1]) : (k ? p.b[0] : p.s[0])) + (size_t)row0 * lay.ng, lay.plane(), bar);
}
// A warp's part p of a tile in shared memory. MMA row m: copy m % 4, row m / 4 of it; rows g and g + 8 share the copy.
template <bool FOURS>
__device__ __forceinline__ void one_tile_part(const OneTiles& lay, uint8_t* smem, uint32_t slot, uint32_t tile, uint32_t p) {
    const uint32_t lane = threadIdx.x % kWarp, g = lane >> 2, t = lane & 3, rb = lay.ng * 32;
    const uint8_t* at = smem + slot * lay.bytes();
    const uint8_t* codes = at + (g & 3) * lay.copy() + (g >> 2) * rb + t * 8 + p * (kTilePart * 32);
    const uint16_t* sc = reinterpret_cast<const uint16_t*>(at + 4 * lay.copy() + ((g & 3) >> 1) * 2 * lay.plane() + ((g & 1) * 4 + (g >> 2)) * lay.ng * 2) + p * kTilePart;
    const float2 v = one_part<FOURS, false>(codes, codes + 2 * rb, sc, sc + lay.plane() / 2, 2 * lay.ng, reinterpret_cast<const uint32_t*>(smem + lay.off_frag()) + (size_t)p * (kTilePart * 32),
                                     reinterpret_cast<const float*>(smem + lay.off_xsum()) + p * kTilePart, lay.ng - p * kTilePart, false);
    float* dst = reinterpret_cast<float*>(smem + lay.off_sums()) + ((size_t)tile * one_parts(lay.ng) + p) * 16 + g;
    if (t == 0) { dst[0] = v.x; dst[8] = v.y; }
}
// act = half(gelu(gate) * up) of a block's tiles, behind a barrier. HALF_GATE: gate and up are rounded to fp16 first (the shared expert:
// Kernels/MoE/SharedExpertInt4.swift:62-93). resolve(tile, matrices, row0). !live: nothing is stored.
template <bool HALF_GATE, typename Resolve>
__device__ __forceinline__ void one_tiles_finish(const OneTiles& lay, const uint8_t* smem, uint32_t count, const Resolve& resolve, bool live) {
    const uint32_t parts = one_parts(lay.ng);
    const float* sums = reinterpret_cast<const float*>(smem + lay.off_sums());
    for (uint32_t i = threadIdx.x; i < ((count * 16 + 31u) & ~31u); i += blockDim.x) {
        const uint32_t tile = i / 16 < count ? i / 16 : 0u, m = i % 16;
        float acc = one_add_parts(sums + (size_t)tile * parts * 16 + m, 16, parts);
        if constexpr (HALF_GATE) acc = __half2float(__float2half_rn(acc));
        const float up = __shfl_down_sync(kFullMask, acc, 2);
        if (live && i < count * 16 && (m & 2) == 0) {
            OneGateUp mats;
            uint32_t row0;
            resolve(tile, mats, row0);
            mats.out[row0 + (m & 1) * 4 + (m >> 2)] = __half_as_ushort(__float2half_rn(gelu_tanh(acc) * up));
        }
    }
}

// ---- front: norm, router logits, shared gate/up ----
template <bool NORM, bool FOURS>          // FOURS: ng % 4 == 0
__global__ void __launch_bounds__(kOneThreads, 2)
one_token_front_kernel(const OneTokenArgs a, uint32_t most) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float red[kWarp];
    const uint32_t tid = threadIdx.x, warp = tid / kWarp, lane = tid % kWarp, ng = a.d / kGroup;
    const bool router = blockIdx.x < a.router_blocks;
    const uint32_t e0 = blockIdx.x * kOneRouterExperts, expert = e0 + warp;
    const bool scores = router && warp < (uint32_t)kOneRouterExperts && expert < a.experts;
    const OneTiles lay{ng, most, most};
    const uint32_t tiles = a.fs / 8, blocks = gridDim.x - a.router_blocks, block = blockIdx.x - a.router_blocks;
    const uint32_t begin = router ? 0u : (uint32_t)((uint64_t)tiles * block / blocks), count = router ? 0u : (uint32_t)((uint64_t)tiles * (block + 1) / blocks) - begin;
    const OneRouterSmem rlay{ng};
    float* xf = reinterpret_cast<float*>(smem);                                   // router blocks
    const uint16_t* srows = reinterpret_cast<const uint16_t*>(smem + rlay.off_scales());
    const uint16_t* brows = reinterpret_cast<const uint16_t*>(smem + rlay.off_biases());
    const uint32_t base = smem_addr_u32(smem), bar = base + (router ? rlay.off_bar() : lay.off_bars());
    // Weights first: nothing writes them on this stream.
    const auto resolve = [&](uint32_t i, OneGateUp& m, uint32_t& row) {
        m = OneGateUp{{a.shared[0].W, a.shared[1].W}, {a.shared[0].S, a.shared[1].S}, {a.shared[0].B, a.shared[1].B}, a.shared_act};
        row = (begin + i) * 8;
    };
    if (warp == 0) {
        if (router && lane == 0) mbar_init(bar, 1);
        if (!router && lane < most) { mbar_init(bar + lane * 8, 1); mbar_init(bar + (most + lane) * 8, one_parts(ng) < (uint32_t)kOneWarps ? one_parts(ng) : (uint32_t)kOneWarps); }
        fence_proxy_async();
        __syncwarp();
        if (!router) {
            for (uint32_t i = 0; i < count; ++i) {
                OneGateUp m;
                uint32_t row;
                resolve(i, m, row);
                one_request_tile(lay, base + i * lay.bytes(), bar + i * 8, m, row);
            }
        } else if (lane == 0) {
            const uint32_t n = a.experts - e0 < (uint32_t)kOneRouterExperts ? a.experts - e0 : (uint32_t)kOneRouterExperts;
            // planes of fewer rows than a block's may end off the 16-byte grid of a bulk copy: by threads then, below
            mbar_arrive_expect_tx(bar, n * a.d);
            bulk_copy_g2s(base + rlay.off_codes(), a.router.W + (size_t)e0 * a.d, n * a.d, bar);
        }
    } else if (router) {
        const uint32_t n = (a.experts - e0 < (uint32_t)kOneRouterExperts ? a.experts - e0 : (uint32_t)kOneRouterExperts) * ng;
        for (uint32_t i = tid - kWarp; i < n; i += kOneThreads - kWarp) {
            const_cast<uint16_t*>(srows)[i] = a.router.S[(size_t)e0 * ng + i];
            const_cast<uint16_t*>(brows)[i] = a.router.B[(size_t)e0 * ng + i];
        }
    }
    const bool ok = tid < ng * 4;                                                 // sixteen columns each
    uint4 nw[2], ew[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        nw[j] = NORM && ok ? __ldg(reinterpret_cast<const uint4*>(a.norm_w) + tid * 2 + j) : make_uint4(0u, 0u, 0u, 0u);
        ew[j] = router && ok ? __ldg(reinterpret_cast<const uint4*>(a.eff) + tid * 2 + j) : make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();                      // barriers initialised, router planes staged
    // Router and shared expert as two launches (a block forward): the first lets the second in after its own wait, so what the
    // second reads is complete when it starts (see EarlyTable), and it waits only before it ends, for the launches behind it.
    if (a.router_blocks != gridDim.x) pdl_launch_dependents();
    if (!a.behind_router) pdl_wait();
    if (a.router_blocks == gridDim.x) pdl_launch_dependents();
    uint32_t r[8];
    {
        const EarlyTable<uint4> row{reinterpret_cast<const uint4*>(a.x)};
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        const uint4 lo = ok ? row.at<true>(tid * 2) : zero, hi = ok ? row.at<true>(tid * 2 + 1) : zero;
        r[0] = lo.x; r[1] = lo.y; r[2] = lo.z; r[3] = lo.w; r[4] = hi.x; r[5] = hi.y; r[6] = hi.z; r[7] = hi.w;
    }
    if constexpr (NORM) {
        // the sum of squares in the order of residual_rmsnorm_kernel: 128 threads, slices of 8 columns
        constexpr uint32_t kNormThreads = 128, kNormSlices = 3;
        static_assert(kOneMaxGroups * kGroup <= kNormThreads * kNormSlices * 8, "columns");
        if (tid < kNormThreads) {
            uint4 v[kNormSlices];
#pragma unroll
            for (uint32_t s = 0; s < kNormSlices; ++s) {
                const uint32_t i = tid + s * kNormThreads;
                v[s] = i < a.d / 8 ? reinterpret_cast<const uint4*>(a.x)[i] : make_uint4(0u, 0u, 0u, 0u);       // zeros add nothing
            }
            float acc = 0.0f;
#pragma unroll
            for (uint32_t s = 0; s < kNormSlices; ++s) {
                const uint32_t w[4] = {v[s].x, v[s].y, v[s].z, v[s].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                    acc = fmaf(p.x, p.x, acc); acc = fmaf(p.y, p.y, acc);
                }
            }
            acc = warp_sum(acc);
            if (lane == 0) red[warp] = acc;
        }
        __syncthreads();
        const float tot = warp_sum(lane < kNormThreads / kWarp ? red[lane] : 0.0f);
        const float inv = rsqrtf(tot / (float)a.d + a.eps);
        const uint32_t ww[8] = {nw[0].x, nw[0].y, nw[0].z, nw[0].w, nw[1].x, nw[1].y, nw[1].z, nw[1].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&r[j]));
            const __half2 n = __floats2half2_rn(p.x * inv * bf16_bits_to_float((uint16_t)(ww[j] & 0xFFFFu)), p.y * inv * bf16_bits_to_float((uint16_t)(ww[j] >> 16)));
            r[j] = *reinterpret_cast<const uint32_t*>(&n);
        }
        if (blockIdx.x == 0 && ok) {
            reinterpret_cast<uint4*>(a.x_out)[tid * 2] = make_uint4(r[0], r[1], r[2], r[3]);
            reinterpret_cast<uint4*>(a.x_out)[tid * 2 + 1] = make_uint4(r[4], r[5], r[6], r[7]);
        }
    }
    if (!router) {
        if (tid < ((one_parts(ng) * 16 + 31u) & ~31u))
            one_stage_frag(r, tid < one_parts(ng) * 16, tid, reinterpret_cast<uint32_t*>(smem + lay.off_frag()), reinterpret_cast<float*>(smem + lay.off_xsum()));
        __syncthreads();
        const uint32_t parts = one_parts(ng);
        bool landed = true;
        for (uint32_t i = 0; i < count; ++i) {
            landed = mbar_wait(bar + i * 8, 0) && landed;
            for (uint32_t p = warp; p < parts; p += kOneWarps) one_tile_part<FOURS>(lay, smem, i, i, p);
        }
        if (!landed) {
            if (lane == 0) atomicCAS(a.error, 0u, kErrTimeoutOneToken);
            for (uint32_t i = 0; i < count; ++i) mbar_wait(bar + i * 8, 0);           // once more (bounded) for the copies in flight
        }
        __syncthreads();
        one_tiles_finish<true>(lay, smem, count, resolve, true);
        if (a.behind_router) pdl_wait();
        return;
    }
    if (ok) {
        const uint32_t ws[8] = {ew[0].x, ew[0].y, ew[0].z, ew[0].w, ew[1].x, ew[1].y, ew[1].z, ew[1].w};
        float4* dst = reinterpret_cast<float4*>(xf + tid * 16);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 p = __half22float2(*reinterpret_cast<const __half2*>(&r[2 * j])), q = __half22float2(*reinterpret_cast<const __half2*>(&r[2 * j + 1]));
            dst[j] = make_float4(__fmul_rn(p.x, bf16_bits_to_float((uint16_t)(ws[2 * j] & 0xFFFFu))), __fmul_rn(p.y, bf16_bits_to_float((uint16_t)(ws[2 * j] >> 16))),
                                 __fmul_rn(q.x, bf16_bits_to_float((uint16_t)(ws[2 * j + 1] & 0xFFFFu))), __fmul_rn(q.y, bf16_bits_to_float((uint16_t)(ws[2 * j + 1] >> 16))));
        }
    }
    __syncthreads();
    if (!scores) return;
    if (!mbar_wait(bar, 0)) {
        if (lane == 0) atomicCAS(a.error, 0u, kErrTimeoutOneToken);
        mbar_wait(bar, 0);                              // once more (bounded) for the copy in flight
    }
    // the canonical logit (router.cu)
    float acc = 0.0f;
    const uint8_t* codes = smem + rlay.off_codes() + warp * a.d + lane * 2;
    const float* xl = xf + lane * 2;
#pragma unroll 4
    for (uint32_t g = 0; g < ng; ++g) {
        const uint32_t w = *reinterpret_cast<const uint16_t*>(codes + g * kGroup);
        // byte -> float through the 2^23 mantissa trick (exact for 0...255)
        const float q0 = __uint_as_float(0x4B000000u | (w & 0xFFu)) - 8388608.0f, q1 = __uint_as_float(0x4B000000u | (w >> 8)) - 8388608.0f;
        const float2 xv = *reinterpret_cast<const float2*>(xl + g * kGroup);
        const float p = __fmaf_rn(q1, xv.y, __fmul_rn(q0, xv.x));
        acc = __fmaf_rn(bf16_bits_to_float(srows[warp * ng + g]), p, acc);
        acc = __fmaf_rn(bf16_bits_to_float(brows[warp * ng + g]), __fadd_rn(xv.x, xv.y), acc);
    }
    float logit = warp_sum(acc);
    if (a.logit_bias) logit = __fadd_rn(logit, a.logit_bias[expert]);
    if (lane == 0) a.logits[expert] = logit;
}

// ---- the selected experts, in every block that needs them ----
struct OneTokenSelection {
    float score[TF_MAX_ROUTER_EXPERTS];        // later the block's hidden values
    __align__(16) uint32_t key[TF_MAX_ROUTER_EXPERTS];
    uint32_t expert[TF_MAX_TOP_K];             // by rank
    uint16_t weight[TF_MAX_TOP_K];
};
// The experts of warp_select_topk, by counting: an expert's rank is the number of higher scores, two threads per expert. Equal scores
// meet at one rank: the lowest index takes it, and if that leaves a rank of the top_k empty, equal scores of lower indices
// are counted, too. The selection's rounds of warp-wide maxima take 1.5 us, this 0.2. Rows with fewer than top_k selectable logits go
// through the rounds. Logits come past L1: the caller may not have waited (see EarlyTable).
__device__ __forceinline__ void rank_experts(const OneTokenArgs& a, OneTokenSelection& sel, bool live) {
    const uint32_t tid = threadIdx.x, E = a.experts, words = (E + 3) / 4;
    bool selectable = false;
    if (tid < words * 4) {
        const EarlyTable<uint32_t> logits{reinterpret_cast<const uint32_t*>(a.logits)};
        float v = tid < E ? (float)tid : -INFINITY;               // !live: any order
        if (live && tid < E) v = __uint_as_float(logits.at<true>(tid));
        const uint32_t key = tid < E ? topk_score_key(v) : 0u;
        sel.score[tid] = v;
        sel.key[tid] = key;
        selectable = key > 0x007FFFFFu;             // above -inf
    }
    if (tid < TF_MAX_TOP_K) sel.expert[tid] = 0xFFFFFFFFu;
    const uint32_t n = (uint32_t)__syncthreads_count(selectable);
    if (n < a.top_k) {
        if (tid < kWarp) warp_select_topk(sel.score, E, a.top_k, a.per_expert_scale, sel.expert, sel.weight, (int)tid);
        __syncthreads();
        return;
    }
    const uint32_t half = tid & 1u, mid = words / 2, first = half ? mid : 0u, last = half ? words : mid;
    const uint4* keys = reinterpret_cast<const uint4*>(sel.key);
    for (uint32_t base = 0; base < E; base += blockDim.x / 2) {
        const uint32_t e = base + (tid >> 1);
        if (base + (tid & ~31u) / 2 >= E) break;                        // whole warps
        const uint32_t mine = e < E ? sel.key[e] : 0u;
        uint32_t better = 0;
#pragma unroll 8
        for (uint32_t w = first; w < last; ++w) {
            const uint4 k = keys[w];
            better += (k.x > mine ? 1u : 0u) + (k.y > mine ? 1u : 0u) + (k.z > mine ? 1u : 0u) + (k.w > mine ? 1u : 0u);
        }
        better += __shfl_xor_sync(kFullMask, better, 1);
        if (half == 0 && mine > 0x007FFFFFu && better < a.top_k) atomicMin(&sel.expert[better], e);
    }
    __syncthreads();
    bool empty = false;
#pragma unroll
    for (int r = 0; r < TF_MAX_TOP_K; ++r) empty = empty || ((uint32_t)r < a.top_k && sel.expert[r] == 0xFFFFFFFFu);
    if (!empty) return;
    __syncthreads();
    for (uint32_t e = tid; e < E; e += blockDim.x) {
        const uint32_t mine = sel.key[e];
        uint32_t better = 0;
        for (uint32_t o = 0; o < E; ++o) better += sel.key[o] > mine || (sel.key[o] == mine && o < e) ? 1u : 0u;
        if (mine > 0x007FFFFFu && better < a.top_k) sel.expert[better] = e;
    }
    __syncthreads();
}

// ---- routed gate/up: persistent blocks, all tiles of a block requested at once (five at the production width) ----
template <bool FOURS>
__global__ void __launch_bounds__(kOneThreads + kWarp, 2)
one_token_gate_up_kernel(const OneTokenArgs a, uint32_t slots, uint32_t most) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ OneTokenSelection sel;
    const uint32_t tid = threadIdx.x, warp = tid / kWarp, lane = tid % kWarp, ng = a.d / kGroup, per_expert = a.f / 8;
    const OneTiles lay{ng, slots, most};
    const uint32_t base = smem_addr_u32(smem), bars = base + lay.off_bars();
    if (tid < slots) { mbar_init(bars + tid * 8, 1); mbar_init(bars + (slots + tid) * 8, one_parts(ng) < (uint32_t)kOneWarps ? one_parts(ng) : (uint32_t)kOneWarps); }
    if (warp == 0) fence_proxy_async();
    const uint32_t blocks = gridDim.x - 1;
    if (blockIdx.x == blocks) {
        // the last block: ids, weights and the routing tables
        pdl_wait();
        pdl_launch_dependents();
        if (tid < a.experts) sel.score[tid] = a.logits[tid];
        __syncthreads();
        if (warp == 0) warp_select_topk(sel.score, a.experts, a.top_k, a.per_expert_scale, a.indices, a.weights, (int)tid);
        __syncthreads();
        group_one_token(a.indices, a.weights, a.top_k, a.experts, a.routes, smem);
        return;
    }
    const uint32_t total = per_expert * a.top_k;
    const uint32_t begin = (uint32_t)((uint64_t)total * blockIdx.x / blocks), count = (uint32_t)((uint64_t)total * (blockIdx.x + 1) / blocks) - begin;
    const auto resolve = [&](uint32_t i, OneGateUp& m, uint32_t& row0) {
        const uint32_t slot = (begin + i) / per_expert;
        row0 = (begin + i - slot * per_expert) * 8;
        const uint8_t* blob = a.pool + (uint64_t)sel.expert[slot] * a.stride;
        m.w[0] = blob + a.off.gate_w_off; m.w[1] = blob + a.off.up_w_off;
        m.s[0] = reinterpret_cast<const uint16_t*>(blob + a.off.gate_s_off); m.s[1] = reinterpret_cast<const uint16_t*>(blob + a.off.up_s_off);
        m.b[0] = reinterpret_cast<const uint16_t*>(blob + a.off.gate_b_off); m.b[1] = reinterpret_cast<const uint16_t*>(blob + a.off.up_b_off);
        m.out = a.acts + (size_t)slot * a.f;
    };
    // Twice: the first pass, while the launch waits, moves no data and stores nothing; it brings the instructions into the SM's cache (some
    // 45 ns for every eight of them otherwise, on the way from the logits to the activations).
#pragma unroll 1
    for (uint32_t pass = 0; pass < 2; ++pass) {
        const bool live = pass == 1, ok = live && tid < ng * 4;
        if (live) {
            pdl_wait();
            pdl_launch_dependents();      // after the wait: the down launch reads the logits and the shared activations early
        }
        uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
        if (ok) { lo = reinterpret_cast<const uint4*>(a.x)[tid * 2]; hi = reinterpret_cast<const uint4*>(a.x)[tid * 2 + 1]; }
        rank_experts(a, sel, live);                 // with block barriers: the mbarriers are initialised
        // a tile by each of the last warps (the first ones stage the activations)
        for (uint32_t i = kOneWarps - warp; live && i < slots && i < count; i += kOneWarps + 1) {
            OneGateUp m;
            uint32_t row0;
            resolve(i, m, row0);
            one_request_tile(lay, base + i * lay.bytes(), bars + i * 8, m, row0);
        }
        const uint32_t r[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        if (tid < ((one_parts(ng) * 16 + 31u) & ~31u))
            one_stage_frag(r, tid < one_parts(ng) * 16, tid, reinterpret_cast<uint32_t*>(smem + lay.off_frag()), reinterpret_cast<float*>(smem + lay.off_xsum()));
        __syncthreads();
        const uint32_t n = live ? count : 1u, parts = one_parts(ng);
        bool landed = true;
        uint32_t slot = 0, use = 0;
        if (warp < (uint32_t)kOneWarps) {
            for (uint32_t i = 0; i < n && warp < parts; ++i) {
                if (live && !mbar_wait(bars + slot * 8, use & 1)) {
                    landed = false;
                    // once more (bounded) for the copies in flight: this tile's and those of the other slots, no others have been requested
                    // since this slot is not free
                    for (uint32_t k = i; k < n && k < i + slots; ++k) mbar_wait(bars + k % slots * 8, (k / slots) & 1);
                    break;
                }
                for (uint32_t p = warp; p < parts; p += kOneWarps) one_tile_part<FOURS>(lay, smem, slot, i, p);
                __syncwarp();                // the sums, of all loads from the slot, have been stored
                if (live && lane == 0) mbar_arrive(bars + (slots + slot) * 8);
                if (++slot == slots) { slot = 0; ++use; }
            }
        } else if (live) {
            // the last warp requests the other tiles as slots become free
            for (uint32_t i = slots; i < count; ++i) {
                if (!mbar_wait(bars + (slots + slot) * 8, use & 1)) { landed = false; break; }
                if (lane == 0) fence_proxy_async();          // the slot was last read through the generic proxy
                __syncwarp();
                OneGateUp m;
                uint32_t row0;
                resolve(i, m, row0);
                one_request_tile(lay, base + slot * lay.bytes(), bars + slot * 8, m, row0);
                if (++slot == slots) { slot = 0; ++use; }
            }
        }
        if (!landed && lane == 0) atomicCAS(a.error, 0u, kErrTimeoutOneToken);
        __syncthreads();
        one_tiles_finish<false>(lay, smem, n, resolve, live);
        __syncthreads();
    }
}

// ---- down ----
// A block takes `rows` rows, 16 and a multiple of four more, or four less (one block per SM: 20 and 16 at the production width). Shared memory: codes
// of the shared matrix' rows and of the slots', their scales and biases, x fragments, sums. A plane of scales need not start or end on
// the 16 bytes of a bulk copy: the copy takes the whole 16-byte words around it.
struct OneDownSmem {
    uint32_t ngs, ngf, slots, rows;            // groups of the shared matrix (0: not part of the launch) and of a slot
    __host__ __device__ uint32_t codes(uint32_t ng) const { return ng * 32 * rows; }
    __host__ __device__ uint32_t plane(uint32_t ng) const { return ((ng * 2 * rows + 15u) & ~15u) + 16; }
    __host__ __device__ uint32_t matrix(uint32_t ng) const { return ng ? codes(ng) + 2 * plane(ng) : 0u; }          // codes, scales, biases
    __host__ __device__ uint32_t vectors() const { return parts() * kTilePart; }                              // groups, in whole parts
    __host__ __device__ uint32_t off_slot(uint32_t s) const { return matrix(ngs) + s * matrix(ngf); }
    __host__ __device__ uint32_t off_frag() const { return off_slot(slots); }
    __host__ __device__ uint32_t off_xsum() const { return off_frag() + vectors() * 128; }
    __host__ __device__ uint32_t parts() const { return one_parts(ngs) + slots * one_parts(ngf); }
    __host__ __device__ uint32_t off_sums() const { return off_xsum() + vectors() * 4; }
    __host__ __device__ uint32_t off_bars() const { return off_sums() + ((parts() * rows * 4 + 15u) & ~15u); }
    __host__ __device__ size_t total() const { return off_bars() + 16; }
};
// Lane 0: n rows' codes, scales and biases from row0 on; the bytes that will land.
__device__ __forceinline__ uint32_t one_plane_bytes(uint32_t ng, uint32_t row0, uint32_t n) {
    return (((row0 + n) * ng * 2 + 15u) & ~15u) - ((row0 * ng * 2) & ~15u);
}
__device__ __forceinline__ void one_request_rows(const OneDownSmem& lay, uint32_t smem, uint32_t bar, const uint8_t* w, const uint8_t* s, const uint8_t* b, uint32_t ng,
                                                 uint32_t row0, uint32_t n) {
    const uint32_t first = (row0 * ng * 2) & ~15u, bytes = one_plane_bytes(ng, row0, n);
    bulk_copy_g2s(smem, w + (size_t)row0 * (ng * 32), n * ng * 32, bar);
    bulk_copy_g2s(smem + lay.codes(ng), s + first, bytes, bar);
    bulk_copy_g2s(smem + lay.codes(ng) + lay.plane(ng), b + first, bytes, bar);
}

template <bool SHARED, bool ROUTED>
__global__ void __launch_bounds__(kOneDownThreads, 2)
one_token_down_kernel(const OneTokenArgs a, uint32_t rows) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ OneTokenSelection sel;
    const uint32_t tid = threadIdx.x, warp = tid / kWarp, lane = tid % kWarp, quads = a.d / 4;
    const uint32_t row0 = quads * blockIdx.x / gridDim.x * 4, n = quads * (blockIdx.x + 1) / gridDim.x * 4 - row0;            // at most `rows`
    const OneDownSmem lay{SHARED ? a.fs / kGroup : 0u, a.f / kGroup, ROUTED ? a.top_k : 0u, rows};
    const uint32_t base = smem_addr_u32(smem), bar = base + lay.off_bars();       // [0] shared, [1] slots
    uint32_t* frag = reinterpret_cast<uint32_t*>(smem + lay.off_frag());
    float* xsum = reinterpret_cast<float*>(smem + lay.off_xsum());
    float* sums = reinterpret_cast<float*>(smem + lay.off_sums());
    pdl_launch_dependents();
    if (tid == 0) {
        mbar_init(bar, 1); mbar_init(bar + 8, 1);
        fence_proxy_async();
        if constexpr (SHARED) {
            mbar_arrive_expect_tx(bar, n * lay.ngs * 32 + 2 * one_plane_bytes(lay.ngs, row0, n));
            one_request_rows(lay, base, bar, a.shared[2].W, reinterpret_cast<const uint8_t*>(a.shared[2].S), reinterpret_cast<const uint8_t*>(a.shared[2].B), lay.ngs, row0, n);
        }
    }
    // The gate/up launch let this one in after its own wait, so the logits are complete: the experts are known, and their weights on
    // their way, while gate/up still runs.
    if constexpr (ROUTED) {
        rank_experts(a, sel, true);               // with block barriers: the mbarriers are initialised
        if (warp == 0) {
            if (lane == 0) mbar_arrive_expect_tx(bar + 8, a.top_k * (n * lay.ngf * 32 + 2 * one_plane_bytes(lay.ngf, row0, n)));
            __syncwarp();
            if (lane < a.top_k) {
                const uint8_t* blob = a.pool + (uint64_t)sel.expert[lane] * a.stride;
                one_request_rows(lay, base + lay.off_slot(lane), bar + 8, blob + a.off.down_w_off, blob + a.off.down_s_off, blob + a.off.down_b_off, lay.ngf, row0, n);
            }
        }
    } else {
        __syncthreads();
    }
    // First the shared expert's parts: its activations are complete (gate/up waited for them before it let this launch in). Then, behind
    // the wait for gate/up, the slots'; the first weights are in registers by then. One loop for both: the second time its instructions
    // are in the cache.
    const uint32_t parts_s = one_parts(lay.ngs), parts_f = one_parts(lay.ngf), g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (uint32_t phase = SHARED ? 0u : 1u; phase < (ROUTED ? 2u : 1u); ++phase) {
        const uint32_t begin = phase ? parts_s : 0u, end = phase ? lay.parts() : parts_s, ng = phase ? lay.ngf : lay.ngs, per = phase ? parts_f : parts_s;
        // Units of 16 rows x 4 groups. The rows beyond the 16th: a second such unit of the shared matrix (rows past the block's read its last
        // one and are not stored); of the slots two rows of all of them, row g of the MMA is slot g and its activations are column g.
        const uint32_t whole = end - begin, units = whole + (n <= (uint32_t)kTileRows16 ? 0u : phase ? (n - kTileRows16) / 2 * per : whole);
        const uint32_t rb = ng * 32, shift = ((row0 * ng * 2) & 15u) / 2;
        if (phase) {
            pdl_wait();
            if (SHARED && tid < n) sel.score[tid] = f16_bits_to_float(a.hidden[row0 + tid]);
            if (SHARED && tid < a.top_k) sel.weight[tid] = a.weights[tid];
        }
        // sixteen columns of a vector to a thread; vectors are filled up with zeros to whole parts
        for (uint32_t j = tid; j < ((whole * 16 + 31u) & ~31u); j += kOneDownThreads) {          // whole warps
            const uint32_t i = begin * 16 + j, slot = (j / 16) / per, in = j - slot * per * 16;
            uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
            if (j < whole * 16 && in < ng * 4) {
                const EarlyTable<uint4> row{reinterpret_cast<const uint4*>(phase ? a.acts + (size_t)slot * a.f : a.shared_act)};
                lo = row.at<true>(in * 2); hi = row.at<true>(in * 2 + 1);
            }
            const uint32_t r[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            one_stage_frag(r, j < whole * 16, i, frag, xsum);
        }
        __syncthreads();
        if (!mbar_wait(bar + phase * 8, 0)) {
            if (lane == 0) atomicCAS(a.error, 0u, kErrTimeoutOneToken);
            mbar_wait(bar + phase * 8, 0);              // once more (bounded) for the copies in flight
        }
        uint32_t q = 0, part = warp;                    // matrix (columns: pair of rows) and part of unit u
        bool second = false;
#pragma unroll 1
        for (uint32_t u = warp; u < units; u += kOneDownWarps, part += kOneDownWarps) {
            if (!second && u >= whole) { second = true; q = 0; part = u - whole; }
            while (part >= per) { part -= per; ++q; }
            const bool columns = phase && second;
            const uint32_t slot = columns ? (g < lay.slots ? g : 0u) : phase ? q : 0u;
            const uint32_t s0 = columns ? kTileRows16 + 2 * q : second ? kTileRows16 + g : g, s1 = columns ? s0 + 1 : s0 + 8;
            const uint32_t r0 = s0 < rows ? s0 : rows - 1, r1 = s1 < rows ? s1 : rows - 1;
            const uint8_t* m = smem + (phase ? lay.off_slot(slot) : 0u);
            const uint8_t* codes = m + part * (kTilePart * 32) + t * 8;
            const uint16_t* sc = reinterpret_cast<const uint16_t*>(m + lay.codes(ng)) + shift + r0 * ng + part * kTilePart;
            const uint32_t p = begin + slot * per + part;
            const float2 y = one_part<false, true>(codes + r0 * rb, codes + r1 * rb, sc, sc + lay.plane(ng) / 2, (r1 - r0) * ng, frag + (size_t)p * (kTilePart * 32),
                                            xsum + p * kTilePart, ng - part * kTilePart, columns && (g & 1));
            if (columns ? t == (g >> 1) && g < lay.slots : t == 0) {
                if (s0 < n) sums[p * rows + s0] = y.x;
                if (s1 < n) sums[p * rows + s1] = y.y;
            }
        }
    }
    if constexpr (!ROUTED) pdl_wait();
    __syncthreads();
    // a thread per row of every matrix adds the parts; the shared expert's output is stored as fp16
    const uint32_t mats = (SHARED ? 1u : 0u) + lay.slots;
    for (uint32_t i = tid; i < mats * rows; i += kOneDownThreads) {
        const uint32_t m = i / rows, row = i - m * rows;
        if (row >= n) continue;
        const bool shared = SHARED && m == 0;
        const uint32_t s = m - (SHARED ? 1u : 0u), first = shared ? 0u : parts_s + s * parts_f;
        float v = one_add_parts(sums + first * rows + row, rows, shared ? parts_s : parts_f);
        if (shared) v = __half2float(__float2half_rn(v));
        if constexpr (SHARED && ROUTED) sums[first * rows + row] = v;              // read by this thread only until now
        else if constexpr (SHARED) a.shared_y[row0 + row] = __half_as_ushort(__float2half_rn(v));
        else a.partials[(size_t)s * a.d + row0 + row] = v;
    }
    if constexpr (SHARED && ROUTED) {
        __syncthreads();
        if (tid < n) {
            float v[TF_MAX_TOP_K], acc = sums[tid];
#pragma unroll
            for (int s = 0; s < TF_MAX_TOP_K; ++s) v[s] = (uint32_t)s < a.top_k ? sums[(parts_s + s * parts_f) * rows + tid] : 0.0f;
#pragma unroll
            for (int s = 0; s < TF_MAX_TOP_K; ++s)
                if ((uint32_t)s < a.top_k) acc = __fadd_rn(acc, __fmul_rn(f16_bits_to_float(sel.weight[s]), v[s]));                    // moe.metal:473-480
            const float y = __half2float(__float2half_rn(acc));
            a.hidden[row0 + tid] = __half_as_ushort(__float2half_rn(sel.score[tid] + y));
        }
    }
}

// ---- host ----

// Blocks of the down launch, one per SM at the most or 16 rows each, their most rows and the shared memory of one (of the launch of both parts).
struct OneDownGrid { uint32_t blocks, rows; size_t bytes; };
static OneDownGrid one_down_grid(const tf_context* ctx, uint32_t d, uint32_t f, uint32_t fs, uint32_t top_k) {
    const uint32_t quads = d / 4, sixteens = d / kTileRows16;
    auto rows = [&](uint32_t blocks) { const uint32_t r = (quads + blocks - 1) / blocks * 4; return r < (uint32_t)kTileRows16 ? (uint32_t)kTileRows16 : r; };
    uint32_t blocks = sixteens < (uint32_t)ctx->sm_count ? sixteens : (uint32_t)ctx->sm_count;
    if (rows(blocks) > 2 * kTileRows16 || OneDownSmem{fs / kGroup, f / kGroup, top_k, rows(blocks)}.total() > kOneDownBytes) blocks = sixteens;
    return {blocks, rows(blocks), OneDownSmem{fs / kGroup, f / kGroup, top_k, rows(blocks)}.total()};
}
// Sizes that these launches take. A stack's layer: a block of the down launch has a place beside one of the gate/up launch (kOneDownBytes); a larger one
// requests its weights only when that has ended. us a layer, layered and here (d x f x fs, top_k; KB of a down block): 2816 x 704 x 2112, 8
// (105) 22.8, 19.5; 3072 x 1280 x 1152, 6 (98) 32.3, 27.3; 1024 x 2048 x 1024, 4 (101) 20.2, 18.6; 2816 x 960 x 2112, 8 (110) 31.1, 27.6;
// 2816 x 1088 x 1024, 8 (111) 22 to 31, 33; 2048 x 1408 x 2816, 6 (126) 24.8, 24.2; 2816 x 2816 x 704, 4 (132) 31.7, 35.6;
// 2048 x 1536 x 1536, 8 (153) 21.6, 27.6; 256 x 1024 x 2048, 8 (113) 18.7, 19.5; 3072 x 1536 x 3072, 8 (169) 29, 44.
// A block's two down launches have such a place up to larger sizes, and no side stream: 2048 x 1408 x 2816, 6 33.4, 28.0; 2048 x 1536 x 1536, 8
// 33.0, 29.2; 1024 x 1536 x 1536, 8 27.6, 26.4; but 512 x 1536 x 1536, 8 24.6, 25.0; 2816 x 2816 x 704, 4 31.0, 34.5; 3072 x 1536 x 3072, 8 42.5, 43.
static bool one_token_size(const tf_context* ctx, const tf_moe_layer* l, bool stack) {
    const size_t bytes = one_down_grid(ctx, l->d, l->f, l->fs, l->top_k).bytes;
    return bytes <= kOneDownBytes || (!stack && bytes <= kOneBlockDownBytes && l->d >= kOneBlockMinD && l->f <= kOneBlockMaxF);
}
// What the layered launches accept and these do not: other shapes, an 8-bit shared expert, workspaces of more tokens (fp16 partials), a
// tensor-core threshold of one token. Arguments that the layered launches refuse go there, too, and are refused.
bool one_token_eligible(const tf_context* ctx, const tf_moe_layer* l, const tf_workspace* ws, bool stack) {
    const bool shape = l->d % kGroup == 0 && l->f % kGroup == 0 && l->fs % kGroup == 0 && l->d > 0 && l->f > 0 && l->fs > 0 &&
                       l->d <= kOneMaxGroups * kGroup && l->f <= kOneMaxGroups * kGroup && l->fs <= kOneMaxGroups * kGroup &&
                       l->top_k > 0 && l->top_k <= TF_MAX_TOP_K && l->top_k <= l->num_experts && l->num_experts <= TF_MAX_ROUTER_EXPERTS;
    if (!shape || l->shared_bits == 8 || ws->max_tokens > 64 || ctx->shared_tensorcore_min_tokens <= 1 ||
        (ctx->tensorcore_min_tokens <= 1 && ws->x_sorted != nullptr))
        return false;
    const tf_projection* ps[4] = {&l->router, &l->shared_gate, &l->shared_up, &l->shared_down};
    const uint32_t rows[4] = {l->num_experts, l->fs, l->fs, l->d}, cols[4] = {l->d, l->d, l->d, l->fs};
    for (int i = 0; i < 4; ++i) {
        if (!ps[i]->weights || !ps[i]->scales || !ps[i]->biases || ps[i]->rows != rows[i] || ps[i]->cols != cols[i] ||
            !aligned(byte_ptr(ps[i]->weights, ps[i]->weights_off), 16) || !aligned(byte_ptr(ps[i]->scales, ps[i]->scales_off), 16) ||
            !aligned(byte_ptr(ps[i]->biases, ps[i]->biases_off), 16))
            return false;
    }
    const tf_expert_offsets& o = l->offsets;
    const uint32_t all[9] = {o.gate_w_off, o.gate_s_off, o.gate_b_off, o.up_w_off, o.up_s_off, o.up_b_off, o.down_w_off, o.down_s_off, o.down_b_off};
    for (uint32_t v : all)
        if (v % 16 != 0) return false;
    return l->pool_layer_base && aligned(l->pool_layer_base, 16) && l->expert_stride % 16 == 0 && l->effective_scale && aligned(l->effective_scale, 16) &&
           l->per_expert_scale && aligned(l->per_expert_scale, 2) && aligned(l->logit_bias, 4) &&
           one_token_size(ctx, l, stack);
}

static OneTokenArgs one_token_args(const tf_context* ctx, const tf_moe_layer* l, tf_workspace* ws) {
    auto planes = [](const tf_projection& p) {
        return OnePlanes{byte_ptr(p.weights, p.weights_off), reinterpret_cast<const uint16_t*>(byte_ptr(p.scales, p.scales_off)),
                         reinterpret_cast<const uint16_t*>(byte_ptr(p.biases, p.biases_off))};
    };
    OneTokenArgs a{};
    a.d = l->d; a.f = l->f; a.fs = l->fs; a.experts = l->num_experts; a.top_k = l->top_k;
    a.router = planes(l->router);
    a.eff = static_cast<const uint16_t*>(l->effective_scale);
    a.logit_bias = l->logit_bias;
    a.logits = ws->one_token_logits;
    a.shared[0] = planes(l->shared_gate); a.shared[1] = planes(l->shared_up); a.shared[2] = planes(l->shared_down);
    a.shared_act = ws->shared_act;
    a.pool = static_cast<const uint8_t*>(l->pool_layer_base);
    a.stride = l->expert_stride;
    a.off = l->offsets;
    a.per_expert_scale = static_cast<const uint16_t*>(l->per_expert_scale);
    a.indices = ws->indices; a.weights = ws->weights;
    a.routes = RouterGroupOut{static_cast<tf_pair*>(ws->routes.sorted_pairs), static_cast<uint32_t*>(ws->routes.per_expert_offsets),
                              static_cast<uint32_t*>(ws->routes.per_expert_counts), static_cast<tf_group*>(ws->routes.groups),
                              static_cast<uint32_t*>(ws->routes.chunk_group), static_cast<uint32_t*>(ws->routes.chunk_start),
                              static_cast<uint32_t*>(ws->routes.counters)};
    a.acts = ws->acts;
    a.shared_y = ws->shared_y;
    a.partials = static_cast<float*>(ws->partials);
    a.error = ctx->device_error;
    return a;
}

// All shared memory of an SM for these kernels: a block of the down launch fits beside one of the gate/up launch (138 + 90 KB), a carveout
// made for the latter alone would not leave it room.
template <typename Kernel>
static tf_status one_carveout(tf_context* ctx, Kernel kernel, DeviceSmemCache& done) {
    const int dev = ctx->device >= 0 && ctx->device < kMaxDevices ? ctx->device : -1;
    std::lock_guard<std::mutex> lock(done.mu);
    if (dev >= 0 && done.bytes[dev]) return TF_OK;
    TF_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (dev >= 0) done.bytes[dev] = 1;
    return TF_OK;
}
static uint32_t one_router_blocks(const OneTokenArgs& a) { return (a.experts + kOneRouterExperts - 1) / kOneRouterExperts; }
template <bool NORM, bool FOURS>
static tf_status launch_front_as(tf_context* ctx, cudaStream_t st, const OneTokenArgs& a, uint32_t shared_blocks) {
    auto kern = one_token_front_kernel<NORM, FOURS>;
    const uint32_t ng = a.d / kGroup, most = shared_blocks ? (a.fs / 8 + shared_blocks - 1) / shared_blocks : 1u;
    const size_t tiles = shared_blocks ? OneTiles{ng, most, most}.total() : 0, router = OneRouterSmem{ng}.total();
    size_t smem = tiles > router ? tiles : router;
    if (a.router_blocks && shared_blocks && smem < kOneFrontBytes) smem = kOneFrontBytes;
    static DeviceSmemCache configured, carved;
    if (tf_status s = ensure_dynamic_smem(ctx, kern, configured, smem)) return s;
    if (tf_status s = one_carveout(ctx, kern, carved)) return s;
    launch_pdl(kern, dim3(a.router_blocks + shared_blocks), dim3(kOneThreads), smem, st, a, most);
    return check_launch(ctx, "one_token_front");
}
// One block per SM, those of the router included.
static uint32_t one_shared_blocks(const tf_context* ctx, const OneTokenArgs& a) {
    const uint32_t tiles = a.fs / 8, sms = (uint32_t)ctx->sm_count, left = sms > a.router_blocks ? sms - a.router_blocks : 1u;
    return tiles < left ? tiles : left;
}
template <bool NORM>
static tf_status launch_front(tf_context* ctx, cudaStream_t st, const OneTokenArgs& a, uint32_t shared_blocks) {
    return a.d / kGroup % 4 == 0 ? launch_front_as<NORM, true>(ctx, st, a, shared_blocks) : launch_front_as<NORM, false>(ctx, st, a, shared_blocks);
}
template <bool FOURS>
static tf_status launch_gate_up_as(tf_context* ctx, cudaStream_t st, const OneTokenArgs& a) {
    auto kern = one_token_gate_up_kernel<FOURS>;
    // one SM is left to the block of the tables, which would otherwise start when another one ends
    const uint32_t sms = ctx->sm_count > 1 ? (uint32_t)ctx->sm_count - 1 : 1u;
    const uint32_t tiles = a.f / 8 * a.top_k, blocks = tiles < sms ? tiles : sms, most = (tiles + blocks - 1) / blocks, slots = most < kOneSlots ? most : kOneSlots;
    const size_t tables = router_group_smem_bytes(a.top_k, a.experts, false), need = OneTiles{a.d / kGroup, slots, most}.total();
    size_t smem = need > tables ? need : tables;
    if (smem < kOneAloneBytes) smem = kOneAloneBytes;
    static DeviceSmemCache configured, carved;
    if (tf_status s = ensure_dynamic_smem(ctx, kern, configured, smem)) return s;
    if (tf_status s = one_carveout(ctx, kern, carved)) return s;
    launch_pdl(kern, dim3(blocks + 1), dim3(kOneThreads + kWarp), smem, st, a, slots, most);
    return check_launch(ctx, "one_token_gate_up");
}
static tf_status launch_gate_up(tf_context* ctx, cudaStream_t st, const OneTokenArgs& a) {
    return a.d / kGroup % 4 == 0 ? launch_gate_up_as<true>(ctx, st, a) : launch_gate_up_as<false>(ctx, st, a);
}
template <bool SHARED, bool ROUTED>
static tf_status launch_down(tf_context* ctx, cudaStream_t st, const OneTokenArgs& a) {
    auto kern = one_token_down_kernel<SHARED, ROUTED>;
    const OneDownGrid grid = one_down_grid(ctx, a.d, a.f, a.fs, a.top_k);
    const OneDownSmem lay{SHARED ? a.fs / kGroup : 0u, a.f / kGroup, ROUTED ? a.top_k : 0u, grid.rows};
    static DeviceSmemCache configured, carved;
    if (tf_status s = ensure_dynamic_smem(ctx, kern, configured, lay.total())) return s;
    if (tf_status s = one_carveout(ctx, kern, carved)) return s;
    launch_pdl(kern, dim3(grid.blocks), dim3(kOneDownThreads), lay.total(), st, a, grid.rows);
    return check_launch(ctx, "one_token_down");
}

tf_status one_token_layer(tf_context* ctx, void* stream, const tf_moe_layer* layer, const void* norm_weight_bf16, void* hidden, float eps, tf_workspace* ws) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    OneTokenArgs a = one_token_args(ctx, layer, ws);
    a.router_blocks = one_router_blocks(a);
    a.x = static_cast<const uint16_t*>(hidden); a.norm_w = static_cast<const uint16_t*>(norm_weight_bf16); a.x_out = ws->x_norm; a.eps = eps;
    if (tf_status s = launch_front<true>(ctx, st, a, one_shared_blocks(ctx, a))) return s;
    a.x = ws->x_norm;
    if (tf_status s = launch_gate_up(ctx, st, a)) return s;
    a.hidden = static_cast<uint16_t*>(hidden);
    return launch_down<true, true>(ctx, st, a);
}

tf_status one_token_block(tf_context* ctx, void* stream, const tf_moe_layer* layer, const void* x, void* y, tf_workspace* ws) {
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    OneTokenArgs a = one_token_args(ctx, layer, ws);
    a.x = static_cast<const uint16_t*>(x);
    a.router_blocks = one_router_blocks(a);
    if (tf_status s = launch_front<false>(ctx, st, a, 0)) return s;
    a.router_blocks = 0; a.behind_router = 1;
    if (tf_status s = launch_front<false>(ctx, st, a, one_shared_blocks(ctx, a))) return s;
    if (tf_status s = launch_gate_up(ctx, st, a)) return s;
    if (tf_status s = launch_down<true, false>(ctx, st, a)) return s;
    if (tf_status s = launch_down<false, true>(ctx, st, a)) return s;
    return tf_moe_reduce_token_major(ctx, stream, ws->partials, 1, ws->weights, ws->shared_y, a.d, y, a.d, 1, a.top_k, a.d);
}

}  // namespace tf
