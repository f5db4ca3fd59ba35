// Streaming int4 GEMVs for large matrices: y[m] = deq4(W[m,n]) . x[n] at HBM speed.
// Second implementation of dequant_int4_gemv_simd (Metal/Quant/dequant_int4.metal:93-191) for the sizes where
// the warp-per-row kernel of gemv.cu is bound by its instruction count (about three CUDA-core instructions per
// weight: extract, convert, multiply-add), e.g. the LM-head-sized instance 262144 x 2816.
//
// Here a weight costs half an instruction. Each warp owns 16 rows and walks the columns in 64-column groups;
// per group it loads 8 bytes of packed codes per lane for rows g and g + 8 straight from global memory (every
// 32-byte sector fully used), masks them into fp16 subnormals (q * 2^-24, or q * 2^-20 against activations
// pre-scaled by 1/16: one AND per two codes) and feeds them as the A operand of mma.sync.m16n8k16. The vector x
// is column 0 of the B operand (the other seven columns are zero), pre-arranged once per block in shared
// memory in fragment order. Scale and bias are applied per group to the fp32 accumulator, acc += s * (q . x)
// + b * sum(x), the reference's algebra (dequant_int4.metal:132-170). Four groups are in flight as
// independent MMA chains, and the next four groups' codes are loaded before the current ones are consumed.
// That is gemv_mma_kernel: batches of small matrices, rows of few columns, smaller greedy heads. gemv_stream_kernel below does the
// same arithmetic on whole rows that bulk copies bring to shared memory; gs_teams says which one a product takes.
#include "async_copy.cuh"
#include "mma_gemv.cuh"

namespace tf {

constexpr int kGmWarps = 8;                 // 16 rows each: 128 rows per block (one large matrix)
constexpr int kGmBatchWarps = 4;            // 64 rows per block for batches of expert-sized matrices (704 = 11 x 64)
constexpr int kGmBlockGroups = 4;           // groups per inner step (independent MMA chains)

// Shared memory: B fragments of x [ng][4 lanes t][8 words], group sums [ng], scale and bias planes of the block's
// 128 rows [128][ng] each.
// A batch (blockIdx.y) walks matrices that share one layout: matrix b has its three planes `plane_stride` bytes
// after those of matrix b - 1 (e.g. the same tensor of consecutive expert blobs), its activations x_stride and its
// results y_stride elements further on (x_stride 0: one vector for all).
struct GemvBatch {
    uint64_t plane_stride;
    uint32_t x_stride, y_stride;
};

__device__ __forceinline__ unsigned long long argmax_key(float z, uint32_t row) {
    return isfinite(z) ? ((unsigned long long)ordered_key(z) << 32) | (unsigned long long)(~row) : 0ull;
}

// x in MMA operand order and its group sums, by the whole block: the 16 values x0..x15 at columns 64 G + 16 t feed four MMAs,
//   j = 0: (x0,x4),(x2,x6)   j = 1: (x1,x5)/16,(x3,x7)/16   j = 2, 3: the same for x8..x15
// (odd columns are pre-scaled by 1/16 because their codes sit four mantissa bits higher)
__device__ __forceinline__ void gm_stage_x(const uint16_t* x, uint32_t ng, uint32_t* xfrag, float* xsum, uint32_t threads) {
    for (uint32_t idx = threadIdx.x; idx < ((ng * 4 + 31u) & ~31u); idx += threads) {   // whole warps: the sums use shuffles
        const bool ok = idx < ng * 4;
        const uint32_t G = idx >> 2, tt = idx & 3;
        const uint4* p = reinterpret_cast<const uint4*>(x + G * kGroup + tt * 16);
        uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
        if (ok) { lo = p[0]; hi = p[1]; }
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
        if (tt == 0) xsum[G] = sum;
        uint32_t f[8];
        gm_make_frag(r, f);
        uint4* dst = reinterpret_cast<uint4*>(xfrag + idx * 8);
        dst[0] = make_uint4(f[0], f[1], f[2], f[3]);
        dst[1] = make_uint4(f[4], f[5], f[6], f[7]);
    }
}

// Row sums of four groups for rows g and g + 8 of a warp's 16: c[i][0] and c[i][2] of the lanes with t == 0. fr: the B fragments of
// the groups (x lives in column 0 only: lanes with g == 0).
__device__ __forceinline__ void gm_four_groups(const uint2 (&ca)[kGmBlockGroups], const uint2 (&cb)[kGmBlockGroups], const uint32_t* fr, int g,
                                               const float (&zc)[4], float (&c)[kGmBlockGroups][4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int i = 0; i < kGmBlockGroups; ++i) {
            uint2 bf = make_uint2(0u, 0u);
            if (g == 0) bf = *reinterpret_cast<const uint2*>(fr + i * 32 + j * 2);
            const uint32_t wx = (j < 2) ? ca[i].x : ca[i].y, wy = (j < 2) ? cb[i].x : cb[i].y;
            const uint32_t mask = (j & 1) ? 0x00F000F0u : 0x000F000Fu;
            const uint32_t a0 = wx & mask, a1 = wy & mask, a2 = (wx >> 8) & mask, a3 = (wy >> 8) & mask;
            if (j == 0) gm_mma(c[i], a0, a1, a2, a3, bf.x, bf.y, zc);
            else gm_mma(c[i], a0, a1, a2, a3, bf.x, bf.y, c[i]);
        }
    }
}
// acc += s * (q . x) + b * sum(x) for four groups; vs, vb: scale and bias of rows g (0) and g + 8 (1). The codes entered the MMA as
// q * 2^-24: 2^24 is folded into the scale.
template <bool SB_FP16>
__device__ __forceinline__ void gm_scale_four(const float (&c)[kGmBlockGroups][4], const uint2& vs0, const uint2& vs1, const uint2& vb0,
                                              const uint2& vb1, const float4& xs, float& acc0, float& acc1) {
    const float xsv[4] = {xs.x, xs.y, xs.z, xs.w};
#pragma unroll
    for (int i = 0; i < kGmBlockGroups; ++i) {
        const uint32_t sv0 = i < 2 ? vs0.x : vs0.y, sv1 = i < 2 ? vs1.x : vs1.y;
        const uint32_t bv0 = i < 2 ? vb0.x : vb0.y, bv1 = i < 2 ? vb1.x : vb1.y;
        const uint16_t s0b = (uint16_t)((i & 1) ? sv0 >> 16 : sv0 & 0xFFFFu), s1b = (uint16_t)((i & 1) ? sv1 >> 16 : sv1 & 0xFFFFu);
        const uint16_t b0b = (uint16_t)((i & 1) ? bv0 >> 16 : bv0 & 0xFFFFu), b1b = (uint16_t)((i & 1) ? bv1 >> 16 : bv1 & 0xFFFFu);
        const float s0 = sb_to_float<SB_FP16>(s0b) * 16777216.0f, s1 = sb_to_float<SB_FP16>(s1b) * 16777216.0f;
        const float b0 = sb_to_float<SB_FP16>(b0b), b1 = sb_to_float<SB_FP16>(b1b);
        acc0 = fmaf(s0, c[i][0], fmaf(b0, xsv[i], acc0));
        acc1 = fmaf(s1, c[i][2], fmaf(b1, xsv[i], acc1));
    }
}
// The largest key of a block -> *argmax. per_warp: one word per warp.
__device__ __forceinline__ void gm_fold_argmax(unsigned long long mine, unsigned long long* per_warp, unsigned long long* argmax) {
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
#pragma unroll
    for (int o = kWarp / 2; o >= 4; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(kFullMask, mine, o);
        mine = other > mine ? other : mine;
    }
    if (lane == 0) per_warp[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t w = 1; w < blockDim.x / kWarp; ++w) mine = per_warp[w] > mine ? per_warp[w] : mine;
        if (mine) atomicMax(argmax, mine);
    }
}

// What becomes of the row sums: stored as fp16, or (the greedy LM head) only the largest fp32 one is kept. ARGMAX: the launch
// follows the call's own norm kernel and nothing else, so weights are requested before that kernel has ended, and every block
// folds its rows into *argmax (ordered logit << 32 | ~row) without waiting for the result. Storing 262144 logits and a second
// kernel over them took 6 us; a count of finished blocks that lets the last one decode the token held every block up for a
// fence and an atomic's return, longer than a third launch of one thread.
template <bool SB_FP16, bool ARGMAX, int WARPS>
__global__ void __launch_bounds__(WARPS * kWarp)
gemv_mma_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                const uint16_t* x, uint16_t* __restrict__ y, uint32_t m, uint32_t n, const GemvBatch bt,
                unsigned long long* argmax) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int kGmRows = WARPS * 16, kGmThreads = WARPS * kWarp;
    {
        const size_t b = blockIdx.y;
        W += b * bt.plane_stride;
        S = reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(S) + b * bt.plane_stride);
        B = reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(B) + b * bt.plane_stride);
        x += b * bt.x_stride;
        y += b * bt.y_stride;
    }
    const uint32_t ng = n / kGroup;
    uint32_t* xfrag = reinterpret_cast<uint32_t*>(smem);                       // ng * 32 words
    float* xsum = reinterpret_cast<float*>(smem + (size_t)ng * 128);           // ng floats
    uint16_t* sS = reinterpret_cast<uint16_t*>(smem + (size_t)ng * 132);       // 128 * ng
    uint16_t* sB = sS + (size_t)kGmRows * ng;
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t row_base = blockIdx.x * kGmRows;

    pdl_launch_dependents();
    if constexpr (!ARGMAX) pdl_wait();
    // the first groups' codes are on their way while scales, biases and x are staged
    const uint32_t r0 = row_base + warp * 16 + g, r1 = r0 + 8;
    const uint32_t row_bytes = n / 2;
    // rows past the matrix read the last row (their results are not stored)
    const uint8_t* W0 = W + (size_t)(r0 < m ? r0 : m - 1) * row_bytes + t * 8;
    const uint8_t* W1 = W + (size_t)(r1 < m ? r1 : m - 1) * row_bytes + t * 8;
    uint2 wa[kGmBlockGroups], wb[kGmBlockGroups];
#pragma unroll
    for (int i = 0; i < kGmBlockGroups; ++i) { wa[i] = gm_ldg64(W0 + i * 32); wb[i] = gm_ldg64(W1 + i * 32); }
    // ---- scale and bias planes of the block's rows (contiguous in global memory) ----
    {
        const uint32_t rows_here = m - row_base < (uint32_t)kGmRows ? m - row_base : (uint32_t)kGmRows;
        const uint32_t words = rows_here * ng / 2;                             // rows * ng is even (ng % 4 == 0)
        const uint32_t* gs = reinterpret_cast<const uint32_t*>(S + (size_t)row_base * ng);
        const uint32_t* gb = reinterpret_cast<const uint32_t*>(B + (size_t)row_base * ng);
        uint32_t* ds = reinterpret_cast<uint32_t*>(sS);
        uint32_t* db = reinterpret_cast<uint32_t*>(sB);
        for (uint32_t i = threadIdx.x; i < words; i += kGmThreads) { ds[i] = __ldg(gs + i); db[i] = __ldg(gb + i); }
    }
    if constexpr (ARGMAX) pdl_wait();
    gm_stage_x(x, ng, xfrag, xsum, kGmThreads);
    __syncthreads();

    const uint16_t* s0p = sS + (size_t)(warp * 16 + g) * ng;
    const uint16_t* s1p = s0p + 8 * ng;
    const uint16_t* b0p = sB + (size_t)(warp * 16 + g) * ng;
    const uint16_t* b1p = b0p + 8 * ng;
    float zc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) asm volatile("mov.f32 %0, 0f00000000;" : "=f"(zc[j]));

    float acc0 = 0.0f, acc1 = 0.0f;
    for (uint32_t G0 = 0; G0 < ng; G0 += kGmBlockGroups) {
        uint2 ca[kGmBlockGroups], cb[kGmBlockGroups];
#pragma unroll
        for (int i = 0; i < kGmBlockGroups; ++i) { ca[i] = wa[i]; cb[i] = wb[i]; }
        if (G0 + kGmBlockGroups < ng) {
#pragma unroll
            for (int i = 0; i < kGmBlockGroups; ++i) {
                wa[i] = gm_ldg64(W0 + (G0 + kGmBlockGroups + i) * 32);
                wb[i] = gm_ldg64(W1 + (G0 + kGmBlockGroups + i) * 32);
            }
        }
        float c[kGmBlockGroups][4];
        gm_four_groups(ca, cb, xfrag + (G0 * 4 + t) * 8, g, zc, c);
        // scale and bias of the four groups for rows g and g + 8 (8-byte aligned: ng % 4 == 0)
        gm_scale_four<SB_FP16>(c, *reinterpret_cast<const uint2*>(s0p + G0), *reinterpret_cast<const uint2*>(s1p + G0),
                               *reinterpret_cast<const uint2*>(b0p + G0), *reinterpret_cast<const uint2*>(b1p + G0),
                               *reinterpret_cast<const float4*>(xsum + G0), acc0, acc1);
    }
    if constexpr (ARGMAX) {
        __shared__ unsigned long long per_warp[WARPS];
        unsigned long long mine = 0ull;                 // 0 = no finite candidate
        if (t == 0 && r0 < m) mine = argmax_key(acc0, r0);
        if (t == 0 && r1 < m) { const unsigned long long k = argmax_key(acc1, r1); mine = k > mine ? k : mine; }
        gm_fold_argmax(mine, per_warp, argmax);
    } else if (t == 0) {
        if (r0 < m) y[r0] = __half_as_ushort(__float2half_rn(acc0));
        if (r1 < m) y[r1] = __half_as_ushort(__float2half_rn(acc1));
    }
}

// The same product by a persistent block per SM: teams of four warps take tiles of 16 whole rows, a quarter of the columns per warp,
// each team through two slots of its own in shared memory that it refills itself with six bulk copies (four rows of codes per copy,
// the tile's scales, its biases): one slot is on its way while the other is multiplied. (One slot per team and twice the teams
// went through load and multiply in step, 4.6 TB/s.) gemv_mma_kernel's loads of eight bytes per lane touch eight lines per
// instruction and kept it at 0.75 of the HBM rate. 262144 x 2816, the whole greedy call: 92.2 -> 71.4 us (5.8 TB/s); 16384 x 4096
// out of L2: 26.6 -> 11.3.
// Four rows of codes are followed by 32 bytes of padding, and MMA row m is weight row 4 (m mod 4) + m / 4, so that the rows that a
// half warp reads together lie in different banks (row lengths are multiples of 128 bytes).
constexpr int kGsTeams = 4, kGsTeamWarps = 4;
__host__ __device__ inline uint32_t gs_stage_bytes(uint32_t n) { return 16 * (n / 2) + 4 * 32 + 2 * 16 * (n / kGroup) * 2; }
__host__ __device__ inline uint32_t gs_x_bytes(uint32_t n) { return (n / kGroup) * 132; }      // a multiple of 16: n % 256 == 0
constexpr uint32_t kErrGemvTimeout = 0x7B000001u;
template <bool SB_FP16, bool ARGMAX>
__global__ void __launch_bounds__(kGsTeams * kGsTeamWarps * kWarp, 1)
gemv_stream_kernel(const uint8_t* __restrict__ W, const uint16_t* __restrict__ S, const uint16_t* __restrict__ B,
                   const uint16_t* x, uint16_t* __restrict__ y, uint32_t m, uint32_t n, unsigned long long* argmax, uint32_t* error) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(8) unsigned long long bars[kGsTeams][2];
    __shared__ unsigned long long per_warp[kGsTeams * kGsTeamWarps];
    __shared__ float2 sums[kGsTeams][2][kGsTeamWarps - 1][8];  // row sums of a team's other warps, for tiles taken in turns
    const uint32_t teams = blockDim.x / (kGsTeamWarps * kWarp);
    const int warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp, team = warp / kGsTeamWarps, part = warp % kGsTeamWarps;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t ng = n / kGroup, row_bytes = n / 2, plane_bytes = 16 * ng * 2;
    uint32_t* xfrag = reinterpret_cast<uint32_t*>(smem);
    float* xsum = reinterpret_cast<float*>(smem + (size_t)ng * 128);
    const uint32_t stage_bytes = gs_stage_bytes(n);
    uint8_t* slots = smem + gs_x_bytes(n) + (size_t)team * 2 * stage_bytes;
    const uint32_t slots_addr = smem_addr_u32(slots), bar0 = smem_addr_u32(&bars[team][0]);
    const uint32_t tiles = (m + 15) / 16;
    const uint32_t step = gridDim.x * teams;
    uint32_t tile = blockIdx.x + gridDim.x * team;            // all blocks read one stretch of the matrix at a time
    // the last tile of a matrix whose rows are no multiple of 16 repeats rows of the one before
    auto first_row = [&](uint32_t tl) { const uint32_t r = tl * 16; return r + 16 <= m ? r : m - 16; };
    auto request = [&](uint32_t tl, uint32_t which) {
        const uint32_t row = first_row(tl), bar = bar0 + which * 8, slot = slots_addr + which * stage_bytes;
        if (lane == 0) {
            fence_proxy_async();                               // the slot was last read through the generic proxy
            mbar_arrive_expect_tx(bar, 16 * row_bytes + 2 * plane_bytes);
        }
        __syncwarp();
        if (lane < 4)
            bulk_copy_g2s(slot + lane * (4 * row_bytes + 32), W + (size_t)(row + 4 * lane) * row_bytes, 4 * row_bytes, bar);
        else if (lane < 6)
            bulk_copy_g2s(slot + 16 * row_bytes + 128 + (lane - 4) * plane_bytes, (lane == 4 ? S : B) + (size_t)row * ng, plane_bytes, bar);
    };
    pdl_launch_dependents();
    if (part == 0 && lane < 2) mbar_init(bar0 + lane * 8, 1);
    __syncwarp();
    if constexpr (!ARGMAX) pdl_wait();                         // (ARGMAX: see gemv_mma_kernel)
    if (part == 0) {
        if (tile < tiles) request(tile, 0);
        if (tile + step < tiles) request(tile + step, 1);
    }
    if constexpr (ARGMAX) pdl_wait();
    gm_stage_x(x, ng, xfrag, xsum, blockDim.x);
    __syncthreads();
    float zc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) asm volatile("mov.f32 %0, 0f00000000;" : "=f"(zc[j]));
    const uint32_t r_lo = 4 * (g & 3) + (g >> 2), r_hi = r_lo + 2;            // weight rows of the tile behind MMA rows g and g + 8
    const uint8_t* c_lo = slots + r_lo * row_bytes + (r_lo / 4) * 32 + t * 8;
    const uint8_t* c_hi = slots + r_hi * row_bytes + (r_hi / 4) * 32 + t * 8;
    const uint16_t* planes = reinterpret_cast<const uint16_t*>(slots + 16 * row_bytes + 128);
    const uint16_t *s_lo = planes + r_lo * ng, *s_hi = planes + r_hi * ng, *b_lo = s_lo + 16 * ng, *b_hi = s_hi + 16 * ng;
    unsigned long long best = 0ull;                            // 0 = no finite candidate
    uint32_t fail = 0;
    const uint32_t blocks = ng / kGmBlockGroups, g_begin = blocks * part / kGsTeamWarps * kGmBlockGroups,
                   g_end = blocks * (part + 1) / kGsTeamWarps * kGmBlockGroups;
    for (uint32_t use = 0; tile < tiles; tile += step, ++use) {
        const uint32_t which = use & 1, off = which * stage_bytes, off16 = off / 2;
        // (a warp whose wait has run out keeps its place at the team's barrier below, without waiting again)
        if (!fail && !mbar_wait(bar0 + which * 8, (use >> 1) & 1)) fail = kErrGemvTimeout;
        float acc0 = 0.0f, acc1 = 0.0f;
        for (uint32_t G0 = g_begin; G0 < g_end; G0 += kGmBlockGroups) {
            uint2 ca[kGmBlockGroups], cb[kGmBlockGroups];
#pragma unroll
            for (int i = 0; i < kGmBlockGroups; ++i) {
                ca[i] = *reinterpret_cast<const uint2*>(c_lo + off + (G0 + i) * 32);
                cb[i] = *reinterpret_cast<const uint2*>(c_hi + off + (G0 + i) * 32);
            }
            float c[kGmBlockGroups][4];
            gm_four_groups(ca, cb, xfrag + (G0 * 4 + t) * 8, g, zc, c);
            gm_scale_four<SB_FP16>(c, *reinterpret_cast<const uint2*>(s_lo + off16 + G0), *reinterpret_cast<const uint2*>(s_hi + off16 + G0),
                                   *reinterpret_cast<const uint2*>(b_lo + off16 + G0), *reinterpret_cast<const uint2*>(b_hi + off16 + G0),
                                   *reinterpret_cast<const float4*>(xsum + G0), acc0, acc1);
        }
        if (part && t == 0) sums[team][which][part - 1][g] = make_float2(acc0, acc1);
        asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kGsTeamWarps * kWarp) : "memory");      // the slot has been read, the sums are there
        if (part) continue;                                    // (it writes this half of sums again after the next tile's barrier)
        if (tile + 2 * step < tiles) request(tile + 2 * step, which);
#pragma unroll
        for (int p = 0; p < kGsTeamWarps - 1; ++p) { acc0 += sums[team][which][p][g].x; acc1 += sums[team][which][p][g].y; }
        const uint32_t row = first_row(tile);
        if (t == 0) {
            if constexpr (ARGMAX) {
                const unsigned long long k0 = argmax_key(acc0, row + r_lo), k1 = argmax_key(acc1, row + r_hi);
                best = k0 > best ? k0 : best;
                best = k1 > best ? k1 : best;
            } else {
                y[row + r_lo] = __half_as_ushort(__float2half_rn(acc0));
                y[row + r_hi] = __half_as_ushort(__float2half_rn(acc1));
            }
        }
    }
    if (fail) {              // the copies get one more bounded wait before the block leaves
        if (lane == 0) atomicCAS(error, 0u, fail);
        for (uint32_t par = 0; par < 4; ++par) mbar_wait(bar0 + (par & 1) * 8, par >> 1);
    }
    if constexpr (ARGMAX) gm_fold_argmax(best, per_warp, argmax);
}
// Teams of a block, 0 where the kernel does not apply: two slots of whole rows for at least two teams, planes of the last tile (which
// may repeat rows; callers have 4096 and more) on a 16-byte boundary, rows of 1024 columns and more (a team's slots hold too
// little otherwise; us, with gemv_mma_kernel and here: 65536 x 512 7.1 and 8.3, 65536 x 1024 12.2 and 11.3, 32768 x 1024 8.5 and 7.0,
// 8192 x 2816 11.8 and 5.7). The greedy LM head waits for its norm at the start, which a block of many small tiles hides
// better: from 1536 columns and 2^27 weights on (262144 rows of 1024 columns 38.2 and 41.6, of 1280 45.8 and 46.7, of 1536 52.0
// and 47.4; 2816 columns, 32000 rows out of L2 18.2 and 20.6, 65536 rows 30.5 and 26.8, 131072 rows 48.4 and 41.3), for rows of more
// than 4096 columns, whose few large slots start and end slowly, from 2^28 (5120 columns, 32000 rows 34.6 and 37.4, 48000 rows
// 45.6 and 51.6, 65536 rows 59.5 and 58.9, 262144 rows 178.7 and 158.9).
constexpr uint32_t kGsMinColumns = 1024, kGsMinArgmaxColumns = 1536, kGsLongColumns = 4096;
constexpr uint64_t kGsMinArgmaxWeights = 1ull << 27, kGsMinArgmaxWeightsLong = 1ull << 28;
static uint32_t gs_teams(uint32_t m, uint32_t n, bool greedy) {
    if (n < (greedy ? kGsMinArgmaxColumns : kGsMinColumns)) return 0;
    if (greedy && (uint64_t)m * n < (n > kGsLongColumns ? kGsMinArgmaxWeightsLong : kGsMinArgmaxWeights)) return 0;
    if (m % 16 != 0 && ((uint64_t)m * (n / kGroup)) % 8 != 0) return 0;
    const uint32_t x_bytes = gs_x_bytes(n), two = 2 * gs_stage_bytes(n), budget = 220u * 1024u;
    const uint32_t fit = x_bytes < budget ? (budget - x_bytes) / two : 0u, teams = fit < (uint32_t)kGsTeams ? fit : (uint32_t)kGsTeams;
    return teams >= 2 ? teams : 0;
}
template <bool SB_FP16, bool ARGMAX>
static tf_status launch_gemv_stream(tf_context* ctx, void* stream, uint32_t teams, const uint8_t* W, const uint16_t* S, const uint16_t* B,
                                    const uint16_t* x, uint16_t* y, uint32_t m, uint32_t n, unsigned long long* argmax, const char* name) {
    const size_t smem = gs_x_bytes(n) + (size_t)teams * 2 * gs_stage_bytes(n);
    auto k = gemv_stream_kernel<SB_FP16, ARGMAX>;
    static DeviceSmemCache configured;
    if (tf_status st = ensure_dynamic_smem(ctx, k, configured, smem)) return st;
    const uint32_t tiles = (m + 15) / 16, grid = tiles < (uint32_t)ctx->sm_count ? tiles : (uint32_t)ctx->sm_count;
    launch_pdl(k, dim3(grid), dim3(teams * kGsTeamWarps * kWarp), smem, static_cast<cudaStream_t>(stream), W, S, B, x, y, m, n, argmax, ctx->device_error);
    return check_launch(ctx, name);
}

static size_t gemv_mma_smem_bytes_for(uint32_t n, int warps) {
    const size_t ng = n / kGroup;
    return ng * 132 + (size_t)2 * warps * 16 * ng * 2;
}
size_t gemv_mma_smem_bytes(uint32_t n) { return gemv_mma_smem_bytes_for(n, kGmWarps); }

// Eligible: large, 16-byte aligned planes, a multiple of 256 columns (scale rows are read four groups at a time).
bool gemv_mma_eligible(const void* W, const void* S, const void* B, const void* x, uint32_t m, uint32_t n) {
    return m >= 4096 && n % 256 == 0 && aligned(W, 16) && aligned(S, 16) && aligned(B, 16) && aligned(x, 16) &&
           gemv_mma_smem_bytes(n) <= 100 * 1024;
}

tf_status launch_gemv_mma(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B,
                          const uint16_t* x, uint16_t* y, uint32_t m, uint32_t n, bool sb_fp16, const char* name) {
    if (const uint32_t teams = gs_teams(m, n, false))
        return sb_fp16 ? launch_gemv_stream<true, false>(ctx, stream, teams, W, S, B, x, y, m, n, nullptr, name)
                       : launch_gemv_stream<false, false>(ctx, stream, teams, W, S, B, x, y, m, n, nullptr, name);
    const size_t smem = gemv_mma_smem_bytes(n);
    auto k = sb_fp16 ? gemv_mma_kernel<true, false, kGmWarps> : gemv_mma_kernel<false, false, kGmWarps>;
    static DeviceSmemCache configured[2];
    if (tf_status st = ensure_dynamic_smem(ctx, k, configured[sb_fp16 ? 1 : 0], smem)) return st;
    launch_pdl(k, dim3((m + kGmWarps * 16 - 1) / (kGmWarps * 16)), dim3(kGmWarps * kWarp), smem, static_cast<cudaStream_t>(stream), W, S, B, x, y,
               m, n, GemvBatch{0, 0, 0}, nullptr);
    return check_launch(ctx, name);
}

// The greedy LM head's product: *argmax is zero before. Must follow, on the stream, the
// launch that writes x, and that launch must start after everything before it (no programmatic launch of its own).
// Short of gs_teams' line blocks of 128 rows, as for the stored form (64 rows took as long when both were measured).
tf_status launch_gemv_mma_argmax(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B,
                                 const uint16_t* x, uint32_t m, uint32_t n, unsigned long long* argmax, const char* name) {
    if (const uint32_t teams = gs_teams(m, n, true))
        return launch_gemv_stream<false, true>(ctx, stream, teams, W, S, B, x, nullptr, m, n, argmax, name);
    const size_t smem = gemv_mma_smem_bytes(n);
    auto k = gemv_mma_kernel<false, true, kGmWarps>;
    static DeviceSmemCache configured;
    if (tf_status st = ensure_dynamic_smem(ctx, k, configured, smem)) return st;
    launch_pdl(k, dim3((m + kGmWarps * 16 - 1) / (kGmWarps * 16)), dim3(kGmWarps * kWarp), smem, static_cast<cudaStream_t>(stream),
               W, S, B, x, nullptr, m, n, GemvBatch{0, 0, 0}, argmax);
    return check_launch(ctx, name);
}

// `count` GEMVs over matrices of one shape whose planes repeat every plane_stride bytes, in one launch.
tf_status launch_gemv_mma_batched(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B,
                                  uint64_t plane_stride, const uint16_t* x, uint32_t x_stride, uint16_t* y, uint32_t y_stride,
                                  uint32_t m, uint32_t n, uint32_t count, bool sb_fp16, const char* name) {
    const size_t smem = gemv_mma_smem_bytes_for(n, kGmBatchWarps);
    auto k = sb_fp16 ? gemv_mma_kernel<true, false, kGmBatchWarps> : gemv_mma_kernel<false, false, kGmBatchWarps>;
    static DeviceSmemCache configured[2];
    if (tf_status st = ensure_dynamic_smem(ctx, k, configured[sb_fp16 ? 1 : 0], smem)) return st;
    const uint32_t rows_per_block = kGmBatchWarps * 16;
    for (uint32_t first = 0; first < count; first += 65535u) {        // gridDim.y limit
        const uint32_t nb = count - first < 65535u ? count - first : 65535u;
        dim3 grid((m + rows_per_block - 1) / rows_per_block, nb);
        launch_pdl(k, grid, dim3(kGmBatchWarps * kWarp), smem, static_cast<cudaStream_t>(stream),
            W + (size_t)first * plane_stride,
            reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(S) + (size_t)first * plane_stride),
            reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(B) + (size_t)first * plane_stride),
            x + (size_t)first * x_stride, y + (size_t)first * y_stride, m, n, GemvBatch{plane_stride, x_stride, y_stride}, nullptr);
        if (tf_status st = check_launch(ctx, name)) return st;
    }
    return TF_OK;
}

}  // namespace tf
