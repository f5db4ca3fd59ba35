// Grouped int4 GEMM on the 5th-generation tensor cores (tcgen05 / TMEM) for batches of eight tokens and more.
//
// Replaces mpp_prefill_affine_threadgroup_f16 (Metal/TensorCore/tensorops.metal:13-105; wrapper
// Kernels/TensorCore/MPPPrefillInt4QMM.swift:34-78), the reference's "dequantise a weight tile to half,
// then matrix-unit MMA with an fp32 accumulator" kernel, and the routed prefill kernels
// prefill_grouped_routed_moe_batched_phase1 / _down (Metal/Prefill/prefill.metal:598-670), which the
// reference runs as scalar per-thread dot products.
//
//   D[128 or 256 weight rows x N tokens] += W_tile[rows x 256] . X_tile[N x 256]^T     per stage of four 64-column groups
//
// Weights are the A operand and are fed to the MMA from TENSOR MEMORY; tokens are the B operand (N = the tile's token count
// rounded up, carried in the instruction descriptor) in shared memory, K-major with the 128-byte swizzle. Data path of the
// weights, which carry nearly all the bytes:
//   HBM --TMA tile load--> shared memory (packed, 128 bytes per row and stage)
//       --LDS.128--> registers --one HFMA2 per two codes--> w = half(q * s + b)     (tensorops.metal:60-75)
//       --tcgen05.st--> tensor memory --tcgen05.mma--> fp32 accumulators in tensor memory.
// The dequantised tile never touches shared memory: an fp16 copy of the weights is four times the packed
// bytes, and writing it to shared memory and reading it back for the MMA would cost more shared-memory
// bandwidth than the whole HBM stream.
// A gate/up tile holds 64 gate rows over 64 up rows, so that one accumulator of 128 lanes carries both, 704 rows are eleven
// whole tiles, and all forms of the kernel have one layout; the epilogue warps of the two halves exchange values.
// Roles of the 24 warps: warp 0 issues the copies of packed codes and of a tile's scale and bias planes (1-D bulk copies; kQmmWide:
// warp 3), warp 2 those of activations (one 3-D box of 16 to 128 rows x 256 columns per stage), warp 1 the MMAs (kQmmFew: in turn
// with warp 3), and commits stages back through mbarriers; warps 4-19 dequantise in two teams that take turns, a thread two
// groups of one row per stage (kQmmWide: in one, a thread one group);
// warps 20-23 read the accumulators with tcgen05.ld, apply GeGLU or nothing, and store through a staging tile as 16-byte words,
// masked to the group's real tokens. Accumulators are double-buffered, so that the epilogue overlaps the next tile's MMAs.
// A persistent grid walks (group, token tile, weight-row tile) work items derived on the device from the
// routing metadata. Every mbarrier wait is bounded; on expiry the kernel records a code, waits for its copies and leaves.
//
// Three forms (clock counters around the waits of each role; 128 experts of 704 x 2816, uniform routing):
// kQmmPair, many tokens: with one CTA per tile of 128 rows x 128 tokens a stage took 1700 clocks, 640 of them waits for activations
// (64 KB per stage and SM out of L2). A pair of CTAs (cta_group::2) shares them: each holds those of half the tokens. 1240 clocks
// at 104 tokens per tile (MMAs 830), most of the rest the instructions of the one warp that issues them. 4096 tokens: gate/up 281
// -> 240 us, down 161 -> 141; dense 4096 x 2112 x 2816: 44 us = 1.11 PFLOP/s. (Arrivals on the other CTA's barriers must not
// be releases at cluster scope: with those a stage took 2150 clocks.)
// kQmmFew: the one warp that issued the MMAs bounded the kernel (waits, 16 MMAs and commits: 1250 of 1250 clocks
// without any copy outstanding at 1170), so two warps take turns, each with an accumulator, and activations come by one copy per
// stage instead of four. 333 tokens, 21 per expert: 1010 clocks a stage, of which an SM's share of the HBM rate is 790 and the
// dequantisers' instructions about 550; gate/up 109 -> 74 us, down 70 -> 46.
// kQmmWide, dense launches of more than 64 tokens per tile whose tiles have few stages: there start and end count, which take a pair
// about 1 us longer, and tiles of 64 tokens would be twice as many. 2000 x 1024 x 512: 8.5 us in the better of the other two, 7.5
// here; 500 x 4096 x 512 8.5 and 7.7; 500 x 8192 x 256 9.1 and 8.2. (Activations by half stages: up to 7 % slower.)
//
// Column order. The cheapest nibble extraction yields the eight codes of a 32-bit word in the order
// (0,4,1,5,2,6,3,7). A dot product does not care about the order as long as both operands agree, so the
// routed path stores its activations (the gathered rows and the GeGLU output) in that order within every
// eight columns (PERMUTED_K) and skips the four byte-permutes per word; the dense entry points take
// caller-owned activations in natural order and pay them.
#include <cuda.h>

#include "async_copy.cuh"

namespace tf {

constexpr int kQmmRows = 128;          // M of a CTA's MMA: weight rows per tile (gate/up: 64 gate rows over 64 up rows)
constexpr int kQmmBoxMax = 64;         // activation rows that a CTA holds per tile: tokens of a tile (kQmmPair: half of them; kQmmWide: up to 128)
constexpr int kQmmStageK = 256;        // columns per stage: four quantisation groups
constexpr uint32_t kQmmRawBytes = kQmmRows * (kQmmStageK / 2);      // 16 KB of packed codes
constexpr uint32_t kQmmRowBytes = kQmmStageK * 2;                   // one activation row of a stage
constexpr int kQmmRawMax = 4, kQmmBMax = 12, kQmmScMax = 4;         // ring depths (the launch picks them to fit, see QmmPlan)
constexpr int kQmmASlots = 2;          // slots of a dequantised stage (128 TMEM columns), used in turn
constexpr int kQmmFirstDequantWarp = 4, kQmmDequantWarps = 16;
constexpr int kQmmFirstEpilogueWarp = 20, kQmmEpilogueWarps = 4;
constexpr int kQmmThreads = (kQmmFirstEpilogueWarp + kQmmEpilogueWarps) * 32;
constexpr int kQmmTmemCols = 512;      // columns 0..255: accumulators; 256..511: the teams' slots of dequantised weights
constexpr int kQmmAccCols = 256;
constexpr uint32_t kQmmStageBytes = 16384;    // output staging of the epilogue
constexpr uint32_t kQmmSpin = 1u << 22;
constexpr uint32_t kErrQmmTimeout = 0x7E000000u;
static_assert(TF_MAX_ROUTER_EXPERTS <= kQmmThreads, "one thread per group");
static_assert(kQmmFirstEpilogueWarp % 4 == 0 && kQmmFirstDequantWarp % 4 == 0, "warp w touches TMEM lanes 32 * (w % 4)");

// How a launch divides its shared memory (offsets from a 1024-byte aligned base); computed on the host from K.
struct QmmPlan {
    uint32_t raw_stages;    // packed-code stages of 16 KB
    uint32_t b_bytes;       // activation ring
    uint32_t sc_bufs;       // scale-plane buffers
    uint32_t plane_bytes;   // one scale or bias plane of a tile (128 / NMAT rows)
    uint32_t sc_bytes;      // one buffer: NMAT x (scale plane, bias plane)
    uint32_t off_b, off_sc, off_stage, off_table, off_bars, total;
};

struct QmmArgs {
    // planes of matrix m of expert e at S[m] + e * expert_stride bytes (dense: one expert)
    const uint16_t* S[2];
    const uint16_t* B[2];
    uint64_t expert_stride;
    // groups of the launch, filled by qmm_prepare_kernel: {first token tile, first row, tokens, expert | tokens per tile << 16},
    // and {groups, token tiles, largest N}
    EarlyTable<uint4> groups;
    EarlyTable<uint32_t> totals;
    // their source; routed: what the grouping kernels left on the device; dense (NULL): one group
    const tf_group* route_groups;
    const uint32_t* route_counters;
    uint32_t dense_tokens, dense_per_tile;
    uint32_t ctas;          // CTAs of a tile: 2 for pairs
    uint32_t step_tok, step_row;      // what the grid's number of tiles is in whole token tiles and weight-row tiles
    uint32_t after_gate_up; // down launch whose predecessor on the stream is the gate/up launch of the same call
    // problem
    uint32_t rows;          // weight rows (output features)
    uint32_t k;             // columns (input features)
    uint16_t* out;          // [tokens, out_stride] fp16
    uint32_t out_stride;
    uint32_t out_vec;       // rows of out start on 16-byte boundaries
    uint32_t round_gate_up; // shared expert: gate and up rounded to fp16 before the activation
    uint32_t* error;
    QmmPlan plan;
};

// ---- PTX wrappers ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void q_mbar_init(uint32_t addr, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count) : "memory");
}
__device__ __forceinline__ void q_mbar_arrive(uint32_t addr) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void q_mbar_expect_tx(uint32_t addr, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(addr), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool q_mbar_wait(uint32_t addr, uint32_t parity) {
    for (uint32_t i = 0; i < kQmmSpin; ++i) {
        uint32_t ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// One look at a barrier, without waiting.
__device__ __forceinline__ bool q_mbar_test(uint32_t addr, uint32_t parity) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
    return ok != 0;
}
// The same shared-memory address in the first CTA of the pair.
__device__ __forceinline__ uint32_t q_in_leader(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// Relaxed: what these arrivals publish is tensor memory, whose accesses the tcgen05 waits and fences order, not memory.
__device__ __forceinline__ void q_mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void q_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Into this CTA's shared memory, counted on a barrier of the pair's first CTA.
__device__ __forceinline__ void tma_load_3d_pair(uint32_t smem_dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(mbar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t mbar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(mbar) : "memory");
}
__device__ __forceinline__ void q_bulk_g2s(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_dst), "l"(gsrc), "r"(bytes), "r"(mbar) : "memory");
}
// One lane of a converged warp; the address arithmetic around the elected instruction stays warp-uniform, so the
// compiler keeps descriptors in uniform registers instead of moving them over for every instruction.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile("{\n\t.reg .pred px;\n\telect.sync _|px, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, px;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void q_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Arrives at mbar (PAIR: at this address in both CTAs) once the MMAs issued so far have completed.
template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(mbar), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor]; PAIR: 128 rows of A and D in each CTA, half of B's rows in each.
template <bool PAIR>
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 32 consecutive 32-bit columns of this thread's TMEM lane <- 32 registers (eight uint4)
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint4 (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w),
                   "r"(v[2].x), "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w),
                   "r"(v[4].x), "r"(v[4].y), "r"(v[4].z), "r"(v[4].w), "r"(v[5].x), "r"(v[5].y), "r"(v[5].z), "r"(v[5].w),
                   "r"(v[6].x), "r"(v[6].y), "r"(v[6].z), "r"(v[6].w), "r"(v[7].x), "r"(v[7].y), "r"(v[7].z), "r"(v[7].w) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint4 q_lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t q_lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}

// K-major operand tile with the 128-byte swizzle: rows of 128 bytes, 8-row atoms of 1024 bytes.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16, fp16 x fp16 -> fp32, both operands K-major, M = m, N = n (a multiple of 16, of 32 for M = 256).
__device__ __forceinline__ uint32_t qmm_idesc(uint32_t m, uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// Eight packed codes (one 32-bit word) -> eight fp16 weights w = half(q * s + b).
// A nibble inside the ten mantissa bits of a half is a subnormal: q * 2^-22 at bits 2..5, q * 2^-20 at bits 4..7,
// q * 2^-18 at bits 6..9, so one HFMA2 with s times the opposite power of two gives fma(q, s, b) rounded once
// (tensorops.metal:60-75 stores half(fma(q, s, b))); the scaled s is exact in fp16 (s is a bf16) while it is finite.
// The kernel is bound by the integer pipe, which takes half a warp per clock, so what counts is its instructions per
// word: permuted order (k0,k4,k1,k5,k2,k6,k3,k7) two shifts and four masks (|s| < 2^-6), natural order one shift, four
// byte permutes and four masks (|s| < 2^-5). Larger scales take the two-step form (1024 + q) - 1024.
template <bool NATURAL_K>
struct FastScale {
    __half2 lo, hi;      // permuted: s * 2^22, s * 2^18; natural: both s * 2^20
    static constexpr float kLimit = NATURAL_K ? 0.03125f : 0.015625f;
    __device__ __forceinline__ explicit FastScale(float s) {
        if (NATURAL_K) { lo = __float2half2_rn(s * 1048576.0f); hi = lo; }
        else { lo = __float2half2_rn(s * 4194304.0f); hi = __float2half2_rn(s * 262144.0f); }
    }
};
__device__ __forceinline__ uint32_t q_hfma2(uint32_t a, __half2 s, __half2 b) {
    const __half2 r = __hfma2(*reinterpret_cast<__half2*>(&a), s, b);
    return *reinterpret_cast<const uint32_t*>(&r);
}
template <bool NATURAL_K>
__device__ __forceinline__ uint4 dequant8_fast(uint32_t w, const FastScale<NATURAL_K>& s, __half2 b) {
    if (NATURAL_K) {
        const uint32_t x = w << 4;
        uint32_t t0, t1, t2, t3;                                        // low half: nibble of byte i in x, high half: in w
        asm("prmt.b32 %0, %1, %2, 0x7470;" : "=r"(t0) : "r"(x), "r"(w));
        asm("prmt.b32 %0, %1, %2, 0x7571;" : "=r"(t1) : "r"(x), "r"(w));
        asm("prmt.b32 %0, %1, %2, 0x7672;" : "=r"(t2) : "r"(x), "r"(w));
        asm("prmt.b32 %0, %1, %2, 0x7773;" : "=r"(t3) : "r"(x), "r"(w));
        return make_uint4(q_hfma2(t0 & 0x00F000F0u, s.lo, b), q_hfma2(t1 & 0x00F000F0u, s.lo, b),
                          q_hfma2(t2 & 0x00F000F0u, s.lo, b), q_hfma2(t3 & 0x00F000F0u, s.lo, b));
    }
    const uint32_t a = w << 2, c = w >> 6;
    return make_uint4(q_hfma2(a & 0x003C003Cu, s.lo, b), q_hfma2(a & 0x03C003C0u, s.hi, b),      // (k0, k4), (k1, k5)
                      q_hfma2(c & 0x003C003Cu, s.lo, b), q_hfma2(c & 0x03C003C0u, s.hi, b));     // (k2, k6), (k3, k7)
}
template <bool NATURAL_K>
__device__ __forceinline__ uint4 dequant8_wide(uint32_t w, __half2 s, __half2 b) {
    const __half2 k1024 = __half2half2(__ushort_as_half(0x6400));
    uint32_t t[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        t[i] = ((w >> (4 * i)) & 0x000F000Fu) | 0x64006400u;
        const __half2 q = __hsub2(*reinterpret_cast<__half2*>(&t[i]), k1024);
        o[i] = q_hfma2(*reinterpret_cast<const uint32_t*>(&q), s, b);
    }
    if (!NATURAL_K) return make_uint4(o[0], o[1], o[2], o[3]);
    uint4 r;
    asm("prmt.b32 %0, %1, %2, 0x5410;" : "=r"(r.x) : "r"(o[0]), "r"(o[1]));   // (k0, k1)
    asm("prmt.b32 %0, %1, %2, 0x5410;" : "=r"(r.y) : "r"(o[2]), "r"(o[3]));   // (k2, k3)
    asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(r.z) : "r"(o[0]), "r"(o[1]));   // (k4, k5)
    asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(r.w) : "r"(o[2]), "r"(o[3]));   // (k6, k7)
    return r;
}

// Position of column k within its eight-column block in the PERMUTED order.
__device__ __forceinline__ uint32_t permuted_col(uint32_t k) { return (k & ~7u) | ((k & 3u) << 1) | ((k >> 2) & 1u); }

// Tokens per tile of a group: as few tiles as 64 * ctas tokens each allow, of equal size (a multiple of 16 per CTA, the step
// of the MMA's N). 256 + 14 tokens are three tiles of 96, not 128 + 128 + 14: the weights are dequantised once per tile, and
// below about 80 tokens that takes longer than the tile's MMAs.
__host__ __device__ inline uint32_t qmm_tokens_per_tile(uint32_t count, uint32_t ctas) {
    const uint32_t most = ctas * kQmmBoxMax, step = ctas * 16u;
    const uint32_t tiles = (count + most - 1) / most;
    return ((count + tiles - 1) / tiles + step - 1) / step * step;
}

// The group table of a launch: one thread per group, the tile counts scanned over the block. (One thread that walked the
// groups took 29 us for 128 of them, on the critical path before every routed GEMM; this takes about 2.)
__global__ void __launch_bounds__(TF_MAX_ROUTER_EXPERTS)
qmm_prepare_kernel(uint4* __restrict__ groups, uint32_t* __restrict__ totals, const tf_group* route_groups,
                   const uint32_t* route_counters, uint32_t dense_tokens, uint32_t dense_per_tile, uint32_t ctas) {
    __shared__ uint32_t warp_tiles[TF_MAX_ROUTER_EXPERTS / kWarp], warp_top[TF_MAX_ROUTER_EXPERTS / kWarp];
    const uint32_t warp = threadIdx.x / kWarp, lane = threadIdx.x % kWarp;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t ngroups = route_groups ? min(route_counters[0], (uint32_t)TF_MAX_ROUTER_EXPERTS) : 1u;
    const uint32_t step = ctas * 16u;
    uint32_t row = 0, count = 0, expert = 0, per = step;
    if (threadIdx.x < ngroups) {
        if (route_groups) {
            const tf_group rg = route_groups[threadIdx.x];
            row = rg.pair_start; count = rg.pair_count; expert = rg.expert;
            per = qmm_tokens_per_tile(count > 0 ? count : 1u, ctas);
        } else {
            count = dense_tokens; per = dense_per_tile;
        }
    }
    const uint32_t tiles = (count + per - 1) / per;
    uint32_t incl = tiles;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    const uint32_t top = __reduce_max_sync(kFullMask, min((count + step - 1) / step * step, per));
    if (lane == kWarp - 1) { warp_tiles[warp] = incl; warp_top[warp] = top; }
    __syncthreads();
    uint32_t before = 0, all = 0, n_top = step;
#pragma unroll
    for (uint32_t w = 0; w < TF_MAX_ROUTER_EXPERTS / kWarp; ++w) {
        before += w < warp ? warp_tiles[w] : 0u;
        all += warp_tiles[w];
        n_top = max(n_top, warp_top[w]);
    }
    if (threadIdx.x < ngroups) groups[threadIdx.x] = make_uint4(before + incl - tiles, row, count, expert | (per << 16));
    if (threadIdx.x == 0) { totals[0] = ngroups; totals[1] = all; totals[2] = n_top; }
}

// A role's place in its CTA's (or pair's) sequence of tiles, which is tile first, first + step, ... Tiles only move forward: the
// group is found by stepping through the table in shared memory, 32 entries to a look, without a division.
struct QmmTile {
    uint32_t tglob, wt;         // token tile over all groups; weight-row tile (of a pair: the two CTAs' tiles 2 wt, 2 wt + 1)
    uint32_t dt, dw;            // their step
    uint32_t wrow_tiles;
    uint32_t gi = 0;            // group
    uint32_t row0 = 0;          // first activation / output row
    uint32_t ntok = 0;          // real tokens
    uint32_t expert = 0;
    __device__ __forceinline__ QmmTile(uint32_t first, uint32_t step_tok, uint32_t step_row, uint32_t tiles)
        : tglob(first / tiles), wt(first - tglob * tiles), dt(step_tok), dw(step_row), wrow_tiles(tiles) {}
    __device__ __forceinline__ void locate(const uint4* table, uint32_t ngroups, uint32_t lane) {
        for (uint32_t ahead = ngroups > 1 ? kWarp : 0; ahead == kWarp;) {      // group starts grow: the votes are a prefix of the lanes
            const uint32_t g = gi + 1 + lane;
            ahead = __popc(__ballot_sync(kFullMask, g < ngroups && table[g].x <= tglob));
            gi += ahead;
        }
        const uint4 g = table[gi];                                  // tile start, first row, tokens, expert | tokens per tile << 16
        const uint32_t per = g.w >> 16, done = (tglob - g.x) * per;
        expert = g.w & 0xFFFFu;
        row0 = g.y + done;
        ntok = g.z - done < per ? g.z - done : per;
    }
    __device__ __forceinline__ void next() {
        tglob += dt; wt += dw;
        if (wt >= wrow_tiles) { wt -= wrow_tiles; ++tglob; }
    }
};

// kQmmPair: two CTAs of a cluster (two SMs that share their tensor cores' operands, cta_group::2) take one tile of 2 x 128 weight
// rows x up to 128 tokens. Each dequantises its own 128 rows and holds half of the tokens' activations, the first one issues the
// MMAs. kQmmFew: a CTA takes 128 rows x up to 64 tokens, and two warps issue MMAs, one for each team of dequantisers. kQmmWide:
// a CTA takes 128 rows x up to 128 tokens, one warp issues.
// x_map0 ... x_map3: boxes of 16, 32, 48 and 64 activation rows; kQmmWide: of a full tile's and of the last tile's rows.
enum QmmForm { kQmmFew, kQmmWide, kQmmPair };
template <int NMAT, bool NATURAL_K, QmmForm FORM>
__global__ void __launch_bounds__(kQmmThreads, 1)
qmm_tcgen05_kernel(const __grid_constant__ CUtensorMap x_map0, const __grid_constant__ CUtensorMap x_map1,
                   const __grid_constant__ CUtensorMap x_map2, const __grid_constant__ CUtensorMap x_map3,
                   const __grid_constant__ CUtensorMap w_map0, const __grid_constant__ CUtensorMap w_map1, const QmmArgs args) {
    extern __shared__ uint8_t smem_raw[];
    constexpr bool PAIR = FORM == kQmmPair, kTwoIssuers = FORM == kQmmFew;
    constexpr uint32_t kMatRows = kQmmRows / NMAT;                     // rows of one matrix in a tile
    constexpr uint32_t kCtas = PAIR ? 2 : 1;                           // CTAs of a tile
    // One team of dequantisers, a group of a row per thread and stage, or two that take turns, two groups per thread: the latter
    // hide one another's waits, the former has a tile's first stage ready sooner, which is what counts for tiles of few stages.
    constexpr uint32_t kTeams = FORM == kQmmWide ? 1 : 2, kTeamWarps = kQmmDequantWarps / kTeams;
    constexpr uint32_t kStep = 16 * kCtas;                             // N of an MMA is a multiple of it
    constexpr uint32_t kAccTok = kTwoIssuers ? 64 : 128;               // columns of an accumulator
    const QmmPlan& plan = args.plan;
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;                      // swizzle atoms need 1024-byte alignment
    uint8_t* base_ptr = smem_raw + (base - raw);
    const uint32_t bars = base + plan.off_bars;
    // barrier map (8 bytes each); L: in a pair only the first CTA's are used
    auto bar_full_raw = [&](uint32_t s) { return bars + s * 8; };                            // 4: TMA tx
    auto bar_empty_raw = [&](uint32_t s) { return bars + (4 + s) * 8; };                     // 4: the team's warps
    auto bar_full_b = [&](uint32_t s) { return bars + (8 + s) * 8; };                        // 12 L: TMA tx
    auto bar_empty_b = [&](uint32_t s) { return bars + (20 + s) * 8; };                      // 12: tcgen05.commit
    auto bar_full_a = [&](uint32_t t) { return bars + (32 + t) * 8; };                       // 2 L: the team's warps, of both CTAs
    auto bar_empty_a = [&](uint32_t t) { return bars + (34 + t) * 8; };                      // 2: tcgen05.commit
    auto bar_full_sc = [&](uint32_t b) { return bars + (40 + b) * 8; };                      // 4: bulk-copy tx
    auto bar_empty_sc = [&](uint32_t b) { return bars + (44 + b) * 8; };                     // 4: dequant warps
    auto bar_acc_full = [&](uint32_t i, uint32_t b) { return bars + (48 + 2 * i + b) * 8; }; // 4: tcgen05.commit
    auto bar_acc_empty = [&](uint32_t b) { return bars + (52 + b) * 8; };                    // 2 L: epilogue warps, of both CTAs
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + plan.off_bars + 54 * 8);   // TMEM base
    uint4* table = reinterpret_cast<uint4*>(base_ptr + plan.off_table);
    uint32_t* totals = reinterpret_cast<uint32_t*>(base_ptr + plan.off_bars + 55 * 8);

    // The shuffle makes the warp index uniform for the compiler: the roles' branches and their operands then stay in uniform
    // registers, where the MMA and copy instructions want them (the MMA issuer's loop was 10 to 15 % slower without).
    const int warp = __shfl_sync(kFullMask, (int)(threadIdx.x / kWarp), 0), lane = threadIdx.x % kWarp;
    const uint32_t rank = PAIR ? blockIdx.x & 1 : 0;                   // CTA within the pair
    const uint32_t ng = args.k / kGroup;
    const uint32_t ksteps = (ng + 3) / 4;                              // stages per tile
    const uint32_t wrow_tiles = (args.rows + kCtas * kMatRows - 1) / (kCtas * kMatRows);

    constexpr bool kRoutedGateUp = NMAT == 2 && !NATURAL_K;
    if (!kRoutedGateUp) pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < (uint32_t)kQmmRawMax; ++s) { q_mbar_init(bar_full_raw(s), 1); q_mbar_init(bar_empty_raw(s), kTeamWarps); }
        for (uint32_t s = 0; s < (uint32_t)kQmmBMax; ++s) { q_mbar_init(bar_full_b(s), 1); q_mbar_init(bar_empty_b(s), 1); }
        for (uint32_t t = 0; t < (uint32_t)kQmmASlots; ++t) { q_mbar_init(bar_full_a(t), kCtas * kTeamWarps); q_mbar_init(bar_empty_a(t), 1); }
        for (uint32_t b = 0; b < (uint32_t)kQmmScMax; ++b) { q_mbar_init(bar_full_sc(b), 1); q_mbar_init(bar_empty_sc(b), kQmmDequantWarps); }
        for (uint32_t b = 0; b < 2; ++b) {
            for (uint32_t i = 0; i < 2; ++i) q_mbar_init(bar_acc_full(i, b), 1);
            q_mbar_init(bar_acc_empty(b), kCtas * kQmmEpilogueWarps);
        }
        if constexpr (PAIR) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        q_fence_async_smem();
    }
    if (warp == 1) {
        const uint32_t slot = smem_u32(const_cast<uint32_t*>(tmem_slot));
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"((uint32_t)kQmmTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"((uint32_t)kQmmTmemCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    // The routed down launch takes its tables and weights while the last gate/up tiles are still being computed elsewhere; only the
    // copies of its activations wait. The tables are complete (see EarlyTable): gate/up lets its dependent start after its own wait.
    const bool early = NMAT == 1 && args.after_gate_up;
    if (!early) pdl_wait();                                             // routes and activations come from the kernels before this one
    if (kRoutedGateUp) pdl_launch_dependents();
    // The whole table and the totals in one round trip, a thread per entry (rows past the groups are copied and never used).
    if (threadIdx.x < (args.route_groups ? (uint32_t)TF_MAX_ROUTER_EXPERTS : 1u)) table[threadIdx.x] = args.groups.at<NMAT == 1>(threadIdx.x);
    else if (threadIdx.x - TF_MAX_ROUTER_EXPERTS < 3u) totals[threadIdx.x - TF_MAX_ROUTER_EXPERTS] = args.totals.at<NMAT == 1>(threadIdx.x - TF_MAX_ROUTER_EXPERTS);
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) q_cluster_sync();                              // the other CTA's barriers are initialised, too
    tc_fence_after();
    const uint32_t ngroups = totals[0], total_tiles = totals[1] * wrow_tiles, n_top = totals[2];
    const uint32_t tmem_base = *tmem_slot;
    // Activation ring: slots of a whole stage of the launch's largest tile, as many as fit. With two MMA issuers an even number,
    // as for the packed codes, so that a slot always belongs to the same one and a wait never sees the phase of another use.
    // Where too few slots would fit beside four stages of packed codes, those make do with two.
    const uint32_t b_slot = n_top / kCtas * kQmmRowBytes;
    const uint32_t raw_stages = !PAIR && plan.b_bytes < (kTwoIssuers ? 4 : 3) * b_slot ? 2u : plan.raw_stages;
    const uint32_t off_b = raw_stages * kQmmRawBytes, b_bytes = plan.off_b + plan.b_bytes - off_b;
    const uint32_t b_fit = kTwoIssuers ? b_bytes / b_slot & ~1u : b_bytes / b_slot;
    const uint32_t b_stages = b_fit < (uint32_t)kQmmBMax ? b_fit : (uint32_t)kQmmBMax;
    const uint32_t a_ring = tmem_base + kQmmAccCols;
    const uint32_t first_tile = blockIdx.x / kCtas, tile_step = gridDim.x / kCtas;

    uint32_t fail = 0;
    QmmTile tl(first_tile, args.step_tok, args.step_row, wrow_tiles);

    // Scale and bias planes of tile tl; false when the wait for the buffer ran out.
    uint32_t pl_buf = 0, pl_use = 0;
    auto copy_planes = [&]() {
        const uint32_t first = (tl.wt * kCtas + rank) * kMatRows;
        if (pl_use > 0 && !q_mbar_wait(bar_empty_sc(pl_buf), (pl_use - 1) & 1)) return false;
        if (elect_one()) {
            const uint32_t left = first < args.rows ? args.rows - first : 0;      // a pair's second tile may be past the matrix
            const uint32_t bytes = (left < kMatRows ? left : kMatRows) * ng * 2;  // a multiple of 16: rows are a multiple of 8
            const size_t off = (size_t)tl.expert * args.expert_stride + (size_t)first * ng * 2;
            q_mbar_expect_tx(bar_full_sc(pl_buf), NMAT * 2 * bytes);
            if (bytes > 0) {
#pragma unroll
                for (int m = 0; m < NMAT; ++m) {
                    const uint32_t dst = base + plan.off_sc + pl_buf * plan.sc_bytes + m * 2 * plan.plane_bytes;
                    q_bulk_g2s(dst, reinterpret_cast<const uint8_t*>(args.S[m]) + off, bytes, bar_full_sc(pl_buf));
                    q_bulk_g2s(dst + plan.plane_bytes, reinterpret_cast<const uint8_t*>(args.B[m]) + off, bytes, bar_full_sc(pl_buf));
                }
            }
        }
        __syncwarp();
        if (++pl_buf == plan.sc_bufs) { pl_buf = 0; ++pl_use; }
        return true;
    };
    auto drain_planes = [&]() {
        for (uint32_t s = 0; s < plan.sc_bufs; ++s) q_mbar_wait(bar_full_sc(s), (s < pl_buf ? pl_use : pl_use + 1) & 1);
    };
    if (warp == 0) {
        // ===================== copy issuer: scale and bias planes of a tile, packed codes =====================
        uint32_t sr = 0, ur = 0;
        for (uint32_t tile = first_tile; tile < total_tiles && !fail; tile += tile_step, tl.next()) {
            tl.locate(table, ngroups, lane);
            const uint32_t first = (tl.wt * kCtas + rank) * kMatRows;
            // (the dequantisers of the tile that used this buffer last are as far as the ring of codes asks for below, or one tile
            // ahead of it where the planes have one buffer)
            if (FORM != kQmmWide && !copy_planes()) { fail = kErrQmmTimeout | 6; break; }
            for (uint32_t ks = 0; ks < ksteps; ++ks) {
                if (ur > 0 && !q_mbar_wait(bar_empty_raw(sr), (ur - 1) & 1)) { fail = kErrQmmTimeout | 1; break; }
                if (elect_one()) {
                    const uint32_t dst = base + sr * kQmmRawBytes;
                    q_mbar_expect_tx(bar_full_raw(sr), kQmmRawBytes);
                    tma_load_3d(dst, &w_map0, (int)(ks * (kQmmStageK / 2)), (int)first, (int)tl.expert, bar_full_raw(sr));
                    if (NMAT == 2)
                        tma_load_3d(dst + kQmmRawBytes / 2, &w_map1, (int)(ks * (kQmmStageK / 2)), (int)first, (int)tl.expert, bar_full_raw(sr));
                }
                __syncwarp();
                if (++sr == raw_stages) { sr = 0; ++ur; }
            }
        }
        if (fail) {          // the copies already issued land before the CTA's shared memory goes away (bounded)
            for (uint32_t s = 0; s < raw_stages; ++s) q_mbar_wait(bar_full_raw(s), (s < sr ? ur : ur + 1) & 1);
            if (FORM != kQmmWide) drain_planes();
        }
    } else if (FORM == kQmmWide && warp == 3) {
        // ===================== copy issuer: scale and bias planes, beside the codes =====================
        for (uint32_t tile = first_tile; tile < total_tiles && !fail; tile += tile_step, tl.next()) {
            tl.locate(table, ngroups, lane);
            if (!copy_planes()) fail = kErrQmmTimeout | 6;
        }
        if (fail) drain_planes();
    } else if (warp == 2) {
        // ===================== copy issuer: activations, one copy per stage =====================
        uint32_t sb = 0, ub = 0;
        if (early) pdl_wait();
        for (uint32_t tile = first_tile; tile < total_tiles && !fail; tile += tile_step, tl.next()) {
            tl.locate(table, ngroups, lane);
            const uint32_t box = (tl.ntok + kStep - 1) / kStep * 16;  // rows per CTA
            const CUtensorMap* map = FORM == kQmmWide ? (box == args.dense_per_tile ? &x_map0 : &x_map1)
                                                      : box == 64 ? &x_map3 : box == 48 ? &x_map2 : box == 32 ? &x_map1 : &x_map0;
            const int row = (int)(tl.row0 + rank * box);
            for (uint32_t ks = 0; ks < ksteps; ++ks) {
                if (ub > 0 && !q_mbar_wait(bar_empty_b(sb), (ub - 1) & 1)) { fail = kErrQmmTimeout | 7; break; }
                if (elect_one()) {                                    // groups past K arrive as zeros and are not multiplied
                    const uint32_t dst = base + off_b + sb * b_slot;
                    if (rank == 0) q_mbar_expect_tx(bar_full_b(sb), kCtas * box * kQmmRowBytes);
                    if constexpr (PAIR) tma_load_3d_pair(dst, map, 0, row, (int)(4 * ks), q_in_leader(bar_full_b(sb)));
                    else tma_load_3d(dst, map, 0, row, (int)(4 * ks), bar_full_b(sb));
                }
                __syncwarp();
                if (++sb == b_stages) { sb = 0; ++ub; }
            }
        }
        if (fail && rank == 0)       // counts the copies of both CTAs, which leave together
            for (uint32_t s = 0; s < b_stages; ++s) q_mbar_wait(bar_full_b(s), (s < sb ? ub : ub + 1) & 1);
    } else if (warp == 1 || warp == 3) {
        // ===================== MMA issuers =====================
        // One issuer: warp 1 of the (first) CTA issues every stage. Two: the warps take turns, each with an accumulator of its own
        // (the epilogue adds them).
        const uint32_t who = warp == 1 ? 0 : 1;
        const bool mine = kTwoIssuers || (rank == 0 && who == 0);
        uint32_t sb = 0, ub = 0, count = 0, buf = 0, uacc = 0;        // count: stages so far; stage c is the (c / 2)-th use of its team's slot
        const uint64_t b_desc0 = umma_smem_desc(base + off_b);
        bool ready = false;                                           // the next stage's operands were there at the last look
        for (uint32_t tile = first_tile; mine && tile < total_tiles && !fail; tile += tile_step, tl.next()) {
            tl.locate(table, ngroups, lane);
            const uint32_t n = (tl.ntok + kStep - 1) / kStep * kStep;
            const uint32_t idesc = qmm_idesc(kCtas * kQmmRows, n);
            const uint32_t b_block = (n / kCtas * 128) >> 4;         // 64 columns of a slot, in units of the descriptor
            // Only for a tile that this warp has a stage of: the parity tells phases apart only while the barrier is at most one
            // phase ahead of the wait, and a tile of one stage can be multiplied and emptied without the other issuer.
            const bool takes_part = !kTwoIssuers || ksteps > 1 || (count & 1) == who;
            if (takes_part && uacc > 0 && !q_mbar_wait(bar_acc_empty(buf), (uacc - 1) & 1)) { fail = kErrQmmTimeout | 2; break; }
            tc_fence_after();
            const uint32_t acc = tmem_base + (kTwoIssuers ? 2 * buf + who : buf) * kAccTok;
            uint32_t accumulate = 0;
            for (uint32_t ks = 0; ks < ksteps; ++ks) {
                if (!kTwoIssuers || (count & 1) == who) {
                    const uint32_t t = count & 1;
                    if (!ready && (!q_mbar_wait(bar_full_b(sb), ub & 1) || !q_mbar_wait(bar_full_a(t), (count >> 1) & 1))) {
                        fail = kErrQmmTimeout | 3;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = a_ring + t * 128;
                    const uint32_t groups = ng - 4 * ks;              // groups left; those past K are skipped
                    const uint64_t b_desc = b_desc0 + (uint64_t)((sb * b_slot) >> 4);
                    auto multiply = [&](uint32_t g) {                 // one group: 16 columns of K per MMA, 8 TMEM columns of A, 32 bytes of B
                        if (g > 0 && groups <= g) return;
#pragma unroll
                        for (uint32_t j = 0; j < 4; ++j)
                            tc_mma_f16_ts<PAIR>(acc, a + g * 32 + j * 8, b_desc + (uint64_t)(g * b_block + j * 2), idesc, g + j > 0 ? 1u : accumulate);
                    };
                    const bool leader = elect_one();
                    if (leader) {
#pragma unroll
                        for (uint32_t g = 0; g < 3; ++g) multiply(g);
                    }
                    if constexpr (!kTwoIssuers) {
                        // A look at the next stage while these MMAs run: a wait on a barrier that is ready takes about 100 clocks,
                        // in which the tensor cores would run dry. (With few tokens the next operands are never there this early.)
                        __syncwarp();
                        const uint32_t nsb = sb + 1 < b_stages ? sb + 1 : 0;
                        ready = __all_sync(kFullMask, q_mbar_test(bar_full_b(nsb), (nsb > sb ? ub : ub + 1) & 1) &&
                                                          q_mbar_test(bar_full_a(t ^ 1), ((count + 1) >> 1) & 1));
                    }
                    if (leader) {
                        multiply(3);
                        tc_commit<PAIR>(bar_empty_a(t));              // both slots are free once these MMAs have read them
                        tc_commit<PAIR>(bar_empty_b(sb));
                        if (ks + (kTwoIssuers ? 2 : 1) >= ksteps) tc_commit<PAIR>(bar_acc_full(who, buf));
                    }
                    __syncwarp();
                    accumulate = 1;
                }
                ++count;
                if (++sb == b_stages) { sb = 0; ++ub; }
            }
            if (++buf == 2) { buf = 0; ++uacc; }
        }
    } else if (warp < kQmmFirstEpilogueWarp) {
        // ===================== dequantisers =====================
        // Two teams of eight warps: each takes every other stage, a thread two quantisation groups of one weight row. While a team
        // waits for codes, for its slot or for its stores, the other one computes. One team: every stage, a group per thread.
        const uint32_t dw = warp - kQmmFirstDequantWarp;
        const uint32_t q = dw & 3, gc = (dw >> 2) % (4 / kTeams) * kTeams;       // TMEM lane quarter; first group within the stage
        const uint32_t team = dw / kTeamWarps;
        const uint32_t r = q * kWarp + lane;                     // row within the tile = TMEM lane
        // packed codes of the row: 128 bytes whose 16-byte chunks sit at chunk ^ (row % 8) (128-byte TMA swizzle)
        const uint32_t raw_off = base + r * 128 + (((2 * gc) ^ (r & 7u)) << 4);
        const uint32_t sc_off = base + plan.off_sc + (r / kMatRows) * 2 * plan.plane_bytes + (r % kMatRows) * ng * 2 + gc * 2;
        const uint32_t a_lane = a_ring + ((q * kWarp) << 16) + gc * 32;
        uint32_t sr = 0, ur = 0, sc = 0, uc = 0, count = 0;      // count: stages so far; stage c is the (c / 2)-th use of slot c % 2
        for (uint32_t tile = first_tile; tile < total_tiles && !fail; tile += tile_step) {
            if (!q_mbar_wait(bar_full_sc(sc), uc & 1)) { fail = kErrQmmTimeout | 8; break; }
            const uint32_t sc_base = sc_off + sc * plan.sc_bytes;
            for (uint32_t ks = 0; ks < ksteps; ++ks) {
                const uint32_t slot = count & 1, ua = count >> 1;
                if (kTeams == 1 || slot == team) {
                    const uint32_t left = ng - 4 * ks > gc ? ng - 4 * ks - gc : 0;         // groups past K are neither dequantised nor multiplied
                    float sf[kTeams], bf[kTeams];
                    bool fast[kTeams];
#pragma unroll
                    for (uint32_t h = 0; h < kTeams; ++h) {
                        sf[h] = left > h ? bf16_bits_to_float((uint16_t)q_lds16(sc_base + ks * 8 + h * 2)) : 0.0f;
                        bf[h] = left > h ? bf16_bits_to_float((uint16_t)q_lds16(sc_base + plan.plane_bytes + ks * 8 + h * 2)) : 0.0f;
                        fast[h] = __all_sync(kFullMask, fabsf(sf[h]) < FastScale<NATURAL_K>::kLimit);
                    }
                    if (!q_mbar_wait(bar_full_raw(sr), ur & 1)) { fail = kErrQmmTimeout | 4; break; }
                    const uint32_t src = raw_off + sr * kQmmRawBytes;
                    uint4 c[2 * kTeams];
#pragma unroll
                    for (uint32_t i = 0; i < 2 * kTeams; ++i) c[i] = q_lds128(src ^ (i << 4));
#pragma unroll
                    for (uint32_t h = 0; h < kTeams; ++h) {
                        const uint4 c0 = c[2 * h], c1 = c[2 * h + 1];
                        uint4 out[8];
                        if (fast[h]) {                            // one branch per warp and group, both arms straight-line
                            const FastScale<NATURAL_K> s2(sf[h]);
                            const __half2 b2 = __float2half2_rn(bf[h]);
                            out[0] = dequant8_fast<NATURAL_K>(c0.x, s2, b2); out[1] = dequant8_fast<NATURAL_K>(c0.y, s2, b2);
                            out[2] = dequant8_fast<NATURAL_K>(c0.z, s2, b2); out[3] = dequant8_fast<NATURAL_K>(c0.w, s2, b2);
                            out[4] = dequant8_fast<NATURAL_K>(c1.x, s2, b2); out[5] = dequant8_fast<NATURAL_K>(c1.y, s2, b2);
                            out[6] = dequant8_fast<NATURAL_K>(c1.z, s2, b2); out[7] = dequant8_fast<NATURAL_K>(c1.w, s2, b2);
                        } else {
                            const __half2 s2 = __float2half2_rn(sf[h]), b2 = __float2half2_rn(bf[h]);
                            out[0] = dequant8_wide<NATURAL_K>(c0.x, s2, b2); out[1] = dequant8_wide<NATURAL_K>(c0.y, s2, b2);
                            out[2] = dequant8_wide<NATURAL_K>(c0.z, s2, b2); out[3] = dequant8_wide<NATURAL_K>(c0.w, s2, b2);
                            out[4] = dequant8_wide<NATURAL_K>(c1.x, s2, b2); out[5] = dequant8_wide<NATURAL_K>(c1.y, s2, b2);
                            out[6] = dequant8_wide<NATURAL_K>(c1.z, s2, b2); out[7] = dequant8_wide<NATURAL_K>(c1.w, s2, b2);
                        }
                        if (h == 0) {
                            __syncwarp();
                            if (lane == 0) {                      // the codes are in registers
                                if constexpr (kTeams == 2) mbar_arrive_after(bar_empty_raw(sr), c[0].x | c[1].x | c[2].x | c[3].x);
                                else mbar_arrive_after(bar_empty_raw(sr), c[0].x | c[1].x);
                            }
                            if (ua > 0 && !q_mbar_wait(bar_empty_a(slot), (ua - 1) & 1)) { fail = kErrQmmTimeout | 5; break; }
                            tc_fence_after();
                        }
                        if (left > h) tc_st32(a_lane + slot * 128 + h * 32, out);
                    }
                    if (fail) break;
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (PAIR) q_mbar_arrive_cluster(q_in_leader(bar_full_a(slot)));
                        else q_mbar_arrive(bar_full_a(slot));
                    }
                }
                ++count;
                if (++sr == raw_stages) { sr = 0; ++ur; }
            }
            __syncwarp();
            if (lane == 0) q_mbar_arrive(bar_empty_sc(sc));       // done with this tile's scale planes
            if (++sc == plan.sc_bufs) { sc = 0; ++uc; }
        }
    } else {
        // ===================== epilogue: TMEM -> registers -> shared memory -> 16-byte stores =====================
        // A lane holds one weight row and a register one token, but the output is [token][row]: 32 tokens at a time go
        // through a staging tile, so that a token's rows leave as whole 16-byte words.
        const uint32_t q = warp & 3;                              // TMEM lane quarter this warp may read
        const uint32_t r = q * kWarp + lane;                      // row within the tile = TMEM lane
        const uint32_t et = threadIdx.x - kQmmFirstEpilogueWarp * kWarp;
        constexpr uint32_t kTokBytes = kMatRows * 2;              // staged bytes per token
        const uint32_t xch = base + plan.off_stage;               // gate/up: 32 tokens x 64 rows fp32
        const uint32_t stage0 = NMAT == 2 ? xch + 8192 : xch;     // two staging tiles of 32 tokens
        const uint32_t mrow = r % kMatRows;
        const uint32_t pos = (NMAT == 2 && !NATURAL_K) ? permuted_col(mrow) : mrow;      // the GeGLU output feeds the down GEMM
        uint32_t buf = 0, uacc = 0, flip = 0, turn = 0;
        for (uint32_t tile = first_tile; tile < total_tiles && !fail; tile += tile_step, tl.next()) {
            tl.locate(table, ngroups, lane);
            const uint32_t first = (tl.wt * kCtas + rank) * kMatRows;
            const uint32_t left = first < args.rows ? args.rows - first : 0, nrows = left < kMatRows ? left : kMatRows;
            const bool two = kTwoIssuers && ksteps > 1;                     // both issuers had stages of the tile
            const uint32_t one = kTwoIssuers ? turn : 0;                     // the issuer of its first stage
            if (!q_mbar_wait(bar_acc_full(one, buf), uacc & 1)) fail = kErrQmmTimeout | 9;
            if (two && !q_mbar_wait(bar_acc_full(one ^ 1, buf), uacc & 1)) fail = kErrQmmTimeout | 9;
            turn ^= ksteps & 1;
            // every warp of the role leaves together: the barriers below count all four
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                         : "=r"(flip) : "r"(fail) : "memory");
            if (flip) { if (!fail) fail = kErrQmmTimeout | 9; break; }
            tc_fence_after();
            const uint32_t acc = tmem_base + ((q * kWarp) << 16) + (kTwoIssuers ? 2 * buf + one : buf) * kAccTok;
            const uint32_t acc2 = tmem_base + ((q * kWarp) << 16) + (2 * buf + (one ^ 1)) * kAccTok;      // the other issuer's
            uint32_t which = 0;
            for (uint32_t c0 = 0; c0 < tl.ntok; c0 += 32, which ^= 1) {
                uint32_t va[16], vb[16];
                tc_ld16(acc + c0, va);
                tc_ld16(acc + c0 + 16, vb);                       // past the tile's tokens: stale columns of the buffer, never stored
                tc_wait_ld();
                if constexpr (kTwoIssuers) {
                    if (two) {
                        uint32_t v2[16];
                        tc_ld16(acc2 + c0, v2);
                        tc_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; ++j) va[j] = __float_as_uint(__uint_as_float(va[j]) + __uint_as_float(v2[j]));
                        tc_ld16(acc2 + c0 + 16, v2);
                        tc_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; ++j) vb[j] = __float_as_uint(__uint_as_float(vb[j]) + __uint_as_float(v2[j]));
                    }
                }
                if (c0 + 32 >= tl.ntok) {                         // the accumulators are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if constexpr (PAIR) q_mbar_arrive_cluster(q_in_leader(bar_acc_empty(buf)));
                        else q_mbar_arrive(bar_acc_empty(buf));
                    }
                }
                const uint32_t stage = stage0 + which * (32 * kTokBytes) + pos * 2;
                if constexpr (NMAT == 2) {
                    // lanes 0..63 hold gate rows, 64..127 up rows: each side hands half of the tokens to the other
                    const bool gate_side = q < 2;
                    const uint32_t xrow = xch + mrow * 4, give = xrow + (gate_side ? 16 * 256 : 0), take = xrow + (gate_side ? 0 : 16 * 256);
                    uint32_t own[16], other[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        own[j] = gate_side ? va[j] : vb[j];
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(give + j * 256), "r"(gate_side ? vb[j] : va[j]) : "memory");
                    }
                    asm volatile("barrier.sync 1, 128;" ::: "memory");
                    // all loads, then the arithmetic of all sixteen, then the stores: one value at a time is a chain of
                    // shared-memory and special-function latencies (340 clocks each), longer than a tile's MMAs
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(other[j]) : "r"(take + j * 256));
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float gt = __uint_as_float(gate_side ? own[j] : other[j]), up = __uint_as_float(gate_side ? other[j] : own[j]);
                        if (args.round_gate_up) {                 // Kernels/MoE/SharedExpertInt4.swift:62-93
                            gt = __half2float(__float2half_rn(gt));
                            up = __half2float(__float2half_rn(up));
                        }
                        own[j] = __half_as_ushort(__float2half_rn(gelu_tanh(gt) * up));        // prefill.metal:634-636
                    }
                    const uint32_t out_tok = stage + (gate_side ? 0 : 16) * kTokBytes;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        asm volatile("st.shared.b16 [%0], %1;" ::"r"(out_tok + j * kTokBytes), "h"((uint16_t)own[j]) : "memory");
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const uint16_t y0 = __half_as_ushort(__float2half_rn(__uint_as_float(va[j])));
                        const uint16_t y1 = __half_as_ushort(__float2half_rn(__uint_as_float(vb[j])));
                        asm volatile("st.shared.b16 [%0], %1;" ::"r"(stage + j * kTokBytes), "h"(y0) : "memory");
                        asm volatile("st.shared.b16 [%0], %1;" ::"r"(stage + (16 + j) * kTokBytes), "h"(y1) : "memory");
                    }
                }
                asm volatile("barrier.sync 1, 128;" ::: "memory");
                // (a staging tile is written again two chunks later, after a barrier that follows these reads)
                constexpr uint32_t kVecs = kTokBytes / 16;        // 16-byte words per token
                const uint32_t src = stage0 + which * (32 * kTokBytes);
                constexpr int kPer = 32 * kVecs / 128;
                uint4 d[kPer];
#pragma unroll
                for (int i = 0; i < kPer; ++i) {
                    const uint32_t v = et + i * 128;
                    d[i] = q_lds128(src + (v / kVecs) * kTokBytes + (v % kVecs) * 16);
                }
#pragma unroll
                for (int i = 0; i < kPer; ++i) {
                    const uint32_t v = et + i * 128, tok = v / kVecs, c = v % kVecs;
                    if (c0 + tok < tl.ntok && c * 8 < nrows) {
                        uint16_t* o = args.out + (size_t)(tl.row0 + c0 + tok) * args.out_stride + first + c * 8;
                        if (args.out_vec) {
                            *reinterpret_cast<uint4*>(o) = d[i];
                        } else {
                            const uint32_t w4[4] = {d[i].x, d[i].y, d[i].z, d[i].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) { o[2 * e] = (uint16_t)(w4[e] & 0xFFFFu); o[2 * e + 1] = (uint16_t)(w4[e] >> 16); }
                        }
                    }
                }
            }
            if (++buf == 2) { buf = 0; ++uacc; }
        }
    }
    if (fail && lane == 0) atomicCAS(args.error, 0u, fail);
    tc_fence_before();
    __syncthreads();
    if constexpr (PAIR) q_cluster_sync();      // the other CTA's MMAs, copies and arrivals no longer need this one
    if (warp == 1) {
        tc_fence_after();
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kQmmTmemCols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)kQmmTmemCols) : "memory");
    }
}

// ---- host side ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// fp16 matrix [rows, k] with a row stride, seen as [k / 64][rows][64]: one copy brings a stage, four blocks of 64 columns x
// box_rows rows, each block laid out as the MMA wants it (128-byte swizzle, rows of 128 bytes); zero fill outside.
static tf_status make_x_map(tf_context* ctx, CUtensorMap* map, const void* x, uint64_t rows, uint32_t k, uint32_t stride_elems,
                            uint32_t box_rows, const char* name) {
    EncodeTiledFn fn = encode_tiled_fn();
    TF_REQUIRE(ctx, fn != nullptr, TF_ERR_UNSUPPORTED, "%s: cuTensorMapEncodeTiled is not available in this driver", name);
    const cuuint64_t dims[3] = {64, rows, k / 64};
    const cuuint64_t strides[2] = {(cuuint64_t)stride_elems * 2, 128};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, kQmmStageK / 64};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(x), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TF_REQUIRE(ctx, r == CUDA_SUCCESS, TF_ERR_CUDA, "%s: cuTensorMapEncodeTiled(activations) failed (%d)", name, (int)r);
    return TF_OK;
}

// Packed int4 weights as bytes [experts, rows, k / 2]: box = 128 bytes x (128 / NMAT) rows x 1 expert, 128-byte swizzle
// (the 16-byte chunks of a row are permuted by row % 8, which makes the row-per-lane LDS.128 conflict
// free); rows past the matrix and bytes past the row read as zero.
static tf_status make_w_map(tf_context* ctx, CUtensorMap* map, const void* w, uint32_t rows, uint32_t k, uint64_t experts,
                            uint64_t expert_stride, uint32_t box_rows, const char* name) {
    EncodeTiledFn fn = encode_tiled_fn();
    TF_REQUIRE(ctx, fn != nullptr, TF_ERR_UNSUPPORTED, "%s: cuTensorMapEncodeTiled is not available in this driver", name);
    const cuuint64_t dims[3] = {k / 2, rows, experts};
    const cuuint64_t strides[2] = {(cuuint64_t)(k / 2), expert_stride};
    const cuuint32_t box[3] = {(cuuint32_t)(kQmmStageK / 2), (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(w), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TF_REQUIRE(ctx, r == CUDA_SUCCESS, TF_ERR_CUDA, "%s: cuTensorMapEncodeTiled(weights) failed (%d)", name, (int)r);
    return TF_OK;
}

// Divides the 227 KB of shared memory for K columns. Packed codes first (four stages keep 48 to 64 KB in flight, what an
// SM's share of the HBM rate needs at its latency), the activation ring takes what the scale planes leave: three slots of
// 64 rows at K = 2816. Long rows give up stages, then (from K = 7040 on) the second buffer of scale planes: the next tile's
// planes are then copied between two tiles, which costs less than halving the tokens per tile (2000 x 2112 x 8192: 104 us with
// one buffer, 152 with two and tiles of 64 tokens).
constexpr uint32_t kQmmMaxK = 9024;
static bool qmm_plan(uint32_t k, uint32_t nmat, QmmPlan* p) {
    if (k > kQmmMaxK) return false;
    const uint32_t budget = 227u * 1024u - 1024u;                  // less the alignment slack
    const uint32_t ng = k / kGroup;
    p->plane_bytes = ((kQmmRows / nmat) * ng * 2u + 15u) & ~15u;
    p->sc_bytes = nmat * 2 * p->plane_bytes;
    const uint32_t slot = kQmmBoxMax * kQmmRowBytes;                // 32 KB
    uint32_t fixed = 0;
    p->raw_stages = 0;
    for (p->sc_bufs = 4 * p->sc_bytes <= 48u * 1024u ? 4u : 2u;; p->sc_bufs = 1) {
        fixed = p->sc_bufs * p->sc_bytes + kQmmStageBytes + TF_MAX_ROUTER_EXPERTS * 16u + 1024u;
        for (uint32_t raw = kQmmRawMax; raw >= 2 && !p->raw_stages; raw -= 2)         // even: a slot belongs to one team of dequantisers
            if (fixed + raw * kQmmRawBytes + 2 * slot <= budget) p->raw_stages = raw;
        if (p->raw_stages) break;
        if (p->sc_bufs == 1) return false;
    }
    p->b_bytes = (budget - fixed - p->raw_stages * kQmmRawBytes) & ~2047u;
    p->off_b = p->raw_stages * kQmmRawBytes;
    p->off_sc = p->off_b + p->b_bytes;
    p->off_stage = p->off_sc + p->sc_bufs * p->sc_bytes;
    p->off_table = p->off_stage + kQmmStageBytes;
    p->off_bars = p->off_table + TF_MAX_ROUTER_EXPERTS * 16u;
    p->total = p->off_bars + 1024u + 1024u;
    return true;
}

// Form and tokens per tile of a dense launch: the least of rounds of the grid x (a tile's stages + what a tile takes besides) + what
// the call takes besides. Fitted to 1500 launches of 13 matrices (256 x 256 to 8192 x 768 and 4096 x 2816) x 65 to 4096 tokens in every
// form and tile size; what it picks takes 0.3 % longer than the best of them on average, 6 % at the most. us, kQmmFew, kQmmWide and
// kQmmPair at their best sizes: 333 x 2112 x 2816 11.8, 13.1, 13.4; 1000 x 4096 x 512 11.1, 9.8, 10.6; 700 x 2816 x 704 9.2, 8.8, 9.6;
// 1000 x 2112 x 2816 19.2, 16.0, 15.4; 4096 x 4096 x 2816 102, 81, 70.
struct QmmDense {
    QmmForm form;
    uint32_t per_tile;
};
static QmmDense qmm_dense_tiles(uint32_t tokens, uint32_t rows, uint32_t mat_rows, uint32_t stages, uint32_t sms, uint32_t most_wide) {
    struct Cost { uint32_t stage, token, tile, call; };               // in units of 50 ps; token: per token of the tile and stage
    constexpr Cost kCost[3] = {{7800, 65, 7400, 94800}, {6000, 98, 9800, 91200}, {9800, 44, 10400, 118600}};      // by form
    QmmDense best{kQmmFew, 16};
    uint64_t best_cost = ~0ull;
    for (const QmmForm form : {kQmmFew, kQmmWide, kQmmPair}) {
        const uint32_t ctas = form == kQmmPair ? 2 : 1, step = ctas * 16u;
        if (ctas > sms) continue;
        const uint32_t least = form == kQmmWide ? kQmmBoxMax + step : step;
        for (uint32_t per = form == kQmmWide ? most_wide : ctas * kQmmBoxMax; per >= least; per -= step) {
            const uint64_t tiles = (uint64_t)((rows + ctas * mat_rows - 1) / (ctas * mat_rows)) * ((tokens + per - 1) / per);
            const uint64_t rounds = (tiles + sms / ctas - 1) / (sms / ctas);
            const Cost& c = kCost[form];
            const uint64_t cost = rounds * ((uint64_t)stages * (c.stage + c.token * per) + c.tile) + c.call;
            if (cost < best_cost) { best_cost = cost; best = {form, per}; }
        }
    }
    return best;
}
// Tokens of a kQmmWide tile: two slots of the activation ring have to fit beside two stages of packed codes.
static uint32_t qmm_most_wide(const QmmPlan& p) {
    const uint32_t fit = (p.off_b + p.b_bytes - 2 * kQmmRawBytes) / (2 * kQmmRowBytes) & ~15u;
    return fit < 128u ? fit : 128u;
}

// Fills a's group table (a.plan and the groups' source are set). The context has three: one for dense launches, which may run
// on another stream at the same time, and one for each half of a routed pair, so that both can be filled before the first.
constexpr int kQmmGateUpTable = 0, kQmmDownTable = 1, kQmmDenseTable = 2;
static tf_status launch_qmm_prepare(tf_context* ctx, void* stream, QmmArgs& a, int table, const char* name) {
    TF_REQUIRE(ctx, ctx->qmm_groups != nullptr, TF_ERR_OUT_OF_MEMORY, "%s: context scratch missing", name);
    uint4* groups = static_cast<uint4*>(ctx->qmm_groups) + table * (TF_MAX_ROUTER_EXPERTS + 1);
    uint32_t* totals = reinterpret_cast<uint32_t*>(groups + TF_MAX_ROUTER_EXPERTS);
    a.groups = {groups};
    a.totals = {totals};
    launch_pdl(qmm_prepare_kernel, dim3(1), dim3(TF_MAX_ROUTER_EXPERTS), 0, static_cast<cudaStream_t>(stream), groups, totals,
               a.route_groups, a.route_counters, a.dense_tokens, a.dense_per_tile, a.ctas);
    return check_launch(ctx, "qmm_prepare");
}

// W[m]: base of matrix m's packed plane for expert 0 (dense: the matrix itself); a.S, a.B likewise. A routed launch's table
// has been filled by the caller.
template <int NMAT, bool NATURAL_K, QmmForm FORM>
static tf_status launch_qmm_kernel(tf_context* ctx, void* stream, QmmArgs& a, const void* x, uint64_t x_rows, uint32_t x_stride,
                            const uint8_t* const* W, uint64_t experts, uint64_t expert_stride, bool dense, const char* name) {
    TF_REQUIRE(ctx, a.k % kGroup == 0 && a.k >= (uint32_t)kGroup, TF_ERR_INVALID_ARGUMENT, "%s: K must be a positive multiple of 64", name);
    TF_REQUIRE(ctx, a.rows % 8 == 0 && a.rows > 0, TF_ERR_INVALID_ARGUMENT, "%s: the weight rows must be a positive multiple of 8", name);
    TF_REQUIRE(ctx, aligned(x, 16) && (x_stride * 2) % 16 == 0, TF_ERR_ALIGNMENT, "%s: activation rows must be 16-byte aligned", name);
    TF_REQUIRE(ctx, qmm_plan(a.k, NMAT, &a.plan), TF_ERR_UNSUPPORTED, "%s: K=%u needs more shared memory for the scale planes than there is", name, a.k);
    constexpr uint32_t kMatRows = kQmmRows / NMAT;
    // Activation boxes: see the kernel. A dense launch knows its tiles (full ones and a last one) and encodes only the boxes of
    // those: an encode is most of a microsecond of host time, and small products are bound by it.
    constexpr uint32_t kCtas = FORM == kQmmPair ? 2 : 1;
    uint32_t box[4] = {16, 32, 48, 64};           // 0: not wanted
    if (dense) {
        const uint32_t rest = a.dense_tokens % a.dense_per_tile;
        const uint32_t full_box = a.dense_tokens >= a.dense_per_tile ? a.dense_per_tile / kCtas : 0u;
        const uint32_t rest_box = (rest + 16 * kCtas - 1) / (16 * kCtas) * 16;
        if (FORM == kQmmWide) {
            box[0] = full_box ? full_box : rest_box == a.dense_per_tile ? rest_box : 0u;
            box[1] = rest_box == a.dense_per_tile ? 0u : rest_box;
            box[2] = box[3] = 0;
        } else {
            for (uint32_t& b : box) b = b == full_box || b == rest_box ? b : 0u;
        }
    }
    CUtensorMap xmap[4], wmap[2];
    int some = -1;
    for (int i = 0; i < 4; ++i) {
        if (box[i] == 0) continue;
        if (tf_status s = make_x_map(ctx, &xmap[i], x, x_rows, a.k, x_stride, box[i], name)) return s;
        some = i;
    }
    for (int i = 0; i < 4; ++i)
        if (box[i] == 0) xmap[i] = xmap[some];
    for (int m = 0; m < NMAT; ++m)
        if (tf_status s = make_w_map(ctx, &wmap[m], W[m], a.rows, a.k, experts, dense ? (uint64_t)a.rows * (a.k / 2) : expert_stride, kMatRows, name)) return s;
    if (NMAT == 1) wmap[1] = wmap[0];
    a.expert_stride = dense ? 0 : expert_stride;
    a.out_vec = aligned(a.out, 16) && a.out_stride % 8 == 0 ? 1u : 0u;
    a.error = ctx->device_error;
    if (dense)
        if (tf_status s = launch_qmm_prepare(ctx, stream, a, kQmmDenseTable, name)) return s;
    auto kern = qmm_tcgen05_kernel<NMAT, NATURAL_K, FORM>;
    static DeviceSmemCache configured;
    if (tf_status s = ensure_dynamic_smem(ctx, kern, configured, a.plan.total)) return s;
    uint32_t grid = (uint32_t)ctx->sm_count / kCtas;
    const uint32_t wrow_tiles = (a.rows + kCtas * kMatRows - 1) / (kCtas * kMatRows);
    if (dense) {
        const uint64_t tiles = (uint64_t)wrow_tiles * ((a.dense_tokens + a.dense_per_tile - 1) / a.dense_per_tile);
        if (tiles < grid) grid = (uint32_t)tiles;
    }
    a.step_tok = grid / wrow_tiles; a.step_row = grid % wrow_tiles;
    launch_pdl_cluster(kern, dim3(grid * kCtas), dim3(kQmmThreads), a.plan.total, static_cast<cudaStream_t>(stream), kCtas, xmap[0], xmap[1],
                       xmap[2], xmap[3], wmap[0], wmap[1], a);
    return check_launch(ctx, name);
}
template <int NMAT, bool NATURAL_K>
static tf_status launch_qmm(tf_context* ctx, void* stream, QmmArgs& a, const void* x, uint64_t x_rows, uint32_t x_stride,
                            const uint8_t* const* W, uint64_t experts, uint64_t expert_stride, bool dense, const char* name) {
    if constexpr (NATURAL_K) {             // the dense launches
        const QmmDense t = qmm_dense_tiles(a.dense_tokens, a.rows, kQmmRows / NMAT, (a.k + kQmmStageK - 1) / kQmmStageK, (uint32_t)ctx->sm_count,
                                           qmm_plan(a.k, NMAT, &a.plan) ? qmm_most_wide(a.plan) : 0u);
        a.ctas = t.form == kQmmPair ? 2 : 1; a.dense_per_tile = t.per_tile;
        if (t.form == kQmmWide)
            return launch_qmm_kernel<NMAT, NATURAL_K, kQmmWide>(ctx, stream, a, x, x_rows, x_stride, W, experts, expert_stride, dense, name);
    }
    return a.ctas == 2 ? launch_qmm_kernel<NMAT, NATURAL_K, kQmmPair>(ctx, stream, a, x, x_rows, x_stride, W, experts, expert_stride, dense, name)
                       : launch_qmm_kernel<NMAT, NATURAL_K, kQmmFew>(ctx, stream, a, x, x_rows, x_stride, W, experts, expert_stride, dense, name);
}

tf_status launch_qmm_generic(tf_context* ctx, void* stream, const uint8_t* W, const uint16_t* S, const uint16_t* B,
                             const uint16_t* X, uint16_t* Y, uint32_t m, uint32_t n, uint32_t k, const char* name);   // qmm_generic.cu

}  // namespace tf

extern "C" {

tf_status tf_grouped_moe_tensorcore(tf_context* ctx, void* stream, const void* x_sorted, uint32_t x_rows,
                                    const void* pool_layer_base, uint64_t expert_stride, uint32_t num_experts,
                                    const tf_expert_offsets* offsets, const tf_device_routes* routes,
                                    void* acts_scratch, void* out_rows, uint32_t d, uint32_t f) {
    const char* name = "tf_grouped_moe_tensorcore";
    TF_REQUIRE(ctx, ctx != nullptr, TF_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", name);
    TF_REQUIRE(ctx, x_sorted && pool_layer_base && offsets && routes && acts_scratch && out_rows, TF_ERR_INVALID_ARGUMENT, "%s: NULL argument", name);
    TF_REQUIRE(ctx, d % 64 == 0 && f % 64 == 0 && d > 0 && f > 0, TF_ERR_INVALID_ARGUMENT, "%s: D and F must be positive multiples of 64", name);
    TF_REQUIRE(ctx, num_experts > 0 && num_experts <= TF_MAX_ROUTER_EXPERTS, TF_ERR_INVALID_ARGUMENT, "%s: numExperts must be in 1...256", name);
    const uint32_t all[9] = {offsets->gate_w_off, offsets->gate_s_off, offsets->gate_b_off, offsets->up_w_off, offsets->up_s_off,
                             offsets->up_b_off, offsets->down_w_off, offsets->down_s_off, offsets->down_b_off};
    for (uint32_t v : all) TF_REQUIRE(ctx, v % 16 == 0, TF_ERR_ALIGNMENT, "%s: blob sub-tensor offset %u is not a multiple of 16 bytes", name, v);
    TF_REQUIRE(ctx, tf::aligned(pool_layer_base, 16) && expert_stride % 16 == 0, TF_ERR_ALIGNMENT, "%s: pool must be 16-byte aligned", name);
    if (x_rows == 0) return TF_OK;
    const uint8_t* pool = static_cast<const uint8_t*>(pool_layer_base);
    tf::QmmArgs a{};
    auto plane = [&](uint32_t off) { return reinterpret_cast<const uint16_t*>(pool + off); };
    a.S[0] = plane(offsets->gate_s_off); a.B[0] = plane(offsets->gate_b_off);
    a.S[1] = plane(offsets->up_s_off);   a.B[1] = plane(offsets->up_b_off);
    a.route_groups = routes->groups; a.route_counters = routes->counters;
    a.rows = f; a.k = d; a.out = static_cast<uint16_t*>(acts_scratch); a.out_stride = f; a.round_gate_up = 0;
    tf::QmmArgs b{};
    b.S[0] = plane(offsets->down_s_off); b.B[0] = plane(offsets->down_b_off);
    b.route_groups = routes->groups; b.route_counters = routes->counters;
    b.rows = d; b.k = f; b.out = static_cast<uint16_t*>(out_rows); b.out_stride = d;
    b.after_gate_up = 1;
    // Pairs of CTAs from 40 rows per expert on. Both GEMMs of a layer of 128 experts, one CTA / pairs: 333 tokens (21 rows) 126 / 150
    // us with uniform and 70 / 62 with Zipf routing, 700 (44 rows) 159 / 157 and 105 / 94, 1000 190 / 165, 4096 518 / 385.
    a.ctas = b.ctas = (uint64_t)x_rows >= 40ull * num_experts ? 2 : 1;
    // both tables first: between the two GEMMs the second one's would wait for the first to end
    TF_REQUIRE(ctx, tf::qmm_plan(d, 2, &a.plan) && tf::qmm_plan(f, 1, &b.plan), TF_ERR_UNSUPPORTED,
               "%s: D=%u or F=%u needs more shared memory for the scale planes than there is", name, d, f);
    if (tf_status s = tf::launch_qmm_prepare(ctx, stream, a, tf::kQmmGateUpTable, name)) return s;
    if (tf_status s = tf::launch_qmm_prepare(ctx, stream, b, tf::kQmmDownTable, name)) return s;
    const uint8_t* w_gu[2] = {pool + offsets->gate_w_off, pool + offsets->up_w_off};
    if (tf_status s = tf::launch_qmm<2, false>(ctx, stream, a, x_sorted, x_rows, d, w_gu, num_experts, expert_stride, false,
                                                "tf_grouped_moe_tensorcore(gate/up)")) return s;
    const uint8_t* w_dn[2] = {pool + offsets->down_w_off, pool + offsets->down_w_off};
    return tf::launch_qmm<1, false>(ctx, stream, b, acts_scratch, x_rows, f, w_dn, num_experts, expert_stride, false,
                                    "tf_grouped_moe_tensorcore(down)");
}

tf_status tf_int4_qmm_with_path(tf_context* ctx, void* stream, const void* weights, uint64_t weights_off, const void* scales,
                                uint64_t scales_off, const void* biases, uint64_t biases_off, const void* x, uint64_t x_off,
                                void* y, uint64_t y_off, uint32_t m, uint32_t n, uint32_t k, tf_qmm_path* path_out) {
    const char* name = "tf_int4_qmm";
    if (path_out) *path_out = TF_QMM_PATH_UNAVAILABLE;
    TF_REQUIRE(ctx, ctx != nullptr, TF_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", name);
    TF_REQUIRE(ctx, weights && scales && biases && x && y, TF_ERR_INVALID_ARGUMENT, "%s: NULL buffer", name);
    const uint8_t* wp = tf::byte_ptr(weights, weights_off);
    const uint8_t* sp = tf::byte_ptr(scales, scales_off);
    const uint8_t* bp = tf::byte_ptr(biases, biases_off);
    const uint8_t* xp = tf::byte_ptr(x, x_off);
    uint8_t* yp = tf::byte_ptr(y, y_off);
    // the reference's guard (MPPPrefillInt4QMM.swift:43-55): positive sizes, K % 64 == 0, even 16-bit plane offsets
    const bool supported = m > 0 && n > 0 && k > 0 && k % 64 == 0 && tf::aligned(sp, 2) && tf::aligned(bp, 2) &&
                           tf::aligned(xp, 2) && tf::aligned(yp, 2);
    if (!supported) {
        if (path_out) return TF_OK;         // the reference reports .unavailable and the caller falls back
        TF_REQUIRE(ctx, m == 0 || n == 0 || (k % 64 == 0 && k > 0), TF_ERR_INVALID_ARGUMENT, "%s: K must be a positive multiple of 64", name);
        if (m == 0 || n == 0) return TF_OK;
        return tf::fail(ctx, TF_ERR_ALIGNMENT, "%s: scale, bias, x and y offsets must be even", name);
    }
    const bool tensor = n % 8 == 0 && tf::aligned(wp, 16) && tf::aligned(sp, 16) && tf::aligned(bp, 16) && tf::aligned(xp, 16);
    if (!tensor) {
        // odd row counts or planes off the 16-byte grid: the CUDA-core kernel takes any byte offset
        tf_status s = tf::launch_qmm_generic(ctx, stream, wp, reinterpret_cast<const uint16_t*>(sp), reinterpret_cast<const uint16_t*>(bp),
                                             reinterpret_cast<const uint16_t*>(xp), reinterpret_cast<uint16_t*>(yp), m, n, k, name);
        if (!s && path_out) *path_out = TF_QMM_PATH_CUDA_CORES;
        return s;
    }
    tf::QmmArgs a{};
    const uint8_t* w[2] = {wp, wp};
    a.S[0] = reinterpret_cast<const uint16_t*>(sp);
    a.B[0] = reinterpret_cast<const uint16_t*>(bp);
    a.dense_tokens = m; a.rows = n; a.k = k;
    a.out = reinterpret_cast<uint16_t*>(yp); a.out_stride = n;
    tf_status s = tf::launch_qmm<1, true>(ctx, stream, a, xp, m, k, w, 1, 0, true, name);
    if (!s && path_out) *path_out = TF_QMM_PATH_TENSORCORE;
    return s;
}

tf_status tf_int4_qmm(tf_context* ctx, void* stream, const void* weights, uint64_t weights_off, const void* scales,
                      uint64_t scales_off, const void* biases, uint64_t biases_off, const void* x, uint64_t x_off,
                      void* y, uint64_t y_off, uint32_t m, uint32_t n, uint32_t k) {
    return tf_int4_qmm_with_path(ctx, stream, weights, weights_off, scales, scales_off, biases, biases_off, x, x_off, y, y_off,
                                 m, n, k, nullptr);
}

tf_status tf_shared_expert_int4_tensorcore(tf_context* ctx, void* stream, const void* x, uint32_t x_stride_elements,
                                           const tf_projection* gate, const tf_projection* up, const tf_projection* down,
                                           void* y, uint32_t y_stride_elements, void* scratch_act, uint32_t rows) {
    const char* name = "tf_shared_expert_int4_tensorcore";
    TF_REQUIRE(ctx, ctx != nullptr, TF_ERR_INVALID_ARGUMENT, "%s: ctx is NULL", name);
    TF_REQUIRE(ctx, x && gate && up && down && y && scratch_act, TF_ERR_INVALID_ARGUMENT, "%s: NULL argument", name);
    TF_REQUIRE(ctx, gate->rows == up->rows && gate->cols == up->cols && down->rows == gate->cols && down->cols == gate->rows,
               TF_ERR_DIMENSION_MISMATCH, "SharedExpert dimension mismatch: gate=(%u,%u) up=(%u,%u) down=(%u,%u)",
               gate->rows, gate->cols, up->rows, up->cols, down->rows, down->cols);
    if (rows == 0) return TF_OK;
    const uint32_t fs = gate->rows, d = gate->cols;
    const tf_projection* ps[3] = {gate, up, down};
    const uint8_t* W[3]; const uint16_t* S[3]; const uint16_t* B[3];
    for (int i = 0; i < 3; ++i) {
        W[i] = tf::byte_ptr(ps[i]->weights, ps[i]->weights_off);
        S[i] = reinterpret_cast<const uint16_t*>(tf::byte_ptr(ps[i]->scales, ps[i]->scales_off));
        B[i] = reinterpret_cast<const uint16_t*>(tf::byte_ptr(ps[i]->biases, ps[i]->biases_off));
        TF_REQUIRE(ctx, tf::aligned(W[i], 16) && tf::aligned(S[i], 16) && tf::aligned(B[i], 16), TF_ERR_ALIGNMENT, "%s: planes must be 16-byte aligned", name);
    }
    tf::QmmArgs a{};
    a.S[0] = S[0]; a.B[0] = B[0];
    a.S[1] = S[1]; a.B[1] = B[1];
    a.dense_tokens = rows; a.rows = fs; a.k = d; a.out = static_cast<uint16_t*>(scratch_act); a.out_stride = fs; a.round_gate_up = 1;
    const uint8_t* w_gu[2] = {W[0], W[1]};
    if (tf_status s = tf::launch_qmm<2, true>(ctx, stream, a, x, rows, x_stride_elements, w_gu, 1, 0, true,
                                               "tf_shared_expert_int4_tensorcore(gate/up)")) return s;
    tf::QmmArgs b{};
    b.S[0] = S[2]; b.B[0] = B[2];
    b.dense_tokens = rows; b.rows = d; b.k = fs; b.out = static_cast<uint16_t*>(y); b.out_stride = y_stride_elements;
    const uint8_t* w_dn[2] = {W[2], W[2]};
    return tf::launch_qmm<1, true>(ctx, stream, b, scratch_act, rows, fs, w_dn, 1, 0, true, "tf_shared_expert_int4_tensorcore(down)");
}

}  // extern "C"
