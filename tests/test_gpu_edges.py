"""Edges of the tiles and of the dispatch rules of the kernels behind the block: token tiles of the tensor-core GEMM, the
few-row router, chunks of 16 tokens against chunks of 8, and the 16-row tiles of the one-token kernels."""
import numpy as np
import pytest

from tests.helpers import blob_table, config0_matrix, dev_zeros_u16, from_dev, to_dev
from turbo_fieldfare_b200._capi import ExpertOffsets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tf_ctx():
    """A context of this module's own: at its defaults whatever thresholds other modules have set on theirs."""
    from turbo_fieldfare_b200.kernels import TurboContext
    ctx = TurboContext(0)
    yield ctx
    ctx.close()


def _dense(o, mat):
    """The matrix in 64 bits."""
    q = np.empty((mat.packed.shape[0], mat.packed.shape[1] * 2), np.float64)
    q[:, 0::2], q[:, 1::2] = mat.packed & 15, mat.packed >> 4
    s, b = (np.repeat(o.bf16_to_f32(p).astype(np.float64), 64, axis=1) for p in (mat.scales, mat.biases))
    return q * s + b


# K: one group, an odd last group, whole and partial stages of four groups, the longest rows (whose scale planes leave room for one
# buffer: from 7040 on, with one and with two tiles per block); N: below, at and beyond a 128-row tile; M: tiles of one MMA
# step, of unequal last steps, exactly full, and several of equal size. y_off = 2 takes the element stores.
@pytest.mark.parametrize("M,N,K,y_off", [(1, 8, 64, 0), (15, 72, 128, 0), (16, 128, 192, 2), (17, 136, 320, 0), (63, 256, 704, 0), (65, 128, 2112, 2),
                                         (113, 264, 448, 0), (128, 2112, 256, 0), (129, 128, 2816, 0), (270, 384, 704, 0), (1000, 40, 4096, 0),
                                         (300, 64, 8192, 0), (128, 128, 6976, 0), (129, 136, 7040, 0), (1200, 2112, 7104, 0), (600, 5000, 8256, 0),
                                         (33, 72, 9024, 0)])
def test_qmm_token_tiles(tf_ctx, oracle, M, N, K, y_off):
    import torch
    from turbo_fieldfare_b200.kernels import MPPPrefillInt4QMM
    o = oracle
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    mat = config0_matrix(o, N, K, rng)
    x16 = o.f32_to_f16(rng.standard_normal((M, K)).astype(np.float32))
    y = dev_zeros_u16(M * N + 16, fill=0x7E00)
    MPPPrefillInt4QMM(tf_ctx).encode(to_dev(mat.packed), to_dev(mat.scales), to_dev(mat.biases), to_dev(x16), y, M, N, K, y_offset=y_off)
    torch.cuda.synchronize()
    assert tf_ctx.device_status() == 0
    out = from_dev(y, np.uint16)
    got = o.f16_to_f32(out[y_off // 2:y_off // 2 + M * N]).reshape(M, N)
    assert np.all(out[:y_off // 2] == 0x7E00) and np.all(out[y_off // 2 + M * N:] == 0x7E00)      # nothing beyond the result
    # weights and results rounded to fp16: 2^-11 each, a third of it in the root mean square
    assert o.rel_l2(got, o.f16_to_f32(x16).astype(np.float64) @ _dense(oracle, mat).T) < 1e-3


@pytest.mark.parametrize("rows", [65, 200, 255, 256, 297, 593, 1184, 1185])
def test_few_row_router_equals_the_one_launch_kernel(oracle, rows):
    """Indices and weights of the small-tile pass with eight, four, two or one warp per token in the re-check: byte for byte
    those of the kernel that computes every canonical logit."""
    import torch
    from turbo_fieldfare_b200.kernels import PrefillRouter, TurboContext
    o = oracle
    E, D, K = 128, 2816, 8
    rng = np.random.default_rng(rows)
    mat = config0_matrix(o, E, D, rng, bits=8)
    mat.packed[7], mat.scales[7], mat.biases[7] = mat.packed[3], mat.scales[3], mat.biases[3]       # exact ties
    W, S, B = to_dev(mat.packed), to_dev(mat.scales), to_dev(mat.biases)
    x = rng.standard_normal((rows, D)).astype(np.float32)
    x[1, 5] = np.nan
    x[2] *= 1e-4
    hid = to_dev(o.f32_to_f16(x))
    eff, gain = to_dev(o.f32_to_bf16(np.full(D, D ** -0.5, np.float32))), to_dev(o.f32_to_bf16(np.ones(E, np.float32)))

    ctx = TurboContext(0)               # whose threshold the test sets

    def run(min_rows):
        ctx.set_router_tensorcore_min_rows(min_rows)
        idx, w = torch.full((rows, K), -1, dtype=torch.int32, device="cuda"), dev_zeros_u16(rows * K)
        PrefillRouter(ctx).encode_gemma4_block(W, S, B, hid, eff, gain, idx, w, rows, E, D, K, D)
        torch.cuda.synchronize()
        return from_dev(idx, np.uint32), from_dev(w, np.uint16)

    try:
        one, two, again = run(0xFFFFFFFF), run(65), run(65)
    finally:
        ctx.close()
    for got in (two, again):
        assert np.array_equal(got[0], one[0]) and np.array_equal(got[1], one[1])


@pytest.fixture(scope="module")
def layer(tf_ctx):
    from turbo_fieldfare_b200.stack import ExpertPool, MoEBlockLayer
    pool = ExpertPool(tf_ctx, 1, 128, 2816, 704)
    pool.fill_synthetic(11)
    layer = MoEBlockLayer(tf_ctx, pool, 0, 2816, 704, 2112, 128, 8)
    layer.fill_synthetic(12)
    yield layer
    pool.close()


def _forward(tf_ctx, layer, ws, x):
    import torch
    from turbo_fieldfare_b200.stack import MoEBlock
    y = torch.zeros_like(x)
    MoEBlock(tf_ctx, layer).forward(x, y, x.shape[0], ws)
    torch.cuda.synchronize()
    assert tf_ctx.device_status() == 0
    return y


@pytest.mark.parametrize("tokens,skew", [(65, 0.0), (130, 6.0), (200, 0.0), (255, 0.0), (255, 9.0), (65, -np.inf), (201, -np.inf)])
def test_block_routing_tables_equal_the_two_calls(tf_ctx, layer, tokens, skew):
    """Block forwards of 65 to 255 tokens group in the last block of the router's second launch: every table equals what the
    router and the grouping launch write. With -inf only three experts stay selectable and the selection repeats expert 0.
    One row has a NaN. Twice, to show that the ticket is reset."""
    import torch
    from turbo_fieldfare_b200.kernels import DeviceRoutes, PrefillGroupedRoutedMoE, PrefillRouter
    from turbo_fieldfare_b200.stack import MoEBlock, Workspace, device_view_u8
    E, D, K, n = 128, 2816, 8, tokens * 8
    bias = np.zeros(E, np.float32)
    bias[[3, E - 1]] = skew, skew / 2
    if skew == -np.inf:
        bias[:] = skew
        bias[[2, 5, E - 1]] = 0.0
    layer.set_logit_bias(bias)
    try:
        gen = torch.Generator(device="cuda").manual_seed(tokens)
        x = torch.randn(tokens, D, generator=gen, device="cuda").half()
        x[7, 100] = float("nan")
        r = layer.router
        idx, w, ref = torch.full((tokens, K), -1, dtype=torch.int32, device="cuda"), dev_zeros_u16(n), DeviceRoutes(tokens, K, E)
        PrefillRouter(tf_ctx).encode_gemma4_block(r.buffer, r.buffer, r.buffer, x, layer.effective_scale, layer.per_expert_scale, idx, w, tokens, E,
                                                  D, K, D, logit_bias=layer.logit_bias, scales_offset=r.s_off, biases_offset=r.b_off)
        PrefillGroupedRoutedMoE(tf_ctx).encode_group_routes(idx, w, tokens, K, E, ref)
        torch.cuda.synchronize()
        ng, nch = ref.counters[:2].tolist()
        assert ref.counters[2].item() == n and ref.per_expert_counts.sum().item() == n
        if skew == -np.inf:
            assert ng == 4 and ref.per_expert_counts[0].item() == (tokens - 1) * (K - 3) + K         # the NaN row has nothing else
        ws, y = Workspace(tf_ctx, tokens, D, 704, 2112, K, E), torch.zeros_like(x)
        sizes = dict(sorted_pairs=n * 4, per_expert_offsets=E, per_expert_counts=E, groups=ng * 3, chunk_group=nch, chunk_start=ng, counters=4)
        for attempt in range(2):
            MoEBlock(tf_ctx, layer).forward(x, y, tokens, ws)
            torch.cuda.synchronize()
            got_idx, got_w = ws.routing(tokens)
            assert np.array_equal(got_idx.reshape(-1), from_dev(idx, np.uint32).reshape(-1)) and np.array_equal(got_w.reshape(-1), from_dev(w, np.uint16))
            tables = tf_ctx.lib.tf_workspace_routes(ws.handle).contents
            for name, words in sizes.items():
                got = device_view_u8(getattr(tables, name), words * 4).view(torch.int32)
                assert torch.equal(got, getattr(ref, name)[:words]), (name, attempt)
        assert tf_ctx.device_status() == 0
    finally:
        layer.set_logit_bias(None)


# 103 / 104 tokens lie on either side of the rule for 16-token chunks; a bias towards few experts gives them chunks of every fill
@pytest.mark.parametrize("tokens,skew", [(103, 0.0), (104, 0.0), (128, 4.0), (255, 0.0), (255, 8.0)])
def test_wide_chunks_equal_narrow_ones(tf_ctx, layer, tokens, skew):
    """A token's sums do not depend on the chunk that it sits in: a block of many tokens has the bits of the same tokens in
    blocks of 40, whose experts' rows (and the shared expert's) are taken eight at a time or in other places, and which route and
    group in one launch instead of two."""
    import torch
    from turbo_fieldfare_b200.stack import Workspace
    bias = np.zeros(128, np.float32)
    bias[[3, 60, 127]] = skew
    layer.set_logit_bias(bias)
    try:
        gen = torch.Generator(device="cuda").manual_seed(tokens)
        x = torch.randn(tokens, 2816, generator=gen, device="cuda").half()
        ws = Workspace(tf_ctx, tokens, 2816, 704, 2112, 8, 128)
        whole = _forward(tf_ctx, layer, ws, x)
        parts = torch.cat([_forward(tf_ctx, layer, ws, x[i:i + 40].contiguous()) for i in range(0, tokens, 40)])
        eight = torch.cat([_forward(tf_ctx, layer, ws, x[i:i + 7].contiguous()) for i in range(0, min(tokens, 63), 7)])
        assert torch.equal(whole, parts)
        assert torch.equal(whole[:eight.shape[0]], eight)
    finally:
        layer.set_logit_bias(None)


def test_one_token_block_equals_its_row_in_a_pair(tf_ctx, layer):
    """The one-token kernels against the grouped ones. Both add exact products in fp32, in an order of their own; the grouped
    ones hold odd activations at 1/16 (below 2^-10 that costs up to 2^-25 each): within two fp16 roundings of each other."""
    import torch
    from turbo_fieldfare_b200.stack import Workspace
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(2, 2816, generator=gen, device="cuda").half()
    ws = Workspace(tf_ctx, 2, 2816, 704, 2112, 8, 128)
    pair = _forward(tf_ctx, layer, ws, x)
    for i in range(2):
        one = _forward(tf_ctx, layer, ws, x[i:i + 1].contiguous())
        assert (one[0].double() - pair[i].double()).norm() / pair[i].double().norm() < 1e-3


@pytest.mark.parametrize("scale", [1.0, 1e-4])
@pytest.mark.parametrize("m,n", [(1, 64), (15, 128), (16, 192), (17, 2112), (704, 2816), (4095, 320), (33, 16384), (700, 4160), (2368, 4096),
                                 (2369, 4160)])
def test_tile_gemv(tf_ctx, oracle, m, n, scale):
    """Remainders of the 16-row tile and of the four-group part, both sides of the rule for sixteen warps (more than 4096
    columns, a block per SM at most); small activations keep their bits."""
    import torch
    from turbo_fieldfare_b200.kernels import DequantInt4GEMV
    o = oracle
    rng = np.random.default_rng(m * 5 + n)
    mat = config0_matrix(o, m, n, rng)
    x16 = o.f32_to_f16((rng.standard_normal(n) * scale).astype(np.float32))
    y = dev_zeros_u16(m + 8, fill=0x7E00)
    DequantInt4GEMV(tf_ctx).encode(to_dev(mat.packed), to_dev(mat.scales), to_dev(mat.biases), to_dev(x16), y, m, n)
    torch.cuda.synchronize()
    out = from_dev(y, np.uint16)
    assert np.all(out[m:] == 0x7E00)
    ref = _dense(o, mat) @ o.f16_to_f32(x16).astype(np.float64)
    # the result's rounding (2^-11, or half a subnormal step) and fp32 sums of up to 16384 products
    bound = np.abs(ref) * 2.0 ** -11 + 2.0 ** -25 + (np.abs(_dense(o, mat)) + 0.1) @ np.abs(o.f16_to_f32(x16).astype(np.float64)) * 2.0 ** -20
    assert np.all(np.abs(o.f16_to_f32(out[:m]) - ref) <= bound)


# The streaming product: remainders of the 16-row tile (the last tile repeats rows), fewer tiles than teams and than slots, rows of 1024
# columns up to the widest that leave two teams (5888), and what stays with the other kernels (fewer or more columns, planes of
# the last tile off the 16-byte grid).
@pytest.mark.parametrize("m,n", [(4096, 1024), (4104, 1280), (4100, 2816), (5002, 2816), (4112, 4096), (40008, 1024), (4096, 5632), (4104, 5888),
                                 (4096, 6144), (4099, 1280), (4098, 768)])
def test_streaming_gemv(tf_ctx, oracle, m, n):
    test_tile_gemv(tf_ctx, oracle, m, n, 1.0)


# The greedy head on both sides of the streaming form's lines (2^27 weights; fewer than 1536 columns; 2^28 weights of more than 4096
# columns), ragged vocabularies.
@pytest.mark.parametrize("d,v", [(2816, 47660), (2816, 47664), (2816, 47666), (2816, 50008), (1280, 104872), (1536, 87376), (1536, 87390),
                                 (4096, 32776), (5120, 52424), (5120, 52434)])
def test_lm_head_rows_around_the_streaming_line(tf_ctx, oracle, d, v):
    from tests.test_gpu_decode import _lm_head_gpu
    o = oracle
    rng = np.random.default_rng(v)
    mat = config0_matrix(o, v, d, rng)
    norm = o.f32_to_bf16((1.0 + 0.02 * rng.standard_normal(d)).astype(np.float32))
    hidden = o.f32_to_f16(rng.standard_normal(d).astype(np.float32))
    want, logits = o.lm_head_greedy(hidden, norm, mat)
    got = _lm_head_gpu(tf_ctx, o, hidden, norm, mat, d, v)
    assert got == want or abs(float(logits[got]) - float(logits[want])) <= 1e-5 * max(1.0, abs(float(logits[want])))


def test_lm_head_ties_and_non_finite_logits_of_the_streaming_form(tf_ctx, oracle):
    from tests.test_gpu_decode import test_lm_head_greedy_streaming_ties_and_non_finite_logits as ties
    ties(tf_ctx, oracle, 2816, 47680)


# Shared memory of the down kernel on either side of what a launch may use unasked (48 KB, the static part included): K * F / 64
# of 368, then 369 to 372. Smaller sizes first: the limit, once raised, stays raised.
@pytest.mark.parametrize("K,F", [(8, 2944), (3, 7872), (5, 4736), (7, 3392), (6, 3968), (8, 8192)])
def test_phase2_shared_memory_limit(tf_ctx, oracle, K, F):
    import torch
    from turbo_fieldfare_b200.kernels import MoE
    o = oracle
    D = 72
    rng = np.random.default_rng(K * F)
    downs = [config0_matrix(o, D, F, rng) for _ in range(K)]
    blobs = [to_dev(np.concatenate([m.packed.reshape(-1), m.scales.view(np.uint8).reshape(-1), m.biases.view(np.uint8).reshape(-1)])) for m in downs]
    coff = ExpertOffsets(0, 0, 0, 0, 0, 0, 0, D * F // 2, D * F // 2 + D * (F // 64) * 2)
    acts16, w16 = o.f32_to_f16(rng.standard_normal((K, F)).astype(np.float32)), o.f32_to_f16(rng.dirichlet(np.ones(K)).astype(np.float32))
    res16 = o.f32_to_f16(rng.standard_normal(D).astype(np.float32))
    y = dev_zeros_u16(D + 8, fill=0x7E00)
    MoE(tf_ctx).encode_routed_phase2_reduce(blob_table(blobs), coff, to_dev(acts16), to_dev(w16), to_dev(res16), y, D, F, K)
    torch.cuda.synchronize()
    out = from_dev(y, np.uint16)
    assert np.all(out[D:] == 0x7E00)
    x64, w64 = o.f16_to_f32(acts16).astype(np.float64), o.f16_to_f32(w16).astype(np.float64)
    dense = [_dense(o, m) for m in downs]
    ref = o.f16_to_f32(res16) + sum(w64[k] * (dense[k] @ x64[k]) for k in range(K))
    # the result's rounding and fp32 sums of up to 8 x 8192 products
    bound = np.abs(ref) * 2.0 ** -11 + 2.0 ** -25 + sum(w64[k] * ((np.abs(dense[k]) + 0.1) @ np.abs(x64[k])) for k in range(K)) * 2.0 ** -20
    assert np.all(np.abs(o.f16_to_f32(out[:D]) - ref) <= bound)


def _kernels_of(forward, path):
    """Text of a captured forward's graph, with the names of its kernels."""
    import torch
    from cuda.bindings import runtime
    forward()                                           # outside the capture: function attributes, side stream
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        forward()
    assert runtime.cudaGraphDebugDotPrint(graph.raw_cuda_graph(), str(path).encode(), 1)[0] == runtime.cudaError_t.cudaSuccess
    return path.read_text()


@pytest.mark.parametrize("rows,two_launches", [(None, True), (65, True), (200, True), (201, False), (256, False), (1000, False), (0xFFFFFFFF, False)])
def test_router_threshold_holds_for_block_forwards(layer, tmp_path, rows, two_launches):
    """A block forward of 200 rows takes the two-launch router by default, and below a threshold that was set the one-launch one."""
    import torch
    from turbo_fieldfare_b200.kernels import TurboContext
    from turbo_fieldfare_b200.stack import MoEBlock, Workspace
    ctx = TurboContext(0)
    try:
        if rows is not None:
            ctx.set_router_tensorcore_min_rows(rows)
        x = torch.randn(200, 2816, device="cuda").half()
        y, ws, block = torch.zeros_like(x), Workspace(ctx, 200, 2816, 704, 2112, 8, 128), MoEBlock(ctx, layer)
        text = _kernels_of(lambda: block.forward(x, y, 200, ws), tmp_path / "graph.dot")
        assert "grouped_ksplit_kernel" in text
        assert ("router_recheck_kernel" in text) is two_launches
        ws.close()
    finally:
        ctx.close()


@pytest.mark.parametrize("d", [1, 64, 255, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 3072, 3073, 4096, 4097])
@pytest.mark.parametrize("bf16,weighted", [(False, True), (True, True), (False, False)])
def test_rmsnorm_row_lengths(tf_ctx, oracle, d, bf16, weighted):
    """Both sides of every row length at which the norm takes another form; the padding between rows stays as it was."""
    import torch
    from turbo_fieldfare_b200.kernels import RMSNorm
    o, rows, stride = oracle, 5, d + 3
    rng = np.random.default_rng(d)
    to_bits, to_float = (o.f32_to_bf16, o.bf16_to_f32) if bf16 else (o.f32_to_f16, o.f16_to_f32)
    x16, w16 = to_bits(rng.standard_normal((rows, stride)).astype(np.float32)), o.f32_to_bf16(1 + 0.1 * rng.standard_normal(d).astype(np.float32))
    y = dev_zeros_u16(rows * stride, fill=0x3C01)
    RMSNorm(tf_ctx).encode(to_dev(x16), to_dev(w16) if weighted else None, y, rows, d, stride, act_dtype=0 if bf16 else 1)
    torch.cuda.synchronize()
    out = from_dev(y, np.uint16).reshape(rows, stride)
    assert np.all(out[:, d:] == 0x3C01)
    x = to_float(x16)[:, :d].astype(np.float64)
    ref = x / np.sqrt((x * x).mean(axis=1, keepdims=True) + 1e-6) * (o.bf16_to_f32(w16).astype(np.float64) if weighted else 1.0)
    # the result's rounding (8 or 11 significant bits), fp32 sums of up to 4097 squares (half of their relative error) and three fp32
    # roundings
    bound = np.abs(ref) * ((2.0 ** -8 if bf16 else 2.0 ** -11) + 2.0 ** -18) + 2.0 ** -25
    assert np.all(np.abs(to_float(out[:, :d]) - ref) <= bound)


@pytest.mark.parametrize("E,D,rows,two_launches", [(16, 256, None, False), (128, 512, None, False), (64, 1280, None, True), (16, 256, 65, True)])
def test_router_size_decides_until_a_threshold_is_set(tmp_path, E, D, rows, two_launches):
    """Block forwards of 70 tokens with up to 65536 router codes keep the one-launch router, and both routes give the same bits."""
    import torch
    from turbo_fieldfare_b200.kernels import TurboContext
    from turbo_fieldfare_b200.stack import ExpertPool, MoEBlock, MoEBlockLayer, Workspace
    ctx = TurboContext(0)
    pool = ExpertPool(ctx, 1, E, D, 64)
    try:
        pool.fill_synthetic(3)
        layer = MoEBlockLayer(ctx, pool, 0, D, 64, 64, E, 8)
        layer.fill_synthetic(4)
        if rows is not None:
            ctx.set_router_tensorcore_min_rows(rows)
        x = torch.randn(70, D, device="cuda").half()
        y, z, ws, block = torch.zeros_like(x), torch.zeros_like(x), Workspace(ctx, 70, D, 64, 64, 8, E), MoEBlock(ctx, layer)
        text = _kernels_of(lambda: block.forward(x, y, 70, ws), tmp_path / "graph.dot")
        assert ("router_recheck_kernel" in text) is two_launches
        ctx.set_router_tensorcore_min_rows(1000 if two_launches else 65)         # the other route
        block.forward(x, z, 70, ws)
        torch.cuda.synchronize()
        assert ctx.device_status() == 0 and torch.equal(y, z)
        ws.close()
    finally:
        pool.close()
        ctx.close()


# 296 and 376 blocks of 16 rows over all slots, on either side of the rule for rows of more than 3072 columns, and a split call
@pytest.mark.parametrize("D,F", [(3072, 752), (3136, 592), (3136, 752)])
def test_phase1_long_rows(tf_ctx, oracle, D, F):
    import torch
    from turbo_fieldfare_b200.kernels import MoE
    o, K = oracle, 8
    rng = np.random.default_rng(D + F)
    mats = [(config0_matrix(o, F, D, rng), config0_matrix(o, F, D, rng)) for _ in range(K)]
    parts = lambda m: [m.packed.reshape(-1), m.scales.view(np.uint8).reshape(-1), m.biases.view(np.uint8).reshape(-1)]
    blobs = [to_dev(np.concatenate(parts(g) + parts(u))) for g, u in mats]
    w, s = F * D // 2, F * (D // 64) * 2
    coff = ExpertOffsets(0, w, w + s, w + 2 * s, 2 * w + 2 * s, 2 * w + 3 * s, 0, 0, 0)
    x16 = o.f32_to_f16(rng.standard_normal(D).astype(np.float32))
    table, x, moe = blob_table(blobs), to_dev(x16), MoE(tf_ctx)
    whole, split = dev_zeros_u16(K * F + 8, fill=0x7E00), dev_zeros_u16(K * F + 8, fill=0x7E00)
    moe.encode_routed_phase1(table, coff, x, whole, D, F, K)
    moe.encode_routed_phase1_subset(table, coff, x, split, D, F, K, to_dev(np.array([6, 1], np.uint32)), 2)
    moe.encode_routed_phase1_subset(table, coff, x, split, D, F, K, to_dev(np.array([0, 2, 3, 4, 5, 7], np.uint32)), 6)
    torch.cuda.synchronize()
    assert torch.equal(whole, split)
    out, x64 = from_dev(whole, np.uint16), o.f16_to_f32(x16).astype(np.float64)
    assert np.all(out[K * F:] == 0x7E00)
    for k, (g, u) in enumerate(mats):
        gt, up = _dense(o, g) @ x64, _dense(o, u) @ x64
        ref = 0.5 * gt * (1 + np.tanh(np.clip(0.7978845608028654 * (gt + 0.044715 * gt ** 3), -20, 20))) * up
        # the result's rounding (2^-11, a third of it in the root mean square) and fp32 sums of 3136 products
        assert o.rel_l2(o.f16_to_f32(out[k * F:(k + 1) * F]), ref) < 5e-4
