"""GPU tests of the one-token launches (block forward and stack step) against the launches of two tokens, whose sums have the same
order: the same token in both rows must give the same bits, whatever the sizes and whatever the router selects."""
import numpy as np
import pytest

from helpers import from_dev, to_dev

pytestmark = pytest.mark.gpu

# (d, f, fs, experts, top_k): production; parts of four groups full and partial in d, f and fs; one tile per block, several and more than are in
# flight at once; few and most experts; down blocks near the shared memory that they have beside a gate/up block, and beyond it (there a
# stack takes the layered launches; a block, too, for few columns, long experts or still larger blocks)
SIZES = [(2816, 704, 2112, 128, 8), (256, 128, 192, 16, 8), (320, 64, 64, 9, 8), (64, 64, 64, 4, 2), (1088, 192, 448, 256, 7),
         (2752, 1024, 576, 24, 8), (3072, 1280, 1152, 16, 6), (1088, 1408, 2816, 16, 6), (512, 1536, 1536, 16, 8), (1024, 2816, 704, 9, 4),
         (3072, 1536, 3072, 16, 8), (3072, 3072, 3072, 9, 8)]
LAYERED_STACKS, LAYERED_BLOCKS = SIZES[-5:], SIZES[-4:]


def _rows(o, rng, d):
    return o.f32_to_f16(rng.standard_normal((1, d)).astype(np.float32))


@pytest.mark.parametrize("d,f,fs,experts,top_k", SIZES)
def test_one_token_block_and_stack_have_the_bits_of_two_equal_tokens(tf_ctx, oracle, d, f, fs, experts, top_k):
    import torch
    from turbo_fieldfare_b200.stack import MoEBlock, MoEStack
    o = oracle
    stack = MoEStack(tf_ctx, layers=3, d=d, f=f, fs=fs, num_experts=experts, top_k=top_k, seed=7, align=256)
    try:
        rng = np.random.default_rng(d + f)
        x16 = _rows(o, rng, d)
        ws1, ws2 = stack.workspace(1), stack.workspace(2)
        one, two = to_dev(x16.copy()), to_dev(np.concatenate([x16, x16]))
        for _ in range(2):                               # the second step runs on what the first one left in the workspace
            stack.forward(one, 1, ws1)
            stack.forward(two, 2, ws2)
        torch.cuda.synchronize()
        assert tf_ctx.device_status() == 0
        a, b = from_dev(one, np.uint16).reshape(-1), from_dev(two, np.uint16).reshape(2, d)
        assert np.array_equal(b[0], b[1]) and np.array_equal(a, b[0])
        idx1, w1 = ws1.routing(1)
        idx2, w2 = ws2.routing(2)
        assert np.array_equal(idx1[0], idx2[0]) and np.array_equal(w1[0], w2[0])
        y1, y2 = torch.zeros(d, dtype=torch.int16, device="cuda"), torch.zeros(2 * d, dtype=torch.int16, device="cuda")
        x1, x2 = to_dev(x16), to_dev(np.concatenate([x16, x16]))
        MoEBlock(tf_ctx, stack.layers[1]).forward(x1, y1, 1, ws1)
        MoEBlock(tf_ctx, stack.layers[1]).forward(x2, y2, 2, ws2)
        torch.cuda.synchronize()
        assert tf_ctx.device_status() == 0
        assert np.array_equal(from_dev(y1, np.uint16), from_dev(y2, np.uint16)[:d])
        assert np.array_equal(ws1.routing(1)[0][0], ws2.routing(2)[0][0])
    finally:
        stack.close()


@pytest.mark.parametrize("d,f,fs,experts,top_k", SIZES)
def test_one_token_takes_its_own_launches(tf_ctx, oracle, tmp_path, d, f, fs, experts, top_k):
    """Three a layer of a stack and, in a block, kernels of their own; the layered ones for sizes that those take less time for."""
    import torch
    from test_gpu_edges import _kernels_of
    from turbo_fieldfare_b200.stack import MoEBlock, MoEStack
    stack = MoEStack(tf_ctx, layers=2, d=d, f=f, fs=fs, num_experts=experts, top_k=top_k, seed=7, align=256)
    try:
        h = to_dev(_rows(oracle, np.random.default_rng(d), d))
        y = torch.zeros(d, dtype=torch.int16, device="cuda")
        ws = stack.workspace(1)
        before = tf_ctx.launch_count
        stack.forward(h, 1, ws)
        launches = tf_ctx.launch_count - before
        text = _kernels_of(lambda: MoEBlock(tf_ctx, stack.layers[1]).forward(h, y, 1, ws), tmp_path / "graph.dot")
        torch.cuda.synchronize()
        assert tf_ctx.device_status() == 0
        size = (d, f, fs, experts, top_k)
        assert (launches == 3 * 2) is (size not in LAYERED_STACKS)
        kernels = ("one_token_front_kernel", "one_token_gate_up_kernel", "one_token_down_kernel")
        assert [k in text for k in kernels] == [size not in LAYERED_BLOCKS] * 3
    finally:
        stack.close()


@pytest.mark.parametrize("case", ["ties", "few", "none", "nan"])
@pytest.mark.parametrize("experts,top_k", [(128, 8), (20, 8), (256, 3)])
def test_one_token_selection_of_ties_and_masked_experts(tf_ctx, oracle, case, experts, top_k):
    """Logit biases decide: equal logits at and around the last rank (the lower index wins), fewer selectable experts than ranks, none at
    all, and NaN logits (never selected)."""
    import torch
    from turbo_fieldfare_b200.stack import MoEStack
    o = oracle
    d = 256
    stack = MoEStack(tf_ctx, layers=1, d=d, f=128, fs=192, num_experts=experts, top_k=top_k, seed=3, align=256)
    try:
        rng = np.random.default_rng(experts)
        bias = np.full(experts, -np.inf, np.float32)
        if case == "ties":
            bias = np.where(rng.random(experts) < 0.5, np.float32(1e30), np.float32(2e30)).astype(np.float32)     # swallows the logits
        elif case == "few":
            bias[rng.permutation(experts)[:max(1, top_k - 2)]] = 0.0
        elif case == "nan":
            bias = rng.standard_normal(experts).astype(np.float32)
            bias[rng.permutation(experts)[:experts // 2]] = np.nan
        stack.set_logit_bias(bias)
        x16 = _rows(o, rng, d)
        ws1, ws2 = stack.workspace(1), stack.workspace(2)
        one, two = to_dev(x16.copy()), to_dev(np.concatenate([x16, x16]))
        stack.forward(one, 1, ws1)
        stack.forward(two, 2, ws2)
        torch.cuda.synchronize()
        assert tf_ctx.device_status() == 0
        assert np.array_equal(ws1.routing(1)[0][0], ws2.routing(2)[0][0])
        assert np.array_equal(ws1.routing(1)[1][0], ws2.routing(2)[1][0])
        assert np.array_equal(from_dev(one, np.uint16).reshape(-1), from_dev(two, np.uint16).reshape(2, d)[0])
    finally:
        stack.close()
