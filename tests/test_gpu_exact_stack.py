"""GPU tests of the stacks whose experts run on the tensor cores with exact weights (65 to 255 tokens, the routed ones from 7 rows per expert on)
against the CUDA-core kernels, which a context takes once its tensor-core threshold has been set. Both add exact products in fp32 and round the activations,
the partials and the hidden state to fp16 in the same places, so a row differs by single fp16 steps of those: less than 2^-10 of its norm."""
import numpy as np
import pytest

from helpers import from_dev, to_dev

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -10


def _spread(o, rng, rows, groups):
    """Scales and biases of many magnitudes within a row and over the rows, of either sign, unrelated; some rows without scales, some without
    biases."""
    s = np.exp2(rng.uniform(-20, -4, (rows, groups))) * rng.choice([-1.0, 1.0], (rows, groups))
    b = np.exp2(rng.uniform(-16, 0, (rows, groups))) * rng.choice([-1.0, 1.0], (rows, groups))
    s[::7] = 0.0
    b[3::7] = 0.0
    s *= np.exp2(rng.uniform(-12, 0, (rows, 1)))
    b *= np.abs(s).max(axis=1, keepdims=True) / np.maximum(np.abs(b).max(axis=1, keepdims=True), 1e-30)
    b += 2.0 ** -6 * (s == 0).all(axis=1, keepdims=True)
    return o.f32_to_bf16(s.astype(np.float32)), o.f32_to_bf16(b.astype(np.float32))


def _both(o, tokens, d, f, fs, experts, top_k, layers=1, zipf=False, spread=None, shared_bits=4):
    """(hidden states of the default context, of one whose threshold was set, launches of either)."""
    import torch
    from turbo_fieldfare_b200.kernels import TurboContext
    from turbo_fieldfare_b200.stack import MoEBlockLayer, MoEStack
    out, launches = [], []
    h16 = o.f32_to_f16(np.random.default_rng(tokens + d).standard_normal((tokens, d)).astype(np.float32))
    for set_threshold in (False, True):
        ctx = TurboContext(0)
        if set_threshold:
            ctx.set_tensorcore_min_tokens(256)
        stack = MoEStack(ctx, layers=layers, d=d, f=f, fs=fs, num_experts=experts, top_k=top_k, seed=5, align=256)
        try:
            if shared_bits == 8:
                stack.layers[0] = MoEBlockLayer(ctx, stack.pool, 0, d, f, fs, experts, top_k, shared_bits=8)
                stack.layers[0].fill_synthetic(6)
                stack._build()
            if zipf:
                stack.set_logit_bias((-1.1 * np.log(np.random.default_rng(1).permutation(experts) + 1.0)).astype(np.float32))
            if spread is not None:
                spread(stack)
            ws = stack.workspace(255)
            first = None
            for _ in range(4):
                h = to_dev(h16.copy())
                before = ctx.launch_count
                stack.forward(h, tokens, ws)
                count = ctx.launch_count - before
                first = h if first is None else first
                assert torch.equal(first, h)
            torch.cuda.synchronize()
            assert ctx.device_status() == 0
            launches.append(count)
            out.append(o.f16_to_f32(from_dev(first, np.uint16)).astype(np.float64).reshape(tokens, d))
        finally:
            torch.cuda.synchronize()
            stack.close()
            ctx.close()
    return out[0], out[1], launches


def _row_errors(a, b):
    return np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)


# (tokens, d, f, fs, experts, top_k, launches more): the production layer from the shared expert's first size on, on either side of seven rows per
# expert; groups of a row that fill a stage or not (d, f, fs / 64 mod 4 = 0 ... 3), one, three and several 64-column blocks of extra groups;
# few and most experts; the widest rows; a shared expert of 8 bits, which stays on the other kernels
SIZES = [(65, 2816, 704, 2112, 128, 8, 1), (111, 2816, 704, 2112, 128, 8, 1), (112, 2816, 704, 2112, 128, 8, 1), (255, 2816, 704, 2112, 128, 8, 1),
         (255, 1088, 192, 1088, 16, 8, 1), (255, 448, 320, 2432, 8, 8, 1), (65, 2752, 576, 1600, 4, 4, 1), (255, 640, 704, 1728, 256, 8, 1),
         (130, 3072, 3072, 3072, 8, 2, 1), (200, 3072, 1280, 2112, 16, 4, 0)]


@pytest.mark.parametrize("tokens,d,f,fs,experts,top_k,more", SIZES)
def test_exact_stack_matches_the_cuda_core_stack(tf_ctx, oracle, tokens, d, f, fs, experts, top_k, more):
    a, b, launches = _both(oracle, tokens, d, f, fs, experts, top_k, shared_bits=4 if more else 8)
    assert launches[0] - launches[1] == more                 # copies with extra columns more, a reduction less: the new route
    assert _row_errors(a, b).max() < TOL


def test_exact_stack_of_two_layers_with_skewed_routing(tf_ctx, oracle):
    a, b, launches = _both(oracle, 190, 2816, 704, 2112, 128, 8, layers=2, zipf=True)
    assert launches[0] > launches[1]
    # near-ties of the second layer's router may fall either way
    assert np.median(_row_errors(a, b)) < TOL and (_row_errors(a, b) > TOL).mean() < 0.05


def test_exact_stack_with_scales_and_biases_of_many_magnitudes(tf_ctx, oracle):
    o = oracle
    d, f, fs, experts = 1088, 576, 1088, 8

    def spread(stack):
        rng = np.random.default_rng(12)
        off, layer = stack.pool.offsets, stack.layers[0]
        for e in range(experts):
            blob = stack.pool.download(0, e).copy()
            for name, rows, cols in (("gate", f, d), ("up", f, d), ("down", d, f)):
                for field, plane in zip("sb", _spread(o, rng, rows, cols // 64)):
                    at = getattr(off, f"{name}_{field}_off")
                    blob[at:at + plane.size * 2] = plane.reshape(-1).view(np.uint8)
            stack.pool.upload(0, e, blob)
        for t in (layer.shared_gate, layer.shared_up, layer.shared_down):
            packed, _, _ = t.download()
            t.upload(packed, *_spread(o, rng, t.rows, t.cols // 64))

    a, b, launches = _both(oracle, 240, d, f, fs, experts, 4, spread=spread)
    assert launches[0] > launches[1]
    assert np.isfinite(b).all() and np.isfinite(a).all() and _row_errors(a, b).max() < TOL


def test_up_to_64_tokens_nothing_changes(tf_ctx, oracle):
    a, b, launches = _both(oracle, 64, 2816, 704, 2112, 128, 8)
    assert launches[0] == launches[1] and np.array_equal(a, b)
