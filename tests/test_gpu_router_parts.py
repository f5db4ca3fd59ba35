"""GPU tests of the two-launch router whose approximate logits are summed in parts of the columns: indices and weights of the one-launch kernel, bit
for bit, on either side of every rule that picks the parts, and in stacks, where the launch begins before the rows it reads are written."""
import numpy as np
import pytest

from helpers import from_dev

pytestmark = pytest.mark.gpu


# (rows, experts, d, stride): one round of the few-row blocks and just more; two rounds of one-chunk blocks and just more (592 of them at 148 SMs);
# one chunk, an even and an odd number of them, parts that end with fewer chunks than the others; one, two and partial blocks of experts;
# the last tokens of a block missing; rows wider than the matrix
CASES = [(256, 128, 2816, 2816), (296, 128, 2816, 2816), (297, 128, 2816, 2816), (848, 128, 2816, 2880), (865, 128, 2816, 2816), (1500, 20, 2816, 2816),
         (433, 256, 2816, 2816), (600, 200, 256, 256), (3000, 129, 512, 512), (1100, 128, 1024, 1032), (2400, 128, 1280, 1280), (700, 64, 3072, 3072)]


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("rows,experts,d,stride", CASES)
def test_router_in_parts_equals_the_one_launch_router(tf_ctx, rows, experts, d, stride, bf16):
    import torch
    from turbo_fieldfare_b200.kernels import TurboContext
    from turbo_fieldfare_b200.stack import AffineTensor, _ptr
    gen = torch.Generator(device="cuda").manual_seed(rows + experts)
    x = torch.randn(rows, stride, generator=gen, device="cuda").to(torch.bfloat16 if bf16 else torch.float16)
    eff = (1.0 + 0.1 * torch.randn(d, generator=gen, device="cuda")).to(torch.bfloat16)
    gain = (0.5 + torch.rand(experts, generator=gen, device="cuda")).to(torch.bfloat16)
    out = []
    for threshold in (65, 0xFFFFFFFF):
        ctx = TurboContext(0)
        try:
            ctx.set_router_tensorcore_min_rows(threshold)
            w = AffineTensor(experts, d, 8)
            w.fill_synthetic(ctx, 7)
            idx = torch.zeros(rows * 8, dtype=torch.int32, device="cuda")
            wt = torch.zeros(rows * 8, dtype=torch.int16, device="cuda")
            p = w.projection()
            for _ in range(2):                     # the second call finds its scratch
                ctx.check(ctx.lib.tf_router_gemma4_block(ctx.handle, 0, p.weights, p.weights_off, p.scales, p.scales_off, p.biases, p.biases_off, _ptr(x), 0,
                                                         0 if bf16 else 1, _ptr(eff), 0, _ptr(gain), 0, None, _ptr(idx), 0, _ptr(wt), 0, None,
                                                         rows, experts, d, 8, stride))
            torch.cuda.synchronize()
            assert ctx.device_status() == 0
            out.append((from_dev(idx, np.uint32), from_dev(wt, np.uint16)))
        finally:
            ctx.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


# up to 255 tokens the re-check groups, too: pairs that fill no round of 32 to a warp, and all of its counters
@pytest.mark.parametrize("tokens,experts", [(66, 256), (112, 128), (113, 128), (131, 200), (255, 20), (255, 256), (300, 64), (880, 64)])
def test_stacks_route_on_the_rows_of_their_own_layer(tf_ctx, tokens, experts):
    import torch
    from turbo_fieldfare_b200.kernels import TurboContext
    from turbo_fieldfare_b200.stack import MoEStack
    x = torch.randn(tokens, 2816, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").half()
    out = []
    for threshold in (65, 0xFFFFFFFF):
        ctx = TurboContext(0)
        ctx.set_router_tensorcore_min_rows(threshold)
        stack = MoEStack(ctx, layers=4, d=2816, f=128, fs=128, num_experts=experts, top_k=8, seed=3, align=256)
        try:
            ws = stack.workspace(tokens)
            for _ in range(1 if out else 20):
                h = x.clone()
                stack.forward(h, tokens, ws)
                out.append(h)
            torch.cuda.synchronize()
            assert ctx.device_status() == 0
        finally:
            torch.cuda.synchronize()
            stack.close()
            ctx.close()
    assert all(torch.equal(out[0], h) for h in out[1:])


# Calls of fewer rows may need more scratch (more parts): 600 and 848 rows outgrow what 1024 rows left. A graph that was captured before keeps its
# buffer; under capture a call takes as many parts as the buffer holds, or, where there is none yet, one launch.
@pytest.mark.parametrize("before,captured,after", [([1024], 1024, [600, 848]), ([1500], 600, [848, 4096]), ([333], 1024, [848]), ([], 700, [700, 1500])])
def test_a_captured_router_keeps_its_scratch(before, captured, after):
    import torch
    from turbo_fieldfare_b200.kernels import TurboContext
    from turbo_fieldfare_b200.stack import AffineTensor, _ptr
    d, experts = 2816, 128
    ctx, plain = TurboContext(0), TurboContext(0)
    try:
        plain.set_router_tensorcore_min_rows(0xFFFFFFFF)
        gen = torch.Generator(device="cuda").manual_seed(captured)
        most = max(before + [captured] + after)
        x = torch.randn(most, d, generator=gen, device="cuda").half()
        eff = (1.0 + 0.1 * torch.randn(d, generator=gen, device="cuda")).to(torch.bfloat16)
        gain = (0.5 + torch.rand(experts, generator=gen, device="cuda")).to(torch.bfloat16)
        w = AffineTensor(experts, d, 8)
        w.fill_synthetic(ctx, 7)
        p = w.projection()
        torch.cuda.synchronize()

        def route(c, rows, idx, wt, stream=0):
            c.check(c.lib.tf_router_gemma4_block(c.handle, stream, p.weights, p.weights_off, p.scales, p.scales_off, p.biases, p.biases_off, _ptr(x), 0, 1,
                                                 _ptr(eff), 0, _ptr(gain), 0, None, _ptr(idx), 0, _ptr(wt), 0, None, rows, experts, d, 8, d))

        def outputs(rows):
            return torch.zeros(rows * 8, dtype=torch.int32, device="cuda"), torch.zeros(rows * 8, dtype=torch.int16, device="cuda")

        def expected(rows):
            idx, wt = outputs(rows)
            route(plain, rows, idx, wt)
            torch.cuda.synchronize()
            return idx, wt

        for rows in before:
            route(ctx, rows, *outputs(rows))
        torch.cuda.synchronize()
        idx, wt = outputs(captured)
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            route(ctx, captured, idx, wt, stream.cuda_stream)
        for rows in after:
            got, want = outputs(rows), expected(rows)
            route(ctx, rows, *got)
            torch.cuda.synchronize()
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        want = expected(captured)
        for _ in range(3):
            idx.zero_()
            wt.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(idx, want[0]) and torch.equal(wt, want[1])
        assert ctx.device_status() == 0
        del graph
    finally:
        torch.cuda.synchronize()
        ctx.close()
        plain.close()
