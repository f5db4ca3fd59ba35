"""The work that a user of this framework has it do, as cases with inputs, one pass and the result's tolerance.

Sizes are those of the repository's own model configuration (hidden 2816, 128 experts of 704, top 8, shared expert of
2112, 30 layers, a vocabulary of 262144 rows) and of its benchmark; token counts run over the range in between.

Kinds of work:
  step       one decode step of the 30-layer stack for a batch of sequences, one token each, replayed as a CUDA graph
             (how a server runs its decode loop)
  prefill    the 30-layer stack over one block of prompt tokens, called eagerly
  block      one MoE block, called eagerly, fp16 or bf16 rows, optionally with popular and rare experts (a Zipf bias on
             the router's logits)
  operators  one MoE layer for one token through the single operators, as a host that keeps the reference's per-operator
             calls makes them: router, blob table, shared expert, gate/up phase, down phase with the weighted sum
  lm_head    final norm, tied int4 LM head and greedy token for one sequence
  gemv       one int4 matrix-vector product
  qmm        one dense int4 matrix-matrix product (prompt rows through one projection)
"""
import math

import numpy as np
import torch

from turbo_fieldfare_b200 import stack as tf_stack
from turbo_fieldfare_b200.kernels import (DequantInt4GEMV, LMHeadChainInt4, MoE, MPPPrefillInt4QMM, SharedExpertInt4,
                                          SharedExpertProjection, TurboContext)

D, F, FS, E, K = tf_stack.GEMMA4_D, tf_stack.GEMMA4_F, tf_stack.GEMMA4_FS, tf_stack.GEMMA4_E, tf_stack.GEMMA4_K
LAYERS, VOCAB = tf_stack.GEMMA4_LAYERS, 262144

_contexts = {}


def _context():
    """One library context per device, kept for the program's life as a server keeps it."""
    device = torch.cuda.current_device()
    if device not in _contexts:
        _contexts[device] = TurboContext(device)
    return _contexts[device]


def listed():
    return [
        # a single chat user: latency of one token through the whole stack
        {"name": "step_1", "kind": "step", "tokens": 1},
        # a handful of sequences decoded together (an odd number: sequences come and go)
        {"name": "step_11", "kind": "step", "tokens": 11},
        # the benchmark's batched decode
        {"name": "step_64", "kind": "step", "tokens": 64},
        # a busy server's decode batch, ragged
        {"name": "step_200", "kind": "step", "tokens": 200},
        # a short prompt, or a chunk of a chunked prefill
        {"name": "prefill_333", "kind": "prefill", "tokens": 333},
        # the benchmark's prompt block
        {"name": "prefill_4096", "kind": "prefill", "tokens": 4096},
        # the smallest call of the block: one token, called eagerly
        {"name": "block_1", "kind": "block", "tokens": 1, "dtype": "f16", "zipf": False},
        # the benchmark's prompt block in bf16 with skewed expert popularity
        {"name": "block_4096_bf16_zipf", "kind": "block", "tokens": 4096, "dtype": "bf16", "zipf": True},
        # a host that calls operator by operator
        {"name": "operators_1", "kind": "operators"},
        # the token at the end of every decode step
        {"name": "lm_head", "kind": "lm_head", "vocab": VOCAB},
        # one expert's gate matrix alone: the smallest launch there is
        {"name": "gemv_704", "kind": "gemv", "rows": F, "cols": D},
        # the shared expert's gate projection over a ragged block of prompt rows
        {"name": "qmm_1000", "kind": "qmm", "m": 1000, "n": FS, "k": D},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "prefill", "prefill", "block", "block", "lm_head", "gemv", "qmm"])
    if kind == "step":
        return {"kind": kind, "tokens": _log_int(rng, 1, 255)}
    if kind == "prefill":
        return {"kind": kind, "tokens": _log_int(rng, 64, 4096)}
    if kind == "block":
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096), "dtype": rng.choice(["f16", "bf16"]),
                "zipf": rng.random() < 0.5}
    if kind == "lm_head":
        return {"kind": kind, "vocab": 8 * _log_int(rng, 4000, VOCAB // 8)}
    if kind == "gemv":
        return {"kind": kind, "rows": _log_int(rng, 64, 65536), "cols": 64 * _log_int(rng, 4, 64)}
    return {"kind": kind, "m": _log_int(rng, 16, 4096), "n": 8 * _log_int(rng, 32, 1024), "k": 64 * _log_int(rng, 4, 64)}


def _rows(seed, tokens, cols, dtype=torch.float16):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(tokens, cols, generator=gen, device="cuda", dtype=torch.float32).to(dtype)


def _zipf_bias(seed):
    rng = np.random.default_rng(seed)
    p = 1.0 / (rng.permutation(E) + 1) ** 1.1
    return np.log(p / p.sum()).astype(np.float32)


def _layer(ctx, seed, zipf):
    """One production layer: 128 experts, router and shared expert."""
    pool = tf_stack.ExpertPool(ctx, 1, E, D, F)
    pool.fill_synthetic(seed)
    layer = tf_stack.MoEBlockLayer(ctx, pool, 0, D, F, FS, E, K)
    layer.fill_synthetic(seed + 1)
    if zipf:
        layer.set_logit_bias(_zipf_bias(seed))
    return pool, layer


def _affine(ctx, seed, rows, cols):
    mat = tf_stack.AffineTensor(rows, cols, 4)
    mat.fill_synthetic(ctx, seed)
    return mat


def _shared_projection(t):
    return SharedExpertProjection(t.buffer, t.buffer, t.buffer, t.rows, t.cols, 0, t.s_off, t.b_off)


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = {"kind": kind, "case": case}
    if kind in ("step", "prefill"):
        tokens = case["tokens"]
        model = tf_stack.MoEStack(ctx, layers=LAYERS, seed=seed)
        s.update(model=model, ws=model.workspace(tokens), x=_rows(seed, tokens, D))
        s["h"] = torch.empty_like(s["x"])
        if kind == "step":
            # a server captures its decode step once per batch size and replays it
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                s["h"].copy_(s["x"])
                model.forward(s["h"], tokens, s["ws"], stream=stream)
                stream.synchronize()
                s["graph"] = torch.cuda.CUDAGraph()
                with torch.cuda.graph(s["graph"], stream=stream):
                    model.forward(s["h"], tokens, s["ws"], stream=torch.cuda.current_stream())
            torch.cuda.current_stream().wait_stream(stream)
    elif kind == "block":
        tokens = case["tokens"]
        pool, layer = _layer(ctx, seed, case["zipf"])
        x = _rows(seed, tokens, D, torch.bfloat16 if case["dtype"] == "bf16" else torch.float16)
        s.update(pool=pool, layer=layer, block=tf_stack.MoEBlock(ctx, layer), x=x, y=torch.empty_like(x),
                 ws=tf_stack.Workspace(ctx, tokens, D, F, FS, K, E))
    elif kind == "operators":
        pool, layer = _layer(ctx, seed, False)
        half = dict(dtype=torch.float16, device="cuda")
        s.update(pool=pool, layer=layer, x=_rows(seed, 1, D), moe=MoE(ctx), shared=SharedExpertInt4(ctx),
                 projections=[_shared_projection(t) for t in (layer.shared_gate, layer.shared_up, layer.shared_down)],
                 indices=torch.zeros(K, dtype=torch.int32, device="cuda"), weights=torch.zeros(K, **half),
                 blobs=torch.zeros(K, dtype=torch.int64, device="cuda"), acts=torch.zeros(K * F, **half),
                 shared_y=torch.zeros(D, **half), y=torch.zeros(D, **half),
                 scratch=[torch.zeros(FS, **half) for _ in range(3)])
    elif kind == "lm_head":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        norm = (1.0 + 0.02 * torch.randn(D, generator=gen, device="cuda")).to(torch.bfloat16)
        s.update(head=LMHeadChainInt4(ctx), w=_affine(ctx, seed, case["vocab"], D), norm=norm, x=_rows(seed, 1, D),
                 token=torch.zeros(1, dtype=torch.int32, device="cuda"))
    elif kind == "gemv":
        s.update(gemv=DequantInt4GEMV(ctx), w=_affine(ctx, seed, case["rows"], case["cols"]), x=_rows(seed, 1, case["cols"]),
                 y=torch.zeros(case["rows"], dtype=torch.float16, device="cuda"))
    elif kind == "qmm":
        s.update(qmm=MPPPrefillInt4QMM(ctx), w=_affine(ctx, seed, case["n"], case["k"]), x=_rows(seed, case["m"], case["k"]),
                 y=torch.zeros(case["m"], case["n"], dtype=torch.float16, device="cuda"))
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "step":
        s["h"].copy_(s["x"])            # this step's input; the stack works in place
        s["graph"].replay()
        return s["h"]
    if kind == "prefill":
        s["h"].copy_(s["x"])
        s["model"].forward(s["h"], case["tokens"], s["ws"])
        return s["h"]
    if kind == "block":
        forward = s["block"].forward_bf16 if case["dtype"] == "bf16" else s["block"].forward
        forward(s["x"], s["y"], case["tokens"], s["ws"])
        return s["y"]
    if kind == "operators":
        layer, pool, moe, x = s["layer"], s["pool"], s["moe"], s["x"]
        r = layer.router
        moe.encode_router_gemma4(r.buffer, r.buffer, r.buffer, x, layer.effective_scale, layer.per_expert_scale, s["indices"],
                                 s["weights"], E, D, K, scales_offset=r.s_off, biases_offset=r.b_off)
        moe.encode_expert_table(pool.ptr(0, 0), pool.stride, s["indices"], K, E, s["blobs"])
        s["shared"].encode(x, *s["projections"], s["shared_y"], *s["scratch"])
        moe.encode_routed_phase1(s["blobs"], pool.offsets, x, s["acts"], D, F, K)
        moe.encode_routed_phase2_reduce(s["blobs"], pool.offsets, s["acts"], s["weights"], s["shared_y"], s["y"], D, F, K)
        return {"indices": s["indices"], "weights": s["weights"], "y": s["y"]}
    w = s["w"]
    if kind == "lm_head":
        s["head"].encode_greedy_decode(s["x"], s["norm"], w.buffer, w.buffer, w.buffer, s["token"], D, case["vocab"],
                                       scales_offset=w.s_off, biases_offset=w.b_off)
        return s["token"]
    if kind == "gemv":
        s["gemv"].encode(w.buffer, w.buffer, w.buffer, s["x"], s["y"], case["rows"], case["cols"], scales_offset=w.s_off,
                         biases_offset=w.b_off)
        return s["y"]
    s["qmm"].encode(w.buffer, w.buffer, w.buffer, s["x"], s["y"], case["m"], case["n"], case["k"], scales_offset=w.s_off,
                    biases_offset=w.b_off)
    return s["y"]


# ---- the same results in 64 bits, in plain torch on the bytes that the state holds ----

def _plain(buf, rows, cols, bits, w_off, s_off, b_off):
    """A quantised matrix as float64: code * scale + bias, 64 columns to a group, the low nibble first."""
    groups, nbytes = cols // 64, rows * cols * bits // 8
    q = buf[w_off:w_off + nbytes].view(rows, -1)
    if bits == 4:
        q = torch.stack((q & 15, q >> 4), dim=-1)
    sb = [buf[o:o + rows * groups * 2].view(torch.bfloat16).view(rows, groups, 1).double() for o in (s_off, b_off)]
    return (q.reshape(rows, groups, 64).double() * sb[0] + sb[1]).view(rows, cols)


def _plain_tensor(t):
    return _plain(t.buffer, t.rows, t.cols, t.bits, 0, t.s_off, t.b_off)


def _plain_mlp(x, gate, up, down):
    return (torch.nn.functional.gelu(x @ gate.T, approximate="tanh") * (x @ up.T)) @ down.T


def _plain_block(layer, x):
    """(indices, weights, y) of one MoE block for float64 rows."""
    logits = (x * layer.effective_scale.view(torch.bfloat16).double()) @ _plain_tensor(layer.router).T
    if layer.logit_bias is not None:
        logits = logits + layer.logit_bias.double()
    top, idx = torch.topk(logits, K, dim=-1)
    weights = torch.softmax(top, dim=-1) * layer.per_expert_scale.view(torch.bfloat16).double()[idx]
    y = _plain_mlp(x, *(_plain_tensor(t) for t in (layer.shared_gate, layer.shared_up, layer.shared_down)))
    pool, o = layer.pool, layer.pool.offsets
    for e in torch.unique(idx).tolist():
        blob = tf_stack.device_view_u8(pool.ptr(layer.layer_index, e), pool.stride)
        token, rank = torch.nonzero(idx == e, as_tuple=True)
        out = _plain_mlp(x[token], _plain(blob, F, D, 4, o.gate_w_off, o.gate_s_off, o.gate_b_off),
                         _plain(blob, F, D, 4, o.up_w_off, o.up_s_off, o.up_b_off),
                         _plain(blob, D, F, 4, o.down_w_off, o.down_s_off, o.down_b_off))
        y.index_add_(0, token, out * weights[token, rank][:, None])
    return idx, weights, y


def exact(case, seed):
    s = prepare(case, seed)
    kind, x = case["kind"], s["x"].double()
    if kind in ("step", "prefill"):
        if case["tokens"] > 512:
            return None                 # takes too long in 64 bits
        model = s["model"]
        for layer, w in zip(model.layers, model.norm_weights):
            normed = x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + model.eps) * w.view(torch.bfloat16).double()
            x = x + _plain_block(layer, normed)[2]
        return x
    if kind == "block":
        return _plain_block(s["layer"], x)[2]
    if kind == "operators":
        idx, weights, y = _plain_block(s["layer"], x)
        return {"indices": idx[0].int(), "weights": weights[0], "y": y[0]}
    w = s["w"]
    if kind == "lm_head":
        normed = x * torch.rsqrt(x.square().mean(dim=-1, keepdim=True) + 1e-6) * s["norm"].double()
        return (_plain_tensor(w) @ normed[0]).argmax().int().view(1)
    y = x @ _plain_tensor(w).T
    return y[0] if kind == "gemv" else y


def _affine_bytes(rows, cols, bits):
    return rows * cols * bits // 8 + 2 * rows * (cols // 64) * 2


def _block_work(tokens):
    """Weights that one block reads (the experts that a uniform router would touch, the shared expert, the router) and its
    multiply-adds; activation rows are counted by the caller."""
    touched = E * (1.0 - (1.0 - K / E) ** tokens)
    expert = 2 * _affine_bytes(F, D, 4) + _affine_bytes(D, F, 4)
    shared = 2 * _affine_bytes(FS, D, 4) + _affine_bytes(D, FS, 4)
    flops = 2.0 * tokens * (K * 3 * D * F + 3 * D * FS + E * D)
    return touched * expert + shared + _affine_bytes(E, D, 8), flops


def work(case):
    kind = case["kind"]
    if kind in ("step", "prefill"):
        nbytes, flops = _block_work(case["tokens"])
        return {"bytes": LAYERS * (nbytes + D * 2) + 2 * case["tokens"] * D * 2, "flops": LAYERS * flops}
    if kind == "block":
        nbytes, flops = _block_work(case["tokens"])
        return {"bytes": nbytes + 2 * case["tokens"] * D * 2, "flops": flops}
    if kind == "operators":
        nbytes, flops = _block_work(1)
        return {"bytes": nbytes + 2 * D * 2, "flops": flops}
    if kind == "lm_head":
        return {"bytes": _affine_bytes(case["vocab"], D, 4) + 2 * D * 2 + 4, "flops": 2.0 * case["vocab"] * D}
    if kind == "gemv":
        return {"bytes": _affine_bytes(case["rows"], case["cols"], 4) + 2 * (case["rows"] + case["cols"]),
                "flops": 2.0 * case["rows"] * case["cols"]}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": _affine_bytes(n, k, 4) + 2 * m * (n + k), "flops": 2.0 * m * n * k}


def tolerance(case):
    if case["kind"] == "block" and case["dtype"] == "bf16":
        return {"rel": 2.5e-3, "max": 3e-2}
    return TOLERANCE[case["kind"]]


# About four times what was seen between two correct evaluations: stacks and blocks with their expert products on the other
# kernel family (other summation order, weights rounded to fp16 or not; fp16 outputs 2.4e-4 and 5e-3 at the most, rows of
# bf16 6.5e-4 and 7.8e-3), the single products against sums in 64 bits (2.1e-4 and 5e-4: the rounding of the fp16 result).
TOLERANCE = {
    "step": {"rel": 1.4e-3, "max": 2e-2},
    "prefill": {"rel": 1.4e-3, "max": 2e-2},
    "block": {"rel": 1e-3, "max": 8e-3},
    "operators": {"rel": 8e-4, "max": 4e-3},
    "lm_head": "exact",
    "gemv": {"rel": 8e-4, "max": 2e-3},
    "qmm": {"rel": 8e-4, "max": 2e-3},
}
