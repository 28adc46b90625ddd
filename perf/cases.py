"""The work users have this framework do, as measurable cases: training steps of streaming attention, its
inference forms, and the two standalone operators, each through the public entry points.

A case names its ``kind`` and its sizes.  Sizes are those of the repository's own benchmark and tests, or lie
between them.  One program keeps to a few (dtype, heads, head dim) combinations, as a model does: the padded
operator is compiled once for each, and drawn cases stay with the listed ones.
"""

from __future__ import annotations

import math
import random

import torch

from kernels_b200 import synthetic
from kernels_b200.self_attention import self_attention
from kernels_b200.sharding import useful_pairs
from kernels_b200.softmax import softmax
from kernels_b200.streaming_attention import (
    output_projection,
    qkv_rope_projection,
    quantize_fp8_tiles,
    rope_tables,
    streaming_attention,
    streaming_attention_fp8,
    streaming_attention_step,
    streaming_attention_varlen,
)

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ELSIZE = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # training step at the size of a unit test or a debugging run: launches and host time are what it costs
        dict(name="train_f32_small", kind="train", dtype="f32", B=2, H=4, T=512, D=64, c=32, back=2, len_lo=256, len_hi=512),
        # training step of a small model kept in full precision
        dict(name="train_f32", kind="train", dtype="f32", B=16, H=4, T=2000, D=64, c=32, back=4, len_lo=1000, len_hi=2000),
        # training step with short chunks: many utterances, 100 visible frames, an odd length
        dict(name="train_f16_c10", kind="train", dtype="f16", B=64, H=12, T=1353, D=64, c=10, back=9, len_lo=676, len_hi=1353),
        # training step of a streaming encoder: head dim 64, ragged lengths
        dict(name="train_f16", kind="train", dtype="f16", B=8, H=16, T=4096, D=64, c=128, back=4, len_lo=2048, len_hi=4096),
        # training step on long sequences without padding: the benchmark's default workload
        dict(name="train_bf16_long", kind="train", dtype="bf16", B=4, H=32, T=16384, D=128, c=256, back=2, len_lo=0, len_hi=0),
        # training step with chunks shorter than a tile and a long look-back: one GPU's share of the 8-GPU workload
        dict(name="train_bf16_c64", kind="train", dtype="bf16", B=8, H=32, T=8192, D=128, c=64, back=8, len_lo=4096, len_hi=8192),
        # training step on a packed batch: sequences one after the other instead of padded
        dict(name="train_packed", kind="packed", dtype="bf16", seqs=256, H=16, D=128, c=64, back=2, len_lo=128, len_hi=1024),
        # one chunk of a few live streams against their caches: a server's smallest call
        dict(name="step_small", kind="step", dtype="f16", B=2, H=8, H_kv=8, Tq=64, T=256, D=64, c=64, back=3),
        # a layer's attention block on a prompt: projections with rotary embedding, attention with shared key/value
        # heads, output projection
        dict(name="layer_prefill", kind="layer", dtype="bf16", B=4, T=2048, E=4096, H=32, H_kv=8, D=128, c=256, back=2),
        # inference with 8-bit attention: q, k, v come in 16 bits, are quantised and attended
        dict(name="forward_fp8", kind="fp8", dtype="bf16", B=2, H=32, T=8192, D=128, c=256, back=2),
        # dense self-attention forward with key padding
        dict(name="dense_f16", kind="dense", dtype="f16", B=16, H=16, T=2048, D=64, len_lo=1024, len_hi=2048),
        # row softmax over a large matrix
        dict(name="softmax_f32", kind="softmax", dtype="f32", rows=65536, cols=4096),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# what a drawn case may cost at most: two thirds of the largest listed case of the same arithmetic
_MOST_FLOPS = {"f32": 3.0e10, "f16": 1.5e12, "bf16": 1.8e12}
_MOST_BYTES = 2.0e9


def draw(rng: random.Random):
    for _ in range(1000):
        case = _draw_one(rng)
        w = work(case)
        if w["flops"] <= _MOST_FLOPS[case["dtype"]] and w["bytes"] <= _MOST_BYTES:
            return case
    raise RuntimeError("no case within the ranges")


def _draw_one(rng: random.Random):
    kind = rng.choice(["train", "train", "train", "packed", "step", "layer", "fp8", "dense", "softmax"])
    if kind == "train":
        dtype, H, D = rng.choice([("f32", 4, 64), ("f16", 12, 64), ("f16", 16, 64), ("bf16", 32, 128)])
        T = _log_int(rng, 200, 4000 if dtype == "f32" else 16384)
        B = _log_int(rng, 2, 64)
        c = _log_int(rng, 10, 300)
        back = rng.randint(2, 10)
        lens = not (dtype == "bf16" and rng.random() < 0.5)
        return dict(kind=kind, dtype=dtype, B=B, H=H, T=T, D=D, c=c, back=back, len_lo=T // 2 if lens else 0, len_hi=T if lens else 0)
    if kind == "packed":
        hi = _log_int(rng, 200, 4000)
        return dict(kind=kind, dtype=rng.choice(["f16", "bf16"]), seqs=_log_int(rng, 4, 256), H=rng.choice([8, 16]), D=rng.choice([64, 128]),
                    c=_log_int(rng, 10, 300), back=rng.randint(0, 8), len_lo=hi // 8, len_hi=hi)
    if kind == "step":
        c, back = _log_int(rng, 16, 300), rng.randint(0, 8)
        H = rng.choice([8, 16, 32])
        return dict(kind=kind, dtype=rng.choice(["f16", "bf16"]), B=_log_int(rng, 1, 128), H=H, H_kv=rng.choice([H, H // 4]), Tq=c,
                    T=c * (back + 1), D=rng.choice([64, 128]), c=c, back=back)
    if kind == "layer":
        return dict(kind=kind, dtype="bf16", B=_log_int(rng, 2, 16), T=_log_int(rng, 100, 8192), E=rng.choice([2048, 4096]), H=32, H_kv=8,
                    D=128, c=_log_int(rng, 32, 300), back=rng.randint(2, 8))
    if kind == "fp8":
        return dict(kind=kind, dtype="bf16", B=_log_int(rng, 1, 16), H=rng.choice([16, 32]), T=_log_int(rng, 200, 16384), D=128,
                    c=_log_int(rng, 32, 300), back=rng.randint(0, 8))
    if kind == "dense":
        T = _log_int(rng, 200, 4096)
        return dict(kind=kind, dtype=rng.choice(["f16", "bf16"]), B=_log_int(rng, 1, 64), H=rng.choice([6, 16]), T=T, D=rng.choice([64, 128]),
                    len_lo=T // 2, len_hi=T)
    return dict(kind=kind, dtype=rng.choice(["f32", "f16", "bf16"]), rows=_log_int(rng, 128, 65536), cols=_log_int(rng, 128, 20000))


def _randn(gen, shape, dtype, scale=1.0):
    x = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=gen)
    return x.mul_(scale) if scale != 1.0 else x


def _lens(case, seed):
    return synthetic.make_lens(case["B"], case["len_lo"], case["len_hi"], seed) if case["len_hi"] else None


def _packed_lens(case, seed):
    """The same lengths in another order for every seed: the tensors' shapes belong to the case."""
    lens = synthetic.make_lens(case["seqs"], case["len_lo"], case["len_hi"])
    return lens[torch.randperm(len(lens), generator=torch.Generator().manual_seed(seed))]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    if kind == "train":
        shape = (case["B"], case["H"], case["T"], case["D"])
        # 16-bit head-dim-64 models scale q, k, v down, as the benchmark's workload does
        qk = case["D"] ** -0.25 if case["dtype"] == "f16" else 1.0
        q, k, v = (_randn(gen, shape, dtype, qk).requires_grad_() for _ in range(3))
        do = _randn(gen, shape, dtype)
        lens = _lens(case, seed)
        return dict(case=case, q=q, k=k, v=v, do=do, lens=None if lens is None else lens.cuda())
    if kind == "packed":
        lens = _packed_lens(case, seed)
        cu = torch.zeros(len(lens) + 1, dtype=torch.int32)
        cu[1:] = lens.cumsum(0)
        shape = (int(cu[-1]), case["H"], case["D"])
        q, k, v = (_randn(gen, shape, dtype).requires_grad_() for _ in range(3))
        return dict(case=case, q=q, k=k, v=v, do=_randn(gen, shape, dtype), cu=cu)
    if kind == "step":
        kv = (case["B"], case["H_kv"], case["T"], case["D"])
        q = _randn(gen, (case["B"], case["H"], case["Tq"], case["D"]), dtype)
        return dict(case=case, q=q, k=_randn(gen, kv, dtype), v=_randn(gen, kv, dtype))
    if kind == "layer":
        E, D = case["E"], case["D"]
        n_qkv = (case["H"] + 2 * case["H_kv"]) * D
        x = _randn(gen, (case["B"], case["T"], E), dtype)
        w_qkv, w_o = _randn(gen, (n_qkv, E), dtype, E**-0.5), _randn(gen, (E, case["H"] * D), dtype, (case["H"] * D) ** -0.5)
        cos, sin = rope_tables(case["T"], D, device="cuda")
        return dict(case=case, x=x, w_qkv=w_qkv, w_o=w_o, cos=cos, sin=sin)
    if kind == "fp8":
        shape = (case["B"], case["H"], case["T"], case["D"])
        return dict(case=case, q=_randn(gen, shape, dtype), k=_randn(gen, shape, dtype), v=_randn(gen, shape, dtype))
    if kind == "dense":
        shape = (case["B"], case["H"], case["T"], case["D"])
        q, k, v = (_randn(gen, shape, dtype) for _ in range(3))
        return dict(case=case, q=q, k=k, v=v, lens=_lens(case, seed).cuda())
    return dict(case=case, x=_randn(gen, (case["rows"], case["cols"]), dtype, 2.0))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        q, k, v = state["q"], state["k"], state["v"]
        o = streaming_attention(q, k, v, state["lens"], case["c"], case["back"])
        return (o, *torch.autograd.grad(o, (q, k, v), state["do"]))
    if kind == "packed":
        q, k, v = state["q"], state["k"], state["v"]
        o = streaming_attention_varlen(q, k, v, state["cu"], case["c"], case["back"])
        return (o, *torch.autograd.grad(o, (q, k, v), state["do"]))
    with torch.no_grad():
        if kind == "step":
            return streaming_attention_step(state["q"], state["k"], state["v"], None, case["c"], case["back"])
        if kind == "layer":
            q, k, v = qkv_rope_projection(state["x"], state["w_qkv"], case["H"], case["H_kv"], case["D"], state["cos"], state["sin"])
            return output_projection(streaming_attention(q, k, v, None, case["c"], case["back"]), state["w_o"])
        if kind == "fp8":
            q8, k8, v8 = (quantize_fp8_tiles(state[n]) for n in "qkv")
            return streaming_attention_fp8(q8[0], k8[0], v8[0], q8[1], k8[1], v8[1], None, case["c"], case["back"])
        if kind == "dense":
            return self_attention(state["q"], state["k"], state["v"], state["lens"])
        return softmax(state["x"])


def work(case):
    """Every input read once, every output written once; matrix products over the unmasked (query, key) pairs.
    Ragged lengths count with their mean."""
    kind, e = case["kind"], ELSIZE[case["dtype"]]
    if kind == "softmax":
        n = case["rows"] * case["cols"]
        return dict(bytes=2 * n * e, flops=0)
    D, H = case["D"], case["H"]
    if kind == "packed":
        ls = _packed_lens(case, 0).tolist()
    elif kind in ("train", "dense"):
        ls = [(case["len_lo"] + case["len_hi"]) // 2 or case["T"]] * case["B"]
    else:
        ls = [case["T"]] * case["B"]
    if kind == "step":
        pairs = H * case["B"] * case["Tq"] * case["T"]
        rows_q, rows_kv = H * case["B"] * case["Tq"], case["H_kv"] * case["B"] * case["T"]
        return dict(bytes=(2 * rows_q + 2 * rows_kv) * D * e, flops=4 * D * pairs)
    if kind == "dense":
        return dict(bytes=4 * H * sum(ls) * D * e, flops=4 * D * H * sum(n * n for n in ls))
    pairs, rows = H * sum(useful_pairs(n, case["c"], case["back"]) for n in ls), H * sum(ls)
    if kind in ("train", "packed"):  # forward q, k, v -> o; backward q, k, v, dO -> dq, dk, dv
        return dict(bytes=11 * rows * D * e, flops=14 * D * pairs)
    if kind == "layer":
        tokens, E, n_qkv = case["B"] * case["T"], case["E"], (H + 2 * case["H_kv"]) * D
        return dict(bytes=2 * tokens * E * e + (n_qkv + H * D) * E * e, flops=2 * tokens * E * (n_qkv + H * D) + 4 * D * pairs)
    return dict(bytes=4 * rows * D * e, flops=4 * D * pairs)  # fp8: 16-bit q, k, v -> o


def tolerance(case):
    """About four times the relative error measured against the same path in 64 bits (gradients included)."""
    kind, dtype = case["kind"], case["dtype"]
    if kind == "softmax":
        return {"rel": {"f32": 4e-7, "f16": 8e-4, "bf16": 6.5e-3}[dtype]}
    if kind == "fp8":  # two implementations round the probabilities to three mantissa bits: 2.5e-2 each
        return {"rel": 5e-2}
    if kind == "layer":
        return {"rel": 1.6e-2}
    return {"rel": {"f32": 2.6e-6, "f16": 1.2e-3, "bf16": 1e-2}[dtype]}


def _exact_streaming(q, k, v, do, length, c, back, q_start=0):
    """One sequence of one batch entry in 64 bits: ``q [H, Tq, D]`` holds positions ``q_start ..``, ``k``, ``v``
    ``[H, T, D]``.  Chunk by chunk against the chunk's key window; ``(o, dq, dk, dv)``, the gradients None without
    ``do``."""
    q, k, v = q.double(), k.double(), v.double()
    scale = q.shape[-1] ** -0.5
    o = torch.zeros_like(q)
    dq, dk, dv = (None, None, None) if do is None else (torch.zeros_like(t) for t in (q, k, v))
    for lo in range(q_start // c * c, length, c):
        r0, r1 = max(lo, q_start), min(lo + c, length)
        k0 = max(lo - back * c, 0)
        qi, ki, vi = q[:, r0 - q_start:r1 - q_start], k[:, k0:r1], v[:, k0:r1]
        if r0 >= r1:
            continue
        p = torch.softmax(qi @ ki.mT * scale, dim=-1)
        o[:, r0 - q_start:r1 - q_start] = p @ vi
        if do is not None:
            doi = do[:, r0:r1].double()
            dv[:, k0:r1] += p.mT @ doi
            ds = p * (doi @ vi.mT - (doi * (p @ vi)).sum(-1, keepdim=True)) * scale
            dq[:, r0:r1] = ds @ ki
            dk[:, k0:r1] += ds.mT @ qi
    return o, dq, dk, dv


def exact(case, seed):
    """What ``run`` returns, in 64 bits; None where the chunks are too many for a loop over them."""
    kind = case["kind"]
    if kind == "softmax":
        return torch.cat([torch.softmax(x.double(), dim=-1) for x in prepare(case, seed)["x"].split(4096)])
    if kind == "dense":
        st = prepare(case, seed)
        return torch.stack([_exact_streaming(st["q"][b], st["k"][b], st["v"][b], None, int(n), case["T"], 0)[0]
                            for b, n in enumerate(st["lens"].tolist())])
    seqs = case["seqs"] if kind == "packed" else case["B"]
    chunks = seqs * (case["len_hi"] if kind == "packed" else case["T"]) // case["c"]
    rows = seqs * case["H"] * (case["len_hi"] if kind == "packed" else case["T"])
    if chunks > 20000 or rows * case["D"] > 3.0e8:
        return None
    st = prepare(case, seed)
    c, back = case["c"], case["back"]
    if kind == "packed":
        outs = [torch.zeros(st[n].shape, dtype=torch.float64, device="cuda") for n in ("q", "q", "k", "v")]
        cu = st["cu"].tolist()
        for a, z in zip(cu, cu[1:]):
            heads = (st[n].detach()[a:z].transpose(0, 1) for n in ("q", "k", "v", "do"))
            for out, got in zip(outs, _exact_streaming(*heads, z - a, c, back)):
                out[a:z] = got.transpose(0, 1)
        return tuple(outs)
    if kind == "layer":
        H, Hk, D = case["H"], case["H_kv"], case["D"]
        w_qkv, w_o, cos, sin = (st[n].double() for n in ("w_qkv", "w_o", "cos", "sin"))
        ys = []
        for x in st["x"]:
            q, k, v = (x.double() @ w_qkv.T).view(-1, H + 2 * Hk, D).transpose(0, 1).split((H, Hk, Hk))
            q, k = (torch.cat([t[..., :D // 2] * cos.T - t[..., D // 2:] * sin.T,
                               t[..., D // 2:] * cos.T + t[..., :D // 2] * sin.T], dim=-1) for t in (q, k))
            k, v = (t.repeat_interleave(H // Hk, dim=0) for t in (k, v))
            o = _exact_streaming(q, k, v, None, x.shape[0], c, back)[0]
            ys.append(o.transpose(0, 1).reshape(-1, H * D) @ w_o.T)
        return torch.stack(ys)
    q, k, v = (st[n].detach() for n in "qkv")
    group = q.shape[1] // k.shape[1]
    k, v = (t.repeat_interleave(group, dim=1) for t in (k, v))
    lens = st.get("lens")
    lens = [case["T"]] * case["B"] if lens is None else lens.tolist()
    do = st.get("do")
    q_start = case["T"] - case["Tq"] if kind == "step" else 0
    per_seq = [_exact_streaming(q[b], k[b], v[b], None if do is None else do[b], int(n), c, back, q_start) for b, n in enumerate(lens)]
    outs = [torch.stack(ts) for ts in zip(*per_seq) if ts[0] is not None]
    return tuple(outs) if kind == "train" else outs[0]
