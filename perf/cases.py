"""The work that users of the attention operators have them do, as measurable cases.

Every case is one call of a public entry point (or the two calls of a step that belong together) on inputs made
from a seed. The kinds:

    decode         one new token per sequence against a contiguous cache (small interactive batches)
    decode_paged   one new token per sequence against a paged cache, every sequence attends to its whole context
    decode_topk    one new token per sequence, a given list of gathered positions through a paged cache
    decode_select  the positions are selected first (``topk_indices`` over a score per key), then attended to; FP8 cache
    prefill        forward over whole sequences; 16-bit, or FP8 tensors with per-tensor scales
    prefill_chunk  a chunk of new queries at the end of a paged cache, with the log-sum-exps that merging needs
    train          forward and backward: dense, or sparse (tile skipping) with an optional causal window
    train_packed   forward and backward over packed sequences of unequal length
    train_gated    forward and backward of the gated operator, one window per KV head

Inputs are iid N(0, 1) (nothing is skipped then) unless ``data`` is "llm", which has the structure of the
repository's long-context benchmark: attention concentrates on the own 1024-token block and on a sink.
"""

import math
import os
import random
import sys

import torch

# the package's folder is not an importable name: it goes on the path like the tests and the benchmark put it there
sys.path.insert(0, os.path.join(os.getcwd(), "flash-sparse-attention_b200"))

import flash_sparse_attn as fsa  # noqa: E402
from flash_sparse_attn.utils.mask import topk_indices  # noqa: E402

DEV = "cuda"
DTYPE = {"bf16": torch.bfloat16, "fp16": torch.float16, "e4m3": torch.float8_e4m3fn}
ELEM = {"bf16": 2, "fp16": 2, "e4m3": 1}
GATED_WINDOWS = (512, 1024, 2048, 4096)  # KV head h looks back over GATED_WINDOWS[h % 4] tokens


def listed():
    return [
        # an interactive decode step of a small model: one sequence, a few thousand cached tokens; launches and latency
        dict(name="decode_one", kind="decode", batch=1, ctx=4000, hq=8, hkv=2, d=64, dtype="bf16"),
        # a serving batch that attends to everything it has, contexts of very different lengths, paged cache
        dict(name="decode_paged", kind="decode_paged", batch=32, ctx_lo=1000, ctx_hi=16000, page=128, hq=32, hkv=8, d=128,
             dtype="bf16"),
        # the long-context serving benchmark: 2048 gathered positions out of 4K-128K through 256-token pages
        dict(name="decode_topk", kind="decode_topk", batch=64, ctx_lo=4096, ctx_hi=131072, topk=2048, page=256, hq=64, hkv=8,
             d=128, dtype="bf16"),
        # a sparse decode step as it runs in a model: score the keys, pick positions, attend to them; FP8 cache
        dict(name="decode_select", kind="decode_select", batch=16, ctx_lo=8000, ctx_hi=32000, topk=1024, page=64, hq=32, hkv=8,
             d=128, dtype="e4m3"),
        # a short prompt of a small model
        dict(name="prefill_small", kind="prefill", op="dense", batch=1, seqlen=1024, hq=8, hkv=2, d=64, dtype="bf16", data="iid"),
        # a long prompt, sparse operator at its default threshold, on inputs whose attention is concentrated
        dict(name="prefill_long", kind="prefill", op="sparse", batch=1, seqlen=16384, hq=32, hkv=8, d=128, dtype="bf16",
             data="llm"),
        # prompts with quantised q, k, v
        dict(name="prefill_fp8", kind="prefill", op="dense", batch=2, seqlen=6000, hq=32, hkv=8, d=128, dtype="e4m3", data="iid"),
        # chunked prefill: the next 500 tokens of four sequences against what they have cached
        dict(name="prefill_chunk", kind="prefill_chunk", batch=4, chunk=500, ctx_lo=2000, ctx_hi=12000, page=256, hq=32, hkv=8,
             d=128, dtype="bf16"),
        # training with a 1024-token causal window (the headline benchmark)
        dict(name="train_window", kind="train", op="sparse", batch=2, seqlen=4096, window=1024, hq=32, hkv=8, d=128,
             dtype="bf16", data="iid"),
        # training, full causal attention, fp16
        dict(name="train_causal", kind="train", op="dense", batch=1, seqlen=8192, window=0, hq=32, hkv=8, d=128, dtype="fp16",
             data="iid"),
        # training on packed documents of 256 to 4096 tokens
        dict(name="train_packed", kind="train_packed", n_seq=16, lo=256, hi=4096, hq=32, hkv=8, d=128, dtype="bf16"),
        # training with gates and per-head windows
        dict(name="train_gated", kind="train_gated", batch=4, seqlen=8192, hq=32, hkv=8, d=128, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kind and its sizes; nothing drawn costs more than the largest listed case."""
    kind = rng.choice(["decode", "decode_paged", "decode_topk", "decode_select", "prefill", "prefill_long", "prefill_fp8",
                       "prefill_chunk", "train_window", "train_causal", "train_packed", "train_gated"])
    heads = rng.choice([(8, 2), (16, 4), (32, 8), (32, 4), (64, 8)])
    hq, hkv = heads
    d = rng.choice([64, 128, 128, 128])
    h16 = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "decode":
        return dict(kind=kind, batch=_log_int(rng, 1, 16), ctx=_log_int(rng, 500, 32000), hq=hq, hkv=hkv, d=d, dtype=h16)
    if kind == "decode_paged":
        hi = _log_int(rng, 2000, 32000)
        return dict(kind=kind, batch=_log_int(rng, 2, 64), ctx_lo=max(16, hi // 16), ctx_hi=hi, page=rng.choice([64, 128, 256]),
                    hq=hq, hkv=hkv, d=d, dtype=h16)
    if kind in ("decode_topk", "decode_select"):
        hi = _log_int(rng, 8000, 64000)
        f8 = kind == "decode_select"
        return dict(kind=kind, batch=_log_int(rng, 2, 64), ctx_lo=max(4200, hi // 8), ctx_hi=hi, topk=_log_int(rng, 200, 4096),
                    page=rng.choice([64, 128, 256]), hq=hq, hkv=hkv, d=128 if f8 else d, dtype="e4m3" if f8 else h16)
    if kind == "prefill":
        return dict(kind=kind, op=rng.choice(["dense", "sparse"]), batch=rng.randint(1, 4), seqlen=_log_int(rng, 200, 6000),
                    hq=hq, hkv=hkv, d=d, dtype=h16, data="iid")
    if kind == "prefill_long":
        return dict(kind="prefill", op="sparse", batch=1, seqlen=_log_int(rng, 6000, 16384), hq=32, hkv=8, d=128, dtype="bf16",
                    data="llm")
    if kind == "prefill_fp8":
        return dict(kind="prefill", op="dense", batch=rng.randint(1, 4), seqlen=_log_int(rng, 1000, 6000), hq=hq, hkv=hkv, d=128,
                    dtype="e4m3", data="iid")
    if kind == "prefill_chunk":
        hi = _log_int(rng, 3000, 16000)
        chunk = _log_int(rng, 60, 1500)
        return dict(kind=kind, batch=rng.randint(1, 6), chunk=chunk, ctx_lo=max(chunk, hi // 8), ctx_hi=hi,
                    page=rng.choice([128, 256]), hq=hq, hkv=hkv, d=d, dtype=h16)
    if kind == "train_window":
        return dict(kind="train", op="sparse", batch=rng.randint(1, 2), seqlen=_log_int(rng, 1000, 8192),
                    window=_log_int(rng, 256, 2048), hq=hq, hkv=hkv, d=d, dtype=h16, data="iid")
    if kind == "train_causal":
        return dict(kind="train", op=rng.choice(["dense", "sparse"]), batch=1, seqlen=_log_int(rng, 1000, 8192), window=0,
                    hq=min(hq, 32), hkv=min(hkv, 8), d=d, dtype=h16, data="iid")
    if kind == "train_packed":
        return dict(kind=kind, n_seq=rng.randint(3, 16), lo=_log_int(rng, 64, 512), hi=_log_int(rng, 800, 4096),
                    hq=min(hq, 32), hkv=min(hkv, 8), d=d, dtype=h16)
    return dict(kind=kind, batch=rng.randint(1, 2), seqlen=_log_int(rng, 700, 8192), hq=min(hq, 32), hkv=min(hkv, 8), d=d,
                dtype=h16)


# ---------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------
def _lengths(case):
    """Lengths that belong to the case and not to the inputs: spread evenly over [lo, hi], odd ones among them."""
    if case["kind"] == "train_packed":
        lo, hi, n = case["lo"], case["hi"], case["n_seq"]
    else:
        lo, hi, n = case["ctx_lo"], case["ctx_hi"], case["batch"]
    got = [lo + (hi - lo) * i // max(n - 1, 1) for i in range(n)] if n > 1 else [hi]
    random.Random(n).shuffle(got)
    return got


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=g, device=DEV, dtype=dtype)


def _cache(g, case, pages):
    """K and V of a paged cache, in the case's type. FP8: values as a quantiser leaves them, with one scale per tensor."""
    shape = (pages, case["page"], case["hkv"], case["d"])
    if case["dtype"] != "e4m3":
        return _randn(g, *shape, dtype=DTYPE[case["dtype"]]), _randn(g, *shape, dtype=DTYPE[case["dtype"]]), {}
    k, v = ((_randn(g, *shape) * 64).to(torch.float8_e4m3fn) for _ in range(2))
    scale = torch.full((1,), 1.0 / 64, device=DEV, dtype=torch.float32)
    return k, v, dict(is_quant=True, query_scale=scale, key_scale=scale, value_scale=scale)


def _query(g, case, *shape):
    if case["dtype"] == "e4m3":
        return (_randn(g, *shape) * 64).to(torch.float8_e4m3fn)
    return _randn(g, *shape, dtype=DTYPE[case["dtype"]])


def _pages(g, lens, page):
    """A page table that scatters the sequences' pages over the cache."""
    per = [-(-n // page) for n in lens]
    perm = torch.randperm(sum(per), generator=g, device=DEV).to(torch.int32)
    table = torch.zeros(len(lens), max(per), dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(per):
        table[b, :n] = perm[at:at + n]
        at += n
    return table, sum(per)


def _llm_like(g, b, s, hq, hkv, d, dtype):
    """0.35 noise + 0.65 position features + 0.75 latent of the 1024-token block (+ sink latent on the first 64 keys)."""
    pairs = (d + 1) // 2
    freqs = torch.exp(torch.linspace(math.log(1.0 / max(float(s), 1024.0)), math.log(1.0 / 64.0), pairs, device=DEV))
    ang = torch.arange(s, device=DEV, dtype=torch.float32)[:, None] * freqs[None, :]
    pos = torch.cat([ang.sin(), ang.cos()], dim=-1)[:, :d].to(dtype)
    kv_of = torch.arange(hq, device=DEV) // (hq // hkv)
    q, k, v = (_randn(g, b, s, h, d, dtype=dtype) for h in (hq, hkv, hkv))
    blk = torch.arange(s, device=DEV) // 1024
    lat = _randn(g, b, (s + 1023) // 1024, hkv, d, dtype=dtype)
    q.mul_(0.35).add_(pos[None, :, None, :], alpha=0.65).add_(lat[:, blk][:, :, kv_of, :], alpha=0.75)
    k.mul_(0.35).add_(pos[None, :, None, :], alpha=0.65).add_(lat[:, blk], alpha=0.75)
    sink = _randn(g, b, hkv, d, dtype=dtype)
    q.add_(sink[:, None, kv_of, :], alpha=0.45)
    k[:, :64].add_(sink[:, None], alpha=1.10)
    v[:, :64].mul_(1.15)
    return q, k, v


def prepare(case, seed):
    g = _gen(seed)
    kind, hq, hkv, d = case["kind"], case["hq"], case["hkv"], case["d"]
    if kind == "decode":
        t = DTYPE[case["dtype"]]
        q = _randn(g, case["batch"], hq, d, dtype=t)
        k, v = (_randn(g, case["batch"], case["ctx"], hkv, d, dtype=t) for _ in range(2))
        return dict(case=case, q=q, k=k, v=v)
    if kind.startswith("decode") or kind == "prefill_chunk":
        lens = _lengths(case)
        table, pages = _pages(g, lens, case["page"])
        k, v, scales = _cache(g, case, pages)
        used = torch.tensor(lens, dtype=torch.int32, device=DEV)
        st = dict(case=case, k=k, v=v, scales=scales, table=table, used=used)
        if kind == "prefill_chunk":
            st["q"] = _query(g, case, case["batch"], case["chunk"], hq, d)
            return st
        st["q"] = _query(g, case, case["batch"], hq, d)
        if kind in ("decode_topk", "decode_select"):
            width = max(lens)
            score = torch.randn(case["batch"], width, generator=g, device=DEV)
            score.masked_fill_(torch.arange(width, device=DEV)[None, :] >= used[:, None], float("-inf"))
            if kind == "decode_select":
                st["score"] = score
            else:  # the positions as some selection left them: distinct, in no order
                st["idx"] = score.topk(case["topk"], dim=-1, sorted=True).indices.to(torch.int32)
        return st
    if kind == "prefill":
        b, s = case["batch"], case["seqlen"]
        if case["data"] == "llm":
            q, k, v = _llm_like(g, b, s, hq, hkv, d, DTYPE[case["dtype"]])
        else:
            q, k, v = (_query(g, case, b, s, h, d) for h in (hq, hkv, hkv))
        scales = {}
        if case["dtype"] == "e4m3":
            one = torch.full((1,), 1.0 / 64, device=DEV, dtype=torch.float32)
            scales = dict(is_quant=True, query_scale=one, key_scale=one, value_scale=one)
        return dict(case=case, q=q, k=k, v=v, scales=scales)
    # training
    t = DTYPE[case["dtype"]]
    st = dict(case=case)
    if kind == "train_packed":
        lens = _lengths(case)
        cu = torch.zeros(len(lens) + 1, dtype=torch.int32)
        cu[1:] = torch.tensor(lens).cumsum(0)
        total = int(cu[-1])
        st.update(cu=cu.to(DEV), longest=max(lens), lens=lens)
        lead = (total,)
    else:
        lead = (case["batch"], case["seqlen"])
    st["q"] = _randn(g, *lead, hq, d, dtype=t).requires_grad_(True)
    st["k"], st["v"] = (_randn(g, *lead, hkv, d, dtype=t).requires_grad_(True) for _ in range(2))
    st["dout"] = _randn(g, *lead, hq, d, dtype=t)
    if kind == "train_gated":
        st["alpha"] = _randn(g, *lead, hq, dtype=t).requires_grad_(True)
        st["delta"] = _randn(g, *lead, hkv, dtype=t).requires_grad_(True)
    w = _windows(case)
    st["windows"] = None if w is None else torch.tensor([[0, x, 0, 0] for x in w], dtype=torch.int32, device=DEV)
    return st


def _windows(case):
    """Tokens that each KV head looks back over, or None."""
    if case["kind"] == "train_gated":
        return [GATED_WINDOWS[h % 4] for h in range(case["hkv"])]
    if case["kind"] == "train" and case["window"]:
        return [case["window"]] * case["hkv"]
    return None


# ---------------------------------------------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "decode":
        return fsa.flash_dense_attn_with_kvcache_func(st["q"], st["k"], st["v"])
    if kind == "decode_paged":
        return fsa.flash_dense_attn_with_kvcache_func(st["q"], st["k"], st["v"], page_table=st["table"], seqused_k=st["used"],
                                                      **st["scales"])
    if kind == "decode_topk":
        return fsa.flash_sparse_attn_with_kvcache_func(st["q"], st["k"], st["v"], page_table=st["table"],
                                                       gather_kv_indices=st["idx"], seqused_k=st["used"], **st["scales"])
    if kind == "decode_select":
        idx = topk_indices(st["score"], case["topk"], dtype=torch.int32)
        out = fsa.flash_sparse_attn_with_kvcache_func(st["q"], st["k"], st["v"], page_table=st["table"], gather_kv_indices=idx,
                                                      seqused_k=st["used"], **st["scales"])
        return out, idx
    if kind == "prefill":
        op = fsa.flash_dense_attn_func if case["op"] == "dense" else fsa.flash_sparse_attn_func
        return op(st["q"], st["k"], st["v"], is_causal=True, **st["scales"])
    if kind == "prefill_chunk":
        return fsa.flash_dense_attn_func(st["q"], st["k"], st["v"], is_causal=True, is_split_kv=True, page_table=st["table"],
                                         seqused_k=st["used"], return_lse=True)
    leaves = [st["q"], st["k"], st["v"]]
    if kind == "train":
        kw = dict(is_causal=True, window_sizes=st["windows"], is_split_kv=True, is_split_qo=True)
        op = fsa.flash_dense_attn_func if case["op"] == "dense" else fsa.flash_sparse_attn_func
        out = op(*leaves, **kw)
    elif kind == "train_packed":
        out = fsa.flash_sparse_attn_varlen_func(*leaves, st["cu"], st["cu"], st["longest"], st["longest"], is_causal=True,
                                                is_split_kv=True, is_split_qo=True)
    else:
        leaves += [st["alpha"], st["delta"]]
        out = fsa.flash_gated_attn_func(*leaves, is_causal=True, window_sizes=st["windows"])
    grads = torch.autograd.grad(out, leaves, st["dout"])
    return (out.detach(),) + tuple(grads)


# ---------------------------------------------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def _causal_pairs(sq, sk, window=0):
    """(query, key) pairs of a causal head whose queries are the last sq of sk positions."""
    first = sk - sq  # keys before the first query's own
    if not window or window >= sk:
        return sq * first + sq * (sq + 1) // 2
    ramp = max(0, min(sq, window - first - 1))  # rows that see fewer keys than the window is wide
    return ramp * (first + 1) + ramp * (ramp - 1) // 2 + (sq - ramp) * window


def work(case):
    kind, hq, hkv, d, e = case["kind"], case["hq"], case["hkv"], case["d"], ELEM[case["dtype"]]
    out_e = 2
    if kind == "decode":
        keys = case["batch"] * case["ctx"]
        return dict(bytes=keys * hkv * d * 2 * e + case["batch"] * hq * d * (e + out_e), flops=4.0 * d * hq * keys)
    if kind.startswith("decode"):
        lens, b = _lengths(case), case["batch"]
        keys, extra = sum(lens), 4 * b * (-(-max(lens) // case["page"]))
        if kind != "decode_paged":
            keys = b * case["topk"]
            extra = 4 * keys
        if kind == "decode_select":
            extra += 4 * sum(lens) + 4 * keys  # the scores, and the positions written
        return dict(bytes=keys * hkv * d * 2 * e + b * hq * d * (e + out_e) + extra, flops=4.0 * d * hq * keys)
    if kind == "prefill":
        b, s = case["batch"], case["seqlen"]
        pairs = b * _causal_pairs(s, s)
        # "llm": which tiles are skipped depends on the scores, and only those are certain to be computed
        flops = (2.0 if case["data"] == "llm" else 4.0) * d * hq * pairs
        return dict(bytes=b * s * d * (hq * (e + out_e) + 2 * hkv * e), flops=flops)
    if kind == "prefill_chunk":
        lens, c = _lengths(case), case["chunk"]
        pairs = sum(_causal_pairs(c, n) for n in lens)
        q = case["batch"] * c * hq
        return dict(bytes=q * (d * (e + out_e) + 4) + sum(lens) * hkv * d * 2 * e, flops=4.0 * d * hq * pairs)
    if kind == "train_packed":
        lens = _lengths(case)
        rows, pairs = sum(lens), hq * sum(_causal_pairs(n, n) for n in lens)
    else:
        rows = case["batch"] * case["seqlen"]
        w = _windows(case) or [0] * hkv
        pairs = case["batch"] * (hq // hkv) * sum(_causal_pairs(case["seqlen"], case["seqlen"], x) for x in w)
    # read q, k, v, dout; write out, dq, dk, dv (gated: alpha, delta and their gradients too)
    nbytes = rows * d * 2 * (4 * hq + 4 * hkv) + (rows * 2 * 2 * (hq + hkv) if kind == "train_gated" else 0)
    return dict(bytes=nbytes, flops=14.0 * d * pairs)


# ---------------------------------------------------------------------------------------------------------------
# how far two correct implementations may be apart, and the results in 64 bits
# ---------------------------------------------------------------------------------------------------------------
def tolerance(case):
    if case["dtype"] == "e4m3" and case["kind"] == "prefill":
        return {"rel": 0.03, "max": 0.99}  # the probabilities are rounded to e4m3
    if case["kind"] == "prefill" and case["data"] == "llm":
        return {"rel": 0.02, "max": 0.99}  # tiles on the line of the skip rule may go either way
    if case["kind"] == "decode_select":
        return {"rel": 0.01, "max": 0.4, "differ": 0.0}
    return {"rel": 0.01, "max": 0.4}


def _attend(q, k, v, group, mask_of, add_of=None):
    """q [S, Hq, D], k / v [T, Hkv, D] in 64 bits, one head at a time -> out [S, Hq, D], lse [Hq, S]."""
    outs, lses = [], []
    scale = q.shape[-1] ** -0.5
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // group].T
        if add_of is not None:
            s = s + add_of(h)
        s = s * scale
        m = mask_of(h)
        if m is not None:
            s = s.masked_fill(~m, float("-inf"))
        lse = torch.logsumexp(s, dim=-1)
        outs.append(torch.exp(s - lse[:, None]) @ v[:, h // group])
        lses.append(lse)
    return torch.stack(outs, dim=1), torch.stack(lses)


def _band(sq, sk, window):
    dist = torch.arange(sq, device=DEV)[:, None] + (sk - sq) - torch.arange(sk, device=DEV)[None, :]
    return (dist >= 0) if not window else (dist >= 0) & (dist < window)


def _grads(q, k, v, do, group, windows, alpha=None, delta=None):
    """Output and gradients of one sequence, head by head (a head's probabilities at a time)."""
    scale = q.shape[-1] ** -0.5
    o, dq, dk, dv = torch.empty_like(q), torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    da = torch.empty_like(alpha) if alpha is not None else None
    dd = torch.zeros_like(delta) if delta is not None else None
    masks = {}
    for h in range(q.shape[1]):
        n = h // group
        w = windows[n] if windows else 0
        if w not in masks:
            masks[w] = _band(q.shape[0], k.shape[0], w)
        s = q[:, h] @ k[:, n].T
        if alpha is not None:
            s += torch.nn.functional.logsigmoid(alpha[:, h, None] * delta[None, :, n])
        p = torch.softmax((s * scale).masked_fill_(~masks[w], float("-inf")), dim=-1)
        del s
        o[:, h] = p @ v[:, n]
        dv[:, n] += p.T @ do[:, h]
        ds = do[:, h] @ v[:, n].T
        ds = p.mul_(ds - (do[:, h] * o[:, h]).sum(-1, keepdim=True)).mul_(scale)
        dq[:, h] = ds @ k[:, n]
        dk[:, n] += ds.T @ q[:, h]
        if alpha is not None:
            ds = ds * torch.sigmoid(-alpha[:, h, None] * delta[None, :, n])
            da[:, h] = ds @ delta[:, n]
            dd[:, n] += ds.T @ alpha[:, h]
    return (o, dq, dk, dv) if alpha is None else (o, dq, dk, dv, da, dd)


def exact(case, seed):
    st = prepare(case, seed)
    kind, hq, hkv = case["kind"], case["hq"], case["hkv"]
    group = hq // hkv
    unscale = 1.0 / 64 if case["dtype"] == "e4m3" else 1.0

    def wide(t):
        return (t.detach().float() if t.dtype == torch.float8_e4m3fn else t.detach()).double() * unscale

    if kind.startswith("decode") or kind == "prefill_chunk":
        outs, lses = [], []
        idx = st.get("idx")
        if kind == "decode_select":
            idx = st["score"].topk(case["topk"], dim=-1).indices.sort(dim=-1).values.to(torch.int32)
        for b in range(case["batch"]):
            if kind == "decode":
                k, v = st["k"][b], st["v"][b]
            else:
                pos = idx[b].long() if idx is not None else torch.arange(int(st["used"][b]), device=DEV)
                row = st["table"][b].long()[pos // case["page"]] * case["page"] + pos % case["page"]
                # (bytes: indexing is not there for every FP8 type)
                k, v = (t.view(-1, hkv, case["d"]).view(torch.uint8)[row].view(t.dtype) for t in (st["k"], st["v"]))
            q = st["q"][b] if kind == "prefill_chunk" else st["q"][b:b + 1]
            ok = _band(q.shape[0], k.shape[0], 0) if kind == "prefill_chunk" else None
            o, lse = _attend(wide(q), wide(k), wide(v), group, lambda h: ok)
            outs.append(o if kind == "prefill_chunk" else o[0])
            lses.append(lse)
        if kind == "prefill_chunk":
            return torch.stack(outs), torch.stack(lses)
        return (torch.stack(outs), None) if kind == "decode_select" else torch.stack(outs)
    if kind == "prefill":
        # without skipping: what it leaves out at the default threshold is part of the operator's own error
        ok = _band(case["seqlen"], case["seqlen"], 0)
        return torch.stack([_attend(wide(st["q"][b]), wide(st["k"][b]), wide(st["v"][b]), group, lambda h: ok)[0]
                            for b in range(case["batch"])])
    names = ("q", "k", "v", "dout") + (("alpha", "delta") if kind == "train_gated" else ())
    if kind == "train_packed":
        at, parts = 0, []
        for n in st["lens"]:
            q, k, v, do = (wide(st[x][at:at + n]) for x in names)
            parts.append(_grads(q, k, v, do, group, None))
            at += n
        return tuple(torch.cat(x) for x in zip(*parts))
    w = _windows(case)
    parts = []
    for b in range(case["batch"]):
        q, k, v, do, *gate = (wide(st[x][b]) for x in names)
        parts.append(_grads(q, k, v, do, group, w, *gate))
    return tuple(torch.stack(x) for x in zip(*parts))
