"""Forward over sequences of unequal length: the CTAs start in the order of their key tiles, worked out on the device. Which
CTA computes a tile changes nothing about its arithmetic, so a batch has to equal its sequences called one by one, bit for bit. That
holds for calls with lengths of their own, pages or keys in front of the queries at every size, and between those and dense calls over
whole sequences up to 896 tokens: from 897 on the latter may have their key tiles shared inside a cluster (fsa_fwd_cluster_size), each
share summed for itself, and equal the others up to the rounding of 16-bit probabilities."""

import pytest
import torch

import flash_sparse_attn as fsa

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _randn(*shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.bfloat16)


def _cu(lens):
    return torch.tensor([0] + list(lens), dtype=torch.int32).cumsum(0).to(torch.int32).to(DEV)


# (lengths, query heads, KV heads): packed self-attention, at both sides of every limit of the ranking; "ragged" is ranked without
# the causal mask. Ties, empty sequences and lengths at the edges of tiles
@pytest.mark.parametrize("lens, hq, hkv", [
    ([1, 700, 0, 256, 257, 511, 512, 30], 16, 4),
    ([300] * 9, 32, 8),
    ([128 + 7 * i for i in range(64)], 8, 2),
    ([129 + i for i in range(128)], 4, 2),
    ([129 + i for i in range(129)], 4, 2),
], ids=["ragged", "equal", "many", "limit", "past_limit"])
@pytest.mark.parametrize("causal", [True, False])
def test_packed_batch_equals_its_sequences(lens, hq, hkv, causal):
    total = sum(lens)
    q, k, v = _randn(total, hq, 64, seed=1), _randn(total, hkv, 64, seed=2), _randn(total, hkv, 64, seed=3)
    cu = _cu(lens)
    out = fsa.flash_dense_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), is_causal=causal)
    at = 0
    for n in lens:
        if n:
            s = slice(at, at + n)
            alone = fsa.flash_dense_attn_func(q[None, s], k[None, s], v[None, s], is_causal=causal)
            assert torch.equal(out[s], alone[0])
        at += n
    fsa.check_status()


# 896 tokens are the most that no cluster shares; 897, 1000 and 2000 at 8 / 2 heads are shared by four, four and two CTAs, but not
# when five of them are one dense batch
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_up_to_where_whole_sequences_have_the_bits_of_a_batch(head_dim, causal):
    lens, hq, hkv = [896, 897, 1000, 2000], 8, 2
    q, k, v = _randn(sum(lens), hq, head_dim, seed=1), _randn(sum(lens), hkv, head_dim, seed=2), _randn(sum(lens), hkv, head_dim, seed=3)
    packed = lambda s, n: fsa.flash_dense_attn_varlen_func(q[s], k[s], v[s], _cu(n), _cu(n), max(n), max(n), is_causal=causal)  # noqa: E731
    out = packed(slice(None), lens)
    at = 0
    for n in lens:
        s = slice(at, at + n)
        assert torch.equal(out[s], packed(s, [n]))  # packed: at every size
        alone = fsa.flash_dense_attn_func(q[None, s], k[None, s], v[None, s], is_causal=causal)[0]
        five = fsa.flash_dense_attn_func(*(t[None, s].repeat(5, 1, 1, 1) for t in (q, k, v)), is_causal=causal)
        assert all(torch.equal(five[i], out[s]) for i in range(5))
        if n <= 896:
            assert torch.equal(alone, out[s])
        # Each side rounds its probabilities and its results to bf16: four roundings of 2^-9 of a value at most, 2^-9 / sqrt(3) in the
        # root mean square, independent of one another and, as the values have random signs, over the keys: 2^-9 * sqrt(4 / 3) together.
        x, y = alone.double(), out[s].double()
        assert (x - y).norm() <= 2.0 ** -8 * y.norm()
        at += n
    fsa.check_status()


Q_LENS = [300, 17, 129, 256, 257, 1, 128, 200]
K_LENS = [600, 2000, 129, 1300, 700, 1999, 128, 1024]


# queries in front of whose own keys others lie, so the causal forms are ranked: every kind, the packed heads, the CTA of one query
# tile (head sizes above 128), and as many items as a CTA ranks
@pytest.mark.parametrize("form", ["dense", "sparse", "gated", "fp8", "pack_gqa", "sparse_wide", "gated_wide", "full", "most_items"])
def test_longer_keys_equal_single_calls(form):
    q_lens, k_lens, hq, hkv, d = Q_LENS, K_LENS, 16, 4, 64
    kw = dict(is_causal=form != "full")
    if form == "most_items":  # 128 sequences of one pair of query tiles each
        q_lens, k_lens, hq, hkv = [1 + 2 * i for i in range(128)], [1 + 2 * i + (i * 1237) % 3840 for i in range(127)] + [4096], 4, 2
    kind = "sparse" if form.startswith("sparse") else "gated" if form.startswith("gated") else "dense"
    if form.endswith("wide"):
        d = 192
    kw.update(dict(pack_gqa=True) if form == "pack_gqa" else {})
    q, k, v = _randn(sum(q_lens), hq, d, seed=1), _randn(sum(k_lens), hkv, d, seed=2), _randn(sum(k_lens), hkv, d, seed=3)
    if form == "fp8":
        d = 128
        q, k, v = ((_randn(sum(n), h, d, seed=i) * 64).to(torch.float8_e4m3fn)
                   for i, (n, h) in enumerate(((q_lens, hq), (k_lens, hkv), (k_lens, hkv))))
        scale = torch.full((1,), 1.0 / 64, device=DEV)
        kw.update(is_quant=True, query_scale=scale, key_scale=scale, value_scale=scale)
    gate = [_randn(sum(q_lens), hq, seed=4), _randn(sum(k_lens), hkv, seed=5)] if kind == "gated" else []
    batched, single = (getattr(fsa, f"flash_{kind}_attn_{x}") for x in ("varlen_func", "func"))
    out = batched(q, k, v, *gate, _cu(q_lens), _cu(k_lens), max(q_lens), max(k_lens), **kw)
    at_q = at_k = 0
    for nq, nk in zip(q_lens, k_lens):
        sq, sk = slice(at_q, at_q + nq), slice(at_k, at_k + nk)
        alone = single(q[None, sq], k[None, sk], v[None, sk], *([gate[0][None, sq], gate[1][None, sk]] if gate else []), **kw)
        assert torch.equal(out[sq], alone[0]), (nq, nk)
        at_q, at_k = at_q + nq, at_k + nk
    fsa.check_status()


def test_used_queries_equal_single_calls():
    hq, hkv, d, n = 16, 4, 128, len(Q_LENS)
    q, k, v = (_randn(n, length, h, d, seed=i) for i, (length, h) in enumerate(((300, hq), (2000, hkv), (2000, hkv))))
    used_q, used_k = (torch.tensor(x, dtype=torch.int32, device=DEV) for x in (Q_LENS, K_LENS))
    out = fsa.flash_dense_attn_varlen_func(q.flatten(0, 1), k.flatten(0, 1), v.flatten(0, 1), _cu([300] * n), _cu([2000] * n), 300,
                                           2000, is_causal=True, seqused_q=used_q, seqused_k=used_k).view(n, 300, hq, d)
    for b, (nq, nk) in enumerate(zip(Q_LENS, K_LENS)):
        alone = fsa.flash_dense_attn_func(q[b:b + 1, :nq], k[b:b + 1, :nk], v[b:b + 1, :nk], is_causal=True)
        assert torch.equal(out[b, :nq], alone[0]), (nq, nk)
    fsa.check_status()


@pytest.mark.parametrize("splits", [1, 3])
def test_chunks_over_cached_keys_equal_single_calls(splits):
    used = [130, 4000, 700, 2049, 128]
    chunk, page, hq, hkv = 300, 128, 32, 8
    per = [-(-n // page) for n in used]
    k, v = _randn(sum(per), page, hkv, 128, seed=4), _randn(sum(per), page, hkv, 128, seed=5)
    table = torch.zeros(len(used), max(per), dtype=torch.int32, device=DEV)
    at = 0
    for b, n in enumerate(per):
        table[b, :n] = torch.arange(at, at + n, device=DEV, dtype=torch.int32)
        at += n
    q = _randn(len(used), chunk, hq, 128, seed=6)
    lens = torch.tensor(used, dtype=torch.int32, device=DEV)
    kw = dict(is_causal=True, is_split_kv=splits > 1, num_splits=splits, return_lse=True)
    out, lse = fsa.flash_dense_attn_func(q, k, v, page_table=table, seqused_k=lens, **kw)
    for b in range(len(used)):
        o1, l1 = fsa.flash_dense_attn_func(q[b:b + 1], k, v, page_table=table[b:b + 1], seqused_k=lens[b:b + 1], **kw)
        assert torch.equal(out[b], o1[0]) and torch.equal(lse[b], l1[0])
    fsa.check_status()
