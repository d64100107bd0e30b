"""Forward over sequences of unequal length: the CTAs start in the order of their key tiles, worked out on the device. Which
CTA computes a tile changes nothing about its arithmetic, so a batch has to equal its sequences called one by one, bit for bit."""

import pytest
import torch

import flash_sparse_attn as fsa

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _randn(*shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.bfloat16)


# (lengths, query heads, KV heads): two to 128 items are ranked (a pair of 128-row query tiles of a sequence is an item), 129 are
# not; ties, empty sequences and lengths at the edges of tiles
@pytest.mark.parametrize("lens, hq, hkv", [
    ([1, 700, 0, 256, 257, 511, 512, 30], 16, 4),
    ([300] * 9, 32, 8),
    ([128 + 7 * i for i in range(64)], 8, 2),    # up to 569 rows: 3 pairs x 64, not ranked
    ([129 + i for i in range(128)], 4, 2),       # 1 pair x 128: the most that is ranked
    ([129 + i for i in range(129)], 4, 2),       # one more: not ranked
], ids=["ragged", "equal", "many", "limit", "past_limit"])
@pytest.mark.parametrize("causal", [True, False])
def test_packed_batch_equals_its_sequences(lens, hq, hkv, causal):
    total = sum(lens)
    q, k, v = _randn(total, hq, 64, seed=1), _randn(total, hkv, 64, seed=2), _randn(total, hkv, 64, seed=3)
    cu = torch.tensor([0] + lens, dtype=torch.int32).cumsum(0).to(torch.int32).to(DEV)
    out = fsa.flash_dense_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), is_causal=causal)
    at = 0
    for n in lens[:12]:
        if n:
            s = slice(at, at + n)
            alone = fsa.flash_dense_attn_func(q[None, s], k[None, s], v[None, s], is_causal=causal)
            assert torch.equal(out[s], alone[0])
        at += n
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
