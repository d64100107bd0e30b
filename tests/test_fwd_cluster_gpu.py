"""Dense calls of few CTAs, whose key tiles are shared by the CTAs of a cluster: at the sizes where the cluster grows (none, two, four,
eight CTAs on 148 SMs), with tiles that are not full, shares without a tile, and what keeps a call out of it. test_fwd_cluster_rule.py
says which size a form takes."""

import pytest
import torch

from fixtures import assert_close, seeded_qkv
from oracle import eager

pytestmark = pytest.mark.gpu


# causal, 2 query heads to a KV head: 700 tokens 3 pairs of query tiles a head over 6 key tiles, 1000: 4 over 8, 2050: 9 over 17
@pytest.mark.parametrize("seqlen, hq", [(641, 4), (700, 4), (1000, 2), (1000, 8), (1025, 2), (2050, 4), (2050, 8), (3000, 2)])
@pytest.mark.parametrize("head_dim", [48, 64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_shares_of_the_keys(seqlen, hq, head_dim, causal):
    import flash_sparse_attn as fsa

    q, k, v = seeded_qkv(seqlen + hq, 1, seqlen, seqlen, hq, hq // 2, head_dim)
    q = q * 3  # maxima that differ between the shares
    ref, lse_ref = eager.forward(q, k, v, None, causal, return_lse=True)
    out, lse = fsa.flash_dense_attn_func(*(t.cuda() for t in (q, k, v)), is_causal=causal, return_lse=True)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)
    assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3)


# by the rule: eight CTAs (9 and 12 pairs of query tiles over 17 and 24 key tiles), four where the batch is two, two at 16 heads
@pytest.mark.parametrize("batch, seqlen, hq, hkv, pack", [(1, 2050, 1, 1, False), (1, 3000, 1, 1, False), (2, 2050, 1, 1, False),
                                                          (2, 1000, 8, 2, False), (1, 1000, 4, 1, True), (1, 1300, 2, 1, True)])
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_clusters_of_eight_batches_and_packed_heads(batch, seqlen, hq, hkv, pack, head_dim, causal, dtype):
    import flash_sparse_attn as fsa

    q, k, v = seeded_qkv(seqlen + hq, batch, seqlen, seqlen, hq, hkv, head_dim, dtype)
    q = q * 3
    ref, lse_ref = eager.forward(q, k, v, None, causal, return_lse=True)
    out, lse = fsa.flash_dense_attn_func(*(t.cuda() for t in (q, k, v)), is_causal=causal, pack_gqa=pack, return_lse=True)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)
    assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3)


def test_packed_heads_infinite_keys_and_a_second_stream():
    import flash_sparse_attn as fsa

    q, k, v = (t.cuda() for t in seeded_qkv(7, 1, 1000, 1000, 8, 2, 64))
    k[0, 300:310] = float("inf")  # a share whose scores are not numbers makes the rows that see it so
    out = fsa.flash_dense_attn_func(q, k, v, is_causal=True)
    assert torch.isnan(out[0, 310:]).all() and torch.isfinite(out[0, :300]).all()
    k[0, 300:310] = 0
    ref = fsa.flash_dense_attn_func(q, k, v, is_causal=True)
    assert_close("packed", fsa.flash_dense_attn_func(q, k, v, is_causal=True, pack_gqa=True), ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = fsa.flash_dense_attn_func(q, k, v, is_causal=True)
    assert torch.equal(fsa.flash_dense_attn_func(q, k, v, is_causal=True), ref)  # the same bits on every run
    side.synchronize()
    assert torch.equal(other, ref)
    fsa.check_status()


# Key tiles that score -inf for every second row, and once for all rows (a product that overflows: masking by an extra column does
# that). 897 tokens x 8 heads: clusters of four, the next two of two, one head: of eight. Every CTA but the one of the last share begins
# with tiles that carry no mask
@pytest.mark.parametrize("seqlen, hq, hkv", [(897, 8, 2), (1024, 16, 4), (2304, 8, 2), (2050, 1, 1)])
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_shares_that_begin_at_minus_infinity(seqlen, hq, hkv, head_dim, causal):
    import flash_sparse_attn as fsa

    q, k, v = seeded_qkv(seqlen + head_dim, 1, seqlen, seqlen, hq, hkv, head_dim)
    tiles = seqlen // 128
    # one tile; two neighbours; the whole of the first share of two; all but the first and the last; every second one
    for out_tiles in ([3], [1, 2], range(1, tiles // 2), range(1, tiles), range(tiles - 1, 0, -2)):
        qq, kk = q.clone(), k.clone()
        qq[..., 5], kk[..., 5] = 0, 0
        qq[:, ::2, :, 5] = 1e20
        for t in out_tiles:
            kk[:, 128 * t:128 * (t + 1), :, 5] = -1e20
        ref, lse_ref = eager.forward(qq, kk, v, None, causal, return_lse=True)
        out, lse = fsa.flash_dense_attn_func(*(t.cuda() for t in (qq, kk, v)), is_causal=causal, return_lse=True)
        assert torch.isfinite(lse_ref).all()  # keys 0 to 127 are there for every row
        assert_close(f"out {list(out_tiles)}", out, ref)
        assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3), list(out_tiles)
    # no key is left to any row: probability zero for every one, as where everything is masked
    if causal:
        qq, kk = q.clone(), k.clone()
        qq[..., 5], kk[..., 5] = 1e20, -1e20
        out, lse = fsa.flash_dense_attn_func(*(t.cuda() for t in (qq, kk, v)), is_causal=True, return_lse=True)
        assert (out == 0).all() and torch.isneginf(lse).all()
    fsa.check_status()
