"""Decode calls whose splits are merged inside a thread-block cluster (all CTAs resident at once, two to eight splits), at
the edges of that rule, against the eager oracle."""

import pytest
import torch

from fixtures import assert_close
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_splits", [1, 2, 3, 7, 8, 9])  # 9 goes through partials and the second launch
@pytest.mark.parametrize("hq,hkv,d", [(1, 1, 16), (8, 1, 64), (12, 3, 128), (16, 1, 128), (17, 1, 128), (16, 2, 256)])
def test_cluster_merge(num_splits, hq, hkv, d):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(num_splits + hq + d)
    mk = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    b, sk = 3, 333
    q, k, v = mk(b, hq, d), mk(b, sk, hkv, d), mk(b, sk, hkv, d)
    used = torch.tensor([333, 40, 1], dtype=torch.int32)  # splits without a key among them
    ref, lse_ref = eager.decode(q, k, v, seqused_k=used, return_lse=True)
    out, lse = fsa.flash_dense_attn_with_kvcache_func(q.cuda(), k.cuda(), v.cuda(), seqused_k=used.cuda(),
                                                      num_splits=num_splits, return_lse=True)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)
    assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3)
    used[1] = 0  # no key at all: zeros and -inf
    out, lse = fsa.flash_dense_attn_with_kvcache_func(q.cuda(), k.cuda(), v.cuda(), seqused_k=used.cuda(),
                                                      num_splits=num_splits, return_lse=True)
    assert (out[1] == 0).all() and torch.isneginf(lse[1]).all()


@pytest.mark.parametrize("num_splits", [1, 2, 8, 9])  # unsplit, cluster merge, partials and combine
@pytest.mark.parametrize("hq,d", [(4, 64), (12, 128)])
def test_rows_of_out_on_4_byte_boundaries(num_splits, hq, d):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(hq)
    q, k, v = (torch.randn(*s, generator=g).to(torch.bfloat16).cuda() for s in ((3, hq, d), (3, 333, 1, d), (3, 333, 1, d)))
    buf = torch.full((3, hq, d + 2), 7.0, dtype=torch.bfloat16, device="cuda")
    want = fsa.flash_dense_attn_with_kvcache_func(q, k, v, num_splits=num_splits)
    out = buf[..., 2:]
    assert out.data_ptr() % 8 == 4 and out.stride(1) % 4 == 2
    fsa.flash_dense_attn_with_kvcache_func(q, k, v, num_splits=num_splits, out=out)
    assert torch.equal(out, want) and (buf[..., :2] == 7).all()
