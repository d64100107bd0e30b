"""Decode: 64-wide rows on both sides of the deeper ring (thirty-two tiles of 16 keys a warp in one round of CTAs, sixteen in several)."""

import pytest
import torch

from fixtures import assert_close
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keys", [1025, 2032, 2048, 2049, 2500])  # 65, 127, 128, 129, 157 tiles for four warps
@pytest.mark.parametrize("kind", ["dense", "sparse", "gated"])
def test_deep_ring(keys, kind):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(keys)
    mk = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    q, k, v = mk(2, 6, 64), mk(2, keys, 2, 64), mk(2, keys, 2, 64)
    used = torch.tensor([keys, 17], dtype=torch.int32)
    gate = dict(alpha=mk(2, 6), delta=mk(2, keys, 2)) if kind == "gated" else {}
    kw = {} if kind == "dense" else dict(softmax_threshold=-128.0)
    if kind == "gated":
        kw["gate_threshold"] = -128.0
    ref = eager.decode(q, k, v, seqused_k=used, **gate)
    fn = getattr(fsa, f"flash_{kind}_attn_with_kvcache_func")
    out = fn(*(t.cuda() for t in (q, k, v)), *(t.cuda() for t in gate.values()), seqused_k=used.cuda(), num_splits=1, **kw)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)


# CTAs on 148 SMs, two KV heads: 370 take the deeper ring, 400, nearly three to an SM, do not; 460 do in rounds of two to an SM, 456 keys are too few
@pytest.mark.parametrize("batch, keys", [(185, 2100), (200, 2100), (230, 1040), (230, 456)])
def test_many_sequences(batch, keys):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(batch)
    q, k, v = (torch.randn(*s, 64, generator=g).to(torch.bfloat16) for s in ((batch, 4), (batch, keys, 2), (batch, keys, 2)))
    out = fsa.flash_dense_attn_with_kvcache_func(*(t.cuda() for t in (q, k, v)), num_splits=1)
    assert_close("out", out, eager.decode(q, k, v))
    fsa.check_status()
