"""Decode: 64-wide rows on both sides of the deeper ring (sixteen tiles of 16 keys a warp)."""

import pytest
import torch

from fixtures import assert_close
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keys", [1008, 1024, 1025, 1500])  # 63, 64, 65, 94 tiles for four warps
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
