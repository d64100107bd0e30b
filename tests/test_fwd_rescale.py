"""Rescaling of the forward's output when a row's maximum moves: right at every width of the loop over its columns."""

import pytest
import torch

from fixtures import assert_close, seeded_qkv
from oracle import eager

@pytest.mark.gpu
@pytest.mark.parametrize("head_dim", [64, 128, 192, 256])
@pytest.mark.parametrize("kind", ["dense", "sparse", "gated"])
def test_maxima_that_move_often(head_dim, kind):
    import flash_sparse_attn as fsa

    q, k, v = seeded_qkv(head_dim, 1, 300, 700, 4, 2, head_dim)
    q = q * 6  # in 16 bits a score is off by 2^-9 of itself, which the comparison shares: both sides start from these q, k, v
    kw, gate = {}, {}
    if kind != "dense":
        kw["softmax_threshold"] = -128.0  # nothing is skipped
    if kind == "gated":
        g = torch.Generator().manual_seed(1)
        gate = dict(alpha=torch.randn(1, 300, 4, generator=g).to(q.dtype), delta=torch.randn(1, 700, 2, generator=g).to(q.dtype))
        kw["gate_threshold"] = -128.0
    ref = eager.forward(q, k, v, None, False, **gate)
    fn = getattr(fsa, f"flash_{kind}_attn_func")
    out = fn(*(t.cuda() for t in (q, k, v)), *(t.cuda() for t in gate.values()), **kw)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close(f"{kind}-hd{head_dim}", out, ref)
