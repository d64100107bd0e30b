"""Gated forward: two threads share a row's key columns, 64 each, and their maxima and sums: key counts around the border between the
halves, rows whose largest score moves from one half to the other, both gates."""

import pytest
import torch

from fixtures import assert_close, seeded_qkv
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keys", [1, 63, 64, 65, 127, 128, 129, 193, 700])
@pytest.mark.parametrize("head_dim", [32, 64, 128])
@pytest.mark.parametrize("logsigmoid", [True, False])
def test_halves_of_a_row(keys, head_dim, logsigmoid):
    import flash_sparse_attn as fsa

    sq = min(keys, 300)
    q, k, v = seeded_qkv(keys + head_dim, 1, sq, keys, 4, 2, head_dim)
    k[:, keys // 2:] *= 3  # the maxima of later keys lie far above those of earlier ones, or far below
    g = torch.Generator().manual_seed(keys)
    alpha, delta = (torch.randn(1, n, h, generator=g).to(q.dtype) for n, h in ((sq, 4), (keys, 2)))
    for causal in (True, False):
        ref, lse_ref = eager.forward(q, k, v, None, causal, alpha=alpha, delta=delta, is_logsigmoid_gate=logsigmoid, return_lse=True)
        out, lse = fsa.flash_gated_attn_func(*(t.cuda() for t in (q, k, v, alpha, delta)), is_causal=causal, softmax_threshold=-128.0,
                                             gate_threshold=-128.0, is_logsigmoid_gate=logsigmoid, return_lse=True)
        torch.cuda.synchronize()
        fsa.check_status()
        assert_close(f"causal {causal}", out, ref)
        assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3)
