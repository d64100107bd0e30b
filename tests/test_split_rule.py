"""The rule that picks the number of KV / QO splits when the caller leaves it open, and the merge of many splits."""

import pytest
import torch

from fixtures import assert_close, seeded_qkv
from flash_sparse_attn.ops.triton import utils
from flash_sparse_attn.ops.triton.flash_bwd import backward_num_splits
from flash_sparse_attn.ops.triton.flash_fwd import forward_num_splits
from oracle import eager


def test_forward_num_splits():
    f = lambda b, sq, sk, hq, d=128, ragged=False, local=False: forward_num_splits(  # noqa: E731
        b, sq, sk, hq, max(hq // 4, 1), d, 1, local, ragged, 148)
    assert f(4, 500, 12000, 32, ragged=True) == 1   # 256 CTAs: two rounds already (37 splits: 1072 us, one: 365 us)
    assert f(3, 300, 12000, 16, 64, ragged=True) == 3   # 96 CTAs of unequal length (one split: 207 us, three: 132 us)
    assert f(2, 200, 12000, 32, ragged=True) == 4   # 143 us with two splits, 107 us with four
    assert f(1, 586, 6400, 16) == 3                 # 48 equal CTAs: one round (three splits 70 us, four 87 us)
    assert f(1, 1112, 1112, 16, 256) == 1           # one query tile a CTA: 144 of them (38 us, two splits 60 us)
    assert f(1, 100, 500, 2) == 1                   # four key tiles: never split
    assert f(4, 500, 12000, 32, ragged=True, local=True) == utils.num_splits_heuristic(500, 12000, 148, 128, 128, True, 8)
    assert f(0, 500, 12000, 32) >= 1                # an empty batch
    for sq in (1, 130, 2000):
        for sk in (1, 513, 4000, 16000):
            for ragged in (False, True):
                n = f(2, sq, sk, 8, ragged=ragged)
                assert 1 <= n <= utils.num_splits_heuristic(sq, sk, 148, 128, 128)


def test_backward_num_splits():
    f = lambda b, sq, sk, hq, hkv, d=128, kind="dense", causal=True, local=False: backward_num_splits(  # noqa: E731
        kind, b, sq, sk, b * sk, hq, hkv, d, causal, local, 148)
    assert f(2, 1318, 1318, 8, 8) == 1           # 176 CTAs: 80 us, eleven splits 233 us
    assert f(1, 3838, 3838, 32, 4, 64) >= 3    # 120 CTAs, the longest of 30 steps: 602 us, four splits 332 us
    assert f(2, 2933, 2933, 8, 2) >= 3        # 92 CTAs: 273 us, three splits 155 us
    assert f(1, 249, 249, 32, 8) == 1            # two query tiles: 84 us, two splits 101 us
    assert f(4, 8192, 8192, 32, 8) == 1
    assert f(0, 500, 500, 8, 2) == f(1, 500, 0, 8, 2) == 1
    assert f(1, 3838, 3838, 32, 4, local=True) == utils.num_splits_heuristic(3838, 3838, 148, 128, 128, True, 4)
    for sq in (1, 300, 5000):
        for sk in (1, 300, 5000):
            for causal in (True, False):
                assert 1 <= f(1, sq, sk, 8, 2, causal=causal) <= -(-sq // 128)


@pytest.mark.gpu
@pytest.mark.parametrize("num_splits", [None, 2, 33, 40])  # 32 splits are merged at a time
@pytest.mark.parametrize("sq,sk", [(70, 5300), (300, 900)])
def test_split_forward_and_backward(num_splits, sq, sk):
    import flash_sparse_attn as fsa

    q, k, v = seeded_qkv(sq + sk, 1, sq, sk, 4, 2, 64)
    ref, lse_ref = eager.forward(q, k, v, None, True, return_lse=True)
    dout = torch.randn(q.shape, generator=torch.Generator().manual_seed(1)).to(q.dtype)
    leaves = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    out, lse = fsa.flash_dense_attn_func(*leaves, is_causal=True, is_split_kv=True, is_split_qo=True,
                                         num_splits=num_splits, return_lse=True)
    grads = torch.autograd.grad(out, leaves, dout.cuda())
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)
    assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3)
    for name, got, want in zip(("dq", "dk", "dv"), grads, eager.backward(q, k, v, dout, None, True)):
        assert_close(name, got, want)
