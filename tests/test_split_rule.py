"""The rule that picks the number of KV / QO splits when the caller leaves it open, and the merge of many splits."""

import pytest
import torch

from fixtures import assert_close, seeded_qkv
from flash_sparse_attn.ops.triton import utils
from flash_sparse_attn.ops.triton.flash_bwd import backward_num_splits
from oracle import eager


def test_balanced_num_splits():
    f = lambda ctas, steps: utils.balanced_num_splits(ctas, steps, 1.5, 7.0, 0.5, 148)  # noqa: E731
    assert f(256, 1) == 1 and f(1, 0) == 1
    assert utils.balanced_num_splits(290, 94, 1.5, 7.0, 50.0, 148) == 1  # the partials would cost more
    assert f(4, 120) > 4                       # four CTAs would leave the GPU idle
    # unequal sequences: fewer CTAs than SMs whose steps last long are split (three sequences of 300 queries against up to
    # 12000 keys, 16 heads of 64: 207 us with one split, 132 us with three)
    assert utils.balanced_num_splits(96, 94, 1.5, 7.0, 1.5, 148) > 1
    # nearly two CTAs per SM are not (1000 queries against 16000 keys, 64 heads: 668 us, 709 us with two splits)
    assert utils.balanced_num_splits(256, 126, 1.5, 7.0, 13.1, 148) == 1
    for ctas in (1, 8, 100, 147, 149, 295):
        for steps in (1, 2, 7, 64, 1000):
            n = f(ctas, steps)
            assert 1 <= n <= min(max(steps, 1), 64)


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
