"""Passes around the backward: a lane group takes two consecutive query rows of a head, so a pair may span two sequences or batches, and
the last one may be a single row."""

import itertools

import pytest
import torch

from fixtures import assert_close
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("heads", [1, 5])
@pytest.mark.parametrize("lens", [[1], [3, 3, 3], [1, 2, 127, 1, 64]], ids=str)
def test_pairs_of_rows(lens, heads, head_dim):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(sum(lens) + heads)
    q, k, v, do = (torch.randn(sum(lens), heads, head_dim, generator=g).to(torch.bfloat16) for _ in range(4))
    cu = torch.tensor([0] + list(itertools.accumulate(lens)), dtype=torch.int32)
    ref = eager.varlen_backward(q, k, v, do, cu, cu, None, True)
    dev = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    if len(set(lens)) == 1:
        shape = (len(lens), lens[0], heads, head_dim)
        out = fsa.flash_dense_attn_func(*(t.view(shape) for t in dev), is_causal=True).view(q.shape)
    else:
        out = fsa.flash_dense_attn_varlen_func(*dev, cu.cuda(), cu.cuda(), max(lens), max(lens), is_causal=True)
    got = torch.autograd.grad(out, dev, do.cuda())
    torch.cuda.synchronize()
    fsa.check_status()
    for name, a, b in zip(("dq", "dk", "dv"), got, ref):
        assert_close(name, a, b)


@pytest.mark.parametrize("batch", [4095, 4096])  # 16 380 and 16 384 blocks: the pass behind the main kernel starts early or after it
def test_many_blocks(batch):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(batch)
    q, k, v, do = (torch.randn(batch, 4, 32, 64, generator=g).to(torch.bfloat16) for _ in range(4))
    dev = [t.cuda().requires_grad_(True) for t in (q, k, v)]
    for _ in range(2):  # behind itself, too
        got = torch.autograd.grad(fsa.flash_dense_attn_func(*dev, is_causal=True), dev, do.cuda())
    torch.cuda.synchronize()
    fsa.check_status()
    # The extremes of 33 million elements. dS is rounded to 16 bits: its magnitudes in a row add up to 30 at most (a quarter of the spread
    # of dP, 60, above the mean and below it), |k| is below 5.7, the scale 1/8: 30 x 5.7 / 8 x 2^-9 = 0.042. The rounded output moves a
    # row's dpsum by up to 0.027 (five deviations of 64 products), which times 5.7 / 8 gives 0.019. Together 0.061.
    for name, a, b in zip(("dq", "dk", "dv"), got, eager.backward(q, k, v, do, None, True)):
        assert_close(name, a, b, ew_atol=6.1e-2)
