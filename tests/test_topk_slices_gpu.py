"""Top-k selection at the sizes where a row changes from one CTA to a cluster, where the cluster grows, and from registers to re-reading
its slice; one call set up while the one in front of it still runs."""

import numpy as np
import pytest
import torch

from oracle import topk as oracle_topk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 16, 19, 34, 75, 150])  # clusters of 8, 4, 4, 2, 1 and 1 at most on 148 SMs
@pytest.mark.parametrize("n", [4095, 8191, 8192, 8193, 16384, 16385, 32768, 32769, 70001])  # of 1, 1, 1, 2, 2, 4, 4, 8 and 8 at most
def test_slices(rows, n):
    from flash_sparse_attn.utils.mask import topk_indices

    g = torch.Generator().manual_seed(rows + n)
    x = torch.randn(rows, n, generator=g)
    x[:, n // 2:] = x[:, n // 2:].round(decimals=1)  # many equal scores in the second half
    x[rows // 2, : n // 3] = float("-inf")
    k = min(n, 1 + n // 5)
    ref = oracle_topk.topk_indices(x.numpy(), k)
    got = topk_indices(x.cuda(), k, dtype=torch.int32).cpu().numpy()
    assert np.array_equal(got, ref)


def test_calls_in_a_row():
    from flash_sparse_attn.utils.mask import topk_indices

    x = torch.randn(32, 20000, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()  # 128 CTAs, two of which an SM could hold
    want = topk_indices(x, 300)
    torch.cuda.synchronize()
    ref = oracle_topk.topk_indices(x.float().cpu().numpy(), 300)
    assert np.array_equal(want.cpu().numpy(), ref)
    assert all(torch.equal(topk_indices(x, 300), want) for _ in range(20))
