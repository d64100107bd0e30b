"""Top-k selection at the sizes where a row changes from one CTA to a cluster, and from registers to re-reading its slice."""

import numpy as np
import pytest
import torch

from oracle import topk as oracle_topk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 16, 19, 34, 75, 150])  # clusters of 8, 4, 4, 2, 1 and 1 on 148 SMs
@pytest.mark.parametrize("n", [4095, 4096, 8191, 8193, 16385, 70001])
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
