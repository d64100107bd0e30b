"""Decode of FP8 rows at the query heads per KV head where the products change sides (up to eight: keys on the M side)."""

import pytest
import torch

from fixtures import assert_close
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq", [1, 7, 8, 9, 16])  # query heads of the one KV head
@pytest.mark.parametrize("fp8", [torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("num_splits", [1, 3])
def test_fp8_rows(hq, fp8, num_splits):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(hq)
    q, k, v = ((torch.randn(*s, generator=g) * 4).to(fp8) for s in ((2, hq, 128), (2, 301, 1, 128), (2, 301, 1, 128)))
    scale = torch.tensor([0.25])
    ref = eager.decode(*((t.float() * 0.25).to(torch.bfloat16) for t in (q, k, v)))  # exact: a power of two
    out = fsa.flash_dense_attn_with_kvcache_func(*(t.cuda() for t in (q, k, v)), is_quant=True, num_splits=num_splits,
                                                 query_scale=scale.cuda(), key_scale=scale.cuda(), value_scale=scale.cuda())
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)
