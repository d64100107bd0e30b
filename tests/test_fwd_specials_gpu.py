"""Forward: rows without any key, logits far apart, NaN keys."""

import pytest
import torch

from fixtures import assert_close, seeded_qkv
from oracle import eager

pytestmark = pytest.mark.gpu


def _run(q, k, v, **kw):
    import flash_sparse_attn as fsa

    out, lse = fsa.flash_dense_attn_func(q.cuda(), k.cuda(), v.cuda(), return_lse=True, **kw)
    torch.cuda.synchronize()
    fsa.check_status()
    return out.float().cpu(), lse.cpu()


@pytest.mark.parametrize("d", [64, 128, 256])
def test_rows_without_keys(d):
    # more queries than keys under a causal mask: the first rows see nothing
    q, k, v = seeded_qkv(3, 1, 400, 250, 2, 1, d)
    out, lse = _run(q, k, v, is_causal=True)
    assert (out[:, :150] == 0).all() and torch.isneginf(lse[:, :, :150]).all()
    ref = eager.forward(q, k, v, None, True)
    assert_close("out", out, ref)


@pytest.mark.parametrize("scale", [1e-3, 1.0, 30.0])
def test_logits_far_apart(scale):
    # probabilities from one to far below the smallest normal number; the log-sum-exp carries fp32 error only
    q, k, v = seeded_qkv(5, 1, 300, 700, 2, 1, 128)
    out, lse = _run(q, k, v, softmax_scale=scale)
    s = torch.einsum("bqhd,bkd->bhqk", q.double(), k[:, :, 0].double()) * scale
    want = torch.logsumexp(s, -1)
    # base-2 logits of size m carry an error of m * 2^-23, the sum of 700 terms 700 * 2^-22 at most
    bound = 2e-4 + want.abs().max().item() * 2.0 ** -21
    assert (lse.double() - want).abs().max().item() < bound
    p = torch.softmax(s, -1)
    ref = torch.einsum("bhqk,bkd->bqhd", p, v[:, :, 0].double())
    assert (out.double() - ref).norm() / ref.norm() < 1e-2


def test_nan_keys():
    q, k, v = seeded_qkv(7, 1, 512, 512, 2, 1, 128)
    for col in (0, 3, 130, 131, 383):  # first, inner and last columns of key tiles
        kk = k.clone()
        kk[0, col] = float("nan")
        out, lse = _run(q, kk, v, is_causal=True)
        assert torch.isnan(out[0, col:]).all(), col
        assert not torch.isnan(out[0, :col]).any(), col


@pytest.mark.parametrize("op", ["dense", "sparse"])
def test_infinite_keys(op):
    # one infinite component in a key: rows whose query is negative there see it with probability zero, rows whose query is
    # positive have no finite softmax
    import flash_sparse_attn as fsa

    fn = fsa.flash_dense_attn_func if op == "dense" else fsa.flash_sparse_attn_func
    q, k, v = seeded_qkv(9, 1, 512, 512, 2, 1, 128)
    for col in (0, 130, 383):
        qq, kk = q.clone(), k.clone()
        qq[..., 5] = -q[..., 5].abs() - 0.5
        qq[:, col + 40, :, 5] = 0.5
        kk[0, col, 0, 5] = float("inf")
        out = fn(qq.cuda(), kk.cuda(), v.cuda(), is_causal=True).float().cpu()
        torch.cuda.synchronize()
        fsa.check_status()
        s = torch.einsum("bqhd,bkd->bhqk", qq.double(), kk[:, :, 0].double()) * 128 ** -0.5
        s = s.masked_fill(torch.ones(512, 512).triu(1).bool(), float("-inf"))
        ref = torch.einsum("bhqk,bkd->bqhd", torch.softmax(s, -1), v[:, :, 0].double())
        assert torch.isnan(out[0, col + 40]).all(), col
        rows = [i for i in range(512) if i != col + 40 and (i, col) != (0, 0)]  # row 0 has no other key than key 0
        assert_close(f"column {col}", out[:, rows], ref[:, rows].float())
