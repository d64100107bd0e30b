"""Calls that no gradient is asked of go past the autograd Function, and only those; top-k positions and FP8 scales through the native
launcher equal those of the Python one."""

import pytest
import torch

DEV = "cuda"


def test_what_the_function_has_to_see():
    from flash_sparse_attn.ops.triton.interface import _nothing_to_record as plain

    x, leaf = torch.zeros(2), torch.zeros(2, requires_grad=True)
    assert plain(x, x, None) and not plain(x, leaf, None) and not plain(leaf * 2)
    assert not plain(torch.nn.Parameter(x)) and not plain(torch.nn.Parameter(x, requires_grad=False))
    with torch.no_grad():
        assert plain(x, leaf) and not plain(torch.nn.Parameter(x))
    with torch.autograd.forward_ad.dual_level():
        assert not plain(x)
    seen = []
    torch.func.vmap(lambda t: (seen.append(plain(t)), t)[1])(x)
    torch.func.grad(lambda t: (seen.append(plain(t)), t.sum())[1])(x)
    torch.jit.trace(lambda t: (seen.append(plain(t)), t + 1)[1], x, check_trace=False)
    assert seen == [False, False, False]


@pytest.mark.parametrize("asked", ["query", "key", "value", "query_scale", "key_scale", "value_scale", None])
def test_every_tensor_that_asks_for_a_gradient_is_recorded(asked, monkeypatch):
    from flash_sparse_attn.ops.triton import interface

    class Function:
        apply = staticmethod(lambda *a: "recorded")

    monkeypatch.setattr(interface, "_AttnFunc", Function)
    monkeypatch.setattr(interface, "_forward", lambda *a: ("not recorded",) * 13)
    one = {n: torch.ones(1) for n in ("query_scale", "key_scale", "value_scale")}
    x = {n: torch.zeros(1, 4, 1, 128) for n in ("query", "key", "value")}
    for t in (x, one):
        if asked in t:
            t[asked].requires_grad_(True)
    want = "not recorded" if asked is None else "recorded"
    assert interface.flash_dense_attn_func(**x, is_quant=True, **one) == want
    assert interface.flash_sparse_attn_func(**x, is_quant=True, **one) == want
    with torch.no_grad():
        assert interface.flash_dense_attn_func(**x, is_quant=True, **one) == "not recorded"


@pytest.mark.gpu
def test_same_results_and_refusals():
    import flash_sparse_attn as fsa
    from fixtures import seeded_qkv

    q, k, v = (t.to(DEV) for t in seeded_qkv(1, 2, 300, 300, 4, 2, 64))
    out, lse = fsa.flash_sparse_attn_func(q, k, v, is_causal=True, return_lse=True)
    leaf = q.clone().requires_grad_(True)
    with_graph = fsa.flash_sparse_attn_func(leaf, k, v, is_causal=True)
    assert torch.equal(out, with_graph) and with_graph.grad_fn is not None and out.grad_fn is None and not out.requires_grad
    with torch.no_grad():
        assert torch.equal(out, fsa.flash_sparse_attn_func(leaf, k, v, is_causal=True))
    buf = torch.empty_like(out)  # a caller's buffer comes back through the Function, as a view of its own
    assert fsa.flash_sparse_attn_func(q, k, v, is_causal=True, out=buf) is not buf and torch.equal(buf, out)
    alpha, delta = torch.randn(2, 300, 4, device=DEV, dtype=q.dtype), torch.randn(2, 300, 2, device=DEV, dtype=q.dtype)
    gated = fsa.flash_gated_attn_func(q, k, v, alpha, delta, is_causal=True)
    assert torch.equal(gated, fsa.flash_gated_attn_func(leaf, k, v, alpha, delta, is_causal=True))
    with pytest.raises(RuntimeError, match="vmap"):
        torch.func.vmap(lambda a: fsa.flash_sparse_attn_func(a, k, v))(q[None])
    with torch.autograd.forward_ad.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
        fsa.flash_sparse_attn_func(torch.autograd.forward_ad.make_dual(q, torch.ones_like(q)), k, v)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_native_topk_equals_the_python_launcher(dtype, monkeypatch):
    from flash_sparse_attn import _lib
    from flash_sparse_attn.utils.mask import topk_indices

    x = torch.randn(3, 4, 1000, device=DEV).to(dtype)
    forms = [x, x[0], x[0, 0], x[..., :900][0], x[:, :2], x.transpose(0, 1), x[0, ::2, :], x[..., ::2], x[:, :, None, :]]
    want = [topk_indices(t.contiguous(), 64, dtype=i) for t in forms for i in (torch.int32, torch.int64)]
    got = [topk_indices(t, 64, dtype=i) for t in forms for i in (torch.int32, torch.int64)]
    monkeypatch.setattr(_lib, "native", lambda: None)
    python = [topk_indices(t, 64, dtype=i) for t in forms for i in (torch.int32, torch.int64)]
    for a, b, c in zip(want, got, python):
        assert a.dtype == b.dtype == c.dtype and a.shape == b.shape == c.shape and torch.equal(a, b) and torch.equal(a, c)
    monkeypatch.undo()
    for bad in (0, 1001):
        with pytest.raises(AssertionError):
            topk_indices(x, bad)
    with pytest.raises((KeyError, AssertionError, RuntimeError, TypeError), match="int32"):
        topk_indices(torch.zeros(4, 10, dtype=torch.int32, device=DEV), 2)
    stored = torch.randn(2, 1000, device=DEV, requires_grad=True)
    assert not topk_indices(stored, 5).requires_grad


@pytest.mark.gpu
@pytest.mark.parametrize("scale_type", [torch.float32, torch.bfloat16, torch.float16])
def test_scales_packed_by_the_native_launcher(scale_type, monkeypatch):
    import flash_sparse_attn as fsa
    from flash_sparse_attn import _lib

    fp8 = torch.float8_e4m3fn
    q, k, v = ((torch.randn(2, 200, h, 128, device=DEV) * 4).to(fp8) for h in (4, 2, 2))
    kw = dict(is_quant=True, query_scale=torch.tensor([0.25], device=DEV, dtype=scale_type),
              key_scale=torch.tensor(0.5, device=DEV, dtype=scale_type), value_scale=torch.tensor([[2.0]], device=DEV, dtype=scale_type))
    calls = [lambda: fsa.flash_dense_attn_func(q, k, v, is_causal=True, **kw),
             lambda: fsa.flash_sparse_attn_with_kvcache_func(q[:, 0], k, v, **kw)]
    got = [c() for c in calls]
    monkeypatch.setattr(_lib, "native", lambda: None)
    for g, c in zip(got, calls):
        assert torch.equal(g, c())
    fsa.check_status()
