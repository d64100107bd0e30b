"""Calls that feed one another without a synchronisation in between: kernels are set up while those in front of them run, so each has
to wait for what it reads and for what still reads what it writes. Same bits as with a synchronisation after every call, on the
default stream, on a side stream, between kernels of torch, and from a captured graph."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(state, sync):
    """Selection, scales and FP8 decode, 16-bit decode in splits, prompt, forward and backward; every output is an input of the next."""
    import flash_sparse_attn as fsa
    from flash_sparse_attn.utils.mask import topk_indices

    def done():
        if sync:
            torch.cuda.synchronize()

    got = []
    q, k, v, score, one = (state[n] for n in ("q", "k", "v", "score", "one"))
    for _ in range(3):
        idx = topk_indices(score, 256, dtype=torch.int32)
        done()
        q8, k8, v8 = ((t * 16).to(torch.float8_e4m3fn) for t in (q[:, -1], k, v))
        dec = fsa.flash_sparse_attn_with_kvcache_func(q8, k8, v8, gather_kv_indices=idx, is_quant=True, query_scale=one, key_scale=one,
                                                      value_scale=one)
        done()
        dec = fsa.flash_dense_attn_with_kvcache_func(dec, k, v, num_splits=9)
        done()
        dec = fsa.flash_dense_attn_with_kvcache_func(dec, k, v, num_splits=3)
        done()
        q = q + dec[:, None]
        out = fsa.flash_dense_attn_func(q, k, v, is_causal=True)
        done()
        out = fsa.flash_sparse_attn_func(out, k, v, is_causal=True, is_split_kv=True, num_splits=2)
        done()
        gated = fsa.flash_gated_attn_func(out, k, v, out[..., 0], k[..., 0], is_causal=True)
        done()
        q = (out + gated) * 0.5
        score = score + q[:, :1, 0, :1].float().flatten(1)
        got += [idx, dec, out, gated]
    return got


def _state():
    g = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    return dict(q=mk(2, 1000, 4, 128), k=mk(2, 1000, 2, 128), v=mk(2, 1000, 2, 128), score=mk(2, 1000).float(),
                one=torch.full((1,), 1 / 16, device="cuda"))


def test_chain_equals_its_calls():
    import flash_sparse_attn as fsa

    state = _state()
    want = _chain(state, True)
    for _ in range(5):
        for a, b in zip(_chain(state, False), want):
            assert torch.equal(a, b)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = _chain(state, False)
    torch.cuda.current_stream().wait_stream(side)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = _chain(state, False)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    fsa.check_status()


def test_two_streams_that_join():
    """Chains on two streams at a time, and a call that reads what both wrote: eagerly and from one captured graph."""
    import flash_sparse_attn as fsa

    state = _state()
    other = {n: t.flip(0).contiguous() for n, t in state.items()}
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]

    def both(sync):
        here = torch.cuda.current_stream()
        got = []
        for s, x in zip(streams, (state, other)):
            s.wait_stream(here)
            with torch.cuda.stream(s):
                got.append(_chain(x, sync))
        for s in streams:
            here.wait_stream(s)
        out = fsa.flash_dense_attn_func(got[0][-2], got[1][-1], got[0][-1], is_causal=True)
        return got[0] + got[1] + [fsa.flash_dense_attn_with_kvcache_func(out[:, -1], got[1][-2], got[0][-2], num_splits=3)]

    state["k"] = state["k"].repeat_interleave(2, 2)  # as many KV heads as query heads: results serve as keys and values
    state["v"], other["k"], other["v"] = (t.repeat_interleave(2, 2) for t in (state["v"], other["k"], other["v"]))
    want = both(True)
    torch.cuda.synchronize()
    for _ in range(3):
        got = both(False)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = both(False)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    fsa.check_status()


def test_backward_passes_in_a_row():
    import flash_sparse_attn as fsa

    s = _state()
    leaves = [s[n].clone().requires_grad_(True) for n in "qkv"]
    do = torch.randn_like(leaves[0])

    def grads(sync):
        got = []
        x = do
        for _ in range(3):
            out = fsa.flash_dense_attn_func(*leaves, is_causal=True, is_split_kv=True, is_split_qo=True, num_splits=2)
            if sync:
                torch.cuda.synchronize()
            got += torch.autograd.grad(out, leaves, x)
            if sync:
                torch.cuda.synchronize()
            x = got[-3] * 0.5  # the next pass starts from this one's dq
        return got

    fsa.set_deterministic(True)
    try:
        want = grads(True)
        for _ in range(3):
            for a, b in zip(grads(False), want):
                assert torch.equal(a, b)
    finally:
        fsa.set_deterministic(False)
    fsa.check_status()


def test_a_refused_launch_is_reported_once():
    # A launch into a capture that something else has spoilt is refused on the host. The call says so, and the next one, whose launch
    # asks for the last error, knows nothing of it.
    import ctypes

    from flash_sparse_attn import _lib
    from flash_sparse_attn.ops.triton import quant

    lib = _lib.load()
    rt = ctypes.CDLL("libcudart.so.12")  # torch's; the library has a runtime of its own
    x = torch.ones(64, device="cuda").to(torch.float8_e4m3fn)
    one, out = torch.ones(1, device="cuda"), torch.empty(3, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    stream = ctypes.c_void_p(side.cuda_stream)
    graph = ctypes.c_void_p()
    assert rt.cudaStreamBeginCapture(stream, 1) == 0  # 1: thread local
    try:
        assert rt.cudaStreamSynchronize(stream) != 0  # not allowed in a capture, which is spoilt by it
        rc = lib.fsa_pack_scales(one.data_ptr(), one.data_ptr(), one.data_ptr(), 4, out.data_ptr(), stream)  # 4: FSA_DT_F32
    finally:
        rt.cudaStreamEndCapture(stream, ctypes.byref(graph))
        rt.cudaGetLastError()
    assert rc == -3, rc  # FSA_ERR_LAUNCH
    assert torch.equal(quant.widen_fp8(x).float(), torch.ones(64, device="cuda"))
