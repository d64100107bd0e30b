"""Decode calls whose splits are merged inside a thread-block cluster (two to eight splits, as many clusters as are resident
at once) and through partials and the combine kernel, at the edges of that rule and for every form, against the eager oracle."""

import pytest
import torch

from fixtures import assert_close
from oracle import eager

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("num_splits", [1, 2, 3, 7, 8, 9])  # 9 goes through partials and the second launch
@pytest.mark.parametrize("hq,hkv,d", [(1, 1, 16), (8, 1, 64), (12, 3, 128), (16, 1, 128), (17, 1, 128), (16, 2, 256)])
def test_cluster_merge(num_splits, hq, hkv, d):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(num_splits + hq + d)
    mk = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    b, sk = 3, 333
    q, k, v = mk(b, hq, d), mk(b, sk, hkv, d), mk(b, sk, hkv, d)
    used = torch.tensor([333, 40, 1], dtype=torch.int32)  # splits without a key among them
    ref, lse_ref = eager.decode(q, k, v, seqused_k=used, return_lse=True)
    out, lse = fsa.flash_dense_attn_with_kvcache_func(q.cuda(), k.cuda(), v.cuda(), seqused_k=used.cuda(),
                                                      num_splits=num_splits, return_lse=True)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)
    assert torch.allclose(lse.cpu(), lse_ref, rtol=0, atol=2e-3)
    used[1] = 0  # no key at all: zeros and -inf
    out, lse = fsa.flash_dense_attn_with_kvcache_func(q.cuda(), k.cuda(), v.cuda(), seqused_k=used.cuda(),
                                                      num_splits=num_splits, return_lse=True)
    assert (out[1] == 0).all() and torch.isneginf(lse[1]).all()


@pytest.mark.parametrize("num_splits", [1, 2, 8, 9])  # unsplit, cluster merge, partials and combine
@pytest.mark.parametrize("hq,d", [(4, 64), (12, 128)])
def test_rows_of_out_on_4_byte_boundaries(num_splits, hq, d):
    import flash_sparse_attn as fsa

    g = torch.Generator().manual_seed(hq)
    q, k, v = (torch.randn(*s, generator=g).to(torch.bfloat16).cuda() for s in ((3, hq, d), (3, 333, 1, d), (3, 333, 1, d)))
    buf = torch.full((3, hq, d + 2), 7.0, dtype=torch.bfloat16, device="cuda")
    want = fsa.flash_dense_attn_with_kvcache_func(q, k, v, num_splits=num_splits)
    out = buf[..., 2:]
    assert out.data_ptr() % 8 == 4 and out.stride(1) % 4 == 2
    fsa.flash_dense_attn_with_kvcache_func(q, k, v, num_splits=num_splits, out=out)
    assert torch.equal(out, want) and (buf[..., :2] == 7).all()


def _graph_nodes(fn):
    """Kernels that one call launches: the nodes of a CUDA graph that captured it."""
    import ctypes

    fn()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    count = ctypes.c_size_t(0)
    runtime = ctypes.CDLL("libcudart.so.12")
    assert runtime.cudaGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(count)) == 0
    return count.value


# (sequences x KV heads, splits): 42 clusters of 7 and 49 of 6 would need all but two of the 296 slots that 148 SMs have for
# two CTAs each, and 18 of 8 or 21 of 7 nearly every SM; GPCs, inside which a cluster has to fit, are not of such sizes
@pytest.mark.parametrize("pairs,splits,launches", [(4, 8, 1), (42, 7, 2), (49, 6, 2), (18, 8, 2), (21, 7, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
def test_clusters_only_where_they_are_resident(dtype, pairs, splits, launches):
    import flash_sparse_attn as fsa

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the numbers are those of 148 SMs")
    g = torch.Generator().manual_seed(pairs)
    q, k, v = (torch.randn(*s, generator=g).to(torch.bfloat16) for s in ((pairs, 4, 128), (pairs, 200, 1, 128), (pairs, 200, 1, 128)))
    ref = eager.decode(q, k, v)
    kw = {}
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    if dtype != torch.bfloat16:
        q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
        ref = eager.decode(*(t.cpu().to(torch.bfloat16) for t in (q, k, v)))
        one = torch.ones(1, device="cuda")
        kw = dict(is_quant=True, query_scale=one, key_scale=one, value_scale=one)
    out, lse = torch.empty(pairs, 4, 128, dtype=torch.bfloat16, device="cuda"), torch.empty(pairs, 4, device="cuda")
    call = lambda: fsa.flash_dense_attn_with_kvcache_func(q, k, v, num_splits=splits, out=out, lse=lse, **kw)  # noqa: E731
    assert _graph_nodes(call) == launches + (1 if kw else 0)  # FP8: one more packs the scales
    call()
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close("out", out, ref)


@pytest.mark.parametrize("num_splits", [2, 8, 9])
def test_partials_are_written_either_way(num_splits):
    """The split partials are a documented output of the library's decode call; a caller that brings the buffers may read them."""
    from flash_sparse_attn.ops.triton.flash_dec import attn_decode

    g = torch.Generator().manual_seed(num_splits)
    q, k, v = (torch.randn(*s, generator=g).to(torch.bfloat16).cuda() for s in ((2, 6, 96), (2, 150, 3, 96), (2, 150, 3, 96)))
    used = torch.tensor([150, 20], dtype=torch.int32, device="cuda")  # splits without a key among them
    want = attn_decode("dense", q, k, v, seqused_k=used, num_splits=num_splits, partial_only=True)
    got = tuple(torch.full_like(t, float("nan")) for t in want)
    attn_decode("dense", q, k, v, seqused_k=used, num_splits=num_splits, workspace=got)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("num_splits", [3, 9])  # cluster merge; partials and combine
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float8_e4m3fn])
@pytest.mark.parametrize("form", ["window", "paged", "gather", "paged gather", "varlen", "gated", "gated gather"])
def test_both_merges_of_every_form(form, dtype, num_splits):
    import flash_sparse_attn as fsa

    fp8 = dtype != torch.bfloat16
    g = torch.Generator().manual_seed(len(form) + num_splits)
    b, sk, hq, hkv, d, page = 2, 320, 6, 2, 128, 32
    mk = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    q, k, v, al, de = mk(b, hq, d), mk(b, sk, hkv, d), mk(b, sk, hkv, d), mk(b, hq), mk(b, sk, hkv)
    if fp8:  # scales of one: the oracle takes the rounded values
        q, k, v = (t.to(dtype).to(torch.bfloat16) for t in (q, k, v))
    put = lambda t: t.to(dtype).cuda()  # noqa: E731
    args, kw, opts = [put(q), put(k), put(v)], {}, {}
    fn = fsa.flash_sparse_attn_with_kvcache_func
    kw["softmax_threshold"] = -128.0  # nothing is skipped
    if form == "window":
        opts = dict(is_local=True, window_sizes=torch.tensor([[8, 60, 40, 90], [0, 100, 0, 33]], dtype=torch.int32))
        kw["window_sizes"] = opts["window_sizes"].cuda()
    if "paged" in form:
        table = torch.randperm(b * sk // page, generator=g).to(torch.int32)
        for i, t in ((1, k), (2, v)):
            pages = torch.empty(b * sk // page, page, hkv, d, dtype=torch.bfloat16)
            pages[table.long()] = t.reshape(pages.shape)
            args[i] = put(pages)
        kw["page_table"] = table.reshape(b, -1).cuda()
    gate = dict(alpha=al, delta=de) if "gated" in form else {}
    if gate:
        fn = fsa.flash_gated_attn_with_kvcache_func
        args += [al.cuda(), de.cuda()]
        kw["gate_threshold"] = -128.0
    if fp8:
        one = torch.ones(1, device="cuda")
        kw.update(is_quant=True, query_scale=one, key_scale=one, value_scale=one)
    if "gather" in form:
        idx = torch.stack([torch.randperm(sk, generator=g)[:200] for _ in range(b)]).to(torch.int32)
        idx[:, 3::11] = -1
        kw["gather_kv_indices"] = idx.cuda()
        ref = eager.gather_decode(q, k, v, idx, return_lse=True, **gate)
    elif form == "varlen":
        cu = torch.tensor([0, 300, 433], dtype=torch.int32)
        k, v = k.reshape(-1, hkv, d)[:433], v.reshape(-1, hkv, d)[:433]
        ref = eager.varlen_decode(q, k, v, cu, return_lse=True)
        fn, args = fsa.flash_sparse_attn_varlen_with_kvcache_func, [put(q), put(k), put(v), cu.cuda(), 300]
    else:
        ref = eager.decode(q, k, v, return_lse=True, **opts, **gate)
    out, lse = fn(*args, num_splits=num_splits, return_lse=True, **kw)
    torch.cuda.synchronize()
    fsa.check_status()
    assert_close(form, out, ref[0], rtol=2.5e-2, atol=2.5e-2)
    assert torch.allclose(lse.cpu(), ref[1], rtol=0, atol=2e-3)
