"""The native launcher of the common calls against the Python launchers: the same results for every form it takes, and
None (the Python launcher runs, with its errors) for the others."""

import pytest
import torch

DEV = "cuda"


def test_decode_split_rule_is_the_same():
    from flash_sparse_attn import _lib
    from flash_sparse_attn.ops.triton.flash_dec import decode_num_splits

    _lib.load()
    for batch in (1, 2, 7, 64, 300):
        for hkv in (1, 2, 8, 40):
            for keys in (0, 1, 511, 512, 2048, 5000, 131072, 1 << 20):
                for sms in (1, 100, 148):
                    assert _lib._host.decode_num_splits(batch, hkv, keys, sms) == decode_num_splits(batch, hkv, keys, sms)


def test_refuses_what_is_not_on_a_gpu():
    from flash_sparse_attn import _lib

    _lib.load()
    q, k = torch.zeros(1, 4, 64, dtype=torch.bfloat16), torch.zeros(1, 8, 2, 64, dtype=torch.bfloat16)
    args = [0, q, k, k, None, None, None, False, None, None, None, None, None, None, None, None, None]
    assert _lib._host.decode(*args) is None  # not on a GPU
    assert _lib._host.decode(*args[:-1]) is None and _lib._host.forward() is None


@pytest.mark.parametrize("module", ["missing", "other abi", "other torch", "old", "fewer entry points"])
def test_package_works_without_it(monkeypatch, module):
    """A launcher that is missing or built for something else is left out, with one warning; the Python launchers remain."""
    import sys
    import types

    from flash_sparse_attn import _lib

    lib = _lib.load()
    good = _lib._host
    fake = None if module == "missing" else types.ModuleType("_host")
    if module.startswith("other"):
        fake.ABI_VERSION = good.ABI_VERSION + (module == "other abi")
        fake.TORCH_VERSION = good.TORCH_VERSION if module == "other abi" else "1.0.0"
    elif module == "fewer entry points":  # built before the launcher took the addresses of top-k and of the packing of scales
        def init(*addresses):
            if len(addresses) != 2:
                raise TypeError("init takes two addresses")

        fake.ABI_VERSION, fake.TORCH_VERSION, fake.init = good.ABI_VERSION, good.TORCH_VERSION, init
    monkeypatch.setitem(sys.modules, "flash_sparse_attn._host", fake)
    try:
        with pytest.warns(RuntimeWarning, match="Python launchers"):
            _lib._load_host(lib)
        assert _lib.native() is None and _lib.native() is None
    finally:
        monkeypatch.undo()
        _lib._load_host(lib)
    assert _lib.native() is good


def test_status_word_is_one_for_all_threads(monkeypatch):
    """Threads that make a device's first call at the same time share one status word: the native launcher keeps the one it is
    given first, and check_status reads the one in the table."""
    import threading
    import time

    from flash_sparse_attn import _lib

    _lib.load()
    zeros, seen = torch.zeros, []

    def slow_zeros(*a, **kw):
        t = zeros(*a, **kw)
        time.sleep(0.05)
        return t

    monkeypatch.setattr(torch, "zeros", slow_zeros)
    device = torch.device("cpu", 7)
    threads = [threading.Thread(target=lambda: seen.append(_lib.status_word(device))) for _ in range(4)]
    try:
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert len(seen) == 4 and all(t is seen[0] for t in seen) and _lib._status_words[("cpu", 7)] is seen[0]
    finally:
        _lib._status_words.pop(("cpu", 7), None)


def _both(monkeypatch, fn):
    """fn() through the native launcher (which must take the call) and through the Python one."""
    from flash_sparse_attn import _lib

    fn()  # registers the device
    taken = []
    host = _lib.native()

    class Spy:
        def __getattr__(self, name):
            f = getattr(host, name)

            def call(*a):
                r = f(*a)
                taken.append(r is not None)
                return r
            return call

    monkeypatch.setattr(_lib, "native", lambda: Spy())
    got = fn()
    assert taken and all(taken)
    monkeypatch.setattr(_lib, "native", lambda: None)
    want = fn()
    monkeypatch.undo()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride() and torch.equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float8_e4m3fn])
@pytest.mark.parametrize("form", ["plain", "strided", "paged", "gather", "paged_gather", "varlen", "window", "buffers"])
def test_decode_forms(monkeypatch, dtype, form):
    import flash_sparse_attn as fsa

    g = torch.Generator(device=DEV).manual_seed(1)
    f8 = dtype == torch.float8_e4m3fn
    mk = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    b, hq, hkv, d, sk = 3, 16, 4, 128, 1536
    q, kw = mk(b, hq, d), {}
    k, v = mk(b, sk, hkv, d), mk(b, sk, hkv, d)
    fn = fsa.flash_sparse_attn_with_kvcache_func
    if form == "strided":
        q, k, v = mk(hq, b, d).transpose(0, 1), mk(b, hkv, sk, d).transpose(1, 2), mk(b, hkv, sk, d).transpose(1, 2)
    if "paged" in form:
        k, v = mk(30, 64, hkv, d), mk(30, 64, hkv, d)
        kw.update(page_table=torch.randperm(30, generator=g, device=DEV).to(torch.int32).reshape(3, 10),
                  seqused_k=torch.tensor([600, 1, 77], dtype=torch.int32, device=DEV))
    if "gather" in form:
        kw.update(gather_kv_indices=torch.randint(-1, 600, (b, 100), generator=g, device=DEV, dtype=torch.int32))
    if form == "window":
        kw.update(window_sizes=torch.tensor([[4, 100, 30, 60]] * hkv, dtype=torch.int32, device=DEV), num_splits=3)
    if form == "buffers":
        kw.update(out=torch.empty(b, hq, d, device=DEV, dtype=torch.bfloat16 if f8 else dtype),
                  lse=torch.empty(b, hq, device=DEV))
    if f8:
        s = torch.full((1,), 0.5, device=DEV, dtype=torch.bfloat16)
        kw.update(is_quant=True, query_scale=s, key_scale=s, value_scale=s)
    if form == "varlen":
        cu = torch.tensor([0, 700, 700, 1500], dtype=torch.int32, device=DEV)
        k, v = mk(1500, hkv, d), mk(1500, hkv, d)
        fn = lambda q, k, v, **a: fsa.flash_sparse_attn_varlen_with_kvcache_func(q, k, v, cu, 800, **a)  # noqa: E731
    _both(monkeypatch, lambda: tuple(t.clone() for t in fn(q, k, v, return_lse=True, **kw)))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float8_e4m3fn])
@pytest.mark.parametrize("form", ["plain", "pack", "split", "paged", "varlen", "varlen_used", "window", "local", "buffers"])
def test_forward_forms(monkeypatch, dtype, form):
    import flash_sparse_attn as fsa

    g = torch.Generator(device=DEV).manual_seed(2)
    f8 = dtype == torch.float8_e4m3fn
    mk = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    b, s, hq, hkv, d = 2, 333, 8, 2, 128
    q, k, v, kw = mk(b, s, hq, d), mk(b, s, hkv, d), mk(b, s, hkv, d), dict(is_causal=True)
    fn = fsa.flash_sparse_attn_func
    if form == "pack":
        kw.update(pack_gqa=True)
    if form == "split":
        kw.update(num_splits=3)
    if form == "paged":
        k, v = mk(8, 128, hkv, d), mk(8, 128, hkv, d)
        kw.update(page_table=torch.randperm(8, generator=g, device=DEV).to(torch.int32).reshape(2, 4),
                  seqused_k=torch.tensor([400, 350], dtype=torch.int32, device=DEV), is_split_kv=True)
    if form == "window":
        kw.update(window_sizes=torch.tensor([[4, 100, 30, 60]] * hkv, dtype=torch.int32, device=DEV))
    if form == "local":
        kw.update(is_local=True)
    if form == "buffers":
        kw.update(out=torch.empty(b, s, hq, d, device=DEV, dtype=torch.bfloat16 if f8 else dtype),
                  lse=torch.empty(b, hq, s, device=DEV))
    if f8:
        sc = torch.full((1,), 0.5, device=DEV)
        kw.update(is_quant=True, query_scale=sc, key_scale=sc, value_scale=sc)
    if "varlen" in form:
        cu = torch.tensor([0, 200, 200, 500], dtype=torch.int32, device=DEV)
        q, k, v = mk(500, hq, d), mk(500, hkv, d), mk(500, hkv, d)
        if form == "varlen_used":
            kw.update(seqused_k=torch.tensor([150, 0, 300], dtype=torch.int32, device=DEV))
        fn = lambda q, k, v, **a: fsa.flash_sparse_attn_varlen_func(q, k, v, cu, cu, 300, 300, **a)  # noqa: E731
    _both(monkeypatch, lambda: tuple(t.clone() for t in fn(q, k, v, return_lse=True, **kw)))


@pytest.mark.gpu
def test_refuses_one_wrong_argument():
    """Calls that it takes, and the same ones with one argument replaced, which it leaves to the Python launcher."""
    import flash_sparse_attn as fsa
    from flash_sparse_attn import _lib

    bf = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device=DEV)  # noqa: E731
    i32 = lambda *s: torch.zeros(*s, dtype=torch.int32, device=DEV)  # noqa: E731
    q, k = bf(2, 4, 64), bf(2, 32, 2, 64)
    fsa.flash_dense_attn_with_kvcache_func(q, k, k)  # registers the device
    host = _lib._host

    def check(fn, base, wrong):
        assert type(fn(*base)) is tuple, "the base call is not taken"
        for i, bads in wrong.items():
            for bad in bads:
                assert fn(*(base[:i] + [bad] + base[i + 1:])) is None, (i, bad if not torch.is_tensor(bad) else bad.shape)
        assert fn(*base[:-1]) is None
        torch.cuda.synchronize()

    ints = lambda *s: [i32(*s).long(), i32(*s).cpu(), i32(*s).float(), "x"]  # noqa: E731  (wrong type, device, kind)
    window = torch.tensor([[0, 16, 0, 8]] * 2, dtype=torch.int32, device=DEV)
    out_wrong = lambda *s: [bf(*s).half(), bf(*s).cpu(), bf(*s[:-1], 32), bf(*s[:-1], 128)[..., ::2], "x"]  # noqa: E731
    lse_wrong = lambda *s: [bf(*s), torch.zeros(*s), torch.zeros(*s, 1, device=DEV), "x"]  # noqa: E731
    q_wrong = [None, "q", q.cpu(), q.half(), q.float(), bf(2, 3, 64), bf(2, 4, 72), bf(2, 4, 128)[..., ::2], bf(8, 64)]
    k_wrong = [None, k.half(), bf(3, 32, 2, 64), bf(2, 32, 2, 128)[..., ::2], bf(2, 2, 32, 64).transpose(1, 2), bf(64, 2, 64)]
    # kind, q, k, v, scale, windows, threshold, local, splits, table, gather, used, cu, max_k, out, lse, fp8 scales
    base = [0, q, k, k, None, None, None, False, None, None, None, None, None, None, None, None, None]
    check(host.decode, base, {0: [1.5, None], 1: q_wrong, 2: k_wrong, 4: ["1", [1.0]], 5: [window], 6: ["1"], 7: [1, True],
                              8: ["two", -1, 1 << 40, 2.0], 10: ints(2, 5) + [i32(3, 5), i32(5), i32(2, 10)[:, ::2]],
                              11: ints(2) + [i32(1), i32(2, 1)], 12: [i32(3)], 14: out_wrong(2, 4, 64),
                              15: lse_wrong(2, 4), 16: [torch.ones(3, device=DEV)]})
    local = base[:5] + [window, None, True] + base[8:]
    check(host.decode, local, {5: [None, window.long(), window.cpu(), window[:1], i32(2, 3), i32(8)], 7: [False]})
    paged = base[:2] + [k, k] + base[4:9] + [i32(2, 1)] + base[10:]
    check(host.decode, paged, {9: ints(2, 1) + [i32(3, 1), i32(2)], 12: [i32(3)]})
    packed = [0, q, bf(64, 2, 64), bf(64, 2, 64)] + base[4:12] + [i32(3), 32] + base[14:]
    check(host.decode, packed, {9: [i32(2, 1)], 12: ints(3) + [i32(2), None], 13: [None, "x", -1, 1.0]})

    q, k = bf(2, 32, 4, 64), bf(2, 32, 2, 64)
    q_wrong = [None, q.cpu(), q.half(), bf(2, 32, 3, 64), bf(2, 32, 4, 128)[..., ::2], bf(2, 4, 32, 64).transpose(1, 2)]
    # kind, q, k, v, causal, scale, windows, threshold, local, splits, pack, cu_q, cu_k, max_q, max_k, table, used_q, used_k, out,
    # lse, fp8 scales
    base = [0, q, k, k, True, None, None, None, False, 1, False, None, None, None, None, None, None, None, None, None, None]
    check(host.forward, base, {0: [1.5], 1: q_wrong, 2: k_wrong, 4: [1], 5: ["1"], 6: [window], 7: ["1"], 8: [True, 0],
                               9: [0, -1, None, 2.0], 10: [1], 11: [i32(3)], 12: [i32(3)], 16: ints(2) + [i32(1)],
                               17: ints(2) + [i32(1)], 18: out_wrong(2, 32, 4, 64), 19: lse_wrong(2, 4, 32),
                               20: [torch.ones(3, device=DEV)]})
    packed = [0, bf(64, 4, 64), bf(64, 2, 64), bf(64, 2, 64)] + base[4:9] + [2] + base[10:11] + [i32(3), i32(3), 32, 32] + base[15:]
    check(host.forward, packed, {11: ints(3) + [None, i32(2)], 12: ints(3) + [None, i32(2)], 13: [None, -1, 1.0], 14: [None, "x"],
                                 15: [i32(2, 1)], 16: [i32(2)]})  # used_q with splits: its partials want a fill


@pytest.mark.gpu
def test_unused_query_rows_with_splits():
    """The declined form: packed sequences of which only some query rows are used, over KV splits."""
    import flash_sparse_attn as fsa
    from fixtures import assert_close
    from oracle import eager

    g = torch.Generator().manual_seed(4)
    mk = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16)  # noqa: E731
    q, k, v = mk(400, 4, 64), mk(1500, 2, 64), mk(1500, 2, 64)
    cu_q, cu_k = torch.tensor([0, 150, 400], dtype=torch.int32), torch.tensor([0, 900, 1500], dtype=torch.int32)
    used = torch.tensor([100, 250], dtype=torch.int32)
    out, lse = fsa.flash_dense_attn_varlen_func(q.to(DEV), k.to(DEV), v.to(DEV), cu_q.to(DEV), cu_k.to(DEV), 250, 900,
                                                is_split_kv=True, num_splits=3, seqused_q=used.to(DEV), return_lse=True)
    for s in range(2):
        rows, keys = slice(cu_q[s], cu_q[s] + used[s]), slice(cu_k[s], cu_k[s + 1])
        ref = eager.forward(q[None, rows], k[None, keys], v[None, keys], None, False)
        assert_close(f"sequence {s}", out[None, rows], ref)
    assert torch.isneginf(lse[:, 100:150]).all()  # rows that are not used


@pytest.mark.gpu
def test_threads_and_streams():
    """Two threads, each with its own stream and inputs, get what one thread gets."""
    import threading

    import flash_sparse_attn as fsa

    g = torch.Generator(device=DEV).manual_seed(6)
    mk = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    jobs = [(mk(2, 8, 64), mk(2, 700, 2, 64), mk(1, 300, 8, 64), mk(1, 300, 2, 64)) for _ in range(2)]

    def run(job):
        q, k, qf, kf = job
        return (fsa.flash_dense_attn_with_kvcache_func(q, k, k, num_splits=9),
                fsa.flash_sparse_attn_func(qf, kf, kf, is_causal=True, is_split_kv=True, num_splits=2))

    want = [run(j) for j in jobs]
    torch.cuda.synchronize()
    got = [None, None]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got[i] = run(jobs[i])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, want):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.gpu
def test_errors_are_those_of_the_contract():
    import flash_sparse_attn as fsa

    q, k = (torch.zeros(1, *s, 64, dtype=torch.bfloat16, device=DEV) for s in ((4,), (8, 2)))
    fsa.flash_dense_attn_with_kvcache_func(q, k, k)
    with pytest.raises(AssertionError, match="same dtype"):
        fsa.flash_dense_attn_with_kvcache_func(q, k.half(), k.half())
    with pytest.raises(AssertionError, match="multiple of 16"):
        fsa.flash_dense_attn_with_kvcache_func(q[..., :40], k[..., :40], k[..., :40])
    with pytest.raises(AssertionError, match="int32"):
        fsa.flash_dense_attn_with_kvcache_func(q, k, k, seqused_k=torch.ones(1, dtype=torch.int64, device=DEV))
    with pytest.raises(RuntimeError):
        fsa.flash_dense_attn_with_kvcache_func(q.cpu(), k.cpu(), k.cpu())


@pytest.mark.gpu
def test_out_of_memory_keeps_its_type(monkeypatch):
    # a workspace of terabytes: the allocation is refused by the allocator, on either route with the class callers catch
    import flash_sparse_attn as fsa
    from flash_sparse_attn import _lib

    q, k = (torch.zeros(1, *s, 64, dtype=torch.bfloat16, device=DEV) for s in ((64,), (8, 2)))
    calls = [lambda n: fsa.flash_dense_attn_with_kvcache_func(q, k, k, num_splits=n),
             lambda n: fsa.flash_dense_attn_func(q[:, None], k, k, is_split_kv=True, num_splits=n)]
    for call in calls:
        call(2)
        with pytest.raises(torch.OutOfMemoryError):
            call(1 << 30)
    monkeypatch.setattr(_lib, "native", lambda: None)
    for call in calls:
        with pytest.raises(torch.OutOfMemoryError):
            call(1 << 30)


@pytest.mark.gpu
def test_gil_is_free_during_the_launch():
    # the library calls are replaced by CPython's own "does this thread hold the GIL": 0 reads as success, 1 as an error
    import ctypes

    import flash_sparse_attn as fsa
    from flash_sparse_attn import _lib

    q, k = (torch.zeros(1, *s, 64, dtype=torch.bfloat16, device=DEV) for s in ((4,), (8, 2)))
    fsa.flash_dense_attn_with_kvcache_func(q, k, k)  # registers the device
    host, lib = _lib._host, _lib.load()
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value  # noqa: E731
    host.init(address(ctypes.pythonapi.PyGILState_Check), address(ctypes.pythonapi.PyGILState_Check))
    try:
        dec = host.decode(0, q, k, k, None, None, None, False, 2, None, None, None, None, None, None, None, None)
        fwd = host.forward(0, q[:, None], k, k, False, None, None, None, False, 2, False, None, None, None, None, None, None,
                           None, None, None, None)
    finally:
        host.init(address(lib.fsa_decode), address(lib.fsa_fwd))
    assert type(dec) is tuple and type(fwd) is tuple


@pytest.mark.gpu
def test_scales_are_packed_once(monkeypatch):
    """By the native launcher where it takes the call, by the Python one where it declines: both reach the library's entry point, whose
    calls are counted on either way."""
    import ctypes

    import flash_sparse_attn as fsa
    from flash_sparse_attn import _lib

    lib, count = _lib.load(), []
    real = lib.fsa_pack_scales
    address = lambda f: ctypes.cast(f, ctypes.c_void_p).value  # noqa: E731
    stub = ctypes.CFUNCTYPE(ctypes.c_int, *real.argtypes)(lambda *a: count.append("native") or real(*a))
    monkeypatch.setattr(lib, "fsa_pack_scales", lambda *a: count.append("python") or real(*a))
    one = torch.ones(1, device=DEV)
    kw = dict(is_quant=True, query_scale=one, key_scale=one, value_scale=one)

    def packed(d, prompt):
        x = lambda *s: torch.randn(*s, d, device=DEV).to(torch.float8_e4m3fn)  # noqa: E731
        count.clear()
        if prompt:
            fsa.flash_dense_attn_func(x(2, 50, 4), x(2, 50, 2), x(2, 50, 2), **kw)
        else:
            fsa.flash_dense_attn_with_kvcache_func(x(2, 4), x(2, 50, 2), x(2, 50, 2), **kw)
        return list(count)

    _lib._host.init(address(lib.fsa_decode), address(lib.fsa_fwd), address(lib.fsa_topk_indices), address(stub))
    try:
        for prompt in (False, True):
            assert packed(128, prompt) == ["native"]
            assert packed(64, prompt) == ["python"]  # native FP8 has 128 columns
    finally:
        _lib._host.init(address(lib.fsa_decode), address(lib.fsa_fwd), address(lib.fsa_topk_indices), address(real))
    fsa.check_status()
