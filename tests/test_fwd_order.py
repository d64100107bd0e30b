"""The rule that has the forward's CTAs rank their work by length, from the header that the launcher takes it from."""

import ctypes
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "flash-sparse-attention_b200", "csrc", "fsa_schedule.h")
SMS = 148


@pytest.fixture(scope="module")
def longest_first(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(f'#include "{os.path.abspath(HEADER)}"\n'
                                'extern "C" int rule(int c, int l, long long b, long long p, long long s, long long h, long long q, '
                                'long long k, int n) { return fsa_fwd_longest_first(c, l, b, p, s, h, q, k, n); }\n')
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "rule.so")).rule
    fn.argtypes = [ctypes.c_int] * 2 + [ctypes.c_longlong] * 6 + [ctypes.c_int]

    def call(batch, sq, sk, heads, causal=True, local=False, splits=1):
        return bool(fn(causal, local, batch, -(-sq // 256), splits, heads, sq, sk, SMS))

    return call


def test_chunks_in_front_of_cached_keys_are_ranked(longest_first):
    f = longest_first
    assert f(4, 500, 12000, 32)       # 2000 to 12000 keys: 329 us, ranked 245
    assert f(8, 1000, 8000, 8)        # 1000 to 8000 keys: 206 us, ranked 140
    assert f(64, 100, 8000, 8)        # 333 us, ranked 279
    assert f(2, 8000, 16000, 32)      # 1450 us, ranked 1365
    assert not f(4, 500, 12000, 8)    # 64 CTAs: all start at once
    assert not f(1, 4000, 16000, 32)
    assert not f(4, 500, 12000, 32, local=True)


def test_packed_self_attention_is_not_ranked(longest_first):
    f = longest_first
    # causal: a pair's key tiles grow with its position alone, so the last pairs first are the longest first already
    assert not f(128, 128, 128, 32)   # 232 us, ranked 276 (one tile a CTA: the ranking is longer than the work)
    assert not f(16, 2000, 2000, 32)  # 337 us, ranked 379
    assert not f(8, 4000, 4000, 8)    # 127 us, ranked 148
    assert not f(4, 8000, 8000, 32)   # 846 us, ranked 887
    assert not f(4, 1000, 1024, 64)   # a first chunk over a cache of whole pages


def test_ranking_has_to_be_short_beside_the_work(longest_first):
    f = longest_first
    assert f(4, 8000, 8000, 8, causal=False)       # 436 us, ranked 397
    assert f(8, 4000, 4000, 32, causal=False)      # 872 us, ranked 832
    assert not f(64, 512, 512, 32, causal=False)   # 284 us, ranked 323
    assert not f(16, 2048, 2048, 32, causal=False)  # 128 items before 16 key tiles
    assert not f(64, 60, 512, 32)
    assert not f(32, 300, 8000, 8, splits=4)       # 64 items before 16 key tiles a split
    assert f(128, 256, 8000, 32) and not f(129, 256, 8000, 32)  # the most that a CTA ranks
