"""The rules that set a decode call up while the kernel in front of it still runs, and that give a warp of 64-wide rows a deeper ring, from
the header that the launcher takes them from. (us:
the same call over and over, one split unless clusters are named, 4 KV heads.)"""

import ctypes
import os
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "flash-sparse-attention_b200", "csrc", "fsa_schedule.h")
SMS = 148
ROOM = {2: 148, 3: 93, 4: 71, 5: 57, 6: 45, 7: 37, 8: 33}  # clusters with two CTAs on an SM
LONE = {2: 74, 3: 46, 4: 33, 5: 27, 6: 20, 7: 18, 8: 15}   # and with one


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(f'#include "{os.path.abspath(HEADER)}"\n'
                                'extern "C" int rule(long long c, int occ, int cluster, int room, int splits, long long bytes, int sms) {\n'
                                '  const FsaDecLaunch r = fsa_dec_launch(c, occ, cluster, room, splits, bytes, sms); return r.early ? r.per_sm : -1; }\n'
                                'extern "C" int deep(long long c, int occ, long long tiles, int sms) {\n'
                                '  return fsa_dec_deep_ring(c, occ, tiles, sms); }\n')
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-o", str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "rule.so"))
    fn = lib.rule
    fn.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]

    def call(ctas, occ=3, cluster=1, keys=1000, splits=1, row=256):
        """-1: behind the kernel in front, otherwise the CTAs an SM may hold (0: as many as find room)."""
        room = (LONE if ctas <= SMS else ROOM).get(cluster, 0)
        return fn(ctas, occ, cluster, room, splits, -(-keys // 16) // (4 * splits) * 16 * row, SMS)

    call.deep = lambda ctas, occ, keys: bool(lib.deep(ctypes.c_longlong(ctas), occ, ctypes.c_longlong(-(-keys // 16) // 4), SMS))
    return call


def test_several_rounds(rule):
    assert rule(448) == rule(512, occ=2) == rule(900, keys=2500) == 0
    assert rule(100, occ=1) == rule(148, occ=1, keys=9000) == rule(300, occ=1) == 0  # an SM never holds two


def test_an_even_share(rule):
    assert rule(1) == rule(148, keys=9000) == 1 and rule(149) == rule(296, keys=2500) == 2
    assert rule(280, keys=300) == 2                                          # 9.8 us with as many as fit, 8.9 so
    assert rule(16, occ=2, cluster=8) == rule(128, occ=2, cluster=4) == 1    # 128 in fours: 13.6 and 13.0


def test_what_waits(rule):
    assert rule(280, occ=2, cluster=5) == -1 and rule(240, occ=2, cluster=5) == 0   # 15.8 us early, 12.6 not; 12.3 and 12.7
    assert rule(279, occ=2, cluster=3) == rule(259, occ=2, cluster=7) == -1         # 93 of three 15.3 us early, 12.3 not; 37 of seven 14.3 and 12.9
    assert rule(296, occ=2, cluster=2) == rule(284, occ=2, cluster=4) == rule(264, occ=2, cluster=8) == 0
    assert rule(340, keys=300) == 0 and rule(340, keys=1000) == -1    # 10.2 us early, 10.6 not; 32.1 and 31.5
    assert rule(360, keys=7540, splits=3) == 0    # 52.2 us early, 53.6 not
    assert rule(416, keys=482) == -1 and rule(416, keys=482, row=128) == 0    # dense 17.2 us early, 16.0 not; rows of 64 columns 10.3 and 10.8
    assert rule(444, keys=768) == -1 and rule(296, occ=2, keys=2500) == -1


def test_deep_ring(rule):
    # thirty-two tiles a warp in one round, sixteen in several (1100 keys: 200 CTAs 16.3 us with two tiles, 17.0 with four)
    assert rule.deep(128, 3, 2033) and not rule.deep(128, 3, 2032)
    assert rule.deep(500, 2, 1009) and not rule.deep(500, 2, 1008)
    # 2500 keys, two tiles and four: 360 CTAs 43.3 and 41.5 us, 400 43.2 and 45.1, 440 46.5 and 49.1
    assert rule.deep(300, 3, 2500) and rule.deep(360, 3, 2500) and rule.deep(380, 3, 2500)
    assert not rule.deep(384, 3, 4700) and not rule.deep(400, 3, 2500) and not rule.deep(444, 3, 2500)
    assert rule.deep(592, 2, 2500)                                    # 72.0 and 64.6
    assert rule.deep(800, 3, 6000) and not rule.deep(840, 3, 6000)    # two rounds of 444: 185 and 181, 191 and 201
    assert not rule.deep(1776, 3, 2375)                               # 74 sequences of 9500 keys, 8 KV heads, three splits: 221.6 and 230.6
