"""The rule that sets a decode call up while the kernel in front of it still runs, from the header that the launcher takes it from. (us:
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
                                'extern "C" int rule(long long c, int occ, int cluster, int room, long long tiles, int sms) {\n'
                                '  const FsaDecLaunch r = fsa_dec_launch(c, occ, cluster, room, tiles, sms); return r.early ? r.per_sm : -1; }\n')
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-o", str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "rule.so")).rule
    fn.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_int]

    def call(ctas, occ=3, cluster=1, keys=1000):
        """-1: behind the kernel in front, otherwise the CTAs an SM may hold (0: as many as find room)."""
        room = (LONE if ctas <= SMS else ROOM).get(cluster, 0)
        return fn(ctas, occ, cluster, room, -(-keys // 16) // 4, SMS)

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
    assert rule(296, occ=2, cluster=2) == 0 and rule(256, occ=2, cluster=4) == 0
    assert rule(340, keys=300) == 0 and rule(340, keys=1000) == -1    # 10.2 us early, 10.6 not; 32.1 and 31.5
    assert rule(444, keys=768) == -1 and rule(296, occ=2, keys=2500) == -1
