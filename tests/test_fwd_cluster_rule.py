"""The rule that shares the key tiles of a dense call inside clusters, from the header that the launcher takes it from: the cluster
sizes of the forms that test_fwd_cluster_gpu.py runs, and both sides of each of its lines."""

import ctypes
import os
import re
import subprocess

import pytest

CSRC = os.path.abspath(os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "flash-sparse-attention_b200", "csrc"))
SMS = 148
ROOM = {2: 74, 4: 33, 8: 15}  # what a B200 says of clusters whose CTAs fill an SM each: one has to fit inside a GPC


@pytest.fixture(scope="module")
def size(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(f'#include "{CSRC}/fsa_schedule.h"\n'
                                'extern "C" int rule(long long ctas, int tiles, int sms, const int* room) {\n'
                                '  return fsa_fwd_cluster_size(ctas, tiles, sms, [&](int size) { return room[size]; }); }\n')
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-o", str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "rule.so")).rule
    fn.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]

    def call(seqlen, heads, batch=1, room=ROOM):
        table = (ctypes.c_int * 9)(*[room.get(i, 0) for i in range(9)])
        return fn(batch * heads * -(-seqlen // 256), -(-seqlen // 128), SMS, table)

    return call


def test_sizes(size):
    assert size(1024, 8) == 4         # 18.0 us, shared 14.3
    assert size(2000, 8) == 2         # 31.7 us, shared 24.8
    assert size(500, 8) == 1          # 12.3 us, shared 17.1
    assert size(896, 8) == 1 and size(897, 8) == 4      # two CTAs would save three of seven tiles
    assert size(2050, 1) == size(3000, 1) == 8 and size(2050, 1, batch=2) == 4
    assert size(1024, 16) == 2 and size(2304, 8) == 2 and size(2305, 8) == 1 and size(1024, 8, batch=6) == 1
    assert size(3840, 1) == 8 and size(4097, 1) == 4    # 15 clusters of eight find room, 17 do not
    assert size(1024, 8, room={2: 70}) == 2 and size(1024, 8, room={}) == 1
    for heads in (1, 2, 8, 16):
        for seqlen in range(1, 6000, 37):
            n, ctas = size(seqlen, heads), heads * -(-seqlen // 256)
            assert n == 1 or (ctas * n <= SMS and ctas <= ROOM[n])


def test_a_kernel_asks_for_its_own_room():
    # Kernels with the same parameters are of one type, so an array that is static in a template over the type of the kernel would hold
    # the first one's answer for all of them.
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"template <typename Kernel>", text):
            at = text.index("{", m.end())
            depth, i = 1, at + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            assert not re.search(r"\bstatic\b", text[at:i]), (name, text[m.start():at])
