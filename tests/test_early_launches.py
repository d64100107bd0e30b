"""Kernels that are set up while the one in front of them runs: which of them wait, and when they let the next one be set up. A
mistake here is a race on memory, or room on the SMs held during a wait for another GPU, that a run on one GPU does not show: the
source is what is looked at."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "flash-sparse-attention_b200", "csrc")


def _code(name):
    """The file's text without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _kernels():
    """Name and body of every kernel."""
    got = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = _code(name)
        for m in re.finditer(r"__global__[^{;]*?\b(\w+_kernel)\(", text):
            at = text.index("{", m.end())
            depth, i = 1, at + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            got[m.group(1)] = text[at + 1:i - 1]
    return got


def _early():
    """Names of the kernels that are launched early: those that no source launches by their name in the plain form."""
    text = "".join(_code(n) for n in sorted(os.listdir(CSRC)) if n.endswith(".cu"))
    return set(_kernels()) - set(re.findall(r"\b(\w+_kernel)\s*(?:<[^;(){}]*>)?\s*<<<", text))


def test_kernels_that_are_launched_early_wait_before_they_touch_memory():
    kernels, early = _kernels(), _early()
    assert {"fwd_kernel", "bwd_kernel", "dec_kernel", "topk_kernel", "combine_kernel", "bwd_pre_kernel", "bwd_post_kernel"} <= early
    for name in early:
        body = kernels[name]
        at = re.search(r"\b(after_previous|wait_for_previous)\(\);", body)
        assert at, name
        # in front of it: constants, types and static assertions only
        for statement in body[:at.start()].split(";"):
            assert re.match(r"\s*(constexpr\b|using\b|static_assert\b|namespace\b|$)", statement), (name, statement)


@pytest.mark.parametrize("name", sorted(_kernels()))
def test_a_wait_for_another_gpu_comes_before_the_next_kernel_is_set_up(name):
    # combine_kernel is the one that waits; blocks of the next kernel would sit on the SMs for as long as it does
    body = _kernels()[name]
    waits = [m.start() for m in re.finditer(r"\.sys\.", body)]
    lets = [m.start() for m in re.finditer(r"\b(after_previous|let_next_be_set_up)\(\);", body)]
    if name == "combine_kernel":
        assert waits and lets
    if waits and lets:
        assert max(waits) < min(lets)
