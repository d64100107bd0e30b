"""Which lane of the MMA issuer does what. PTX does not say which lane ``elect.sync`` picks, so what one lane writes for a later
commit to announce has to be written by the lane that commits: only then program order puts the write first. A mistake here is a
race on shared memory that a GPU run shows by chance at best, so the source is what is looked at."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "flash-sparse-attention_b200", "csrc")


def _code(name):
    """The file's text without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _rest_of_block(text, at):
    """From `at` to the end of the innermost block around it."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth < 0:
            return text[at:i]
    raise AssertionError("unbalanced braces")


@pytest.mark.parametrize("name", ["fsa_fwd_sm100.cu", "fsa_bwd_sm100.cu"])
def test_issuer_works_through_its_elected_lane(name):
    text = _code(name)
    roles = [_rest_of_block(text, m.start()) for m in re.finditer(r"lead\s*=\s*elect_one\(\)", text)]
    assert roles and all("umma_commit_lead(lead" in r for r in roles)
    for role in roles:
        assert not re.search(r"\blane\s*==", role), "a fixed lane does part of the elected lane's work"


def test_a_warp_waits_until_every_lane_has_seen_the_phase():
    # A lane acquires what a barrier announces by its own test of the phase; a vote carries the news to the other lanes, but orders
    # no memory for them. "Any lane" would let the elected lane run ahead of its own acquire.
    votes = [(name, m.group(0)) for name in sorted(os.listdir(CSRC))
             for m in re.finditer(r"__(any|all|ballot)_sync\([^;]*mbar_\w*wait", _code(name))]
    assert votes and all(v.startswith("__all_sync") for _, v in votes), votes


def test_backward_producer_waits_for_tiles_that_nobody_uses():
    # a CTA without a step (an empty split, keys that no window reaches) must not leave while its K and V are on their way into
    # its shared memory: only the issuer of a CTA with steps waits for them otherwise
    text = _code("fsa_bwd_sm100.cu")
    producer = _rest_of_block(text, text.index("mbar_arrive_expect_tx(&bars->kv_full"))
    first_walk = producer[producer.index("bool more = walk_next("):producer.index("for (int it = 0")]
    assert re.search(r"if \(!more\)\s*mbar_wait\(&bars->kv_full, 0, abort_flag\);", first_walk)
