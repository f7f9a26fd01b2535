"""The tensor-core kernels hand a place of a shared-memory ring back only after the words read from it have arrived: the
next copy lands there. The outcome is a race that no run can be relied on to show, so the sources are looked at: a
worker's arrival on the `empty` barrier of a ring whose words it read into registers depends on those words
(tc_mbar_arrive_used), or comes behind the instruction that stores them (the weights: to tensor or shared memory)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pelica_b200", "csrc")


def source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("name", ["prefill_tc.cu", "prefill_mx.cu", "prefill_mx8.cu", "prefill_q32.cu"])
def test_places_go_back_after_their_words_arrived(name):
    text = source(name)
    # the ring of work items, the ring of the tokens' blocks
    assert re.search(r"tc_mbar_arrive_used\(it_empty \+ s, [^;]*it\.t\.x[^;]*it\.r0", text)
    for ring in ("it_empty", "empty_b"):
        assert not re.search(r"tc_mbar_arrive\(%s" % ring, text), ring
    # the ring of the weights: between the last read of the box and the arrival its words are stored
    read = [m.end() for m in re.finditer(r"\bq?\[?[^;\n]*=\s*\*\(const uint4 \*\)\(r(?:aw|q|h)\b[^;]*;|unpack_q[46]\(raw", text)]
    for back in [m.start() for m in re.finditer(r"tc_mbar_arrive\(empty_raw", text)]:
        last = max(r for r in read if r < back)
        assert re.search(r"tc_st(16|32)\(|\*\(uint2 \*\)\(dst", text[last:back]), text[last:back]


def test_the_arrival_depends_on_the_words():
    helper = source("tcgen.cuh").split("tc_mbar_arrive_used")[1].split("tc_mbar_expect")[0]
    assert re.search(r"and\.b32 a, %1, %2;.*add\.u32 a, a, %0;.*arrive[^;]*\[a\]", helper.replace("\n", " "))


def test_copies_in_flight_are_waited_for():
    """No CTA ends with a copy on its way into its shared memory, also where a wait ran out: every ring's last copies are
    waited for, each ring by its own count, with a limit that a caller's short one does not shorten."""
    rings = {"prefill_tc.cu": ("full_raw", "full_b"), "prefill_mx.cu": ("full_raw", "full_b"),
             "prefill_mx8.cu": ("full_raw", "a_ready"), "prefill_q32.cu": ("full_raw", "full_b")}
    for name, bars in rings.items():
        text = source(name)
        for bar in bars:
            assert re.search(r"tc_landed\(%s \+" % bar, text), (name, bar)
        assert "< A.wait_ns" not in text, name
    assert "wait_ns" not in source("tcgen.cuh").split("TC_LANDED_NS")[1].split("tc_pack2")[0]
    few = source("kernels_basic.cu").split("k_route_plan_small")[1].split("the last CTA")[0]
    assert re.search(r"atomicCAS\(err, 0, 9\);\s*wait\(ph, \d+ull\);", few)
