"""Orders in the tensor-core kernels whose violation is a race that no run can be relied on to show, so the sources are looked at.
(1) A place of a shared-memory ring goes back only after the words read from it have arrived - the next copy lands there: a
worker's arrival on the `empty` barrier of a ring whose words it read into registers depends on those words (tc_mbar_arrive_used),
or comes behind the instruction that stores them (the weights: to tensor memory); a ring that no worker reads goes back by the
products' commit. (2) No CTA ends with a copy in flight. (3) A producer that begins before griddepcontrol.wait reads the tile list
and weights only, and the launch in front lets it in only after its own wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pelica_b200", "csrc")
PRODUCTS = ["prefill_tc.cu", "prefill_few.cu", "prefill_mx.cu", "prefill_mx8.cu", "prefill_q32.cu"]
EARLY = [n for n in PRODUCTS if n != "prefill_mx.cu"]
ARRIVE = r"tc_mbar_arrive\([^;]*\b%s\b"  # (also `cond ? one : other`)


def source(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def body(text, name):
    """A kernel's text, up to the end of its function."""
    return re.search(r"__global__[^;{]*\b%s\(.*?\n}\n" % name, text, re.S).group(0)


@pytest.mark.parametrize("name", PRODUCTS)
def test_places_go_back_after_their_words_arrived(name):
    text = source(name)
    # the ring of work items, the ring of the tokens' blocks
    assert re.search(r"tc_mbar_arrive_used\(it_empty \+ s, [^;]*it\.t\.x[^;]*it\.r0", text)
    for ring in ("it_empty", "empty_b"):
        assert not re.search(ARRIVE % ring, text), ring
    if name == "prefill_mx8.cu":  # nobody reads operand A, its scales or the pieces into registers: the commits give them back
        assert not re.search(r"tc_mbar_arrive(_used)?\([^;]*\b(empty_raw|a_free)\b", text)
        for ring in ("empty_raw", "a_free"):
            assert re.search(r"tc_commit\(%s \+ st\)" % ring, text) and re.search(r"tc_mbar_init\(%s \+ i, 1\)" % ring, text), ring
        # the scales are written into a place that has come back, and handed on behind the fence
        assert re.search(r"tc_wait\(empty_raw \+ sr, pr,.*?\*\(uint4 \*\)\(sSA \+ sr.*?fence\.proxy\.async.*?tc_mbar_arrive\(full_raw \+ sr\)",
                         text.split("TcBytes8 nx")[1], re.S)
        return
    # the ring of the weights: between the last read of the box and the arrival its words are stored
    read = [m.end() for m in re.finditer(r"=\s*\*\(const uint4 \*\)\(r(?:aw|q|h|p)\b[^;]*;|unpack_q[46]\(raw", text)]
    backs = [m.start() for m in re.finditer(ARRIVE % "empty_raw", text)]
    assert backs
    for back in backs:
        last = max(r for r in read if r < back)
        assert re.search(r"tc_st(16|32)\(", text[last:back]), text[last:back]


def test_the_arrival_depends_on_the_words():
    helper = source("tcgen.cuh").split("tc_mbar_arrive_used")[1].split("tc_mbar_expect")[0]
    assert re.search(r"and\.b32 a, %1, %2;.*add\.u32 a, a, %0;.*arrive[^;]*\[a\]", helper.replace("\n", " "))


def test_copies_in_flight_are_waited_for():
    """No CTA ends with a copy on its way into its shared memory, also where a wait ran out: every ring's last copies are
    waited for, each ring by its own count, with a limit that a caller's short one does not shorten."""
    for name in PRODUCTS:
        text = source(name)
        for bar in ("full_raw", "a_ready" if name == "prefill_mx8.cu" else "full_b"):
            assert re.search(r"tc_landed\(%s \+" % bar, text), (name, bar)
        assert "< A.wait_ns" not in text, name
    assert "wait_ns" not in source("tcgen.cuh").split("TC_LANDED_NS")[1].split("tc_pack2")[0]
    few = source("kernels_basic.cu").split("k_route_plan_small")[1].split("the last CTA")[0]
    assert re.search(r"atomicCAS\(err, 0, 9\);\s*wait\(ph, \d+ull\);", few)


@pytest.mark.parametrize("name", EARLY)
def test_early_producers_start_weights_only(name):
    text = source(name)
    assert len(re.findall(r"if \(warp != MW \+ 1\) (?:\{\s*)?pm_pdl_wait\(\);", text)) == 1  # every other warp waits first
    producer = text[text.index("} else if (warp == MW + 1) {"):]
    before, after = producer.split("pm_pdl_wait();", 1)
    # the tile list past L1, tensor copies of the weights; no operand, no counter, no item, no write
    assert "__ldcg(A.tiles" in before and "__ldcg(A.n_tiles)" in before and "tc_tma3(" in before
    for late in ("cp.async.bulk.shared", "A.rec", "atomicAdd", "items[", "it_full", "A.out", "A.next", "__ldg"):
        assert late not in before, late
    for late in ("cp.async.bulk.shared", "A.rec", "atomicAdd", "items[", "it_full"):
        assert late in after, late


def test_launches_in_front_of_early_producers_wait_before_they_let_them_in():
    common = source("common.cuh")
    assert re.search(r"void pm_pdl\(\) \{\s*pm_pdl_wait\(\);\s*pm_pdl_trigger\(\);\s*\}", common)
    for name, kernels in {"prefill_tc.cu": ("k_tc_quant_rows", "k_tc_rows"), "prefill_mx8.cu": ("k_mx8_rows",),
                          "prefill_q32.cu": ("k_q32_rows",)}.items():
        for k in kernels:
            b = body(source(name), k)
            assert b.count("pm_pdl();") == 1 and not re.search(r"pm_pdl_(early|trigger)|launch_dependents", b), k
            assert b.index("pm_pdl();") < b.index("tiles[blockIdx.y]"), k
    # (the down products of k_tc_mx8 follow its gate/up products)
    b = body(source("prefill_mx8.cu"), "k_tc_mx8")
    assert re.findall(r"(?:if \(\S+\) )?pm_pdl_trigger\(\);", b) == ["if (DOWN) pm_pdl_trigger();", "if (!DOWN) pm_pdl_trigger();"]
    assert b.index("pm_pdl_wait();") < b.index("if (!DOWN) pm_pdl_trigger();")
    # on the host a rows' kernel stands in front of every product that needs one
    api = source("api.cu")
    for f in ("dev_experts", "dev_shared"):
        text = re.search(r"static int32_t %s\(.*?\n}\n" % f, api, re.S).group(0)
        seen = []
        for call in re.findall(r"\blaunch_\w+", text):
            if call in ("launch_tc", "launch_tc_q32"):
                assert any(s.endswith("_rows") for s in seen), (f, call)
                seen = []
            else:
                seen.append(call)
    mx = re.search(r"if \(path\.mx\) \{.*?\n  \}\n", api, re.S).group(0)
    assert re.findall(r"\blaunch_\w+", mx)[:4] == ["launch_mx8_rows", "launch_mx_rows", "launch_tc_mx8", "launch_tc_mx"]
