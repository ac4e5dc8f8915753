"""Instructions that all 32 lanes of a warp have to execute together (PTX `.aligned`, and bar.sync) are issued only by helpers
of ptx.cuh that bring the warp together first. A kernel that gets this wrong may work or hang depending on what the compiler
made of the branch before, so the rule is checked in the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rocmlir_b200", "csrc")
COLLECTIVE = re.compile(r'"[^"\n]*(?:\.aligned\b|\bbar\.sync\b|\bbarrier\.(?:cluster|cta)\b)[^"\n]*"')


def code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def bodies(text):
    """(name, body) of every function of a header whose functions close with a brace in the first column."""
    return re.findall(r"^(?:static )?__device__ __forceinline__ [\w ]*?(\w+)\([^{;]*\) \{(.*?)^\}|^\Z", text, re.M | re.S)


def test_collective_instructions_stand_in_the_ptx_helpers_only():
    for root, _, files in os.walk(CSRC):
        for name in files:
            if name.endswith((".cu", ".cuh", ".h")) and name != "ptx.cuh":
                assert not COLLECTIVE.search(code(os.path.join(root, name))), name


def test_every_collective_helper_brings_the_warp_together_first():
    text = code(os.path.join(CSRC, "ptx.cuh"))
    found = 0
    for name, body in bodies(text):
        hits = [m.start() for m in COLLECTIVE.finditer(body)]
        if hits:
            assert 0 <= body.find("__syncwarp()") < hits[0], name
            found += len(hits)
    assert found == len(COLLECTIVE.findall(text)) >= 10


def test_waits_of_the_softmax_warps_end_alike_in_all_lanes():
    """A wait that runs out in some lanes only would leave the others at the next collective: warps that go on to one wait
    through the helper that polls once for the whole warp."""
    text = code(os.path.join(CSRC, "attention_sm100.cu"))
    assert not re.search(r"\bmbar_wait\(&?(?:s_full|pv_done)\b", text)
