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
    """The waits for loads and stores are the exception: they follow the access, which has brought the warp together. The raw load is
    for the helpers of this header, which do it for several of them at once."""
    text = code(os.path.join(CSRC, "ptx.cuh"))
    found = 0
    for name, body in bodies(text):
        hits = [m.start() for m in COLLECTIVE.finditer(body)]
        if hits:
            found += len(hits)
            if name not in ("tmem_ld_wait", "tmem_st_wait", "tmem_ld32_raw"):
                assert 0 <= body.find("__syncwarp()") < hits[0], name
        if "tmem_ld32_raw(" in body:
            assert 0 <= body.find("__syncwarp()") < body.find("tmem_ld32_raw("), name
    assert found == len(COLLECTIVE.findall(text)) >= 12


def test_waits_follow_their_accesses():
    """Between an access to tensor memory and its wait no lane leaves the others, or the warp meets again."""
    for root, _, files in os.walk(CSRC):
        for name in files:
            if not name.endswith((".cu", ".cuh")) or name == "ptx.cuh":
                continue
            text = code(os.path.join(root, name))
            for m in re.finditer(r"\btmem_(ld|st)_wait\(\);", text):
                before = text[:m.start()]
                access = max(before.rfind(f"tmem_{m.group(1)}{n}(") for n in (16, 32, 64))
                between = before[access:]
                parted = re.search(r"\blane(?:_id\(\))? == 0|\bvalid\b|\brow_ok\b|\bleader\b", between)
                assert access >= 0 and (not parted or between.rfind("__syncwarp()") > parted.start()), (name, between[-200:])


def test_waits_of_the_softmax_warps_end_alike_in_all_lanes():
    """A wait that runs out in some lanes only would leave the others at the next collective: warps that go on to one wait
    through the helper that polls once for the whole warp."""
    text = code(os.path.join(CSRC, "attention_sm100.cu"))
    assert not re.search(r"\bmbar_wait\(&?(?:s_full|pv_done)\b", text)
