"""What the estimate that chooses tiles and K ranges of a GEMM may not change (no GPU needed: configuration and workspace queries). An
explicit variant word without tile fields keeps the rule."""
import ctypes as C
import math
import random

import pytest

from rocmlir_b200 import _lib as L

RULE = 1 << 27
RESULTS = {L.F16: (L.F16, L.F32), L.BF16: (L.BF16, L.F32), L.F32: (L.F32,), L.I8: (L.I32, L.I8, L.F32), L.F8E4M3: (L.BF16, L.F32)}


def query(p, variant):
    lib, info = L.lib(), L.RbGemmConfigInfo()
    lib.rbSetGemmVariant(variant)
    L.check(lib.rbGemmGetConfig(C.byref(p), C.byref(info)))
    return info, int(lib.rbGemmWorkspaceSize(C.byref(p)))


def products(count):
    # (g, m, n, k, trans_b, type, result): three that the estimate used to cut
    yield from [(1, 282, 4871, 5040, 1, L.F16, L.F16), (1, 340, 4713, 7770, 0, L.F16, L.F32), (1, 290, 4971, 5412, 0, L.BF16, L.BF16)]
    rng = random.Random(2)
    for _ in range(count):
        m, n, k = (max(1, round(math.exp(rng.uniform(math.log(64), math.log(9000))))) for _ in range(3))
        if rng.random() < 0.5:
            m, n, k = (max(64, v // 64 * 64) for v in (m, n, k))
        t = rng.choice(list(RESULTS))
        yield rng.choice([1, 1, 3]), m, n, k, rng.randrange(2), t, rng.choice(RESULTS[t])


def test_ranges_and_workspace_stay_within_the_rule():
    changed = 0
    for g, m, n, k, tb, t, ct in products(6000):
        p = L.RbGemmProblem(g, m, n, k, 0, tb, 0, t, ct, 0, 0)
        (rule, rule_ws), (got, ws) = query(p, RULE), query(p, 0)
        changed += (rule.tile_m, rule.tile_n, rule.splits) != (got.tile_m, got.tile_n, got.splits)
        what = (g, m, n, k, tb, t, ct)
        if rule.splits == 1:   # one kernel stays one kernel
            assert got.splits == 1 and ws <= rule_ws, what
        if ct == L.F32 and t != L.I8:   # sums of no more elements in one accumulator
            blocks = -(-k // rule.tile_k)
            assert -(-blocks // got.splits) <= -(-blocks // rule.splits), what
    assert changed > 1000   # the estimate is at work


def test_eight_bit_results_of_several_waves_keep_wide_tiles():
    """896 x 6016 x 1024, requantised: tiles of 64 columns take 22 us, of 128 17, the rule's 20."""
    p = L.RbGemmProblem(1, 896, 6016, 1024, 0, 1, 0, L.I8, L.I8, 0, 0)
    assert query(p, 0)[0].tile_n >= 128


def test_dimensions_of_a_handle_are_those_of_the_one_kernel():
    """K is cut for the sake of the f32 sums: the handle names the grid of the kernel that a client launches itself, which sums all of K. Cut for
    speed there is no such kernel, and the grid is the library's."""
    from rocmlir_b200 import miir
    for m, n, k, cut, one in ((384, 4288, 1472, True, True), (64, 576, 8192, True, False), (4096, 4096, 1024, False, False)):
        p = L.RbGemmProblem(1, m, n, k, 0, 0, 0, L.F16, L.F32, 0, 0)
        info, ws = query(p, 0)
        assert (info.splits > 1) == cut and (ws > 0) == cut
        with miir.Handle(f"--operation gemm --arch sm_100a -t f16 -out_datatype f32 -transA false -transB false -g 1 -m {m} -n {n} -k {k}") as h:
            h.lower_bin()
            glob, loc = h.execution_dims()
            assert (glob // loc != info.grid) == one


@pytest.mark.parametrize("m,n,k,trans_a,trans_b,tile", [
    (704, 3098, 128, 0, 1, (128, 64)), (1218, 1823, 150, 0, 0, (128, 64)), (2304, 2157, 384, 0, 0, (256, 128)), (2267, 2297, 740, 0, 1, (256, 128)),
    (3405, 1344, 192, 1, 0, (256, 128)), (3246, 1541, 263, 0, 0, (256, 128)), (2368, 1920, 640, 0, 1, (128, 128))])
def test_f32_products_of_several_waves(m, n, k, trans_a, trans_b, tile):
    """The tile that was the fastest of those measured, rows of C on and off 16 bytes (others took 1.1 to 1.4 times as long)."""
    info, _ = query(L.RbGemmProblem(1, m, n, k, trans_a, trans_b, 0, L.F32, L.F32, 0, 0), 0)
    assert (info.tile_m, info.tile_n, info.splits) == (*tile, 1)
