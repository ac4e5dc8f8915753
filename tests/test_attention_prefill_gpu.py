"""Attention over more than one query tile without side tensors (attention_prefill_sm100.cu): edges of query tiles and key blocks, pairs
whose second tile is missing, fewer and more items than SMs, every operand order, both element types.

The bound: each probability is rounded once to the element type (half an ulp, u, of relative error) before it meets V, and the
result once more, so an element is off by at most 2u * max|V|; the f32 arithmetic around that is a thousand times finer (5 % for it).
"""
import math

import pytest

pytestmark = pytest.mark.gpu


def reference(q, k, v, scale, causal):
    s = (q.double() @ k.double().transpose(1, 2)) * scale
    if causal:
        s.masked_fill_(s.new_ones(s.shape[1:]).triu(1).bool(), -math.inf)
    return s.softmax(-1) @ v.double()


def check(got, q, k, v, scale, causal):
    u = 2.0 ** -11 if got.element_size() == 2 and got.dtype.is_floating_point and "bfloat" not in str(got.dtype) else 2.0 ** -8
    err = (got.double() - reference(q, k, v, scale, causal)).abs().max().item()
    assert err <= 2.1 * u * v.double().abs().max().item(), err


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("g,sq,sk,d,dv,causal,trans_k", [
    (1, 129, 1, 64, 64, False, True), (2, 129, 127, 128, 64, False, True), (3, 255, 128, 64, 128, False, False),
    (2, 256, 129, 128, 128, False, True), (2, 257, 264, 128, 128, True, False), (5, 385, 385, 64, 64, True, True),
    (2, 300, 129, 128, 128, True, True), (2, 129, 900, 40, 24, True, True), (160, 130, 130, 64, 64, True, True),
    (149, 129, 256, 128, 128, False, True), (40, 1025, 1025, 128, 128, True, True), (37, 640, 1000, 72, 120, False, False)])
def test_prefill_matches_reference(cuda_device, dtype, g, sq, sk, d, dv, causal, trans_k):
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.attention import attention
    gen = torch.Generator(device="cuda").manual_seed(sq * 1000 + sk)
    q, k, v = (torch.randn(s, device="cuda", generator=gen).to(getattr(torch, dtype)) for s in ((g, sq, d), (g, sk, d), (g, sk, dv)))
    scale = 1.0 / math.sqrt(d)
    got = attention(q, k if trans_k else k.transpose(1, 2).contiguous(), v, trans_k=trans_k, scale=scale, causal=causal)
    torch.cuda.synchronize()
    assert L.kernel_status() == 0
    check(got, q, k, v, scale, causal)


@pytest.mark.parametrize("causal", [False, True])
def test_maximum_that_grows_from_block_to_block(cuda_device, causal):
    """The exponentials of a block begin on the guess that the row maximum has not outgrown its reference by 2^8. Here it does in some
    rows and not in others, in every block, by 2^5 to 2^40."""
    import torch
    from rocmlir_b200.attention import attention
    g, s, d = 3, 700, 64
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn((g, s, d), device="cuda", generator=gen) for _ in range(3))
    k = k * (1 + 2 * (torch.arange(s, device="cuda") // 128))[None, :, None]
    q = q * torch.where(torch.arange(s, device="cuda") % 3 == 0, 0.5, 2.0)[None, :, None]
    q, k, v = q.half(), k.half(), v.half()
    check(attention(q, k, v, trans_k=True, scale=0.25, causal=causal), q, k, v, 0.25, causal)


def test_two_streams_and_a_graph_give_the_same_bits(cuda_device):
    """Work items are claimed from CTAs of the same launch only: launches side by side and replays agree with one alone."""
    import torch
    from rocmlir_b200.attention import attention
    q, k, v = (torch.randn((50, 900, 64), device="cuda").half() for _ in range(3))
    f = lambda out: attention(q, k, v, trans_k=True, scale=0.125, causal=True, out=out)
    want = f(torch.empty_like(q)).clone()
    outs = [torch.zeros_like(q) for _ in range(6)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for i, o in enumerate(outs[:4]):
        with torch.cuda.stream(streams[i % 2]):
            f(o)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        f(outs[4])
        f(outs[5])
    graph.replay()
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, want)


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
def test_scores_that_are_not_finite(cuda_device, bad):
    """A key whose scores are NaN or +inf makes the rows that see it NaN; one at -inf weighs nothing."""
    import torch
    from rocmlir_b200.attention import attention
    q, k, v = (torch.rand((2, 300, 64), device="cuda").half() + 0.1 for _ in range(3))
    k[1, 200, 3] = bad
    got = attention(q, k, v, trans_k=True, scale=0.125, causal=True)
    want = reference(q, k, v, 0.125, True)
    seen = torch.zeros((2, 300, 1), dtype=torch.bool, device="cuda")
    seen[1, 200:] = bad != -math.inf
    assert torch.equal(got.isnan(), seen.expand_as(got))
    ok = ~seen.expand_as(got)
    assert (got.double() - want)[ok].abs().max().item() <= 2.1 * 2.0 ** -11 * v.max().item()


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("scale", [0.0, -0.0, 2.0 ** -149, 2.0 ** -126])
@pytest.mark.parametrize("g,s,sk,d,causal", [(2, 129, 128, 64, True), (2, 256, 256, 128, True), (3, 300, 300, 64, True), (1, 129, 1, 64, False),
                                             (2, 257, 130, 128, False), (2, 900, 897, 64, False), (2, 256, 256, 64, False)])
def test_scale_of_zero(cuda_device, dtype, scale, g, s, sk, d, causal):
    """Every visible key weighs the same; keys past the end and above the diagonal weigh nothing."""
    import torch
    from rocmlir_b200.attention import attention
    gen = torch.Generator(device="cuda").manual_seed(s + sk)
    q, k, v = (torch.randn(shape, device="cuda", generator=gen).to(getattr(torch, dtype)) for shape in ((g, s, d), (g, sk, d), (g, sk, d)))
    check(attention(q, k, v, trans_k=True, scale=scale, causal=causal), q, k, v, scale, causal)
