"""GPU parity of the attention kernel for at most 128 queries when a cluster of CTAs divides a query tile's keys (few tiles),
and of its mask reads, against the double-precision oracle."""
import math

import numpy as np
import pytest

import oracle
from test_attention_gpu import make_qkv, run_attention

pytestmark = pytest.mark.gpu

# (g, sq, sk, d, dv): clusters of 2, 4 and 8; one query and a full tile; a last key block of one key; more parts than the
# blocks fill (nine blocks over eight parts: five of two); head dimensions below the 64 / 128 the kernel works on
SHAPES = [(3, 1, 1000, 128, 128), (2, 16, 1025, 64, 64), (1, 128, 2048, 128, 64), (40, 5, 384, 64, 128), (60, 33, 256, 128, 128),
          (1, 2, 1100, 40, 24), (160, 3, 640, 128, 128)]


def check(got, ref, code):
    # P and O carry one rounding to the element type each (2^-11 f16, 2^-8 bf16, relative); the f32 sums add far less
    ulp = 2.0 ** -10 if code == oracle.F16 else 2.0 ** -7
    assert np.abs(got - ref).max() <= 2.0 * ulp * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16])
@pytest.mark.parametrize("g,sq,sk,d,dv", SHAPES)
def test_split_keys(cuda_device, g, sq, sk, d, dv, code):
    (q, qraw), (k, kraw), (v, vraw) = make_qkv(g, sq, sk, d, dv, code)
    scale = 1.0 / math.sqrt(d)
    ref = oracle.attention(q, k, v, elem_type=oracle.F64, scale_scalar=scale, threads=oracle.max_threads())
    got = run_attention(qraw, kraw, vraw, code, scale=scale)
    check(got, ref, code)
    turned = run_attention(qraw, np.ascontiguousarray(np.swapaxes(kraw, 1, 2)), vraw, code, scale=scale, trans_k=True)
    np.testing.assert_array_equal(turned, got)
    swapped = run_attention(qraw, kraw, vraw, code, scale=scale, trans_o=True)
    np.testing.assert_array_equal(np.swapaxes(swapped.reshape(g, dv, sq), 1, 2), got.reshape(g, sq, dv))


# at most four queries: one byte per key and thread, keys divided over a cluster or not. Above: mask rows on 16-byte boundaries
# are read as words, others byte by byte, both with the keys divided (few tiles) and not; a ragged last block of keys; one,
# two and three live warps of a query tile
@pytest.mark.parametrize("fill", [float("-inf"), -1000.0, float(np.finfo(np.float32).min)])
@pytest.mark.parametrize("g,sq,sk,d,dv", [(3, 4, 1040, 128, 128), (2, 4, 1001, 64, 64), (150, 2, 272, 64, 64),
                                          (3, 16, 1040, 128, 128), (2, 37, 1296, 64, 64), (1, 70, 2048, 64, 128), (2, 40, 1001, 64, 64),
                                          (2, 37, 272, 64, 64), (150, 7, 272, 64, 128), (150, 6, 277, 128, 64)])
def test_split_keys_with_mask(cuda_device, g, sq, sk, d, dv, fill):
    """A row without any key left, and one whose keys all lie in the first block, so that the other CTAs of the cluster
    contribute nothing."""
    (q, qraw), (k, kraw), (v, vraw) = make_qkv(g, sq, sk, d, dv, oracle.F16)
    scale = 1.0 / math.sqrt(d)
    mask = (np.random.Generator(np.random.PCG64(4)).random((g, sq, sk)) > 0.4).astype(np.int8)
    mask[0, 0, :] = 0
    mask[0, 1, 5:] = 0
    mask[0, 1, :5] = 1
    got = run_attention(qraw, kraw, vraw, oracle.F16, scale=scale, mask=mask, mask_fill=fill).reshape(g, sq, dv)
    if fill == -1000.0:
        ref = oracle.attention(q, k, v, elem_type=oracle.F64, scale_scalar=scale, mask=mask, mask_fill=fill, threads=oracle.max_threads())
    else:   # (the lowest float times log2(e) is -inf as well)
        ref = oracle.attention(q, k, v, elem_type=oracle.F64, scale_scalar=scale, mask=mask, mask_fill=float("-inf"), threads=oracle.max_threads())
        assert not got[0, 0].any()
        got, ref = got.reshape(g * sq, dv)[1:], np.asarray(ref).reshape(g * sq, dv)[1:]
    check(got.reshape(-1), np.asarray(ref).reshape(-1), oracle.F16)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("sk", [256, 700])
@pytest.mark.parametrize("g,sq", [(2, 1), (160, 2), (2, 3), (2, 4), (2, 8), (160, 8)])
def test_scale_and_bias_tensors(cuda_device, g, sq, sk, masked):
    """Every element of the side tensors differs, so that a wrong row, key or group shows; the fill of masked keys replaces the
    biased score."""
    import torch
    from rocmlir_b200.attention import attention
    d = 64
    gen = torch.Generator(device="cuda").manual_seed(7)
    q, k, v = (torch.randn(s, device="cuda", generator=gen).half() for s in ((g, sq, d), (g, sk, d), (g, sk, d)))
    st, bias = (torch.randn((g, sq, sk), device="cuda", generator=gen).half() for _ in range(2))
    mask = (torch.rand((g, sq, sk), device="cuda", generator=gen) > 0.3).to(torch.int8) if masked else None
    got = attention(q, k, v, trans_k=True, scale=0.1, scale_tensor=st, bias=bias, mask=mask, mask_fill=-2.0).double()
    s = q.double() @ k.double().transpose(1, 2) * 0.1 * st.double() + bias.double()
    if masked:
        s = torch.where(mask != 0, s, torch.full_like(s, -2.0))
    ref = s.softmax(-1) @ v.double()
    check(got.cpu().numpy(), ref.cpu().numpy(), oracle.F16)


@pytest.mark.parametrize("code", [oracle.F16, oracle.BF16])
@pytest.mark.parametrize("g,sq,sk", [(2, 2, 100), (2, 3, 300), (160, 4, 300), (2, 4, 128), (3, 1, 300), (2, 9, 300)])
def test_causal_few_queries(cuda_device, g, sq, sk, code):
    """Query i sees keys 0 .. i, whatever the number of keys: one key block at most."""
    (q, qraw), (k, kraw), (v, vraw) = make_qkv(g, sq, sk, 64, 64, code)
    mask = np.ascontiguousarray(np.broadcast_to(np.tril(np.ones((sq, sk), np.int8)), (g, sq, sk)))
    ref = oracle.attention(q, k, v, elem_type=oracle.F64, scale_scalar=0.125, mask=mask, mask_fill=float("-inf"),
                           threads=oracle.max_threads())
    got = run_attention(qraw, kraw, vraw, code, scale=0.125, causal=True)
    check(got.reshape(-1), np.asarray(ref).reshape(-1), code)
    check(run_attention(qraw, kraw, vraw, code, scale=0.125, mask=mask).reshape(-1), np.asarray(ref).reshape(-1), code)


@pytest.mark.parametrize("g,sq,sk,causal,masked", [(2, 300, 2048, False, False), (2, 300, 2048, True, False), (1, 700, 1000, True, False),
                                                   (2, 300, 1040, False, True), (200, 150, 400, True, False)])
def test_negative_scale_over_several_query_tiles(cuda_device, g, sq, sk, causal, masked):
    """A negative scale keeps more than 128 queries on the single-tile kernel: several tiles of a group with their keys divided
    or not, under the causal flag each tile with its own number of key blocks and parts that have none."""
    import torch
    from rocmlir_b200.attention import attention
    gen = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(s, device="cuda", generator=gen).half() for s in ((g, sq, 64), (g, sk, 64), (g, sk, 64)))
    mask = (torch.rand((g, sq, sk), device="cuda", generator=gen) > 0.3).to(torch.int8) if masked else None
    got = attention(q, k, v, trans_k=True, scale=-0.125, causal=causal, mask=mask).double()
    s = q.double() @ k.double().transpose(1, 2) * -0.125
    if causal:
        s = s.masked_fill(torch.ones((sq, sk), dtype=torch.bool, device="cuda").triu(1), -float("inf"))
    if masked:
        s = s.masked_fill(mask == 0, -float("inf"))
    check(got.cpu().numpy(), (s.softmax(-1) @ v.double()).cpu().numpy(), oracle.F16)


@pytest.mark.parametrize("g,sq,sk,masked", [(64, 1, 4096, True), (3, 4, 1000, False), (2, 37, 1296, True), (1, 128, 2048, False)])
def test_divided_keys_repeat_exactly(cuda_device, g, sq, sk, masked):
    """The parts of a divided row are added in the order of their ranks: the same bits on every call."""
    import torch
    from rocmlir_b200.attention import attention
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(s, device="cuda", generator=gen).half() for s in ((g, sq, 128), (g, sk, 128), (g, sk, 128)))
    mask = (torch.rand((g, sq, sk), device="cuda", generator=gen) > 0.3).to(torch.int8) if masked else None
    first = attention(q, k, v, trans_k=True, scale=0.1, mask=mask)
    for _ in range(20):
        assert torch.equal(attention(q, k, v, trans_k=True, scale=0.1, mask=mask), first)


@pytest.mark.parametrize("g,sq,sk,masked", [(2, 3, 640, False), (2, 40, 640, False), (2, 40, 640, True), (160, 100, 256, False)])
def test_quantised_form_with_few_queries(cuda_device, g, sq, sk, masked):
    """First product in int8, with the keys divided over a cluster and not; the reference rounds to f16 where the form does."""
    import torch
    from rocmlir_b200.attention import attention
    d = 64
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k = (torch.randint(-8, 9, s, device="cuda", generator=gen, dtype=torch.int8) for s in ((g, sq, d), (g, sk, d)))
    v = torch.randn((g, sk, d), device="cuda", generator=gen).half()
    mask = (torch.rand((g, sq, sk), device="cuda", generator=gen) > 0.3).to(torch.int8) if masked else None
    qb, qs = torch.tensor([3], dtype=torch.int8, device="cuda"), torch.tensor([0.0078125], dtype=torch.float16, device="cuda")
    got = attention(q, k, v, trans_k=True, scale=1.0, mask=mask, quant_bias=qb, quant_scale=qs).double()
    s = (q.double() @ k.double().transpose(1, 2) - 3.0).half() * qs
    if masked:
        s = s.masked_fill(mask == 0, -float("inf"))
    ref = s.double().softmax(-1) @ v.double()
    check(got.cpu().numpy(), ref.cpu().numpy(), oracle.F16)


def test_split_keys_with_side_tensors_and_infinities(cuda_device):
    """Scale and bias tensors on the split form, and an infinite value of V: infinite (not NaN) where its key has weight."""
    import torch
    from rocmlir_b200.attention import attention
    g, sq, sk, d = 2, 8, 700, 64
    gen = torch.Generator(device="cuda").manual_seed(2)
    q, k, v = (torch.randn(s, device="cuda", generator=gen).half() for s in ((g, sq, d), (g, sk, d), (g, sk, d)))
    st, bias = (torch.randn((g, sq, sk), device="cuda", generator=gen).half() for _ in range(2))
    got = attention(q, k, v, trans_k=True, scale=0.1, scale_tensor=st, bias=bias).double()
    s = q.double() @ k.double().transpose(1, 2) * 0.1 * st.double() + bias.double()
    ref = s.softmax(-1) @ v.double()
    assert (got - ref).abs().max() <= 2.0 * 2.0 ** -10 * max(1.0, float(ref.abs().max()))
    v[1, 650, 3] = float("inf")
    got = attention(q, k, v, trans_k=True, scale=0.1)
    assert torch.isinf(got[1, :, 3]).all() and (got[1, :, 3] > 0).all()
    got[1, :, 3] = 0
    assert torch.isfinite(got).all()


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 16])
@pytest.mark.parametrize("g,sq,sk", [(2, 5, 128), (2, 16, 129), (3, 7, 300), (150, 9, 255), (1, 6, 1), (1, 100, 1023)])
def test_mask_rows_anywhere(cuda_device, g, sq, sk, offset):
    """Masks whose rows start on any byte, in a tensor that begins and ends on any byte: equal, bit for bit, to the same mask as a
    bias-free general call (a bias tensor of zeros takes the element-wise path)."""
    import torch
    from rocmlir_b200 import _lib as L
    from rocmlir_b200.attention import attention
    gen = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn(s, device="cuda", generator=gen).half() for s in ((g, sq, 64), (g, sk, 64), (g, sk, 64)))
    buf = torch.full((g * sq * sk + 64,), 1, dtype=torch.int8, device="cuda")
    mask = buf[offset:offset + g * sq * sk].view(g, sq, sk)
    mask.copy_((torch.rand((g, sq, sk), device="cuda", generator=gen) > 0.4).to(torch.int8))
    got = attention(q, k, v, trans_k=True, scale=0.125, mask=mask)
    zeros = torch.zeros((g, sq, sk), dtype=torch.float16, device="cuda")
    ref = attention(q, k, v, trans_k=True, scale=0.125, mask=mask.clone(), bias=zeros)
    torch.cuda.synchronize()
    assert torch.equal(got, ref) and L.kernel_status() == 0
