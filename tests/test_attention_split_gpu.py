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


@pytest.mark.parametrize("fill", [float("-inf"), -1000.0, float(np.finfo(np.float32).min)])
@pytest.mark.parametrize("g,sq,sk,d,dv", [(3, 4, 1040, 128, 128), (2, 4, 1001, 64, 64), (150, 2, 272, 64, 64)])
def test_split_keys_with_mask(cuda_device, g, sq, sk, d, dv, fill):
    """Mask rows on 16-byte boundaries (read as words) and off them; a row without any key left, and one whose keys all lie
    in the first block, so that the other CTAs of the cluster contribute nothing."""
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
