"""The vector forms of the quantizers and the dequantizer at the edges of their dispatch: rows that
cross a warp's run of groups, ragged block tails, rows longer than a block holds in registers,
quotients at and next to half-integers (where the reciprocal cannot decide), unaligned views and
odd widths (the element-wise kernels).  Everything is bit for bit against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from full_inference_engine_b200.kernels import w4a16_format as w4
from full_inference_engine_b200.kernels import w4a16_linear, w8a8_linear, w8a16_linear
from oracle import wq_oracle as oracle
from tests.helpers import bits_equal, to_np

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float16, torch.float32]


def _near_ties(n: int, k: int) -> torch.Tensor:
    """Rows whose quotients sit on half-integers, or one ulp to either side of them."""
    steps = torch.arange(n * k).reshape(n, k) % 14 - 7 + 0.5
    scale = torch.tensor([0.25, 0.3, 1.7e-3])[torch.arange(n) % 3][:, None]
    w = (steps * scale).float()
    w[:, 0::128] = 7.0 * scale                  # the group maximum: s = scale up to rounding
    toward = torch.where(torch.arange(n * k).reshape(n, k) % 3 == 0, float("inf"), 0.0)
    return torch.where(torch.arange(n * k).reshape(n, k) % 2 == 0, w, torch.nextafter(w, toward))


def _weights(kind: str, n: int, k: int, dtype: torch.dtype) -> torch.Tensor:
    torch.manual_seed(n * 31 + k)
    if kind == "ties":
        return _near_ties(n, k).to(dtype)
    w = torch.randn(n, k) * 0.02
    if kind == "odd":
        w[0] = 0.0
        w[-1] *= 1e-6                           # scales in fp16's subnormal range
        w[n // 2, : k // 2] = 0.0
    return w.to(dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(1, 128), (5, 384), (37, 896), (64, 4096), (3, 12416)])
@pytest.mark.parametrize("kind", ["odd", "ties"])
def test_w4_group128(kind, shape, dtype):
    w = _weights(kind, *shape, dtype)
    packed, scales = w4.quantize_weight_w4_grouped(w.cuda())
    rp, rs = oracle.quantize_w4_grouped(to_np(w))
    assert bits_equal(packed, rp) and bits_equal(scales, rs)
    out = torch.full(shape, float("nan"), device="cuda", dtype=torch.float16)
    w4a16_linear.w4_dequantize_into(out, packed, scales)
    assert bits_equal(out, oracle.unpack_w4(rp, rs, shape[1]))
    packed, scales, zeros = w4.quantize_weight_w4_asym(w.cuda())
    rp, rs, rz = oracle.quantize_w4_asym(to_np(w))
    rz = rz + np.float16(0)                     # an all-zero group: the oracle says -0, the kernels +0
    assert bits_equal(packed, rp) and bits_equal(scales, rs) and bits_equal(zeros, rz)
    w4a16_linear.w4_dequantize_into(out, packed, scales, zeros=zeros)
    assert bits_equal(out, oracle.unpack_w4_asym(rp, rs, rz, shape[1]))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("shape", [(1, 8), (5, 1000), (7, 2056), (3, 12288), (2, 13000), (4, 1001)])
def test_w8_rows(shape, dtype):
    w = _weights("odd" if shape[0] > 1 else "plain", *shape, dtype)
    q, s = w8a16_linear.quantize_weight_per_channel(w.cuda())
    rq, rs = oracle.quantize_w8_per_channel(to_np(w))
    assert bits_equal(q, rq) and bits_equal(s, rs)
    q, s = w8a16_linear.quantize_weight_per_channel_fp32_scales(w.cuda())
    rq, rs = oracle.quantize_w8_int8linear(to_np(w))
    assert bits_equal(q, rq) and bits_equal(s, rs)


def test_unaligned_weight_views_take_the_element_wise_kernels():
    torch.manual_seed(2)
    big = (torch.randn(24, 1032) * 0.02).to(torch.bfloat16).cuda()
    view = big[:, 4:4 + 1024 - 4 * 128]          # rows start 8 bytes off a 16-byte boundary
    packed, scales = w4.quantize_weight_w4_grouped(view)
    rp, rs = oracle.quantize_w4_grouped(to_np(view))
    assert bits_equal(packed, rp) and bits_equal(scales, rs)
    q, s = w8a16_linear.quantize_weight_per_channel(view)
    rq, rs = oracle.quantize_w8_per_channel(to_np(view))
    assert bits_equal(q, rq) and bits_equal(s, rs)
    out = torch.full((24, 520), float("nan"), device="cuda", dtype=torch.float16)[:, 4:516]
    w4a16_linear.w4_dequantize_into(out, packed, scales)
    assert bits_equal(out, oracle.unpack_w4(to_np(packed), to_np(scales), 512))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shape", [(3, 8), (65, 2048), (70, 2056), (2, 12288), (2, 13000), (64, 16)])
def test_activation_rows(shape, dtype):
    torch.manual_seed(shape[1])
    x = (torch.randn(shape) * 3).to(dtype)
    x[0, 1:] = x[0, 0] * (torch.arange(1, shape[1]) % 127 + 0.5).to(dtype) / 127      # next to half steps
    q, scales = w8a8_linear.quantize_activations_per_row(x.cuda())
    rq, rs = oracle.quantize_rows_int8(to_np(x))
    assert np.array_equal(q.cpu().numpy(), rq) and bits_equal(scales, rs)
