"""The stream-K kernel's warp-level multiply: every token-tile width, ragged channels, and its argmax."""

import numpy as np
import pytest
import torch

from full_inference_engine_b200 import _lib
from full_inference_engine_b200.kernels import argmax
from full_inference_engine_b200.kernels import w4a16_format as w4
from full_inference_engine_b200.kernels import w4a16_linear, w8a16_linear

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _weights(fmt, n, k):
    weight = torch.randn(n, k, device=DEV) * 0.02
    if fmt == "w8":
        q, scales = w8a16_linear.quantize_weight_per_channel(weight)
        return (q, scales, None), q.double() * scales.double()[:, None]
    quantize = w4.quantize_weight_w4_grouped if fmt == "ref" else w4.quantize_weight_w4_asym
    packed, scales, zeros = (*quantize(weight), None)[:3]
    dense = torch.empty(n, k, dtype=torch.float16, device=DEV)
    w4a16_linear.w4_dequantize_into(dense, packed, scales, zeros=zeros)
    return (packed, scales, zeros), dense.double()


def _forward(fmt, x, weights, **kw):
    if fmt == "w8":
        return w8a16_linear.w8a16_linear(x, weights[0], weights[1], kernel="streamk", **kw)
    return w4a16_linear.w4a16_linear(x, weights[0], weights[1], zeros=weights[2], kernel="streamk", **kw)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("fmt", ["ref", "asym", "w8"])
@pytest.mark.parametrize("m,n,k", [(1, 130, 1024), (8, 4099, 2048), (9, 1027, 5120), (16, 640, 1024), (17, 2050, 3072),
                                   (32, 1285, 4096), (33, 384, 1024), (48, 777, 2048), (49, 129, 1024), (64, 1030, 2048)])
def test_every_tile_width_is_as_exact_as_its_output_type(m, n, k, fmt, dtype):
    """2-norm error against the products in 64 bits.  What is rounded: the output, once (relative error at most
    2^-11 in fp16, 2^-8 in bf16; 2^-11 / sqrt(3) and 2^-8 / sqrt(3) in the mean over a binade's worst end), and,
    for 4-bit weights with bf16 activations, the format's fp16 products, which the kernel does not round (2^-11).
    Sums of at most 5120 products in fp32 stay below 1e-5 of the result."""
    torch.manual_seed(m * n + k)
    weights, dense = _weights(fmt, n, k)
    x = torch.randn(m, k, device=DEV).to(dtype)
    truth = x.double() @ dense.T
    for _ in range(2):                                   # the second call sees what the first left behind
        y = _forward(fmt, x, weights)
        err = float((y.double() - truth).norm() / truth.norm())
        assert err <= (2.0 ** -11 if dtype is torch.float16 else 2.0 ** -8) / 3 ** 0.5 + 2.0 ** -12 + 1e-5
    assert torch.equal(y, _forward(fmt, x, weights))
    workspace = _lib.workspace_for(torch.device("cuda", torch.cuda.current_device()), 256)
    assert _lib.library().b200q_workspace_status(workspace.data_ptr(), _lib.stream_ptr(x.device)) == _lib.OK
    assert not bool(workspace[128 * 1024:128 * 1024 + 5 * 1024 * 1024].any()), "the exchange region was not left empty"


def test_int8_extremes_are_exact_in_both_types():
    """Every int8 value against one-hot activations: integers below 2^8 are exact in fp16 and bf16."""
    n, k = 256, 1024
    q = (torch.arange(n * k, device=DEV) % 256 - 128).to(torch.int8).reshape(n, k)
    q = torch.roll(q, 3, 0)
    for dtype in (torch.float16, torch.bfloat16):
        x = torch.zeros(16, k, device=DEV, dtype=dtype)
        for row in range(16):
            x[row, (row * 67) % k] = 1.0
        y = w8a16_linear.w8a16_linear(x, q, torch.ones(n, device=DEV), kernel="streamk")
        assert torch.equal(y.float(), x.float() @ q.float().T)


@pytest.mark.parametrize("fmt", ["ref", "w8"])
@pytest.mark.parametrize("m", [1, 9, 31, 32])
def test_argmax_takes_the_route_of_the_plain_call(m, fmt):
    """A head large enough for the stream-K kernel: the fused argmax is the plain call's, ties to the smallest channel."""
    torch.manual_seed(m)
    n, k = 12005, 2048
    weights, _ = _weights(fmt, n, k)
    for dtype in (torch.float16, torch.bfloat16):
        x = torch.randn(m, k, device=DEV).to(dtype)
        if fmt == "w8":
            dense, picked = (w8a16_linear.w8a16_linear(x, weights[0], weights[1], _argmax=a) for a in (False, True))
            if m == 1:                                   # a single int8 row may be the CUDA-core kernel's
                dense = w8a16_linear.w8a16_linear(x, weights[0], weights[1], kernel="dot")
        else:
            dense = w4a16_linear.w4a16_linear(x, weights[0], weights[1])
            picked = argmax.w4a16_linear_argmax(x, weights[0], weights[1])
        assert torch.equal(picked, dense.argmax(dim=-1))
        zeros = torch.zeros_like(x)
        if fmt == "ref":
            assert not bool(argmax.w4a16_linear_argmax(zeros, weights[0], weights[1]).any())


def test_shared_scale_chunks_of_a_deep_matrix_restart_at_a_tile():
    """One-hot columns read single weights back across chunk and tile boundaries."""
    n, k = 300, 2048
    packed, scales = w4.quantize_weight_w4_grouped(torch.randn(n, k, device=DEV) * 0.3)
    dense = w4.unpack_w4_reference(packed, scales, k) if hasattr(w4, "unpack_w4_reference") else None
    x = torch.zeros(8, k, device=DEV, dtype=torch.float16)
    columns = [0, 63, 64, 127, 128, 1023, 1024, k - 1]
    for row, column in enumerate(columns):
        x[row, column] = 1.0
    y = w4a16_linear.w4a16_linear(x, packed, scales, kernel="streamk")
    if dense is None:
        dense = torch.empty(n, k, dtype=torch.float16, device=DEV)
        w4a16_linear.w4_dequantize_into(dense, packed, scales)
    assert np.array_equal(y.cpu().numpy(), dense[:, columns].T.half().cpu().numpy())
