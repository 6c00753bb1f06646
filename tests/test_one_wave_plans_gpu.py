"""Tile-kernel plans of one-wave problems (33 to 256 tokens): every token tile, block shape and split they choose."""

import pytest
import torch

from full_inference_engine_b200 import _lib
from full_inference_engine_b200.kernels import w4a16_format as w4
from full_inference_engine_b200.kernels import w4a16_linear, w8a16_linear

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("fmt", ["w8", "w4"])
@pytest.mark.parametrize("m", [33, 64, 65, 97, 144, 160, 193, 255, 256])
@pytest.mark.parametrize("n,k", [(128, 512), (1000, 1024), (1024, 2048), (3072, 1024), (2050, 4096), (6144, 1152), (18900, 640)])
def test_matches_the_products_in_64_bits(n, k, m, fmt):
    """2-norm error: the output's one rounding to fp16 (2^-11) and fp32 sums of at most 4096 products (below 1e-5)."""
    torch.manual_seed(n + k + m)
    weight = torch.randn(n, k, device=DEV) * 0.02
    x = torch.randn(m, k, device=DEV).half()
    bias = torch.randn(n, device=DEV).half()
    if fmt == "w8":
        q, scales = w8a16_linear.quantize_weight_per_channel(weight)
        dense = q.double() * scales.double()[:, None]
        y = [w8a16_linear.w8a16_linear(x, q, scales, bias) for _ in range(2)]
    else:
        packed, scales = w4.quantize_weight_w4_grouped(weight)
        half = torch.empty(n, k, dtype=torch.float16, device=DEV)
        dense = w4a16_linear.w4_dequantize_into(half, packed, scales).double()
        y = [w4a16_linear.w4a16_linear(x, packed, scales, bias) for _ in range(2)]
    truth = x.double() @ dense.T + bias.double()
    assert torch.equal(y[0], y[1])
    assert float((y[0].double() - truth).norm() / truth.norm()) <= 2.0 ** -11 + 1e-5
    workspace = _lib.workspace_for(torch.device("cuda", torch.cuda.current_device()), 256)
    assert _lib.library().b200q_workspace_status(workspace.data_ptr(), _lib.stream_ptr(x.device)) == _lib.OK
