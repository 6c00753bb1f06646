"""The CUDA-core kernel starts while its predecessor drains: a chain of dependent calls must not notice."""

import pytest
import torch

from full_inference_engine_b200.kernels import w4a16_format as w4
from full_inference_engine_b200.kernels import w4a16_linear, w8a16_linear

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("fmt", ["w8", "ref", "asym"])
@pytest.mark.parametrize("m,k", [(1, 1024), (1, 2080), (2, 4096), (3, 1056)])
def test_dependent_calls_back_to_back_equal_synchronised_calls(m, k, fmt, static):
    """k columns down to fewer 16-byte vectors than threads, and a remainder in the last round of the K loop."""
    if fmt != "w8":
        k = k // 128 * 128
    torch.manual_seed(k + m)
    layers = []
    for _ in range(6):
        weight = torch.randn(k, k, device=DEV) / k ** 0.5
        if fmt == "w8":
            q, s = w8a16_linear.quantize_weight_per_channel(weight)
            layers.append(lambda x, q=q, s=s: w8a16_linear.w8a16_linear(x, q, s, kernel="gemv", static_weights=static))
        else:
            packed, s, z = (*(w4.quantize_weight_w4_grouped if fmt == "ref" else w4.quantize_weight_w4_asym)(weight), None)[:3]
            layers.append(lambda x, p=packed, s=s, z=z: w4a16_linear.w4a16_linear(
                x, p, s, zeros=z, kernel="gemv", static_weights=static))
    x0 = torch.randn(m, k, device=DEV).half()

    def chain(sync):
        x = x0
        for layer in layers:
            x = layer(x)
            if sync:
                torch.cuda.synchronize()
        return x

    expected = chain(True)
    torch.cuda.synchronize()
    assert torch.equal(chain(False), expected)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = chain(False)
    for _ in range(3):
        graph.replay()
    assert torch.equal(captured, expected)
