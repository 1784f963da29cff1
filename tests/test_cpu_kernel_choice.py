"""What the layers tell the kernels, and which kernel a call takes: rules on the host, checked without a GPU."""
import pytest
import torch

from omni_npu_b200 import ops
from omni_npu_b200.layers.linear import Fp8BlockLinearMethod, UnquantizedLinearMethod
from omni_npu_b200.layers.quant_fp8 import fp8_block_gemm, quantize_weight_block


def _record(monkeypatch, name):
    calls, real = [], getattr(ops, name)

    def wrapped(*a, **k):
        calls.append(k)
        return real(*a, **k)

    monkeypatch.setattr(ops, name, wrapped)
    return calls


def test_only_parameters_are_read_ahead_of_the_kernels_before(monkeypatch):
    """A product may load its weights early only where the caller says that no kernel writes them: a layer's parameters,
    not the expanded copy of e4m3 weights that is made right ahead of the product."""
    calls = _record(monkeypatch, "gemm")
    x, layer = torch.randn(3, 64), torch.nn.Module()
    layer.weight = torch.nn.Parameter(torch.randn(32, 64), requires_grad=False)
    UnquantizedLinearMethod().apply(layer, x, None)
    assert calls.pop()["w_ready"] is True
    wq, ws = quantize_weight_block(torch.randn(32, 64))
    layer.weight, layer.weight_scale_inv = (torch.nn.Parameter(t, requires_grad=False) for t in (wq, ws))
    Fp8BlockLinearMethod().apply(layer, x, None)
    fp8_block_gemm(x, wq, ws, w_ready=True)
    assert len(calls) == 2 and not any(c.get("w_ready", False) for c in calls)
