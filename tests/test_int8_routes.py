"""The route of an int8 layer past the rows `w8a16` is tiled for, looked at on the CPU: as one op of a
full graph under `torch.compile`, and with derivatives."""

from __future__ import annotations

import pytest
import torch
from torch.autograd import forward_ad

from linnet_b200 import kernels, quantized


@pytest.mark.parametrize("group", [0, 32])
@pytest.mark.parametrize("rows", [1, 64, 65, 200])
def test_traced_as_a_full_graph(rows, group):
    """The trace holds one product op, whatever the addresses will be."""
    seen = []

    def record(module, inputs):
        seen.extend(str(node.target) for node in module.graph.nodes if node.op == "call_function")
        return lambda *args: (torch.zeros(rows, 48, dtype=torch.bfloat16),)

    weight = torch.zeros(48, 128, dtype=torch.int8)
    scale = torch.ones(48, 128 // group) if group else torch.ones(48)
    torch._dynamo.reset()
    compiled = torch.compile(lambda x: quantized._weight_only(x, weight, scale, group), backend=record, fullgraph=True)
    y = compiled(torch.zeros(rows, 128, dtype=torch.bfloat16))
    assert y.shape == (rows, 48)
    want = "gemv8" if rows == 1 else "w8a16" if rows <= quantized.TILED_ROWS else "w8a16_many"
    assert [name for name in seen if name.startswith("linnet.")] == [f"linnet.{want}.default"]


DENSE = torch.randn(48, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16)


@pytest.fixture
def dense_only(monkeypatch):
    """A stand-in for the dequantized weight; the kernels themselves must not be reached."""
    def refuse(*args, **kwargs):
        raise AssertionError("a kernel without a derivative was reached")

    monkeypatch.setattr(kernels, "dequantize8", lambda *args: DENSE)
    monkeypatch.setattr(kernels, "w8a16_any_rows", lambda *args: True)
    monkeypatch.setattr(kernels, "_eight_bit", refuse)
    weight, scale = torch.zeros(48, 128, dtype=torch.int8), torch.ones(48)
    return lambda x: quantized._weight_only(x, weight, scale)


def test_derivatives_past_the_tiled_rows(dense_only):
    """The gradient with respect to the activations, backward and forward, and batched rows."""
    gen = torch.Generator().manual_seed(2)
    x = torch.randn(70, 128, generator=gen).to(torch.bfloat16)
    g = torch.randn(70, 48, generator=gen).to(torch.bfloat16)
    leaf = x.clone().requires_grad_()
    dense_only(leaf).backward(g)
    torch.testing.assert_close(leaf.grad, g @ DENSE)
    with forward_ad.dual_level():
        tangent = forward_ad.unpack_dual(dense_only(forward_ad.make_dual(x, x))).tangent
        torch.testing.assert_close(tangent, x @ DENSE.T)
    torch.testing.assert_close(torch.func.jvp(dense_only, (x,), (x,))[1], x @ DENSE.T)
    torch.testing.assert_close(torch.func.vmap(dense_only)(torch.stack((x, x)))[1], x @ DENSE.T)


def test_nothing_to_differentiate_takes_the_kernel(dense_only):
    with pytest.raises(AssertionError, match="without a derivative"):
        dense_only(torch.zeros(70, 128, dtype=torch.bfloat16))
    with torch.no_grad(), pytest.raises(AssertionError, match="without a derivative"):
        dense_only(torch.zeros(70, 128, dtype=torch.bfloat16, requires_grad=True))
