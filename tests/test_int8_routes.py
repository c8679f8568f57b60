"""The route of an int8 layer past the rows `w8a16` is tiled for, looked at on the CPU: as one op of a
full graph under `torch.compile`."""

from __future__ import annotations

import pytest
import torch

from linnet_b200 import quantized


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
