"""Weights and scales that a wrapper copies right before the launch are not fetched ahead of the
kernel that copies them: the call asks for plain stream order (`B200Q_NO_OVERLAP`).  The requests are
recorded on the CPU by a stand-in for the library; the GPU tests run such calls, eagerly and in a
replayed graph whose allocator hands the same addresses to other layers' copies."""

from __future__ import annotations

import contextlib

import pytest
import torch

from linnet_b200 import _lib, kernels
from oracle import linear_oracle as lo

FLAGS_AT = {"b200q_int8_linear_ex": 9, "b200q_int4_linear_ex": 10}


class Recorder:
    """Answers every entry point with OK and keeps the flags of the calls."""

    def __init__(self):
        self.flags = []

    def __getattr__(self, name):
        def call(*args):
            self.flags.append(args[FLAGS_AT[name]])
            return _lib.OK
        return call


@pytest.fixture
def recorder(monkeypatch):
    record = Recorder()
    monkeypatch.setattr(_lib, "load", lambda: record)
    monkeypatch.setattr(kernels, "_on_gpu", lambda who, *tensors: tensors[0].device)
    monkeypatch.setattr(kernels, "_Device", lambda device: contextlib.nullcontext())
    monkeypatch.setattr(kernels, "_stream", lambda device: 0)
    return record


@pytest.mark.parametrize("rows", [1, 8, 40])
def test_int8_copies_ask_for_stream_order(recorder, rows):
    x = torch.zeros(rows, 64, dtype=torch.bfloat16)
    weight, scale = torch.zeros(32, 64, dtype=torch.int8), torch.ones(32)
    call = kernels.gemv8 if rows == 1 else kernels.w8a16
    call(x, weight, scale, False, 0, 1)
    assert recorder.flags == [0]
    for w, s in ((weight, scale.half()), (weight, scale.bfloat16()), (weight, torch.ones(64)[::2]),
                 (torch.zeros(64, 32, dtype=torch.int8).t(), scale)):
        call(x, w, s, False, 0, 1)
    assert recorder.flags[1:] == [_lib.NO_OVERLAP] * 4


def test_int8_entry_takes_the_flag():
    """No launch: no rows."""
    lib = _lib.load()
    arguments = (None, None, None, None, 0, 64, 32, 0, _lib.BF16)
    assert lib.b200q_int8_linear_ex(*arguments, _lib.NO_OVERLAP, None) == _lib.OK
    assert lib.b200q_int8_linear_ex(*arguments, 1 << 10, None) == _lib.ERROR


@pytest.mark.parametrize("rows", [1, 12, 40])
def test_int4_entry_refuses_unknown_flags(rows):
    """Whatever kernel would serve the call; refused before any launch."""
    lib = _lib.load()
    address = 1 << 12
    assert lib.b200q_int4_linear_ex(address, address, address, address, address, rows, 64, 32, 64, _lib.BF16, 1 << 10,
                                    None) == _lib.ERROR
    assert "unknown flag bits" in _lib.last_error()


def int8_layer(depth, out, seed):
    gen = torch.Generator().manual_seed(seed)
    weight = torch.randint(-127, 128, (out, depth), generator=gen, dtype=torch.int8)
    # scales that f16 holds, so that the copy is the only difference
    return weight, (torch.rand(out, generator=gen) * 0.01 + 1e-3).half()


def int8_close(got, x, weight, scale):
    """Against the f64 product: one rounding of each weight and of the result, f32 sums."""
    want = x.double() @ lo.int8_weight(weight, scale.float(), x.dtype).double().T
    torch.testing.assert_close(got.double().cpu(), want, rtol=1e-2, atol=1e-2 * float(want.abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 8, 40])
def test_int8_copied_weights_and_scales(rows):
    """A transposed weight and f16 scales against the same product of tensors kept as they are."""
    depth, out = 1024, 3072
    x = torch.randn(rows, depth, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16)
    layers = [int8_layer(depth, out, seed) for seed in range(3)]
    given = [(w.t().contiguous().cuda().t(), s.cuda()) for w, s in layers]
    kept = [(w.cuda(), s.float().cuda()) for w, s in layers]
    assert not any(w.is_contiguous() for w, _ in given)
    call = kernels.gemv8 if rows == 1 else kernels.w8a16
    inputs = x.cuda()
    want = [call(inputs, w, s, False, 0, 1) for w, s in kept]
    for y, (w, s) in zip(want, layers):
        int8_close(y, x, w, s)

    def forward():
        return [call(inputs, w, s, False, 0, 1) for w, s in given]

    for y, ref in zip(forward(), want):
        assert torch.equal(y, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = forward()
    for _ in range(3):
        graph.replay()
        for y, ref in zip(captured, want):
            assert torch.equal(y, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 4, 12, 40])
@pytest.mark.parametrize("group", [64, 128])
def test_int4_copied_weights(rows, group):
    """Strided packed weights, scales and zero points, through every kernel that few rows reach,
    against the same product of tensors kept as they are."""
    depth, out = 2048, 3000
    gen = torch.Generator().manual_seed(rows + group)
    inputs = torch.randn(rows, depth, generator=gen).to(torch.bfloat16).cuda()
    kept, given = [], []
    for _ in range(3):
        packed = torch.randint(0, 256, (out, depth // group, group // 2), generator=gen, dtype=torch.uint8)
        scale = (torch.rand(out, depth // group, generator=gen) * 0.02 + 1e-3).to(torch.bfloat16)
        zero = torch.randint(0, 16, (out, depth // group), generator=gen, dtype=torch.uint8)
        layer = [t.cuda() for t in (packed, scale, zero)]
        kept.append(layer)
        given.append([torch.stack((t, t), dim=-1)[..., 0] for t in layer])
    assert not any(t.is_contiguous() for layer in given for t in layer)
    want = [kernels.int4_linear(inputs, *layer) for layer in kept]
    for y, ref in zip((kernels.int4_linear(inputs, *layer) for layer in given), want):
        assert torch.equal(y, ref)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = [kernels.int4_linear(inputs, *layer) for layer in given]
    for _ in range(3):
        graph.replay()
        for y, ref in zip(captured, want):
            assert torch.equal(y, ref)
