"""The one- and two-row kernels where a warp takes several items of a tile and a block's last round of
tiles is short: a warp whose last tile lies in the round before still counts that round as a whole
one when it looks for its stage of the ring."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

# (inputs, tiles of 16 rows a block, 148 blocks): items a warp and tile, warps a tile, tiles in work
INT8 = [(5376, 3),    # 3, 7, 2
        (6400, 4),    # 5, 5, 3
        (6400, 5),
        (8704, 9)]    # 17, 2, 8
INT4 = [(10752, 3),   # 3, 7, 2
        (12800, 4),   # 5, 5, 3
        (12800, 5),
        (8704, 18)]   # 17, 1, 16


def check(got, x, w):
    """Against the f64 product of the unrounded weights: one rounding of the result (2^-9 of it at the
    worst, 2^-10 on average) and f32 sums; a stage read in the wrong place is off by about 1."""
    from linnet_b200 import _lib

    _lib.check(_lib.load().b200q_int4_gemm_status())
    want = x.double() @ w.T
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 2])
@pytest.mark.parametrize(("depth", "tiles"), INT8)
def test_int8(depth, tiles, rows, dtype):
    from linnet_b200 import kernels

    gen = torch.Generator(device="cuda").manual_seed(depth + tiles)
    for out in (16 * 148 * tiles, 16 * 148 * tiles - 1000):  # blocks with one tile less too
        w = torch.randint(-127, 128, (out, depth), device="cuda", dtype=torch.int8, generator=gen)
        s = torch.rand(out, device="cuda", generator=gen) * 0.01 + 1e-3
        x = torch.randn(rows, depth, device="cuda", generator=gen).to(dtype)
        got = (kernels.gemv8 if rows == 1 else kernels.w8a16)(x, w, s, False, 0, 1)
        check(got, x, w.double() * s.double()[:, None])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [1, 2])
@pytest.mark.parametrize(("depth", "tiles"), INT4)
def test_int4(depth, tiles, rows, dtype):
    from linnet_b200 import kernels

    gen = torch.Generator(device="cuda").manual_seed(depth + tiles)
    groups = depth // 128
    for out in (16 * 148 * tiles, 16 * 148 * tiles - 1000):
        packed = torch.randint(0, 256, (out, groups, 64), device="cuda", dtype=torch.uint8, generator=gen)
        scale = (torch.rand(out, groups, device="cuda", generator=gen) * 0.02 + 1e-3).to(dtype)
        zero = torch.randint(0, 16, (out, groups), device="cuda", dtype=torch.uint8, generator=gen)
        x = torch.randn(rows, depth, device="cuda", generator=gen).to(dtype)
        levels = torch.stack((packed & 15, packed >> 4), dim=-1).reshape(out, groups, 128)
        w = ((levels.short() - zero.short()[..., None]).double() * scale.double()[..., None]).reshape(out, depth)
        check(kernels.int4_linear(x, packed, scale, zero), x, w)
