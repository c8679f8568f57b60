"""The tensor-core product of 16-bit activations and quantized weights at the sizes where it can go
wrong: one row to several tiles of rows, K that ends in half an item (64 of 128 inputs), one item
a tile, ragged N, every group size it takes, both 16-bit types, scales at the ends of their range,
values that are not finite."""

from __future__ import annotations

import pytest
import torch

from oracle import linear_oracle as lo

pytestmark = pytest.mark.gpu


def make_int4(out, depth, group, dtype, gen, magnitude=1.0):
    packed = torch.randint(0, 256, (out, depth // group, group // 2), generator=gen, dtype=torch.uint8)
    scale = ((torch.rand(out, depth // group, generator=gen) * 0.9 + 0.1) * magnitude).to(dtype)
    zero = torch.randint(0, 16, (out, depth // group), generator=gen, dtype=torch.uint8)
    return packed, scale, zero


def make_int8(out, depth, group, gen):
    weight = torch.randint(-128, 128, (out, depth), generator=gen, dtype=torch.int8)
    return weight, torch.rand(out, depth // (group or depth), generator=gen) * 0.01 + 1e-4


def check(got, x, w):
    """Against the f64 product of the same rounded weights: one rounding to the result's type plus
    f32 sums of `depth` products, each addition off by at most an ulp (2^-23, the tensor cores
    truncate) of the sum of magnitudes."""
    exact = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    ulp = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -11
    bound = ulp * exact.abs() + x.shape[1] * 2.0 ** -23 * size + 1e-30
    assert bool(((got.double().cpu() - exact).abs() <= 1.01 * bound).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("group", [16, 32, 64, 128, 384])
def test_int4_weights_are_exact(dtype, group):
    """The identity times W^T is W bit for bit, also where the fast conversion's power of two would
    leave the type's range (scales near its largest value) and for subnormal scales."""
    from linnet_b200 import kernels

    depth, out = 768, 200
    gen = torch.Generator().manual_seed(group)
    top = 2.0 ** 124 if dtype == torch.bfloat16 else 2000.0  # 15 times the scale is still finite
    for magnitude in (0.01, top, 2.0 ** -130 if dtype == torch.bfloat16 else 2.0 ** -20):
        packed, scale, zero = make_int4(out, depth, group, dtype, gen, magnitude)
        got = kernels.int4_linear(torch.eye(depth, dtype=dtype).cuda(), packed.cuda(), scale.cuda(), zero.cuda())
        want = lo.int4_weight(packed, scale, zero, dtype)
        assert torch.equal(got.t().cpu().float(), want.float())


# (rows, depth, out): few rows (the smallest stay with the decode kernels), a last item of half, wide
# and narrow weights, short and long K, several tiles of rows with a ragged last one.  Which tile shape
# and K split a size gets is the cost model's choice.
SHAPES = [(1, 64, 128), (9, 128, 100), (17, 192, 1000), (33, 4160, 130), (64, 4096, 512), (16, 1024, 28680),
          (100, 320, 20000), (200, 448, 3000), (256, 1088, 4096), (257, 640, 5000), (1000, 256, 9001)]


@pytest.mark.parametrize(("rows", "depth", "out"), SHAPES)
@pytest.mark.parametrize(("group", "dtype"), [(64, torch.bfloat16), (32, torch.float16), (16, torch.bfloat16)])
def test_int4_product(rows, depth, out, group, dtype):
    from linnet_b200 import kernels

    gen = torch.Generator().manual_seed(rows + depth + out + group)
    packed, scale, zero = make_int4(out, depth, group, dtype, gen, 0.02)
    x = torch.randn(rows, depth, generator=gen).to(dtype)
    got = kernels.int4_linear(x.cuda(), packed.cuda(), scale.cuda(), zero.cuda())
    check(got, x, lo.int4_weight(packed, scale, zero, dtype))


@pytest.mark.parametrize(("rows", "depth", "out"), SHAPES)
@pytest.mark.parametrize(("group", "dtype"), [(0, torch.bfloat16), (32, torch.bfloat16), (64, torch.float16)])
def test_int8_product(rows, depth, out, group, dtype):
    from linnet_b200 import quantized

    if rows <= 2 and not group:
        pytest.skip("one or two rows with one scale a row run another kernel")
    gen = torch.Generator().manual_seed(rows + depth + out + group)
    weight, scale = make_int8(out, depth, group, gen)
    x = torch.randn(rows, depth, generator=gen).to(dtype)
    if group:
        got = quantized.int8_group_linear(x.cuda(), quantized.int8_group_operands(weight.cuda(), scale.cuda()), None)
    else:
        got = quantized.int8_linear(x.cuda(), quantized.int8_operands(weight.cuda(), scale.cuda(), 0), None)
    check(got, x, lo.int8_weight(weight, scale if group else scale.reshape(-1), dtype))


# One item of half or whole size a tile, for one tile in all and for three and more tiles a block, so
# that a tile's single item falls to either issuer and accumulator.
ONE_ITEM = [(16, 64, 128), (16, 128, 100), (16, 64, 60000), (16, 128, 60000), (16, 128, 75001), (40, 64, 57000),
            (70, 128, 60000), (200, 128, 60000), (256, 64, 58000)]


@pytest.mark.parametrize(("rows", "depth", "out"), ONE_ITEM)
@pytest.mark.parametrize(("group", "dtype"), [(64, torch.bfloat16), (16, torch.float16)])
def test_int4_one_item_a_tile(rows, depth, out, group, dtype):
    test_int4_product(rows, depth, out, group, dtype)


@pytest.mark.parametrize(("rows", "depth", "out"), ONE_ITEM)
@pytest.mark.parametrize(("group", "dtype"), [(0, torch.float16), (64, torch.bfloat16), (16, torch.bfloat16)])
def test_int8_one_item_a_tile(rows, depth, out, group, dtype):
    test_int8_product(rows, depth, out, group, dtype)


@pytest.mark.parametrize("group", [16, 48 * 16, 0])
def test_int8_groups(group):
    """The smallest group, one that is no power of two, and one scale a row, over a K that ends in half
    an item."""
    for rows in (16, 33, 150):
        test_int8_product(rows, 768 * 3 + (0 if group > 16 else 64), 1500, group, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows", [20, 80])
def test_infinities_and_nan_stay_where_they_are(rows, dtype):
    """An activation that is not finite makes its own row not finite, a scale its own column; every
    other result is as without them."""
    from linnet_b200 import kernels

    depth, out, group = 512, 700, 64
    gen = torch.Generator().manual_seed(rows)
    packed, scale, zero = make_int4(out, depth, group, dtype, gen, 0.02)
    zero = zero.clamp(max=14)  # a level equal to the zero point would make 0 times infinity
    packed |= 0xFF             # every level is 15
    weight, scale8 = make_int8(out, depth, group, gen)
    weight = weight.clamp(min=1)
    x = torch.randn(rows, depth, generator=gen).to(dtype)
    odd, odd4, odd8 = x.clone(), scale.clone(), scale8.clone()
    odd[3, 5], odd[7, 100] = float("inf"), float("nan")
    odd4[11, 2], odd4[600, 0] = float("inf"), float("nan")
    odd8[11, 2], odd8[600, 0] = float("inf"), float("nan")
    calls = [(lambda x, s: kernels.int4_linear(x.cuda(), packed.cuda(), s.cuda(), zero.cuda()), scale, odd4),
             (lambda x, s: kernels.w8a16(x.cuda(), weight.cuda(), s.cuda(), False, group, 1), scale8, odd8)]
    for call, plain, spoiled in calls:
        want = call(x, plain).cpu()
        got = call(odd, plain).cpu()
        rest = [i for i in range(rows) if i not in (3, 7)]
        assert not bool(torch.isfinite(got[[3, 7]]).any()) and bool(torch.isinf(got[3]).all())
        assert torch.equal(got[rest], want[rest])
        got = call(x, spoiled).cpu()
        rest = [i for i in range(out) if i not in (11, 600)]
        assert bool(torch.isnan(got[:, 600]).all()) and not bool(torch.isfinite(got[:, 11]).any())
        assert torch.equal(got[:, rest], want[:, rest])


def test_slow_scales_do_not_outrun_the_weights():
    """Groups of 32 over a wide weight, many launches: the scattered scale loads keep the load unit
    busy while the stages of packed weights are handed back (results are the same every time)."""
    from linnet_b200 import _lib, kernels

    gen = torch.Generator().manual_seed(2)
    packed, scale, zero = (t.cuda() for t in make_int4(14336, 4096, 32, torch.bfloat16, gen, 0.02))
    x = torch.randn(300, 4096, generator=gen).to(torch.bfloat16).cuda()
    first = kernels.int4_linear(x, packed, scale, zero)
    check(first[:, :256], x.cpu(), lo.int4_weight(packed[:256].cpu(), scale[:256].cpu(), zero[:256].cpu(), torch.bfloat16))
    for _ in range(10):
        assert torch.equal(kernels.int4_linear(x, packed, scale, zero), first)
    assert _lib.load().b200q_int4_gemm_status() == 0


def test_unaligned_activations_keep_the_library_route():
    """int8 rows that do not start on 16 bytes: what the tiled copies cannot read is still taken."""
    from linnet_b200 import kernels, quantized

    gen = torch.Generator().manual_seed(4)
    weight, scale = make_int8(256, 512, 0, gen)
    x = torch.randn(100 * 512 + 1, generator=gen).to(torch.bfloat16)
    inner = x.cuda()[1:].view(100, 512)
    operands = quantized.int8_operands(weight.cuda(), scale.cuda(), 0)
    assert not kernels.w8a16_any_rows(inner, operands[0], operands[1], 0)
    got = quantized.int8_linear(inner, operands, None)
    check(got, x[1:].view(100, 512), lo.int8_weight(weight, scale.reshape(-1), torch.bfloat16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize(("rows", "depth", "out"), [
    (9, 8192, 5120), (16, 8192, 7168), (12, 4096, 14336), (16, 12288, 4608),  # the decode kernel's
    (9, 4096, 16384), (16, 8192, 8192), (12, 2048, 5120), (16, 1024, 1024), (11, 7168, 2050), (17, 8192, 5120),  # the product's
])
def test_int4_nine_to_sixteen_rows(rows, depth, out, dtype):
    """Either kernel may take these rows of groups of 128, by its estimated time; both round every
    weight once."""
    from linnet_b200 import kernels

    gen = torch.Generator().manual_seed(rows + depth + out)
    packed, scale, zero = make_int4(out, depth, 128, dtype, gen, 0.02)
    x = torch.randn(rows, depth, generator=gen).to(dtype)
    check(kernels.int4_linear(x.cuda(), packed.cuda(), scale.cuda(), zero.cuda()), x, lo.int4_weight(packed, scale, zero, dtype))


@pytest.mark.parametrize(("rows", "depth", "out", "dtype"), [
    (17, 1536, 4096, torch.bfloat16), (18, 5632, 1000, torch.bfloat16), (33, 1536, 4096, torch.float16),
    (50, 2560, 4096, torch.float16), (65, 2048, 4096, torch.float16), (130, 4096, 4096, torch.float16),
])
def test_int4_rows_past_the_passes_keep_unrounded_weights(rows, depth, out, dtype):
    """The one or two rows that passes of the decode kernels leave over come from the one- and
    two-row kernel, bit for bit, which takes zero points and scales unrounded."""
    from linnet_b200 import kernels

    gen = torch.Generator().manual_seed(rows + depth)
    packed, scale, zero = (t.cuda() for t in make_int4(out, depth, 128, dtype, gen, 0.02))
    x = torch.randn(rows, depth, generator=gen).to(dtype).cuda()
    last = rows % 16
    got = kernels.int4_linear(x, packed, scale, zero)
    assert torch.equal(got[-last:], kernels.int4_linear(x[-last:], packed, scale, zero))
    check(got[:-last], x[:-last].cpu(), lo.int4_weight(packed.cpu(), scale.cpu(), zero.cpu(), dtype))


@pytest.mark.parametrize(("rows", "dtype"), [(17, torch.bfloat16), (18, torch.float16), (33, torch.float16),
                                             (34, torch.bfloat16), (50, torch.bfloat16), (66, torch.bfloat16)])
def test_int8_rows_past_the_passes_keep_unrounded_weights(rows, dtype):
    """The same for int8 with one scale a row, at any row count of `w8a16`; an int8 layer past the
    rows `w8a16` is tiled for rounds every weight, as its dense route does."""
    from linnet_b200 import kernels, quantized

    depth, out = 4096, 3000
    gen = torch.Generator().manual_seed(rows)
    weight, scale = make_int8(out, depth, 0, gen)
    x = torch.randn(rows, depth, generator=gen).to(dtype)
    w, s, rounded = weight.cuda(), scale.reshape(-1).cuda(), lo.int8_weight(weight, scale.reshape(-1), dtype)
    last = rows % 16
    got = kernels.w8a16(x.cuda(), w, s, False, 0, 1)
    few = kernels.gemv8 if last == 1 else kernels.w8a16
    assert torch.equal(got[-last:], few(x[-last:].cuda(), w, s, False, 0, 1))
    check(got[:-last], x[:-last], rounded)
    if rows > quantized.TILED_ROWS:
        check(quantized.int8_linear(x.cuda(), quantized.int8_operands(w, s, 0), None), x, rounded)
