"""The fp16 contraction kernel (neoml_b200/csrc/contraction_split.cu) at the edges of its tiles and of its number range.

Bound of the comparison, against sums in double precision and relative to sum |a||b| of each result: three split errors of
at most 2^-22, and one truncation of at most 2^-22 for each of the ceil(K / 16) accumulations (main and cross) and for the
epilogue's four roundings."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from neoml_b200 import ops as module
    return module


def bound(k: int) -> float:
    return (3 + math.ceil(k / 16) + 4) * 2.0 ** -22


def worst(got, a, b, extra=None):
    want = a.double() @ b.double().transpose(-1, -2)
    size = a.abs().double() @ b.abs().double().transpose(-1, -2)
    if extra is not None:
        want, size = want + extra.double(), size + extra.abs().double()
    assert bool((got[size == 0] == 0).all())
    return float(((got.double() - want).abs() / size.clamp_min(1e-300)).max())


def rows_of(kind: str, m: int, k: int, g) -> torch.Tensor:
    a = torch.empty(m, k, device="cuda").normal_(generator=g)
    if kind == "zeros":          # rows without anything, rows that begin with empty K blocks, a ReLU's half
        a.clamp_(min=0)
        a[::2, : k // 2] = 0
        a[::5] = 0
    elif kind == "scales":       # every row of another magnitude
        a *= torch.logspace(-30, 30, m, device="cuda")[:, None]
    elif kind == "rising":       # every K block beyond the range of the one before: the row scales move in mid-tile
        a *= torch.pow(2.0, 7.0 * (torch.arange(k, device="cuda") // 32).clamp(max=12))
    elif kind == "jump":         # some rows of a warp move, others do not; the last block included
        a[::3, k // 2:] *= 1e4
        a[1::7, k - 1] *= 1e6
    return a


# m x k x n: 75 row tiles are the fewest that one column tile takes to this kernel, 160 = five K blocks the shortest depth; the
# last four have few tiles and split K (into 2, 8, with 33 K blocks 3, and 4 parts)
@pytest.mark.parametrize("m,k,n", [(75 * 128 - 127, 160, 32), (9700, 132, 57), (9600, 190, 64), (9601, 576, 96), (4800, 320, 129),
                                   (1024, 333 * 4, 1300), (5000, 2064, 260), (4116, 1024, 256),
                                   (1029, 2304, 128), (1100, 1044, 132), (1024, 768, 512)])
@pytest.mark.parametrize("kind", ["normal", "zeros", "scales", "rising", "jump"])
def test_products(ops, m, k, n, kind):
    g = torch.Generator(device="cuda")
    g.manual_seed(m + k)
    a, b = rows_of(kind, m, k, g), torch.empty(n, k, device="cuda").normal_(generator=g)
    b *= torch.logspace(-3, 3, n, device="cuda")[:, None]
    got = ops.MultiplyMatrixByTransposedMatrix(a, b)
    assert worst(got, a, b) < bound(k)
    assert torch.equal(got, ops.MultiplyMatrixByTransposedMatrix(a, b))
    if kind in ("normal", "jump"):
        bias, res = torch.empty(n, device="cuda").normal_(generator=g), torch.empty(m, n, device="cuda").normal_(generator=g)
        got = ops.MultiplyMatrixByTransposedMatrix(a, b, free_term=bias, residual=res)
        assert worst(got, a, b, extra=bias + res) < bound(k)


@pytest.mark.parametrize("m,k,n", [(9601, 160, 40), (1100, 1044, 132)])
def test_tiny_rows(ops, m, k, n):
    """Rows whose first K block, or which altogether, lie at the lower end of fp32; zeros among them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    a, b = torch.empty(m, k, device="cuda").normal_(generator=g), torch.empty(n, k, device="cuda").normal_(generator=g)
    a[:, :32] *= torch.logspace(-37, -30, m, device="cuda")[:, None]
    a[:, 1:32:3] = 0
    first = a[:, :32].clone()
    a[::7, :32] *= 1e-6       # with the line before: a first block of zeros and subnormal numbers for some
    b[::3] *= torch.logspace(-33, -29, b[::3].shape[0], device="cuda")[:, None]
    b[::3, ::4] = 0
    got = ops.MultiplyMatrixByTransposedMatrix(a, b)
    assert bool(torch.isfinite(got).all()) and worst(got, a, b) < bound(k)
    a[::2, 32:] = 0           # nothing but the tiny block
    a[:, :32] = first
    b[::3] = torch.empty(b[::3].shape, device="cuda").normal_(generator=g) * 1e33
    got = ops.MultiplyMatrixByTransposedMatrix(a, b)
    assert bool(torch.isfinite(got).all()) and worst(got[:, ::3], a, b[::3]) < bound(k)


@pytest.mark.parametrize("m,k,n", [(9601, 160, 40), (4800, 192, 129), (1100, 1044, 132)])
def test_both_scales_over_the_whole_range(ops, m, k, n):
    """Rows of every magnitude by columns of every magnitude: a result is finite and right wherever fp32 holds it."""
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    a, b = torch.empty(m, k, device="cuda").normal_(generator=g), torch.empty(n, k, device="cuda").normal_(generator=g)
    a *= torch.logspace(-32, 36, m, device="cuda")[:, None]
    b *= torch.logspace(-32, 36, n, device="cuda")[:, None]
    got = ops.MultiplyMatrixByTransposedMatrix(a, b)
    size = a.abs().double() @ b.abs().double().T
    held = (size > 1e-30) & (size < 3e38)
    assert float(held.double().mean()) > 0.7 and bool(torch.isfinite(got[held]).all())
    err = (got.double() - a.double() @ b.double().T).abs() / size
    assert float(err[held].max()) < bound(k)


def opposed(kind: str, m: int, k: int, n: int, g):
    """Operands whose large elements meet small ones, or none, on the other side, down to subnormal numbers."""
    a, b = torch.empty(m, k, device="cuda").normal_(generator=g), torch.empty(n, k, device="cuda").normal_(generator=g)
    sign = 1.0 - 2.0 * (torch.arange(k, device="cuda") % 2)
    if kind == "decades":        # the odd and the even columns up to 34 decades apart, the other way round in the other operand
        a *= torch.pow(10.0, torch.linspace(0, 17, m, device="cuda")[:, None] * sign)
        b *= torch.pow(10.0, -torch.linspace(0, 17, n, device="cuda")[:, None] * sign)
    elif kind == "shadowed":     # one element each that towers over its row and meets a zero
        a[:, 40], b[:, 40], a[:, 77], b[:, 77] = 1e12, 0.0, 0.0, 1e12
    elif kind == "last":         # the same in the last column, after the row's scale has settled, and for some rows only
        a[::3, k - 1], b[:, k - 1] = 1e15, 0.0
    elif kind == "subnormal":
        a *= 1e-37
        a[:, ::2] *= 1e-3
        a[::5] *= 1e-3
        b *= 1e25
    return a, b


@pytest.mark.parametrize("m,k,n", [(9700, 132, 57), (9601, 576, 96), (4800, 160, 129), (1024, 1332, 330), (1029, 2304, 128)])
@pytest.mark.parametrize("kind", ["decades", "shadowed", "last", "subnormal"])
def test_opposed_ranges(ops, m, k, n, kind):
    g = torch.Generator(device="cuda")
    g.manual_seed(m + k)
    a, b = opposed(kind, m, k, n, g)
    got = ops.MultiplyMatrixByTransposedMatrix(a, b)
    assert worst(got, a, b) < bound(k)
    bias = torch.empty(n, device="cuda").normal_(generator=g)
    got = ops.MultiplyMatrixByTransposedMatrix(a, b, free_term=bias)
    assert worst(got, a, b, extra=bias.expand(m, n)) < bound(k)


@pytest.mark.parametrize("shape,k,r,stride,pad,dil", [((5, 45, 47, 64), 70, 3, 1, 1, 1), ((3, 61, 59, 32), 128, 5, 2, 2, 1),
                                                      ((9, 31, 33, 32), 96, 3, 1, 2, 2), ((4, 75, 90, 3), 64, 7, 2, 3, 1),
                                                      ((5, 60, 70, 4), 40, 5, 1, 2, 1), ((6, 14, 14, 512), 160, 3, 1, 1, 1)])
@pytest.mark.parametrize("decades", [6, 15])
def test_convolutions_of_opposed_ranges(ops, shape, k, r, stride, pad, dil, decades):
    """The same through im2col, row windows (3 and 4 channels) and split K (the last): channels of opposed magnitude."""
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    x, f = torch.empty(shape, device="cuda").normal_(generator=g), torch.empty(k, r, r, shape[3], device="cuda").normal_(generator=g)
    scale = torch.pow(10.0, decades * (1.0 - 2.0 * (torch.arange(shape[3], device="cuda") % 2)))
    x, f = x * scale, f / scale
    f[1] = 0.0                                    # a filter of zeros
    got = ops.BlobConvolution(x, f, padding=(pad, pad), stride=(stride, stride), dilation=(dil, dil))
    conv = lambda p, q: torch.nn.functional.conv2d(p.double().permute(0, 3, 1, 2), q.double().permute(0, 3, 1, 2), stride=stride,
                                                   padding=pad, dilation=dil).permute(0, 2, 3, 1)
    size = conv(x.abs(), f.abs())
    assert bool((got[size == 0] == 0).all())
    assert float(((got.double() - conv(x, f)).abs() / size.clamp_min(1e-300)).max()) < bound(r * r * shape[3])


def test_batches_and_infinities(ops):
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    a = torch.empty(7, 1100, 160, device="cuda").normal_(generator=g)
    b = torch.empty(7, 200, 160, device="cuda").normal_(generator=g)
    assert worst(ops.BatchMultiplyMatrixByTransposedMatrix(a, b), a, b) < bound(160)
    a[2, 5, 3], a[2, 7, 159] = float("inf"), float("nan")
    got = ops.BatchMultiplyMatrixByTransposedMatrix(a, b)
    assert not bool(torch.isfinite(got[2, 5]).any()) and bool(torch.isnan(got[2, 7]).all())
    a[2, 5, 3] = a[2, 7, 159] = 0.0
    rest = ops.BatchMultiplyMatrixByTransposedMatrix(a, b)
    keep = torch.ones(7, 1100, dtype=torch.bool, device="cuda")
    keep[2, 5] = keep[2, 7] = False
    assert torch.equal(got[keep], rest[keep])      # the other rows of the tile do not notice


@pytest.mark.parametrize("shape,k,r,stride,pad,dil", [((5, 45, 47, 64), 70, 3, 1, 1, 1), ((3, 61, 59, 32), 128, 5, 2, 2, 1),
                                                      ((9, 31, 33, 32), 96, 3, 1, 2, 2), ((4, 75, 90, 3), 64, 7, 2, 3, 1)])
def test_convolutions(ops, shape, k, r, stride, pad, dil):
    """im2col and row-window operands; the padding's zeros come first in the border rows."""
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    x, f = torch.empty(shape, device="cuda").normal_(generator=g), torch.empty(k, r, r, shape[3], device="cuda").normal_(generator=g)
    got = ops.BlobConvolution(x, f, padding=(pad, pad), stride=(stride, stride), dilation=(dil, dil))
    conv = lambda p, q: torch.nn.functional.conv2d(p.double().permute(0, 3, 1, 2), q.double().permute(0, 3, 1, 2), stride=stride,
                                                   padding=pad, dilation=dil).permute(0, 2, 3, 1)
    err = (got.double() - conv(x, f)).abs() / conv(x.abs(), f.abs()).clamp_min(1e-300)
    assert float(err.max()) < bound(r * r * shape[3])


# rows of 4k + 1..3 floats: both operands are copied into 16-byte rows first.  Where the product then runs on the TF32
# kernel unsplit it forms the same sums in the same order as the kernel that gathers the rows as they are
@pytest.mark.parametrize("batch,m,k,n,same", [(1, 1, 5, 1, True), (3, 40, 33, 50, True), (2, 129, 127, 97, True), (90, 65, 61, 33, True),
                                              (1, 200, 1001, 131, False), (1, 2000, 1003, 905, False), (2, 5000, 131, 70, False)])
@pytest.mark.parametrize("precision", [0, 1])
def test_odd_depths(ops, batch, m, k, n, same, precision):
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    a, b = torch.empty(batch, m, k, device="cuda").normal_(generator=g), torch.empty(batch, n, k, device="cuda").normal_(generator=g)
    got = ops.BatchMultiplyMatrixByTransposedMatrix(a, b, precision=precision)
    gathered = ops.BatchMultiplyMatrixByTransposedMatrix(a, b, precision=precision, use_scratch=False)
    if same:
        assert torch.equal(got, gathered)
    # TF32 operands are rounded to 11 bits: two errors of 2^-12 more; the TF32 kernel accumulates 8 products at a time
    limit = 2 * bound(k) + (2.0 ** -11 if precision else 0.0)
    assert worst(got, a, b) < limit
    odd = torch.nn.functional.pad(a[0], (0, 2)).contiguous()     # an odd row length in memory, too
    wide = ops.MultiplyMatrixByTransposedMatrix(odd, b[0], first_width=k, precision=precision, first_row_size=k + 2)
    assert worst(wide, a[0], b[0]) < limit


# unsplit products of few K blocks: the tile width follows from the waves, the K blocks and whether result rows are whole 16-byte
# pieces (here 96, 96, 64, 128 and then 32 columns, most with a remainder)
@pytest.mark.parametrize("m,k,n", [(20000, 32, 576), (20001, 16, 1300), (60000, 32, 320), (18900, 128, 250 * 4), (20000, 24, 130),
                                   (3000, 16, 259), (9001, 100, 64), (300, 20, 33)])
@pytest.mark.parametrize("precision", [0, 1])
def test_tile_widths(ops, m, k, n, precision):
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    a, b = torch.empty(m, k, device="cuda").normal_(generator=g), torch.empty(n, k, device="cuda").normal_(generator=g)
    res = torch.empty(m, n, device="cuda").normal_(generator=g)
    # 8 products at a time; plain TF32 rounds both operands to 11 bits
    limit = 2 * bound(k) + (2.0 ** -10 if precision else 0.0)
    got = ops.MultiplyMatrixByTransposedMatrix(a, b, residual=res, precision=precision)
    assert worst(got, a, b, extra=res) < limit
    bias = torch.empty(n, device="cuda").normal_(generator=g)
    got = ops.MultiplyMatrixByTransposedMatrix(a, b, free_term=bias, precision=precision)
    assert worst(got, a, b, extra=bias.expand(m, n)) < limit
    clamped = ops.MultiplyMatrixByTransposedMatrix(a, b, free_term=bias, act=ops.ACT_RELU, act_param=2.5, precision=precision)
    assert torch.equal(clamped, got.clamp(0.0, 2.5))


@pytest.mark.parametrize("shape,k,r,stride,pad", [((5, 45, 47, 64), 70, 3, 1, 1), ((9, 40, 40, 160), 96, 1, 1, 0),
                                                  ((4, 75, 90, 3), 64, 7, 2, 3), ((6, 14, 14, 512), 160, 3, 1, 1)])
@pytest.mark.parametrize("precision", [0, 1])
def test_prepared_filters(ops, shape, k, r, stride, pad, precision):
    """A filter prepared once (im2col, plain rows, row windows, split K) gives the bits of one prepared in the call, and its other
    form serves a single image, which the TF32 kernel takes."""
    capi, lib = ops.capi, ops.capi.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    x, f = torch.empty(shape, device="cuda").normal_(generator=g), torch.empty(k, r, r, shape[3], device="cuda").normal_(generator=g)
    bias = torch.empty(k, device="cuda").normal_(generator=g)
    ho, wo = (ops.conv_output_size(v, r, pad, stride) for v in shape[1:3])
    desc = lambda n: capi.ConvDesc(n, *shape[1:], k, r, r, pad, pad, stride, stride, 1, 1, ho, wo)
    stream, epi = torch.cuda.current_stream().cuda_stream, capi.Epilogue(bias.data_ptr(), None, k, capi.ACT_NONE, 0.0, 0, None)
    prepared = torch.empty(lib.nb200_blob_convolution_prepared_filter_floats(desc(shape[0])), device="cuda")
    capi.check("prepare", lib.nb200_blob_convolution_prepare_filter(stream, desc(shape[0]), f.data_ptr(), prepared.data_ptr(), precision))
    for n in (shape[0], 1):
        y = torch.empty(n, ho, wo, k, device="cuda")
        scratch = torch.empty(lib.nb200_blob_convolution_scratch_floats(desc(n)) + 1, device="cuda")
        capi.check("convolution", lib.nb200_blob_convolution_with_prepared_filter(
            stream, desc(n), x.data_ptr(), f.data_ptr(), prepared.data_ptr(), y.data_ptr(), scratch.data_ptr(), epi, precision))
        if n == shape[0]:
            assert torch.equal(y, ops.BlobConvolution(x, f, bias, padding=(pad, pad), stride=(stride, stride), precision=precision))
        conv = lambda p, q: torch.nn.functional.conv2d(p.double().permute(0, 3, 1, 2), q.double().permute(0, 3, 1, 2), stride=stride,
                                                       padding=pad).permute(0, 2, 3, 1)
        err = (y.double() - conv(x[:n], f) - bias.double()).abs() / (conv(x[:n].abs(), f.abs()) + bias.abs().double())
        # the TF32 kernel accumulates 8 products at a time; plain TF32 rounds both operands to 11 bits
        assert float(err.max()) < 2 * bound(r * r * shape[3]) + (2.0 ** -10 if precision else 0.0)
