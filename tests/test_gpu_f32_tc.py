"""Float32 activations on the tensor cores at the sizes where the split can go wrong -- one row more than the few-rows kernel
keeps, chunks of 16, 32 and 48 rows and one more, a last step of K that is half or a quarter full, one tile and a ragged last one, one to eight
CTAs to a tile, tables whose rows start on no word, biases that are not the centre's -- against the exact product of the oracle. Needs a B200.

Tolerance: 4e-7 of the result's norm (2^-24 = 6e-8 for each of: an activation's three pieces, which are exact; a tensor core's truncated sum
of 16 products, four in a row; the scaled sums of up to 8 groups and of up to 8 CTAs, square roots of that many)."""

import numpy as np
import pytest
import torch

from helpers import activations, affine_case, mxfp4_case, to_numpy, to_torch
from metaljax_b200 import _lib, qmm
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _case(m, k, n, kind, gs, tdt, seed=0):
    rng = np.random.default_rng(m * k + n + seed)
    if kind == "mxfp4":
        w, s, b, kw = *mxfp4_case(rng, n, k)[-2:], None, dict(group_size=32, bits=4, mode="mxfp4")
    else:
        (w, s, b), kw = affine_case(rng, n, k, gs, int(kind[3:]), tdt)[1:], dict(group_size=gs, bits=int(kind[3:]))
    xs = activations(rng, (m, k), "f32")
    exact = O.qmm_exact(xs, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    return xs, [to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV)], kw, exact


def _product(x, *args, **kw):
    """On the tensor-core kernel, or not at all."""
    with _lib.force_route("f32_tc"):
        return qmm.quantized_matmul(x, *args, **kw)


def _far(y, exact):
    return np.linalg.norm(to_numpy(y).astype(np.float64) - exact) / np.linalg.norm(exact)


@pytest.mark.parametrize("m,k,n,kind,gs,tdt,plan", [
    (9, 64, 1, "int4", 64, "f32", (16, 1, 2)),              # half a step
    (16, 96, 127, "mxfp4", 32, None, (16, 1, 2)),           # three quarters of one
    (17, 160, 129, "int4", 32, "bf16", (16, 2, 2)),         # two steps, the last a quarter full; two tiles
    (33, 4096, 1790, "int4", 64, "f32", (48, 8, 1)),        # 48 rows, eight CTAs, one partial tile on its way
    (33, 4096, 640, "int4", 64, "f32", (16, 8, 2)),         # three chunks of 16
    (49, 4096, 2500, "int4", 128, "f16", (32, 8, 2)),       # two chunks, more tiles than clusters
    (64, 2112, 385, "int8", 64, "f32", (16, 8, 2)),         # 17 steps over eight CTAs
    (100, 1088, 257, "int8", 32, "bf16", (16, 4, 2)),
    (12, 14336, 256, "int4", 128, "f32", (16, 8, 2)),       # the longest stretch of K that 16 rows leave room for
    (12, 12288, 300, "int8", 64, "f32", (16, 8, 1)),        # ... of 8-bit codes: one partial tile on its way
    (48, 2880, 700, "mxfp4", 32, None, (16, 8, 2)),         # 90 table bytes a row
    (31, 320, 200, "int8", 64, "f16", (16, 2, 2)),
    (200, 576, 19300, "int4", 64, "f32", (32, 1, 2)),       # many tiles, no cluster
])
def test_float32_rows(m, k, n, kind, gs, tdt, plan):
    xs, args, kw, exact = _case(m, k, n, kind, gs, tdt)
    with _lib.force_route("f32_tc"):
        assert qmm.float32_plan(m, k, n, table_dtype=args[1].dtype, **kw) == plan
    y = _product(to_torch(xs, DEV), *args, **kw)
    assert _far(y, exact) <= 4e-7
    assert _lib.poll_status() == 0


def test_float32_rows_that_do_not_fit():
    """32 codes more than 16 rows' stretches leave room for: the few-rows kernel's."""
    xs, args, kw, exact = _case(20, 14368, 130, "mxfp4", 32, None)
    with pytest.raises(_lib.QmmError):
        _product(to_torch(xs, DEV), *args, **kw)
    assert _far(qmm.quantized_matmul(to_torch(xs, DEV), *args, **kw), exact) <= 4e-7


def test_float32_rows_with_biases_of_their_own():
    """(b + C s) sum x is left out where it is nought for a warp's rows: here one row of a tile has one."""
    xs, (w, s, b), kw, _ = _case(40, 512, 300, "int4", 64, "f32")
    b = -8 * s
    b[200, 3] = 0.7
    exact = O.qmm_exact(xs, to_numpy(w), to_numpy(s), to_numpy(b), 64, 4)
    assert _far(_product(to_torch(xs, DEV), w, s, b, **kw), exact) <= 4e-7


@pytest.mark.parametrize("m,kind,gs,k,tdt", [(48, "int4", 64, 4096, "f32"), (33, "int4", 32, 1056, "f32"), (20, "int4", 128, 2688, "f16"), (48, "int8", 128, 3200, "f32"),
                                             (17, "int8", 32, 2080, "bf16"), (64, "int8", 64, 8256, "f32"), (12, "int4", 32, 14336, "f32")])
def test_float32_rows_with_zero_points(m, kind, gs, k, tdt):
    """Every group has a bias of its own: exact, and no further off than eight rows at a time (see below)."""
    xs, (w, s, b), kw, _ = _case(m, k, 900, kind, gs, tdt, 5)
    b = b + s * torch.randint(-5, 6, s.shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)).to(s.dtype)
    exact = O.qmm_exact(xs, to_numpy(w), to_numpy(s), to_numpy(b), gs, kw["bits"])
    x = to_torch(xs, DEV)
    by_eight = torch.cat([qmm.quantized_matmul(x[i:i + 8], w, s, b, **kw) for i in range(0, m, 8)])
    far = _far(_product(x, w, s, b, **kw), exact)
    assert far <= 4e-7 and far <= 1.05 * _far(by_eight, exact)      # (10800 results at least: their root mean square varies by 1 %)


def test_float32_rows_infinite_beside_biases_of_their_own():
    """A weight row with centred biases makes of an infinity what its weight does, whatever the biases of the rows beside it."""
    xs, (w, s, b), kw, _ = _case(20, 256, 140, "int4", 64, "f32")
    b = -8 * s
    b[7] += s[7]
    column = O.qmm_exact(np.eye(256, dtype=np.float32)[77:78], to_numpy(w), to_numpy(s), to_numpy(b), 64, 4)[0]
    xs[2, 77] = np.inf
    y = to_numpy(_product(to_torch(xs, DEV), w, s, b, **kw))
    with np.errstate(invalid="ignore"):
        want = np.float32(np.inf) * column.astype(np.float32)
    rest = np.arange(140) != 7
    assert np.array_equal(np.isnan(y[2][rest]), np.isnan(want[rest]))
    finite = rest & ~np.isnan(want)
    assert np.array_equal(y[2][finite], want[finite])


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float16])
def test_float32_rows_to_16_bits(out):
    xs, args, kw, exact = _case(37, 1024, 260, "int4", 64, "f32")
    y = _product(to_torch(xs, DEV), *args, **kw, out_dtype=out)
    assert torch.equal(y, _product(to_torch(xs, DEV), *args, **kw).to(out))


@pytest.mark.parametrize("m", [12, 40])            # with slices of 512 codes, and with one for all of a stretch
@pytest.mark.parametrize("kind,k,power", [("int8", 1088, 120), ("int8", 1088, 118), ("int8", 1088, -118), ("int8", 640, -128),
                                          ("mxfp4", 1120, 118), ("mxfp4", 1120, -116), ("mxfp4", 640, -128), ("int4", 1088, 120), ("int4", 1088, -108)])
def test_float32_rows_at_the_ends_of_their_range(m, kind, k, power):
    """Activations of up to some 2^122 whose results fit, and such that have no 24 bits above bf16's smallest number, keep the precision of the middle
    of the range; slices that lie 2^60 apart do not share a scale."""
    xs, args, kw, _ = _case(m, k, 200, kind, 32 if kind == "mxfp4" else 64, "f32")
    xs = np.ldexp(xs, power)
    if power < 0 and kind != "int4":
        xs[1, 512:] = np.ldexp(xs[1, 512:], 60)
    exact = O.qmm_exact(xs, to_numpy(args[0]), to_numpy(args[1]), None if args[2] is None else to_numpy(args[2]), kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    y = to_numpy(_product(to_torch(xs, DEV), *args, **kw)).astype(np.float64)
    assert np.isfinite(y).all()
    far = np.linalg.norm(y - exact, axis=1) / np.linalg.norm(exact, axis=1)      # of each row: they are as far apart as their slices
    assert far.max() <= 4e-7


@pytest.mark.parametrize("kind,gs,k,one_sign", [("int4", 64, 14336, True), ("int4", 32, 8192, True), ("int4", 128, 4096, False), ("int8", 128, 4096, False),
                                                ("int8", 64, 12288, True), ("mxfp4", 32, 4096, False), ("mxfp4", 32, 14336, True)])
def test_float32_rows_are_as_exact_as_eight_at_a_time(kind, gs, k, one_sign):
    """Against the few-rows kernel, which calls of eight rows take: no further from the exact product (the errors of 49152 results have a root
    mean square that varies by 0.4 %: 2 % is five times that)."""
    xs, args, kw, _ = _case(48, k, 1024, kind, gs, "f32" if kind != "mxfp4" else None, 3)
    if one_sign:
        xs = np.abs(xs)
    exact = O.qmm_exact(xs, to_numpy(args[0]), to_numpy(args[1]), None if args[2] is None else to_numpy(args[2]), gs, kw["bits"], mode=kw.get("mode", "affine"))
    x = to_torch(xs, DEV)
    by_eight = torch.cat([qmm.quantized_matmul(x[i:i + 8], *args, **kw) for i in range(0, 48, 8)])
    assert _far(_product(x, *args, **kw), exact) <= 1.02 * _far(by_eight, exact)


def test_float32_rows_below_the_range_of_4_bit_codes():
    """Below 2^-110 an activation is rounded to a multiple of 2^-133, the smallest bf16: an error of 2^-133 / sqrt(12) each, and a quarter more."""
    xs, args, kw, _ = _case(40, 1024, 200, "int4", 64, "f32")
    xs = np.ldexp(xs, -122)
    w, s, b = (to_numpy(a) for a in args)
    dense = O.qmm_exact(np.eye(1024, dtype=np.float32), w, s, b, 64, 4)
    y = to_numpy(_product(to_torch(xs, DEV), *args, **kw)).astype(np.float64)
    assert np.linalg.norm(y - O.qmm_exact(xs, w, s, b, 64, 4)) <= 1.25 * 2.0 ** -133 / np.sqrt(12) * np.sqrt(len(xs)) * np.linalg.norm(dense)


@pytest.mark.parametrize("kind", ["mxfp4", "int4", "int8"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_float32_rows_that_are_not_finite(value, kind):
    """An infinity times a positive, a negative or a zero weight, as a sum of products has it; the rows beside it as ever."""
    xs, args, kw, exact = _case(20, 1120, 300, kind, 32, None if kind == "mxfp4" else "f32")
    w, s, b = (None if a is None else to_numpy(a) for a in args)
    column = O.qmm_exact(np.eye(1120, dtype=np.float32)[17:18], w, s, b, 32, kw["bits"], mode=kw.get("mode", "affine"))[0]
    xs[3, 17] = value
    y = to_numpy(_product(to_torch(xs, DEV), *args, **kw))
    with np.errstate(invalid="ignore"):
        want = (np.float32(value) * column.astype(np.float32))
    assert np.array_equal(np.isnan(y[3]), np.isnan(want)) and np.array_equal(y[3][~np.isnan(want)], want[~np.isnan(want)])
    rest = np.arange(20) != 3
    assert _far(to_torch(y[rest], "cpu"), exact[rest]) <= 4e-7


def test_float32_rows_replay():
    xs, args, kw, exact = _case(64, 2048, 1024, "int4", 64, "f32")
    x, y = to_torch(xs, DEV), torch.zeros((64, 1024), device=DEV)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        _product(x, *args, out=y, **kw)
        stream.synchronize()
        first = y.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(3):
                _product(x, *args, out=y, **kw)
        y.zero_()
        graph.replay()
        stream.synchronize()
    assert torch.equal(y, first) and _far(first, exact) <= 4e-7
    assert _lib.poll_status() == 0
