"""The few-rows kernel at the sizes where its split can go wrong -- chunks of 4, 8 and 16 rows, slices and clusters
along K and their remainders, tables whose rows start on no word, experts of nought to twenty rows --
against the exact product of the oracle. Needs a B200.

Tolerances are the parity gates of the package: 1e-2 of the largest result for 16-bit activations (the output
is rounded to 8 bits: 2^-9 of each value; everything before it is kept in 21 bits or more), 1e-5 for
float32 (sums of K terms in float32, in pieces of 512: below 2^-24 * 512)."""

import numpy as np
import pytest
import torch

from helpers import activations, affine_case, mxfp4_case, to_numpy, to_torch
from metaljax_b200 import _lib, moe, qmm
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
TOL = {"bf16": 1e-2, "f16": 1e-2, "f32": 1e-5}


def _case(rng, kind, n, k, gs, tdt, lead=()):
    if kind == "mxfp4":
        out = mxfp4_case(rng, n, k, lead=lead)
        return (*out[-2:], None), dict(group_size=32, bits=4, mode="mxfp4")
    return affine_case(rng, n, k, gs, int(kind[3:]), tdt, lead=lead)[1:], dict(group_size=gs, bits=int(kind[3:]))


@pytest.fixture(autouse=True)
def _no_wait_ran_out():
    yield
    assert _lib.poll_status() == 0


@pytest.mark.parametrize("kind,gs,x,tdt", [
    ("int4", 64, "bf16", "bf16"), ("int4", 32, "bf16", "f32"), ("int4", 128, "f16", "f16"), ("int8", 32, "f16", "f16"),
    ("int8", 64, "bf16", "bf16"), ("mxfp4", 32, "bf16", None), ("int4", 64, "f32", "f32"), ("int8", 128, "f32", "bf16"), ("mxfp4", 32, "f32", None),
])
@pytest.mark.parametrize("m,k,n", [
    (2, 128, 1), (7, 384, 33), (8, 512, 300), (9, 640, 31), (16, 1152, 65), (5, 4480, 130), (3, 16384, 48), (12, 34048, 20), (17, 2176, 100),
])
def test_rows_at_the_edges(kind, gs, x, tdt, m, k, n):
    if m > 16 and x != "f32":
        pytest.skip("more rows of 16-bit activations are the tensor-core kernel's")
    rng = np.random.default_rng(m * k + n)
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt)
    xs = activations(rng, (m, k), x)
    args = [to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV)]
    if x == "f32":
        y = qmm.quantized_matmul(*args, **kw)
    else:
        with _lib.force_route("gemv_fmma"):                   # (a long K has the tensor-core kernel by default)
            y = qmm.quantized_matmul(*args, **kw)
    exact = O.qmm_exact(xs, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    assert O.rel_err(to_numpy(y).astype(np.float32), exact) <= TOL[x]


@pytest.mark.parametrize("sizes", [[1], [0, 3, 0, 1], [20, 0, 17, 8, 9, 1, 0, 2], [0, 0, 0], [1] * 40])
@pytest.mark.parametrize("kind,x", [("int4", "bf16"), ("int8", "f16"), ("mxfp4", "bf16")])
def test_few_rows_per_expert(kind, x, sizes):
    rng = np.random.default_rng(len(sizes) + sum(sizes))
    k, n, total = 672 if kind == "mxfp4" else 704, 90, sum(sizes) + 1
    (w, s, b), kw = _case(rng, kind, n, k, 64, x, lead=(len(sizes),))
    xs = activations(rng, (total, k), x)
    gsz = np.array(sizes, np.int32)
    y = moe.ragged_dot(to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV), torch.from_numpy(gsz).to(DEV), **kw)
    got = to_numpy(y).astype(np.float32)
    assert not got[sum(sizes):].any()
    if sum(sizes):
        assert O.rel_err(got, O.ragged_qmm_exact(xs, w, s, b, gsz, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))) <= 1e-2


def _styled(rng, shape, style):
    """Activations N(0, 1), of one sign, or with outliers of 300."""
    v = rng.standard_normal(shape)
    if style == "one sign":
        v = np.abs(v)
    elif style == "outliers":
        v[..., ::97] *= 300.0
    return v.astype(np.float32)


def _weight64(w, s, b, kw):
    """The weight in float64 (the oracle's is rounded to float32 element by element)."""
    if b is None:
        return O.dequantize(w, s, None, 32, 4, "mxfp4").astype(np.float64)
    gs = kw["group_size"]
    codes = O.dequantize(w, np.ones(s.shape, np.float32), np.zeros(s.shape, np.float32), gs, kw["bits"], "affine").astype(np.float64)
    return codes * np.repeat(s.astype(np.float64), gs, -1) + np.repeat(b.astype(np.float64), gs, -1)


@pytest.mark.parametrize("style", ["normal", "one sign", "outliers"])
@pytest.mark.parametrize("kind,gs,tdt", [("int4", 32, "f32"), ("int4", 128, "bf16"), ("int8", 32, "bf16"), ("int8", 128, "f32"), ("mxfp4", 32, None)])
@pytest.mark.parametrize("m,k,n", [(3, 512, 130), (33, 5632, 96)])
def test_float32_is_as_exact_as_plain_float32(kind, gs, tdt, style, m, k, n):
    """Against the SIMT kernel, which sums float32 products one by one: the few-rows kernel is no further from the exact product.
    Both errors are sums of roundings of 2^-24 that scatter by a few percent; a quarter is allowed for that."""
    rng = np.random.default_rng(m + k)
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt)
    xs = _styled(rng, (m, k), style)
    args = [to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV)]
    exact = xs.astype(np.float64) @ _weight64(w, s, b, kw).T
    error = lambda y: np.linalg.norm(to_numpy(y).astype(np.float64) - exact) / np.linalg.norm(exact)
    got = error(qmm.quantized_matmul(*args, **kw))
    with _lib.force_route("simt"):
        plain = error(qmm.quantized_matmul(*args, **kw))
    assert got <= 1.25 * plain


@pytest.mark.parametrize("x", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_infinite_activations_are_summed_as_they_are(x, value):
    """MXFP4 has no bias: an infinity times a positive, a negative or a zero weight, and the rows beside it as ever."""
    rng = np.random.default_rng(5)
    (w, s, _), kw = _case(rng, "mxfp4", 70, 1120, 32, None)
    xs = activations(rng, (3, 1120), x)
    xs[1, 17] = value
    y = to_numpy(qmm.quantized_matmul(to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None, out_dtype=torch.float32, **kw))
    column = O.qmm_exact(np.eye(1120, dtype=np.float32)[17:18], w, s, None, 32, 4, mode="mxfp4")[0]      # the weights that the infinity meets
    with np.errstate(invalid="ignore"):
        np.testing.assert_array_equal(y[1], np.float32(value) * column.astype(np.float32))
    rest = O.qmm_exact(xs[[0, 2]], w, s, None, 32, 4, mode="mxfp4")
    assert O.rel_err(y[[0, 2]], rest) <= 1e-5


@pytest.mark.parametrize("kind,gs", [("int4", 64), ("int8", 64), ("mxfp4", 32)])
@pytest.mark.parametrize("size", [2.0 ** 120, 2.0 ** -100])
def test_large_and_small_float32_activations(kind, gs, size):
    """Finite results of finite activations, whatever their size: as exact as those near one (the gate for float32)."""
    rng = np.random.default_rng(6)
    (w, s, b), kw = _case(rng, kind, 70, 1152, gs, "f32")
    xs = activations(rng, (5, 1152), "f32") * np.float32(size / 8)
    y = qmm.quantized_matmul(to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV), **kw)
    exact = O.qmm_exact(xs.astype(np.float64) / size, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    assert O.rel_err(to_numpy(y).astype(np.float64) / size, exact) <= 1e-5


@pytest.mark.parametrize("sizes", [[3, 0, 9, 1, 20, 2], [5, 1, 0, 8, 1, 1]])
def test_half_nibbles_of_one_sign(sizes):
    """4-bit codes against f16 of one sign, where the sums are far larger than the results: no further from the exact product than the
    tensor-core kernel, whose weights are rounded to f16."""
    rng = np.random.default_rng(sum(sizes))
    (w, s, b), kw = _case(rng, "int4", 96, 2048, 64, "f16", lead=(len(sizes),))
    xs = np.abs(activations(rng, (sum(sizes), 2048), "f16"))
    gsz = np.array(sizes, np.int32)
    args = [to_torch(a, DEV) for a in (xs, w, s, b)] + [torch.from_numpy(gsz).to(DEV)]
    exact = O.ragged_qmm_exact(xs, w, s, b, gsz, kw["group_size"], kw["bits"]).astype(np.float64)
    error = lambda y: np.linalg.norm(to_numpy(y).astype(np.float64) - exact) / np.linalg.norm(exact)
    got = error(moe.ragged_dot(*args, out_dtype=torch.float32, **kw))
    with _lib.force_route("gemm_tc"):
        assert got <= error(moe.ragged_dot(*args, out_dtype=torch.float32, **kw))


@pytest.mark.parametrize("kind,x", [("int4", "bf16"), ("int4", "f16"), ("int8", "bf16"), ("int8", "f16")])
@pytest.mark.parametrize("m,k", [(17, 2048), (32, 32)])
def test_gathers_of_many_rows_sum_in_plain_float32(kind, x, m, k):
    """Unsorted gathers of more than 16 rows, activations of one sign, a float32 result: no further from the exact product than the SIMT kernel
    (a quarter for the scatter of the roundings, as above)."""
    rng = np.random.default_rng(m + k)
    (w, s, b), kw = _case(rng, kind, 96, k, 32, x, lead=(4,))
    xs = np.abs(activations(rng, (5, m, k), x))
    li, ri = rng.integers(0, 5, 9), rng.integers(0, 4, 9)
    args = [to_torch(a, DEV) for a in (xs, w, s, b)] + [torch.from_numpy(i).to(DEV) for i in (li, ri)]
    exact = np.stack([xs[i].astype(np.float64) @ _weight64(w[j], s[j], b[j], kw).T for i, j in zip(li, ri)])
    error = lambda y: np.linalg.norm(to_numpy(y).astype(np.float64) - exact) / np.linalg.norm(exact)
    got = error(moe.gather_qmm(*args, out_dtype=torch.float32, **kw))
    with _lib.force_route("simt"):
        assert got <= 1.25 * error(moe.gather_qmm(*args, out_dtype=torch.float32, **kw))


@pytest.mark.parametrize("kind", ["int4", "int8", "mxfp4"])
@pytest.mark.parametrize("m,k", [(9, 4224), (16, 5760)])
def test_nine_to_sixteen_rows_keep_float32_weights(kind, m, k):
    """A float32 result of bf16 activations. 4-bit codes are summed as 128 + q, of which 128 of some 10 cancel: 2^-24 * 16 of a term, of which K
    random ones add up as their root does and so do the results; 2^-18 leaves four times that. (Weights rounded to bf16 are 2^-10 off.)"""
    rng = np.random.default_rng(m + k)
    (w, s, b), kw = _case(rng, kind, 96, k, 64, "bf16")
    xs = activations(rng, (m, k), "bf16")
    args = [to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV)]
    y = to_numpy(qmm.quantized_matmul(*args, out_dtype=torch.float32, **kw)).astype(np.float64)
    exact = xs.astype(np.float64) @ _weight64(w, s, b, kw).T
    assert np.linalg.norm(y - exact) <= 2.0 ** -18 * np.linalg.norm(exact)


@pytest.mark.parametrize("sizes", [[0, 64, 0, 0, 0, 0, 0, 0], [32, 0, 0, 0, 0, 0, 0, 32], [57, 1, 1, 1, 1, 1, 1, 1], [0, 0, 0, 65, 0, 0, 0, 0], [0, 0, 128, 0, 0, 0, 0, 0]])
@pytest.mark.parametrize("kind,x", [("int4", "bf16"), ("mxfp4", "f16")])
def test_skewed_routing(kind, x, sizes):
    """All or nearly all rows on one or two experts, on either side of the rule that picks the kernel by the average."""
    rng = np.random.default_rng(sum(sizes) + sizes[0])
    (w, s, b), kw = _case(rng, kind, 90, 704, 64, x, lead=(8,))
    xs = activations(rng, (sum(sizes), 704), x)
    gsz = np.array(sizes, np.int32)
    y = moe.ragged_dot(to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV), torch.from_numpy(gsz).to(DEV), **kw)
    exact = O.ragged_qmm_exact(xs, w, s, b, gsz, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    assert O.rel_err(to_numpy(y).astype(np.float32), exact) <= TOL[x]


@pytest.mark.parametrize("kind,gs,x,tdt", [("int4", 64, "bf16", "bf16"), ("int4", 128, "f16", "f16"), ("int4", 32, "bf16", "f32"), ("mxfp4", 32, "bf16", None)])
@pytest.mark.parametrize("k", [1024, 5632, 14336])
@pytest.mark.parametrize("n", [16, 33, 528, 6000])
def test_tiles_of_a_cluster_are_finished_a_lap_late(kind, gs, x, tdt, k, n):
    """K of one CTA, of clusters of two and of four; from one tile to a dozen of a cluster, so that the last lap of leaders is whole, partial or the only one.
    The result is float32: every term is a product of 16-bit numbers, and what the sums round off is below 2^-24 of the largest of them, 128 sum |x| s
    against a result of some 8 sum |x| s sqrt(1 / K): 1e-4 of the largest result."""
    rng = np.random.default_rng(n + k)
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt)
    xs = activations(rng, (5, k), x)
    args = [to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV)]
    with _lib.force_route("gemv_fmma"):
        y = qmm.quantized_matmul(*args, out_dtype=torch.float32, **kw)
    exact = O.qmm_exact(xs, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    assert O.rel_err(to_numpy(y).astype(np.float32), exact) <= 1e-4


@pytest.mark.parametrize("kind,gs,x,tdt", [("int4", 64, "bf16", "bf16"), ("int4", 32, "f16", "f32"), ("int8", 128, "f16", "f16"), ("mxfp4", 32, "bf16", None)])
@pytest.mark.parametrize("m,k,n", [(2, 128, 1), (8, 512, 16), (5, 1152, 17), (9, 4224, 300), (16, 5632, 40), (3, 640, 2500)])
def test_two_products_and_their_gate_in_one_launch(kind, gs, x, tdt, m, k, n):
    """silu(x . Wg) * (x . Wu) with the weights' rows side by side in a tile, against the exact products, gate and all in float64: the results are rounded to 16 bits
    four times (both products, the gate, their product: 2^-9 each for bf16), and the three launches that it stands for are as far off."""
    rng = np.random.default_rng(m * k + n)
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt)
    (w2, s2, b2), _ = _case(rng, kind, n, k, gs, tdt)
    xs = activations(rng, (m, k), x) * np.float32(0.05)
    xt = to_torch(xs, DEV).to(DT[x])
    xs = to_numpy(xt).astype(np.float32)
    y = torch.full((m, n), float("nan"), dtype=DT[x], device=DEV)
    one, two = ([to_torch(a, DEV) if a is not None else None for a in weight] for weight in ((w, s, b), (w2, s2, b2)))
    v = _lib.Views()
    _lib.check(_lib.lib().qmm_gated_matmul(v(xt), *(v(a) for a in one), *(v(a) for a in two), v(y), kw["group_size"], kw["bits"], int(kind == "mxfp4"), torch.cuda.current_stream().cuda_stream))
    gate = O.qmm_exact(xs, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine")).astype(np.float64)
    up = O.qmm_exact(xs, w2, s2, b2, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine")).astype(np.float64)
    assert O.rel_err(to_numpy(y).astype(np.float32), (gate / (1.0 + np.exp(-gate)) * up).astype(np.float32)) <= 1e-2
    apart = moe.silu_mul(qmm.quantized_matmul(xt, *one, **kw), qmm.quantized_matmul(xt, *two, **kw)) if m <= 8 and m * n % 8 == 0 else None
    if apart is not None:
        assert O.rel_err(to_numpy(y).astype(np.float32), to_numpy(apart).astype(np.float32)) <= 1e-2


def test_what_one_launch_does_not_take_is_refused():
    rng = np.random.default_rng(0)
    (w, s, b), kw = _case(rng, "int4", 64, 256, 64, "bf16")
    weight = [to_torch(a, DEV) for a in (w, s, b)]
    for m, x, out in ((1, "bf16", "bf16"), (17, "bf16", "bf16"), (4, "f32", "f32"), (4, "bf16", "f32")):
        xt, y = torch.zeros((m, 256), dtype=DT[x], device=DEV), torch.zeros((m, 64), dtype=DT[out], device=DEV)
        v = _lib.Views()
        before = _lib.lib().qmm_launch_count()
        assert _lib.lib().qmm_gated_matmul(v(xt), *(v(a) for a in weight), *(v(a) for a in weight), v(y), 64, 4, 0, torch.cuda.current_stream().cuda_stream) == 7
        assert _lib.lib().qmm_launch_count() == before


@pytest.mark.parametrize("kind,gs,tdt", [("int4", 32, "f32"), ("int4", 64, "bf16"), ("int8", 64, "f32"), ("int8", 128, "bf16")])
@pytest.mark.parametrize("x", ["bf16", "f16"])
@pytest.mark.parametrize("m", [5, 24])
@pytest.mark.parametrize("style", ["one sign", "outliers", "binades"])
def test_float32_results_of_uneven_activations(kind, gs, tdt, x, m, style):
    """Activations of one sign, with one in 97 300 times as large, and of 22 binades. Everything is a product of 16-bit numbers and a float32 sum: what is rounded or cut off is below 2^-24 of what has been
    added up, (2^bits sum |x| s) at most, over 16 additions one after another in an MMA and K / 512 of them; 24 rows are a gather, which takes the codes without the magic number: sum |x (q - centre)| s."""
    k, n, bits = 2176, 200, int(kind[3:])
    rng = np.random.default_rng(gs + m + len(style))
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt)
    xs = activations(rng, (m, k), x).astype(np.float32)
    if style == "one sign":
        xs = np.abs(xs)
    elif style == "outliers":
        xs[:, ::97] *= 300
    else:
        xs = np.sign(xs) * np.exp2(rng.uniform(-12, 10, xs.shape)).astype(np.float32)
    xt = torch.from_numpy(xs).to(DEV).to(DT[x])
    wt, st, bt = (to_torch(a, DEV) for a in (w, s, b))
    if m == 5:
        with _lib.force_route("gemv_fmma"):
            y = qmm.quantized_matmul(xt, wt, st, bt, out_dtype=torch.float32, **kw)
    else:
        idx = torch.zeros(1, dtype=torch.int32, device=DEV)
        y = moe.gather_qmm(xt[None], wt[None], st[None], bt[None], idx, idx, out_dtype=torch.float32, **kw)[0]
    codes = wt.view(torch.uint8).reshape(n, -1)
    codes = codes if bits == 8 else torch.stack((codes & 15, codes >> 4), -1).reshape(n, k)
    wide = lambda t: t.double().repeat_interleave(gs, -1)
    exact = xt.double() @ (codes.double() * wide(st) + wide(bt)).T
    largest = 2.0 ** (bits if m == 24 else bits + 4 if bits == 4 else bits + 3)               # (a code under the magic number is below 256 or 2048)
    assert bool(((y.double() - exact).abs() <= (16 + k / 512) * 2.0 ** -24 * largest * (xt.double().abs() @ wide(st).abs().T)).all())


def _dequantized(w, s, b, kind, gs):
    """The weight in float64, on the device."""
    codes = w.view(torch.uint8)
    codes = codes if kind == "int8" else torch.stack((codes & 15, codes >> 4), -1)
    codes = codes.reshape(*w.shape[:-1], -1)
    if kind == "mxfp4":
        values = torch.tensor([0, 0.5, 1, 1.5, 2, 3, 4, 6, 0, -0.5, -1, -1.5, -2, -3, -4, -6], dtype=torch.float64, device=w.device)
        return values[codes.long()] * torch.exp2(s.double() - 127).repeat_interleave(32, -1)
    return codes.double() * s.double().repeat_interleave(gs, -1) + b.double().repeat_interleave(gs, -1)


def _gated(xt, one, two, y, kw, kind):
    v = _lib.Views()
    _lib.check(_lib.lib().qmm_gated_matmul(v(xt), *(v(a) for a in one), *(v(a) for a in two), v(y), kw["group_size"], kw["bits"], int(kind == "mxfp4"), torch.cuda.current_stream().cuda_stream))
    return y


@pytest.mark.parametrize("kind,gs,x,tdt", [("int4", 64, "bf16", "bf16"), ("int4", 32, "f16", "f32"), ("int8", 128, "bf16", "bf16"), ("mxfp4", 32, "bf16", None)])
@pytest.mark.parametrize("m,k,n", [(5, 4096, 6000), (12, 5632, 6000), (8, 14336, 3000), (16, 4224, 4500), (9, 1088, 9001)])
def test_gated_tiles_that_follow_one_another(kind, gs, x, tdt, m, k, n):
    """Several tiles a worker -- slots of the ring used again, chunks of 8 rows one after the other in one CTA, laps of a cluster's leaders -- with table rows of whole 16 bytes, of words
    and of neither. Against float64: four roundings to 16 bits, 2^-9 each for bf16, as when each step is a launch."""
    if k % gs:
        pytest.skip("not whole groups")
    rng = np.random.default_rng(m + k + n)
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt)
    (w2, s2, b2), _ = _case(rng, kind, n, k, gs, tdt)
    xt = to_torch(activations(rng, (m, k), x) * np.float32(0.05), DEV).to(DT[x])
    one, two = ([to_torch(a, DEV) if a is not None else None for a in weight] for weight in ((w, s, b), (w2, s2, b2)))
    y = _gated(xt, one, two, torch.full((m, n), float("nan"), dtype=DT[x], device=DEV), kw, kind)
    gate, up = (xt.double() @ _dequantized(*weight, kind, gs).T for weight in (one, two))
    exact = gate / (1.0 + torch.exp(-gate)) * up
    assert ((y.double() - exact).abs().max() / exact.abs().max()).item() <= 1e-2
    assert ((y.double() - exact).norm() / exact.norm()).item() <= 2.0 ** -7


@pytest.mark.parametrize("x", ["bf16", "f16"])
def test_gates_that_are_not_finite(x):
    """Infinities and NaN of either product, and gates so negative that their exponential overflows, come out as from the three launches."""
    k, n, gs = 256, 64, 64
    rng = np.random.default_rng(3)
    (w, s, b), kw = _case(rng, "int4", n, k, gs, x)
    (w2, s2, b2), _ = _case(rng, "int4", n, k, gs, x)
    xt = to_torch(activations(rng, (8, k), x), DEV).to(DT[x])
    xt[1, 7], xt[2, 100], xt[3, 200] = float("inf"), float("-inf"), float("nan")
    xt[4] = 200.0 * xt[4].sign()
    xt[5] = 0.0
    one, two = ([to_torch(a, DEV) for a in weight] for weight in ((w, s, b), (w2, s2, b2)))
    y = _gated(xt, one, two, torch.zeros((8, n), dtype=DT[x], device=DEV), kw, "int4")
    apart = moe.silu_mul(qmm.quantized_matmul(xt, *one, **kw), qmm.quantized_matmul(xt, *two, **kw))
    assert torch.equal(y.isnan(), apart.isnan()) and torch.equal(y.isinf(), apart.isinf()) and bool(y.isnan().any())
    fine = apart.isfinite()
    assert torch.equal(y.sign()[fine], apart.sign()[fine]) and (y - apart)[fine].abs().max() <= 1e-2 * apart[fine].abs().max()


@pytest.mark.parametrize("kind,gs,x,tdt", [("int8", 64, "bf16", "bf16"), ("int8", 128, "f16", "f32")])
@pytest.mark.parametrize("sizes,k,n", [([5], 5632, 6000), ([5], 14336, 3000), ([3, 0, 9, 1], 5632, 2500), ([8, 2], 14336, 1500)])
def test_laps_of_leaders_with_8_bit_codes_and_with_experts(kind, gs, x, tdt, sizes, k, n):
    """What the leaders of a cluster add up a lap late, of 8-bit codes, dense (one size) and grouped: a dozen tiles a cluster, whose last lap is partial. Against float64, the result rounded to 16 bits."""
    rng = np.random.default_rng(k + n + len(sizes))
    dense = len(sizes) == 1
    (w, s, b), kw = _case(rng, kind, n, k, gs, tdt, lead=() if dense else (len(sizes),))
    xt = to_torch(activations(rng, (sum(sizes), k), x), DEV).to(DT[x])
    args = [to_torch(a, DEV) for a in (w, s, b)]
    weights = _dequantized(*args, kind, gs)
    if dense:
        y, exact = qmm.quantized_matmul(xt, *args, **kw), xt.double() @ weights.T
    else:
        y = moe.ragged_dot(xt, *args, torch.tensor(sizes, device=DEV), **kw)
        exact = torch.cat([rows @ e.T for rows, e in zip(xt.double().split(sizes), weights)])
    assert ((y.double() - exact).abs().max() / exact.abs().max()).item() <= 1e-2
    assert ((y.double() - exact).norm() / exact.norm()).item() <= 2.0 ** -8


@pytest.mark.parametrize("kind,x", [("int4", "bf16"), ("int4", "f32"), ("int8", "f16"), ("int8", "f32")])
@pytest.mark.parametrize("m,k,n", [(2, 32, 1), (5, 288, 33), (8, 512, 300), (8, 3232, 700), (3, 4096, 129), (7, 14368, 48)])
def test_rows_of_float32_entries_in_groups_of_32(kind, x, m, k, n):
    """A word of one row's entries a lane where rows start on no 16 bytes (K no multiple of 128), 16 or 8 bytes where they do; one group, a slice that ends in the middle of its entries, clusters. The file's tolerances."""
    rng = np.random.default_rng(m + k + n)
    (w, s, b), kw = _case(rng, kind, n, k, 32, "f32")
    xt = to_torch(activations(rng, (m, k), x), DEV).to(DT[x])
    args = [to_torch(a, DEV) for a in (w, s, b)]
    exact = xt.double() @ _dequantized(*args, kind, 32).T
    if x == "f32":
        y = qmm.quantized_matmul(xt, *args, **kw)
    else:
        with _lib.force_route("gemv_fmma"):
            y = qmm.quantized_matmul(xt, *args, **kw)
    assert ((y.double() - exact).abs().max() / exact.abs().max()).item() <= TOL[x]
