"""The tensor-core kernel where its split of the work can go wrong, against the exact product of the oracle: one K block and
ragged ones, tables whose rows start on no word, tiles added up by clusters, by a second kernel and from worker to
worker, pairs of CTAs whose second half has no features or no tokens. Needs a B200.

Tolerance: the package's parity gate (1e-2 of the largest result): weights and results are rounded to 8 bits (2^-9 of each
value), sums are float32."""

import functools

import numpy as np
import pytest
import torch

from helpers import activations, affine_case, mxfp4_case, to_numpy, to_torch
from metaljax_b200 import _lib, qmm
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@functools.lru_cache(maxsize=None)
def _case(m, k, n, kind, gs, x, tdt):
    rng = np.random.default_rng(m * 7 + k + n)
    if kind == "mxfp4":
        w, s, b, kw = *mxfp4_case(rng, n, k)[1:], None, dict(group_size=32, bits=4, mode="mxfp4")
    else:
        (w, s, b), kw = affine_case(rng, n, k, gs, int(kind[3:]), tdt)[1:], dict(group_size=gs, bits=int(kind[3:]))
    xs = activations(rng, (m, k), x)
    exact = O.qmm_exact(xs, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    return [to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV)], kw, exact


@pytest.mark.parametrize("m,k,n,kind,gs,x,tdt", [
    (17, 96, 130, "int4", 32, "bf16", "bf16"),          # one box and a half block
    (33, 2176, 1300, "int8", 128, "f16", "f16"),        # 17 table entries a row: no word boundary; clusters
    (64, 4160, 700, "int4", 64, "bf16", "f32"),         # few tiles: a second kernel adds up
    (65, 1184, 2200, "int4", 32, "f16", "bf16"),        # 128-row tiles, an odd number of K blocks
    (64, 2048, 19200, "int4", 64, "bf16", "bf16"),      # 150 tiles of 8 boxes: too short to share out
    (64, 4096, 19200, "int4", 64, "bf16", "bf16"),      # ... of 16 boxes: the last round shared out from worker to worker
    (128, 4096, 19200, "int4", 64, "f16", "f16"),       # ... 128 tokens wide
    (64, 7168, 12800, "int4", 64, "bf16", "bf16"),      # 100 tiles, less than a round: all of them shared out
    (33, 4160, 19100, "int8", 32, "bf16", "f32"),       # ... of 33 boxes of two blocks, the last one half empty; no whole last tile
    (300, 4096, 9984, "int4", 64, "bf16", "bf16"),      # 78 tiles of pairs
    (300, 1024, 2050, "int8", 32, "bf16", "f32"),       # pairs in clusters, two features in the last tile
    (513, 2912, 1300, "mxfp4", 32, "bf16", None),       # one token in the last tile, 91 scale bytes a row
    (2048, 3008, 2560, "int4", 64, "bf16", "bf16"),     # 80 tiles on 74 pairs
    (257, 4224, 129, "int8", 128, "bf16", "bf16"),      # one pair, whose second CTA has one feature
])
def test_tensor_core_splits(m, k, n, kind, gs, x, tdt):
    args, kw, exact = _case(m, k, n, kind, gs, x, tdt)
    with _lib.force_route("gemm_tc"):
        y = qmm.quantized_matmul(*args, **kw)
    assert O.rel_err(to_numpy(y).astype(np.float32), exact) <= 1e-2
    assert _lib.poll_status() == 0


SHARED_OUT = [(64, 4096, 19200), (128, 4096, 19200), (64, 7168, 12800), (300, 4096, 9984), (2048, 3008, 2560)]


@pytest.mark.parametrize("m,k,n", SHARED_OUT + [(64, 2048, 19200), (64, 4160, 700), (65, 1184, 2200), (300, 1024, 2304)])
def test_which_products_are_shared_out(m, k, n):
    """Scratch and one launch: handed over from worker to worker. Scratch and two: a second kernel adds up. No scratch: clusters, or a tile each."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the tile counts are for 148 SMs")
    args, kw, _ = _case(m, k, n, "int4", 32 if k % 64 else 64, "bf16", "bf16")
    with _lib.force_route("gemm_tc"):
        qmm.quantized_matmul(*args, **kw)
        allocs, launches = _lib.alloc_count(), _lib.launch_count()
        qmm.quantized_matmul(*args, **kw)
        made = (_lib.alloc_count() - allocs, _lib.launch_count() - launches)
    assert (made == (1, 1)) == ((m, k, n) in SHARED_OUT), made
    assert _lib.poll_status() == 0


@pytest.mark.parametrize("m,k,n", SHARED_OUT)
def test_shared_out_products_replay(m, k, n):
    """A captured launch replays over the scratch it left behind, whose flags must say nothing by then: replayed with other activations, a
    worker that took an earlier replay's partial tile for this one's would show."""
    args, kw, _ = _case(m, k, n, "int4", 64, "bf16", "bf16")
    others = [args[0], args[0].flip(0).contiguous(), (args[0] * -2).contiguous()]
    x, y = torch.empty_like(args[0]), torch.zeros((m, n), device=DEV, dtype=torch.bfloat16)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), _lib.force_route("gemm_tc"):
        want = [qmm.quantized_matmul(o, *args[1:], **kw) for o in others]
        x.copy_(others[0])
        qmm.quantized_matmul(x, *args[1:], out=y, **kw)
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            qmm.quantized_matmul(x, *args[1:], out=y, **kw)
        for i in (0, 1, 2, 1, 0, 2):
            x.copy_(others[i])
            graph.replay()
            stream.synchronize()
            assert torch.equal(y, want[i])
    assert _lib.poll_status() == 0


@pytest.mark.parametrize("m,k,n", [(64, 2048, 19200), (64, 4160, 700), (300, 1024, 2304)])
def test_tensor_core_splits_replay(m, k, n):
    """A captured launch replays over the scratch it left behind (clusters, a second kernel, tiles that are whole)."""
    args, kw, exact = _case(m, k, n, "int4", 32 if k % 64 else 64, "bf16", "bf16")
    y = torch.zeros((m, n), device=DEV, dtype=torch.bfloat16)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream), _lib.force_route("gemm_tc"):
        qmm.quantized_matmul(*args, out=y, **kw)
        stream.synchronize()
        first = y.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(3):
                qmm.quantized_matmul(*args, out=y, **kw)
        for _ in range(3):
            y.zero_()
            graph.replay()
            stream.synchronize()
            assert torch.equal(y, first)
    assert O.rel_err(to_numpy(first).astype(np.float32), exact) <= 1e-2
    assert _lib.poll_status() == 0
