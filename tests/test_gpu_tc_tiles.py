"""Tiles of fewer tokens than the tensor-core kernel's widest, which it takes where those would leave pairs of CTAs without one, and MXFP4 codes
looked up in bytes of their scaled magnitudes, against the exact product of the oracle. Needs a B200.

Tolerance: the package's parity gate (1e-2 of the largest result): weights and results are rounded to 8 bits (2^-9 of each
value), sums are float32."""

import numpy as np
import pytest

from helpers import activations, affine_case, mxfp4_case, to_numpy, to_torch
from metaljax_b200 import _lib, qmm
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("m,k,n,kind,gs,x", [
    (512, 704, 5760, "mxfp4", 32, "bf16"),      # 46 tiles of 256, 69 of 192
    (449, 576, 6144, "int4", 64, "bf16"),       # 48, 72 of 160, the last of 129
    (600, 320, 4608, "int8", 32, "f16"),        # 54, 72 of 160
    (130, 96, 11000, "mxfp4", 32, "f16"),       # one short tile of tokens
    (64, 2080, 300, "mxfp4", 32, "bf16"),
])
def test_tiles_of_fewer_tokens(m, k, n, kind, gs, x):
    rng = np.random.default_rng(m + k + n)
    if kind == "mxfp4":
        w, s, b, kw = *mxfp4_case(rng, n, k)[-2:], None, dict(group_size=32, bits=4, mode="mxfp4")
    else:
        (w, s, b), kw = affine_case(rng, n, k, gs, int(kind[3:]), x)[1:], dict(group_size=gs, bits=int(kind[3:]))
    xs = activations(rng, (m, k), x)
    exact = O.qmm_exact(xs, w, s, b, kw["group_size"], kw["bits"], mode=kw.get("mode", "affine"))
    with _lib.force_route("gemm_tc"):
        y = qmm.quantized_matmul(to_torch(xs, DEV), to_torch(w, DEV), to_torch(s, DEV), None if b is None else to_torch(b, DEV), **kw)
    assert O.rel_err(to_numpy(y).astype(np.float32), exact) <= 1e-2
    assert _lib.poll_status() == 0
