"""How the few-rows kernel shares a product out, asked without a device (on a machine of 148 SMs)."""

import pytest
import torch

from metaljax_b200 import _lib, qmm

BF16, F16, F32 = torch.bfloat16, torch.float16, torch.float32


def plan(*args, gated=0, **kw):
    out = (_lib.ctypes.c_int32 * 5)(7, 7, 7, 7, 7)
    _lib.check(_lib.lib().qmm_few_rows_plan(_lib.ctypes.byref(qmm._problem(*args, **kw)), gated, out))
    return tuple(out)


@pytest.mark.parametrize("m,k,n,kw,want", [
    (2, 4096, 24576, dict(), (2, 1, 8, 2, 148)),                                                       # two sequences' gate and up, four CTAs of two warps a tile instead: 8 % of a step
    (1, 2048, 28480, dict(bits=8, x_dtype=F32, table_dtype=BF16), (1, 1, 4, 2, 296)),                    # 17.3 us, with clusters of two 25.7
    (1, 4096, 14336, dict(bits=8, x_dtype=F32, table_dtype=BF16), (1, 1, 8, 2, 148)),                    # 18.2 / 25.8
    (2, 14208, 3164, dict(group_size=128, x_dtype=F32), (2, 4, 7, 2, 148)),                              # 17.2 / 18.3 with tiles of 16 rows
    (48, 2816, 8576, dict(group_size=128, bits=8, batch=8, ragged=True), (2, 1, 6, 2, 148)),             # 48 rows of 8 experts: the block 169 / 196 us
])
def test_the_memory_of_tables_and_sums_leaves_the_plan(m, k, n, kw, want):
    """Plans that a few hundred bytes more per warp had changed for slower ones."""
    assert plan(m, k, n, **kw) == want


def test_what_has_no_plan():
    assert plan(1, 4096, 4096) == (0, 0, 0, 0, 0)                          # one row: another kernel's
    assert plan(17, 4096, 4096) == (0, 0, 0, 0, 0)                         # the tensor cores'
    assert plan(8, 4096, 4096, gated=1) != (0, 0, 0, 0, 0) == plan(8, 4096, 4096, gated=1, x_dtype=F32)
    assert _lib.lib().qmm_few_rows_plan(None, 0, (_lib.ctypes.c_int32 * 5)()) == 1


@pytest.mark.parametrize("kind", [dict(), dict(group_size=32), dict(bits=8, group_size=128), dict(mode="mxfp4", group_size=32)])
@pytest.mark.parametrize("x", [BF16, F32])
def test_clusters_are_of_three_warps_and_more(kind, x):
    """Smaller ones were up to 1.7 times slower than what comes next, and chosen by a hair."""
    for k in range(512, 17408, 512):
        for n in (64, 4096, 14336, 24576, 28480):
            for m in (2, 8) if x == BF16 else (1, 4, 8):
                blocks, cluster, warps, ring, ctas = plan(m, k, n, x_dtype=x, **kind)
                assert warps and (cluster == 1 or warps >= 3) and ctas % cluster == 0


@pytest.mark.parametrize("m,k,n,kw,pays", [
    (4, 2048, 5632, dict(), True), (16, 4096, 14336, dict(group_size=128, x_dtype=F16), True),             # us on a B200, one launch / three: 9 / 13.5
    (2, 1280, 11080, dict(bits=8, group_size=128, x_dtype=F16), True),                                     # 11.8 / 14.3
    (4, 3968, 14720, dict(bits=8, group_size=128), False), (16, 3968, 18968, dict(bits=8, group_size=128), False),      # 37.4 / 32.7, 83.0 / 61.7
    (1, 4096, 14336, dict(), False), (17, 4096, 14336, dict(), False), (12, 8192, 1024, dict(), False),    # other kernels'
    (4, 2048, 5632, dict(x_dtype=F32), False), (4, 2048, 5632, dict(y_dtype=F32), False), (4, 0, 64, dict(), False), (4, 64, 0, dict(), False),
    (4, 2048, 5632, dict(group_size=48), False), (4, 2048, 5632, dict(batch=2), False), (4, 2048, 5632, dict(batch=4, ragged=True), False),
])
def test_two_products_and_their_gate_in_one_launch_where_that_is_faster(m, k, n, kw, pays):
    assert _lib.lib().qmm_gated_matmul_pays(_lib.ctypes.byref(qmm._problem(m, k, n, **kw))) == pays
    assert _lib.lib().qmm_gated_matmul_pays(None) == 0
