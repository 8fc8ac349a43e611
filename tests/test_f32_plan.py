"""Which products of float32 activations the tensor-core kernel takes, and in what plan: asked without a device."""

import pytest
import torch

from metaljax_b200 import _lib, qmm


def test_rows_that_are_few_enough_for_the_few_rows_kernel():
    assert qmm.float32_plan(8, 4096, 4096) is None
    assert qmm.float32_plan(9, 4096, 4096) is not None
    with _lib.force_route("f32_tc"):
        assert qmm.float32_plan(8, 4096, 4096) is not None
    with _lib.force_route("simt"):
        assert qmm.float32_plan(9, 4096, 4096) is None


@pytest.mark.parametrize("kind,gs,longest", [("affine", 64, 14336), ("affine8", 64, 12288), ("mxfp4", 32, 14336)])
def test_the_longest_contraction(kind, gs, longest):
    kw = dict(group_size=gs, bits=8 if kind == "affine8" else 4, mode="mxfp4" if kind == "mxfp4" else "affine")
    with _lib.force_route("f32_tc"):
        assert qmm.float32_plan(64, longest, 4096, **kw)[1] == 8
        with pytest.raises(_lib.QmmError):
            qmm.float32_plan(64, longest + gs, 4096, **kw)
    assert qmm.float32_plan(64, longest + gs, 4096, **kw) is None


def test_48_rows_have_no_more_than_512_codes_to_a_cta():
    """Their sums have one level (and one scale)."""
    with _lib.force_route("f32_tc"):
        for k in range(128, 14337, 128):
            rows, cluster, slots = qmm.float32_plan(48, k, 14336)
            assert rows in (16, 32, 48) and cluster in (1, 2, 4, 8) and slots in (1, 2)
            assert rows < 48 or -(-k // 128) <= 4 * cluster


def test_what_it_does_not_take():
    p = qmm._problem(64, 4096, 4096, x_dtype=torch.float32, batch=2)
    plan = (_lib.ctypes.c_int32 * 3)(7, 7, 7)
    _lib.check(_lib.lib().qmm_float32_plan(_lib.ctypes.byref(p), plan))
    assert list(plan) == [0, 0, 0]
    assert _lib.lib().qmm_float32_plan(None, plan) == 1


@pytest.mark.parametrize("m,k,n,kw,taken", [
    (9, 8576, 160, dict(group_size=32, mode="mxfp4"), False),       # us on a B200, few-rows / tensor cores: 9.0 / 16.5
    (14, 8192, 160, dict(group_size=32), False),                    # 9.7 / 15.0
    (44, 2304, 128, dict(group_size=32, bits=8), False),            # 7.5 / 10.5
    (9, 4096, 4096, dict(), True),                                  # 18.2 / 14.0
    (33, 4096, 4096, dict(), True),                                 # 35.5 / 25.0
    (64, 14336, 4096, dict(group_size=32), True),                   # 272 / 185
    (16, 4096, 14336, dict(group_size=32, mode="mxfp4"), True),     # 88 / 47
    (64, 1024, 1024, dict(group_size=128, bits=8), True),           # 14.5 / 8.6
])
def test_the_kernel_that_is_expected_to_be_the_faster(m, k, n, kw, taken):
    plan = qmm.float32_plan(m, k, n, **kw)
    assert (plan is not None) == taken
