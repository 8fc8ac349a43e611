"""`g * logistic(g) * u` of a program in one pass, against float64: operands in either order, element counts that are
and are not whole 16-byte pieces, an inner value that is also returned (never fused). Needs a B200."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _program(shape, el, swap, keep):
    t = f"tensor<{shape[0]}x{shape[1]}x{el}>"
    inner, outer = ("%0, %arg0", "%arg1, %1") if swap else ("%arg0, %0", "%1, %arg1")
    out, types = ("%2, %1", f"{t}, {t}") if keep else ("%2", t)
    return (f"module @gate {{\n  func.func public @main(%arg0: {t}, %arg1: {t}) -> ({types}) {{\n"
            f"    %0 = stablehlo.logistic %arg0 : {t}\n    %1 = stablehlo.multiply {inner} : {t}\n"
            f"    %2 = stablehlo.multiply {outer} : {t}\n    return {out} : {types}\n  }}\n}}\n")


@pytest.mark.parametrize("shape", [(1, 8), (3, 5), (1, 2056), (7, 1001), (512, 11264)])
@pytest.mark.parametrize("el,dtype,unit", [("bf16", torch.bfloat16, 2.0 ** -8), ("f16", torch.float16, 2.0 ** -11)])
@pytest.mark.parametrize("swap,keep", [(False, False), (True, False), (False, True)])
def test_gate(shape, el, dtype, unit, swap, keep):
    from metaljax_b200 import recognizer
    g = torch.Generator(device=DEV).manual_seed(shape[1])
    gate, up = (torch.randn(shape, generator=g, device=DEV).to(dtype) for _ in range(2))
    it = recognizer.Interpreter(_program(shape, el, swap, keep))
    got = it.execute([gate, up])[0]
    assert len(it._qmm.plan) == (3 if keep else 1)
    exact = gate.double() * torch.sigmoid(gate.double()) * up.double()
    # Three roundings at most, each of `unit` = half of the spacing above 1 (bf16 keeps 8 bits: 2^-8; f16 11: 2^-11); f16 results below 2^-14 round to multiples of 2^-24.
    assert got.dtype == dtype and ((got.double() - exact).abs() <= 3.1 * unit * exact.abs() + 2.0 ** -22 * (1 + up.double().abs())).all()
