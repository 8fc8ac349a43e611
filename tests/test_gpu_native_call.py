"""The calls that go from torch to the library natively: what they decline or meet on the way has to end as it does on
the ctypes way -- in torch's own error, or in the result. Needs a B200."""

import numpy as np
import pytest
import torch

from helpers import activations, affine_case, to_torch
from metaljax_b200 import qmm

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _operands(m=3, n=64, k=128):
    rng = np.random.default_rng(m + n + k)
    return [to_torch(a, DEV) for a in (activations(rng, (m, k)), *affine_case(rng, n, k, 64, 4)[1:])]


def test_a_tensor_without_storage_is_an_error():
    """Inside vmap a tensor has no memory of its own: torch throws where its address is asked for."""
    x, w, s, b = _operands()
    with pytest.raises(Exception, match="(?i)storage|data pointer|dlpack|functorch|vmap"):
        torch.vmap(lambda t: qmm.quantized_matmul(t, w, s, b))(x[None].expand(2, -1, -1))
    assert qmm.quantized_matmul(x, w, s, b).shape == (3, 64)


def test_memory_that_runs_out_is_torchs_error():
    x, w, s, b = _operands(n=1 << 16)
    with pytest.raises(torch.OutOfMemoryError):
        qmm.quantized_matmul(x[:1].expand(1 << 22, -1), w, s, b)       # a result of 512 GiB
