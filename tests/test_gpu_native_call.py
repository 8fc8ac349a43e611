"""The calls that go from torch to the library natively: what they decline or meet on the way has to end as it does on
the ctypes way -- in torch's own error, or in the result. Needs a B200."""

import ctypes
import importlib.machinery
import importlib.util
import shutil
import subprocess
import threading
import time

import numpy as np
import pytest
import torch

from helpers import activations, affine_case, to_torch
from metaljax_b200 import _lib, qmm

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


_SLOW = """
#include <unistd.h>
int slow_product() { usleep(300000); return 0; }
long long slow_workspace() { return 4096; }
int slow_block() { usleep(300000); return 0; }
"""


@pytest.mark.parametrize("call", ["quantized_matmul", "moe_experts"])
def test_other_threads_run_while_a_call_waits(call, tmp_path):
    """An enqueue can wait for the device (its launch queue is full), and the device for another thread of Python. The binding is given
    entry points that take 0.3 s and do nothing: another thread has to get on meanwhile."""
    source, library = tmp_path / "slow.c", tmp_path / "slow.so"
    source.write_text(_SLOW)
    subprocess.check_call([shutil.which("gcc") or "cc", "-shared", "-fPIC", str(source), "-o", str(library)])
    slow = ctypes.CDLL(str(library))
    loader = importlib.machinery.ExtensionFileLoader("_native", _lib.NATIVE_PATH)
    native = importlib.util.module_from_spec(importlib.util.spec_from_loader("_native", loader))
    loader.exec_module(native)
    ours = [ctypes.cast(getattr(_lib.lib(), name), ctypes.c_void_p).value for name in ("qmm_quantized_matmul", "qmm_moe_workspace_bytes", "qmm_moe_experts_checked")]
    x, w, s, b = _operands(m=4, n=128, k=128)
    idx = torch.zeros((4, 1), dtype=torch.int64, device=DEV)
    weights = torch.ones((4, 1), device=DEV)
    expert = (w[None].contiguous(), s[None].contiguous(), b[None].contiguous())
    ticks, done = [], threading.Event()

    def tick():
        while not done.is_set():
            ticks.append(time.monotonic())
            time.sleep(0.002)

    other = threading.Thread(target=tick)
    other.start()
    try:
        native.bind(*(ctypes.cast(getattr(slow, name), ctypes.c_void_p).value for name in ("slow_product", "slow_workspace", "slow_block")))
        before = len(ticks)
        start = time.monotonic()
        if call == "quantized_matmul":
            native.quantized_matmul(x, w, s, b, True, 64, 4, 0, None, None)
        else:
            native.moe_experts(x, idx, weights, *expert, *expert, *expert, 64, 4, 0)
        took, ran = time.monotonic() - start, len(ticks) - before
    finally:
        native.bind(*ours)                         # (the addresses are the module's, and a module is loaded once)
        done.set()
        other.join()
    assert took >= 0.3 and ran >= 20               # 150 ticks of 2 ms fit; with the lock held it is one or two
