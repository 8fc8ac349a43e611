"""A stored int4 Dense layer packed on the device against the same call on host arrays (the general way):
every word and table entry the same, at the edges of the 64 x 256 tile, odd column counts, group sizes that
allow 128, 64 and 32 codes per table entry, and tables that have to stay float32. Needs a B200."""

import ctypes

import pytest
import torch

from metaljax_b200 import _lib, qmm

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


@pytest.mark.parametrize("k,n,groups,sdt,zdt,constant", [
    (32, 1, 1, torch.bfloat16, torch.bfloat16, False), (256, 64, 2, torch.bfloat16, torch.int8, False),
    (288, 65, 3, torch.float16, torch.float16, False), (320, 63, 5, torch.float32, torch.float32, False),
    (1024, 130, 32, torch.bfloat16, None, False), (1024, 130, 32, torch.bfloat16, torch.uint8, True),
    (512, 7, 8, torch.float16, None, False), (4096, 200, 32, torch.bfloat16, torch.bfloat16, False),
])
def test_device_pack_is_the_host_pack(k, n, groups, sdt, zdt, constant):
    g = torch.Generator().manual_seed(k + n)
    packed = torch.randint(-128, 128, (k, -(-n // 2)), generator=g, dtype=torch.int8)
    if n % 2:
        packed[:, -1] &= 15                                   # (the column past the last one is zero)
    rows = 1 if constant else groups
    scale = (torch.rand((rows, n), generator=g) * 0.02 + 0.01).to(sdt).expand(groups, n).contiguous()
    zero = None
    if zdt is not None:
        zero = torch.randint(0, 5, (rows, n), generator=g).to(zdt).expand(groups, n).contiguous()
    want = qmm.from_keras_int4(packed, scale, zero, columns=n)
    got = qmm.from_keras_int4(packed.to(DEV), scale.to(DEV), None if zero is None else zero.to(DEV), columns=n)
    assert (got.gs, got.bits, got.mode, got.scales.dtype) == (want.gs, want.bits, want.mode, want.scales.dtype)
    assert torch.equal(got.w.cpu().view(torch.int32), want.w.view(torch.int32))
    assert torch.equal(got.scales.cpu(), want.scales) and torch.equal(got.biases.cpu(), want.biases)


def test_device_pack_rejects_what_the_host_pack_rejects():
    packed = torch.zeros((256, 3), dtype=torch.int8, device=DEV)
    scale = torch.full((4, 6), 0.5, device=DEV)
    zero = torch.full((4, 6), 0.5, device=DEV)                # no integer
    with pytest.raises(qmm._Reject):
        qmm.from_keras_int4(packed, scale, zero, columns=6)


def test_a_longer_layer_than_the_device_kernels_take():
    k, n = 1 << 24, 2
    packed = torch.arange(k, dtype=torch.int64).to(torch.int8)[:, None].contiguous()
    scale = torch.full((k // 128, n), 0.5)
    want = qmm.from_keras_int4(packed, scale, columns=n)
    got = qmm.from_keras_int4(packed.to(DEV), scale.to(DEV), columns=n)
    assert (got.gs, got.bits) == (want.gs, want.bits)
    assert torch.equal(got.w.cpu().view(torch.int32), want.w.view(torch.int32)) and torch.equal(got.biases.cpu(), want.biases)


def test_layers_packed_one_after_another_and_by_several_threads():
    """What a layer's blocks add up is nought again when the next one starts, and each call has sums of its own."""
    import threading

    layers, want = [], []
    for i in range(6):
        g = torch.Generator().manual_seed(i)
        packed = torch.randint(-128, 128, (256 + 128 * i, 40), generator=g, dtype=torch.int8)
        scale = (torch.rand((packed.shape[0] // 64, 80), generator=g) * 0.02 + 0.01).to(torch.bfloat16)
        layers.append((packed.to(DEV), scale.to(DEV)))
        want.append(qmm.from_keras_int4(packed, scale))
    wrong = []

    def pack(turn):
        with torch.cuda.stream(torch.cuda.Stream()):
            for i in range(len(layers)):
                at = (i + turn) % len(layers)
                got = qmm.from_keras_int4(*layers[at])
                torch.cuda.current_stream().synchronize()
                if not (torch.equal(got.w.cpu().view(torch.int32), want[at].w.view(torch.int32)) and torch.equal(got.scales.cpu(), want[at].scales)
                        and torch.equal(got.biases.cpu(), want[at].biases)):
                    wrong.append(at)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=pack, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def _layer(packed, scale, zero, group, narrow=False, scale_dtype=None):
    """qmm_pack_dense_layer itself: (status, words, scales, biases, digest, facts)."""
    k, n = packed.shape[0], scale.shape[1]
    words = torch.empty((n, k // 8), dtype=torch.uint32, device=DEV)
    tables = [torch.empty((n, k // group), dtype=scale.dtype if narrow else torch.float32, device=DEV) for _ in range(2)]
    digest, facts = ctypes.c_uint64(), ctypes.c_uint32()
    rc = _lib.lib().qmm_pack_dense_layer(packed.data_ptr(), words.data_ptr(), scale.data_ptr(), None if zero is None else zero.data_ptr(),
                                         _lib.ELEM[scale.dtype] if scale_dtype is None else scale_dtype, 0 if zero is None else _lib.ELEM[zero.dtype],
                                         tables[0].data_ptr(), tables[1].data_ptr(), int(narrow), scale.shape[0], n, k, group, ctypes.byref(digest), ctypes.byref(facts),
                                         _lib.stream_ptr(packed))
    return rc, words, *tables, digest.value, facts.value


def test_what_a_layer_keeps_is_counted_and_given_back():
    """A call's sums and host words stay for the next one; a call that is refused takes none."""
    packed, scale = torch.zeros((64, 4), dtype=torch.int8, device=DEV), torch.ones((1, 8), device=DEV)
    lib = _lib.lib()
    _lib.release_scratch()
    before = _lib.alloc_count()
    for _ in range(3):
        assert _layer(packed, scale, None, 64, scale_dtype=_lib.ELEM[torch.uint8])[0] == 2
    assert _lib.alloc_count() == before and b"scales" in lib.qmm_last_error()
    for _ in range(3):
        assert _layer(packed, scale, None, 64)[0] == 0
    assert _lib.alloc_count() == before + 1
    _lib.release_scratch()
    assert _layer(packed, scale, None, 64)[0] == 0
    assert _lib.alloc_count() == before + 2
