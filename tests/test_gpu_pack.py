"""A stored int4 Dense layer packed on the device against the same call on host arrays (the general way):
every word and table entry the same, at the edges of the 128 x 256 tile, odd column counts, group sizes that
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
    (224, 127, 7, torch.bfloat16, torch.int8, False), (256, 128, 4, torch.bfloat16, None, False),        # a column less, a whole tile,
    (288, 129, 9, torch.float32, torch.uint8, False), (512, 256, 4, torch.float16, torch.int8, False),   # one more (bytes of a row in fours and not), two tiles
    (544, 257, 17, torch.bfloat16, None, False),
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


def _dense(k, n, groups, sdt, zdt, seed=0):
    g = torch.Generator().manual_seed(seed + k + n)
    packed = torch.randint(-128, 128, (k, -(-n // 2)), generator=g, dtype=torch.int8)
    if n % 2:
        packed[:, -1] &= 15
    scale = (torch.rand((groups, n), generator=g) * 0.02 + 0.01).to(sdt)
    zero = None if zdt is None else torch.randint(0, 5, (groups, n), generator=g).to(zdt)
    return packed.to(DEV), scale.to(DEV), None if zero is None else zero.to(DEV)


@pytest.mark.parametrize("k,n", [(256, 128), (288, 129), (224, 127)])
def test_the_digest_tells_layers_apart(k, n):
    """Equal codes have an equal digest, however their bytes lie; one code more or less, or two that change places, another."""
    packed, scale, _ = _dense(k, n, k // 32, torch.float32, None)
    first = _layer(packed, scale, None, 32)
    assert first[0] == 0 and _layer(packed.clone(), scale, None, 32)[4] == first[4]
    shifted = torch.empty(packed.numel() + 1, dtype=torch.int8, device=DEV)[1:].view(packed.shape)      # starts on no word
    shifted.copy_(packed)
    assert _layer(shifted, scale, None, 32)[4] == first[4]
    seen = {first[4]}
    for row, col in ((0, 0), (k - 1, packed.shape[1] - 1), (k // 2, 1)):
        other = packed.clone()
        other[row, col] ^= 1
        seen.add(_layer(other, scale, None, 32)[4])
    other = packed.clone()
    other[[3, 4]] = packed[[4, 3]]
    seen.add(_layer(other, scale, None, 32)[4])
    assert len(seen) == 5


@pytest.mark.parametrize("k,n,groups,sdt,zdt", [(288, 129, 9, torch.bfloat16, torch.int8), (512, 256, 4, torch.float16, None), (1024, 63, 8, torch.float32, torch.float32)])
def test_the_steps_in_a_captured_stream_are_the_layer(k, n, groups, sdt, zdt):
    """Codes, facts and tables by their own entries, which a stream that is being captured takes, against all of it in one, which it does not."""
    packed, scale, zero = _dense(k, n, groups, sdt, zdt)
    group = next(s for s in (128, 64, 32) if k // groups % s == 0)
    _, words, scales, biases, digest, facts = _layer(packed, scale, zero, group)
    lib, types = _lib.lib(), (_lib.ELEM[sdt], 0 if zdt is None else _lib.ELEM[zdt])
    tables = (scale.data_ptr(), None if zero is None else zero.data_ptr(), *types)
    got = [torch.zeros_like(words), torch.zeros_like(scales), torch.zeros_like(biases)]
    sums = torch.zeros(2, dtype=torch.int64, device=DEV)
    stream, refused = torch.cuda.Stream(), []
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        st = stream.cuda_stream
        sums.zero_()
        _lib.check(lib.qmm_pack_dense_codes(packed.data_ptr(), got[0].data_ptr(), k, n, sums.data_ptr(), st))
        _lib.check(lib.qmm_pack_dense_facts(*tables, groups, n, k, sums.data_ptr() + 8, st))
        _lib.check(lib.qmm_pack_dense_tables(*tables, got[1].data_ptr(), got[2].data_ptr(), 0, groups, n, k, group, st))
        d, f = ctypes.c_uint64(), ctypes.c_uint32()
        refused.append(lib.qmm_pack_dense_layer(packed.data_ptr(), words.data_ptr(), *tables, scales.data_ptr(), biases.data_ptr(), 0, groups, n, k, group,
                                                ctypes.byref(d), ctypes.byref(f), st))
    assert refused == [7]
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got[0].view(torch.int32), words.view(torch.int32)) and torch.equal(got[1], scales) and torch.equal(got[2], biases)
    assert sums[0].item() % (1 << 64) == digest and sums[1].item() == facts


@pytest.mark.parametrize("skew", [1, 2, 3])
@pytest.mark.parametrize("k,n", [(32, 1), (288, 9), (256, 262), (544, 515)])
def test_codes_that_start_on_no_word(k, n, skew):
    """Rows of 1, 5, 131 and 258 bytes, the first of which starts on no word, with nothing allocated before or behind it that is this layer's; the words written on no 16 bytes."""
    g = torch.Generator().manual_seed(k + n + skew)
    rows = torch.randint(-128, 128, (k, -(-n // 2)), generator=g, dtype=torch.int8)
    scale = torch.full((k // 32, n), 0.5)
    want = qmm.from_keras_int4(rows, scale, columns=n)
    flat = torch.empty(skew + rows.numel(), dtype=torch.int8, device=DEV)
    packed = flat[skew:].view(rows.shape)
    packed.copy_(rows)
    got = qmm.from_keras_int4(packed, scale.to(DEV), columns=n)
    assert torch.equal(got.w.cpu().view(torch.int32), want.w.view(torch.int32))
    words = torch.zeros(n * (k // 8) + 2, dtype=torch.int32, device=DEV)
    digest = torch.zeros(1, dtype=torch.int64, device=DEV)
    _lib.check(_lib.lib().qmm_pack_dense_codes(packed.data_ptr(), words.data_ptr() + 4, k, n, digest.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(words[1:-1].cpu(), want.w.view(torch.int32).reshape(-1)) and words[0] == 0 and words[-1] == 0


def test_a_tensor_that_requires_a_gradient_is_packed_all_the_same():
    """What the native call declines takes the way through ctypes: the same words."""
    g = torch.Generator().manual_seed(5)
    packed = torch.randint(-128, 128, (256, 33), generator=g, dtype=torch.int8).to(DEV)
    scale = (torch.rand((4, 66), generator=g) * 0.02 + 0.01).to(DEV)
    got, want = qmm.from_keras_int4(packed, scale.clone().requires_grad_()), qmm.from_keras_int4(packed, scale)
    assert torch.equal(got.w.view(torch.int32), want.w.view(torch.int32)) and torch.equal(got.biases, want.biases)
