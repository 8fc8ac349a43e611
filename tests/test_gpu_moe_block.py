"""The expert block in one native call against its steps one by one and against the oracle's product pair by pair, at the edges of
the pair sort (one pair, experts without a pair, more pairs than a warp, more than a block's warps) and on either product
kernel. Needs a B200."""

import threading

import numpy as np
import pytest
import torch

from helpers import activations, affine_case, mxfp4_case, to_numpy, to_torch
from metaljax_b200 import _lib, moe
from oracle import qmm_oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _case(rng, kind, n, k, tdt, lead):
    if kind == "mxfp4":
        return (*mxfp4_case(rng, n, k, lead=lead)[1:], None), dict(group_size=32, bits=4, mode="mxfp4")
    return affine_case(rng, n, k, 64, 4, tdt, lead=lead)[1:], dict(group_size=64, bits=4)


def _exact_block(xs, idx, wts, packs, gs, mode):
    """The block in float64 on the dequantized weights, nothing rounded in between."""
    w1, w3, w2 = (O.dequantize(w, s, b, gs, 4, mode).astype(np.float64) for w, s, b in packs)
    out = np.zeros((len(xs), w2.shape[1]))
    for t, x in enumerate(xs.astype(np.float64)):
        for e, weight in zip(idx[t], wts[t].astype(np.float64)):
            gate = w1[e] @ x
            out[t] += weight * (w2[e] @ (gate / (1.0 + np.exp(-gate)) * (w3[e] @ x)))
    return out


@pytest.mark.parametrize("tokens,experts,k", [(1, 4, 1), (3, 8, 2), (33, 40, 4), (150, 4, 2)])
@pytest.mark.parametrize("kind,x,index", [("int4", "bf16", torch.int64), ("mxfp4", "f16", torch.int32)])
def test_expert_block_in_one_call(kind, x, index, tokens, experts, k):
    """Against the block's steps one by one: the same kernels on either side of the same 16-bit hand-offs, so
    what differs is the order of float32 sums (a chunk of rows may be another width) and what 8 bits make of that: the parity gate. And against
    float64: gate, up, SwiGLU (twice) and down are rounded to 16 bits, five independent errors of 2^-9 a value of which
    the down projection averages four over 320 terms: the parity gate again."""
    rng = np.random.default_rng(tokens + experts)
    d, f = 192, 320
    packs, host, kw = [], [], None
    for n, kk in ((f, d), (f, d), (d, f)):
        arrays, kw = _case(rng, kind, n, kk, x, lead=(experts,))
        host.append(arrays)
        packs.append(tuple(None if a is None else to_torch(a, DEV) for a in arrays))
    xs_host = activations(rng, (tokens, d), x, 0.5)
    xs = to_torch(xs_host, DEV)
    idx = torch.from_numpy(np.stack([rng.permutation(experts)[:k] for _ in range(tokens)])).to(index).to(DEV)
    wts = torch.from_numpy(rng.random((tokens, k)).astype(np.float32)).to(DEV)
    got = moe.moe_experts(xs, idx, wts, *packs, **kw)
    exact = _exact_block(xs_host, idx.cpu().numpy(), wts.cpu().numpy(), host, kw["group_size"], kw.get("mode", "affine"))
    assert O.rel_err(to_numpy(got).astype(np.float32), exact) <= 1e-2
    order, tok, sizes = moe.sort_pairs(idx.to(torch.int64), experts)
    rows = xs.index_select(0, tok)
    act = moe.silu_mul(moe.ragged_dot(rows, *packs[0], sizes, **kw), moe.ragged_dot(rows, *packs[1], sizes, **kw))
    want = moe.routed_sum(moe.ragged_dot(act, *packs[2], sizes, **kw), order, wts, tokens, k)
    assert O.rel_err(to_numpy(got).astype(np.float32), to_numpy(want).astype(np.float64)) <= 1e-2
    for outside in (experts, -1, 1 << 20):                    # an index outside the experts: refused, never followed
        bad = idx.clone()
        bad[-1, -1] = outside
        with pytest.raises(RuntimeError):
            moe.moe_experts(xs, bad, wts, *packs, **kw)
    assert torch.equal(moe.moe_experts(xs, idx, wts, *packs, **kw), got) and _lib.poll_status() == 0


def test_activations_at_any_address():
    """A contiguous view that starts on no 16-byte boundary: the same result as a copy of it."""
    rng = np.random.default_rng(3)
    d, f, t = 192, 320, 5
    packs = []
    for n, kk in ((f, d), (f, d), (d, f)):
        arrays, kw = _case(rng, "int4", n, kk, "bf16", lead=(4,))
        packs.append(tuple(to_torch(a, DEV) for a in arrays))
    flat = to_torch(activations(rng, (4 + t * d,)), DEV)
    x = flat[4:].view(t, d)
    assert x.data_ptr() % 16
    idx = torch.from_numpy(rng.integers(0, 4, (t, 2))).to(DEV)
    wts = torch.rand((t, 2), device=DEV)
    got, want = moe.moe_experts(x, idx, wts, *packs, **kw), moe.moe_experts(x.clone(), idx, wts, *packs, **kw)
    assert O.rel_err(to_numpy(got).astype(np.float32), to_numpy(want).astype(np.float64)) <= 1e-2


def _small_block(t=6, experts=4, d=192, f=320):
    rng = np.random.default_rng(9)
    packs = []
    for n, kk in ((f, d), (f, d), (d, f)):
        arrays, kw = _case(rng, "int4", n, kk, "bf16", lead=(experts,))
        packs.append(tuple(to_torch(a, DEV) for a in arrays))
    x = to_torch(activations(rng, (t, d), "bf16", 0.5), DEV)
    idx = torch.from_numpy(rng.integers(0, experts, (t, 2))).to(DEV)
    return x, idx, torch.rand((t, 2), device=DEV), packs, kw


def test_captured_block():
    """In a graph nothing can be looked at by the host: a replay computes, and an index out of range is reported by the status."""
    x, idx, wts, packs, kw = _small_block()
    want = moe.moe_experts(x, idx, wts, *packs, **kw)
    index, stream = idx.clone(), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        y = moe.moe_experts(x, index, wts, *packs, **kw)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and _lib.poll_status() == 0
    index[0, 0] = 4
    graph.replay()
    with pytest.raises(_lib.QmmError):
        _lib.poll_status()


def test_blocks_of_several_threads():
    """Every call waits for the report of its own sort: one thread's indices are out of range, and it alone is refused."""
    x, idx, wts, packs, kw = _small_block()
    want = moe.moe_experts(x, idx, wts, *packs, **kw)
    bad = idx.clone()
    bad[3, 1] = -7
    torch.cuda.synchronize()
    outcome = {}

    def calls(number):
        refused, right = 0, 0
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(25):
                try:
                    y = moe.moe_experts(x, bad if number == 2 else idx, wts, *packs, **kw)
                    torch.cuda.current_stream().synchronize()
                    right += bool(torch.equal(y, want))
                except _lib.QmmError:
                    refused += 1
        outcome[number] = (refused, right)

    threads = [threading.Thread(target=calls, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert outcome == {0: (0, 25), 1: (0, 25), 2: (25, 0), 3: (0, 25)} and _lib.poll_status() == 0


@pytest.mark.parametrize("kind,d,f,launches", [("int8", 896, 2944, 6), ("int8", 2304, 320, 4), ("int4", 896, 2944, 4)])
def test_both_products_in_one_launch_where_that_is_faster(kind, d, f, launches):
    """8-bit codes of many tiles have both products of the block by themselves and a gate behind them, the others one launch: the sort, that, the down projection and the weighted sum."""
    rng = np.random.default_rng(d + f)
    experts, tokens, k, bits = 8, 6, 2, int(kind[3:])
    host = [affine_case(rng, n, kk, 64, bits, "bf16", lead=(experts,))[1:] for n, kk in ((f, d), (f, d), (d, f))]
    packs = [tuple(to_torch(a, DEV) for a in arrays) for arrays in host]
    xs_host = activations(rng, (tokens, d), "bf16", 0.25)
    xs = to_torch(xs_host, DEV)
    idx = torch.from_numpy(np.stack([rng.permutation(experts)[:k] for _ in range(tokens)])).to(DEV)
    wts = torch.from_numpy(rng.random((tokens, k)).astype(np.float32)).to(DEV)
    kw = dict(group_size=64, bits=bits)
    got = moe.moe_experts(xs, idx, wts, *packs, **kw)
    before = _lib.lib().qmm_launch_count()
    assert torch.equal(moe.moe_experts(xs, idx, wts, *packs, **kw), got)
    assert _lib.lib().qmm_launch_count() - before == launches
    w1, w3, w2 = (O.dequantize(w, s, b, 64, bits, "affine").astype(np.float32) for w, s, b in host)
    exact = np.zeros((tokens, d))
    for t, x in enumerate(xs_host.astype(np.float64)):
        for e, weight in zip(idx[t].tolist(), wts[t].tolist()):
            gate = w1[e] @ x
            exact[t] += weight * (w2[e] @ (gate / (1.0 + np.exp(-gate)) * (w3[e] @ x)))
    assert O.rel_err(to_numpy(got).astype(np.float32), exact) <= 1e-2
