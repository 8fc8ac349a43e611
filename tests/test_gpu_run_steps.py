"""A program of products and gates in one native call, against the same program op by op: equal bit for bit where it is taken, and declined --
not wrong -- where an argument is laid out another way or carries a gradient. Needs a B200."""

import threading

import pytest
import torch

from metaljax_b200 import _lib, recognizer

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
EL = {torch.bfloat16: "bf16", torch.float16: "f16", torch.float32: "f32"}


def program(m, d, f, dtype, gate=True, returns_x=False):
    """silu(x Wg) * (x Wu) Wd, or x Wg Wd; the weights as int8 codes with a scale per group of 32."""
    el, lines, args, count = EL[dtype], [], [f"%arg0: tensor<{m}x{d}x{EL[dtype]}>"], [0]

    def op(text):
        lines.append(f"    %{count[0]} = stablehlo.{text}")
        count[0] += 1
        return f"%{count[0] - 1}"

    def dense(x, k, n):
        i = len(args)
        full, small, wide = f"tensor<{n}x{k}x{el}>", f"tensor<{n}x{k // 32}x{el}>", f"tensor<{n}x{k // 32}x32x{el}>"
        args.extend([f"%arg{i}: tensor<{n}x{k}xi8>", f"%arg{i + 1}: {small}"])
        c = op(f"convert %arg{i} : (tensor<{n}x{k}xi8>) -> {full}")
        b = op(f"broadcast_in_dim %arg{i + 1}, dims = [0, 1] : ({small}) -> {wide}")
        c = op(f"multiply {c}, {op(f'reshape {b} : ({wide}) -> {full}')} : {full}")
        return op(f"dot_general {x}, {c}, contracting_dims = [1] x [1] : (tensor<{m}x{k}x{el}>, {full}) -> tensor<{m}x{n}x{el}>")

    mid = f"tensor<{m}x{f}x{el}>"
    h = dense("%arg0", d, f)
    if gate:
        up = dense("%arg0", d, f)
        act = op(f"multiply {h}, {op(f'logistic {h} : {mid}')} : {mid}")
        h = op(f"multiply {act}, {up} : {mid}")
    y = dense(h, f, d)
    out = f"tensor<{m}x{d}x{el}>"
    results = (f"({out}, {out})", f"return %arg0, {y} : {out}, {out}") if returns_x else (f"({out})", f"return {y} : {out}")
    return "module @jit_f {\n  func.func public @main(" + ", ".join(args) + f") -> {results[0]} {{\n" + "\n".join(lines) + f"\n    {results[1]}\n  }}\n}}\n"


def arguments(m, d, f, dtype, gate=True):
    g = torch.Generator(device=DEV).manual_seed(m + d + f)
    out = [torch.randn((m, d), generator=g, device=DEV).to(dtype)]
    for n, k in ((f, d), (f, d), (d, f)) if gate else ((f, d), (d, f)):
        out.append(torch.randint(-8, 8, (n, k), generator=g, device=DEV, dtype=torch.int8))
        out.append((torch.rand((n, k // 32), generator=g, device=DEV) * 0.018 + 0.002).to(dtype))
    return out


def both(text, args):
    """(in one call or not, the results, the results op by op)"""
    it = recognizer.Interpreter(text)
    it.execute(args)
    plan = it._qmm.plan
    if plan.steps is None:
        return None, None, None
    one = it._run_steps(plan, it._qmm.values, args)
    before = it.fused_calls
    got = it.execute(args)
    assert it.fused_calls == before + plan.products
    steps, plan.steps = plan.steps, None
    want = it.execute(args)
    plan.steps = steps
    assert _lib.poll_status() == 0
    return one is not None, got, want


@pytest.mark.parametrize("m,d,f,dtype,gate,returns_x", [
    (4, 128, 256, torch.bfloat16, True, False), (1, 64, 96, torch.float16, True, True), (33, 160, 288, torch.bfloat16, True, False),
    (200, 256, 512, torch.float16, True, False), (3, 96, 64, torch.float32, False, True), (12, 128, 64, torch.float32, False, False),
])
def test_one_call_equals_op_by_op(m, d, f, dtype, gate, returns_x):
    args = arguments(m, d, f, dtype, gate)
    taken, got, want = both(program(m, d, f, dtype, gate, returns_x), args)
    assert taken
    assert all(torch.equal(a, b) and a.dtype == b.dtype for a, b in zip(got, want))
    if returns_x:
        assert got[0] is args[0]


def test_what_is_not_plain_is_declined():
    text = program(6, 128, 256, torch.bfloat16)
    args = arguments(6, 128, 256, torch.bfloat16)
    wide = torch.randn((6, 256), device=DEV).to(torch.bfloat16)
    for x in (wide[:, ::2], wide[:, 64:192]):
        taken, got, want = both(text, [x, *args[1:]])
        assert taken is False
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    it = recognizer.Interpreter(text)
    it.execute(args)
    with pytest.raises(BufferError):                      # refused, as a call by itself is
        it.execute([args[0].detach().clone().requires_grad_(), *args[1:]])


def test_a_float32_gate_runs_op_by_op():
    args = arguments(4, 64, 96, torch.float32)
    assert both(program(4, 64, 96, torch.float32), args)[0] is None


def test_on_a_stream_of_the_callers():
    """The call enqueues on the current stream: it sees what that stream wrote before, and is replayed from a graph of it."""
    text, args = program(6, 128, 256, torch.bfloat16), arguments(6, 128, 256, torch.bfloat16)
    it = recognizer.Interpreter(text)
    want = it.execute(args)[0].clone()
    other = it.execute([args[0] * 2, *args[1:]])[0].clone()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    x = torch.zeros_like(args[0])
    with torch.cuda.stream(stream):
        torch.cuda._sleep(2_000_000)
        x.copy_(args[0], non_blocking=True)
        got = it.execute([x, *args[1:]])[0]
        stream.synchronize()
        assert torch.equal(got, want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            y = it.execute([x, *args[1:]])[0]
        x.copy_(args[0] * 2)
        graph.replay()
        stream.synchronize()
    assert torch.equal(y, other)


def test_two_threads_at_once():
    """Each on a stream and with arguments of its own, through one interpreter."""
    text = program(5, 128, 256, torch.float16)
    it = recognizer.Interpreter(text)
    sets = [arguments(5, 128, 256, torch.float16) for _ in range(2)]
    sets[1][0] = sets[1][0].flip(0).contiguous()
    want = []
    for args in sets:                                     # (weights of the same values: one plan)
        want.append(it.execute([args[0], *sets[0][1:]])[0].clone())
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(2)

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait()
            for _ in range(200):
                got = it.execute([sets[i][0], *sets[0][1:]])[0]
                torch.cuda.current_stream().synchronize()
                if not torch.equal(got, want[i]):
                    wrong.append(i)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and _lib.poll_status() == 0


@pytest.mark.parametrize("m", [2, 5, 16])
def test_a_product_that_is_read_twice_keeps_its_launch(m):
    """The gate's products are one launch with it (m rows of 2 to 16), but not where the program returns one of them as well."""
    text, args = program(m, 128, 256, torch.bfloat16), arguments(m, 128, 256, torch.bfloat16)
    first = next(line.split("=")[0].strip() for line in text.splitlines() if "dot_general" in line)
    mid, out = f"tensor<{m}x256xbf16>", f"tensor<{m}x128xbf16>"
    last = text.rsplit("return ", 1)[1].split(" ")[0]
    more = text.replace(f"-> ({out}) {{", f"-> ({mid}, {out}) {{").replace(f"return {last} : {out}", f"return {first}, {last} : {mid}, {out}")
    counts = []
    for t in (text, more):
        taken, got, want = both(t, args)
        assert taken and all(torch.equal(a, b) for a, b in zip(got, want))
        it = recognizer.Interpreter(t)
        it.execute(args)
        before = _lib.lib().qmm_launch_count()
        it.execute(args)
        counts.append(_lib.lib().qmm_launch_count() - before)
    assert counts == [2, 4]


@pytest.mark.parametrize("m,d,f,dtype,launches", [(12, 8192, 64, torch.bfloat16, 6), (12, 8160, 64, torch.float16, 2), (1, 128, 256, torch.bfloat16, 4), (17, 128, 256, torch.bfloat16, 4)])
def test_gates_that_keep_their_launches(m, d, f, dtype, launches):
    """One row, 17, and 12 of the longest K are other kernels' than the one that takes both products (the tensor cores' from K = 8192 on, in two launches each): two products, a gate and the product behind it."""
    text, args = program(m, d, f, dtype), arguments(m, d, f, dtype)
    taken, got, want = both(text, args)
    assert taken and all(torch.equal(a, b) for a, b in zip(got, want))
    it = recognizer.Interpreter(text)
    it.execute(args)
    before = _lib.lib().qmm_launch_count()
    it.execute(args)
    assert _lib.lib().qmm_launch_count() - before == launches
