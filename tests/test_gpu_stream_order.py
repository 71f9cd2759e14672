"""Eager calls see what the kernels before them in the stream wrote, inputs and weights alike, although their blocks may be
placed before those have ended (csrc/stream_order.cuh): the same buffers written anew ahead of every call, nothing waited for."""
import ctypes

import pytest
import torch

from qwen38_flash_ops_b200 import ArgmaxRows, DequantWeightBf16, LmHeadArgmax, SharedExpertDown, SkinnyGemm
from qwen38_flash_ops_b200 import workloads as W

pytestmark = pytest.mark.gpu
ROUNDS = 8


def _rand(seed, *shape):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, generator=gen, device="cuda").bfloat16()


def _case(kind, mode, seed):
    """The tensors of a call."""
    K, N = 1024, 4096
    w = W.make_weight(mode, K, N, seed)[0]
    if kind in ("few", "many", "head"):
        return {"x": _rand(seed, 40 if kind == "many" else 4, K), "w": w}
    if kind == "shared":
        return {"g": _rand(seed, 40, K), "u": _rand(seed + 1, 40, K), "w": w, "gx": _rand(seed + 2, 40, 256), "gw": _rand(seed + 3, 256, 1) * 0.02,
                "routed": _rand(seed + 4, 40, N)}
    return {"x": _rand(seed, 16, 40 * N)} if kind == "argmax" else {"w": w}


def _op(kind):
    N = 4096
    if kind in ("few", "many"):
        op = SkinnyGemm([2], [N // 4, 3 * N // 4])
        return lambda t: op(t["x"], t["w"])
    if kind == "head":
        op = LmHeadArgmax()
        return lambda t: list(op(t["x"], t["w"], N))
    if kind == "shared":
        op = SharedExpertDown()
        return lambda t: [op(t["g"], t["u"], t["w"], t["gx"], t["gw"], t["routed"])]
    if kind == "argmax":
        op = ArgmaxRows()
        return lambda t: list(op(t["x"]))
    op = DequantWeightBf16(N)
    return lambda t: op(t["w"])


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("kind", ["few", "many", "head", "shared", "argmax", "dequant"])
def test_inputs_written_just_before(cuda, kind, mode):
    if kind == "head" and mode != 2 or kind == "argmax" and mode != 0:
        pytest.skip("one type is enough")
    op, sources = _op(kind), [_case(kind, mode, 50 * i + mode) for i in range(ROUNDS)]
    alone = []
    for s in sources:
        alone.append([o.clone() for o in op(s)])
        torch.cuda.synchronize()
    shared = {k: torch.empty_like(v) for k, v in sources[0].items()}
    delay = torch.empty(1 << 24, device="cuda")
    got = []
    for s in sources:
        delay.fill_(1.0)  # the copies behind it are in the stream before it is done
        for k, v in s.items():
            shared[k].copy_(v)
        got.append(op(shared))
    torch.cuda.synchronize()
    for a, g in zip(alone, got):
        assert all(torch.equal(p.view(torch.uint8), q.view(torch.uint8)) for p, q in zip(a, g))


def test_calls_of_the_library_in_a_row(cuda):
    """A weight dequantised, multiplied by, its logits sampled: each call reads what the one before it writes."""
    K, N = 2560, 8192
    weights, x = [W.make_weight(2, K, N, i)[0] for i in range(ROUNDS)], _rand(3, 4, K)
    deq, gemm, top = DequantWeightBf16(N), SkinnyGemm([1], [N]), ArgmaxRows()
    w = torch.empty(K, N, dtype=torch.bfloat16, device="cuda")
    got = []
    for s in weights:
        deq(s, out=[w])
        got.append(top(gemm(x, w)[0]))
    torch.cuda.synchronize()
    for s, g in zip(weights, got):
        deq(s, out=[w])
        torch.cuda.synchronize()
        y = gemm(x, w)[0]
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(top(y), g))


# ---- a predecessor that lets its dependents in at its start and writes what they read at its end, 140 us later


class _Early:
    """Ten blocks of a general kernel, which releases its dependents first of all; the other SMs are free for them.  Writes [8, 2560]."""

    def __init__(self):
        self.op = SkinnyGemm([1], [2560], trigger=1)
        self.op.set_option("plan", "direct=0,wn=2,wk=4,cluster=1,ctas=10")
        self.w, self.xs = _rand(900, 8192, 2560) * 0.02, [_rand(901 + i, 8, 8192) for i in range(2)]

    def __call__(self, i, out):
        self.op(self.xs[i % 2], self.w, out=[out])


def _weight_in(mode, buffer):
    """The bytes of a [8, 2560] BF16 buffer as a weight: (weight, K, N)."""
    raw = buffer.view(torch.uint8).reshape(-1)
    if mode == 0:
        return buffer.reshape(80, 256), 80, 256
    return (raw.view(torch.float8_e4m3fn).reshape(160, 256), 160, 256) if mode == 1 else (raw[:280 * 144].reshape(280, 144), 280, 256)


def _successor(kind, reads, mode, plan):
    """A call that reads `reads` out of rows 32 to 39 of a [40, 2560] buffer: buffer -> outputs."""
    K, N = 2560, 1024
    if kind == "argmax":
        op = ArgmaxRows()
        return lambda b: list(op(b[32:]))
    if kind == "dequant":
        op = DequantWeightBf16(256)
        return lambda b: op(_weight_in(mode, b[32:])[0])
    if kind == "head":
        op, w = LmHeadArgmax(), W.make_weight(mode, K, 4096, 7)[0]
        return lambda b: list(op(b[32:], w, 4096))
    many = kind.startswith("many")
    if kind.endswith("shared"):
        op = SharedExpertDown()
        rows = 40 if many else 8
        w, u, gx, gw, routed = W.make_weight(mode, K, N, 7)[0], _rand(8, rows, K), _rand(9, rows, 256), _rand(10, 256, 1) * 0.02, _rand(11, rows, N)
        return lambda b: [op(b if many else b[32:], u, w, gx, gw, routed)]
    if reads == "weight":
        _, K, N = _weight_in(mode, torch.empty(8, 2560, dtype=torch.bfloat16, device="cuda"))
        x = _rand(12, 40 if many else 8, K)
    op = SkinnyGemm([1], [N])
    op.set_option("dense_plan", plan if many else "0")
    if reads == "weight":
        return lambda b: op(x, _weight_in(mode, b[32:])[0])
    w = W.make_weight(mode, K, N, 7)[0]
    return lambda b: op(b if many else b[32:], w)


@pytest.mark.parametrize("kind,reads,mode,plan", [
    ("argmax", "x", 0, ""), ("head", "x", 2, "")] + [(k, r, m, p) for m in (0, 1, 2) for k, r, p in [
        ("dequant", "weight", ""), ("few", "x", ""), ("few", "weight", ""), ("few shared", "x", ""), ("many shared", "x", ""),
        ("many", "x", "48,1,0"), ("many", "x", "48,4,0"), ("many", "x", "64,1,1"), ("many", "x", "256,1,0,1"), ("many", "weight", "48,1,0"),
        ("many", "weight", "48,2,0"), ("many", "weight", "64,1,1"), ("many", "weight", "256,1,0,1")]])
def test_behind_a_predecessor_that_released_its_dependents(cuda, kind, reads, mode, plan):
    early, call, buffer = _Early(), _successor(kind, reads, mode, plan), _rand(920, 40, 2560)
    alone = []
    for i in range(2):
        early(i, buffer[32:])
        torch.cuda.synchronize()
        alone.append([o.clone() for o in call(buffer)])
        torch.cuda.synchronize()
    got = []
    for i in range(12):
        early(i, buffer[32:])
        got.append(call(buffer))
        if i % 3 == 2:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    for i, g in enumerate(got):
        assert all(torch.equal(p.view(torch.uint8), q.view(torch.uint8)) for p, q in zip(alone[i % 2], g)), i


@pytest.mark.parametrize("kind", ["few", "many", "head", "shared", "argmax", "dequant"])
@pytest.mark.parametrize("order", ["event", "default behind blocking"])
def test_inputs_written_by_another_stream(cuda, kind, order):
    """A stream that waits for the writer's event, and the default stream behind a blocking one, with nothing said."""
    mode = 0 if kind == "argmax" else 2
    op, sources = _op(kind), [_case(kind, mode, 50 * i + 1) for i in range(4)]
    alone = []
    for s in sources:
        alone.append([o.clone() for o in op(s)])
        torch.cuda.synchronize()
    shared = {k: torch.empty_like(v) for k, v in sources[0].items()}
    delay = torch.empty(1 << 24, device="cuda")
    runtime, handle = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p()
    if order == "event":
        writer, reader = torch.cuda.Stream(), torch.cuda.Stream()
    else:
        assert runtime.cudaStreamCreate(ctypes.byref(handle)) == 0
        writer, reader = torch.cuda.ExternalStream(handle.value), torch.cuda.default_stream()
    torch.cuda.synchronize()
    got = []
    for s in sources * 2:
        if order == "event":
            writer.wait_stream(reader)
        with torch.cuda.stream(writer):
            delay.fill_(1.0)
            for k, v in s.items():
                shared[k].copy_(v)
        if order == "event":
            reader.wait_stream(writer)
        with torch.cuda.stream(reader):
            got.append(op(shared))
    torch.cuda.synchronize()
    for a, g in zip(alone * 2, got):
        assert all(torch.equal(p.view(torch.uint8), q.view(torch.uint8)) for p, q in zip(a, g))
    if handle.value:
        assert runtime.cudaStreamDestroy(handle) == 0
