"""Eager calls see what the kernels before them in the stream wrote, inputs and weights alike, although their blocks may be
placed before those have ended (csrc/stream_order.cuh): the same buffers written anew ahead of every call, nothing waited for."""
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
