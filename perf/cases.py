"""The calls that a program using this package spends its time in, for timing: the decode projections and the
LM head (one to eight rows of activations against resident weights), the same projections with the rows of a
batch or of a prompt, the shared expert's down projection in both regimes, argmax over logits, and the
dequantisation of a weight.

Shapes are those of the package's workloads, tests and benchmark (K = 5120 and K = 2560 models); activations are
N(0, 1) in BF16, weights N(0, 0.02^2) quantised the way each format is quantised.  A case is a dict:

  op      gemm | lmhead | shared | argmax | dequant
  dtype   bf16 | fp8 | nvfp4 (weights), or bf16 | f16 | f32 (logits)
  rows    rows of x (gemm, lmhead, shared), or of the logits (argmax)
  k       inner dimension (weight rows)
  widths  output widths: "," separates the outputs that slice one weight, "/" separates weights
  scaled  whether the op is given a per-column w_scale
"""
import torch

from qwen38_flash_ops_b200 import ArgmaxRows, DequantWeightBf16, LmHeadArgmax, SharedExpertDown, SkinnyGemm
from qwen38_flash_ops_b200 import workloads as W

_MODE = {"bf16": W.MODE_BF16, "fp8": W.MODE_FP8, "nvfp4": W.MODE_NVFP4}
_LOGITS = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
_GATE = 2560  # length of the shared expert's gate vector: the model width


def _case(name, op, dtype, rows, k, widths, scaled=False):
    c = {"op": op, "dtype": dtype, "rows": rows, "k": k, "widths": widths, "scaled": scaled}
    return {"name": name, **c} if name else c


def listed():
    return [
        # decode, one token: attention output projection, BF16 weights
        _case("decode_o_proj_bf16", "gemm", "bf16", 1, 5120, "5120"),
        # decode, two tokens: q, k and v in one call over three FP8 weights
        _case("decode_qkv_fp8", "gemm", "fp8", 2, 5120, "8192/1024/1024", True),
        # decode, one token: the MLP's gate and up projections, NVFP4 weights
        _case("decode_gate_up_nvfp4", "gemm", "nvfp4", 1, 5120, "17408/17408"),
        # decode with four speculated tokens: the MLP's down projection (long K, narrow N)
        _case("decode_down_nvfp4", "gemm", "nvfp4", 4, 17408, "5120"),
        # the same step's vocabulary projection with the greedy token taken in the kernel
        _case("decode_lm_head_nvfp4", "lmhead", "nvfp4", 4, 5120, "151936"),
        # the smallest call of a decode step: the shared expert of a K = 2560 mixture-of-experts layer
        _case("decode_shared_expert_nvfp4", "shared", "nvfp4", 4, 640, "2560"),
        # a batch of sequences decoded together: more rows than one streaming pass takes, an odd number
        _case("batch_up_nvfp4", "gemm", "nvfp4", 33, 5120, "17408"),
        # the tail of a chunked prompt, a ragged number of rows
        _case("prefill_qkv_fp8", "gemm", "fp8", 509, 5120, "8192/1024/1024", True),
        # a full prompt chunk, weights with a global scale beside the block scales
        _case("prefill_up_nvfp4", "gemm", "nvfp4", 2048, 5120, "17408", True),
        # the shared expert over a prompt
        _case("prefill_shared_expert_fp8", "shared", "fp8", 777, 640, "2560", True),
        # greedy sampling for a batch from logits that another op produced
        _case("sample_argmax_bf16", "argmax", "bf16", 64, 0, "151936"),
        # an NVFP4 weight handed to an op that wants BF16
        _case("dequant_up_nvfp4", "dequant", "nvfp4", 0, 5120, "17408", True),
    ]


def _segments(case):
    return [[int(v) for v in w.split(",")] for w in case["widths"].split("/")]


def _weight_bytes(dtype, k, n):
    return {"bf16": 2 * k * n, "fp8": k * n, "nvfp4": k * n * 9 // 16}[dtype]


def _log_int(rng, lo, hi, step=1):
    v = lo * (hi / lo) ** rng.random()
    return max(lo, min(hi, int(round(v / step)) * step))


def _split(rng, n, step):
    """n columns over one to three outputs, in multiples of `step`."""
    parts = rng.choice([1, 1, 2, 3])
    cuts = sorted({0, n, *(rng.randrange(1, max(2, n // step)) * step for _ in range(parts - 1))})
    return ",".join(str(b - a) for a, b in zip(cuts, cuts[1:]) if b > a)


def draw(rng):
    largest = max(work(c)["flops"] for c in listed())
    op = rng.choice(["gemm"] * 5 + ["batch"] * 4 + ["shared"] * 3 + ["lmhead", "argmax", "dequant"])
    dtype = rng.choice(["bf16", "fp8", "nvfp4"])
    scaled = dtype == "fp8" or (dtype == "nvfp4" and rng.random() < 0.5)
    step = 128 if dtype == "nvfp4" else 16
    if op == "lmhead":
        return _case(None, "lmhead", "nvfp4", rng.randint(1, 8), _log_int(rng, 1024, 5120, 16),
                     str(_log_int(rng, 16384, 151936, 128)))
    if op == "argmax":
        dtype = rng.choice(["bf16", "f16", "f32"])
        return _case(None, "argmax", dtype, _log_int(rng, 1, 128), 0, str(_log_int(rng, 16384, 151936)))
    if op == "dequant":
        n = _log_int(rng, 1024, 17408, step)
        return _case(None, "dequant", dtype, 0, _log_int(rng, 640, 17408, 16), _split(rng, n, step), scaled)
    if op == "shared":
        return _case(None, "shared", dtype, _log_int(rng, 1, 2048), _log_int(rng, 256, 2560, 16),
                     str(_log_int(rng, 1024, 5120, step)), scaled)
    rows = rng.randint(1, 8) if op == "gemm" else _log_int(rng, 9, 2048)
    while True:
        k = _log_int(rng, 320, 17408, 16)
        weights = "/".join(_split(rng, _log_int(rng, 512, 17408, step), step) for _ in range(rng.choice([1, 1, 2, 3])))
        c = _case(None, "gemm", dtype, rows, k, weights, scaled)
        outputs = len(weights.replace("/", ",").split(","))  # one call has at most eight
        if outputs <= 8 and work(c)["flops"] <= largest and work(c)["bytes"] <= 400e6:
            return c


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000 + 17)
    op, rows, k = case["op"], case["rows"], case["k"]
    segs = _segments(case)
    if op == "argmax":
        # logits of a vocabulary projection: about N(0, 1.4^2) in the type the projection wrote
        x = torch.randn(rows, segs[0][0], generator=gen, device="cuda") * 1.4
        return {"op": op, "node": ArgmaxRows(), "x": x.to(_LOGITS[case["dtype"]])}
    weights, scales = [], []
    for i, outs in enumerate(segs):
        n = sum(outs)
        w, s = W.make_weight(_MODE[case["dtype"]], k, n, seed * 1000 + 100 + i)
        if case["scaled"] and s is None:
            # one global scale per weight, given per column
            s = torch.full((n,), 0.5 + torch.rand(1, generator=gen, device="cuda").item(), device="cuda")
        weights.append(w)
        scales.append(s)
    w_scale = torch.cat(scales).cpu().numpy() if case["scaled"] else None
    st = {"op": op, "weights": weights, "n": sum(segs[0]), "scales": scales}
    if op == "dequant":
        st["node"] = DequantWeightBf16(st["n"], widths=segs[0], w_scale=w_scale)
    elif op == "lmhead":
        st["node"] = LmHeadArgmax(w_scale=w_scale)
        st["x"] = W.make_x(rows, k, seed * 1000 + 1)
    elif op == "gemm":
        st["node"] = SkinnyGemm([len(o) for o in segs], [v for o in segs for v in o], w_scale=w_scale)
        st["x"] = W.make_x(rows, k, seed * 1000 + 1)
    else:
        def mk(*shape):
            return torch.randn(*shape, generator=gen, device="cuda").bfloat16()
        st["node"] = SharedExpertDown(w_scale=w_scale)
        st["g"], st["u"], st["gx"] = mk(rows, k), mk(rows, k), mk(rows, _GATE)
        st["gw"] = (torch.randn(_GATE, 1, generator=gen, device="cuda") * 0.02).bfloat16()
        st["routed"] = (torch.randn(rows, st["n"], generator=gen, device="cuda") * 0.5).bfloat16()
    return st


def run(st):
    op, node = st["op"], st["node"]
    if op == "gemm":
        return node(st["x"], *st["weights"])
    if op == "lmhead":
        return node(st["x"], st["weights"][0], st["n"])
    if op == "shared":
        return node(st["g"], st["u"], st["weights"][0], st["gx"], st["gw"], st["routed"])
    if op == "argmax":
        return node(st["x"])
    return node(st["weights"][0])


def _weight_f64(dtype, w, n, scale):
    """The values of a stored weight, in 64 bits."""
    if dtype != "nvfp4":
        v = w.double()
    else:
        e2m1 = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device=w.device)
        e2m1 = torch.cat([e2m1, -e2m1])
        packed, blocks = w[:, :n // 2], w[:, n // 2:]
        v = torch.stack([e2m1[(packed & 15).long()], e2m1[(packed >> 4).long()]], dim=-1).reshape(w.shape[0], n)
        v = v * blocks.contiguous().view(torch.float8_e4m3fn).double().repeat_interleave(16, dim=1)
    return v if scale is None else v * scale.double()


def exact(case, seed):
    st = prepare(case, seed)
    op, dtype = case["op"], case["dtype"]
    if op == "argmax":
        val, idx = st["x"].double().max(dim=-1)
        return idx, val
    segs = _segments(case)

    def bf(t):  # a rounding that the op itself is defined with
        return t.bfloat16().double()

    if op == "dequant":
        return list(torch.split(_weight_f64(dtype, st["weights"][0], st["n"], st["scales"][0]), segs[0], dim=1))
    if op == "shared":
        g, u = st["g"].double(), st["u"].double()
        x = bf(bf(g * bf(torch.sigmoid(g))) * u)
        gate = bf(torch.sigmoid(bf(st["gx"].double() @ st["gw"].double())))
        y = x @ _weight_f64(dtype, st["weights"][0], st["n"], st["scales"][0])
        return st["routed"].double() + bf(y) * gate
    x = st["x"].double()
    if op == "lmhead":
        best = None
        w, n = st["weights"][0], st["n"]
        for c0 in range(0, n, 16384):  # column blocks: the whole weight in 64 bits would be large
            c1 = min(n, c0 + 16384)
            block = torch.cat([w[:, c0 // 2:c1 // 2], w[:, n // 2 + c0 // 16:n // 2 + c1 // 16]], dim=1)
            top = (x @ _weight_f64(dtype, block, c1 - c0, None)).max(dim=-1).values
            best = top if best is None else torch.maximum(best, top)
        return None, best, None  # the index, and the key made of it, may differ where two logits round alike
    outs = []
    for w, s, widths in zip(st["weights"], st["scales"], segs):
        outs += torch.split(x @ _weight_f64(dtype, w, sum(widths), s), widths, dim=1)
    return outs


def work(case):
    op, rows, k = case["op"], case["rows"], case["k"]
    segs = _segments(case)
    n = sum(sum(o) for o in segs)
    if op == "argmax":
        return {"bytes": rows * n * (4 if case["dtype"] == "f32" else 2) + 12 * rows, "flops": 0}
    b = _weight_bytes(case["dtype"], k, n) + (4 * n if case["scaled"] else 0)
    if op == "dequant":
        return {"bytes": b + 2 * k * n, "flops": 0}
    if op == "lmhead":
        b += 2 * rows * k + 20 * rows
    elif op == "gemm":
        b += 2 * rows * (k + n)
    else:
        b += 2 * rows * (2 * k + _GATE + 2 * n) + 2 * _GATE
    return {"bytes": b, "flops": 2 * rows * k * n + (2 * rows * _GATE if op == "shared" else 0)}


def tolerance(case):
    if case["op"] in ("argmax", "dequant"):
        return "exact"
    if case["op"] == "lmhead":
        return {"rel": 1e-2}  # the winning logit is one BF16 value; indices are whole numbers
    # One BF16 rounding (2^-9) of FP32 sums.  Where the call may round the scaled weights to BF16 first (many rows),
    # that moves a result by about as much again.
    return {"rel": 8e-3, "max": 6e-2} if case["rows"] > 8 else {"rel": 4e-3, "max": 3e-2}
