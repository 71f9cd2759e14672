"""The kernel that streams the weights by tensor copies (csrc/skinny_stream.cu) at the edges of its launch shapes, against
the CPU oracle with the tolerances of test_gpu_skinny_gemm.py and test_gpu_shared_expert_down.py."""
import numpy as np
import pytest
import torch

from conftest import bits, to_dev
from oracle import oracle as O
from qwen38_flash_ops_b200 import ArgmaxRows, LmHeadArgmax, QfgError, SharedExpertDown, SkinnyGemm
from qwen38_flash_ops_b200 import packing as P

import _util as U
from test_gpu_shared_expert_down import _check, _inputs

pytestmark = pytest.mark.gpu


def _gemm(rng, mode, M, K, seg_widths, plan, x=None, force_slow=False):
    """One call in the launch shape `plan`; the row-independent check of every output against the oracle."""
    ns = [sum(w) for w in seg_widths]
    x = P.synth_x(rng, M, K) if x is None else x
    made = [U.make_weight(rng, mode, K, n, True) for n in ns]
    scales = [s for _, s in made]
    w_scale = np.concatenate(scales) if mode != 0 else None
    op = SkinnyGemm([len(w) for w in seg_widths], [v for w in seg_widths for v in w], w_scale=w_scale)
    weights = [U.dev_weight(a, mode) for a, _ in made]
    xd = to_dev(x, "bf16")
    op.set_option("stream_plan", plan)
    if force_slow:
        op.set_option("force_slow", 1)
    outs = op(xd, *weights)
    assert f"stream={plan.replace(',', '/')}/0" in op.describe(K, *weights)
    torch.cuda.synchronize()
    o = 0
    for (arr, s), widths, n in zip(made, seg_widths, ns):
        got = np.concatenate([bits(outs[o + j]).reshape(M, -1) for j in range(len(widths))], axis=1)
        U.check_against_oracle(mode, x, arr, n, s if mode != 0 else None, got, K, f"mode{mode} M{M} K{K} {plan}")
        o += len(widths)
    return op, xd, weights, outs


# width,wk,teams,cluster: one and many tiles, a last tile of one granule, warps without columns, more teams or ranks than
# stages, a ring that wraps many times, stages of two boxes
@pytest.mark.parametrize("mode,plan", [
    (0, "3,4,1,1"), (0, "8,4,2,1"), (0, "9,2,2,3"), (0, "24,1,2,2"), (0, "8,8,2,1"), (0, "31,4,1,8"),
    (1, "3,4,1,1"), (1, "8,8,1,1"), (1, "9,2,2,3"), (1, "24,1,2,2"), (1, "8,1,4,5"), (1, "17,4,1,8"),
    (2, "1,4,1,1"), (2, "1,8,2,1"), (2, "2,4,2,3"), (2, "3,2,2,2"), (2, "9,1,2,1"), (2, "1,1,4,8"), (2, "1,9,1,1")])
def test_launch_shapes(cuda, mode, plan):
    rng = np.random.default_rng(1000 * mode + sum(map(ord, plan)))
    # NVFP4 rows of a multiple of 16 bytes, and of an odd multiple of 8
    cases = [(1, 2312, [[1280, 384]]), (5, 1000, [[512], [256, 256]]), (8, 72, [[256]])]
    if mode == 2:
        cases += [(3, 2312, [[640, 384], [896]]), (8, 136, [[384]]), (2, 8, [[128]])]
    else:
        cases += [(3, 2312, [[16 * 37]]), (8, 8, [[16], [48]])]
    for M, K, segs in cases:
        _gemm(rng, mode, M, K, segs, plan)


@pytest.mark.parametrize("mode", [1, 2])
def test_values_outside_the_fp16_range(cuda, mode):
    """Rows whose magnitudes spread too far for FP16, and the forced BF16 path."""
    rng = np.random.default_rng(mode)
    x = P.synth_x(rng, 4, 520)
    x[1, 3] = 0x7180   # 2^100: times 448, the largest E4M3 value, and a few thousand N(0, 1) terms still an FP32 number
    x[2, 7] = 0x0080   # the smallest normal number
    _gemm(rng, mode, 4, 520, [[256]], "1,4,2,1" if mode == 2 else "8,4,2,1", x=x)
    _gemm(rng, mode, 4, 520, [[384]], "1,4,1,2" if mode == 2 else "8,4,1,2", force_slow=True)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("M", [1, 3, 8])
def test_rows_are_independent_and_calls_agree(cuda, mode, M):
    """The same bits in any company, and in every one of many calls (a ring slot read after it was written again would not
    give them)."""
    rng = np.random.default_rng(7 * mode + M)
    plan = "2,2,2,2" if mode == 2 else "16,2,2,2"
    op, x, weights, outs = _gemm(rng, mode, M, 5120, [[512, 256]], plan)
    for m in range(M):
        for one, all_rows in zip(op(x[m:m + 1].contiguous(), *weights), outs):
            assert torch.equal(one[0], all_rows[m])
    for _ in range(50):
        for again, first in zip(op(x, *weights), outs):
            assert torch.equal(again, first)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["1,4,2,1", "1,4,1,3", "2,1,4,1"])
def test_shared_expert(cuda, mode, plan):
    width, rest = plan.split(",", 1)
    plan = plan if mode == 2 else f"{8 * int(width) - 1},{rest}"
    rng = np.random.default_rng(mode + sum(map(ord, plan)))
    for M, K, N, gk in [(1, 640, 256, 2560), (5, 296, 384, 8), (8, 1032, 128, 1000)]:
        arr, s = U.make_weight(rng, mode, K, N, mode != 0)
        g, u, gx, gw, routed = _inputs(rng, M, K, N, gk)
        op = SharedExpertDown(w_scale=s if mode != 0 else None)
        op.set_option("stream_plan", plan)
        args = [to_dev(g, "bf16"), to_dev(u, "bf16"), U.dev_weight(arr, mode), to_dev(gx, "bf16"), to_dev(gw, "bf16"), to_dev(routed, "bf16")]
        out = op(*args)
        y, _, _, shared = O.shared_expert_down(g, u, mode, arr, N, gx, gw, routed, s if mode != 0 else None)
        _check(bits(out), y, shared, O.bf16_to_f32(routed), f"mode {mode} M {M} {plan}")
        for m in range(M):
            row = [a[m:m + 1].contiguous() if a.shape[0] == M and i not in (2, 4) else a for i, a in enumerate(args)]
            assert torch.equal(op(*row)[0], out[m])


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("plan", ["1,4,2,1", "1,4,1,2"])
def test_shared_expert_outside_the_fp16_range(cuda, mode, plan):
    """swish_mul that spreads too far for FP16, in the last row and the last slice of K alone, and the forced BF16 path, whose
    sums are those of the FP16 one."""
    plan = plan if mode == 2 else f"8{plan[1:]}"
    rng = np.random.default_rng(mode)
    M, K, N, gk = 5, 1032, 128, 64
    arr, s = U.make_weight(rng, mode, K, N, True)
    g, u, gx, gw, routed = _inputs(rng, M, K, N, gk)
    op = SharedExpertDown(w_scale=s)
    op.set_option("stream_plan", plan)
    run = lambda u: bits(op(*[to_dev(a, "bf16") if a is not arr else U.dev_weight(arr, mode) for a in (g, u, arr, gx, gw, routed)]))
    plain = run(u)
    for value in (0x7180, 0x0D00):  # 2^100, 2^-101
        wide = u.copy()
        wide[M - 1, K - 1] = value
        y, _, _, shared = O.shared_expert_down(g, wide, mode, arr, N, gx, gw, routed, s)
        got = run(wide)
        _check(got, y, shared, O.bf16_to_f32(routed), f"mode {mode} {plan} {value:x}")
        assert np.array_equal(got[:M - 1], plain[:M - 1])
    op.set_option("force_slow", 1)
    assert np.array_equal(run(u), plain)


@pytest.mark.parametrize("groups", [33, 34])  # rows of 8 modulo 16 bytes, and of 0
@pytest.mark.parametrize("tail", [1, 3])
def test_head_tail(cuda, groups, tail):
    """Left-over column groups in slices of K: the argmax of the kernel's own logits, which are the plain product's."""
    rng = np.random.default_rng(groups + tail)
    N, K, M = 128 * groups, 1032, 5
    w = U.dev_weight(U.make_weight(rng, 2, K, N, False)[0], 2)
    x = to_dev(P.synth_x(rng, M, K), "bf16")
    head, plain = LmHeadArgmax(), SkinnyGemm([1], [N])
    head.set_option("stream_plan", f"2,1,2,1,{tail}")
    plain.set_option("stream_plan", "3,1,2,1")
    for _ in range(3):
        idx, val, _, logits = head(x, w, N, logits=True)
        i, v = ArgmaxRows()(logits)
        assert torch.equal(idx, i) and torch.equal(val, v)
        ref = plain(x, w)[0]
        main = N - 128 * tail
        assert torch.equal(logits[:, :main], ref[:, :main])
        # the tail's sums are FP32 in another order: one BF16 ULP, and K * 2^-24 of the magnitudes where they cancel
        assert torch.allclose(logits.float(), ref.float(), rtol=2.0 ** -7, atol=K * 2.0 ** -24 * float(x.float().abs().sum(1).max()) * 0.2)


def test_shapes_that_do_not_exist_are_refused(cuda):
    w = U.dev_weight(U.make_weight(np.random.default_rng(0), 2, 64, 256, False)[0], 2)
    x = to_dev(np.zeros((1, 64), np.uint16), "bf16")
    for plan in ("1,19,1,1", "19,1,1,1", "0,1,1,1", "1,1,1,9", "1,1,0,1", "1,4", "1,4,1,1,1"):
        op = SkinnyGemm([1], [256])
        op.set_option("stream_plan", plan)
        with pytest.raises(QfgError):
            op(x, w)


@pytest.mark.parametrize("mode,N,plan", [(0, 1040, ""), (1, 1040, "9,2,2,2"), (2, 4224, "2,1,2,1,3"), (2, 4352, "2,1,2,1,1"), (2, 384, "1,4,2,1")])
@pytest.mark.parametrize("pdl_wait", [0, 1])
def test_a_head_that_gave_up_says_so(cuda, mode, N, plan, pdl_wait):
    """As if the wait for x had run out: every logit is NaN although the weights are there, and the next call's are the ones
    before."""
    rng = np.random.default_rng(N + mode)
    K, M = 1032, 5
    x, w = to_dev(P.synth_x(rng, M, K), "bf16"), U.dev_weight(U.make_weight(rng, mode, K, N, False)[0], mode)
    head = LmHeadArgmax()
    head.set_option("stream_plan", plan)
    head.set_option("pdl_wait", pdl_wait)
    first = head(x, w, N, logits=True)
    for _ in range(3):
        head.set_option("give_up", 1)
        _, val, _, logits = head(x, w, N, logits=True)
        assert torch.isnan(val).all() and torch.isnan(logits).all()
        head.set_option("give_up", 0)
        for a, b in zip(head(x, w, N, logits=True), first):
            assert torch.equal(a, b)


# what stands among ordinary values of x: [2^-27, 2^6) is scaled in one look, the rest row by row or not at all
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("kind", ["plain", "cluster", "shared", "head"])
@pytest.mark.parametrize("least,most", [(2.0 ** -22, 1.9921875 * 2.0 ** 10), (1.9921875 * 2.0 ** -23, 1.0), (2.0 ** -10, 2.0 ** 11), (2.0 ** -30, 2.0 ** -4),
                                        (2.0 ** 10, 2.0 ** 36), (2.0 ** -40, 2.0 ** 20), (2.0 ** -130, 1.0), (0.0, float("inf")), (0.0, float("nan"))])
def test_scalings_of_x_agree(cuda, mode, kind, least, most):
    """Scaled or not, the products are exact and so are the powers of two: the bits of the BF16 path, which scales nothing."""
    gen = torch.Generator(device="cuda").manual_seed(mode)
    M, K, N = 3, 1160, 512
    x = (torch.rand(M, K, generator=gen, device="cuda") + 0.5) * torch.where(torch.rand(M, K, generator=gen, device="cuda") < 0.5, 1.0, -1.0)
    if least >= 2.0 ** 10:
        x *= 2.0 ** 12
    if 0 < least < 2.0 ** -22 and most < 1:
        x *= 2.0 ** -5
    x[0, 5], x[0, 1159], x[1, 700], x[2, :64] = least, -most, -least, 0.0
    x = x.bfloat16()
    w = torch.randn(K, N, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    if mode == 2:
        w = torch.randint(0, 256, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)
        w[:, N // 2:] = w[:, N // 2:] % 0x60  # block scales: finite, not negative
    outs = []
    for slow in (0, 1):
        if kind == "head":
            op = LmHeadArgmax()
            op.set_option("force_slow", slow)
            outs.append(op(x, w, N, logits=True)[3])
        elif kind == "shared":
            op = SharedExpertDown()
            op.set_option("force_slow", slow)
            g, one = torch.full_like(x, 16.0), torch.ones(64, 1, dtype=torch.bfloat16, device="cuda")  # bf16(sigmoid(16)) is 1
            outs.append(op(g, (x.float() / 16).bfloat16(), w, torch.ones(M, 64, dtype=torch.bfloat16, device="cuda"), one, torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")))
        else:
            op = SkinnyGemm([1], [N])
            op.set_option("force_slow", slow)
            op.set_option("stream_plan", ("1,4,1,3" if mode == 2 else "8,4,1,3") if kind == "cluster" else "")
            outs.append(op(x, w)[0])
    a, b = outs
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))
    assert torch.isfinite(a).any()


def _rows_of_every_kind(M, K):
    """Rows that the usual scaling of x, exact in [2^-27, 2^6), fits and does not: below it here and there, above it among zeros, below it
    throughout, nothing but zeros, its edges, and both ends of what FP16 holds."""
    gen = torch.Generator(device="cuda").manual_seed(K)
    rand = lambda: torch.rand(K, generator=gen, device="cuda")
    x = (torch.rand(M, K, generator=gen, device="cuda") + 0.5) * torch.where(torch.rand(M, K, generator=gen, device="cuda") < 0.5, 1.0, -1.0)
    x[1 % M, rand() < 0.02] = 1.375 * 2.0 ** -28
    x[1 % M, rand() < 0.1] = 0.0
    if M > 2:
        x[2, rand() < 0.01] = 100.0
        x[2, rand() < 0.5] = 0.0
        x[3] *= 2.0 ** -33
        x[4] = 0.0
    if M > 5:
        x[5, 3::41] = 2.0 ** -27
        x[5, 4::41] = -1.9921875 * 2.0 ** -28  # rounds to the same FP16 number
        x[5, 5::41] = 1.9921875 * 2.0 ** 5
        x[6, K - 1], x[6, 0] = 200.0, -1.5 * 2.0 ** -21
        x[7, K - 5] = 2.0 ** 6
    return x.bfloat16()


# a lane with several rows, with more than 32 pieces of one, with one batch of a row and padding past it, and with one batch
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("M,K,plan", [(8, 10248, "{},1,1,1"), (8, 5128, "{},4,1,1"), (5, 1528, "{},5,1,1"), (8, 2568, "{},8,1,2"), (1, 17408, ""), (8, 5120, "")])
def test_rows_scaled_after_the_first_look(cuda, mode, M, K, plan):
    """The bits of the BF16 path, which scales nothing, whatever the slice was staged from."""
    N = 512
    gen = torch.Generator(device="cuda").manual_seed(mode)
    x = _rows_of_every_kind(M, K)
    w = torch.randn(K, N, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    if mode == 2:
        w = torch.randint(0, 256, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)
        w[:, N // 2:] = w[:, N // 2:] % 0x60
    outs = []
    for slow in (0, 1):
        op = SkinnyGemm([1], [N])
        op.set_option("force_slow", slow)
        op.set_option("stream_plan", plan.format("1" if mode == 2 else "8"))
        outs.append(op(x, w)[0])
    assert torch.isfinite(outs[0]).all() and torch.equal(*outs)


def _quickest(*calls, rounds=9, reps=40):
    """The shortest of several timings of `reps` times each call's list, in turn, in microseconds."""
    best = [float("inf")] * len(calls)
    for _ in range(rounds):
        for i, c in enumerate(calls):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(reps):
                for f in c:
                    f()
            b.record()
            torch.cuda.synchronize()
            best[i] = min(best[i], a.elapsed_time(b) * 1e3 / reps / len(c))
    return best


def test_time_does_not_depend_on_the_activations(cuda):
    """x as a down projection gets it, silu(g) u with g and u of deviation 0.1, against N(0, 1): restaging whole slices took a third
    more for eight rows of FP8 5120 x 10240 (22.3 us, 16.8), and a fifth for four of the shared expert (7.5, 6.2); now 17.9, 16.6 and 6.2, 6.2."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    op, w = SkinnyGemm([1], [10240]), mk(5120, 10240).to(torch.float8_e4m3fn)
    normal = [mk(8, 5120).bfloat16() for _ in range(6)]
    silu = [(torch.nn.functional.silu(mk(8, 5120) * 0.1) * mk(8, 5120) * 0.1).bfloat16() for _ in range(6)]
    a, b = _quickest([lambda x=x: op(x, w) for x in normal], [lambda x=x: op(x, w) for x in silu])
    assert b < 1.2 * a, (a, b)
    K, N, M = 640, 2560, 4
    op, w = SharedExpertDown(), torch.randint(0, 0x60, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)
    rest = mk(M, N).bfloat16(), (mk(N, 1) * 0.02).bfloat16(), mk(M, N).bfloat16()
    pairs = [[((mk(M, K) * s).bfloat16(), (mk(M, K) * s).bfloat16()) for _ in range(6)] for s in (1.0, 0.1)]
    a, b = _quickest(*[[lambda g=g, u=u: op(g, u, w, *rest) for g, u in p] for p in pairs])
    assert b < 1.1 * a, (a, b)
