"""The many-row kernel of SkinnyGemm (csrc/dense_tc.cu) at the edges of its tiles: ragged rows, K that ends inside a
block of 64, column tiles cut short, several weights and outputs, every launch shape, both ways of loading NVFP4 rows."""
import subprocess
import sys

import numpy as np
import pytest
import torch

from conftest import ROOT, bits, to_dev
from oracle import cpu as C
from oracle import oracle as O
from qwen38_flash_ops_b200 import DequantWeightBf16, QfgError, SkinnyGemm
from qwen38_flash_ops_b200 import packing as P

import _util as U

pytestmark = pytest.mark.gpu

# rows, K, widths per weight: NVFP4 in 128-column groups, odd counts of them being the rows that start off 16 bytes
CASES = [
    (17, 72, [[128]]),
    (33, 328, [[256, 128], [128]]),
    (100, 1096, [[640], [128, 256]]),
    (300, 512, [[384]]),
]
# rows per tile, CTAs that split K, pair of CTAs, blocks of 64 k per stage
PLANS = ["", "16,1,0", "48,1,0,1", "48,1,0,2", "256,1,0", "64,2,0,1", "48,3,0,2", "32,8,0", "64,1,1,1", "64,1,1,2", "112,1,1", "256,1,1"]


def _takes_the_kernel(op, *args, **kw):
    """Whether a call goes to the many-row kernel: only there is a launch shape that does not exist an error."""
    op.set_option("dense_plan", "8,1")
    try:
        op(*args, **kw)
    except QfgError as e:
        assert "bad launch shape" in str(e)
        return True
    finally:
        op.set_option("dense_plan", "0")
    return False


def _check(mode, M, K, seg_widths, plan, seed, x_offset=0, out_offset=0, scale_columns=None, route=True):
    rng = np.random.default_rng(seed)
    seg_outs, widths, ns = [len(w) for w in seg_widths], [w for ws in seg_widths for w in ws], [sum(w) for w in seg_widths]
    x = P.synth_x(rng, M, K)
    stored, scales = zip(*[U.make_weight(rng, mode, K, n, True) for n in ns])
    w_scale = np.concatenate(scales) if mode != 0 else None
    if scale_columns is not None and mode != 0:  # a w_scale that ends early: the weights it does not cover have none
        w_scale = w_scale[:scale_columns]
        ends = np.cumsum(ns)
        scales = [s if end <= scale_columns else None for s, end in zip(scales, ends)]
    op = SkinnyGemm(seg_outs, widths, w_scale=w_scale)
    xd = to_dev(x, "bf16")
    if x_offset:
        buf = torch.empty(M * K + x_offset, dtype=torch.bfloat16, device="cuda")
        buf[x_offset:] = xd.reshape(-1)
        xd = buf[x_offset:].view(M, K)
    wd = [U.dev_weight(a, mode) for a in stored]
    outs = None
    if out_offset:  # outputs inside larger buffers, the elements around them watched
        buffers = [torch.full((M * w + 16,), 77.0, device="cuda", dtype=torch.bfloat16) for w in widths]
        outs = [b[out_offset:out_offset + M * w].view(M, w) for b, w in zip(buffers, widths)]
    assert _takes_the_kernel(op, xd, *wd, out=outs) == route
    if plan:
        op.set_option("dense_plan", plan)
    outs = op(xd, *wd, out=outs)
    torch.cuda.synchronize()
    if out_offset:
        for b, w in zip(buffers, widths):
            assert (b[:out_offset] == 77).all() and (b[out_offset + M * w:] == 77).all()
    o = 0
    for i, n in enumerate(ns):
        got = np.concatenate([bits(outs[o + j]).reshape(M, -1) for j in range(seg_outs[i])], axis=1)
        o += seg_outs[i]
        # the weights are rounded to BF16 with w_scale folded in, products and sums are not
        w_bf16 = O.dequant_weight_bf16(mode, stored[i], n, 0, scales[i] if mode != 0 else None)
        _, sums, mags = C.skinny_gemm(0, x, w_bf16, n, None)
        ok = O.gemm_within_tolerance(got, sums, mags, K)
        assert ok.all(), f"weight {i}: {np.count_nonzero(~ok)} of {ok.size} outputs outside tolerance"


# tiles of up to 128 rows hand the weights over in tensor memory: one and several stages of a group, a K
# range shorter than the groups, several tiles per CTA, ranks that add up, pairs
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("plan", ["16,1,0", "48,5,0", "80,1,0", "112,2,0", "128,1,0", "128,8,0", "64,1,1", "96,1,1", "128,1,1"])
def test_weights_through_tensor_memory(cuda, mode, plan):
    for i, (M, K, segs) in enumerate([(17, 72, [[256]]), (100, 2504, [[640 + 128], [128, 256 + 128]]), (300, 512, [[512]]), (129, 1096, [[256 * 45]])]):
        _check(mode, M, K, segs, plan, 900 + 10 * mode + i)
    if plan == "16,1,0":  # 646 tiles: five rounds of both accumulator sets
        _check(mode, 300, 1032, [[2304], [2048]], plan, 990 + mode)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", PLANS)
def test_tile_edges(cuda, mode, plan):
    for i, (M, K, seg_widths) in enumerate(CASES):
        _check(mode, M, K, seg_widths, plan, 1000 * mode + i)


@pytest.mark.parametrize("mode,K,widths,x_offset,route", [
    (0, 64, [[72]], 0, True), (1, 64, [[144]], 0, True),          # the last 16-byte pieces of a row are the tile's last
    (2, 64, [[128]], 0, True), (2, 64, [[256]], 0, True),          # NVFP4 rows off 16 bytes and on them
    (1, 64, [[136]], 0, False), (2, 64, [[192]], 0, False),        # rows the copies cannot address
    (0, 68, [[128]], 0, False), (0, 64, [[128]], 2, False), (2, 128, [[256]], 4, False),  # K or x off 16 bytes
])
def test_layouts_on_either_side_of_the_route(cuda, mode, K, widths, x_offset, route):
    _check(mode, 40, K, widths, "", 77, x_offset, route=route)


# Launch shapes that give a CTA, or a pair, four tiles and more: both accumulator sets come round again, and stages, rings and
# the dequantising groups go on across tiles, with an odd number of k steps (17 blocks of 64, 9 stages' worth of two).
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("M,plan", [(300, "16,1,0,1"), (300, "16,1,0,2"), (1100, "64,1,1,1"), (1100, "64,1,1,2")])
@pytest.mark.parametrize("K,last", [(1032, 1920), (1032, 2048), (64, 1920)])
def test_many_tiles_a_cta(cuda, mode, M, plan, K, last):
    bm, _, pair, _ = map(int, plan.split(","))
    seg_widths = [[1664, 640], [last]]  # NVFP4: at 1920 columns the rows are off 16 bytes
    tiles = sum(-(-sum(w) // (256 if pair else 128)) for w in seg_widths) * -(-M // bm)
    assert tiles > 4 * (74 if pair else 148)
    _check(mode, M, K, seg_widths, plan, 5000 + mode)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["", "64,1,0", "48,3,0", "64,1,1"])
def test_outputs_off_16_bytes_and_short_scales(cuda, mode, plan):
    """Both epilogues' two-byte stores, and weights beyond the end of w_scale."""
    for out_offset in (1, 4):
        _check(mode, 100, 328, [[248, 136], [128 if mode == 2 else 144]], plan, 40 + out_offset, out_offset=out_offset, scale_columns=384)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["256,1,0,1", "128,1,0,1", "256,1,1,1", "64,3,0,2"])
def test_repeated_calls_agree(cuda, mode, plan):
    """A stage handed on before it was read or written shows as a run that differs (5120 rows of K: every ring of the
    kernel goes round many times, and with 256 rows a tile the MMAs are what the other roles wait for)."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    M, K, N = 300, 5120, 2048
    x = torch.randn(M, K, generator=gen, device="cuda").bfloat16()
    if mode == 0:
        w = (torch.randn(K, N, generator=gen, device="cuda") * 0.02).bfloat16()
    elif mode == 1:
        w = torch.randn(K, N, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    else:
        w = torch.randint(0, 256, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)
        w[:, N // 2:] = w[:, N // 2:] % 0x7F  # block scales: finite, not negative
    op = SkinnyGemm([1], [N])
    op.set_option("dense_plan", plan)
    first = op(x, w)[0].clone()
    assert torch.isfinite(first).all()
    # a fault that repeats itself: against the product of the same BF16 weights by another kernel, FP32 sums in another order
    wide = DequantWeightBf16(N)(w)[0] if mode != 0 else w
    want = x.float() @ wide.float()
    bound = 2.0 ** -8 * want.abs() + 2 * K * 2.0 ** -24 * (x.float().abs() @ wide.float().abs())  # one BF16 rounding, the sums' on both sides
    assert torch.all((first.float() - want).abs() <= bound)
    for _ in range(40):
        assert torch.equal(op(x, w)[0], first)


def test_graph_capture_and_bad_launch_shapes(cuda):
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(64, 512, generator=gen, device="cuda").bfloat16()
    w = torch.randn(512, 256, generator=gen, device="cuda").bfloat16()
    op = SkinnyGemm([1], [256])
    eager = op(x, w)[0].clone()
    out = [torch.empty_like(eager)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op(x, w, out=out)
    out[0].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0], eager)
    for plan in ("8,1,0", "272,1,0", "40,1,1", "64,2,1", "64,9,0", "64,1,0,3"):
        op.set_option("dense_plan", plan)
        with pytest.raises(QfgError):
            op(x, w)


@pytest.mark.parametrize("mode,K", [(0, 8), (1, 8), (2, 8), (0, 24), (2, 40)])
def test_k_shorter_than_a_block(cuda, mode, K):
    _check(mode, 33, K, [[128], [256]], "", 5)


def test_first_call_of_a_process_may_be_captured(cuda):
    """Nothing is left for the first call to set up: each kernel's first launch of the process is a captured one."""
    code = """
import torch
from qwen38_flash_ops_b200 import SharedExpertDown, SkinnyGemm
mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()
w = mk(512, 256)
nibbles = torch.randint(0, 256, (512, 144), device="cuda", dtype=torch.uint8)
nibbles[:, 128:] %= 0x7F
gx, gw, routed = mk(64, 64), mk(64, 1), mk(64, 256)
calls = []
for weight in (w, w.to(torch.float8_e4m3fn), nibbles):
    for rows in (64, 700):
        x, op, out = mk(rows, 512), SkinnyGemm([1], [256]), torch.zeros(rows, 256, device="cuda", dtype=torch.bfloat16)
        calls.append(lambda op=op, x=x, weight=weight, out=out: op(x, weight, out=[out])[0])
    x, op = mk(64, 512), SharedExpertDown()
    calls.append(lambda op=op, x=x, weight=weight: op(x, x, weight, gx, gw, routed))
torch.cuda.synchronize()
for call in calls:
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = call()
    graph.replay()
    got = y.clone()
    assert torch.equal(got, call()) and torch.isfinite(got).all() and got.abs().max() > 0
print("ok")
"""
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["48,1,0", "48,1,0,1", "64,4,0", "64,4,0,1", "128,1,1", "96,1,1,1", "256,1,0", "256,1,1"])
def test_waits_that_run_out_give_nan(cuda, mode, plan):
    """x never comes: every output is NaN, none keeps what its memory held, and the next call is whole.  Several tiles a CTA."""
    gen = torch.Generator(device="cuda").manual_seed(mode)
    M, K, N = 300, 1096, 128 * 46 if "4,0" in plan else 128 * 150
    x = torch.randn(M, K, generator=gen, device="cuda").bfloat16()
    w = torch.randn(K, N, generator=gen, device="cuda").bfloat16()
    if mode == 1:
        w = w.to(torch.float8_e4m3fn)
    elif mode == 2:
        w = torch.randint(0, 0x70, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)
    op = SkinnyGemm([1], [N])
    op.set_option("dense_plan", plan)
    first = op(x, w)[0]
    for _ in range(2):
        out = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
        op.set_option("give_up", 1)
        op(x, w, out=[out])
        assert torch.isnan(out).all()
        op.set_option("give_up", 0)
        assert torch.equal(op(x, w)[0], first)
