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
from qwen38_flash_ops_b200 import QfgError, SkinnyGemm
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


def _check(mode, M, K, seg_widths, plan, seed, x_offset=0):
    rng = np.random.default_rng(seed)
    seg_outs, widths, ns = [len(w) for w in seg_widths], [w for ws in seg_widths for w in ws], [sum(w) for w in seg_widths]
    x = P.synth_x(rng, M, K)
    stored, scales = zip(*[U.make_weight(rng, mode, K, n, True) for n in ns])
    op = SkinnyGemm(seg_outs, widths, w_scale=np.concatenate(scales) if mode != 0 else None)
    if plan:
        op.set_option("dense_plan", plan)
    xd = to_dev(x, "bf16")
    if x_offset:
        buf = torch.empty(M * K + x_offset, dtype=torch.bfloat16, device="cuda")
        buf[x_offset:] = xd.reshape(-1)
        xd = buf[x_offset:].view(M, K)
    outs = op(xd, *[U.dev_weight(a, mode) for a in stored])
    torch.cuda.synchronize()
    o = 0
    for i, n in enumerate(ns):
        got = np.concatenate([bits(outs[o + j]).reshape(M, -1) for j in range(seg_outs[i])], axis=1)
        o += seg_outs[i]
        # the weights are rounded to BF16 with w_scale folded in, products and sums are not
        w_bf16 = O.dequant_weight_bf16(mode, stored[i], n, 0, scales[i] if mode != 0 else None)
        _, sums, mags = C.skinny_gemm(0, x, w_bf16, n, None)
        ok = O.gemm_within_tolerance(got, sums, mags, K)
        assert ok.all(), f"weight {i}: {np.count_nonzero(~ok)} of {ok.size} outputs outside tolerance"


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", PLANS)
def test_tile_edges(cuda, mode, plan):
    for i, (M, K, seg_widths) in enumerate(CASES):
        _check(mode, M, K, seg_widths, plan, 1000 * mode + i)


@pytest.mark.parametrize("mode,K,widths,x_offset", [
    (0, 64, [[72]], 0), (1, 64, [[144]], 0),          # the last 16-byte pieces of a row are the tile's last
    (1, 64, [[136]], 0), (2, 64, [[192]], 0),          # rows the copies cannot address
    (0, 68, [[128]], 0), (0, 64, [[128]], 2), (2, 128, [[256]], 4),  # K or x off 16 bytes
])
def test_layouts_on_either_side_of_the_route(cuda, mode, K, widths, x_offset):
    _check(mode, 40, K, widths, "", 77, x_offset)


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
