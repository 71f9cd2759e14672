"""The many-row kernel of SharedExpertDown (csrc/dense_tc.cu) at the edges of its tiles and clusters, and its sigmoid on
every BF16 value."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import bits, to_dev
from oracle import oracle as O
from qwen38_flash_ops_b200 import QfgError, SharedExpertDown, SkinnyGemm
from qwen38_flash_ops_b200 import _lib as L
from qwen38_flash_ops_b200 import packing as P

import _util as U

pytestmark = pytest.mark.gpu


def _run(mode, M, K, N, gk, plan, seed, gx_offset=0, g_offset=0, route=True):
    rng = np.random.default_rng(seed)
    bf = lambda a: P.f32_to_bf16_bits(a.astype(np.float32))
    arr, s = U.make_weight(rng, mode, K, N, mode != 0)
    g, u, gx = bf(rng.standard_normal((M, K)) * 0.8), bf(rng.standard_normal((M, K)) * 0.8), bf(rng.standard_normal((M, gk)) * 0.2)
    gw, routed = bf(rng.standard_normal((gk, 1)) * 0.2), bf(rng.standard_normal((M, N)) * 0.2)

    def dev(a, offset=0):
        t = to_dev(a, "bf16")
        if not offset:
            return t
        buf = torch.empty(t.numel() + offset, dtype=torch.bfloat16, device="cuda")
        buf[offset:] = t.reshape(-1)
        return buf[offset:].view(t.shape)

    op = SharedExpertDown(w_scale=s if mode != 0 else None)
    args = dev(g, g_offset), dev(u), U.dev_weight(arr, mode), dev(gx, gx_offset), dev(gw), dev(routed)
    # only in the many-row kernel is a launch shape that does not exist an error
    op.set_option("dense_plan", "8,1")
    if route:
        with pytest.raises(QfgError, match="bad launch shape"):
            op(*args)
    else:
        op(*args)
    op.set_option("dense_plan", plan or "0")
    out = op(*args)
    torch.cuda.synchronize()
    y, _, _, shared = O.shared_expert_down(g, u, mode, arr, N, gx, gw, routed, s if mode != 0 else None)
    got, gf, yf = bits(out), O.bf16_to_f32(bits(out)), O.bf16_to_f32(y)
    # FP32 sums in another order may cross a BF16 boundary: one ulp of the larger of the two terms
    tol = np.maximum(np.maximum(np.abs(O.bf16_to_f32(routed)), np.abs(shared)), np.abs(yf)) * 2.0 ** -7 + 1e-30
    assert np.all(np.abs(gf - yf) <= tol), f"{np.count_nonzero(np.abs(gf - yf) > tol)} outputs outside one ULP"
    assert np.mean(got == y) > 0.97


# rows per tile, CTAs per cluster (ranks whose warps have no rows of their own among them)
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["", "16,1", "32,4", "48,2", "96,4", "256,1", "256,4"])
def test_tile_and_cluster_edges(cuda, mode, plan):
    for i, (M, K, N, gk) in enumerate([(17, 256, 128, 256), (100, 648, 1152, 1024), (35, 1096, 640, 26)]):
        _run(mode, M, K, N, gk, plan, 100 * mode + i)


# clusters whose CTAs have unequal shares of the rows, or columns past the end
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["32,3,0,1", "48,5,0,1", "64,7,0,1", "80,8,0,1", "160,7,0,1", "256,6,0,1"])
def test_uneven_shares(cuda, mode, plan):
    """Whoever evaluates a row, sums and gates are added in one order: the bits of the launch without clusters."""
    gen = torch.Generator(device="cuda").manual_seed(mode)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    for M, K, N, gk in ((17, 256, 128, 256), (170, 648, 1152, 1000), (35, 1096, 640, 26)):
        w = [mk(K, N), mk(K, N).to(torch.float8_e4m3fn), torch.randint(0, 0x70, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)][mode]
        args = mk(M, K), mk(M, K), w, mk(M, gk) * 0.2, mk(gk, 1) * 0.2, mk(M, N)
        op = SharedExpertDown()
        op.set_option("dense_plan", "32,1")
        want = op(*args)
        op.set_option("dense_plan", plan)
        assert torch.equal(op(*args), want)


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_outputs_off_sixteen_bytes(cuda, mode):
    """routed, and the output that is made beside it, at an odd element: the same values, two bytes at a time."""
    gen = torch.Generator(device="cuda").manual_seed(mode)
    M, K, N = 70, 256, 384
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    w = [mk(K, N), mk(K, N).to(torch.float8_e4m3fn), torch.randint(0, 0x70, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)][mode]
    g, u, gx, gw, routed = mk(M, K), mk(M, K), mk(M, 64), mk(64, 1), mk(M, N)
    op = SharedExpertDown()
    want = op(g, u, w, gx, gw, routed)
    for shift_in, shift_out in ((1, 0), (0, 1), (3, 5)):
        src, dst = torch.zeros(M * N + 8, dtype=torch.bfloat16, device="cuda"), torch.zeros(M * N + 8, dtype=torch.bfloat16, device="cuda")
        src[shift_in:shift_in + M * N] = routed.reshape(-1)
        t = L.Tensor2D(w.data_ptr(), [L.QFG_BFLOAT16, L.QFG_FLOAT8E4M3FN, L.QFG_UINT8][mode], *w.shape)
        code = L.load().qfg_shared_expert_down_compute(op._h, g.data_ptr(), u.data_ptr(), M, K, ctypes.byref(t), gx.data_ptr(), 64, gw.data_ptr(),
                                                       src.data_ptr() + 2 * shift_in, N, dst.data_ptr() + 2 * shift_out, torch.cuda.current_stream().cuda_stream)
        assert code == 0
        assert torch.equal(dst[shift_out:shift_out + M * N].view(M, N), want)
        assert not dst[:shift_out].any() and not dst[shift_out + M * N:].any()


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_layouts_on_either_side_of_the_route(cuda, mode):
    _run(mode, 40, 256, 128, 64, "", 7, gx_offset=1)               # gate read element by element
    _run(mode, 40, 256, 128, 64, "", 7, g_offset=2, route=False)    # rows of g the kernel cannot read: streaming passes
    _run(mode, 40, 260, 192, 64, "", 7, route=False)                # K off 16 bytes, N an odd number of 64
    _run(mode, 40, 256, 256, 64, "", 7)                             # NVFP4 rows on 16 bytes (at 128 columns they are not)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["160,4", "256,4", "64,2", "32,1", "160,7,0,1", "80,8,0,1"])
def test_repeated_calls_agree(cuda, mode, plan):
    """A stage reused before every CTA of the cluster has read it shows as a run that differs."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    M, K, N = 300, 2560, 1152
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    if mode == 0:
        w = mk(K, N) * 0.02
    elif mode == 1:
        w = mk(K, N).to(torch.float8_e4m3fn)
    else:
        w = torch.randint(0, 256, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)
        w[:, N // 2:] = w[:, N // 2:] % 0x7F  # block scales: finite, not negative
    args = (mk(M, K), mk(M, K), w, mk(M, 512), mk(512, 1), mk(M, N))
    op = SharedExpertDown()
    op.set_option("dense_plan", plan)
    first = op(*args).clone()
    assert torch.isfinite(first).all()
    for _ in range(40):
        assert torch.equal(op(*args), first)


def _three_kernels():
    """The many-row kernel, the few-row kernel in passes, the general kernels in passes."""
    many, few, general = SharedExpertDown(), SharedExpertDown(), SharedExpertDown()
    for op in (few, general):
        op.set_option("dense_rows", 0)
    general.set_option("stream_plan", "0")
    return many, few, general


@pytest.mark.parametrize("seed", range(4))
def test_swish_times_u_is_the_streaming_kernels(cuda, seed):
    """Every g beside random u of every size: bf16(bf16(g * bf16(sigmoid(g))) * u), through an identity weight, in the many-row
    and the few-row kernel, which share swish.cuh, against the general kernels, whose sigmoid is expf and a division.  A row holds 64
    values, so g and u stay below 2^60 and sums are one term and zeros.  Products below the normal range may be rounded twice
    (once to FP32's subnormals), so they are compared to one unit in their last place."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16)
    g = torch.where(torch.isfinite(g) & (g.abs() < 2.0 ** 60), g, torch.zeros_like(g))[torch.randperm(65536, generator=gen, device="cuda")].view(1024, 64)
    u = torch.randint(0, 65536, (1024, 64), generator=gen, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    u = torch.where(torch.isfinite(u) & (u.abs() < 2.0 ** 60), u, torch.ones_like(u))
    w = torch.zeros(64, 128, device="cuda")
    w[torch.arange(64), torch.arange(64)] = 1
    gx, gw = torch.ones(1024, 8, device="cuda").bfloat16(), torch.full((8, 1), 10.0, device="cuda").bfloat16()
    routed = torch.zeros(1024, 128, device="cuda").bfloat16()
    many, few, b = (op(g, u, w.bfloat16(), gx, gw, routed) for op in _three_kernels())
    normal = b.float().abs() >= 2.0 ** -126
    for a in (many, few):
        assert torch.equal(a[normal], b[normal])
        assert ((a.double() - b.double()).abs() <= 2.0 ** -133).logical_or(normal).all()
        assert normal[:, :64].sum() > 30000 and torch.count_nonzero(a[:, 64:]) == 0


def test_swish_of_every_bf16_value_is_the_streaming_kernels(cuda):
    """One value per row, u = 1, an identity weight and a gate of one: the output is bf16(g * bf16(sigmoid(g)))."""
    g = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.bfloat16).view(1024, 64)
    w = torch.zeros(64, 128, device="cuda")
    w[torch.arange(64), torch.arange(64)] = 1
    gx, gw = torch.ones(1024, 8, device="cuda").bfloat16(), torch.full((8, 1), 10.0, device="cuda").bfloat16()
    u, routed = torch.ones_like(g), torch.zeros(1024, 128, device="cuda").bfloat16()
    kernels = _three_kernels()
    for j in range(64):
        gj = torch.zeros_like(g)
        gj[:, j] = g[:, j]
        many, few, b = (op(gj, u, w.bfloat16(), gx, gw, routed)[:, j] for op in kernels)
        for a in (many, few):
            assert torch.equal(torch.isnan(a), torch.isnan(b))
            assert torch.equal(torch.nan_to_num(a, nan=7.0), torch.nan_to_num(b, nan=7.0))


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("trigger", [1, 2])
def test_programmatic_launch_behind_an_early_trigger(cuda, mode, trigger):
    """A predecessor that releases its dependents at once writes g; the many-row kernel must not read it before that."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    M, K, N = 200, 640, 1152
    w = [mk(K, N) * 0.02, mk(K, N).to(torch.float8_e4m3fn), torch.randint(0, 0x7F, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)][mode]
    x, wg, u, gx, gw, routed = mk(M, 2560), mk(2560, K) * 0.02, mk(M, K), mk(M, 512), mk(512, 1), mk(M, N)
    before, op, after = SkinnyGemm([1], [K], trigger=1), SharedExpertDown(trigger=trigger), SkinnyGemm([1], [K], trigger=1)
    for node in (before, op, after):
        node.set_option("pdl_wait", 1)
    for node in (before, after):
        node.set_option("dense_rows", 0)
    want = SharedExpertDown()(before(x, wg)[0], u, w, gx, gw, routed)
    wn = mk(N, K) * 0.02
    want_next = after(want, wn)[0]
    torch.cuda.synchronize()

    def chain():
        g = before(x, wg)[0]
        y = op(g, u, w, gx, gw, routed)
        return y, after(y, wn)[0]

    for _ in range(50):
        y, z = chain()
        assert torch.equal(y, want) and torch.equal(z, want_next)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y, z = chain()
    for _ in range(20):
        y.zero_()
        z.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want) and torch.equal(z, want_next)


def test_bad_launch_shapes(cuda):
    z = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda")
    op = SharedExpertDown()
    for plan in ("24,1", "272,1", "48,4", "64,3", "64,8"):
        op.set_option("dense_plan", plan)
        with pytest.raises(QfgError):
            op(z(20, 64), z(20, 64), z(64, 64), z(20, 64), z(64, 1), z(20, 64))


def test_gates_are_fp32_sums(cuda):
    """Gates of 4096 elements of one sign against the 64-bit ones, by a weight that makes them the output.  FP32 sums in any order are off by a
    few 2^-24, one BF16 number in some ten thousand; a tensor core accumulator that runs through k made 91 of 204 800 wrong, rounded sums none."""
    M, K, N, gk = 2048, 64, 128, 4096
    g, u = torch.full((M, K), 16.0, device="cuda").bfloat16(), torch.full((M, K), 1 / 16, device="cuda").bfloat16()  # swish_mul is 1
    w, routed = torch.zeros(K, N, dtype=torch.bfloat16, device="cuda"), torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    w[0] = 1
    op, wrong = SharedExpertDown(), 0
    for seed in range(50):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        gx = torch.randn(M, gk, generator=gen, device="cuda").abs().bfloat16()
        gw = -(torch.randn(gk, 1, generator=gen, device="cuda") * 0.0025).abs().bfloat16()
        logit = (gx.double() @ gw.double()).bfloat16().float()
        wrong += (op(g, u, w, gx, gw, routed) != torch.sigmoid(logit).bfloat16()).any(dim=1).sum().item()
    assert wrong <= 6  # of 102 400: 42 with the running accumulator


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("plan", ["32,1", "64,2", "160,7,0,1"])
def test_waits_that_run_out_give_nan(cuda, mode, plan):
    """swish_mul never comes: every output is NaN, and the next call is whole."""
    gen = torch.Generator(device="cuda").manual_seed(mode)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    M, K, N = 170, 648, 1152
    w = [mk(K, N), mk(K, N).to(torch.float8_e4m3fn), torch.randint(0, 0x70, (K, N * 9 // 16), generator=gen, device="cuda", dtype=torch.uint8)][mode]
    args = mk(M, K), mk(M, K), w, mk(M, 256), mk(256, 1) * 0.02, mk(M, N)
    op = SharedExpertDown()
    op.set_option("dense_plan", plan)
    first = op(*args)
    for _ in range(2):
        op.set_option("give_up", 1)
        assert torch.isnan(op(*args)).all()
        op.set_option("give_up", 0)
        assert torch.equal(op(*args), first)
