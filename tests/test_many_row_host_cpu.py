"""The host side of the many-row calls (csrc/dense_tc.cu, csrc/capi.cc) against a CUDA runtime that runs nothing and
records every launch (fake_cuda.c): devices, set-up, and the way a call goes.  Each case is a process of its own, since the
library's set-up belongs to the process."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PRELUDE = """
import ctypes, importlib.util, json, os
spec = importlib.util.spec_from_file_location("qfg_lib", os.path.join({root!r}, "qwen38_flash_ops_b200", "_lib.py"))
L = importlib.util.module_from_spec(spec)
spec.loader.exec_module(L)
lib, fake = L.load(), ctypes.CDLL({fake!r})
fake.fake_log.restype = ctypes.c_char_p
BF16, FP8, U8 = L.QFG_BFLOAT16, L.QFG_FLOAT8E4M3FN, L.QFG_UINT8
cols = lambda dtype, n: n * 9 // 16 if dtype == U8 else n
P = 1 << 20  # an address nothing reads

def gemm(seg_outs, widths, **options):
    h = ctypes.c_void_p()
    assert lib.qfg_skinny_gemm_create(L.i64_array(seg_outs), len(seg_outs), L.i64_array(widths), len(widths), None, 0, 0, ctypes.byref(h)) == 0
    for k, v in options.items():
        assert lib.qfg_skinny_gemm_set_option(h, k.encode(), str(v).encode()) == 0
    return h

def run_gemm(h, dtype, m, k, widths):
    fake.fake_clear()
    w = (L.Tensor2D * len(widths))(*[L.Tensor2D(P, dtype, k, cols(dtype, sum(o))) for o in widths])
    n = sum(len(o) for o in widths)
    outs = (ctypes.c_void_p * n)(*[P] * n)
    code = lib.qfg_skinny_gemm_compute(h, P, m, k, w, len(widths), outs, n, None)
    return code, (lib.qfg_last_error().decode() if code else ""), fake.fake_log().decode().split("\\n")[:-1]

def shared(**options):
    h = ctypes.c_void_p()
    assert lib.qfg_shared_expert_down_create(None, 0, 0, ctypes.byref(h)) == 0
    for k, v in options.items():
        assert lib.qfg_shared_expert_down_set_option(h, k.encode(), str(v).encode()) == 0
    return h

def run_shared(h, dtype, m, k, n):
    fake.fake_clear()
    w = L.Tensor2D(P, dtype, k, cols(dtype, n))
    code = lib.qfg_shared_expert_down_compute(h, P, P, m, k, ctypes.byref(w), P, 64, P, P, n, P, None)
    return code, (lib.qfg_last_error().decode() if code else ""), fake.fake_log().decode().split("\\n")[:-1]
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cuda.so")
    inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    # found under cuBLAS's name when the library looks for it
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-O1", "-I" + inc, "-Wl,-soname,libcublas.so.12", "-o", so, os.path.join(HERE, "fake_cuda.c")])

    def run(body):
        code = PRELUDE.format(root=ROOT, fake=so) + textwrap.dedent(body)
        r = subprocess.run([sys.executable, "-c", code], env={**os.environ, "LD_PRELOAD": so}, capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout)

    return run


def _kernels(log):
    return [next((k for k in ("DenseTcKernel", "DenseSharedKernel", "DequantKernel", "SkinnyGemm") if k in line), line.split()[0]) for line in log]


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_many_rows_on_a_second_device(fake, dtype):
    """A node is not tied to the device that was current when the process made its first one."""
    out = fake(f"""
        h = gemm([1], [256])
        first = run_gemm(h, {dtype}, 64, 512, [[256]])
        fake.fake_device(1)
        print(json.dumps([first, run_gemm(h, {dtype}, 64, 512, [[256]]), run_gemm(gemm([1], [256]), {dtype}, 2000, 512, [[256]])]))
        """)
    for device, (code, message, log) in zip((0, 1, 1), out):
        assert code == 0, message
        assert _kernels(log) == ["DenseTcKernel"] and f"device={device} " in log[0]


def test_shared_expert_is_refused_on_a_second_device_at_any_row_count(fake):
    few, many = fake("""
        h = shared()
        assert run_shared(h, FP8, 40, 256, 128)[0] == 0
        fake.fake_device(1)
        print(json.dumps([run_shared(h, FP8, 4, 256, 128), run_shared(h, FP8, 40, 256, 128)]))
        """)
    assert few[0] != 0 and few == many


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_first_many_row_call_sets_nothing_up(fake, dtype):
    """Kernel attributes and cluster residency belong to the creation of a node: a first call may be captured."""
    out = fake(f"""
        h, s = gemm([1], [256]), shared()
        calls = fake.fake_setup_calls()
        fake.fake_refuse_setup(1)
        r = [run_gemm(h, {dtype}, 64, 512, [[256]]), run_gemm(h, {dtype}, 1000, 5120, [[256]]), run_shared(s, {dtype}, 40, 256, 128)]
        print(json.dumps([calls, fake.fake_setup_calls(), r]))
        """)
    assert out[0] == out[1]
    for code, message, log in out[2]:
        assert code == 0, message


def test_a_failed_set_up_is_tried_again(fake):
    out = fake("""
        h = gemm([1], [256])
        fake.fake_device(1)
        fake.fake_refuse_setup(1)
        bad = run_gemm(h, FP8, 64, 512, [[256]])
        fake.fake_refuse_setup(0)
        print(json.dumps([bad, run_gemm(h, FP8, 64, 512, [[256]])]))
        """)
    assert out[0][0] != 0 and out[1][0] == 0


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_shared_expert_options_at_any_row_count(fake, dtype):
    """`pdl_wait` reaches the many-row kernel's launch; a pinned launch geometry or load path is the streaming kernels'."""
    out = fake(f"""
        r = [run_shared(shared(), {dtype}, 40, 256, 128), run_shared(shared(pdl_wait=1), {dtype}, 40, 256, 128),
             run_shared(shared(plan="direct=0,wn=2,wk=2,cluster=1"), {dtype}, 40, 256, 128), run_shared(shared(force_slow=1), {dtype}, 40, 256, 128)]
        os.environ["QFG_PLAN"] = "direct=0,wn=2,wk=2,cluster=1"
        print(json.dumps(r + [run_shared(shared(), {dtype}, 40, 256, 128)]))
        """)
    for code, message, log in out:
        assert code == 0, message
    logs = [log for _, _, log in out]
    assert _kernels(logs[0]) == _kernels(logs[1]) == ["DenseSharedKernel"]
    assert logs[0][0].endswith("pdl=0") and logs[1][0].endswith("pdl=1")
    for log in logs[2:]:
        assert _kernels(log) == ["SkinnyGemm"] * 5  # eight rows a pass
    # the three weight types' ring kernels, not whatever the planner prefers
    assert all("SkinnyGemmRingKernel" in line and "threads=128 " in line for line in logs[2] + logs[4])


@pytest.mark.parametrize("dtype", ["BF16", "FP8", "U8"])
def test_what_the_many_row_kernels_cannot_take_goes_the_general_way(fake, dtype):
    """A tensor map that cannot be made, and more rows than the kernel counts: the library branch (with its
    dequantisation) and the streaming kernels take these calls."""
    gemm, shared, rows = fake(f"""
        h, s = gemm([1], [256]), shared()
        fake.fake_refuse_encode(1)
        r = [run_gemm(h, {dtype}, 64, 512, [[256]]), run_shared(s, {dtype}, 40, 256, 256)]
        fake.fake_refuse_encode(0)
        print(json.dumps(r + [run_gemm(h, {dtype}, 2 ** 30, 8, [[256]])]))
        """)
    library = [] if dtype == "BF16" else ["DequantKernel"]
    assert gemm[0] == 0 and _kernels(gemm[2]) == library + ["cublas"], gemm
    assert rows[0] == 0 and _kernels(rows[2]) == library + ["cublas"], rows
    assert shared[0] == 0 and _kernels(shared[2]) == ["SkinnyGemm"] * 5, shared


@pytest.mark.parametrize("resident,clusters", [(132, True), (2, False), (1, False)])
def test_launch_shapes_use_the_clusters_that_the_device_holds(fake, resident, clusters):
    """Both planners ask the device: where it holds one or none at a time, neither splits K nor shares rows over clusters."""
    out = fake(f"""
        fake.fake_resident({resident})
        print(json.dumps([run_gemm(gemm([1], [256]), FP8, 40, 5120, [[256]]), run_shared(shared(), FP8, 777, 640, 2560)]))
        """)
    for code, message, log in out:
        assert code == 0 and len(log) == 1, message
        assert (" cluster=1 " not in log[0]) == clusters, log


@pytest.mark.parametrize("dtype", ["FP8", "U8"])
def test_blocks_per_stage_of_a_pinned_shape(fake, dtype):
    """Two blocks a stage are what tiles of up to 128 rows have anyway; unpaired tiles above have one, and pinning two takes it where there
    is room for two and is refused where there never was."""
    out = fake(f"""
        def launch(plan):
            code, error, log = run_gemm(gemm([1], [512], dense_plan=plan), {dtype}, 300, 2048, [[512]])
            return log if code == 0 else error
        shapes = ["16,1,0", "48,3,0", "128,1,0", "128,8,0", "64,1,1", "128,1,1"]
        print(json.dumps([[(launch(p + b), launch(p)) for p in shapes] for b in (",2", ",1")] + [[launch("160,1,0,2"), launch("160,1,0,1"), launch("256,1,0,2")]]))
        """)
    assert all(a == b for a, b in out[0])
    assert all(len(a) == len(b) == 1 and a != b for a, b in out[1])  # one block a stage: through shared memory
    assert out[2][0] == out[2][1] and "bad launch shape" in out[2][2]
