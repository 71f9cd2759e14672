"""csrc/calls.cc without a GPU: what is not a plain dense CUDA tensor is handed back to the Python code, with no error left
behind."""
import os
import shutil
import subprocess
import sys

import pytest
import torch

import qwen38_flash_ops_b200 as package
from qwen38_flash_ops_b200 import ArgmaxRows, QfgError, _calls
from qwen38_flash_ops_b200 import ops


class Sub(torch.Tensor):
    pass


@pytest.mark.parametrize("x", [torch.zeros(2, 8, dtype=torch.bfloat16), torch.zeros(8, 2, dtype=torch.bfloat16).t(), torch.zeros(()),
                               torch.zeros(2, 8, device="meta"), torch.zeros(2, 8).as_subclass(Sub), None, 3])
def test_other_arguments_are_handed_back(x):
    assert _calls.argmax_rows(x, True) is None
    assert _calls.skinny_gemm(1, x, (x,), [8]) is None
    assert _calls.dequant(1, x, [8]) is None
    assert _calls.shared_expert_down(1, x, x, x, x, x, x) is None
    assert _calls.lmhead(1, x, x, x, 8, 0) is None


def test_odd_arguments_leave_no_error_behind():
    x = torch.zeros(2, 8, dtype=torch.bfloat16)
    for args in [(), (None, x, (x,), [8]), (1, x, [x], [8]), (1, x, (x,), ["8"]), (1, x, (x,), [2 ** 70]), ("1", x, (x,), [8])]:
        assert _calls.skinny_gemm(*args) is None
    assert _calls.lmhead(1, x, x, x, 2.5, "0") is None and _calls.argmax_rows(x, 1) is None


def test_under_vmap_and_functionalisation():
    seen = []

    def f(x):
        seen.append(_calls.argmax_rows(x, True))
        return x

    torch.func.vmap(f)(torch.zeros(3, 2, 8))
    torch.func.functionalize(f)(torch.zeros(2, 8))
    torch.func.grad(lambda x: f(x).sum())(torch.zeros(2, 8))
    assert seen == [None, None, None]


def test_bind_checks_its_addresses():
    with pytest.raises(TypeError):
        _calls.bind(1, 2)
    with pytest.raises(ValueError):
        _calls.bind(0, 1, 1, 1, 1)


def test_errors_are_the_python_codes(monkeypatch):
    ops._load()
    with pytest.raises(QfgError, match="contiguous CUDA tensor"):
        ArgmaxRows()(torch.zeros(2, 8))


@pytest.mark.parametrize("extension", ["absent", "damaged", "for another torch", "without a version"])
def test_ops_without_the_extension(tmp_path, extension):
    """The package with the library alone, or beside an extension that this torch cannot load: the Python code serves the calls."""
    src = os.path.dirname(package.__file__)
    pkg = tmp_path / os.path.basename(src)
    pkg.mkdir()
    for name in os.listdir(src):
        if name.endswith(".py"):
            shutil.copy(os.path.join(src, name), pkg)
    if extension == "damaged":
        (pkg / "_calls.so").write_bytes(b"not a library")
    elif extension != "absent":
        (pkg / "_calls.py").write_text("torch_version = '1.0'\n" if extension == "for another torch" else "")
    code = """
import warnings, torch
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    from qwen38_flash_ops_b200 import ArgmaxRows, QfgError
assert any("_calls" in str(w.message) for w in seen)
try:
    ArgmaxRows()(torch.zeros(2, 8))
except QfgError as e:
    assert "contiguous CUDA tensor" in str(e)
else:
    raise AssertionError("accepted")
"""
    env = {**os.environ, "PYTHONPATH": str(tmp_path), "QFG_LIBRARY": os.path.join(src, "libqfg_b200.so")}
    r = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_the_extension_serves_this_torch():
    assert _calls.torch_version == torch.__version__ and ops._calls is _calls


@pytest.mark.gpu
def test_calls_handed_back_give_the_same(cuda, monkeypatch):
    from qwen38_flash_ops_b200 import DequantWeightBf16, LmHeadArgmax, SharedExpertDown, SkinnyGemm

    gen = torch.Generator(device="cuda").manual_seed(2)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    x, w, g, u, gx, gw, routed = mk(2, 3, 64), mk(64, 256), mk(3, 64), mk(3, 64), mk(3, 32), mk(32, 1), mk(3, 256)

    def every():
        return [*SkinnyGemm([2], [64, 192])(x, w), *ArgmaxRows()(x), ArgmaxRows()(x, with_val=False), *DequantWeightBf16(256, widths=[128, 128])(w),
                *LmHeadArgmax()(x, w, 256), SharedExpertDown()(g, u, w, gx, gw, routed)]

    direct = every()
    for name in ("skinny_gemm", "argmax_rows", "dequant", "lmhead", "shared_expert_down"):
        monkeypatch.setattr(ops._calls, name, lambda *args: None)
    for a, b in zip(direct, every(), strict=True):
        assert a.shape == b.shape and a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)


def _make(*args):
    src = os.path.join(os.path.dirname(package.__file__), "csrc")
    return subprocess.run(["make", "-C", src, *args], capture_output=True, text=True, timeout=300)


def test_make_without_torch_builds_the_rest():
    """Hosts of the C ABI need neither Python nor torch."""
    r = _make("-n", "PYTHON=false", "CALLS=/nonexistent/_calls.so", "LIB=/nonexistent/libqfg.so")
    assert r.returncode == 0 and "libqfg.so" in r.stdout and "calls.cc" not in r.stdout, r.stderr


def test_make_builds_the_extension_anew_for_another_torch(tmp_path):
    python = tmp_path / "python"
    calls = tmp_path / "_calls.so"
    for version, expected in (("1", True), ("1", False), ("2", True)):
        python.write_text(f"#!/bin/sh\necho -DQFG_TORCH_VERSION={version}\n")
        python.chmod(0o755)
        r = _make(f"PYTHON={python}", f"CALLS={calls}", f"OBJ={tmp_path}", "HOSTCXX=true", str(calls))  # compiles nothing
        assert r.returncode == 0 and ("calls.cc" in r.stdout) == expected, (version, r.stdout, r.stderr)
        calls.touch()


@pytest.mark.parametrize("name", ["SkinnyGemm", "DequantWeightBf16", "SharedExpertDown", "LmHeadArgmax"])
def test_a_destroyed_node_is_not_called(name):
    """Its address goes with the handle: the C++ calls hand None back, and the library refuses a null node."""
    freed = []

    class Lib:
        def __getattr__(self, entry):
            return freed.append

    op = object.__new__(getattr(ops, name))
    op._lib, op._h, op._p = Lib(), 1, 1
    op.__del__()
    op.__del__()
    assert freed == [1] and op._h is None and op._p is None
