"""csrc/calls.cc without a GPU: what is not a plain dense CUDA tensor is handed back to the Python code, with no error left
behind."""
import pytest
import torch

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
