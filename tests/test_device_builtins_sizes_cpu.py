"""DeviceBuiltins' checked path, which runs when the native binding declines a call: a tensor shorter than what the builtin
reads or writes is a ValueError before anything is launched, a longer one is accepted.  Stand-ins for tensors and library."""
import math
import types

import pytest

import __graft_entry__ as ge

ge.load_package()
import torch  # noqa: E402
from polarai_framework_b200 import device_builtins  # noqa: E402


class FakeTensor:
    is_cuda, dtype, device = True, torch.float32, "cuda:0"

    def __init__(self, *shape):
        self.shape = shape

    def numel(self):
        return math.prod(self.shape)

    def is_contiguous(self):
        return True

    def data_ptr(self):
        return 256


class Recorder:
    def __init__(self):
        self.calls = []

    def call(self, name, *args):
        self.calls.append(name)


@pytest.fixture
def d(monkeypatch):
    monkeypatch.setattr(device_builtins, "_stream", lambda t: 0)
    b = device_builtins.DeviceBuiltins.__new__(device_builtins.DeviceBuiltins)
    b.lib = Recorder()
    b._native = types.SimpleNamespace(**{n: lambda *a: False for n in (
        "ffill", "fcopy", "fadd", "fmul", "fdivide", "fsigmoid", "fsigmoid_unclamped", "flogloss", "fmulconcat", "frelu", "fsoftmax",
        "fpool", "fconv2d", "ftranspose", "fmatmul")})
    return b


T = FakeTensor
CALLS = {   # of the size that the argument is short or long of: called with it, with one less and with one more
    "fcopy": lambda d, n: d.fcopy(T(n), T(8)), "fadd a": lambda d, n: d.fadd(T(n), 1, T(8), 1, T(8)),
    "fadd b": lambda d, n: d.fadd(T(8), 1, T(n), 1, T(8)), "fmul": lambda d, n: d.fmul(T(n), T(8), T(8)),
    "fdivide": lambda d, n: d.fdivide(T(8), T(n), T(8)), "fsigmoid": lambda d, n: d.fsigmoid(T(n), T(8)),
    "fsigmoid_unclamped": lambda d, n: d.fsigmoid(T(n), T(8), clamp=False), "flogloss": lambda d, n: d.flogloss(T(8), T(n), T(8)),
    "fmulconcat": lambda d, n: d.fmulconcat(T(1), T(n), T(8)), "frelu": lambda d, n: d.frelu(T(n), T(8)),
    "fsoftmax": lambda d, n: d.fsoftmax(T(n), T(8)), "fpool": lambda d, n: d.fpool(T(5, 9), (2, 3), (2, 2), T(n)),
    "fconv2d": lambda d, n: d.fconv2d(T(4, 6), T(3, 3), T(n)), "ftranspose": lambda d, n: d.ftranspose(T(2, 4), T(n)),
    "fslice": lambda d, n: d.fslice(T(n, 1), n - 5, T(4)) if n < 8 else d.fslice(T(n, 1), 1, T(4)),
    "fmatmul_ffma": lambda d, n: d.fmatmul_ffma(0, 0, T(2, 3), T(3, 4), T(n)),
    "fmatmul_tc": lambda d, n: d.fmatmul_tc(0, 0, T(2, 3), T(3, 4), T(n))}


@pytest.mark.parametrize("name", CALLS)
def test_short_tensors_are_refused_and_long_ones_taken(d, name):
    with pytest.raises(ValueError):
        CALLS[name](d, 7)
    assert d.lib.calls == []
    CALLS[name](d, 8)
    CALLS[name](d, 9)
    assert len(d.lib.calls) == 2


@pytest.mark.gpu
def test_the_binding_declines_what_does_not_fit():
    d = device_builtins.DeviceBuiltins()
    new = lambda *s: torch.zeros(s, device="cuda")  # noqa: E731
    before = d.lib.launch_count()
    for call in (lambda: d.fcopy(new(7), new(8)), lambda: d.fadd(new(8), 1, new(7), 1, new(8)), lambda: d.fsoftmax(new(7), new(8)),
                 lambda: d.fmulconcat(new(1), new(7), new(8)), lambda: d.fpool(new(5, 9), (2, 3), (2, 2), new(7)),
                 lambda: d.fconv2d(new(4, 6), new(3, 3), new(7)), lambda: d.ftranspose(new(2, 4), new(7)),
                 lambda: d.fmatmul(0, 0, new(2, 3), new(3, 4), new(7))):
        with pytest.raises((ValueError, IndexError)):
            call()
    assert d.lib.launch_count() == before
    long = torch.full((10,), 7.0, device="cuda")
    assert d.fconv2d(torch.ones((4, 6), device="cuda"), torch.ones((3, 3), device="cuda"), long).tolist() == [9.0] * 8 + [7.0] * 2
