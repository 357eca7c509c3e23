"""CPU checks of the C ABI: the library loads, exports every symbol the headers
declare, and rejects bad arguments with a status (no compute without a GPU)."""
import ctypes
import os
import re

import pytest

import __graft_entry__ as ge

ROOT = ge.ROOT


@pytest.fixture(scope="module")
def library():
    ge.build()
    return ge.load_package().lib()


def declared(header):
    text = open(os.path.join(ROOT, "include", header)).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(polar_b200_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(library):
    names = declared("polar_b200.h")
    assert len(names) >= 20
    for name in names:
        assert hasattr(library.cdll, name), name


def test_binding_table_matches_header(library):
    from polarai_framework_b200.capi import SIGNATURES
    assert sorted(SIGNATURES) == declared("polar_b200.h")


def test_bad_arguments_return_status_not_abort(library):
    c = library.cdll
    assert c.polar_b200_ffill(1.0, None, 4, None) == 1
    assert "null" in library.last_error()
    assert c.polar_b200_fadd(None, 1.0, None, 1.0, None, 0, None) == 0      # n == 0 is a no-op
    assert c.polar_b200_fmatmul(2, 0, 4, 4, 4, None, None, None, None, 0, None) == 1
    assert c.polar_b200_fmatmul(0, 0, 0, 4, 4, None, None, None, None, 0, None) == 0
    assert c.polar_b200_launch_by_name(b"fnope", None, 0, None, 0, None) == 3
    assert c.polar_b200_launch_by_name(None, None, 0, None, 0, None) == 1
    assert library.launch_count() == 0


def test_launch_by_name_checks_argument_patterns(library):
    from polarai_framework_b200.capi import Arg
    c = library.cdll
    shape = (ctypes.c_uint64 * 1)(4)
    args = (Arg * 2)()
    for a in args:
        a.is_tensor = 1
        a.tensor.dims = 1
        a.tensor.shape = shape
    assert c.polar_b200_launch_by_name(b"fadd", args, 2, None, 0, None) == 3   # wrong arity
    assert c.polar_b200_launch_by_name(b"fmatmul_f_f", args, 2, None, 0, None) == 3


def test_a_program_that_no_host_can_hold_returns_status_not_abort(library):
    # in a process of its own: an exception that left the C entry would end it
    import subprocess
    import sys
    code = """
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as ge
c = ge.load_package().lib().cdll
from polarai_framework_b200.capi import Arg, Op
for argc, dims in ((1 << 57, 1), (2, 1 << 59)):
    shape, args, handle = (ctypes.c_uint64 * 1)(4), (Arg * 2)(), ctypes.c_void_p(1)
    for a in args:
        a.is_tensor, a.tensor.dims, a.tensor.shape = 1, dims, shape
    op = Op(b"fcopy", args, argc)
    assert c.polar_b200_program_create(ctypes.byref(op), 1, None, 0, ctypes.byref(handle)) == 1
    assert not handle.value and b"memory" in c.polar_b200_last_error()
"""
    r = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stderr[-500:])


def test_the_binding_declines_tensors_without_data(library):
    # in a process of its own: torch throws where such a tensor's data or an unknown device's stream is asked for
    import subprocess
    import sys
    code = """
import sys
sys.path.insert(0, sys.argv[1])
import torch
import __graft_entry__ as ge
ge.load_package()
from polarai_framework_b200.capi import binding
from torch._subclasses.fake_tensor import FakeTensorMode
b = binding()
with FakeTensorMode():
    a, out = torch.empty(4, 4, device="cuda:0"), torch.empty(4, 4, device="cuda:0")
assert not b.ffill(1.0, out) and not b.fcopy(a, out) and not b.fadd(a, 1.0, a, 1.0, out) and not b.fmul(a, a, out)
assert not b.fmulconcat(a, a, out) and not b.fsoftmax(a, out) and not b.fpool(a, 1, 1, 1, 1, out)
assert not b.fconv2d(a, out, out) and not b.ftranspose(a, out) and not b.fmatmul(0, 0, a, a, out)
try:
    b.run_program(0, 63)
except RuntimeError:
    print("raised")
"""
    r = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True)
    assert r.returncode == 0 and "raised" in r.stdout, (r.returncode, r.stdout, r.stderr[-500:])


def test_matmul_path_selection(library):
    c = library.cdll
    assert c.polar_b200_fmatmul_path(0, 0, 8192, 8192, 8192) == 0     # tensor cores
    assert c.polar_b200_fmatmul_path(0, 0, 65536, 4096, 784) == 0
    assert c.polar_b200_fmatmul_path(1, 0, 784, 4096, 65536) == 0
    assert c.polar_b200_fmatmul_path(0, 0, 65536, 10, 4096) != 0      # row pitch 40 B: no TMA
    assert c.polar_b200_fmatmul_path(0, 0, 256, 1, 784) != 0


def test_runtime_plugin_exports_and_opens_without_a_gpu(library):
    from conftest import skip_without_reference
    skip_without_reference()
    from polarai_framework_b200 import runtime
    cdll = runtime.load_rt_library()           # resolves every declared symbol + initContext/closeContext
    assert sorted(runtime.RT_SIGNATURES) == declared("polar_b200_rt.h")
    import torch
    if not torch.cuda.is_available():
        rt = runtime.Runtime()
        assert rt.device_count() == 0          # no sm_100 device: an empty context, not a crash
        with pytest.raises(Exception):
            rt.tensor((4,))
        rt.close()
