"""Prepared programs: elementwise builtins that share a launch, and the graph replay, give every tensor the
bits of the builtins launched one by one."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    return torch


def inputs(torch, prog, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ins = {t: torch.empty(prog.tensors[t], device="cuda").uniform_(0.05, 0.95, generator=g) for t in prog.inputs}
    if "Y" in ins:
        ins["Y"] = (ins["Y"] < 0.5).float()
    return ins


def one_by_one(torch, prog, ins, passes):
    """The program through polar_b200_launch_by_name, one call per builtin."""
    from polarai_framework_b200.program import DeviceExecutor
    ex = DeviceExecutor(prog)
    ex.set_inputs(**ins)
    s = torch.cuda.current_stream().cuda_stream
    for _ in range(passes):
        for kernel, arr, n in ex._compiled:
            if kernel is not None:
                ex.lib.check(ex._fn(kernel, arr, n, ex._ws_ptr, ex._ws_bytes, s))
    torch.cuda.synchronize()
    return {k: v.clone() for k, v in ex.t.items()}


def chains(n):
    from polarai_framework_b200.program import Program
    p = Program("chains")
    for t in ("a", "b", "c", "d", "e", "f", "g", "h", "i", "P", "Y"):
        p.tensor(t, n)
    p.tensor("s", 1), p.tensor("w", 2 * n), p.tensor("v", 2 * n)
    p.inputs = list(p.tensors)
    new = lambda t: p.tensor(t, n)  # noqa: E731
    p.op("ffill", 0.75, new("t0"))
    p.op("fadd", "a", 1.0, "b", -0.5, new("t1"))
    p.op("fmul", "t1", "t1", new("t2"))                # both operands the previous result
    p.op("fmulconcat", "s", "t1", new("t3"))           # an operand from two instructions back
    p.op("fdivide", "t3", "t0", new("t4"))
    p.op("fsigmoid", "t4", new("t5"))
    p.op("frelu", "t2", new("t6"))
    p.op("fcopy", "a", new("t7"))
    p.op("flogloss", "P", "Y", new("t8"))
    p.op("flogloss", "P", "b", new("t9"))              # soft labels
    p.op("fsigmoid_grad", "t8", "P", new("t10"))
    p.op("fsigmoid_logloss_grad", "P", "Y", new("t11"))
    p.op("fadd", "a", 1.0, "t11", -0.1, "a")           # in place, the old value read above
    p.op("fmul", "a", "t7", new("t12"))                # the new value, beside a copy of the old
    for k, t in enumerate("cdefghi"):                  # more inputs than one launch takes
        p.op("fadd", t, 1.0, "t12", float(k), new(f"u{k}"))
    p.op("fmulconcat", "u6", "u5", new("x"))           # the factor is a result of the same pass: a launch of its own
    p.op("fadd", "w", 0.5, "v", 2.0, "w")              # another element count
    p.op("fmul", "w", "v", "v")
    p.outputs = ["x", "v"]
    return p


@pytest.mark.parametrize("n", [1, 3, 4, 5, 511, 512, 513, 4099, 1_000_001])
def test_chains_give_the_bits_of_single_launches(env, n):
    from polarai_framework_b200.program import DeviceExecutor
    prog = chains(n)
    ins = inputs(env, prog, n)
    for passes in (1, 4):                              # 4: the last two are graph replays
        want = one_by_one(env, prog, ins, passes)
        ex = DeviceExecutor(prog)
        ex.set_inputs(**ins)
        for _ in range(passes):
            ex.run()
        env.cuda.synchronize()
        steps = int(ex.lib.cdll.polar_b200_program_steps(ex._only))
        assert 3 <= steps <= 7 < len(prog.ops)
        for t in prog.tensors:
            assert env.equal(ex.t[t].view(env.int32), want[t].view(env.int32)), (n, passes, t)


@pytest.mark.parametrize("fused", [False, True])
def test_steps_replayed_as_a_graph(env, fused):
    # a training step with weights updated in place: eager runs, replays, a side stream and the caller's
    # own capture all advance it identically
    from polarai_framework_b200.program import DeviceExecutor, fuse_program, mlp_program
    prog = mlp_program(300, 65, 130, 7, 1e-3)
    prog = fuse_program(prog) if fused else prog
    ins = inputs(env, prog, 5)
    want = one_by_one(env, prog, ins, 7)
    ex = DeviceExecutor(prog)
    ex.set_inputs(**ins)
    for _ in range(4):
        ex.run()
    side = env.cuda.Stream()
    side.wait_stream(env.cuda.current_stream())
    with env.cuda.stream(side):
        ex.run()
        graph = env.cuda.CUDAGraph()
        with env.cuda.graph(graph, stream=side):
            ex.run()
        graph.replay()
        ex.run()
    env.cuda.synchronize()
    for t in prog.outputs:
        assert env.equal(ex.t[t].view(env.int32), want[t].view(env.int32)), t


def test_a_changed_wait_limit_makes_the_graph_again(env):
    # (the limit itself shows only where a wait runs out; here every wait ends)
    from polarai_framework_b200.program import DeviceExecutor, mlp_program
    prog = mlp_program(300, 65, 130, 7, 1e-3)
    ins = inputs(env, prog, 6)
    want = one_by_one(env, prog, ins, 9)
    ex = DeviceExecutor(prog)
    ex.set_inputs(**ins)
    try:
        for limit in (0, 500_000_000, 0):
            ex.lib.cdll.polar_b200_set_wait_limit_ns(limit)
            for _ in range(3):
                ex.run()
    finally:
        ex.lib.cdll.polar_b200_set_wait_limit_ns(0)
    env.cuda.synchronize()
    for t in prog.outputs:
        assert env.equal(ex.t[t].view(env.int32), want[t].view(env.int32)), t


def test_bad_programs_are_statuses(env):
    from polarai_framework_b200.capi import Arg, Op, PolarB200Error, lib
    from polarai_framework_b200.program import DeviceExecutor, Program
    handle = ctypes.c_void_p()
    assert lib().cdll.polar_b200_program_create(None, 1, None, 0, ctypes.byref(handle)) == 1
    assert lib().cdll.polar_b200_program_run(None, None) == 1
    ops = (Op * 1)()
    ops[0].name, ops[0].args, ops[0].argc = b"fadd", ctypes.cast((Arg * 2)(), ctypes.POINTER(Arg)), 2
    lib().call("polar_b200_program_create", ops, 1, None, 0, ctypes.byref(handle))
    assert lib().cdll.polar_b200_program_run(handle, None) == 3          # what launch_by_name answers
    lib().cdll.polar_b200_program_destroy(handle)
    p = Program("sizes differ")
    p.tensor("a", 8), p.tensor("b", 9), p.tensor("c", 8)
    p.op("fmul", "a", "a", "c")
    p.op("fmul", "a", "b", "c")
    with pytest.raises(PolarB200Error):
        DeviceExecutor(p).run()


def test_scratch_survives_and_can_be_given_back(env):
    from polarai_framework_b200.device_builtins import HostBuiltins
    gpu = HostBuiltins("cuda:0")
    rng = np.random.default_rng(3)
    l, r = rng.uniform(-1, 1, (512, 256)).astype(np.float32), rng.uniform(-1, 1, (512, 4)).astype(np.float32)
    first = gpu.fmatmul(1, 0, l, r)
    gpu.d.lib.call("polar_b200_trim_scratch", 0)
    assert np.array_equal(gpu.fmatmul(1, 0, l, r), first)
