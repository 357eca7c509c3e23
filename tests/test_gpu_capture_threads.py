"""What one thread runs while another captures in the global mode, the default of torch.cuda.graph: both come out right."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def while_capturing(call):
    """Runs call on a stream and thread of its own while this thread captures."""
    import torch
    x, y = torch.ones(1000, device="cuda"), torch.zeros(1000, device="cuda")
    torch.add(x, 1, out=y)
    torch.mul(y, 2, out=y)
    torch.cuda.synchronize()
    side, errors = torch.cuda.Stream(), []

    def run():
        try:
            with torch.cuda.stream(side):
                call()
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            errors.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        torch.add(x, 1, out=y)
        thread = threading.Thread(target=run)
        thread.start()
        thread.join()
        torch.mul(y, 2, out=y)
    torch.cuda.synchronize()
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert not errors and y.tolist() == [4.0] * 1000


@pytest.mark.parametrize("tl,m,n,k", [(0, 333, 257, 129), (1, 512, 10, 4096)])    # padded copies; partial sums
def test_scratch_is_allocated_while_another_thread_captures(tl, m, n, k):
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    d = DeviceBuiltins()
    left, right = torch.rand((k, m) if tl else (m, k), device="cuda"), torch.rand((k, n), device="cuda")
    want, out = torch.empty((m, n), device="cuda"), torch.empty((m, n), device="cuda")
    d.fmatmul(tl, 0, left, right, want)                      # (the first launch of a kernel loads it)
    d.lib.call("polar_b200_trim_scratch", 0)
    while_capturing(lambda: d.fmatmul(tl, 0, left, right, out))
    assert torch.equal(out, want)


def test_a_program_becomes_a_graph_while_another_thread_captures():
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.program import DeviceExecutor, mlp_program

    def executor():
        ex = DeviceExecutor(mlp_program(100, 31, 52, 7, 0.01), "cuda:0")
        g = torch.Generator(device="cuda").manual_seed(3)
        new = lambda *s: torch.empty(s, device="cuda").uniform_(-0.5, 0.5, generator=g)  # noqa: E731
        ex.set_inputs(X=new(100, 31), Y=(new(100, 7) > 0).float(), W1=new(31, 52), W2=new(52, 7))
        return ex

    want, ex = executor(), executor()
    for _ in range(6):
        want.run()
    while_capturing(lambda: [ex.run() for _ in range(6)])
    assert all(torch.equal(ex.t[n], want.t[n]) for n in ex.program.outputs)
