"""Products with sums of up to 2048 terms whose result is no whole number of vectors (m * n no multiple of four): the
tile choice must not cut their sums, with the library's scratch, a caller workspace and the fused sigmoid."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1025, 1025, 2048), (1281, 1793, 2048), (1537, 1537, 2048), (2049, 1793, 2048), (1999, 1281, 1952),
                                   (1538, 1025, 1536)])
def test_results_that_are_no_vectors(m, n, k):
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    d = DeviceBuiltins()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    left = torch.empty((m, k), device="cuda").uniform_(-1, 1, generator=g)
    right = torch.empty((n, k), device="cuda").uniform_(-1, 1, generator=g)
    ref, mag = left.double() @ right.double().t(), left.abs().double() @ right.abs().double().t()
    out = torch.full((m, n), float("nan"), device="cuda")
    d.fmatmul(0, 1, left, right, out)
    # relative to the sum of magnitudes; toward-zero accumulation in steps of eight terms loses at most k / 8 * 2^-23 = 3e-5 of
    # it, and on zero-mean operands a tenth of that and less.  A shifted cut is off by about 1
    assert float(((out.double() - ref).abs() / mag).max()) <= 5e-6
    need = int(d.lib.cdll.polar_b200_fmatmul_workspace_bytes(0, 1, m, n, k))
    ws = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    again, act = (torch.full((m, n), float("nan"), device="cuda") for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream
    d.lib.call("polar_b200_fmatmul", 0, 1, m, n, k, left.data_ptr(), right.data_ptr(), again.data_ptr(), ws.data_ptr(), need, st)
    assert torch.equal(out, again)
    d.lib.call("polar_b200_fmatmul_sigmoid", 0, 1, m, n, k, left.data_ptr(), right.data_ptr(), act.data_ptr(), None, 0, st)
    assert torch.equal(act, d.fsigmoid(out, torch.empty_like(out)))
    assert d.device_status() == 0
