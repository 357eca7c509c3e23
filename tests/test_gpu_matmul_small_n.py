"""Products with up to 16 columns and a K-major left operand on both sides of the line between the narrow kernels and the
32-column tensor-core tiles: every transpose of the small operand, caller and library scratch, the fused sigmoid."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(300, 10, 4096), (513, 7, 4100), (1000, 16, 1024), (2048, 10, 4096), (2049, 1, 8192), (4000, 4, 2047),
                                   (8192, 10, 4096), (8192, 16, 8192), (16384, 10, 4096), (64, 3, 64)])
@pytest.mark.parametrize("tr", [0, 1])
def test_few_columns(m, n, k, tr):
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    d = DeviceBuiltins()
    g = torch.Generator(device="cuda").manual_seed(m + n + k + tr)
    left = torch.empty((m, k), device="cuda").uniform_(-1, 1, generator=g)
    right = torch.empty((n, k) if tr else (k, n), device="cuda").uniform_(-1, 1, generator=g)
    r = (right.t() if tr else right).double()
    ref, mag = left.double() @ r, left.abs().double() @ r.abs()
    out = torch.full((m, n), float("nan"), device="cuda")
    d.fmatmul(0, tr, left, right, out)
    assert float(((out.double() - ref).abs() / mag).max()) <= 4e-7
    assert float((out.double() - ref).norm() / ref.norm()) <= 3e-7
    need = int(d.lib.cdll.polar_b200_fmatmul_workspace_bytes(0, tr, m, n, k))
    ws = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    again, act, both = (torch.full((m, n), float("nan"), device="cuda") for _ in range(3))
    st = torch.cuda.current_stream().cuda_stream
    rc = d.lib.cdll.polar_b200_fmatmul(0, tr, m, n, k, left.data_ptr(), right.data_ptr(), again.data_ptr(), ws.data_ptr(), need, st)
    assert rc == 0 and torch.equal(out, again)
    rc = d.lib.cdll.polar_b200_fmatmul_sigmoid(0, tr, m, n, k, left.data_ptr(), right.data_ptr(), act.data_ptr(), ws.data_ptr(), need, st)
    assert rc == 0
    d.fsigmoid(out, both)
    assert torch.equal(act, both)
    assert d.device_status() == 0


@pytest.mark.parametrize("m,n,k", [(514, 7, 999), (1001, 10, 2000), (130, 16, 8192), (33, 3, 512), (2049, 16, 700), (514, 10, 300)])
@pytest.mark.parametrize("tr", [0, 1])
def test_few_columns_of_rows_that_are_no_vectors(m, n, k, tr):
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    d = DeviceBuiltins()
    g = torch.Generator(device="cuda").manual_seed(m + n + k + tr)
    left = torch.empty((k, m), device="cuda").uniform_(-1, 1, generator=g)
    right = torch.empty((n, k) if tr else (k, n), device="cuda").uniform_(-1, 1, generator=g)
    r = (right.t() if tr else right).double()
    ref = left.double().t() @ r
    out = torch.full((m, n), float("nan"), device="cuda")
    d.fmatmul(1, tr, left, right, out)
    assert float((out.double() - ref).norm() / ref.norm()) <= 3e-7
    need = int(d.lib.cdll.polar_b200_fmatmul_workspace_bytes(1, tr, m, n, k))
    ws = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    again = torch.full((m, n), float("nan"), device="cuda")
    rc = d.lib.cdll.polar_b200_fmatmul(1, tr, m, n, k, left.data_ptr(), right.data_ptr(), again.data_ptr(), ws.data_ptr(), need,
                                       torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(out, again)
    assert d.device_status() == 0
