"""t_f products with a few rows past their last whole tile: the rows that the 256 x 256-tile kernel takes along, in stream
mode and with fixed cuts of k, against float64 - column tiles cut off, k no multiple of a slab, every number of rows."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(784, 4096, 8192), (772, 1000, 4100), (776, 260, 4097), (780, 4096, 5000),
                                   (1536 + 16, 2048, 4096), (784, 4096, 33000), (784, 516, 65536), (2052, 1024, 4096),
                                   (528, 2048, 8192), (272, 4096, 8192)])
def test_rows_past_the_last_tile(m, n, k):
    import torch
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    d = DeviceBuiltins()
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    left = torch.empty((k, m), device="cuda").uniform_(-1, 1, generator=g)
    right = torch.empty((k, n), device="cuda").uniform_(-1, 1, generator=g)
    buf = torch.full((m * n + 4,), float("nan"), device="cuda")
    ref = left.double().t() @ right.double()
    mag = left.abs().double().t() @ right.abs().double()
    outs = []
    for shift in (0, 1, 0):                                  # a result that is only 4-byte aligned; the same bits run to run
        buf.fill_(float("nan"))
        out = buf[shift:shift + m * n].view(m, n)
        d.fmatmul(1, 0, left, right, out)
        err = ((out.double() - ref).abs() / mag).amax(dim=1)
        assert float(err.max()) <= 5e-6
        past = m - m % 128
        assert float(err[past:].max()) <= 4e-7               # sums in round-to-nearest
        assert torch.isnan(buf[shift + m * n:]).all()
        outs.append(out.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert d.device_status() == 0
