"""The kernels for narrow results at small and unaligned sizes: the k shares of a cluster, one to four rows per warp, rows
that start anywhere - against the CPU oracle, and the fused forms against their two builtins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import HostBuiltins
    return HostBuiltins("cuda:0")


@pytest.fixture(scope="module")
def par_oracle():
    from oracle import oracle as orc
    o = orc.Oracle()
    o.set_threads(o.max_threads())
    return o


@pytest.mark.parametrize("m,n,k", [(1, 1, 32), (1, 10, 4096), (16, 10, 4096), (256, 1, 784), (255, 3, 785), (1200, 10, 130),
                                   (2400, 16, 100), (3001, 7, 33), (4099, 2, 260), (5, 16, 5000), (1, 2, 8191),
                                   (784, 1, 256), (783, 10, 1024), (4097, 5, 999), (907, 1, 67), (2, 4, 1025)])
@pytest.mark.parametrize("tl,tr", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_narrow_results(gpu, par_oracle, tl, tr, m, n, k):
    import torch
    rng = np.random.default_rng(m + 3 * n + 7 * k + tl * 2 + tr)
    l = rng.uniform(-1, 1, (k, m) if tl else (m, k)).astype(np.float32)
    r = rng.uniform(-1, 1, (n, k) if tr else (k, n)).astype(np.float32)
    ref, mag = par_oracle.fmatmul_f64(tl, tr, l, r)
    got = gpu.fmatmul(tl, tr, l, r)
    assert np.max(np.abs(got.astype(np.float64) - ref) / mag) <= 1e-6
    assert np.array_equal(got.view(np.uint32), gpu.fmatmul(tl, tr, l, r).view(np.uint32))
    lib, st = gpu.d.lib, torch.cuda.current_stream().cuda_stream
    L, R, P = torch.from_numpy(l).cuda(), torch.from_numpy(r).cuda(), torch.from_numpy(got).cuda()
    out, want = torch.empty_like(P), torch.empty_like(P)
    lib.call("polar_b200_fmatmul_sigmoid", tl, tr, m, n, k, L.data_ptr(), R.data_ptr(), out.data_ptr(), None, 0, st)
    gpu.d.fsigmoid(P, want)
    assert torch.equal(out.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("rows,kh,n", [(32, 36, 1), (100, 64, 3), (1024, 784, 10), (1025, 40, 10), (600, 2048, 16), (5000, 132, 7)])
def test_one_pass_backward_keeps_the_bits_of_its_builtins(gpu, rows, kh, n):
    import torch
    lib, st = gpu.d.lib, torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(rows + kh + n)
    H = torch.empty((rows, kh), device="cuda").uniform_(1e-5, 1 - 1e-5, generator=g)
    dZ = torch.empty((rows, n), device="cuda").uniform_(-1, 1, generator=g)
    W = torch.empty((kh, n), device="cuda").uniform_(-0.5, 0.5, generator=g)
    want_dw, dw = torch.empty((kh, n), device="cuda"), torch.empty((kh, n), device="cuda")
    want_in, din = torch.empty((rows, kh), device="cuda"), torch.empty((rows, kh), device="cuda")
    gpu.d.fmatmul(1, 0, H, dZ, want_dw)
    lib.call("polar_b200_fmatmul_sigmoid_grad", 0, 1, rows, kh, n, dZ.data_ptr(), W.data_ptr(), H.data_ptr(), want_in.data_ptr(),
             None, 0, st)
    lib.call("polar_b200_fdense_grad", rows, kh, n, dZ.data_ptr(), W.data_ptr(), H.data_ptr(), dw.data_ptr(), din.data_ptr(), None,
             0, st)
    assert torch.equal(dw.view(torch.int32), want_dw.view(torch.int32))
    assert torch.equal(din.view(torch.int32), want_in.view(torch.int32))
