"""The cluster kernel of fmatmul (one 128-row tile per cluster of CTAs) against the CPU oracle: every tile width, cluster
size, orientation and transpose form, on sizes around its tile and slab edges, aligned or not."""
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


def operands(tl, tr, m, n, k):
    rng = np.random.default_rng(m * 7 + n * 3 + k + tl * 2 + tr)
    return (rng.uniform(-1, 1, (k, m) if tl else (m, k)).astype(np.float32),
            rng.uniform(-1, 1, (n, k) if tr else (k, n)).astype(np.float32))


def rel_err(got, ref, mag):
    return float(np.max(np.abs(got.astype(np.float64) - ref) / mag))


@pytest.mark.parametrize("tl,tr", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(128, 128, 32), (1, 64, 40), (127, 129, 257), (130, 257, 1000), (300, 33, 96), (77, 200, 2500)])
def test_every_configuration(gpu, par_oracle, tl, tr, m, n, k):
    l, r = operands(tl, tr, m, n, k)
    ref, mag = par_oracle.fmatmul_f64(tl, tr, l, r)
    for width in (32, 64, 128):
        for cluster in (1, 2, 4, 8):
            if (k + 31) // 32 < cluster:
                continue
            for exchanged in (0, 1000):
                for rounded in (0, 1):
                    run = lambda: gpu.fmatmul(tl, tr, l, r, which="tc", tile_n=2000 + width + exchanged,  # noqa: E731
                                              slab_k=32, splits=cluster, write_hi=rounded)
                    got = run()
                    err = rel_err(got, ref, mag)
                    assert err <= (4e-7 if rounded else 5e-6), (width, cluster, exchanged, rounded, err)
                    assert np.array_equal(got.view(np.uint32), run().view(np.uint32))      # the same bits run to run
    assert gpu.d.device_status() == 0


@pytest.mark.parametrize("m,n,k", [(999, 514, 301), (301, 514, 999), (16, 4096, 784), (33, 17, 50), (5, 7, 31), (64, 48, 32),
                                   (1024, 1024, 1024), (1000, 2001, 130), (2001, 1511, 70), (258, 130, 4097), (1, 1, 1)])
@pytest.mark.parametrize("tl,tr", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_dispatch_on_ragged_and_small_products(gpu, par_oracle, tl, tr, m, n, k):
    # through fmatmul, with the library's own scratch and with a caller workspace; unaligned base pointers; and the
    # fused sigmoid, which has to give the bits of the two builtins
    import torch
    l, r = operands(tl, tr, m, n, k)
    ref, mag = par_oracle.fmatmul_f64(tl, tr, l, r)
    got = gpu.fmatmul(tl, tr, l, r)
    assert rel_err(got, ref, mag) <= 5e-6
    lib, st = gpu.d.lib, torch.cuda.current_stream().cuda_stream
    L, R = torch.from_numpy(l).cuda(), torch.from_numpy(r).cuda()
    need = int(lib.cdll.polar_b200_fmatmul_workspace_bytes(tl, tr, m, n, k))
    ws = torch.empty(need + 16, dtype=torch.uint8, device="cuda")
    out = torch.full((m, n), float("nan"), device="cuda")
    lib.call("polar_b200_fmatmul", tl, tr, m, n, k, L.data_ptr(), R.data_ptr(), out.data_ptr(), ws.data_ptr(), need, st)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), got.view(np.uint32))
    prod = out.clone()
    lib.call("polar_b200_fmatmul_sigmoid", tl, tr, m, n, k, L.data_ptr(), R.data_ptr(), out.data_ptr(), None, 0, st)
    gpu.d.fsigmoid(prod, prod)
    assert torch.equal(out.view(torch.int32), prod.view(torch.int32))
    shifted = torch.zeros(L.numel() + 1, device="cuda")
    shifted[1:] = L.flatten()
    base = torch.full((m * n + 2,), float("nan"), device="cuda")
    lib.call("polar_b200_fmatmul", tl, tr, m, n, k, shifted.data_ptr() + 4, R.data_ptr(), base.data_ptr() + 4, None, 0, st)
    assert rel_err(base[1:-1].cpu().numpy().reshape(m, n), ref, mag) <= 5e-6
    assert bool(torch.isnan(base[0])) and bool(torch.isnan(base[-1]))
    assert gpu.d.device_status() == 0
