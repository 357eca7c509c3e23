"""Products with a NaN or an infinity in an operand: every sum it enters has the class that IEEE arithmetic gives it, and all
other results keep their bits.  One shape per kernel that fmatmul can take, and every configuration of the cluster kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VALUES = [0x7FC00000, 0x7FFFFFFF, 0xFFFFFFFF, 0x7F800001, 0x7F800000, 0xFF800000]   # four NaNs, two infinities


@pytest.fixture(scope="module")
def d():
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import DeviceBuiltins
    return DeviceBuiltins()


def check(run, tl, tr, m, n, k, tensor_core_tiles=False):
    """run(left, right, out).  The 256-column tensor-core tiles make a NaN of an infinity (inf - inf in its lo part)."""
    import torch
    rng = np.random.default_rng(m + n + k + 2 * tl + tr)
    left = rng.uniform(0.5, 1, (k, m) if tl else (m, k)).astype(np.float32) * rng.choice([-1, 1], (k, m) if tl else (m, k)).astype(np.float32)
    right = rng.uniform(0.5, 1, (n, k) if tr else (k, n)).astype(np.float32) * rng.choice([-1, 1], (n, k) if tr else (k, n)).astype(np.float32)
    i, j, kk = m - 1 - m // 3, n // 2, k - 1 - k // 5
    # an infinity meets a zero, and numbers that have no lo part
    if n > 1:
        right[(n - 1, kk) if tr else (kk, n - 1)] = 0
        right[(0, kk) if tr else (kk, 0)] = 1
    if m > 1:
        left[(kk, 0) if tl else (0, kk)] = 0
    L, R = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    clean = torch.full((m, n), -7.0, device="cuda")
    run(L, R, clean)
    assert bool(torch.isfinite(clean).all())
    for bits in VALUES:
        value = float(np.uint32(bits).view(np.float32))
        for in_left in (True, False):
            A, B = L.clone(), R.clone()
            spoilt, at = (A, (kk, i) if tl else (i, kk)) if in_left else (B, (j, kk) if tr else (kk, j))
            spoilt.view(torch.int32)[at] = bits - (bits >> 31 << 32)
            out = torch.full((m, n), -7.0, device="cuda")
            run(A, B, out)
            got = (out[i] if in_left else out[:, j]).cpu().numpy()
            with np.errstate(all="ignore"):
                # what meets the value decides; the other terms are finite
                want = value * ((right[:, kk] if tr else right[kk]) if in_left else (left[kk] if tl else left[:, kk])).astype(np.float64)
            if tensor_core_tiles and np.isinf(value):
                assert not np.isfinite(got).any(), (hex(bits), in_left)
            else:
                assert np.array_equal(np.isnan(got), np.isnan(want)), (hex(bits), in_left)
                assert np.array_equal(got[~np.isnan(want)], want[~np.isnan(want)].astype(np.float32)), (hex(bits), in_left)
            rest = torch.ones((m, n), dtype=torch.bool, device="cuda")
            if in_left:
                rest[i] = False
            else:
                rest[:, j] = False
            assert torch.equal(out[rest], clean[rest]), (hex(bits), in_left)


@pytest.mark.parametrize("tl,tr,m,n,k,tiles", [
    (0, 0, 33, 17, 50, False), (1, 1, 5, 7, 31, False),           # below a tile
    (0, 0, 999, 514, 301, False), (1, 0, 301, 514, 999, False),   # unaligned rows: padded copies, either orientation
    (0, 0, 16, 640, 784, False), (0, 1, 256, 320, 256, False), (0, 0, 512, 512, 512, False),   # clusters on the operands as they are
    (0, 0, 512, 10, 4096, False), (0, 1, 2049, 16, 1000, False), (1, 0, 514, 7, 999, False),   # few columns, 32-column tiles
    (0, 0, 16, 10, 1024, False), (0, 0, 20000, 3, 512, False), (1, 0, 256, 10, 300, False), (1, 0, 512, 10, 4096, False),   # narrow kernels
    (0, 1, 300, 64, 10, False),                                   # few terms
    (0, 0, 2048, 4096, 256, True)])                               # 256-column tiles
def test_products(d, tl, tr, m, n, k, tiles):
    check(lambda a, b, out: d.fmatmul(tl, tr, a, b, out), tl, tr, m, n, k, tiles)


@pytest.mark.parametrize("k", [4096, 40960])
def test_rows_past_the_tiles(d, k):
    # t_f, 772 = 3 * 256 + 4 rows: the last four are no tensor-core rows, the rest are
    import torch
    g = torch.Generator(device="cuda").manual_seed(k)
    left, right = (torch.empty(s, device="cuda").uniform_(0.5, 1, generator=g) for s in ((k, 772), (k, 256)))
    for value in (float("nan"), float("inf")):
        for row in (770, 5):
            spoilt = left.clone()
            spoilt[k // 2, row] = value
            out = torch.zeros((772, 256), device="cuda")
            d.fmatmul(1, 0, spoilt, right, out)
            assert not bool(torch.isfinite(out[row]).any()) and bool(torch.isfinite(out[:row]).all() and torch.isfinite(out[row + 1:]).all())
            assert row == 5 or value != value or bool((out[row] == value).all())


@pytest.mark.parametrize("tl,tr", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_every_configuration_of_the_cluster_kernel(d, tl, tr):
    m, n, k = 131, 66, 101
    for width in (32, 64, 128):
        for exchanged in (0, 1000):
            for rounded in (0, 1):
                check(lambda a, b, out: d.fmatmul_tc(tl, tr, a, b, out, tile_n=2000 + width + exchanged, slab_k=32,   # noqa: B023
                                                     splits=1 + rounded, write_hi=rounded), tl, tr, m, n, k)


@pytest.mark.parametrize("tl,tr,m,n,k", [(0, 0, 140, 70, 301), (1, 1, 70, 140, 96), (0, 1, 512, 10, 4096)])
def test_the_largest_numbers(d, tl, tr, m, n, k):
    # the hi part of the largest numbers rounds to an infinity, the results are finite
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    left, right = (torch.empty(s, device="cuda").uniform_(0.01, 0.1, generator=g) for s in ((k, m) if tl else (m, k), (n, k) if tr else (k, n)))
    for spoilt in (left, right):
        a, b = left.clone(), right.clone()
        (a if spoilt is left else b)[3, 5] = torch.finfo(torch.float32).max
        out = d.fmatmul(tl, tr, a, b, torch.empty((m, n), device="cuda"))
        ref = (a.double().t() if tl else a.double()) @ (b.double().t() if tr else b.double())
        assert float(((out.double() - ref).abs() / ref).max()) <= 4e-7 * (10 if k > 1000 else 1)   # 8 ulp; a sum of thousands
