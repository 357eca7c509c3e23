"""fconv2d, fpool, fsoftmax and frelu around the edges of their tiles and vectors, against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import __graft_entry__ as ge
    ge.load_package()
    from polarai_framework_b200.device_builtins import HostBuiltins
    return HostBuiltins("cuda:0")


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("k", [1, 3, 5, 7, 9])
@pytest.mark.parametrize("oh,ow", [(1, 1), (7, 127), (8, 128), (9, 129), (17, 260), (3, 1000), (300, 5)])
def test_convolution_tiles(gpu, oracle, k, oh, ow):
    rng = np.random.default_rng(k * oh + ow)
    img = rng.uniform(-1, 1, (oh + k - 1, ow + k - 1)).astype(np.float32)
    ker = rng.uniform(-1, 1, (k, k)).astype(np.float32)
    assert np.array_equal(bits(gpu.fconv2d(img, ker)), bits(oracle.fconv2d(img, ker)))


@pytest.mark.parametrize("h,w", [(2, 3), (3, 255), (67, 514), (130, 1025)])
@pytest.mark.parametrize("window,stride", [((2, 2), (2, 2)), ((2, 2), (1, 3)), ((2, 3), (1, 1)), ((3, 3), (3, 3)), ((3, 3), (2, 1))])
def test_pooling_windows(gpu, oracle, h, w, window, stride):
    if window[0] > h or window[1] > w:
        return
    img = np.random.default_rng(h + w).uniform(-1, 1, (h, w)).astype(np.float32)
    img[0, 0] = np.nan
    assert np.array_equal(bits(gpu.fpool(img, window, stride)), bits(oracle.fpool(img, window, stride)))


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1024, 1025, 151_552, 1_000_003])
def test_softmax_and_relu_sizes(gpu, oracle, n):
    import torch
    x = np.random.default_rng(n).uniform(-4, 4, n).astype(np.float32)
    e = np.exp(x.astype(np.float64))                                            # (the oracle sums in float: too coarse here)
    want = e / e.sum()
    got = gpu.fsoftmax(x)
    assert np.max(np.abs(got - want) / want) <= 1e-5
    assert np.array_equal(bits(got), bits(gpu.fsoftmax(x)))                     # the same bits run to run
    X = torch.from_numpy(np.concatenate([[0], x]).astype(np.float32)).cuda()[1:]    # a base that is only 4-byte aligned
    out, ws = torch.empty(n, device="cuda"), torch.empty(1, dtype=torch.float64, device="cuda")
    lib, st = gpu.d.lib, torch.cuda.current_stream().cuda_stream
    lib.call("polar_b200_fsoftmax", X.data_ptr(), out.data_ptr(), n, ws.data_ptr(), 8, st)   # the smallest workspace it takes
    assert np.max(np.abs(out.cpu().numpy() - want) / want) <= 1e-5
    assert np.array_equal(bits(gpu.frelu(x)), bits(oracle.frelu(x)))


@pytest.mark.parametrize("n", [31, 8191, 8193, 32_769, 262_143, 262_144, 262_145, 262_149])
def test_softmax_around_the_limit_of_one_cluster(gpu, n):
    import torch
    x = np.random.default_rng(n).uniform(-4, 4, n).astype(np.float32)
    e = np.exp(x.astype(np.float64))
    want = e / e.sum()
    X = torch.from_numpy(x).cuda()
    st = torch.cuda.current_stream().cuda_stream
    gpu.d.lib.call("polar_b200_fsoftmax", X.data_ptr(), X.data_ptr(), n, None, 0, st)       # in place
    assert np.max(np.abs(X.cpu().numpy() - want) / want) <= 1e-5
