"""Ties in the direct kernel: equal distances within and beyond the gathered
buffer, and points that are all equal, against the oracle bit for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _lattice(n, d, levels, seed):
    return np.random.default_rng(seed).integers(0, levels, (n, d)).astype(np.float32)


@pytest.mark.parametrize("levels", [1, 2, 5])
@pytest.mark.parametrize("n,d,k", [(70, 1, 20), (700, 1, 33), (2433, 2, 24), (3001, 3, 25), (4096, 16, 32), (6000, 8, 20),
                                   (7168, 5, 64)])
def test_ties_bit_exact(n, d, k, levels):
    # points on a lattice: most distances have many equals, a row's k-th among them
    X = _lattice(n, d, levels, n + d)
    dx = torch.from_numpy(X).cuda()
    idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((k, n), device="cuda")
    kd = torch.zeros(n, device="cuda")
    with _culof.Context() as ctx:
        before = _culof.kernel_launch_count()
        ctx.knn_device(dx.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.synchronize()
        assert _culof.kernel_launch_count() - before == 2  # the centring and the direct kernel
    Xc, _, _ = oracle.center(X)
    o_idx, o_d2, o_kd = oracle.knn(Xc, k)
    np.testing.assert_array_equal(kd.cpu().numpy().view(np.uint32), o_kd.view(np.uint32))
    np.testing.assert_array_equal(idx.cpu().numpy(), o_idx)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), o_d2.view(np.uint32))


@pytest.mark.parametrize("n,d,k", [(7168, 8, 20), (7168, 8, 64), (7168, 16, 49), (6144, 12, 20), (4096, 16, 48)])
def test_auto_reaches_the_direct_kernel(n, d, k):
    # at the far end of each of its ranges; the launches tell it from the other
    # paths, which give the same bits
    X = _lattice(n, d, 1000, n + k)
    dx = torch.from_numpy(X).cuda()
    idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((k, n), device="cuda")
    kd = torch.zeros(n, device="cuda")
    with _culof.Context() as ctx:
        before = _culof.kernel_launch_count()
        ctx.knn_device(dx.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.synchronize()
        assert _culof.kernel_launch_count() - before == 2  # the centring and the direct kernel
    Xc, _, _ = oracle.center(X)
    o_idx, _, o_kd = oracle.knn(Xc, k)
    np.testing.assert_array_equal(kd.cpu().numpy().view(np.uint32), o_kd.view(np.uint32))
    np.testing.assert_array_equal(idx.cpu().numpy(), o_idx)
