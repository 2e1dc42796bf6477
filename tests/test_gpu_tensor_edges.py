"""The tensor path at the edges of its bounds scan, lists and splits, against
the oracle bit for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof, synthetic

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [
    # one tile, two tiles, a last tile of one point; k at the list registers'
    # and the group minima's limits (63 + the row itself fill the 64 groups; the
    # scan has two halves above 55); d at the operand boxes' limits
    (100, 16, 20), (129, 42, 32), (256, 43, 33), (1000, 64, 63), (1000, 65, 64), (3001, 128, 50), (20000, 24, 1),
]


@pytest.mark.parametrize("splits", ["1", "3", "4"])
@pytest.mark.parametrize("n,d,k", CASES)
def test_tensor_path_bit_exact(monkeypatch, n, d, k, splits):
    monkeypatch.setenv("CULOF_SPLITS", splits)
    X = synthetic.factor_model(n, d, seed=n + k)
    X[n // 2 : n // 2 + min(5, n // 4)] = X[1]  # a few duplicates
    with _culof.Context() as ctx:
        ctx.set_path(_culof.PATH_TENSOR)
        dx = torch.from_numpy(X).cuda()
        idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
        d2 = torch.zeros((k, n), device="cuda")
        kd = torch.zeros(n, device="cuda")
        ctx.knn_device(dx.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.synchronize()
    Xc, _, _ = oracle.center(X)
    o_idx, o_d2, o_kd = oracle.knn(Xc, k)
    np.testing.assert_array_equal(kd.cpu().numpy().view(np.uint32), o_kd.view(np.uint32))
    np.testing.assert_array_equal(idx.cpu().numpy(), o_idx)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), o_d2.view(np.uint32))


def _check_tensor(X, k, path):
    n, d = X.shape
    with _culof.Context() as ctx:
        ctx.set_path(path)
        dx = torch.from_numpy(X).cuda()
        idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
        d2 = torch.zeros((k, n), device="cuda")
        kd = torch.zeros(n, device="cuda")
        ctx.knn_device(dx.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.synchronize()
        assert ctx.last_path() == _culof.PATH_TENSOR
    Xc, _, _ = oracle.center(X)
    o_idx, o_d2, o_kd = oracle.knn(Xc, k)
    np.testing.assert_array_equal(kd.cpu().numpy().view(np.uint32), o_kd.view(np.uint32))
    np.testing.assert_array_equal(idx.cpu().numpy(), o_idx)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), o_d2.view(np.uint32))


@pytest.mark.parametrize("n,d,k", [(2600, 24, 56), (4200, 40, 64), (4100, 43, 20), (5000, 64, 33), (4300, 100, 64),
                                   (4200, 126, 57), (2600, 200, 20), (2700, 256, 64)])
def test_lists_without_room_turn_exact(n, d, k):
    # clusters far from the origin: a wide filter margin, most rows rescore
    # their candidates exactly, 32 pending pairs at a time
    X = synthetic.clusters_with_outliers(n, d, seed=n + k)
    X[: n // 2] += np.float32(40.0)
    X[20:30] = X[19]
    _check_tensor(X, k, _culof.PATH_TENSOR if d <= 128 else _culof.PATH_AUTO)
