"""The direct two-pass kernel at its dimension, list and row-count edges, and
the tensor path past 128 features, against the oracle bit for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof, synthetic

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

DIRECT = [
    # two points, one step and one more, one staged block and one more, the
    # rows per warp's limits, every padded dimension and list form
    (2, 1, 1), (65, 2, 64), (66, 3, 24), (512, 4, 25), (513, 5, 32), (2432, 6, 33), (2433, 8, 20), (4096, 9, 20),
    (1025, 12, 64), (4095, 16, 40), (7168, 4, 20), (7168, 16, 30),
]


def _knn(ctx, X, k):
    n, d = X.shape
    dx = torch.from_numpy(X).cuda()
    idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((k, n), device="cuda")
    kd = torch.zeros(n, device="cuda")
    ctx.knn_device(dx.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
    ctx.synchronize()
    return idx.cpu().numpy(), d2.cpu().numpy(), kd.cpu().numpy()


def _check(X, k, got):
    Xc, _, _ = oracle.center(X)
    o_idx, o_d2, o_kd = oracle.knn(Xc, k)
    np.testing.assert_array_equal(got[2].view(np.uint32), o_kd.view(np.uint32))
    np.testing.assert_array_equal(got[0], o_idx)
    np.testing.assert_array_equal(got[1].view(np.uint32), o_d2.view(np.uint32))


@pytest.mark.parametrize("dups", [0, 200])
@pytest.mark.parametrize("n,d,k", DIRECT)
def test_direct_bit_exact(n, d, k, dups):
    X = synthetic.clusters_with_outliers(n, d, seed=n + d)
    if dups and n > 600:
        X[5 : 5 + dups] = X[4]  # more equal keys than the gathered buffer holds
    with _culof.Context() as ctx:
        _check(X, k, _knn(ctx, X, k))


@pytest.mark.parametrize("n,d,k", [(2561, 129, 20), (3000, 192, 33), (3000, 193, 63), (2700, 256, 64), (9000, 200, 20)])
def test_tensor_path_past_128_features(n, d, k):
    X = synthetic.factor_model(n, d, seed=n + d)
    X[10:13] = X[9]
    with _culof.Context() as ctx:
        got = _knn(ctx, X, k)
        assert ctx.last_path() == _culof.PATH_TENSOR
    _check(X, k, got)


def test_forced_fused_paths_still_refuse_more_than_128_features():
    X = synthetic.factor_model(3000, 129, seed=1)
    with _culof.Context() as ctx:
        for path in (_culof.PATH_FAST, _culof.PATH_TENSOR):
            ctx.set_path(path)
            with pytest.raises(ValueError):
                ctx.lof(X, 10)


@pytest.mark.parametrize("n", [7169, 8193, 16385, 32769, 65536, 65537])
def test_spatial_order_sorts(n):
    # the one-launch sort's pairs per thread and its limit, through the small-d
    # path (every point is placed once: the k-NN graph is the oracle's)
    X = synthetic.clusters_with_outliers(n, 3, seed=n)
    with _culof.Context() as ctx:
        ctx.set_path(_culof.PATH_FAST)
        got = ctx.lof(X, 12)
    np.testing.assert_array_equal(got.view(np.uint32), oracle.lof(X, 12).view(np.uint32))
