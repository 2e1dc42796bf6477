"""Rows that leave the tensor path for the pass over all points: data on which
the f16 filter decides little or nothing, against the oracle bit for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof, synthetic

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _cauchy(n, d, seed):  # the far points set the filter's scale
    return np.random.default_rng(seed).standard_cauchy((n, d)).astype(np.float32)


def _equal(n, d, seed):
    return np.full((n, d), 1.5, np.float32)


def _lattice(n, d, seed):  # two points: every distance ties with thousands
    return np.random.default_rng(seed).integers(0, 2, (n, 1)).astype(np.float32) * np.ones((1, d), np.float32)


def _some_equal(n, d, seed):  # a few rows leave: their columns are split
    X = synthetic.factor_model(n, d, seed=seed)
    X[n // 3 : n // 3 + 300] = X[1]
    return X


def _far(n, d, seed):  # the filter is off: all rows leave
    X = synthetic.factor_model(n, d, seed=seed)
    return (X * np.float32(1e19)).astype(np.float32)


DATA = {"cauchy": _cauchy, "equal": _equal, "lattice": _lattice, "some_equal": _some_equal, "far": _far}


def _check(X, k, path=_culof.PATH_TENSOR):
    n, d = X.shape
    with _culof.Context() as ctx:
        ctx.set_path(path)
        dx = torch.from_numpy(X).cuda()
        for _ in range(2):  # (the second call finds the first one's lists)
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


@pytest.mark.parametrize("data", DATA)
@pytest.mark.parametrize("n,d,k", [
    # the staged features' and columns' edges, the list forms' (24 / 25, 32 / 33, 64), one
    # share of the columns and several, a last tile of one column
    (400, 9, 24), (1025, 16, 25), (2561, 31, 32), (3000, 32, 20), (2999, 33, 33), (2700, 63, 64), (3001, 128, 48),
    (4000, 5, 20),
])
def test_rows_that_leave(n, d, k, data):
    _check(DATA[data](n, d, n + d), k)


@pytest.mark.parametrize("data", DATA)
@pytest.mark.parametrize("n,d,k", [(2561, 129, 20), (3000, 200, 33), (2700, 255, 64), (2600, 256, 24)])
def test_rows_that_leave_past_128_features(n, d, k, data):
    _check(DATA[data](n, d, n + d), k, _culof.PATH_AUTO)


@pytest.mark.parametrize("shards", [2, 3])
def test_shards_keep_their_rows(shards):
    n, d, k = 3000, 24, 20
    X = _cauchy(n, d, 5)
    dx = torch.from_numpy(X).cuda()
    idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((k, n), device="cuda")
    kd = torch.zeros(n, device="cuda")
    rows = torch.zeros(n, dtype=torch.int32, device="cuda")
    seen = np.zeros(n, np.int64)
    with _culof.Context() as ctx:
        ctx.set_path(_culof.PATH_TENSOR)
        for s in range(shards):
            m = ctx.knn_shard_device(dx.data_ptr(), n, d, k, False, s, shards, idx.data_ptr(), d2.data_ptr(),
                                     kd.data_ptr(), rows.data_ptr())
            ctx.synchronize()
            seen[rows[:m].cpu().numpy()] += 1
    assert (seen == 1).all()
    o_idx, _, o_kd = oracle.knn(oracle.center(X)[0], k)
    np.testing.assert_array_equal(idx.cpu().numpy(), o_idx)
    np.testing.assert_array_equal(kd.cpu().numpy().view(np.uint32), o_kd.view(np.uint32))
