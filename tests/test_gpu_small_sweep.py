"""The small-d k-NN kernel (d <= 8) at the edges of its tiles, windows, list
registers and segments, against the oracle bit for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof, synthetic

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = [
    # n, d, k: one tile, the window alone, one tile past it, a refinement
    # chunk and one point more, the last k of each list form and the first of
    # the next, every padded dimension, two rows per CTA size
    (129, 8, 20), (640, 3, 24), (641, 8, 25), (1024, 1, 32), (1025, 2, 33), (2049, 5, 64), (5000, 6, 20),
    (7001, 7, 32), (16385, 4, 33), (20000, 8, 1), (120001, 8, 20),
]


@pytest.mark.parametrize("iso", ["0", "1"])
@pytest.mark.parametrize("n,d,k", CASES)
def test_small_sweep_bit_exact(monkeypatch, n, d, k, iso):
    if iso == "1" and n > 100_000:
        pytest.skip("isolated rows are on by default at this size")
    monkeypatch.setenv("CULOF_ISO_ROWS", "1" if n > 100_000 else iso)
    monkeypatch.setenv("CULOF_PRUNE_LISTS", "0" if n % 2 else "1")  # odd n: short tile segments
    X = synthetic.clusters_with_outliers(n, d, seed=n + k)
    X[n // 2 : n // 2 + 7] = X[3]  # a few duplicates
    with _culof.Context() as ctx:
        ctx.set_path(_culof.PATH_FAST)
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


@pytest.mark.parametrize("n,d,k", [(8000, 1, 20), (9000, 3, 32), (17000, 8, 33)])
def test_ties_enter_by_index_only(n, d, k):
    # a few distinct points: most distances tie with the k-th
    rng = np.random.default_rng(n)
    X = np.round(rng.random((n, d)) * 2).astype(np.float32)
    with _culof.Context() as ctx:
        ctx.set_path(_culof.PATH_FAST)
        got = ctx.lof(X, k)
    np.testing.assert_array_equal(got.view(np.uint32), oracle.lof(X, k).view(np.uint32))
