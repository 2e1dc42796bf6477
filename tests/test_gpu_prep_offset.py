"""Centring, the offset and the labels at the edges of their kernels' ranges,
against the oracle bit for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof, synthetic

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("normalize", [False, True])
@pytest.mark.parametrize("n,d", [(2, 1), (255, 3), (256, 200), (257, 8), (8192, 16), (8193, 16), (656, 200), (4100, 40)])
def test_centring_bit_exact(n, d, normalize):
    # one CTA per feature up to 8,192 rows and 131,072 values, the separate
    # kernels above; a constant, a tiny and a huge column take the widening
    # and rounding edges
    X = synthetic.clusters_with_outliers(n, d, seed=n + d)
    X[:, 0] *= np.float32(1e-30)
    if d > 2:
        X[:, 1] = np.float32(2.5)
        X[:, 2] *= np.float32(1e6)
    k = min(5, n - 1)
    with _culof.Context() as ctx:
        got = ctx.lof(X, k, normalize)
    np.testing.assert_array_equal(got.view(np.uint32), oracle.lof(X, k, normalize).view(np.uint32))


@pytest.mark.parametrize("c", ["auto", 0.001, 0.01, 0.37, 0.5])
@pytest.mark.parametrize("n", [1, 2, 1023, 8192, 8193, 200_001, 1 << 20, (1 << 20) + 1])
def test_offset_matches_numpy(n, c):
    rng = np.random.default_rng(n)
    nof = -(1.0 + 0.2 * np.abs(rng.standard_normal(n))).astype(np.float32)
    nof[:: max(1, n // 5)] = nof[0]  # ties
    t = torch.from_numpy(nof).cuda()
    off = torch.zeros((), dtype=torch.float64, device="cuda")
    with _culof.Context() as ctx:
        ctx.offset_device(t.data_ptr(), n, c, off.data_ptr())
        ctx.synchronize()
    expect = -1.5 if c == "auto" else float(np.percentile(nof, 100.0 * c))
    assert off.item() == expect


@pytest.mark.parametrize("c", ["auto", 0.02])
@pytest.mark.parametrize("n", [700, 9000, 30_000])
def test_labels_follow_the_offset(n, c):
    X = synthetic.clusters_with_outliers(n, 4, seed=n)
    with _culof.Context() as ctx:
        nof, labels, off = ctx.fit_predict(X, 10, False, c)
    np.testing.assert_array_equal(labels, np.where(nof < off, -1, 1))
