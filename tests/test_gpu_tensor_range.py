"""The tensor path on values whose squared norms overflow float32, or nearly
do, while the distances within a cluster are ordinary, against the oracle bit
for bit."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _far_clusters(n, d, centre, spread, seed):
    rng = np.random.default_rng(seed)
    centres = rng.uniform(-centre, centre, (5, d))
    return (centres[rng.integers(0, 5, n)] + spread * rng.standard_normal((n, d))).astype(np.float32)


@pytest.mark.parametrize("centre,spread", [(5e19, 1e15), (1.5e18, 1e14), (6e17, 1e13), (1e17, 1e13)])
@pytest.mark.parametrize("n,d,k,path", [(3000, 32, 20, _culof.PATH_TENSOR), (5000, 100, 33, _culof.PATH_AUTO),
                                        (4500, 200, 20, _culof.PATH_AUTO)])
def test_norms_at_the_end_of_the_float_range(n, d, k, path, centre, spread):
    X = _far_clusters(n, d, centre, spread, n + d)
    want = oracle.lof(X, k)
    assert np.isfinite(want).all()
    with _culof.Context() as ctx:
        ctx.set_path(path)
        got = ctx.lof(X, k)
        assert ctx.last_path() == _culof.PATH_TENSOR
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("centre,spread", [(5e19, 1e15), (1.5e18, 1e14), (1e17, 1e13)])
@pytest.mark.parametrize("n,d,k", [(129, 9, 9), (1500, 16, 24), (2000, 33, 48), (1000, 128, 64)])
def test_fp32_filter_at_the_end_of_the_float_range(n, d, k, centre, spread):
    # the wide FP32 sweep's filter overflows the same way
    X = _far_clusters(n, d, centre, spread, n + d)
    want = oracle.lof(X, k)
    assert np.isfinite(want).all()
    with _culof.Context() as ctx:
        ctx.set_path(_culof.PATH_FAST)
        got = ctx.lof(X, k)
    np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
