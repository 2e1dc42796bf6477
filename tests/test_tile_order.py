"""The order of the small-d sweep's row tiles is a permutation for any extents
(checked on the host), and inputs that are not finite come out of the sweep."""

import ctypes
import os
import subprocess

import numpy as np
import pytest
from conftest import ROOT

import oracle
from culof_gb300 import _culof, synthetic

RULE = r"""
#include "tile_order.cuh"
extern "C" void ranks(const uint32_t* bits, int m, int* out) {
    using namespace culof_gb300;
    for (int t = 0; t < m; ++t) {
        int r = 0;
        for (int i = 0; i < m; ++i) r += starts_before(extent_key(bits[i]), i, extent_key(bits[t]), t) ? 1 : 0;
        out[t] = r;
    }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "rule.cpp").write_text(RULE)
    so = str(d / "rule.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "culof_gb300", "csrc"),
                    str(d / "rule.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def ranks(extents):
        bits = np.ascontiguousarray(extents, np.float32).view(np.uint32)
        out = np.empty(len(bits), np.int32)
        lib.ranks(ctypes.c_void_p(bits.ctypes.data), len(bits), ctypes.c_void_p(out.ctypes.data))
        return out

    return ranks


def test_ranks_are_a_permutation(rule):
    rng = np.random.default_rng(0)
    nan, inf = np.float32(np.nan), np.float32(np.inf)
    neg_nan = np.uint32(0xFFC00001).view(np.float32)
    for e in ([nan] * 40, [inf] * 7, [0.0] * 9, [nan, 1.0, inf, neg_nan, 0.0, 1.0, inf, nan],
              rng.choice(np.array([nan, neg_nan, inf, 0.0, 1e-45, 3.0], np.float32), 300), rng.random(157)):
        got = rule(np.array(e, np.float32))
        np.testing.assert_array_equal(np.sort(got), np.arange(len(e)))
    # wider first, equal ones by number
    np.testing.assert_array_equal(rule(np.array([1.0, 4.0, 1.0, inf, nan], np.float32)), [3, 2, 4, 1, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["nan", "inf", "overflow"])
@pytest.mark.parametrize("n,d,k", [(9000, 3, 20), (20000, 8, 33)])
def test_inputs_that_are_not_finite_leave_the_sweep(n, d, k, kind):
    # no score is defined (the centring spreads what is not finite over the
    # feature); the call returns, with neighbours among the points, and the
    # context serves the next call
    torch = pytest.importorskip("torch")
    X = synthetic.clusters_with_outliers(n, d, seed=n)
    good = oracle.lof(X[:8000], k)
    Y = X.copy()
    if kind == "overflow":
        # less its mean the first part is infinite: whole tiles of equal infinities
        Y[: n // 16, 1] = 3.4e38
        Y[n // 16 :, 1] = -3.4e38
    else:
        Y[77, 1] = np.nan if kind == "nan" else np.inf
    dx, dy = torch.from_numpy(X[:8000]).cuda(), torch.from_numpy(Y).cuda()
    scores = torch.zeros(n, device="cuda")
    idx = torch.full((k, n), -7, dtype=torch.int32, device="cuda")
    d2, kd = torch.zeros((k, n), device="cuda"), torch.zeros(n, device="cuda")
    with _culof.Context() as ctx:
        ctx.knn_device(dy.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.lof_device(dy.data_ptr(), n, d, k, False, scores.data_ptr())
        ctx.synchronize()
        got = idx.cpu().numpy()
        assert got.min() >= 0 and got.max() < n
        ctx.lof_device(dx.data_ptr(), 8000, d, k, False, scores.data_ptr())
        ctx.synchronize()
    np.testing.assert_array_equal(scores[:8000].cpu().numpy().view(np.uint32), good.view(np.uint32))
