"""LOF scores from a caller's own densities, over the whole float range:
infinite, zero, subnormal and undefined values among them."""

import numpy as np
import pytest

from culof_gb300 import _culof

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [False, True])
@pytest.mark.parametrize("n,k", [(40, 1), (300, 20), (1000, 40)])
def test_scores_of_any_densities(n, k, rows):
    rng = np.random.default_rng(n + k)
    lrd = np.exp(rng.uniform(-100.0, 88.0, n)).astype(np.float32)
    odd = np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, 1e-45, 1.1754942e-38, 3.4028235e38, -2.5, 1.0], np.float32)
    lrd[:: max(1, n // 30)] = np.resize(odd, len(lrd[:: max(1, n // 30)]))
    idx = rng.integers(0, n, (k, n)).astype(np.int32)
    with np.errstate(all="ignore"):
        total = np.zeros(n)
        for t in range(k):  # the sum runs over the slots in order, in 64 bits
            total = total + lrd[idx[t]].astype(np.float64) / lrd.astype(np.float64)
        want = (total / k).astype(np.float32)
    assert np.isposinf(want).any() and np.isnan(want).any() and np.isfinite(want).any()
    di, dl = torch.from_numpy(idx).cuda(), torch.from_numpy(lrd).cuda()
    out = torch.zeros(n, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    if rows:
        listed = torch.arange(n - 1, -1, -1, dtype=torch.int32, device="cuda")
        _culof.compute_scores_rows(stream, di.data_ptr(), dl.data_ptr(), n, k, listed.data_ptr(), n, out.data_ptr())
    else:
        _culof.compute_scores(stream, di.data_ptr(), dl.data_ptr(), n, k, out.data_ptr())
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    np.testing.assert_array_equal(got[ok].view(np.uint32), want[ok].view(np.uint32))
