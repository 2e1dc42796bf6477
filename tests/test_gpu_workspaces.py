"""Device memory that a k-NN call keeps in its context."""

import pytest

from culof_gb300 import _culof

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _kept(n, d, k):
    """Bytes that a fresh context holds after one k-NN call (its caller's buffers aside)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(n, d, generator=g, device="cuda")
    idx = torch.zeros((k, n), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((k, n), device="cuda")
    kd = torch.zeros(n, device="cuda")
    with _culof.Context() as ctx:  # the kernels' own memory, once per process
        ctx.knn_device(x.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.synchronize()
    free = torch.cuda.mem_get_info()[0]
    with _culof.Context() as ctx:
        ctx.knn_device(x.data_ptr(), n, d, k, False, idx.data_ptr(), d2.data_ptr(), kd.data_ptr())
        ctx.synchronize()
        return free - torch.cuda.mem_get_info()[0]


def test_no_lists_for_isolated_rows_that_cannot_leave(monkeypatch):
    n = 400_000
    monkeypatch.setenv("CULOF_ISO_ROWS", "1")
    on = _kept(n, 2, 8)
    monkeypatch.setenv("CULOF_ISO_ROWS", "0")
    off = _kept(n, 2, 8)
    # a list of 32 keys (and its row) for a quarter of the rows and more
    assert on - off > n // 4 * 32 * 8 - (4 << 20)


def test_no_seed_lists_without_a_seed():
    # the tensor path past 8 features starts from none: what it keeps does not
    # grow with k (the split of the columns is the same)
    n = 100_000
    assert abs(_kept(n, 24, 48) - _kept(n, 24, 8)) < 8 << 20
