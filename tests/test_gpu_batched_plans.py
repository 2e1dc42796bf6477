"""Batched LOF: every list form, padded width and kernel of the batched path,
values that are not finite, and plans that are refused."""

import numpy as np
import pytest

import oracle
from culof_gb300 import _culof, synthetic

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Batch:
    def __init__(self, problems, ks):
        self.ks = list(ks)
        self.d = problems[0].shape[1]
        self.off = np.zeros(len(problems) + 1, np.int64)
        self.off[1:] = np.cumsum([len(p) for p in problems])
        self.x = torch.from_numpy(np.concatenate(problems).astype(np.float32)).cuda()
        self.out = torch.zeros(int(self.off[-1]), device="cuda")

    def run(self, ctx, ks=None, normalize=False):
        ctx.lof_batched_device(self.off, self.ks if ks is None else ks, self.x.data_ptr(), self.d, normalize,
                               self.out.data_ptr())
        ctx.synchronize()
        s = self.out.cpu().numpy()
        return [s[self.off[i]:self.off[i + 1]] for i in range(len(self.ks))]


def _same(got, problem, k):
    np.testing.assert_array_equal(got.view(np.uint32), oracle.lof(problem, k).view(np.uint32))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("d", [1, 3, 16, 24])
def test_values_that_are_not_finite_stay_in_their_problem(d, bad):
    probs = [synthetic.clusters_with_outliers(n, d, seed=n) for n in (300, 900, 2000)]
    spoilt = [p.copy() for p in probs]
    spoilt[0][5, 0] = bad  # the first problem: nothing lies before its ranges
    spoilt[1][:, :] = bad
    with _culof.Context() as ctx:
        got = Batch(spoilt, [10, 30, 20]).run(ctx)
        _same(got[2], probs[2], 20)
        for g, p, k in zip(Batch(probs, [10, 30, 20]).run(ctx), probs, [10, 30, 20]):
            _same(g, p, k)


def test_a_refused_layout_is_refused_again():
    # after a valid batch, with the same buffers: neither its graph nor its
    # plan may answer for the layout that was refused
    probs = [synthetic.clusters_with_outliers(n, 4, seed=n) for n in (50, 60, 300)]
    ks = [5, 10, 20]
    with _culof.Context() as ctx:
        b = Batch(probs, ks)
        b.run(ctx)
        for bad in ([50, 10, 20], [5, 10, 49], [5, 0, 20]):
            for _ in range(2):
                b.out.fill_(-1.0)
                with pytest.raises(ValueError, match="k must satisfy"):
                    b.run(ctx, ks=bad)
                assert bool((b.out == -1.0).all())
        for _ in range(2):
            for got, p, k in zip(b.run(ctx), probs, ks):
                _same(got, p, k)
        assert ctx.batched_tuning()["ctas_per_sm"] > 0


@pytest.mark.parametrize("normalize", [False, True])
@pytest.mark.parametrize("d", [2, 4, 5, 8, 9, 12, 13, 16, 17, 32, 33])
def test_every_list_form_in_every_padded_width(d, normalize):
    # the lists' limits in one batch (groups of one launch each), sizes at the
    # tiles' and the window's edges, duplicates more than the gathered buffer holds
    sizes = (25, 64, 65, 128, 129, 640, 641, 900, 2000)
    ks = (24, 25, 32, 33, 48, 1, 24, 33, 20)
    probs = [synthetic.clusters_with_outliers(n, d, seed=n + d) for n in sizes]
    for p in probs:
        p[len(p) // 2:] = p[: len(p) - len(p) // 2] if len(p) < 200 else p[len(p) // 2:]
    probs[7][100:300] = probs[7][7]
    probs[8][::5] = probs[8][3]
    with _culof.Context() as ctx:
        for got, p, k in zip(Batch(probs, ks).run(ctx, normalize=normalize), probs, ks):
            want = oracle.lof(p, k, normalize)
            np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
