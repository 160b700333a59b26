"""Host side of the continuum loop: the splines of several functions solved
together have the bits of one solved alone (the FP64 fit's step count follows
the last bits of the model), and the grouped faces of the box least squares
give the minimiser of a face-by-face search, rank-deficient bins included."""

import numpy as np
import pytest

from picca_gb300 import continuum


@pytest.mark.parametrize("n", [4, 5, 6, 20, 33])
def test_splines_solved_together_bitwise(n):
    rng = np.random.default_rng(n)
    for even in (True, False):
        x = np.linspace(3.55, 3.74, n) if even else np.sort(rng.uniform(3.5, 3.8, n))
        ys = [np.ones(n), rng.normal(size=n), 1e-7 * rng.normal(size=n)]
        breaks, coefs = continuum.cubic_ppolys(x, ys)
        for y, coef in zip(ys, coefs):
            b, c = continuum.cubic_ppoly(x, y)
            assert np.array_equal(breaks, b) and np.array_equal(coef, c)


def test_box_least_squares_is_the_best_face():
    rng = np.random.default_rng(3)
    lo, hi = np.array([0.5, 0.0, 0.0]), np.array([1.5, 0.3, np.inf])
    for trial in range(40):
        a = rng.normal(size=(6, 30, 3)) * np.array([1, 1, 10.0 ** rng.uniform(-2, 2)])
        y = rng.normal(size=(6, 30))
        a[4] = 0.0      # no pixel
        a[5, 1:] = 0.0  # one pixel
        gram, mty = np.einsum("bij,bik->bjk", a, a), np.einsum("bij,bi->bj", a, y)
        x, ok = continuum.box_lsq3_gram(gram, mty, (0.5, 1.5), (0.0, 0.3))
        assert list(ok) == [True] * 4 + [False] * 2
        for b in range(4):
            assert np.all(x[b] >= lo - 1e-15) and np.all(x[b] <= hi + 1e-15)
            cost = np.sum((a[b] @ x[b] - y[b]) ** 2)
            # no feasible random point, near or far, is better
            pts = np.concatenate([x[b] + rng.normal(size=(200, 3)) * s for s in (1e-4, 0.1, 1.0)])
            pts = np.clip(pts, lo, hi)
            assert cost <= np.min(np.sum((pts @ a[b].T - y[b]) ** 2, axis=1)) + 1e-9
