"""The 1D correlation matrices of the Wick terms at the edges of the kernel's
32 x 32 tiles: forests of 1 to 97 pixels and a long one, distances on a bound of
the nearest-neighbour table, a pixel without a distance. Equal to the formula in
FP64, bit for bit (products in its order, an IEEE square root)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_matrices():
    from picca_gb300 import pairs, synthetic, wick
    lengths = [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 300]
    fs = synthetic.make_forests(len(lengths), 3, (150.0, 151.0), (0.0, 1.0), 2.4, 3.0, "uniform")
    rng = np.random.default_rng(2)
    for name in ("r_comov", "dist_m", "z", "delta", "weights", "log_lambda"):
        x, o = np.asarray(getattr(fs, name)), fs.pix_offset
        setattr(fs, name, np.concatenate([np.resize(x[o[f]:o[f + 1]], n)
                                          for f, n in enumerate(lengths)]))
    fs.pix_offset = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    fs.weights = rng.uniform(0.1, 9, fs.weights.size)
    # distances of whole and half steps of the table
    fs.log_lambda = np.log10(3600.0) + 1.5e-4 * rng.integers(0, 900, fs.weights.size)
    k = np.arange(600)
    ones = np.ones(k.size, dtype=np.int64)
    tables = wick.OneDTables({"LLMIN": float(np.log10(3600.0)), "DLL": 3e-4, "nv1d": ones,
                              "v1d": rng.uniform(0.1, 2, k.size), "nb1d": ones,
                              "c1d": rng.normal(size=k.size)})
    fs.log_lambda[5] = np.nan
    arena, offsets, _ = wick.WickEngine().xi_matrices(pairs.DeviceForests(fs, compact=False),
                                                      tables, np.arange(len(lengths)))
    arena, offsets = arena.cpu().numpy(), offsets.cpu().numpy()
    variance = tables.variance(fs.log_lambda)
    for f, n in enumerate(lengths):
        sl = slice(fs.pix_offset[f], fs.pix_offset[f + 1])
        ll, w, v = fs.log_lambda[sl], fs.weights[sl], variance[sl]
        d = np.abs(ll[None, :] - ll[:, None])
        d[np.isnan(d)] = -1.0
        xi = tables.xi_y[np.searchsorted(tables.xi_bounds, d, "left")]
        want = (np.outer(w, w) * xi) * np.sqrt(np.outer(v, v))
        np.fill_diagonal(want, 0.0)
        assert np.array_equal(arena[offsets[f]:offsets[f] + n * n].reshape(n, n), want), f
