"""The FP64 delta x quasar correlation (FP32 decisions, FP64 sums) where its
forms can go wrong: one quasar to more than a block of 4,096 neighbours, r_par
of both signs and a shifted range, redshift cuts, unsorted and zero-weight
pixels. Against the CPU oracle: pair counts are equal, the sums within 1e-12 of
the sum of their terms' magnitudes (a few hundred thousand FP64 additions in
another order)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["one", "few", "many", "shifted", "zcut", "unsorted"])
def test_rows(case):
    from oracle import cpu as oracle
    from picca_gb300 import pairs, synthetic
    side = 0.5 if case == "many" else 1.5
    fs = synthetic.make_forests(3 if case == "many" else 30, 5, (150.0, 150.0 + side),
                                (0.0, side), 2.4, 3.4, "uniform")
    qs = synthetic.make_quasars({"one": 1, "few": 33, "many": 9000}.get(case, 400), 6,
                                (150.0, 150.0 + side), (0.0, side))
    rng = np.random.default_rng(1)
    fs.weights[rng.random(len(fs.weights)) < 0.05] = 0.0
    if case == "unsorted":
        a, b = fs.pix_offset[3], fs.pix_offset[4]
        for name in ("r_comov", "dist_m", "z", "delta", "weights"):
            x = getattr(fs, name)
            x[a:b] = x[a:b][::-1].copy()
    cut = dict(z_min_pairs=2.5, z_max_pairs=2.9) if case == "zcut" else {}
    lo, hi, bins = (20.0, 120.0, 30) if case == "shifted" else (-200.0, 200.0, 100)
    kwargs = dict(r_par_min=lo, r_par_max=hi, r_trans_max=200.0, num_bins_r_par=bins,
                  num_bins_r_trans=50, **cut)
    ang_max = synthetic.correlation_ang_max(200.0, float(fs.z.min()))
    p_or = oracle.make_params(**kwargs)
    off, idx = oracle.neighbours(fs, qs, p_or, ang_max, auto_mode=0, xcf=True)
    ref = oracle.rows(fs, qs, p_or, off, idx, xcf=True)
    fs_abs = __import__("copy").copy(fs)
    fs_abs.delta = np.abs(fs.delta)
    ref_abs = oracle.rows(fs_abs, qs, p_or, off, idx, xcf=True)
    got = pairs.correlate(fs, qs, pairs.make_params(ang_max=ang_max, x_correlation=True, **kwargs),
                          mode=pairs.MODE_FP64, xcf=True)["raw"]
    assert case == "one" or ref[5].sum() > 0
    if case == "many":
        assert np.diff(off).max() > 4096
    assert np.array_equal(got[5], ref[5])
    for k in range(5):
        scale = np.abs(ref_abs[k]) if k != 2 else ref[0] * max(abs(lo), abs(hi))
        assert np.all(np.abs(got[k] - ref[k]) <= 1e-12 * scale + 1e-300), k
