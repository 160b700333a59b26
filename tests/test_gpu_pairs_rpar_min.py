"""Auto-correlation with r_par_min several bins above 0: the band of diagonals
that is swept reaches r_par_max, not r_par_max - r_par_min. Pair counts are
the CPU oracle's in both arithmetic modes."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["MODE_FP64", "MODE_FP32_GUARD"])
@pytest.mark.parametrize("r_par_min,r_par_max,bins", [(8.0, 120.0, 50), (100.0, 200.0, 25)])
def test_counts(mode, r_par_min, r_par_max, bins):
    from oracle import cpu as oracle
    from picca_gb300 import pairs, synthetic
    fs = synthetic.make_forests(24, 5, (150.0, 152.0), (0.0, 2.0), 2.5, 3.5, "uniform")
    kwargs = dict(r_par_min=r_par_min, r_par_max=r_par_max, r_trans_max=200.0,
                  num_bins_r_par=bins, num_bins_r_trans=50)
    ang_max = synthetic.correlation_ang_max(200.0, 2.0)
    p_or = oracle.make_params(**kwargs)
    off, idx = oracle.neighbours(fs, fs, p_or, ang_max, auto_mode=1)
    ref = oracle.rows(fs, fs, p_or, off, idx)
    res = pairs.correlate(fs, None, pairs.make_params(ang_max=ang_max, **kwargs),
                          mode=getattr(pairs, mode))
    assert ref[5].sum() > 0
    assert np.array_equal(res["raw"][5], ref[5])
