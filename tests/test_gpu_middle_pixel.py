"""A forest whose middle pixel, the one that the FP32 distances are taken
relative to, has no finite comoving distance: its other pixels pair as in the
loop with all geometry in FP64 (equal counts)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("xcf", [False, True])
def test_counts(xcf, value):
    from test_gpu_exact_decisions import _counts, _forests
    from picca_gb300 import synthetic
    fs = _forests()
    qs = synthetic.make_quasars(400, 6, (150.0, 150.8), (0.0, 0.8)) if xcf else None
    middle = (fs.pix_offset[:-1] + np.diff(fs.pix_offset) // 2)[::3]
    fs.r_comov = fs.r_comov.copy()
    fs.r_comov[middle] = value
    _counts(fs, qs, dict(r_par_min=-200.0 if xcf else 0.0, r_par_max=200.0, r_trans_max=200.0,
                         num_bins_r_par=50, num_bins_r_trans=50, x_correlation=xcf))
