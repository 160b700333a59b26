"""The precision form near the limit of shared memory, where one warp's buffers
fit beside the histograms and the forest: many bins, long forests. The largest
forests that 227 KB of shared memory hold run; pair counts are the CPU oracle's.
And with few bins and short forests, where the arrays before the staged forest
are smaller than the reach of an idle lane."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(max_pixels, bins, xcf, num):
    from oracle import cpu as oracle
    from picca_gb300 import pairs, synthetic
    fs = synthetic.make_forests(num, 5, (150.0, 150.7), (0.0, 0.7), 2.4, 2.6, "uniform",
                                grid="lin", max_pixels=max_pixels)
    qs = synthetic.make_quasars(12, 6, (150.0, 150.7), (0.0, 0.7)) if xcf else None
    kwargs = dict(r_par_min=-200.0 if xcf else 0.0, r_par_max=200.0, r_trans_max=200.0,
                  num_bins_r_par=bins[0], num_bins_r_trans=bins[1], x_correlation=xcf)
    ang_max = synthetic.correlation_ang_max(200.0, float(fs.z.min()))
    p_or = oracle.make_params(**kwargs)
    if xcf:
        off, idx = oracle.neighbours(fs, qs, p_or, ang_max, 0, xcf=True)
        want = oracle.rows(fs, qs, p_or, off, idx, xcf=True)
    else:
        off, idx = oracle.neighbours(fs, fs, p_or, ang_max, auto_mode=1)
        want = oracle.rows(fs, fs, p_or, off, idx)
    got = pairs.correlate(fs, qs, pairs.make_params(ang_max=ang_max, **kwargs),
                          mode=pairs.MODE_FP32_GUARD, xcf=xcf)["raw"]
    assert int(np.diff(fs.pix_offset).max()) == max_pixels
    assert want[5].sum() > 0 and np.array_equal(got[5], want[5])


@pytest.mark.parametrize("max_pixels,bins", [(500, (80, 80)), (600, (80, 80)), (3, (3, 4)),
                                             (40, (1, 2)), (200, (2, 4))])
def test_auto(max_pixels, bins):
    _case(max_pixels, bins, False, 6)


@pytest.mark.parametrize("max_pixels,bins", [(600, (77, 80)), (574, (79, 80)), (3, (3, 4))])
def test_cross(max_pixels, bins):
    _case(max_pixels, bins, True, 6)
