"""The pair kernels that decide bins in FP32 against the loop with all geometry in
FP64 (pg_plan_set_all_fp64), which shares no decision with them: few forests,
whose neighbours are cut into parts, and quasars around the groups of 32. Pair
counts are equal, also to the CPU oracle's; sums within 2e-6 (precision form)
and 1e-12 (FP64 sums in another order, of the sum of the terms' magnitudes)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(fs, qs, kwargs):
    from oracle import cpu as oracle
    from picca_gb300 import pairs, synthetic
    xcf = qs is not None
    ang_max = synthetic.correlation_ang_max(200.0, float(fs.z.min()))
    params = pairs.make_params(ang_max=ang_max, **kwargs)
    plain = pairs.PairEngine()
    plain.plan.set_all_fp64(True)
    run = lambda mode, engine=None: pairs.correlate(fs, qs, params, mode=mode, xcf=xcf,  # noqa
                                                    engine=engine)["raw"]
    want, fp64 = run(pairs.MODE_FP64, plain), run(pairs.MODE_FP64)
    guard = run(pairs.MODE_FP32_GUARD)
    off, idx = oracle.neighbours(fs, qs if xcf else fs, oracle.make_params(**kwargs), ang_max,
                                 int(not xcf), xcf=xcf)
    counts = oracle.rows(fs, qs if xcf else fs, oracle.make_params(**kwargs), off, idx, xcf=xcf)[5]
    for got in (want, fp64, guard):
        assert np.array_equal(got[5], counts)
    scale = [want[0], None, want[0] * 200.0, want[0] * 200.0, want[4]]
    for k in (0, 2, 3, 4):
        assert np.all(np.abs(fp64[k] - want[k]) <= 1e-12 * scale[k]), k
        assert np.all(np.abs(guard[k] - want[k]) <= 2e-6 * scale[k]), k
    return counts.sum()


@pytest.mark.parametrize("max_pixels", [3, 33, 131, 400])
@pytest.mark.parametrize("forests", [2, 30])
def test_few(forests, max_pixels):
    from picca_gb300 import synthetic
    fs = synthetic.make_forests(forests, 3, (150.0, 150.6), (0.0, 0.6), 2.4, 2.6, "uniform",
                                max_pixels=max_pixels)
    assert _compare(fs, None, dict(r_par_min=0.0, r_par_max=200.0, r_trans_max=200.0,
                                   num_bins_r_par=50, num_bins_r_trans=50)) > 0


@pytest.mark.parametrize("quasars", [31, 33, 1000])
def test_groups(quasars):
    from picca_gb300 import synthetic
    fs = synthetic.make_forests(40, 5, (150.0, 151.0), (0.0, 1.0), 2.4, 3.4, "uniform")
    qs = synthetic.make_quasars(quasars, 6, (150.0, 151.0), (0.0, 1.0))
    assert _compare(fs, qs, dict(r_par_min=-200.0, r_par_max=200.0, r_trans_max=200.0,
                                 num_bins_r_par=100, num_bins_r_trans=50,
                                 x_correlation=True)) > 0


@pytest.mark.parametrize("forests,r_max,bins", [(30, 20.0, 10), (3, 20.0, 10), (30, 80.0, 20),
                                                (2, 2.0, 1), (120, 60.0, 15)])
def test_few_short_range(forests, r_max, bins):
    """Few diagonals within r_par_max: fewer parts a neighbour, down to one."""
    from picca_gb300 import synthetic
    fs = synthetic.make_forests(forests, 3, (150.0, 150.4), (0.0, 0.4), 2.4, 2.6, "uniform")
    assert _compare(fs, None, dict(r_par_min=0.0, r_par_max=r_max, r_trans_max=200.0,
                                   num_bins_r_par=bins, num_bins_r_trans=50)) > 0
