"""The delta x quasar correlation for numbers of quasars around its groups of
32, fewer and more groups than warps: pair counts are the FP64 kernel's, the
other sums within 2e-6 of it (FP32 pair terms, the tolerance of
test_gpu_pairs)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quasars", [1, 31, 33, 150, 300, 1000])
def test_groups(quasars):
    from picca_gb300 import pairs, synthetic
    fs = synthetic.make_forests(40, 5, (150.0, 151.0), (0.0, 1.0), 2.4, 3.4, "uniform")
    qs = synthetic.make_quasars(quasars, 6, (150.0, 151.0), (0.0, 1.0))
    params = pairs.make_params(-200.0, 200.0, 200.0, 100, 50,
                               synthetic.correlation_ang_max(200.0, float(fs.z.min())),
                               x_correlation=True)
    got = pairs.correlate(fs, qs, params, mode=pairs.MODE_FP32_GUARD, xcf=True)["raw"]
    want = pairs.correlate(fs, qs, params, mode=pairs.MODE_FP64, xcf=True)["raw"]
    assert quasars < 31 or want[5].sum() > 0
    assert np.array_equal(got[5], want[5])
    for k in (0, 2, 3, 4):
        scale = np.abs(want[k]) if k != 2 else np.abs(want[0]) * 200.0
        assert np.all(np.abs(got[k] - want[k]) <= 2e-6 * scale + 1e-30), k
