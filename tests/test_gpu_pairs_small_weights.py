"""The precision form with weights whose products lie below the FP32 normal
range (1.2e-38): the counted pairs keep their weight. A product of two FP32
weights is off by at most 2^-150 there, so a bin's sum by 1.4e-45 a pair beside
the 2e-6 of the ordinary sums; the FP64 mode is the other side."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xcf", [False, True])
def test_weights(xcf, scale=1e-22):
    from picca_gb300 import pairs, synthetic
    fs = synthetic.make_forests(40, 5, (150.0, 151.0), (0.0, 1.0), 2.4, 3.4, "uniform")
    fs.weights = fs.weights * scale
    qs = synthetic.make_quasars(300, 6, (150.0, 151.0), (0.0, 1.0)) if xcf else None
    if xcf:
        qs.obj_weight = qs.obj_weight * scale
    params = pairs.make_params(-200.0 if xcf else 0.0, 200.0, 200.0, 50, 50,
                               synthetic.correlation_ang_max(200.0, float(fs.z.min())),
                               x_correlation=xcf)
    got = pairs.correlate(fs, qs, params, mode=pairs.MODE_FP32_GUARD, xcf=xcf)["raw"]
    want = pairs.correlate(fs, qs, params, mode=pairs.MODE_FP64, xcf=xcf)["raw"]
    assert 0 < want[0][want[5] > 0].min() < 1e-38
    assert np.array_equal(got[5], want[5])
    assert np.all(np.abs(got[0] - want[0]) <= 2e-6 * want[0] + 1.5e-45 * want[5])
