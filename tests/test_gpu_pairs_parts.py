"""The auto-correlation where a neighbour forest is cut into parts for the
warps: a handful of neighbours a forest, of 3 to 400 pixels. Pair counts are
the FP64 mode's, the sums within 2e-6 of it (the tolerance of
test_gpu_pairs)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_pixels", [3, 33, 131, 400])
@pytest.mark.parametrize("forests", [2, 5, 30])
def test_few(forests, max_pixels):
    from picca_gb300 import pairs, synthetic
    fs = synthetic.make_forests(forests, 3, (150.0, 150.6), (0.0, 0.6), 2.4, 2.6, "uniform",
                                max_pixels=max_pixels)
    params = pairs.make_params(0.0, 200.0, 200.0, 50, 50,
                               synthetic.correlation_ang_max(200.0, float(fs.z.min())))
    got = pairs.correlate(fs, None, params, mode=pairs.MODE_FP32_GUARD)["raw"]
    want = pairs.correlate(fs, None, params, mode=pairs.MODE_FP64)["raw"]
    assert want[5].sum() > 0
    assert np.array_equal(got[5], want[5])
    for k in (0, 2, 3, 4):
        assert np.all(np.abs(got[k] - want[k]) <= 2e-6 * np.abs(want[k]) + 1e-30), k
