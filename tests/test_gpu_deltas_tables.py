"""The delta extraction with a stack that fits in shared memory and with one that
does not: the same points, and as many again beyond every pixel, give the same
bits; both are the nearest point's values (1e-14: a product and a quotient)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_long_stack():
    from picca_gb300 import continuum, synthetic_spectra
    raw = synthetic_spectra.make_raw_forests(40, 3, z_lo=2.4, z_hi=3.2)
    rng = np.random.default_rng(0)
    x = np.linspace(raw.log_lambda.min() - 0.01, raw.log_lambda.max() + 0.01, 10000)
    y = 1.0 + 0.1 * rng.normal(size=x.size)
    more = x[-1] + 1e-5 * np.arange(1, 10001)
    got = []
    for sx, sy in ((x, y), (np.concatenate([x, more]), np.concatenate([y, np.ones(more.size)]))):
        eng = continuum.Dr16Gpu(raw.grid)
        spectra = continuum.DeviceSpectra(raw, eng.device)
        fit = eng.fit(spectra)
        eng.stack_x, eng.stack_y, eng.force_stack_delta_to_zero = sx, sy, True
        delta, weights = eng.deltas(spectra, fit)
        got.append((delta.cpu().numpy(), weights.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    out = continuum.fit_results_to_host(fit)
    stack = y[np.searchsorted((x[1:] + x[:-1]) / 2, raw.log_lambda, "left")]
    use = got[0][1] > 0
    want = raw.flux[use] / (out["continuum"][use] * stack[use]) - 1
    assert use.any() and np.allclose(got[0][0][use], want, rtol=1e-14, atol=1e-14)
