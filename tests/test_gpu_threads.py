"""Two threads with a plan and a stream each, calling the same kernels with
forests of different lengths at once: every call is launched and gives what
it gives alone (counts equal, fits to the bit)."""

import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run_pairs(fs, repeat):
    from picca_gb300 import pairs, synthetic
    params = pairs.make_params(0.0, 100.0, 100.0, 20, 20,
                               synthetic.correlation_ang_max(100.0, float(fs.z.min())))
    return [pairs.correlate(fs, None, params, mode=pairs.MODE_FP64)["raw"][5]
            for _ in range(repeat)]


def _run_fit(raw, repeat):
    from picca_gb300 import continuum
    out = []
    for _ in range(repeat):
        eng = continuum.Dr16Gpu(raw.grid)
        out.append(continuum.fit_results_to_host(
            eng.fit(continuum.DeviceSpectra(raw, eng.device)))["zero_point"])
    return out


def _both(run, small, large, repeat=15):
    want = [run(x, 1)[0] for x in (small, large)]
    got, errors = [None, None], []

    def work(k, x):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got[k] = run(x, repeat)
        except Exception as exc:  # pylint: disable=broad-except
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(k, x)) for k, x in enumerate((small, large))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for g, w in zip(got, want):
        assert all(np.array_equal(x, w, equal_nan=True) for x in g)


def test_pairs():
    from picca_gb300 import synthetic
    make = lambda n: synthetic.make_forests(8, 5, (150.0, 150.5), (0.0, 0.5), 2.4, 2.6,  # noqa
                                            "uniform", grid="lin", max_pixels=n)
    _both(_run_pairs, make(40), make(600))


def test_fits():
    from picca_gb300 import synthetic_spectra
    make = lambda n: synthetic_spectra.make_raw_forests(n, 3)  # noqa: E731
    _both(_run_fit, make(20), make(3000))
