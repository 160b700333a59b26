"""The metal matrix of forest pairs without a diagonal in the r_par range (far
apart along the line of sight): nothing is added, and pairs beside them are."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_no_diagonal():
    from picca_gb300 import constants, dmat, metal, pairs, synthetic
    fs = synthetic.make_forests(30, 5, (150.0, 151.0), (0.0, 1.0), 2.1, 3.5, "uniform",
                                max_pixels=40)
    r = [fs.r_comov[a:b] for a, b in zip(fs.pix_offset[:-1], fs.pix_offset[1:])]
    apart = lambda f, g: max(r[f].min() - r[g].max(), r[g].min() - r[f].max())  # noqa: E731
    every = [(f, g) for f in range(fs.num) for g in range(f)]
    far = [p for p in every if apart(*p) > 30.0]
    near = [p for p in every if apart(*p) < 0.0]
    assert far and near
    eng = metal.MetalEngine()
    dev = pairs.DeviceForests(fs)
    params = pairs.make_params(0.0, 20.0, 200.0, 10, 10, 0.1)
    dparams = dmat.make_dmat_params(10, 10)
    one = metal.absorber_pixels(dev, constants.Cosmo(Om=0.3147, verbose=False), "LYA", 2.9)

    def run(chosen):
        first, second = (torch.tensor(c, dtype=torch.int32, device="cuda") for c in zip(*chosen))
        sums = eng.alloc_sums(params, dparams)
        eng.run_pass(params, dparams, 1.0, dev, None, one, one, first, second, len(chosen), sums)
        eng.engine.stats()
        return {k: v.cpu().numpy() for k, v in sums.items()}

    assert all(not v.any() for v in run(far).values())
    want = run(near)
    assert want["weights_dmat"].any()
    for key, v in run(far + near).items():
        assert np.all(np.abs(v - want[key]) <= 1e-12 * np.abs(want[key]).max()), key
