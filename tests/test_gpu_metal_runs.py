"""Metal matrices by diagonal sweeps (pg_metal.cu) against the NumPy oracle
where the sweep can go wrong: forests around a warp's 32 diagonals, single
pixels, pixels out of order, absorber pixels dropped at the red end, model
bins finer than the data bins. The sums are the same FP64 terms in another
order (1e-10 of each output's largest value, as in the other metal tests)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[1], [1, 33, 2], [31, 32, 65], [207, 128, 96]])
@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("abs1,abs2,coef", [("LYA", "SiIII(1207)", 1), ("SiII(1190)", "LYA", 2)])
def test_against_oracle(lengths, shuffle, abs1, abs2, coef):
    from oracle import cpu
    from oracle import metal_dmat as omd
    from picca_gb300 import constants, dmat, metal, pairs, synthetic
    from picca_gb300.forests import PIXEL_FIELDS
    num = 7
    rng = np.random.default_rng(5)
    fs = synthetic.make_forests(num, 9, (150.0, 151.0), (0.0, 1.0), 2.6, 3.2, "uniform")
    npix = np.diff(fs.pix_offset)
    want_n = np.minimum(np.resize(lengths, num), npix)
    # the red end of each forest, where SiII(1190) pixels are dropped
    keep = np.concatenate([np.arange(o + n - k, o + n) if not shuffle else
                           rng.permutation(np.arange(o + n - k, o + n))
                           for o, n, k in zip(fs.pix_offset, npix, want_n)])
    for key in PIXEL_FIELDS:
        setattr(fs, key, getattr(fs, key)[keep])
    fs.pix_offset = np.concatenate([[0], np.cumsum(want_n)]).astype(np.int64)
    cosmo = constants.Cosmo(Om=0.3147, verbose=False)
    alpha = {"LYA": 2.9, "SiIII(1207)": 1.0, "SiII(1190)": 1.1}
    p = omd.MetalParams(0.0, 200.0, 200.0, 50, 40, coef_binning_model=coef, z_ref=2.25,
                        alpha_abs=alpha)
    out = omd.new_outputs(p)
    po = fs.pix_offset
    pairs_ = [(f, g) for f in range(num) for g in range(f)]
    for f, g in pairs_:
        ang = cpu.lib().oracle_angle(fs.x_cart[f], fs.y_cart[f], fs.z_cart[f], fs.ra[f],
                                     fs.dec[f], fs.cos_dec[f], fs.x_cart[g], fs.y_cart[g],
                                     fs.z_cart[g], fs.ra[g], fs.dec[g])
        side = lambda h: (fs.log_lambda[po[h]:po[h + 1]], fs.r_comov[po[h]:po[h + 1]],  # noqa
                          fs.dist_m[po[h]:po[h + 1]], fs.weights[po[h]:po[h + 1]], fs.z_qso[h])
        omd.forest_pair(p, cosmo, side(f), side(g), ang, False, abs1, abs2, False, out)
    torch = pytest.importorskip("torch")
    eng = metal.MetalEngine()
    dev = pairs.DeviceForests(fs)
    params = pairs.make_params(0.0, 200.0, 200.0, 50, 40, 0.1)
    dparams = dmat.make_dmat_params(50, 40, coef_binning_model=coef)
    first, second = (torch.tensor(c, dtype=torch.int32, device="cuda") for c in zip(*pairs_))
    sums = eng.alloc_sums(params, dparams)
    eng.run_pass(params, dparams, (1 + 2.25) ** (alpha[abs1] + alpha[abs2] - 2), dev, None,
                 metal.absorber_pixels(dev, cosmo, abs1, alpha[abs1]),
                 metal.absorber_pixels(dev, cosmo, abs2, alpha[abs2]), first, second,
                 len(pairs_), sums)
    eng.engine.stats()
    for key, v in sums.items():
        assert np.all(np.abs(v.cpu().numpy() - out[key]) <= 1e-10 * np.abs(out[key]).max()), key
