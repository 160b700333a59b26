"""What the FP32 decisions of the FP64 kernels cannot decide is decided in FP64:
bins so narrow that FP32 does not resolve them (distances moved off the common
grid, 6e4 to 1e5 bins per Mpc/h), redshifts so large that FP32 sums of two are coarser than
the ordinary band of the z cuts, and distances that are not numbers. The
other side is the loop with all geometry in FP64 (equal pair counts), and the
NumPy oracle for the metal matrix (1e-10, as in its other tests)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _counts(fs, qs, kwargs):
    from picca_gb300 import pairs, synthetic
    params = pairs.make_params(ang_max=synthetic.correlation_ang_max(200.0, 2.4), **kwargs)
    plain = pairs.PairEngine()
    plain.plan.set_all_fp64(True)
    want, got = (pairs.correlate(fs, qs, params, mode=pairs.MODE_FP64, xcf=qs is not None,
                                 engine=e)["raw"][5] for e in (plain, None))
    assert want.sum() > 0 and np.array_equal(got, want)


def _forests(num=20):
    from picca_gb300 import synthetic
    return synthetic.make_forests(num, 5, (150.0, 150.8), (0.0, 0.8), 2.5, 3.4, "uniform")


@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("bins", [(3000, 2, 0.05), (5000, 1, 0.05), (60000, 1, 200.0)])
def test_narrow_bins(bins, signed):
    fs = _forests()
    rng = np.random.default_rng(1)
    fs.r_comov = fs.r_comov + rng.uniform(0.0, 0.1, fs.r_comov.size)
    _counts(fs, None, dict(r_par_min=-bins[2] if signed else 0.0, r_par_max=bins[2],
                           r_trans_max=200.0, num_bins_r_par=bins[0], num_bins_r_trans=bins[1],
                           x_correlation=signed))


def test_narrow_bins_trans():
    _counts(_forests(8), None, dict(r_par_min=0.0, r_par_max=50.0, r_trans_max=200.0,
                                    num_bins_r_par=2, num_bins_r_trans=60000))


@pytest.mark.parametrize("bins", [(3000, 2, 1.0), (5000, 1, 1.0)])
def test_narrow_bins_cross(bins):
    from picca_gb300 import synthetic
    qs = synthetic.make_quasars(400, 6, (150.0, 150.8), (0.0, 0.8))
    _counts(_forests(), qs, dict(r_par_min=-bins[2], r_par_max=bins[2], r_trans_max=200.0,
                                 num_bins_r_par=bins[0], num_bins_r_trans=bins[1],
                                 x_correlation=True))


@pytest.mark.parametrize("cut", ["z_min_pairs", "z_max_pairs"])
@pytest.mark.parametrize("xcf", [False, True])
def test_large_redshifts(cut, xcf):
    from picca_gb300 import synthetic
    fs = _forests()
    qs = synthetic.make_quasars(400, 6, (150.0, 150.8), (0.0, 0.8)) if xcf else None
    fs.z = fs.z * 3000.0
    if xcf:
        qs.z_qso = qs.z_qso * 3000.0
    limit = 0.5 * (float(np.median(fs.z)) + float(np.median(qs.z_qso if xcf else fs.z)))
    _counts(fs, qs, {**dict(r_par_min=-200.0 if xcf else 0.0, r_par_max=200.0, r_trans_max=200.0,
                            num_bins_r_par=50, num_bins_r_trans=50, x_correlation=xcf),
                     cut: limit})


@pytest.mark.parametrize("xcf", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_not_numbers(xcf, value):
    from picca_gb300 import synthetic
    fs = _forests()
    qs = synthetic.make_quasars(400, 6, (150.0, 150.8), (0.0, 0.8)) if xcf else None
    inner = np.concatenate([np.arange(a + 3, b - 3, 17) for a, b in zip(fs.pix_offset[:-1],
                                                                        fs.pix_offset[1:])])
    fs.r_comov = fs.r_comov.copy()
    fs.r_comov[inner[::2]] = value
    _counts(fs, qs, dict(r_par_min=-200.0 if xcf else 0.0, r_par_max=200.0, r_trans_max=200.0,
                         num_bins_r_par=50, num_bins_r_trans=50, x_correlation=xcf))


def test_narrow_bins_metal():
    from oracle import cpu
    from oracle import metal_dmat as omd
    from picca_gb300 import constants, dmat, metal, pairs
    torch = pytest.importorskip("torch")
    fs = _forests(7)
    fs.r_comov = fs.r_comov + np.random.default_rng(1).uniform(0.0, 0.1, fs.r_comov.size)
    cosmo = constants.Cosmo(Om=0.3147, verbose=False)
    p = omd.MetalParams(0.0, 0.05, 200.0, 3000, 1, coef_binning_model=1, z_ref=2.25,
                        alpha_abs={"LYA": 2.9})
    out = omd.new_outputs(p)
    po = fs.pix_offset
    pairs_ = [(f, g) for f in range(fs.num) for g in range(f)]
    for f, g in pairs_:
        ang = cpu.lib().oracle_angle(fs.x_cart[f], fs.y_cart[f], fs.z_cart[f], fs.ra[f],
                                     fs.dec[f], fs.cos_dec[f], fs.x_cart[g], fs.y_cart[g],
                                     fs.z_cart[g], fs.ra[g], fs.dec[g])
        side = lambda h: (fs.log_lambda[po[h]:po[h + 1]], fs.r_comov[po[h]:po[h + 1]],  # noqa
                          fs.dist_m[po[h]:po[h + 1]], fs.weights[po[h]:po[h + 1]], fs.z_qso[h])
        omd.forest_pair(p, cosmo, side(f), side(g), ang, False, "LYA", "LYA", False, out)
    eng = metal.MetalEngine()
    dev = pairs.DeviceForests(fs)
    params = pairs.make_params(0.0, 0.05, 200.0, 3000, 1, 0.1)
    dparams = dmat.make_dmat_params(3000, 1, coef_binning_model=1)
    first, second = (torch.tensor(c, dtype=torch.int32, device="cuda") for c in zip(*pairs_))
    sums = eng.alloc_sums(params, dparams)
    one = metal.absorber_pixels(dev, cosmo, "LYA", 2.9)
    eng.run_pass(params, dparams, (1 + 2.25) ** (2 * 2.9 - 2), dev, None, one, one, first, second,
                 len(pairs_), sums)
    eng.engine.stats()
    assert out["weights_dmat"].sum() > 0
    for key, v in sums.items():
        assert np.all(np.abs(v.cpu().numpy() - out[key]) <= 1e-10 * np.abs(out[key]).max()), key
