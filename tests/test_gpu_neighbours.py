"""Neighbour lists against the CPU oracle at the sizes where the warp-per-
query search can go wrong: query counts around a warp's four queries and a
CTA's 32, candidate counts around a warp and around the staged tile, objects
at the same position, equal thingids and thingids that agree in their low
half, and angles for which the FP32 tests are switched off."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(r_par_min=0.0, r_par_max=200.0, r_trans_max=200.0, num_bins_r_par=50,
          num_bins_r_trans=50)


def _forests(num, seed):
    from picca_gb300 import synthetic
    fs = synthetic.make_forests(num, seed, (150.0, 153.0), (0.0, 3.0), 2.1, 3.5, "uniform")
    if num > 8:
        # repeated positions (equal RA: neither is the other's neighbour in
        # the auto-correlation) and thingids equal in their low 32 bits
        for k in range(0, num - 1, 7):
            for key in ("ra", "dec", "x_cart", "y_cart", "z_cart", "cos_dec"):
                getattr(fs, key)[k + 1] = getattr(fs, key)[k]
        fs.thingid[::5] = fs.thingid[0] + (np.arange(len(fs.thingid[::5])) << 32)
        fs.thingid[3::11] = fs.thingid[2]
    return fs


def _check(fs, other, ang_max, auto, xcf, **kw):
    from oracle import cpu as oracle
    from picca_gb300 import pairs
    kwargs = dict(KW, **kw)
    p_or = oracle.make_params(**kwargs)
    off, idx = oracle.neighbours(fs, other if other is not None else fs, p_or, ang_max,
                                 auto_mode=int(auto), xcf=xcf)
    engine = pairs.PairEngine()
    params = pairs.make_params(ang_max=ang_max, **kwargs)
    d1 = pairs.DeviceForests(fs)
    d2 = pairs.DeviceForests(other) if other is not None else None
    for grouped in (True, False):
        o, i, total = engine.neighbours(params, d1, d2, xcf=xcf, grouped=grouped)
        assert np.array_equal(o.cpu().numpy(), off)
        assert np.array_equal(i.cpu().numpy()[:total], idx)


@pytest.mark.parametrize("num", [1, 3, 5, 31, 33, 130, 1030])
@pytest.mark.parametrize("ang_max", [5e-4, 0.02, 0.06, 3.2])
def test_auto_lists(num, ang_max):
    _check(_forests(num, 3), None, ang_max, True, False)


@pytest.mark.parametrize("num1,num2", [(1, 1500), (4, 32), (33, 31), (65, 1025), (257, 4)])
def test_two_field_lists(num1, num2):
    _check(_forests(num1, 5), _forests(num2, 6), 0.05, False, False)


@pytest.mark.parametrize("num1,num2", [(1, 1500), (5, 33), (67, 1024), (257, 1700)])
@pytest.mark.parametrize("zerr", [False, True])
def test_quasar_lists(num1, num2, zerr):
    from picca_gb300 import synthetic
    qs = synthetic.make_quasars(num2, 8, (150.0, 153.0), (0.0, 3.0), 1.8, 4.0)
    cut = dict(zerr_cut_deg=0.3, zerr_cut_kms=3000.0) if zerr else {}
    # narrow r_par range: many quasars are decided by the distance pre-cut
    _check(_forests(num1, 7), qs, 0.05, False, True, r_par_min=-40.0, r_par_max=40.0, **cut)
