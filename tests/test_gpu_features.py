"""Inputs of the warm-start network at the edges of the kernel's batches and
ranges: forests of 1 to 97 pixels around multiples of 32 and of a batch of 96,
masked and unsorted pixels, and numbers of forests around a CTA's range,
against the FP64 formulas rounded to bf16 (FP32 sums of at most a few dozen
terms per bin: 1e-5, then half a bf16 unit, 2^-8 relative)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _raw(lengths, seed):
    from picca_gb300 import synthetic_spectra
    raw = synthetic_spectra.make_raw_forests(len(lengths), seed, z_lo=2.9, z_hi=3.4)
    rng = np.random.default_rng(seed)
    cols = {k: [] for k in ("log_lambda", "flux", "ivar", "transmission_correction")}
    for f, n in enumerate(lengths):
        o, e = int(raw.pix_offset[f]), int(raw.pix_offset[f + 1])
        take = o + rng.integers(0, e - o, n)
        if f % 3:
            take = np.sort(take)
        for k in cols:
            cols[k].append(getattr(raw, k)[take])
        cols["ivar"][-1] = np.where(rng.random(n) < 0.2, 0.0, cols["ivar"][-1])
    for k, v in cols.items():
        setattr(raw, k, np.concatenate(v))
    raw.pix_offset = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    return raw


@pytest.mark.parametrize("num", [1, 8, 9, 2433])
def test_features(num):
    from picca_gb300 import continuum, learned
    around = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 191, 192, 193]
    lengths = [around[i % len(around)] for i in range(num)]
    raw = _raw(lengths, 7)
    eng = continuum.Dr16Gpu(raw.grid)
    eng.mean_cont_y = 1.0 + 0.2 * np.sin(30 * eng.mean_cont_x)
    model, _keep = eng._model()
    feat, a0 = learned.features(eng, continuum.DeviceSpectra(raw, eng.device), model)
    feat, a0 = feat.float().cpu().numpy(), a0.cpu().numpy()
    rest = raw.grid.log_lambda_rest_frame_grid
    for f in range(min(num, 40)):
        sl = slice(raw.pix_offset[f], raw.pix_offset[f + 1])
        iv, fl, ll = raw.ivar[sl], raw.flux[sl], raw.log_lambda[sl]
        want_a0 = (fl * iv).sum() / iv.sum() if iv.sum() > 0 else 0.0
        scale = np.abs(fl * iv).sum() / iv.sum() if iv.sum() > 0 else 0.0
        assert abs(a0[f] - want_a0) <= 1e-5 * scale
        u = ll - rest[0] - np.log10(1 + raw.z_qso[f])
        pos = u * 64 / (rest[-1] - rest[0])
        x = eng.mean_cont_x - rest[0]
        i = np.clip(np.searchsorted(x, u) - 1, 0, len(x) - 2)
        mc = eng.mean_cont_y[i] + (u - x[i]) * np.diff(eng.mean_cont_y)[i] / np.diff(x)[i]
        mc = mc * raw.transmission_correction[sl]
        ok = (iv > 0) & (mc != 0)
        near = np.abs(pos - np.round(pos)) < 1e-4   # bin decided by rounding
        bins = np.clip(np.floor(pos), 0, 63).astype(int)
        for k in range(64):
            if (near & ((np.round(pos) == k) | (np.round(pos) == k + 1))).any():
                continue
            m = ok & (bins == k)
            want = 0.0
            if m.any() and want_a0 != 0:
                r = (fl[m] / mc[m] * iv[m]) / iv[m].sum() / want_a0
                want = r.sum() - 1
                tol = 1e-5 * (np.abs(r).sum() + 1) * max(1.0, scale / abs(want_a0))
            else:
                tol = 0.0
            assert abs(feat[f, k] - want) <= tol + abs(want) * 2**-8, (f, k)
        if iv.sum() > 0:
            snr = (fl * np.sqrt(iv))[iv > 0].sum() / (iv > 0).sum()
            assert abs(feat[f, 65] - np.log(max(snr, 1e-3))) <= 1e-3 + abs(np.log(max(snr, 1e-3))) * 2**-8
        assert abs(feat[f, 64] - (raw.z_qso[f] - 3)) <= 1e-6 + abs(raw.z_qso[f] - 3) * 2**-8
    assert np.all(feat[:, 66:] == 0)
