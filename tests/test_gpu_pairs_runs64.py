"""FP64 sums with FP32 decisions (pg_pairs_runs64.cu) against the CPU oracle
where the sweep can go wrong: forests around the staged chunk of 64 pixels,
a single pixel, empty forests, pixels out of order, zero weights, few forests
(shared by many CTAs) and many, every cut, one and two fields.

Tolerances: pair counts equal; sums of positive terms differ from the oracle
by the order of at most ~1e5 additions in FP64 (rtol 1e-12), xi by 1e-12 of
the bin's sum of absolute terms."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = dict(r_par_min=0.0, r_par_max=200.0, r_trans_max=200.0, num_bins_r_par=50,
          num_bins_r_trans=50)


def _forests(num, seed, lengths=None, shuffle=False, zero=False, start=1):
    from picca_gb300 import synthetic
    from picca_gb300.forests import PIXEL_FIELDS
    fs = synthetic.make_forests(num, seed, (150.0, 152.0), (0.0, 2.0), 2.5, 3.5, "uniform",
                                thingid_start=start)
    rng = np.random.default_rng(seed)
    if lengths is not None:
        npix = np.diff(fs.pix_offset)
        want = np.minimum(np.resize(lengths, num), npix)
        keep = np.concatenate([np.arange(o, o + n) for o, n in zip(fs.pix_offset, want)])
        for key in PIXEL_FIELDS:
            setattr(fs, key, getattr(fs, key)[keep])
        fs.pix_offset = np.concatenate([[0], np.cumsum(want)]).astype(np.int64)
    if shuffle:
        for f in range(0, num, 2):
            order = fs.pix_offset[f] + rng.permutation(int(np.diff(fs.pix_offset)[f]))
            sl = slice(fs.pix_offset[f], fs.pix_offset[f + 1])
            for key in PIXEL_FIELDS:
                getattr(fs, key)[sl] = getattr(fs, key)[order]
    if zero:
        fs.weights[rng.random(fs.num_pixels) < 0.2] = 0.0
    fs.plate[:] = rng.integers(1, 3, num)
    fs.fiberid[:] = rng.integers(1, 1000, num)
    return fs


def _reference(fs, fs2=None, **kw):
    """Oracle rows, and xi of the absolute deltas (changes the deltas)."""
    from oracle import cpu as oracle
    from picca_gb300 import pairs, synthetic
    kwargs = dict(KW, **kw)
    ang_max = synthetic.correlation_ang_max(200.0, 2.0)
    p_or = oracle.make_params(**kwargs)
    other = fs2 if fs2 is not None else fs
    off, idx = oracle.neighbours(fs, other, p_or, ang_max, auto_mode=int(fs2 is None))
    ref = oracle.rows(fs, other, p_or, off, idx)
    for each in {id(fs): fs, id(other): other}.values():
        each.delta = np.abs(each.delta)
    abs_xi = oracle.rows(fs, other, p_or, off, idx)[1]
    return ref, abs_xi, pairs.make_params(ang_max=ang_max, **kwargs)


def _run(fs, fs2=None, compact=True, **kw):
    from picca_gb300 import pairs
    saved = [s.delta for s in (fs, fs2) if s is not None]
    ref, abs_xi, params = _reference(fs, fs2, **kw)
    for each, delta in zip((fs, fs2), saved):
        each.delta = delta
    engine = pairs.PairEngine()
    d1 = pairs.DeviceForests(fs, compact=compact)
    d2 = pairs.DeviceForests(fs2, compact=compact) if fs2 is not None else None
    offsets, index, total = engine.neighbours(params, d1, d2)
    order, num, _ = engine.work_order(d1, d2, offsets, index, total)
    nbins = params.num_bins_r_par * params.num_bins_r_trans
    rows = engine.alloc_rows(d1.num_rows, nbins)
    engine.accumulate(params, d1, d2, offsets, index, order, num, rows, pairs.MODE_FP64)
    engine.stats()
    got = pairs.rows_to_numpy(rows, d1.num_rows, nbins)
    assert np.array_equal(got[5], ref[5])
    for k in (0, 2, 3, 4):
        assert np.allclose(got[k], ref[k], rtol=1e-12, atol=1e-12), k
    assert np.all(np.abs(got[1] - ref[1]) <= 1e-12 * abs_xi + 1e-300)


@pytest.mark.parametrize("lengths", [[1], [1, 2, 33], [63, 64, 65], [127, 129, 32], [0, 5, 207]])
@pytest.mark.parametrize("num", [2, 9, 40])
def test_lengths(lengths, num):
    _run(_forests(num, 11 + num, lengths))


@pytest.mark.parametrize("kw", [
    dict(z_min_pairs=2.2, z_max_pairs=2.6), dict(zerr_cut_deg=1.0, zerr_cut_kms=4000.0),
    dict(remove_same_half_plate_close_pairs=True), dict(r_par_min=8.0, r_par_max=120.0),
    dict(x_correlation=True, r_par_min=-200.0, num_bins_r_par=100)])
def test_cuts(kw):
    _run(_forests(24, 5), **kw)
    _run(_forests(24, 6), _forests(17, 7, start=900), **kw)


@pytest.mark.parametrize("shuffle,zero,compact", [(True, False, True), (False, True, False),
                                                  (True, True, False)])
def test_order_and_weights(shuffle, zero, compact):
    _run(_forests(20, 9, shuffle=shuffle, zero=zero), compact=compact)
