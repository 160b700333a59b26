"""T1-T3 over row and column segments (pg_wick_segments.cu) against the sweep
over all pairs of listed pixel pairs (wick_t123_kernel, which a work buffer
too small for the segment lists still selects) on forests around the warp's
32 bins and the block's 256 threads, single pixels, folded and signed r_par,
other bin counts, units cut into slices and several batches of pairs.

Both sum the same FP64 terms in another order; the summed magnitudes are the
sums of the same terms with absolute weights and correlations, so the
difference is bounded by 1e-12 of them (below 1e6 terms a cell)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _forests(num, lengths, seed):
    from picca_gb300 import synthetic
    from picca_gb300.forests import PIXEL_FIELDS
    fs = synthetic.make_forests(num, seed, (150.0, 151.5), (0.0, 1.5), 2.5, 3.4, "uniform",
                                grid="lin")
    npix = np.diff(fs.pix_offset)
    want = np.minimum(np.resize(lengths, num), npix)
    keep = np.concatenate([np.arange(o, o + n) for o, n in zip(fs.pix_offset, want)])
    for key in PIXEL_FIELDS:
        setattr(fs, key, getattr(fs, key)[keep])
    fs.pix_offset = np.concatenate([[0], np.cumsum(want)]).astype(np.int64)
    return fs


def _cf1d():
    k = np.arange(1000)
    ones = np.ones(k.size, dtype=np.int64)
    return {"LLMIN": float(np.log10(3600.0)), "DLL": 3e-4, "v1d": 0.1 + 0.05 * np.sin(k / 60.0),
            "nv1d": ones, "c1d": np.where(k == 0, 1.0, 0.05 * np.cos(k / 7.0)), "nb1d": ones}


@pytest.mark.parametrize("lengths,num", [([1], 6), ([1, 2, 31], 8), ([32, 33, 64, 5], 8),
                                         ([150, 257, 96], 7), ([300], 4)])
@pytest.mark.parametrize("unfold,np_,nt", [(False, 50, 50), (True, 40, 10), (False, 7, 13)])
def test_against_sweep(monkeypatch, lengths, num, unfold, np_, nt):
    from picca_gb300 import pairs, wick
    fs = _forests(num, lengths, 3)
    params = pairs.make_params(-200.0 if unfold else 0.0, 200.0, 200.0, np_, nt, 0.06,
                               x_correlation=unfold)
    monkeypatch.setattr(wick, "SLICE_TARGET", 1e7)  # units cut into slices
    engine = wick.WickEngine()
    dev = pairs.DeviceForests(fs, compact=False)
    offsets, index, total = engine.engine.neighbours(params, dev)
    first, second, n = wick.forest_pairs(dev, offsets, index, np.ones(total, dtype=bool))
    zw = torch.from_numpy(wick.evolution(fs.z, 2.25, 2.9)).cuda()
    units = engine.plan_pairs(dev, first, second, n)
    tables = wick.OneDTables(_cf1d())
    arena, x_off, _keep = engine.xi_matrices(dev, tables, np.arange(num))
    nb = np_ * nt
    whole = engine.work_buffer(params, dev.max_pixels, dev.max_pixels, units["num"])
    per_pair = (dev.max_pixels**2 * 12 + (2 * nb + 5) * 4 + 255) // 256 * 256
    runs = {}
    for name, size, xa in (("segments", whole.numel(), arena), ("batches", 2 * per_pair, arena),
                           ("sweep", dev.max_pixels**2 * 4, arena),
                           ("magnitude", dev.max_pixels**2 * 4, arena.abs())):
        engine._work = whole[:size]
        sums = engine.alloc_sums(nb)
        monkeypatch.setattr(engine, "work_buffer", lambda *a: engine._work)
        engine.launch_pairs(params, dev, zw, zw, x_off, xa, units, sums)
        assert engine.stats().status == 0
        runs[name] = {k: v.cpu().numpy() for k, v in sums.items()}
    scale = runs["magnitude"]
    assert runs["sweep"]["num_pairs_wick"].sum() > 0 or max(lengths) < 40
    for name in ("segments", "batches"):
        for key, want in runs["sweep"].items():
            if key == "num_pairs_wick":
                assert np.array_equal(runs[name][key], want), name
            else:
                assert np.all(np.abs(runs[name][key] - want) <= 1e-12 * np.abs(scale[key])), (
                    name, key)
