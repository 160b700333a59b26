"""Wick terms of long forests of the linear grid with the default size of a
slice: a forest pair that pg_cf_wick takes over segments of equal bin is
listed once, one that it sweeps is cut into slices. The sums of both against
each other (a work buffer without room for the lists selects the sweep), to
1e-12 of the same sums of magnitudes, as in test_gpu_wick_segments."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _case(length, num=3):
    from picca_gb300 import pairs, wick
    from test_gpu_wick_segments import _cf1d, _forests
    fs = _forests(num, [length], 3)
    params = pairs.make_params(0.0, 20.0, 100.0, 5, 25, 0.06)
    engine = wick.WickEngine()
    dev = pairs.DeviceForests(fs, compact=False)
    assert dev.max_pixels == length
    offsets, index, total = engine.engine.neighbours(params, dev)
    first, second, n = wick.forest_pairs(dev, offsets, index, np.ones(total, dtype=bool))
    units = engine.plan_pairs(dev, first, second, n)
    return wick, engine, params, fs, dev, units, n, _cf1d()


@pytest.mark.parametrize("length", [300, 545, 600])
def test_listed_once(monkeypatch, length):
    wick, engine, params, fs, dev, units, n, cf1d = _case(length)
    assert n > 0 and units["num"] == n
    zw = torch.from_numpy(wick.evolution(fs.z, 2.25, 2.9)).cuda()
    arena, x_off, _keep = engine.xi_matrices(dev, wick.OneDTables(cf1d), np.arange(fs.num))
    whole = engine.work_buffer(params, length, length, n)
    runs = []
    for size, xa in ((whole.numel(), arena), (length**2 * 4, arena), (length**2 * 4, arena.abs())):
        engine._work = whole[:size]
        monkeypatch.setattr(engine, "work_buffer", lambda *a: engine._work)
        sums = engine.alloc_sums(125)
        engine.launch_pairs(params, dev, zw, zw, x_off, xa, units, sums)
        assert engine.stats().status == 0
        runs.append({k: v.cpu().numpy() for k, v in sums.items()})
    for key, want in runs[1].items():
        if key == "num_pairs_wick":
            assert want.sum() > 0 and np.array_equal(runs[0][key], want)
        else:
            assert np.all(np.abs(runs[0][key] - want) <= 1e-12 * np.abs(runs[2][key])), key


def test_swept_pairs_are_cut(monkeypatch):
    from picca_gb300 import pairs, synthetic
    from picca_gb300 import wick
    fs = synthetic.make_forests(4, 3, (150.0, 150.5), (0.0, 0.5), 2.5, 3.4, "uniform")
    dev = pairs.DeviceForests(fs, compact=False)
    first = torch.tensor([1, 2], dtype=torch.int32, device="cuda")
    second = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    dev.max_pixels, dev.npix = 900, np.full(4, 900)  # what the plan looks at
    units = wick.WickEngine().plan_pairs(dev, first, second, 2)
    assert units["num"] > 2 * 100


def test_operation_count():
    """One bin that holds every pixel pair: a row of n1 has n2 listed pixels to
    add up for each of n2 pixels, and n2 column segments, a product each."""
    from picca_gb300 import pairs, wick
    from test_gpu_wick_segments import _cf1d, _forests
    fs = _forests(2, [40, 70], 3)
    params = pairs.make_params(0.0, 1e4, 1e4, 1, 1, 0.06)
    engine = wick.WickEngine()
    dev = pairs.DeviceForests(fs, compact=False)
    first, second = (torch.tensor([k], dtype=torch.int32, device="cuda") for k in (0, 1))
    zw = torch.from_numpy(wick.evolution(fs.z, 2.25, 2.9)).cuda()
    arena, x_off, _keep = engine.xi_matrices(dev, wick.OneDTables(_cf1d()), np.arange(2))
    sums = engine.accumulate(params, dev, zw, zw, x_off, arena, first, second, 1,
                             engine.alloc_sums(1))
    stats = engine.stats()
    n1, n2 = 40, 70
    assert int(sums["num_pairs_wick"]) == n1 * n2
    assert stats.visited_pairs == (n1 * n2)**2 and stats.gemm_macs == n1 * (n2 * n2 + n2)
