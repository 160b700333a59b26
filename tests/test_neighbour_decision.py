"""FP32 decisions of the neighbour search (nbr_decide in
picca_gb300/csrc/pg_neighbours.cu) emulated on the CPU: whatever the FP32
margins decide is the FP64 decision, for the RA order of the auto-correlation
and for the distance pre-cut of the cross-correlation, also for distances and
limits far from the usual range and for values a few rounding errors apart."""

import numpy as np

f32 = np.float32


def test_ra_order_decisions():
    rng = np.random.default_rng(1)
    ra1 = rng.uniform(0, 2 * np.pi, 400_000)
    ra2 = ra1 + rng.normal(0, 1, ra1.size) * 10.0 ** rng.uniform(-17, 0, ra1.size)
    err = (f32(2e-7) * np.abs(ra1.astype(f32)) + f32(1e-30)).astype(f32)
    d = ra1.astype(f32) - ra2.astype(f32)
    m = err + f32(2e-7) * np.abs(ra2.astype(f32))
    assert not np.any((d < -m) & (ra1 > ra2))
    assert not np.any((d > m) & ~(ra1 > ra2))
    assert np.mean(np.abs(d) > m) > 0.25


def test_distance_precut_decisions():
    rng = np.random.default_rng(2)
    n = 400_000
    for scale, limit in ((4000.0, 200.0), (4000.0, 1e-3), (50.0, 200.0), (1e5, 3e4)):
        robj = scale * rng.uniform(0.9, 1.1, n)
        ang = 10.0 ** rng.uniform(-6, np.log10(2.0), n)
        cos_half = np.cos(ang / 2)
        rmax = limit
        # distances on the edge of the limit, off by many or few roundings
        off = rng.normal(0, 1, n) * scale * 10.0 ** rng.uniform(-12, -1, n)
        rfirst = robj + rmax / cos_half + off
        dot = (np.cos(ang) + rng.uniform(-4e-7, 4e-7, n)).astype(f32)
        xh = f32(0.5) * (f32(1) + dot)
        ch = np.sqrt(np.maximum(xh, f32(0))).astype(f32)
        u = rfirst.astype(f32) - robj.astype(f32)
        p = u * ch
        m = (f32(2e-7) * np.abs(rfirst.astype(f32)) + f32(2e-7) * np.abs(robj.astype(f32)) +
             f32(1e-6) + f32(2e-7) * f32(2 * rmax))
        e = np.abs(u) * f32(5e-6) + m
        est = xh >= f32(0.25)
        exact = (rfirst - robj) * cos_half < rmax
        inside = est & (p < f32(rmax) - e)
        outside = est & (p > f32(rmax) + e)
        assert not np.any(inside & ~exact)
        assert not np.any(outside & exact)
        assert np.mean(inside | outside) > 0.2
