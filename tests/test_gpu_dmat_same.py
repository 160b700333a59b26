"""Equal data and model binnings of the distortion matrix where the kernel's
forms can go wrong, against the FP64 oracle with the bounds of test_gpu_dmat:
pairs that touch a model bin but are not selected (half plate, redshift cut),
forests of more pixels than one strip of bins holds, row chunks, both products."""

import numpy as np
import pytest

import test_gpu_dmat as base
from test_gpu_dmat import cuda  # noqa: F401 (fixture)

pytestmark = pytest.mark.gpu

CASES = {
    "veto": dict(np=10, nt=8, coef=1, zevol=True, shp=True, rmu=False, zcut=(2.3, 2.9), nproc=3,
                 reject=0.85),
    "half_plate": dict(np=15, nt=15, coef=1, zevol=False, shp=True, rmu=False, zcut=None, nproc=2,
                       reject=0.9),
    "fine": dict(np=40, nt=37, coef=1, zevol=True, shp=False, rmu=False, zcut=None, nproc=1,
                 reject=0.95),
}


def _long(seed=7, num=90):
    """Forests of up to 600 pixels of the linear grid."""
    from picca_gb300 import synthetic
    fs = synthetic.make_forests(num, seed, (150.0, 151.5), (0.0, 1.5), grid="lin")
    rng = np.random.default_rng(seed)
    fs.plate = rng.integers(0, 3, fs.num).astype(np.int64)
    fs.fiberid = rng.integers(1, 1000, fs.num).astype(np.int64)
    fs.order = rng.integers(0, 2, fs.num).astype(np.int64)
    return fs


@pytest.mark.parametrize("case", sorted(CASES))
def test_same_binning(cuda, monkeypatch, case):
    monkeypatch.setitem(base.CASES, case, CASES[case])
    base.test_synthetic_matches_oracle(cuda, case)


def test_strips(cuda, monkeypatch):
    monkeypatch.setitem(base.CASES, "long", dict(CASES["veto"], nt=10))
    monkeypatch.setattr(base, "_synthetic", _long)
    assert np.diff(_long().pix_offset).max() > 400
    base.test_synthetic_matches_oracle(cuda, "long")


def test_row_counts(cuda, monkeypatch):
    """Numbers of touched bins around the product's tiles of 32 and 128 rows
    (row chunks of 17 to 300 for a pair's few hundred bins)."""
    from picca_gb300 import dmat
    make = dmat.make_dmat_params
    for capacity in (34, 66, 130, 258, 600):
        monkeypatch.setitem(base.CASES, "rows", dict(CASES["fine"], nt=40, reject=0.985))
        monkeypatch.setattr(dmat, "make_dmat_params", lambda *a, **k: make(
            *a, **dict(k, row_capacity=capacity, product="split_bf16")))
        base.test_synthetic_matches_oracle(cuda, "rows")
