"""The FP64 matrix-unit spread and interpolation at the sizes where they can go
wrong: runs of equal footprint origins shorter than, equal to and longer than
a matrix step (4 and 8 records) and a staged batch (32), chunks of one record
(an empty second team), every kernel support from one warp a record to a team
a record.  Checked against the FP64 direct Fourier transform; the tolerance is
the requested epsilon, which bounds the kernel's aliasing error (rounding,
about 1e-15 times the number of records, is far below it)."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context

pytestmark = pytest.mark.gpu
PX = np.deg2rad(20 / 3600)
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])


def _uvw(runs, rng):
    """One random position per run, repeated."""
    uvw = rng.uniform(-1, 1, (len(runs), 3)) * np.array([900.0, 900.0, 250.0])
    return np.repeat(uvw, runs, axis=0)


RUNS = {
    "one": [1],
    "two": [2],
    "steps": [3, 4, 5, 7, 8, 9, 1, 1, 12],
    "batches": [31, 32, 33, 64, 65],
    "long": [700],
    "singles": [1] * 97,
}


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-4, 1e-5, 1e-6, 1e-7, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12])
@pytest.mark.parametrize("runs", sorted(RUNS))
def test_runs_of_equal_origins(eps, runs):
    rng = np.random.default_rng(len(runs))
    nx, ny = 96, 80
    uvw = _uvw(RUNS[runs], rng)
    vis = rng.normal(size=(len(uvw), 1)) + 1j * rng.normal(size=(len(uvw), 1))
    ctx = Context()
    d = ctx.ms2dirty(uvw, FREQ, vis, nx, ny, PX, PX, eps, precision="fp64", **KW)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, ny, PX, PX, negate_v=True, divide_by_n=False)
    assert O.rel_rms(d, ref) <= eps
    img = np.zeros((nx, ny))
    img[rng.integers(0, nx, 9), rng.integers(0, ny, 9)] = rng.normal(size=9)
    v = ctx.dirty2ms(uvw, FREQ, img, PX, PX, eps, precision="fp64", vis_dtype=np.complex128, **KW)
    vref = O.dft_dirty2ms(uvw, FREQ, img, PX, PX, negate_v=True, divide_by_n=False)
    assert O.rel_rms(v, vref) <= eps
    ctx.close()


@pytest.mark.parametrize("eps", [1e-5, 1e-12])
def test_records_between_plane_passes(eps, monkeypatch):
    """w planes in several passes: the interpolation adds its sums up."""
    monkeypatch.setenv("WSG_MAX_PLANES", "3")
    rng = np.random.default_rng(3)
    nx = 128
    uvw = rng.uniform(-1, 1, (900, 3)) * np.array([900.0, 900.0, 900.0])
    vis = rng.normal(size=(900, 1)) + 1j * rng.normal(size=(900, 1))
    px = 4 * PX
    ctx = Context()
    d = ctx.ms2dirty(uvw / 4, FREQ, vis, nx, nx, px, px, eps, precision="fp64", **KW)
    assert ctx.stats()["nplanes"] > 3
    ref = O.dft_ms2dirty(uvw / 4, FREQ, vis, nx, nx, px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(d, ref) <= eps
    v = ctx.dirty2ms(uvw / 4, FREQ, ref, px, px, eps, precision="fp64", vis_dtype=np.complex128, **KW)
    vref = O.dft_dirty2ms(uvw / 4, FREQ, ref, px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(v, vref) <= eps
    ctx.close()
