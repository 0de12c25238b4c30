"""The FP32 spread and interpolation at the sizes where they can go wrong: runs
of equal footprint origins shorter and longer than a staged batch of 32
records, chunks with fewer records than warps, w planes in several passes, and
the supports whose footprint rows do not fill a warp or a pair of cells (W = 4
to 8).  Checked against the FP64 direct Fourier transform; the tolerance is the
requested epsilon, which bounds the kernel's aliasing error (FP32 rounding is
below 1e-6 here)."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context

pytestmark = pytest.mark.gpu
PX = np.deg2rad(20 / 3600)
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.5, sigma_max=2.0)
FREQ = np.array([1.5e8])
RUNS = {
    "one": [1],
    "two": [2],
    "steps": [3, 4, 5, 7, 8, 9, 1, 1, 12],
    "batches": [31, 32, 33, 64, 65],
    "long": [700],
    "singles": [1] * 97,
}


def _check(ctx, uvw, px, nx, ny, eps, rng, do_w=True):
    vis = (rng.normal(size=(len(uvw), 1)) + 1j * rng.normal(size=(len(uvw), 1))).astype(np.complex64)
    d = ctx.ms2dirty(uvw, FREQ, vis, nx, ny, px, px, eps, do_w, **KW)
    st = ctx.stats()
    u = uvw if do_w else uvw * np.array([1.0, 1.0, 0.0])
    ref = O.dft_ms2dirty(u, FREQ, vis, nx, ny, px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(np.asarray(d, dtype=np.float64), ref) <= eps
    img = np.zeros((nx, ny), dtype=np.float32)
    img[rng.integers(0, nx, 9), rng.integers(0, ny, 9)] = rng.normal(size=9)
    v = ctx.dirty2ms(uvw, FREQ, img, px, px, eps, do_w, **KW)
    vref = O.dft_dirty2ms(u, FREQ, img.astype(np.float64), px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(v, vref) <= eps
    return st


@pytest.mark.parametrize("eps", [5e-2, 1e-2, 1e-3, 1e-4, 1e-5])
@pytest.mark.parametrize("runs", sorted(RUNS))
def test_runs_of_equal_origins(eps, runs):
    rng = np.random.default_rng(len(runs))
    uvw = rng.uniform(-1, 1, (len(RUNS[runs]), 3)) * np.array([900.0, 900.0, 250.0])
    uvw = np.repeat(uvw, RUNS[runs], axis=0)
    ctx = Context()
    _check(ctx, uvw, PX, 96, 80, eps, rng)
    ctx.close()


@pytest.mark.parametrize("eps", [1e-2, 1e-3, 1e-4, 1e-5])
def test_without_w_term(eps):
    """One plane: kernel rows of the other planes are zero."""
    rng = np.random.default_rng(5)
    uvw = rng.uniform(-1, 1, (500, 3)) * np.array([900.0, 900.0, 0.0])
    ctx = Context()
    assert _check(ctx, uvw, PX, 96, 80, eps, rng, do_w=False)["nplanes"] == 1
    ctx.close()


@pytest.mark.parametrize("eps", [1e-3, 1e-5])
def test_records_between_plane_passes(eps, monkeypatch):
    """w planes in several passes: the interpolation adds its sums up."""
    monkeypatch.setenv("WSG_MAX_PLANES", "3")
    rng = np.random.default_rng(3)
    uvw = rng.uniform(-1, 1, (900, 3)) * 225.0
    ctx = Context()
    assert _check(ctx, uvw, 4 * PX, 128, 128, eps, rng)["nplanes"] > 3
    ctx.close()
