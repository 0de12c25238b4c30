"""The 8192-point transforms of the mixed form along u and v: one and two twisted
passes, bands up to and past the rows that can be staged, image sides that
leave odd remainders, an odd number of plane passes; both directions against
the FP64 direct Fourier transform.  The tolerance is the requested epsilon."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
EPS = 1e-5
FREQ = np.array([1.5e8])
LAM = 299792458.0 / FREQ[0]


@pytest.mark.parametrize("side", [4200, 6002, 9002])
@pytest.mark.parametrize("extent", [0.21, 0.30, 0.40, 0.46])
@pytest.mark.parametrize("axis", [0, 1])
def test_long_axis(side, extent, axis, monkeypatch):
    if extent == 0.30:
        monkeypatch.setenv("WSG_MAX_PLANES", "3")
    rng = np.random.default_rng(side + axis)
    npix = [34, 34]
    npix[axis] = side
    px = 0.08 / side
    ext = [0.2, 0.2, 0.01]
    ext[axis] = extent
    uvw = rng.uniform(-1, 1, (200, 3)) * np.array(ext) / px * LAM
    uvw[0, :2] = np.array(ext[:2]) / px * LAM
    uvw[:, 2] *= 20 if extent == 0.30 else 1
    vis = (rng.normal(size=(200, 1)) + 1j * rng.normal(size=(200, 1))).astype(np.complex64)
    ctx = Context()
    d = ctx.ms2dirty(uvw, FREQ, vis, npix[0], npix[1], px, px, EPS, **KW)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, npix[0], npix[1], px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(np.asarray(d, dtype=np.float64), ref) <= EPS
    img = np.zeros(npix, dtype=np.float32)
    img[rng.integers(0, npix[0], 9), rng.integers(0, npix[1], 9)] = rng.normal(size=9)
    img[0, 0] = img[-1, -1] = img[0, -1] = img[-1, 0] = 1.0
    v = ctx.dirty2ms(uvw, FREQ, img, px, px, EPS, **KW)
    vref = O.dft_dirty2ms(uvw, FREQ, img.astype(np.float64), px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(v, vref) <= EPS
    ctx.close()
