"""Calls of up to 16384 visibilities sort in one CTA, larger ones device-wide:
sizes on both sides of every variant's limit, with visibilities that weight,
mask and value make inactive, against the FP64 direct Fourier transform
(tolerance: the requested epsilon), and the two paths against each other on
the same data (a row of zero weight more sends the call to the other path)."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context

pytestmark = pytest.mark.gpu
PX = np.deg2rad(20 / 3600)
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])
SIZES = [1, 1023, 1024, 3072, 3073, 6144, 6145, 9216, 9217, 12288, 12289, 16383, 16384, 16385]


def _data(n, rng):
    uvw = rng.uniform(-1, 1, (n, 3)) * np.array([900.0, 900.0, 250.0])
    vis = rng.normal(size=(n, 1)) + 1j * rng.normal(size=(n, 1))
    wgt = rng.uniform(0.5, 2.0, (n, 1)).astype(np.float32)
    mask = (rng.uniform(size=(n, 1)) > 0.1).astype(np.uint8)
    if n > 10:
        wgt[rng.integers(0, n, n // 10)] = 0
        vis[rng.integers(0, n, n // 10)] = 0
    return uvw, vis, wgt, mask


@pytest.mark.parametrize("prec,eps", [("mixed", 1e-5), ("fp64", 1e-9)])
@pytest.mark.parametrize("n", SIZES)
def test_sizes(n, prec, eps):
    rng = np.random.default_rng(n)
    nx = 64
    uvw, vis, wgt, mask = _data(n, rng)
    cdt = np.complex64 if prec == "mixed" else np.complex128
    vis = vis.astype(cdt)
    ctx = Context()
    kw = dict(KW, precision=prec, wgt=wgt, mask=mask)
    d = ctx.ms2dirty(uvw, FREQ, vis, nx, nx, PX, PX, eps, **kw)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, nx, PX, PX, wgt=wgt, mask=mask, negate_v=True,
                         divide_by_n=False)
    if np.any(ref):
        assert O.rel_rms(np.asarray(d, dtype=np.float64), ref) <= eps
    img = rng.normal(size=(nx, nx))
    img = img.astype(np.float32 if prec == "mixed" else np.float64)
    v = ctx.dirty2ms(uvw, FREQ, img, PX, PX, eps, vis_dtype=cdt, **kw)
    vref = O.dft_dirty2ms(uvw, FREQ, img.astype(np.float64), PX, PX, wgt=wgt, mask=mask,
                          negate_v=True, divide_by_n=False)
    if np.any(vref):
        assert O.rel_rms(v, vref) <= eps
    assert not np.any(v[(wgt == 0) | (mask == 0)])
    ctx.close()


@pytest.mark.parametrize("nchan", [1, 8])
def test_paths_agree(nchan):
    """16384 visibilities against the same ones and more rows of zero weight:
    the same records in the same order, so the degridded values are equal."""
    rng = np.random.default_rng(1)
    n = 16384 // nchan
    freq = np.linspace(1.5e8, 1.52e8, nchan)
    uvw = rng.uniform(-1, 1, (n + 3, 3)) * np.array([900.0, 900.0, 250.0])
    wgt = np.ones((n + 3, nchan), dtype=np.float32)
    wgt[n:] = 0
    img = rng.normal(size=(64, 64)).astype(np.float32)
    ctx = Context()
    a = ctx.dirty2ms(uvw[:n], freq, img, PX, PX, 1e-5, wgt=wgt[:n], **KW)
    b = ctx.dirty2ms(uvw, freq, img, PX, PX, 1e-5, wgt=wgt, **KW)
    assert np.array_equal(a, b[:n]) and not np.any(b[n:])
    ctx.close()
