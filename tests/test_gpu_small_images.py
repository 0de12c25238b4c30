"""Images a few pixels high: the grid along v is shorter than a tile's lines, which
then pass its end twice.  Both precisions and directions, dense enough for the
lines to run over the bounding box, against the FP64 direct Fourier transform to
the requested epsilon."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])
LAM = 299792458.0 / FREQ[0]


@pytest.mark.parametrize("ny", [10, 12, 16, 18, 20, 22, 26, 32, 40])
@pytest.mark.parametrize("precision,eps", [("mixed", 1e-3), ("mixed", 1e-5), ("fp64", 1e-6),
                                           ("fp64", 1e-11)])
def test_few_pixels(ny, precision, eps):
    rng = np.random.default_rng(ny)
    nx, nrow, px = 64, 3000, 2e-3
    uvw = rng.uniform(-1, 1, (nrow, 3)) * np.array([0.05, 0.49, 0.0]) / px * LAM
    uvw[0, 0] = 0.4 / px * LAM
    vis = rng.normal(size=(nrow, 1)) + 1j * rng.normal(size=(nrow, 1))
    img = rng.normal(size=(nx, ny))
    if precision == "mixed":
        vis, img = vis.astype(np.complex64), img.astype(np.float32)
    ctx = Context()
    args = dict(precision=precision, do_wgridding=False, **KW)
    d = ctx.ms2dirty(uvw, FREQ, vis, nx, ny, px, px, eps, **args)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, ny, px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(d.astype(np.float64), ref) <= eps
    v = ctx.dirty2ms(uvw, FREQ, img, px, px, eps, vis_dtype=vis.dtype, **args)
    mref = O.dft_dirty2ms(uvw, FREQ, img.astype(np.float64), px, px, negate_v=True,
                          divide_by_n=False)
    assert O.rel_rms(v, mref) <= eps
    ctx.close()
