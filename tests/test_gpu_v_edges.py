"""Visibilities next to both ends of a v band that is nearly as wide as the
grid: a tile holds footprints of both ends, dense enough for its lines to run
over the bounding box.  Calls, plans and streams, both directions, against the
FP64 direct Fourier transform; the tolerance is the requested epsilon."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context, Plan, Stream, data_extent

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])
LAM = 299792458.0 / FREQ[0]
NX, PX = 64, 0.08 / 256
CASES = [(64, 1e-5, 0.47), (128, 1e-5, 0.47), (160, 1e-5, 0.47), (512, 1e-5, 0.492),
         (160, 1e-4, 0.47), (640, 1e-3, 0.494), (196, 1e-3, 0.47), (180, 1e-4, 0.46),
         (720, 1e-4, 0.488), (322, 1e-5, 0.47), (658, 1e-5, 0.488)]


def _data(ny, vmax_px):
    """4000 rows within 8 cells of +-vmax and a narrow range of u, w = 0."""
    rng = np.random.default_rng(ny)
    n = 4000
    uvw = np.zeros((n, 3))
    uvw[:, 0] = rng.uniform(0.0, 0.02, n)
    uvw[:, 1] = vmax_px * np.where(rng.random(n) < 0.5, 1, -1) * (1 - rng.uniform(0, 8.0 / ny, n))
    uvw[0, :2] = 0.2, vmax_px
    uvw *= LAM / PX
    vis = (rng.normal(size=(n, 1)) + 1j * rng.normal(size=(n, 1))).astype(np.complex64)
    img = rng.normal(size=(NX, ny)).astype(np.float32)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, NX, ny, PX, PX, negate_v=True, divide_by_n=False)
    mref = O.dft_dirty2ms(uvw, FREQ, img.astype(np.float64), PX, PX, negate_v=True,
                          divide_by_n=False)
    return uvw, vis, img, ref, mref


@pytest.mark.parametrize("ny,eps,vmax_px", CASES)
def test_call(ny, eps, vmax_px):
    uvw, vis, img, ref, mref = _data(ny, vmax_px)
    ctx = Context()
    d = ctx.ms2dirty(uvw, FREQ, vis, NX, ny, PX, PX, eps, do_wgridding=False, **KW)
    assert O.rel_rms(d.astype(np.float64), ref) <= eps
    v = ctx.dirty2ms(uvw, FREQ, img, PX, PX, eps, do_wgridding=False, **KW)
    assert O.rel_rms(v, mref) <= eps
    ctx.close()


@pytest.mark.parametrize("ny,eps,vmax_px", CASES[:1] + CASES[2:4] + CASES[-1:])
def test_plan_and_stream(ny, eps, vmax_px):
    import torch
    uvw, vis, img, ref, mref = _data(ny, vmax_px)
    dev = torch.device("cuda", 0)
    u, v, m = (torch.as_tensor(x, device=dev) for x in (uvw, vis, img))
    with Plan(u, FREQ, PX, PX, eps, npix_x=NX, npix_y=ny, do_wgridding=False, **KW) as plan:
        assert O.rel_rms(plan.ms2dirty(v)[0].double().cpu().numpy(), ref) <= eps
        assert O.rel_rms(plan.dirty2ms([m]).cpu().numpy(), mref) <= eps
    with Stream(FREQ, NX, ny, PX, PX, eps, data_extent(uvw, FREQ), nvis=len(uvw),
                do_wgridding=False, **KW) as st:
        st.add(uvw[:2500], vis[:2500])
        st.add(uvw[2500:], vis[2500:])
        assert O.rel_rms(st.finish().astype(np.float64), ref) <= eps
        st.predict_begin(img)
        assert O.rel_rms(st.predict(uvw), mref) <= eps
