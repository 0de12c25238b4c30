"""The pruned v transform of the mixed form over its geometries: every column
transform length (256 to 8192 points), one and several twisted passes, image
heights that are not multiples of 32, v bands as wide as a transform and
(falling back to whole rows) as wide as the grid; both directions against the
FP64 direct Fourier transform.  The tolerance is the requested epsilon, 1e-5."""
import numpy as np
import pytest

import oracle as O
from wsclean_b200.gridder import Context

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
EPS = 1e-5
C = 299792458.0
FREQ = np.array([1.5e8])
LAM = C / FREQ[0]


def _uvw(nrow, umax_px, vmax_px, px, rng):
    """Uniform rows with |u| px, |v| px up to the given fractions of a cycle a pixel."""
    uvw = rng.uniform(-1, 1, (nrow, 3)) * np.array([umax_px, vmax_px, 0.01]) / px * LAM
    uvw[0, :2] = np.array([umax_px, vmax_px]) / px * LAM
    return uvw


@pytest.mark.parametrize("ny", [64, 250, 722, 1502, 2998, 5402])
@pytest.mark.parametrize("vmax_px", [0.03, 0.17, 0.30, 0.47])
def test_v_geometries(ny, vmax_px):
    rng = np.random.default_rng(ny)
    nx = 64
    px = 0.08 / max(ny, 256)
    uvw = _uvw(300, 0.2, vmax_px, px, rng)
    vis = (rng.normal(size=(300, 1)) + 1j * rng.normal(size=(300, 1))).astype(np.complex64)
    ctx = Context()
    d = ctx.ms2dirty(uvw, FREQ, vis, nx, ny, px, px, EPS, **KW)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, ny, px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(np.asarray(d, dtype=np.float64), ref) <= EPS
    img = np.zeros((nx, ny), dtype=np.float32)
    img[rng.integers(0, nx, 9), rng.integers(0, ny, 9)] = rng.normal(size=9)
    img[0, 0] = img[-1, -1] = img[0, -1] = 1.0
    v = ctx.dirty2ms(uvw, FREQ, img, px, px, EPS, **KW)
    vref = O.dft_dirty2ms(uvw, FREQ, img.astype(np.float64), px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(v, vref) <= EPS
    ctx.close()


def test_planes_in_passes(monkeypatch):
    """Plane passes shorter than the layout: rows of a pass start p0 planes in."""
    monkeypatch.setenv("WSG_MAX_PLANES", "2")
    rng = np.random.default_rng(7)
    nx, ny, px = 128, 322, 4e-4
    uvw = _uvw(400, 0.2, 0.2, px, rng)
    uvw[:, 2] *= 20
    vis = (rng.normal(size=(400, 1)) + 1j * rng.normal(size=(400, 1))).astype(np.complex64)
    ctx = Context()
    d = ctx.ms2dirty(uvw, FREQ, vis, nx, ny, px, px, EPS, **KW)
    assert ctx.stats()["plane_batch"] == 2 and ctx.stats()["nplanes"] % 2 == 1
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, ny, px, px, negate_v=True, divide_by_n=False)
    assert O.rel_rms(np.asarray(d, dtype=np.float64), ref) <= EPS
    v = ctx.dirty2ms(uvw, FREQ, d, px, px, EPS, **KW)
    vref = O.dft_dirty2ms(uvw, FREQ, np.asarray(d, dtype=np.float64), px, px, negate_v=True,
                          divide_by_n=False)
    assert O.rel_rms(v, vref) <= EPS
    ctx.close()


@pytest.mark.parametrize("vmax_px", [0.03, 0.30, 0.47])
def test_plan_and_stream_equal_the_call(vmax_px):
    """Plans (facets of unequal heights) and streams use the same rows."""
    import torch
    from wsclean_b200.gridder import Plan, Stream, data_extent
    rng = np.random.default_rng(11)
    nx, ny = 96, 250
    px = 3e-4
    uvw = _uvw(500, 0.2, vmax_px, px, rng)
    vis = (rng.normal(size=(500, 1)) + 1j * rng.normal(size=(500, 1))).astype(np.complex64)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, ny, px, px, negate_v=True, divide_by_n=False)
    dev = torch.device("cuda", 0)
    u, v = torch.as_tensor(uvw, device=dev), torch.as_tensor(vis, device=dev)
    jobs = [dict(npix_x=nx, npix_y=ny), dict(npix_x=64, npix_y=90, center_x=5 * px)]
    with Plan(u, FREQ, px, px, EPS, jobs=jobs, **KW) as plan:
        out = plan.ms2dirty(v)
        assert O.rel_rms(out[0].double().cpu().numpy(), ref) <= EPS
        acc = plan.ms2dirty(v, dirty=[o.clone() for o in out], accumulate=True)
        assert O.rel_rms(acc[0].double().cpu().numpy(), 2 * ref) <= EPS
        model = plan.dirty2ms([out[0], torch.zeros_like(out[1])])
        mref = O.dft_dirty2ms(uvw, FREQ, out[0].double().cpu().numpy(), px, px, negate_v=True,
                              divide_by_n=False)
        assert O.rel_rms(model.cpu().numpy(), mref) <= EPS
    with Stream(FREQ, nx, ny, px, px, EPS, data_extent(uvw, FREQ), nvis=500, **KW) as st:
        st.add(uvw[:200], vis[:200])
        st.add(uvw[200:], vis[200:])
        d = st.finish()
        assert O.rel_rms(d.astype(np.float64), ref) <= EPS
        st.predict_begin(d)
        m = st.predict(uvw)
        mref = O.dft_dirty2ms(uvw, FREQ, d.astype(np.float64), px, px, negate_v=True, divide_by_n=False)
        assert O.rel_rms(m, mref) <= EPS
