"""Memory of resident grids: what a stream reports holds its whole working set,
and plans and streams that are short of memory keep whole band rows."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])
LAM = 299792458.0 / FREQ[0]


def _stored(st, ny, vmax_px):
    """Bytes of the stored columns and of the rows transformed along v."""
    nvs = 2 * math.ceil(vmax_px * st["nv"] + 0.5 * st["supp"] + 2) + 2
    return 8 * st["band_rows"] * st["nplanes"] * (nvs + ny)


def test_stream_reports_both_band_arrays():
    from wsclean_b200.gridder import Stream
    n, px, v = 1024, 1e-4, 0.2
    with Stream(FREQ, n, n, px, px, 1e-5, (0.0, 200.0, v / px, v / px), nvis=10 ** 6, **KW) as st:
        s = st.stats()
        assert s["nv"] % 256 == 0  # a height of the pruned form
        # (and the u-transformed rows and the FP64 image)
        assert s["device_bytes"] >= _stored(s, n, v) + 8 * n * n * (s["nplanes"] + 1)


def _data(nrow, px, v):
    rng = np.random.default_rng(2)
    uvw = rng.uniform(-1, 1, (nrow, 3)) * np.array([0.2, v, 0.004]) / px * LAM
    uvw[0, :2] = np.array([0.2, v]) / px * LAM
    vis = (rng.normal(size=(nrow, 1)) + 1j * rng.normal(size=(nrow, 1))).astype(np.complex64)
    return uvw, vis


@pytest.mark.parametrize("kind", ["stream", "plan"])
def test_whole_rows_where_memory_is_short(kind, monkeypatch):
    """A wide band's stored columns and transformed rows take more memory than
    whole rows transformed in place: with little free, plans and streams keep
    whole rows, with the same results to within epsilon."""
    import torch
    import oracle as O
    from wsclean_b200.gridder import Plan, Stream, data_extent
    nx, ny, px, v, eps = 128, 600, 1e-4, 0.45, 1e-5
    uvw, vis = _data(3000, px, v)
    ref = O.dft_ms2dirty(uvw, FREQ, vis, nx, ny, px, px, negate_v=True, divide_by_n=False)
    dev = torch.device("cuda", 0)
    u, x = torch.as_tensor(uvw, device=dev), torch.as_tensor(vis, device=dev)

    def run():
        if kind == "stream":
            with Stream(FREQ, nx, ny, px, px, eps, data_extent(uvw, FREQ), nvis=3000, **KW) as st:
                st.add(uvw, vis)
                d, s = st.finish().astype(np.float64), st.stats()
                st.predict_begin(d.astype(np.float32))
                return d, st.predict(uvw), s
        jobs = [dict(npix_x=nx, npix_y=ny), dict(npix_x=nx, npix_y=ny - 96)]
        with Plan(u, FREQ, px, px, eps, jobs=jobs, **KW) as p:
            d = p.ms2dirty(x)
            m = p.dirty2ms([d[0], torch.zeros_like(d[1])])
            return d[0].double().cpu().numpy(), m.cpu().numpy(), p.stats()

    d0, m0, s0 = run()
    monkeypatch.setenv("WSG_FREE_MB", "1")
    d1, m1, s1 = run()
    assert s1["device_bytes"] < s0["device_bytes"]
    for d, m in ((d0, m0), (d1, m1)):
        assert O.rel_rms(d, ref) <= eps
        mref = O.dft_dirty2ms(uvw, FREQ, d.astype(np.float32).astype(np.float64), px, px,
                              negate_v=True, divide_by_n=False)
        assert O.rel_rms(m, mref) <= eps
