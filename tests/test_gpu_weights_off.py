"""Turning a stream's imaging weights off concerns the rows added later: those
already added, which may wait in a batch, keep the weights they were added
with.  The parts are compared with one another (the same sums: FP32 rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])
LAM = 299792458.0 / FREQ[0]


def test_rows_keep_their_weights():
    from wsclean_b200.gridder import Context, ImageWeights, Stream
    rng = np.random.default_rng(4)
    nrow, n, px = 6000, 256, 2e-4
    uvw = rng.uniform(-0.35, 0.35, (nrow, 3)) / px * LAM
    uvw[:, 2] *= 0.02
    vis = (rng.normal(size=(nrow, 1)) + 1j * rng.normal(size=(nrow, 1))).astype(np.complex64)
    top = np.abs(uvw).max(axis=0) / LAM
    ctx = Context()

    def image(part, off):
        with ImageWeights("uniform", 0.0, n, n, px, px, context=ctx) as w, \
                Stream(FREQ, n, n, px, px, 1e-5, (0.0, top[2], top[0], top[1]), nvis=nrow,
                       context=ctx, **KW) as st:
            w.grid(uvw, FREQ)
            w.finish()
            if part != "late":
                st.set_imaging_weights(w)
                st.add(uvw[:4000], vis[:4000])
            if off:
                st.set_imaging_weights(None)
            if part != "early":
                st.add(uvw[4000:], vis[4000:])
            return st.finish().astype(np.float64)

    early, late, both = image("early", False), image("late", True), image("both", True)
    assert np.linalg.norm(image("early", True) - early) <= 1e-5 * np.linalg.norm(early)
    assert np.linalg.norm(both - (early + late)) <= 1e-5 * np.linalg.norm(both)
    ctx.close()
