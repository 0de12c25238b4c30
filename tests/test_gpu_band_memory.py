"""Memory of resident grids: what a stream reports holds its whole working set."""
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
        assert s["device_bytes"] >= _stored(s, n, v) + 8 * n * n
