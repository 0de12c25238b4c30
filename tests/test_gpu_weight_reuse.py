"""The buffers of a closed imaging-weight object go to the next one of its
context: a gridding stream of another context, whose lookups of the first
object's grid were queued before it was closed, still sees its weights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KW = dict(negate_v=True, divide_by_n=False, sigma_min=1.1, sigma_max=2.0)
FREQ = np.array([1.5e8])
LAM = 299792458.0 / FREQ[0]


@pytest.mark.parametrize("nrow", [20000, 4000000])
def test_close_with_lookups_in_flight(nrow):
    import torch
    from wsclean_b200.gridder import Context, ImageWeights, Stream
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev)
    gen.manual_seed(nrow)
    n, px = 512, 2e-4
    uvw = (torch.rand((nrow, 3), generator=gen, device=dev, dtype=torch.float64) - 0.5) * (0.7 / px * LAM)
    uvw[:, 2] *= 0.02
    vis = torch.randn((nrow, 1), generator=gen, device=dev, dtype=torch.complex64)
    top = uvw.abs().max(dim=0).values.cpu().numpy() / LAM
    owner, other = Context(), Context()

    def image(close):
        w = ImageWeights("uniform", 0.0, n, n, px, px, context=owner)
        w.grid(uvw, FREQ)
        w.finish()
        # (turning the weights off sorts the rows: their records are then queued)
        with Stream(FREQ, n, n, px, px, 1e-5, (0.0, top[2], top[0], top[1]), nvis=nrow // 8,
                    context=other, **KW) as st:
            st.set_imaging_weights(w)
            st.add(uvw, vis)
            if close:
                st.set_imaging_weights(None)
                w.close()
                w = ImageWeights("natural", 0.0, n, n, px, px, context=owner)
            d = st.finish()
        w.close()
        return d.astype(np.float64)

    want, got = image(False), image(True)
    # (the same sums in the order of the atomics: FP32 rounding)
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
    owner.close()
    other.close()
