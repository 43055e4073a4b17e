"""A phase of few pixels is scored four lanes to a pixel, a longer one a pixel per thread:
against the oracle on frames where scores tie (flat colours: the first of N, S, W, E must
win), where superpixels of one or two pixels dissolve, with noise that keeps many pixels
moving and with so little that phases fall on either side of the line.  Labels are integers:
they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def frame(kind, H, W):
    rng = np.random.default_rng(H * W)
    if kind == "flat":
        return np.full((H, W, 3), 0.25, np.float32)
    steps = (np.indices((H, W)).sum(0) // 11 % 2)[..., None] * np.float32(0.5)
    noise = {"steps": 0.0, "quiet": 0.01, "loud": 0.5}[kind]
    return (0.2 + steps + noise * rng.random((H, W, 3))).astype(np.float32)


@pytest.mark.parametrize("kind", ["flat", "steps", "quiet", "loud"])
@pytest.mark.parametrize("H,W,sp,niters_seg", [(9, 11, 2, 4), (40, 40, 3, 4), (64, 97, 15, 4),
                                               (64, 97, 6, 1), (400, 900, 9, 4)])
def test_few_and_many_pixels_per_phase(kind, H, W, sp, niters_seg):
    from st_spix_gb300 import bist_cuda
    cfg = dict(niters=9, sp_size=sp, sm_period=4, niters_seg=niters_seg)
    img = frame(kind, H, W)
    lab, p = bist_cuda.run_bass(torch.from_numpy(img).cuda(), **cfg)
    st, ref, _, n = O.run_bass(img, O.default_config(**cfg))
    assert st == 0
    assert p.n == n
    np.testing.assert_array_equal(lab.cpu().numpy(), ref)
