"""get_marked_video in one kernel against the oracle: sizes that leave partial blocks and
whose rows cross them, pointers that are not 16-byte aligned, negative labels, colours
outside [0, 1], infinities and NaN (the clamp saturates: a NaN becomes 0)."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,W,skip", [(1, 2, 2, 0), (3, 41, 57, 0), (3, 41, 57, 1),
                                        (2, 33, 512, 0), (2, 2, 1500, 1), (1, 700, 3, 0)])
def test_marked_video_matches_the_oracle(T, H, W, skip):
    from st_spix_gb300 import bist_cuda
    rng = np.random.default_rng(T * H + W)
    vid = rng.uniform(-0.2, 1.2, size=(T + skip, H, W, 3)).astype(np.float32)
    vid[:, 0, 0] = [np.nan, np.inf, -np.inf]
    spix = rng.integers(-1, 4, size=(T + skip, H, W)).astype(np.int32)
    color = np.array([0.25, 0.5, 2.0], np.float32)
    gv, gs = torch.from_numpy(vid).cuda()[skip:], torch.from_numpy(spix).cuda()[skip:]
    out = bist_cuda.get_marked_video(gv, gs, torch.from_numpy(color)).cpu().numpy()
    plain = np.where(np.isnan(vid[skip:]), np.float32(0), vid[skip:])
    ref = O.get_marked_video(plain, spix[skip:], color)
    np.testing.assert_array_equal(out, ref)
