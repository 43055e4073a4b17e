"""The halves of a split are bits set by the warp or block that grows them: superpixels in
one register word, in several, in shared memory (boxes above 128 pixels) and beyond it (above
512), at odd widths, side by side in one word of the bits, and more superpixels than the
launch has warps, against the oracle.  Labels are integers: they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O
from st_spix_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,sp,regions,iters", [
    (40, 33, 4, 20, 9),
    (97, 131, 15, 12, 9),
    (150, 161, 70, 4, 9),           # boxes of 65 to 128 pixels
    (331, 473, 200, 6, 9),          # boxes above 128 pixels
    (523, 607, 600, 2, 5),          # a box above 512 pixels
    (400, 644, 7, 900, 5),          # 6,000 superpixels for 2,432 warps
])
@pytest.mark.parametrize("sp_period", [2, 4])
def test_splits_match_the_oracle(H, W, sp, regions, iters, sp_period):
    from st_spix_gb300 import bist_cuda
    img, _ = synth.voronoi_frame(H, W, regions, 0.03, seed=H)
    cfg = dict(niters=iters, sp_size=sp, sm_period=sp_period)
    lab, p = bist_cuda.run_bass(torch.from_numpy(img).cuda(), **cfg)
    st, ref, _, n = O.run_bass(img, O.default_config(**cfg))
    assert st == 0
    assert p.n == n
    np.testing.assert_array_equal(lab.cpu().numpy(), ref)
