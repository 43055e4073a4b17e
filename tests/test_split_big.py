"""Splits of superpixels whose boxes a block searches in shared memory (129 to 512 pixels) or in
global memory (above), at the edges of its words and rows: a frame of one or a few superpixels,
whose boxes are the frame, against the oracle.  Labels are integers: they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O
from st_spix_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(129, 40), (40, 129), (70, 191), (70, 192), (70, 193), (512, 33),
                                 (513, 33), (33, 512), (33, 513), (300, 449)])
def test_frames_of_one_superpixel(H, W):
    from st_spix_gb300 import bist_cuda
    img, _ = synth.voronoi_frame(H, W, 3, 0.03, seed=H + W)
    cfg = dict(niters=7, sp_size=1000, sm_period=2)
    lab, p = bist_cuda.run_bass(torch.from_numpy(img).cuda(), **cfg)
    st, ref, _, n = O.run_bass(img, O.default_config(**cfg))
    assert st == 0 and p.n == n
    np.testing.assert_array_equal(lab.cpu().numpy(), ref)


def test_large_boxes_of_a_propagated_video():
    from st_spix_gb300 import bist_cuda
    cfg = dict(niters=9, sp_size=180, sm_period=4, prop_niters=9)
    vid, flows, _ = synth.voronoi_video(290, 420, 3, 6, 0.03, seed=4, max_shift=3.0)
    st, ref, _ = O.bist_forward(vid, flows, O.default_config(**cfg), True)
    assert st == 0
    out = bist_cuda.bist_forward(torch.from_numpy(vid).cuda(), torch.from_numpy(flows).cuda(), 9,
                                 180, 0.5, 0.009 ** 2, float(np.log(0.5)), 0.0, True, False,
                                 sm_period=4, prop_niters=9)
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
