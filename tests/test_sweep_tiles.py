"""The four-sweep launches against the oracle at the edges of their rules: each tile size
(by the frame's number of 32x32 tiles), frames smaller than a halo, ragged rights and
bottoms, sweep counts that leave one to three sweeps to the last launch, tiles whose
relabelled pixels touch more labels than the statistics table holds, and colours outside
[0, 1].  Labels are integers: they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,sp,niters,niters_seg,lo,hi", [
    (5, 7, 3, 8, 4, 0.0, 1.0),              # a frame inside one tile's halo
    (33, 65, 9, 12, 4, 0.0, 1.0),
    (97, 131, 3, 8, 4, 0.0, 1.0),           # 9-pixel superpixels: tables overflow
    (96, 128, 15, 12, 1, 0.0, 1.0),
    (96, 128, 15, 12, 3, -0.6, 1.4),
    (96, 128, 15, 12, 6, 0.0, 1.0),
    (331, 1000, 20, 6, 4, 0.0, 1.0),        # 352 tiles: 32x32 by 256 threads, 331 = 10 x 32 + 11
    (715, 1281, 24, 5, 4, 0.0, 1.0),        # 943 tiles: 64x32 tiles, 715 = 22 x 32 + 11
    (715, 1281, 24, 4, 6, -0.6, 1.4),
    (331, 1000, 20, 5, 5, -0.6, 1.4),
    (961, 1361, 25, 5, 4, 0.0, 1.0),        # 1333 tiles: 64x48 tiles, 961 = 20 x 48 + 1
    (961, 1361, 25, 4, 7, 0.0, 1.0),
])
def test_four_sweep_launches_match_the_oracle(H, W, sp, niters, niters_seg, lo, hi):
    from st_spix_gb300 import bist_cuda, synth
    vid, flows, _ = synth.voronoi_video(H, W, 2, max(3, H * W // 900), 0.05, seed=H + niters_seg,
                                        max_shift=2.0)
    vid = (lo + (hi - lo) * vid).astype(np.float32)
    out = bist_cuda.bist_forward(torch.from_numpy(vid).cuda(), torch.from_numpy(flows).cuda(),
                                 niters, sp, 0.5, 0.009 ** 2, float(np.log(0.5)), 0.0, True, False,
                                 niters_seg=niters_seg, prop_niters=niters)
    st, ref, _ = O.bist_forward(vid, flows, O.default_config(niters=niters, sp_size=sp,
                                                             niters_seg=niters_seg,
                                                             prop_niters=niters), True)
    assert st == 0
    np.testing.assert_array_equal(out.cpu().numpy(), ref)


@pytest.mark.parametrize("H,W,sp,niters,period", [
    (96, 128, 15, 9, 1),         # split and merge in one step: the merge reads the border mask
    (96, 128, 15, 9, 2),
    (97, 131, 9, 10, 3),
    (300, 300, 2, 6, 4),         # 23,000 ids: scans of more than one tile
])
def test_split_merge_periods_match_the_oracle(H, W, sp, niters, period):
    from st_spix_gb300 import bist_cuda, synth
    vid, flows, _ = synth.voronoi_video(H, W, 2, max(3, H * W // 900), 0.05, seed=period,
                                        max_shift=3.0)
    out = bist_cuda.bist_forward(torch.from_numpy(vid).cuda(), torch.from_numpy(flows).cuda(),
                                 niters, sp, 0.5, 0.009 ** 2, float(np.log(0.5)), 0.0, True, False,
                                 sm_period=period, prop_niters=niters)
    glog = bist_cuda.frame_log()
    st, ref, _ = O.bist_forward(vid, flows, O.default_config(niters=niters, sp_size=sp,
                                                             sm_period=period,
                                                             prop_niters=niters), True)
    assert st == 0
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
    olog = O.last_log()
    assert (glog.nsplits, glog.nmerges, glog.nrevived, glog.nminted) == \
        (olog.nsplits, olog.nmerges, olog.nrevived, olog.nminted)
