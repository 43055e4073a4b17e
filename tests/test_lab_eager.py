"""stspix_config.lab_ingest on the paths that launch every step (graphs disabled, profiling on):
the labels of the default path."""
import numpy as np
import pytest

from helpers import small_video

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [False, True])
@pytest.mark.parametrize("video_mode", [False, True])
def test_lab_ingest_launched_step_by_step(video_mode, profile):
    from st_spix_gb300 import bist_cuda
    vid, flows = small_video(T=3)
    gv, gf = torch.from_numpy(vid).cuda(), torch.from_numpy(flows).cuda()
    args = (12, 15, 0.5, 0.009 ** 2, float(np.log(0.5)), 0.0, video_mode, False)
    first = bist_cuda.bist_forward(bist_cuda.rgb2lab(gv), gf, *args)
    # (the buffer of converted frames has held others)
    bist_cuda.bist_forward(gv.flip(0).contiguous(), gf, *args, lab_ingest=1)
    ctx = bist_cuda._ctx(gv.device)
    ctx.profile(profile)
    ctx.set_batch_graphs(False)
    try:
        out = bist_cuda.bist_forward(gv, gf, *args, lab_ingest=1)
    finally:
        ctx.profile(False)
        ctx.set_batch_graphs(True)
    assert torch.equal(out, first)
