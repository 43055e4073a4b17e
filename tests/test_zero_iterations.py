"""Frames without iterations beside frames with some: the closing posterior of the former is
their first, and reads nothing of the frame that held the workspace before."""
import numpy as np
import pytest

from st_spix_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("new_first", [True, False])
def test_zero_iterations_beside_a_propagated_frame(graphs, new_first):
    from st_spix_gb300 import batch, bist_cuda
    H, W, cfg = 61, 83, dict(sp_size=9, sm_period=4)
    img = torch.from_numpy(synth.voronoi_frame(H, W, 12, 0.05, seed=1)[0]).cuda()
    other = torch.from_numpy(synth.voronoi_frame(H, W, 30, 0.08, seed=2)[0]).cuda()
    vid, flows, _ = synth.voronoi_video(H, W, 2, 14, 0.05, seed=3, max_shift=2.0)
    vid, flow = torch.from_numpy(vid).cuda(), torch.from_numpy(flows[0]).cuda()

    def videos():
        new, old = batch.Video(H, W), batch.Video(H, W)
        batch.process_batch([batch.Frame(img=vid[0], video=old)], niters=5, **cfg)
        return new, old

    def frames(new, old):
        return [batch.Frame(img=img, video=new), batch.Frame(img=vid[1], flow=flow, video=old)]

    # each alone
    new, old = videos()
    for f in frames(new, old):
        batch.process_batch([f], niters=0, prop_niters=3, **cfg)
    ref = [new.save(), old.save()]
    # together, after the workspace held other frames of these sizes
    ctx = bist_cuda._ctx(img.device)
    ctx.set_batch_graphs(graphs)
    try:
        for _ in range(3):
            new, old = videos()
            batch.process_batch([batch.Frame(img=other), batch.Frame(img=other)], niters=6, **cfg)
            fr = frames(new, old)
            batch.process_batch(fr if new_first else fr[::-1], niters=0, prop_niters=3, **cfg)
            assert [f.niters for f in fr] == [0, 3]
            for a, b in zip((new, old), ref):
                np.testing.assert_array_equal(np.frombuffer(a.save(), np.uint8),
                                              np.frombuffer(b, np.uint8))
    finally:
        ctx.set_batch_graphs(True)
