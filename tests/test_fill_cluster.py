"""The hole fill by one block, by a cluster of blocks and by the loop over all SMs, on either
side of the hole counts where one hands over to the next, against the oracle: labels after
the shift and after the fill, with frames moved far enough that the fill takes hundreds of
iterations or stops at its limit, and for several streams of different counts at
once, replayed from graphs too.  Labels are integers: they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O
from st_spix_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def labelled(H, W, sp, seed):
    img, _ = synth.voronoi_frame(H, W, max(4, H * W // 4000), 0.05, seed=seed)
    st, lab, p, n = O.run_bass(img, O.default_config(niters=1, sp_size=sp))
    assert st == 0
    return lab, p, n


def gpu_params(op, n):
    from st_spix_gb300 import bist_cuda
    p = bist_cuda.SuperpixelParams(n, "cuda")
    p.n = n
    for name, dt, per in bist_cuda.PARAM_FIELDS:
        getattr(p, "_" + name).copy_(torch.from_numpy(np.ascontiguousarray(op[name]).reshape(-1)))
    return p


@pytest.mark.parametrize("H,W,sp,dx,dy", [
    (37, 53, 7, 3.0, 1.0),              # one block
    (96, 128, 9, 40.0, -20.0),          # 5,600 holes: a cluster; 45 iterations
    (130, 700, 20, 300.0, 0.0),
    (24, 1300, 12, 1200.0, 0.0),        # stops at the iteration limit
    (300, 1000, 30, 890.0, 0.0),        # 267,000 holes: above a cluster of 16 blocks
    (620, 700, 40, 300.0, 200.0),
    (280, 1400, 40, 1300.0, 0.0),       # above, and stops at the limit
])
def test_fill_matches_the_oracle(H, W, sp, dx, dy):
    from st_spix_gb300 import bist_cuda
    lab, p, n = labelled(H, W, sp, seed=H)
    rng = np.random.default_rng(W)
    flow = (np.array([dx, dy]) + rng.uniform(-1.5, 1.5, (H, W, 2))).astype(np.float32)
    st, filled, shifted, _ = O.shift_and_fill(lab, p, n, flow)
    assert st == 0
    gf, gs = bist_cuda.shift_and_fill(torch.from_numpy(lab).cuda(), gpu_params(p, n),
                                      torch.from_numpy(flow).cuda())
    np.testing.assert_array_equal(gs.cpu().numpy(), shifted)
    np.testing.assert_array_equal(gf.cpu().numpy(), filled)


@pytest.mark.parametrize("B", [3, 9])
def test_streams_with_different_hole_counts(B):
    """Clusters of 16 and of 8 blocks (more than 8 slots), each slot with its own motion;
    from the third frame on the batch step is a replayed graph."""
    from st_spix_gb300 import batch
    T, cfg = 5, dict(niters=6, sm_period=4, prop_niters=6, sp_size=9)
    vids = [synth.voronoi_video(64 + 32 * (i % 3), 96, T, 20, 0.05, seed=i, max_shift=1.0 + 6.0 * i)
            for i in range(B)]
    refs = []
    for vid, flows, _ in vids:
        st, ref, _ = O.bist_forward(vid, flows, O.default_config(**cfg), True)
        assert st == 0
        refs.append(ref)
    gpu = [(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()) for v, f, _ in vids]
    vs = [batch.Video(v.shape[1], v.shape[2]) for v, _ in gpu]
    for t in range(T):
        fr = [batch.Frame(img=v[t], flow=f[t - 1] if t else None, video=h)
              for (v, f), h in zip(gpu, vs)]
        batch.process_batch(fr, **cfg)
        for f, ref in zip(fr, refs):
            assert f.status == 0
            np.testing.assert_array_equal(f.labels.cpu().numpy(), ref[t])
    for h in vs:
        h.close()
