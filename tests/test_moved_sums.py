"""After a split the statistics are the halves' sums, after a merge (and the relabel before it
on propagated frames) sums added id to id: against the oracle, which sums the pixels again,
where every iteration splits and merges, where many superpixels are revived or minted, at
colours outside [0, 1] and with superpixels of a few pixels.  Labels, counts and sums are
integers: they must be equal."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from st_spix_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 2, 4])
@pytest.mark.parametrize("H,W,sp,lo,hi", [(24, 40, 3, 0.0, 1.0), (97, 131, 12, 0.0, 1.0),
                                          (97, 131, 12, -0.6, 1.4)])
@pytest.mark.parametrize("iters", [6, 9])
def test_sums_after_each_step(P, H, W, sp, lo, hi, iters):
    from st_spix_gb300 import _lib
    img = (lo + (hi - lo) * synth.voronoi_frame(H, W, 30, 0.05, seed=P + H)[0]).astype(np.float32)
    cfg = dict(niters=12, sp_size=sp, sm_period=P)
    st, o_lab, o, o_n, o_mx = O.bass_partial(img, O.default_config(**cfg), iters, 1)
    assert st == 0
    cap = 30 * O.hex_count(H, W, sp)
    cnt = torch.zeros(cap, dtype=torch.int32, device="cuda")
    sums = torch.zeros(cap * 8, dtype=torch.int64, device="cuda")
    d = _lib.DumpC()
    d.count, d.sums, d.capacity = cnt.data_ptr(), sums.data_ptr(), cap
    ctx = _lib.Context(0)
    lab = torch.zeros((H, W), dtype=torch.int32, device="cuda")
    n, mx = C.c_int(0), C.c_int(0)
    g = torch.from_numpy(img).cuda()
    c = _lib.default_config(**cfg)
    assert ctx.lib.stspix_bass_partial(ctx.handle, torch.cuda.current_stream().cuda_stream,
                                       g.data_ptr(), H, W, C.byref(c), iters, 1, lab.data_ptr(),
                                       C.byref(d), C.byref(n), C.byref(mx)) == 0
    torch.cuda.synchronize()
    ctx.close()
    assert (n.value, mx.value) == (o_n, o_mx)
    np.testing.assert_array_equal(lab.cpu().numpy(), o_lab)
    np.testing.assert_array_equal(cnt.cpu().numpy(), o["count"])
    np.testing.assert_array_equal(sums.cpu().numpy(), o["sums"])


@pytest.mark.parametrize("P", [1, 2, 4])
@pytest.mark.parametrize("H,W,sp,shift,seed", [(48, 64, 5, 9.0, 1), (120, 160, 12, 3.0, 2)])
def test_propagated_frames(P, H, W, sp, shift, seed):
    from st_spix_gb300 import bist_cuda
    vid, flows, _ = synth.voronoi_video(H, W, 3, max(6, H * W // 200), 0.08, seed=seed,
                                        max_shift=shift)
    rng = np.random.default_rng(seed)
    vid[1:] = vid[1:, :, :, rng.permutation(3)]       # colours change: revivals and new ids
    out = bist_cuda.bist_forward(torch.from_numpy(vid).cuda(), torch.from_numpy(flows).cuda(), 9,
                                 sp, 0.5, 0.009 ** 2, float(np.log(0.5)), 0.0, True, False,
                                 sm_period=P, prop_niters=9, thresh_relabel=1e-3, thresh_new=5e-3)
    st, ref, _ = O.bist_forward(vid, flows, O.default_config(niters=9, sp_size=sp, sm_period=P,
                                                             prop_niters=9, thresh_relabel=1e-3,
                                                             thresh_new=5e-3), True)
    assert st == 0
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
