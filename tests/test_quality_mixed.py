"""Colour and overlap sums where labels hardly repeat in a warp's 32 x 8 block (after 16 rounds
the rest is added pixel by pixel): ids from all alike to one per pixel, blocks that start
regular and turn to noise, partial blocks, colours of a narrow and a wide range."""
import numpy as np
import pytest

from oracle import quality as Q

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ids", [1, 16, 60, 100, 2000])
@pytest.mark.parametrize("T,H,W", [(2, 41, 75), (1, 8, 32), (3, 9, 33)])
@pytest.mark.parametrize("wide", [False, True])
def test_mixed_labels(ids, T, H, W, wide):
    from st_spix_gb300 import metrics
    rng = np.random.default_rng(ids + W)
    vid = rng.uniform(0, 1, (T, H, W, 3)).astype(np.float32)
    if wide:
        vid[..., 0] *= np.float32(1e-6)
    spix = rng.integers(0, ids, (T, H, W)).astype(np.int32)
    spix[:, : H // 2] = np.arange(W, dtype=np.int32) // 8 % ids    # regular rows first
    spix.reshape(-1)[:ids] = np.arange(min(ids, spix.size))        # every id, as far as they go
    S = int(spix.max()) + 1
    gt = rng.integers(0, 3, (T, H, W)).astype(np.int32)
    pooled, down = (a.cpu().numpy() for a in metrics.sp_pooling(vid, spix, S))
    ref = np.zeros((T, S, 3))
    for t in range(T):
        n = np.bincount(spix[t].ravel(), minlength=S)
        for c in range(3):
            ref[t, :, c] = np.bincount(spix[t].ravel(), vid[t, ..., c].ravel().astype(np.float64),
                                       S) / (n + 1e-8)
    # one FP32 rounding of FP64 means of non-negative values
    np.testing.assert_allclose(down, ref, rtol=2.0 ** -23, atol=1e-45)
    np.testing.assert_array_equal(pooled, np.stack([down[t][spix[t]] for t in range(T)]))
    got, want = metrics.computeSummary(vid, gt, spix), Q.compute_summary(vid, spix, gt)
    for k in ("tex", "szv", "ue2d", "sa2d", "ue3d", "sa3d", "spnum", "ave_nsp", "ev", "ev3d"):
        a, b = float(got[k]), float(want[k])
        assert (np.isnan(a) and np.isnan(b)) or abs(a - b) <= 1e-9 * max(abs(b), 1e-300), (k, a, b)
