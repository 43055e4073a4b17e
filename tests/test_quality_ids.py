"""Overlap scores with very many ground-truth ids (more than 65,535 blocks of 256 of them)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_an_id_per_pixel():
    from st_spix_gb300 import metrics
    H, W = 4096, 4200
    vid = torch.rand((1, H, W, 3), device="cuda")
    spix = torch.zeros((1, H, W), dtype=torch.int32, device="cuda")
    spix[:, :, W // 2:] = 1
    gt = torch.arange(H * W, dtype=torch.int32, device="cuda").reshape(1, H, W)
    s = metrics.computeSummary(vid, gt, spix)
    # every ground-truth id overlaps one superpixel in one pixel: min(out, in) = 1, and no
    # superpixel lies at least half inside it
    assert s["ue2d"] == pytest.approx(1.0 / (H * W), rel=1e-9)
    assert s["ue3d"] == pytest.approx(1.0 / (H * W), rel=1e-9)
    assert s["sa2d"] == 0 and s["sa3d"] == 0


def test_a_missing_id_is_named():
    from st_spix_gb300 import _lib, metrics
    vid = torch.rand((1, 16, 16, 3), device="cuda")
    spix = torch.zeros((1, 16, 16), dtype=torch.int32, device="cuda")
    gt = torch.ones_like(spix)
    gt[0, 0, 0] = 20_000_000
    with pytest.raises(_lib.StspixError, match="id 0 of 0..20000000 never occurs"):
        metrics.computeSummary(vid, gt, spix)
