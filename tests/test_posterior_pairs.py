"""The posterior's shortened arithmetic against the oracle's FP64 division and log at the
inputs where it decides between its pairs of floats and FP64: colour means that are exact or
lie half way between two floats, negative and large sums, superpixels of a few pixels (their
covariance is degenerate) and shapes of every determinant between.  Labels, counts and the
FP32 parameters must be equal (an FP32 value is the rounding of the FP64 one), FP64 ones to
1e-12, as in the parity tests (the inverse covariances and means are quotients, equal too, of
sums both sides hold exactly)."""
import numpy as np
import pytest

from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def frame(kind, H, W):
    rng = np.random.default_rng(len(kind) * 1000 + H)
    img = rng.integers(0, 256, (H // 8 + 1, W // 8 + 1, 3)).repeat(8, 0).repeat(8, 1)[:H, :W] / 255
    if kind == "flat":
        return np.full((H, W, 3), 0.625, np.float32)
    if kind == "ties":        # multiples of 2^-26 next to 1/2: means between two floats
        return (0.5 + rng.integers(0, 8, (H, W, 3)) * 2.0 ** -26 + (img > 0.5) * 0.25).astype(np.float32)
    if kind == "dark":
        return (img * 2.0 ** -20).astype(np.float32)
    if kind == "negative":
        return (img - 1.0).astype(np.float32)
    if kind == "large":
        return (img * 4000 - 1000).astype(np.float32)
    return (img + 0.05 * rng.random((H, W, 3))).clip(0, 1).astype(np.float32)


@pytest.mark.parametrize("kind", ["flat", "ties", "dark", "negative", "large", "noise"])
@pytest.mark.parametrize("H,W,sp", [(5, 7, 2), (64, 33, 3), (96, 128, 15), (130, 70, 40)])
def test_parameters_match_the_oracle(kind, H, W, sp):
    from st_spix_gb300 import bist_cuda
    img = frame(kind, H, W)
    lab, p = bist_cuda.run_bass(torch.from_numpy(img).cuda(), sp_size=sp, niters=10, sm_period=4)
    st, ref, op, n = O.run_bass(img, O.default_config(niters=10, sp_size=sp, sm_period=4))
    assert st == 0
    assert p.n == n
    np.testing.assert_array_equal(lab.cpu().numpy(), ref)
    for name, g in p.as_dict().items():
        g = g.detach().cpu().numpy().reshape(-1)
        o = np.asarray(op[name]).reshape(-1)
        if g.dtype == np.float64:
            np.testing.assert_allclose(g, o, rtol=1e-12, atol=0, err_msg=name)
        else:
            np.testing.assert_array_equal(g, o, err_msg=name)
