"""The hole fill on either side of the largest count a cluster of 16 blocks takes (16 x 12,288),
against the oracle.  Labels are integers: they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O
from test_fill_cluster import gpu_params, labelled

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(192, 1400), (256, 1100)])
@pytest.mark.parametrize("more", [-1, 0, 1, 40])
def test_fill_at_the_limit(H, W, more):
    """A shift by whole columns leaves H dx holes: 16 x 12,288 is 192 x 1024 and 256 x 768."""
    from st_spix_gb300 import bist_cuda
    dx = 16 * 12288 // H + more
    lab, p, n = labelled(H, W, 40, seed=more + 5)
    flow = np.zeros((H, W, 2), np.float32)
    flow[..., 0] = dx
    st, filled, shifted, _ = O.shift_and_fill(lab, p, n, flow)
    assert st == 0 and int((shifted < 0).sum()) == H * dx
    gf, gs = bist_cuda.shift_and_fill(torch.from_numpy(lab).cuda(), gpu_params(p, n),
                                      torch.from_numpy(flow).cuda())
    np.testing.assert_array_equal(gs.cpu().numpy(), shifted)
    np.testing.assert_array_equal(gf.cpu().numpy(), filled)
