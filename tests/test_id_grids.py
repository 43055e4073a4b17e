"""Per-id kernels launch a bounded number of blocks per slot, which loop over the slot's ids
and take their slots in rotated rows: a large frame with several rounds of ids (and of ids in
use for the decisions) beside frames with a few, as a batch and alone, against the oracle.
Labels are integers: they must be equal."""
import numpy as np
import pytest

from oracle import oracle as O
from st_spix_gb300 import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,at", [(24, 0), (24, 17), (3, 2), (1, 0)])
def test_large_frame_among_small_ones(n, at):
    from st_spix_gb300 import batch
    cfg = dict(niters=9, sm_period=4)
    # 5,000 ids in use of 150,000: at 24 frames a slot has 51 blocks of 32 or 256 ids
    sizes = [(8 + 8 * (i % 4), 24, 4 + i % 3) for i in range(n)]
    sizes[at] = (200, 328, 4)
    imgs = [synth.voronoi_frame(h, w, max(2, h * w // 40), 0.05, 7 * i + h)[0]
            for i, (h, w, _) in enumerate(sizes)]
    fr = [batch.Frame(img=torch.from_numpy(im).cuda(), sp_size=sp)
          for im, (_, _, sp) in zip(imgs, sizes)]
    batch.process_batch(fr, **cfg)
    for f, im, (_, _, sp) in zip(fr, imgs, sizes):
        st, lab, _, k = O.run_bass(im, O.default_config(sp_size=sp, **cfg))
        assert st == 0 and f.status == 0
        assert f.nspix == k
        np.testing.assert_array_equal(f.labels.cpu().numpy(), lab)
