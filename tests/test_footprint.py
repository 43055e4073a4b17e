"""stspix_footprint against the buffers of engine.h counted by hand, and the serving form's use
of it."""
import types

import pytest

from st_spix_gb300 import _lib, bist_cuda, serve

# bytes per pixel of a slot: border, d1 d2 smseg hits shifted, best, seg_alt, two change planes
PIX = 1 + 5 * 4 + 8 + 4 + 2
# per id: the working state (twice), split/merge scratch, the other per-id arrays
STATE = (4 + 1 + 1 + 4 + 4 + 4 + 3 * 4 + 2 * 8 + 3 * 8 + 8 + 3 * 4 + 2 * 8 + 3 * 8 + 3 * 8 + 3 * 8
         + 8 * 8 + 48)
SPLIT_MERGE = 4 + 3 * 8 + 3 * 8 + 5 * 8 + 5 * 4 + 1 + 8
OTHER = (5 * 1 + 6 * 4 + 2 * 8 + 2 * 4 + 4 + 2 * 8 + 16 + 8 + 8     # flags .. ccbest
         + 4 * 4 + 9 * 8 + 1 + 3 * 8)                               # bbox, snap, recchg, pscache
PARAMS = 2 * (3 * 4 + 3 * 4 + 2 * 8 + 3 * 8 + 4 + 2 * 8 + 3 * 8 + 3 * 8 + 5 * 4)


@pytest.mark.parametrize("H,W,sp", [(480, 854, 20), (72, 96, 15), (2, 2, 40), (481, 855, 7)])
def test_every_buffer_is_counted(H, W, sp):
    video, slot = _lib.footprint(H, W, sp)
    cap = max(30 * bist_cuda.hex_count(H, W, sp), 64)
    # (each of fewer than 128 buffers is rounded up to 16 bytes, some hold two ids more)
    slack = 128 * 16 + 2 * (SPLIT_MERGE + OTHER)
    want = PIX * H * W + (2 * STATE + SPLIT_MERGE + OTHER) * cap
    assert want <= slot <= want + slack
    want = 4 * H * W + PARAMS * cap
    assert want <= video <= want + slack


@pytest.mark.parametrize("lab", [0, 1])
def test_a_served_slot_counts_the_converted_frame(lab):
    s = serve.Server.__new__(serve.Server)
    s._lib, s.sp_default, s.cfg = _lib, 15, {"lab_ingest": lab}
    req = types.SimpleNamespace(vid=types.SimpleNamespace(shape=(3, 120, 160, 3)), sp_size=0)
    assert s.slot_bytes(req) == _lib.footprint(120, 160, 15)[1] + lab * 12 * 120 * 160
