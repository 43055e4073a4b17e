"""stspix_sp_pooling with ids out of range: refused, and the outputs stay as they were."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [-1, 9, 2 ** 31 - 1, -2 ** 31])
def test_outputs_stay_untouched(bad):
    from st_spix_gb300 import _lib, bist_cuda
    T, H, W, n = 2, 37, 53, 9
    vid = torch.rand((T, H, W, 3), device="cuda")
    spix = torch.randint(0, n, (T, H, W), dtype=torch.int32, device="cuda")
    spix[1, 20, 30] = bad
    down = torch.full((T, n, 3), 7.0, device="cuda")
    pooled = torch.full((T, H, W, 3), 7.0, device="cuda")
    ctx = bist_cuda._ctx(vid.device)
    st = ctx.lib.stspix_sp_pooling(ctx.handle, bist_cuda._stream(vid.device), vid.data_ptr(),
                                   spix.data_ptr(), T, H, W, n, pooled.data_ptr(),
                                   down.data_ptr())
    torch.cuda.synchronize()
    assert st == _lib.STSPIX_ERR_ARG
    assert bool((down == 7.0).all()) and bool((pooled == 7.0).all())
