"""Colour sums of the quality metrics: integer sums scaled to a block's largest exponent, and
FP64 for blocks with a wider range.  Pooled colours are one FP32 rounding (half an ulp, 6e-8)
of FP64 means whose sums err by far less: rtol 2^-23.  Frames whose sizes leave partial
blocks, ids in use that change inside every row, results that are not 16-byte aligned."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _values(kind, rng, shape):
    v = rng.uniform(0, 1, shape)
    if kind == "signed":                   # 8-bit range, negative values
        v = 255 * v - 100
    elif kind == "wide":                   # more than 16 binary orders inside a block
        v = v * 10.0 ** rng.integers(-9, 3, shape)
    elif kind == "tiny":                   # denormals
        v = v * 1e-40
    elif kind == "mixed":                  # exact zeros and values just inside the range
        v = np.where(v < 0.3, 0.0, np.where(v < 0.6, 2.0 ** -16 * (1 + v), 1.0))
    return v.astype(np.float32)


@pytest.mark.parametrize("kind", ["unit", "signed", "wide", "tiny", "mixed"])
@pytest.mark.parametrize("T,H,W", [(2, 37, 53), (3, 5, 700), (1, 64, 64)])
def test_pooled_colours(kind, T, H, W):
    from st_spix_gb300 import metrics
    rng = np.random.default_rng(H + W)
    vid = _values(kind, rng, (T, H, W, 3))
    spix = ((np.arange(H)[:, None] // 6) * 7 + np.arange(W) // 9 + rng.integers(0, 2, (T, H, W)))
    spix = spix.astype(np.int32)
    S = int(spix.max()) + 3
    pooled, down = metrics.sp_pooling(vid, spix, S)
    ref = np.zeros((T, S, 3))
    for t in range(T):
        n = np.bincount(spix[t].ravel(), minlength=S)
        for c in range(3):
            ref[t, :, c] = np.bincount(spix[t].ravel(), vid[t, ..., c].ravel().astype(np.float64),
                                       S) / (n + 1e-8)
    # (signed sums may cancel: the bound is relative to the mean magnitude of the values)
    atol = 2.0 ** -23 * float(np.abs(vid).max()) * (1e-9 if kind != "tiny" else 1) + 1e-45
    np.testing.assert_allclose(down.cpu().numpy(), ref, rtol=2.0 ** -23, atol=atol)
    np.testing.assert_array_equal(pooled.cpu().numpy(),
                                  np.stack([down[t].cpu().numpy()[spix[t]] for t in range(T)]))


def test_infinities_stay_with_their_id():
    from st_spix_gb300 import metrics
    vid = np.full((1, 40, 70, 3), 0.5, np.float32)
    spix = np.tile(np.arange(70, dtype=np.int32) // 10, (1, 40, 1))
    vid[0, 3, 5, 0], vid[0, 9, 25, 1] = np.inf, np.nan
    _, down = metrics.sp_pooling(vid, spix, 7)
    d = down.cpu().numpy()[0]
    assert np.isinf(d[0, 0]) and np.isnan(d[2, 1])
    ok = np.ones((7, 3), bool)
    ok[0, 0] = ok[2, 1] = False
    np.testing.assert_allclose(d[ok], 0.5, rtol=2.0 ** -23)


def test_ids_out_of_range_are_refused():
    from st_spix_gb300 import _lib, metrics
    vid = torch.rand((2, 33, 47, 3), device="cuda")
    spix = torch.zeros((2, 33, 47), dtype=torch.int32, device="cuda")
    spix[1, 32, 46] = 5
    with pytest.raises(_lib.StspixError):
        metrics.sp_pooling(vid, spix, 5)
    spix[1, 32, 46] = -1
    with pytest.raises(_lib.StspixError):
        metrics.sp_pooling(vid, spix, 5)
    counts = metrics.count_spix(spix.clamp(min=0))
    assert counts.cpu().tolist() == [[33 * 47], [33 * 47]]


@pytest.mark.parametrize("sizes", [[(2, 30, 40), (4, 200, 300), (1, 20, 20)]])
def test_calls_on_two_streams_share_no_scratch(sizes):
    """Calls that follow each other on different streams with contexts of their own, and
    calls of growing and shrinking scratch on one stream, give the single-call results."""
    from st_spix_gb300 import metrics
    rng = np.random.default_rng(0)
    ins = []
    for T, H, W in sizes:
        v = torch.from_numpy(rng.uniform(0, 1, (T, H, W, 3)).astype(np.float32)).cuda()
        s = torch.from_numpy(rng.integers(0, 50, (T, H, W)).astype(np.int32)).cuda()
        ins.append((v, s, metrics.sp_pooling(v, s, 64)[1].clone(), metrics.evaluate(v, s, s)))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for rep in range(3):
        outs = []
        for i, (v, s, _, _) in enumerate(ins):
            with torch.cuda.stream(streams[(i + rep) % 2]):
                outs.append((metrics.sp_pooling(v, s, 64)[1], metrics.evaluate(v, s, s)))
        torch.cuda.synchronize()
        for (d, e), (_, _, d0, e0) in zip(outs, ins):
            np.testing.assert_allclose(d.cpu().numpy(), d0.cpu().numpy(), rtol=2.0 ** -23)
            assert abs(e.ev - e0.ev) <= 1e-12 and e.ue2d == e0.ue2d
