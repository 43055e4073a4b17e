"""The two-float forms of the CIELAB conversion (st_spix_gb300/csrc/k_color.cu lin_ff, f_ff and
the outputs) restated in numpy: wherever ff_round accepts an argument of powf it is the
float that the FP64 steps round to, and it accepts nearly all; the outputs are equal.  On the GPU, against the FP64 steps around
torch's powf, to the tolerance that powf's few ulps leave."""
import numpy as np
import pytest

F = np.float32
MARGIN = F(2.0 ** -43)


def fma(a, b, c):
    # the product of two floats is exact in a double
    return (np.asarray(a, np.float64) * np.asarray(b, np.float64) + np.asarray(c, np.float64)).astype(F)


def const(x):
    return F(x), F(x - float(F(x)))


def sum_err(a, b, s):
    bb = s - a
    return (a - (s - bb)) + (b - bb)


def mul_err(ah, al, k, p):
    return fma(al, k[0], fma(ah, k[1], fma(ah, k[0], -p)))


def ff_round(h, e, margin):
    up, dn = h + (e + margin), h + (e - margin)
    return up, up == dn


def values(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.uniform(0, 1, n)
    v[: n // 4] = rng.integers(0, 256, n // 4) / 255.0
    v[n // 4: n // 2] = rng.uniform(-0.5, 3.0, n // 4)
    return v.astype(F)


def test_linearisation_rounds_as_fp64():
    c = values(400000, 0)
    c = c[c > F(0.04045)]
    a, k = const(0.055), const(1 / 1.055)
    s = c + a[0]
    tl = sum_err(c, a[0], s) + a[1]
    p = s * k[0]
    x, ok = ff_round(p, mul_err(s, tl, k, p), p * MARGIN)
    ref = ((c.astype(np.float64) + 0.055) / 1.055).astype(F)
    np.testing.assert_array_equal(x[ok], ref[ok])
    assert ok.mean() > 0.999


def test_division_by_constants_is_correctly_rounded():
    """div_const with the fused multiply-adds in exact rational arithmetic."""
    from fractions import Fraction
    rng = np.random.default_rng(8)
    for b in (12.92, 1.055, 116.0, 0.950456, 1.088754):
        y = 1.0 / b
        x = np.concatenate([rng.uniform(0, 30, 2000), np.exp2(rng.uniform(-80, 80, 2000)),
                            # near the quotients' rounding boundaries
                            (rng.uniform(0, 1, 4000) + 2.0 ** -54) * b])
        for v in x.tolist():
            q = v * y
            r = float(Fraction(v) - Fraction(b) * Fraction(q))
            assert float(Fraction(q) + Fraction(r) * Fraction(y)) == v / b, (v, b)


def test_dark_branch_rounds_as_fp64():
    r, g, b = (abs(values(200000, s)) * F(0.03) for s in (9, 10, 11))
    for c in (r, g, b):
        c[::9] *= F(-3)                             # negative sums: 116 f below 8
    k = const(1 / 12.92)
    ff, f64 = [], []
    for (kr, kg, kb, white) in ((0.4124564, 0.3575761, 0.1804375, 0.950456),
                                (0.2126729, 0.7151522, 0.0721750, 1.0)):
        ks = [const(q / white) for q in (kr, kg, kb)]
        pairs = [(c * k[0], mul_err(c, F(0), k, c * k[0])) for c in (r, g, b)]
        ps = [h * q[0] for (h, _), q in zip(pairs, ks)]
        s = ps[0] + ps[1]
        v = s + ps[2]
        errs = [mul_err(h, l, q, p) for (h, l), q, p in zip(pairs, ks, ps)]
        e = ((errs[0] + errs[1]) + errs[2]) + (sum_err(ps[0], ps[1], s) + sum_err(s, ps[2], v))
        kappa, inv = const(903.3), const(1 / 116.0)
        p = v * kappa[0]
        t = p + F(16)
        w = mul_err(v, e, kappa, p) + sum_err(p, F(16), t)
        q = t * inv[0]
        ff.append((q, mul_err(t, w, inv, q)))
        x = sum(c.astype(np.float64) / 12.92 * m for c, m in zip((r, g, b), (kr, kg, kb))) / white
        f64.append((903.3 * x + 16.0) / 116.0)
    (xh, xl), (yh, yl) = ff
    p = F(116) * yh
    s = p - F(16)
    lab, ok = ff_round(s, fma(F(116), yl, fma(F(116), yh, -p)) + sum_err(p, F(-16), s),
                       F(2.0 ** -38))
    np.testing.assert_array_equal(lab[ok], (116.0 * f64[1] - 16.0).astype(F)[ok])
    assert ok.mean() > 0.99
    d = xh - yh
    lo = sum_err(xh, -yh, d) + (xl - yl)
    q = F(500) * d
    a, ok = ff_round(q, fma(F(500), lo, fma(F(500), d, -q)), F(2.0 ** -35))
    np.testing.assert_array_equal(a[ok], (500.0 * (f64[0] - f64[1])).astype(F)[ok])
    assert ok.mean() > 0.99


def test_tristimulus_rounds_as_fp64():
    rng = np.random.default_rng(1)
    r, g, b = (values(200000, s) for s in (2, 3, 4))
    dark = rng.uniform(0, 1, r.size) < 0.2
    # a channel of the linear branch is a pair, the others single floats
    k = const(1 / 12.92)
    rh = np.where(dark, F(0.04) * r * k[0], r).astype(F)
    rl = np.where(dark, mul_err(F(0.04) * r, F(0), k, F(0.04) * r * k[0]), F(0)).astype(F)
    r64 = np.where(dark, (F(0.04) * r).astype(np.float64) / 12.92, r.astype(np.float64))
    for (kr, kg, kb, white) in ((0.4124564, 0.3575761, 0.1804375, 0.950456),
                                (0.2126729, 0.7151522, 0.0721750, 1.0),
                                (0.0193339, 0.1191920, 0.9503041, 1.088754)):
        ks = [const(q / white) for q in (kr, kg, kb)]
        ps = [rh * ks[0][0], g * ks[1][0], b * ks[2][0]]
        s = ps[0] + ps[1]
        v = s + ps[2]
        e = ((mul_err(rh, rl, ks[0], ps[0]) + mul_err(g, F(0), ks[1], ps[1])) +
             mul_err(b, F(0), ks[2], ps[2])) + (sum_err(ps[0], ps[1], s) + sum_err(s, ps[2], v))
        x, ok = ff_round(v, e, (abs(ps[0]) + abs(ps[1]) + abs(ps[2])) * MARGIN)
        ref = ((r64 * kr + g.astype(np.float64) * kg + b.astype(np.float64) * kb) / white).astype(F)
        np.testing.assert_array_equal(x[ok], ref[ok])
        assert ok.mean() > 0.999


def test_outputs_round_as_fp64():
    fx, fy = values(400000, 5), values(400000, 6)
    fx, fy = abs(fx) + F(0.2), abs(fy) + F(0.2)
    fx[::5] = fy[::5] * F(1 + 2.0 ** -20)          # near-grey: the difference cancels
    fx[1::5] *= F(4.7)                              # up to the bound of 16
    p = F(116) * fy
    ref = (116.0 * fy.astype(np.float64) - 16.0).astype(F)
    np.testing.assert_array_equal((p - F(16)) + fma(F(116), fy, -p), ref)
    d = fx - fy
    p = F(500) * d
    x = p + fma(F(500), sum_err(fx, -fy, d), fma(F(500), d, -p))
    ref = (500.0 * (fx.astype(np.float64) - fy.astype(np.float64))).astype(F)
    np.testing.assert_array_equal(x, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("first_blue", [1, 0])
def test_conversion_edges(first_blue):
    """Dark, out-of-gamut, infinite and NaN pixels next to ordinary ones, an odd pixel count."""
    torch = pytest.importorskip("torch")
    from st_spix_gb300 import bist_cuda, prop_cuda
    v = values(3 * 4999, 7).reshape(-1, 3)
    v[::7] *= F(0.05)
    v[11] = [np.nan, 0.5, 0.5]
    v[12] = 0.0
    g = torch.from_numpy(v).cuda()
    out = (bist_cuda.rgb2lab if first_blue else prop_cuda.rgb_to_lab)(g)
    assert torch.equal(out[11], g[11]) or bool(torch.isnan(out[11, 0]))
    assert out[11, 1] == 0.5 and out[11, 2] == 0.5
    ch = g.double() if not first_blue else g.double().flip(1)
    lin = torch.where(ch <= 0.04045, ch / 12.92,
                      torch.pow(((ch + 0.055) / 1.055).float(), 2.4).double())
    m = torch.tensor([[0.4124564, 0.3575761, 0.1804375], [0.2126729, 0.7151522, 0.0721750],
                      [0.0193339, 0.1191920, 0.9503041]], dtype=torch.float64, device="cuda")
    xyz = lin @ m.T / torch.tensor([0.950456, 1.0, 1.088754], dtype=torch.float64, device="cuda")
    f = torch.where(xyz > 0.008856, torch.pow(xyz.float(), 1.0 / 3.0).double(),
                    (903.3 * xyz + 16.0) / 116.0)
    ref = torch.stack([(116 * f[:, 1] - 16) / -100, 5 * (f[:, 0] - f[:, 1]),
                       2 * (f[:, 1] - f[:, 2])], 1)
    keep = torch.ones(len(v), dtype=torch.bool, device="cuda")
    keep[11] = False
    # powf: 2 ulps in each of two steps of values up to 3, times 5 in the differences
    torch.testing.assert_close(out[keep].double(), ref[keep], rtol=0, atol=5 * 3 * 8 * 2.0 ** -23)
