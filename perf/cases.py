"""The work whose speed this repository is kept to: superpixel labelling of frames and
videos through the public entry points, over the sizes users run (a few thousand pixels
to 4K), and the steps around it (label propagation, border overlay, quality scores,
pooling, colour ingest).

Scenes are the package's seeded synthetic ones (Voronoi regions with noise and affine
motion) at the densities and noise levels of its tests and benchmark; every input is a
function of the case and the seed.

    listed()            the fixed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what a program holds before the call (inputs, streams)
    run(state)          one pass; its outputs
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits, where they are computed numbers
"""
import math

import torch

from st_spix_gb300 import batch, bist_cuda, metrics, synth

LOG_HALF = math.log(0.5)
SIGMA2_APP = 0.009 ** 2
POTTS = 0.5


# ---------------------------------------------------------------------------
# cases
def listed():
    return [
        # the smallest call: one thumbnail-sized frame, default configuration, with the
        # superpixel parameters a caller keeps (the size of the parity tests)
        dict(name="bass_72x96", kind="bass", H=72, W=96, regions=24, noise=0.05, sp_size=15,
             niters=15, sm_period=4),
        # one segmentation-benchmark image run to convergence: 100 iterations
        dict(name="image_240x320_n100", kind="image", H=240, W=320, T=1, regions=200, noise=0.05,
             sp_size=15, niters=100, sm_period=20),
        # a video as the reference's scripts run it: frame after frame, iteration count of
        # a propagated frame by the hole fraction (4, 8 or 12)
        dict(name="video_480x854_ladder", kind="video", H=480, W=854, T=4, regions=400,
             noise=0.03, sp_size=20, niters=20, sm_period=4, prop_niters=0),
        # eight concurrent streams, one batch per time step: the streaming workload
        dict(name="streams8_480x854", kind="streams", B=8, H=480, W=854, T=3, regions=400,
             noise=0.03, sp_size=20, niters=20, sm_period=10, prop_niters=20),
        # one live 720p stream: latency of a frame at a time
        dict(name="stream_720x1280", kind="streams", B=1, H=720, W=1280, T=3, regions=900,
             noise=0.03, sp_size=20, niters=20, sm_period=10, prop_niters=20),
        # an offline batch of independent images of uneven size
        dict(name="batch16_uneven", kind="batch", n=16, sizes=7, lo=240, hi=1080, step=8,
             niters=20, sm_period=10),
        # the largest frames: 4K video
        dict(name="video_2160x3840", kind="video", H=2160, W=3840, T=2, regions=2000, noise=0.03,
             sp_size=25, niters=20, sm_period=10, prop_niters=20),
        # label propagation alone, ragged size: shift by the mean flow and hole filling
        dict(name="shift_fill_481x855", kind="shift", H=481, W=855, regions=400, noise=0.03,
             sp_size=20, niters=20, sm_period=10),
        # borders painted over a labelled clip, as for display
        dict(name="marked_480x854_T8", kind="marked", H=480, W=854, T=8, regions=400, noise=0.03,
             sp_size=20),
        # all quality scores of a labelled clip with ground truth, as an evaluation does
        dict(name="evaluate_480x854_T8", kind="evaluate", H=480, W=854, T=8, regions=400,
             noise=0.03, sp_size=20),
        # superpixel-pooled colours of a labelled clip
        dict(name="pooling_480x854_T8", kind="pooling", H=480, W=854, T=8, regions=400,
             noise=0.03, sp_size=20),
        # 8-bit ingest of a 1080p frame: scaling to float and conversion to CIELAB
        dict(name="lab_1080x1920", kind="lab", H=1080, W=1920),
    ]


def _size(rng, lo_pix, hi_pix):
    """H and W of a frame with lo_pix..hi_pix pixels (spread over their logarithm) and an
    aspect between 1:2 and 2:1, odd values included."""
    n = math.exp(rng.uniform(math.log(lo_pix), math.log(hi_pix)))
    a = math.exp(rng.uniform(-math.log(2.0), math.log(2.0)))
    return max(16, int(round(math.sqrt(n / a)))), max(16, int(round(math.sqrt(n * a))))


def _scene(rng, H, W):
    area = math.exp(rng.uniform(math.log(350.0), math.log(4000.0)))   # pixels per region
    return dict(H=H, W=W, regions=max(4, int(H * W / area)), noise=round(rng.uniform(0.02, 0.08), 3),
                sp_size=rng.choice([12, 15, 16, 20, 25]))


def draw(rng):
    kind = rng.choice(["bass", "image", "video", "streams", "batch", "large", "shift", "marked",
                       "evaluate", "pooling", "lab"])
    sched = dict(niters=rng.randint(10, 24), sm_period=rng.choice([4, 10]))
    if kind == "bass":
        return dict(kind=kind, **_scene(rng, *_size(rng, 4e3, 1e5)), **sched)
    if kind == "image":
        return dict(kind=kind, T=rng.randint(1, 2), **_scene(rng, *_size(rng, 4e4, 4e5)),
                    niters=rng.randint(30, 100), sm_period=rng.choice([4, 20]))
    if kind == "video":
        return dict(kind=kind, T=rng.randint(2, 5), **_scene(rng, *_size(rng, 5e4, 9e5)), **sched,
                    prop_niters=rng.choice([0, 0, 12]))
    if kind == "streams":
        B = rng.randint(1, 8)
        return dict(kind=kind, B=B, T=rng.randint(2, 3),
                    **_scene(rng, *_size(rng, 1e5, min(2e6, 4e6 / B))), **sched,
                    prop_niters=rng.choice([0, 12, 20]))
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(3, 16), sizes=rng.randint(0, 10 ** 6), lo=240, hi=1080,
                    step=rng.choice([1, 8]), **sched)
    if kind == "large":
        s = _scene(rng, *_size(rng, 2e6, 6e6))
        s.update(regions=1500, sp_size=25, niters=rng.randint(10, 20), prop_niters=12)
        return dict(kind="video", T=rng.randint(1, 2), **s, sm_period=sched["sm_period"])
    if kind == "shift":
        return dict(kind=kind, **_scene(rng, *_size(rng, 2e4, 2e6)), **sched)
    if kind == "lab":
        H, W = _size(rng, 1e4, 8e6)
        return dict(kind=kind, H=H, W=W)
    s = _scene(rng, *_size(rng, 3e4, 1e6))
    s["regions"] = min(s["regions"], 600)
    return dict(kind=kind, T=rng.randint(2, 10), **s)


# ---------------------------------------------------------------------------
# inputs
def _uneven(case):
    """Sizes, superpixel sizes and scenes of the frames of a batch (of the case alone, so
    every seed gives other pixels of the same sizes)."""
    import random
    r = random.Random(case["sizes"])
    lo, hi, step = case["lo"], case["hi"], case["step"]
    out = []
    for _ in range(case["n"]):
        out.append((r.randint(lo, hi) // step * step, r.randint(lo, hi) // step * step,
                    r.randint(100, 800), round(r.uniform(0.02, 0.08), 3),
                    r.choice([12, 16, 20, 25])))
    return out


def _video(case, seed, T, regions=False):
    return synth.voronoi_video_device(case["H"], case["W"], T, case["regions"], case["noise"],
                                      seed=seed, regions=regions)


def _forward(vid, flows, case, video_mode, **kw):
    return bist_cuda.bist_forward(vid, flows, case.get("niters", 20), case["sp_size"], POTTS,
                                  SIGMA2_APP, LOG_HALF, 0.0, video_mode, False,
                                  sm_period=case.get("sm_period", 10), **kw)


def _bass_kw(case):
    return dict(niters=case["niters"], sp_size=case["sp_size"], potts=POTTS,
                sigma2_app=SIGMA2_APP, alpha=LOG_HALF, sm_period=case["sm_period"])


def _whole(params, names=None):
    """The parameter arrays as allocated (rows beyond params.n are zero): their shape does
    not depend on how many superpixels the frame ended with."""
    return {f[0]: getattr(params, "_" + f[0]) for f in bist_cuda.PARAM_FIELDS
            if names is None or f[0] in names}


def prepare(case, seed):
    k = case["kind"]
    s = dict(case=dict(case), kind=k)
    if k == "bass":
        s["img"] = _video(case, seed, 1)[0][0].contiguous()
    elif k in ("image", "video"):
        s["vid"], s["flows"] = _video(case, seed, case["T"])
    elif k == "streams":
        s["vids"] = [_video(case, 1000 * seed + b, case["T"]) for b in range(case["B"])]
        s["streams"] = [batch.Video(case["H"], case["W"]) for _ in range(case["B"])]
    elif k == "batch":
        s["imgs"], s["sp"] = [], []
        for i, (H, W, n, noise, sp) in enumerate(_uneven(case)):
            s["imgs"].append(synth.voronoi_video_device(H, W, 1, n, noise,
                                                        seed=1000 * seed + i)[0][0].contiguous())
            s["sp"].append(sp)
    elif k == "shift":
        vid, flows = _video(case, seed, 2)
        s["labels"], s["params"] = bist_cuda.run_bass(vid[0].contiguous(), **_bass_kw(case))
        s["flow"] = flows[0].contiguous()
    elif k in ("marked", "evaluate", "pooling"):
        vid, flows, regs = _video(case, seed, case["T"], regions=True)
        s["vid"] = vid
        # ground-truth ids 0..max, each present
        s["gt"] = torch.unique(regs, return_inverse=True)[1].to(torch.int32).contiguous()
        s["spix"] = _forward(vid, flows, case, True, prop_niters=12)
        s["color"] = torch.tensor([0.0, 0.0, 1.0], device=vid.device)
        # rows of a table with room for ids of later frames
        s["nspix"] = max(8 * bist_cuda.hex_count(case["H"], case["W"], case["sp_size"]),
                         int(s["spix"].max()) + 1)
    elif k == "lab":
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))
        s["u8"] = torch.randint(0, 256, (case["H"], case["W"], 3), generator=g, device="cuda",
                                dtype=torch.uint8)
    else:
        raise KeyError(k)
    return s


# ---------------------------------------------------------------------------
# one pass
def run(s):
    case, k = s["case"], s["kind"]
    if k == "bass":
        labels, params = bist_cuda.run_bass(s["img"], **_bass_kw(case))
        return {"labels": labels, "n": params.n, "params": _whole(params)}
    if k == "image":
        return _forward(s["vid"], s["flows"], case, False)
    if k == "video":
        return _forward(s["vid"], s["flows"], case, True, prop_niters=case["prop_niters"])
    if k == "streams":
        for v in s["streams"]:
            v.reset()
        out = []
        for t in range(case["T"]):
            frames = [batch.Frame(img=vid[t], flow=flows[t - 1] if t else None, video=v)
                      for (vid, flows), v in zip(s["vids"], s["streams"])]
            batch.process_batch(frames, prop_niters=case["prop_niters"], **_bass_kw(case))
            out.append([f.labels for f in frames])
        return out
    if k == "batch":
        frames = [batch.Frame(img=i, sp_size=sp) for i, sp in zip(s["imgs"], s["sp"])]
        batch.process_batch(frames, niters=case["niters"], sm_period=case["sm_period"])
        return [f.labels for f in frames]
    if k == "shift":
        filled, shifted = bist_cuda.shift_and_fill(s["labels"], s["params"], s["flow"])
        return {"filled": filled, "shifted": shifted,
                "params": _whole(s["params"], ("prior_counts", "invalid_counts"))}
    if k == "marked":
        return bist_cuda.get_marked_video(s["vid"], s["spix"], s["color"])
    if k == "evaluate":
        return dict(metrics.computeSummary(s["vid"], s["gt"], s["spix"]))
    if k == "pooling":
        return metrics.sp_pooling(s["vid"], s["spix"], s["nspix"])
    if k == "lab":
        img = bist_cuda.rescale_u8(s["u8"])
        return {"img": img, "lab": bist_cuda.rgb2lab(img)}
    raise KeyError(k)


# ---------------------------------------------------------------------------
# what a pass cannot do without
def work(case):
    """Bytes: every input read and every output written once (colours 12 B, flow 8 B and
    labels 4 B a pixel).  Operations: a labelling compares every pixel with its four
    neighbours in each of the four sweeps of each iteration; the other passes are counted
    by their arithmetic on a pixel."""
    k = case["kind"]
    if k == "batch":
        npix = sum(H * W for H, W, _, _, _ in _uneven(case))
        return {"bytes": 16.0 * npix, "flops": 16.0 * case["niters"] * npix}
    T = case.get("T", 1)
    npix = float(case["H"] * case["W"])
    n = npix * T * case.get("B", 1)
    if k in ("bass", "image"):
        return {"bytes": 16.0 * n, "flops": 16.0 * case["niters"] * n}
    if k in ("video", "streams"):
        first = n / T
        later = n - first
        it = case["prop_niters"] or 4
        return {"bytes": 16.0 * n + 8.0 * later,
                "flops": 16.0 * (case["niters"] * first + it * later)}
    if k == "shift":
        return {"bytes": (4 + 8 + 4 + 4) * npix, "flops": 8.0 * npix}
    if k == "marked":
        return {"bytes": (12 + 4 + 12) * n, "flops": 8.0 * n}
    if k == "evaluate":
        return {"bytes": (12 + 4 + 4) * n, "flops": 30.0 * n}
    if k == "pooling":
        return {"bytes": (12 + 4 + 12) * n, "flops": 3.0 * n}
    if k == "lab":
        return {"bytes": (3 + 12 + 12) * npix, "flops": 60.0 * npix}
    raise KeyError(k)


# ---------------------------------------------------------------------------
# the outputs in 64 bits
def exact(case, seed):
    k = case["kind"]
    if k not in ("marked", "evaluate", "pooling", "lab"):
        return None                     # labels, and the parameters that go with them
    s = prepare(case, seed)
    if k == "lab":
        img = s["u8"].double() / 255.0
        return {"img": img, "lab": _lab64(img)}
    vid, spix = s["vid"].double(), s["spix"].long()
    if k == "marked":
        return _marked64(vid, spix, s["color"].double())
    if k == "pooling":
        down = _pool64(vid, spix, s["nspix"])[0]
        return torch.stack([d[p] for d, p in zip(down, spix)]), down
    return _scores64(vid, spix, s["gt"].long())


def _lab64(img):
    """sRGB (blue first) to CIELAB stored as (L / -100, a / 100, b / 100)."""
    lin = torch.where(img <= 0.04045, img / 12.92, ((img + 0.055) / 1.055).clamp_min(0) ** 2.4)
    b, g, r = lin.unbind(-1)
    X = r * 0.4124564 + g * 0.3575761 + b * 0.1804375
    Y = r * 0.2126729 + g * 0.7151522 + b * 0.0721750
    Z = r * 0.0193339 + g * 0.1191920 + b * 0.9503041

    def f(v):
        return torch.where(v > 0.008856, v.clamp_min(0) ** (1.0 / 3.0), (903.3 * v + 16.0) / 116.0)

    fx, fy, fz = f(X / 0.950456), f(Y), f(Z / 1.088754)
    return torch.stack([(116.0 * fy - 16.0) / -100.0, 5.0 * (fx - fy), 2.0 * (fy - fz)], -1)


def _marked64(vid, spix, color):
    """A pixel is painted when a 4-neighbour carries a smaller label."""
    border = torch.zeros_like(spix, dtype=torch.bool)
    border[:, 1:] |= spix[:, 1:] > spix[:, :-1]
    border[:, :-1] |= spix[:, :-1] > spix[:, 1:]
    border[:, :, 1:] |= spix[:, :, 1:] > spix[:, :, :-1]
    border[:, :, :-1] |= spix[:, :, :-1] > spix[:, :, 1:]
    return torch.where(border[..., None], color, vid.clamp(0.0, 1.0))


def _pool64(vid, spix, S):
    """Mean colour of every id in every frame (sum / (count + 1e-8)), and the counts."""
    T = vid.shape[0]
    sums = torch.zeros(T, S, 3, dtype=torch.float64, device=vid.device)
    cnt = torch.zeros(T, S, dtype=torch.float64, device=vid.device)
    for t in range(T):
        p = spix[t].reshape(-1)
        sums[t].index_add_(0, p, vid[t].reshape(-1, 3))
        cnt[t].index_add_(0, p, torch.ones_like(p, dtype=torch.float64))
    return sums / (cnt + 1e-8)[..., None], cnt, sums


def _scores64(vid, spix, gt):
    """Temporal extent, size variation, explained variance (frame and video), PSNR of the
    pooled video, under-segmentation error and segmentation accuracy (frame and video)."""
    T, H, W = spix.shape
    spix = spix - spix.min()
    S, G = int(spix.max()) + 1, int(gt.max()) + 1
    mean, cnt, sums = _pool64(vid, spix, S)
    alive = cnt > 0
    out = {"tex": float(alive.double().mean(1).mean()), "spnum": S,
           "ave_nsp": float(alive.sum(1).double().mean())}
    n, s1, s2 = alive.sum(0).double(), cnt.sum(0), (cnt * cnt).sum(0)
    keep = n > 1
    var = (n * s2 - s1 * s1)[keep] / (n * (n - 1))[keep]
    out["szv"] = float(var.sqrt().mean()) if bool(keep.any()) else float("nan")
    frame = vid.reshape(T, -1, 3).mean(1)
    pooled = torch.stack([m[p] for m, p in zip(mean, spix)])
    dev = ((vid - frame[:, None, None]) ** 2).reshape(T, -1).sum(1)
    out["ev"] = float((((pooled - frame[:, None, None]) ** 2).reshape(T, -1).sum(1)
                       / (dev + 1e-10)).mean())
    whole = (255.0 * sums.sum(0) / (s1 + 1e-10)[:, None])[spix]
    out["ev3d"] = float((((whole - 255.0 * frame[:, None, None]) ** 2).reshape(T, -1).sum(1)
                         / (255.0 ** 2 * dev + 1e-10)).mean())
    mse = ((vid - pooled) ** 2).reshape(T, -1).mean(1)
    out["pooling"] = float((10.0 * torch.log10(1.0 / mse)).mean())
    ue, sa, size, inside, outside = [], [], [], 0, 0
    for t in range(T):
        J = torch.bincount(spix[t].reshape(-1) * G + gt[t].reshape(-1),
                           minlength=S * G).reshape(S, G).double()
        c = cnt[t][:, None]
        o = torch.where(J > 0, c - J, torch.zeros_like(J))
        ue.append(torch.minimum(o, J).sum(0))
        sa.append(torch.where(2 * J >= c, J, torch.zeros_like(J)).sum(0))
        size.append(J.sum(0))
        inside, outside = inside + J, outside + o
    ue, sa, size = torch.stack(ue), torch.stack(sa), torch.stack(size)
    out["ue2d"] = float((ue / (H * W)).mean())
    z = size[:, 1:]
    out["sa2d"] = float(((sa[:, 1:] / (z + (z == 0))).sum(0) / (z > 0).sum(0)).mean())
    out["ue3d"] = float((torch.minimum(outside, inside).sum(0) / (T * H * W)).mean())
    sa3 = torch.where(2 * inside >= s1[:, None], inside, torch.zeros_like(inside)).sum(0)
    out["sa3d"] = float((sa3[1:] / z.sum(0)).mean())
    out["strred0"] = out["strred1"] = -1.0
    return out
