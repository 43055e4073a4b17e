"""The quality entry points keep device scratch and pinned staging in the context.  Calls that
share a context from several host threads, or come on streams of equal handles, give what
each gives alone."""
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def clip(T, H, W, n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    vid = torch.rand((T, H, W, 3), generator=g, device="cuda")
    y, x = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"),
                          indexing="ij")
    lab = (y * n // H) * n + x * n // W
    spix = lab.to(torch.int32).expand(T, H, W).contiguous()
    gt = (lab % 5).to(torch.int32).expand(T, H, W).contiguous()
    return vid, spix, gt, n * n


def in_threads(jobs, rounds):
    """jobs[i](): run `rounds` times in a thread of its own; all results."""
    out, errors = [[] for _ in jobs], []
    start = threading.Barrier(len(jobs))

    def run(i):
        try:
            start.wait()
            for _ in range(rounds):
                out[i].append(jobs[i]())
        except Exception as e:          # noqa: BLE001 - reported below
            errors.append(e)

    ts = [threading.Thread(target=run, args=(i,)) for i in range(len(jobs))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    return out


def test_threads_on_the_default_stream(monkeypatch):
    """Different sizes, so the scratch grows while other threads use it."""
    from st_spix_gb300 import bist_cuda, metrics
    data = [clip(*a) for a in ((2, 33, 47, 3, 0), (6, 240, 320, 20, 1), (3, 480, 854, 60, 2),
                               (8, 120, 200, 9, 3))]
    ref = [(metrics.sp_pooling(v, s, n), dict(metrics.computeSummary(v, g, s)),
            metrics.count_spix(s)) for v, s, g, n in data]
    torch.cuda.synchronize()
    monkeypatch.setattr(bist_cuda, "_contexts", {})   # a new context: its scratch has to grow
    jobs = [lambda d=d: (metrics.sp_pooling(d[0], d[1], d[3]),
                         dict(metrics.computeSummary(d[0], d[2], d[1])),
                         metrics.count_spix(d[1])) for d in data]
    got = in_threads(jobs, 20)
    for r, gs in zip(ref, got):
        for g in gs:
            # (FP64 sums by atomics: their order moves the last digits)
            torch.testing.assert_close(g[0][0], r[0][0], rtol=2.0 ** -22, atol=0)
            torch.testing.assert_close(g[0][1], r[0][1], rtol=2.0 ** -22, atol=0)
            assert torch.equal(g[2], r[2])
            for k, v in r[1].items():
                assert g[1][k] == pytest.approx(v, rel=1e-9, abs=1e-9, nan_ok=True), k


def test_per_thread_default_streams_of_one_handle():
    """One context, the handle of the per-thread default stream, another stream in each
    thread: the first call returns while its kernels still read the scratch, and the second,
    in a thread that starts then, takes it over."""
    from st_spix_gb300 import _lib
    per_thread = 2
    data = [clip(16, 480, 854, 40, 4), clip(16, 480, 854, 41, 5)]
    ctx = _lib.Context(0)
    outs = [(torch.empty((v.shape[0], n, 3), device="cuda"), torch.empty_like(v))
            for v, _, _, n in data]

    def call(i):
        v, s, _, n = data[i]
        T, H, W = s.shape
        down, pooled = outs[i]
        assert 0 == ctx.lib.stspix_sp_pooling(ctx.handle, per_thread, v.data_ptr(), s.data_ptr(),
                                              T, H, W, n, pooled.data_ptr(), down.data_ptr())

    def other():
        call(1)
        torch.cuda.synchronize()        # (its stream is idle when the thread ends)

    torch.cuda.synchronize()
    ref = []
    for i in (0, 1):
        call(i)
        torch.cuda.synchronize()
        ref.append([o.clone() for o in outs[i]])
    for _ in range(10):
        for o in outs[0] + outs[1]:
            o.zero_()
        torch.cuda.synchronize()
        call(0)
        t = threading.Thread(target=other)
        t.start()
        t.join()
        torch.cuda.synchronize()
        for o, r in zip(outs, ref):
            for a, b in zip(o, r):
                torch.testing.assert_close(a, b, rtol=2.0 ** -22, atol=0)


def test_capture_is_refused_and_leaves_the_context_usable():
    from st_spix_gb300 import metrics
    v, s, _, n = clip(2, 33, 47, 3, 6)
    ref = metrics.sp_pooling(v, s, n)[1]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        metrics.sp_pooling(v, s, n)     # the stream's context and scratch exist
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        g.capture_begin()
        try:
            with pytest.raises(RuntimeError):
                metrics.sp_pooling(v, s, n)
        finally:
            g.capture_end()
        out = metrics.sp_pooling(v, s, n)[1]
    torch.cuda.synchronize()
    torch.testing.assert_close(out, ref, rtol=2.0 ** -22, atol=0)
