"""Graphs recorded from context calls, and what later calls on the same context do to them: calls that use none of a
recorded call's scratch leave its replays as they were, and a call of the same shape is enough to warm up a capture.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Call:
    """ps_mcm_multi_device of some spins on one grid, with its own windows and matrices."""

    def __init__(self, ctx, spins, lmax, mode, lmin=0, seed=1):
        from powerspectra_gpu import synthetic as syn
        self.ctx, self.spins, self.lmin, self.lmax, self.mode = ctx, spins, lmin, lmax, mode
        self.nW, self.n = 2 * lmax + 1, lmax - lmin + 1
        self.W = torch.tensor(np.stack([syn.mask_spectrum(self.nW, 0.5, self.nW / 3.0, seed=seed + s) for s in spins]),
                              device="cuda")
        self.M = torch.zeros((len(spins), self.n, self.n), dtype=torch.float64, device="cuda")

    def __call__(self):
        self.ctx.mcm_multi_device({s: self.W[i].data_ptr() for i, s in enumerate(self.spins)}, self.nW, self.lmin,
                                  self.lmax, {s: self.M[i].data_ptr() for i, s in enumerate(self.spins)}, self.n,
                                  mode=self.mode)

    def direct(self):
        self()
        torch.cuda.synchronize()
        return self.M.clone()

    def record(self, stream):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            self()
        return g

    def replayed(self, g):
        self.M.zero_()
        g.replay()
        torch.cuda.synchronize()
        return self.M


@pytest.fixture
def own():
    """A context of its own on a stream that can be captured."""
    from powerspectra_gpu import Context
    ctx, s = Context(0), torch.cuda.Stream()
    ctx.set_stream(s.cuda_stream)
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        yield ctx, s
        torch.cuda.synchronize()
    ctx.close()


@pytest.mark.parametrize("first,second", [("plain", "chosen"), ("chosen", "plain")])
def test_one_arithmetic_beside_the_other(own, first, second):
    ctx, s = own
    a, b = Call(ctx, (0, 2), 90, first), Call(ctx, (0, 2), 60, second, lmin=2, seed=7)
    want_a, want_b = a.direct(), b.direct()
    ga = a.record(s)  # the other arithmetic's call on another grid came last
    assert bool((a.replayed(ga) == want_a).all())
    assert bool((b.direct() == want_b).all())
    gb = b.record(s)
    for _ in range(2):
        assert bool((a.replayed(ga) == want_a).all())
        assert bool((b.replayed(gb) == want_b).all())


def test_plain_graph_beside_a_larger_quickpol(own):
    """QuickPol in FP64 reads the same factors as the plain kernels, and for a larger lmax needs more of them."""
    ctx, s = own
    a = Call(ctx, (0, 1, 2, 3), 70, "plain")
    want = a.direct()
    g = a.record(s)
    for lmax in (71, 150, 900):
        ctx.quickpol_xi(0, 0, 2, 2, np.ones(2 * lmax + 1), lmax, 3, 3)
        junk = torch.full((1 << 16,), np.nan, dtype=torch.float64, device="cuda")  # fresh memory, were any given back
        assert bool((a.replayed(g) == want).all())
        assert bool((a.direct() == want).all())
        del junk


@pytest.mark.parametrize("lmax", [64, 520])  # without and with the table of square-root ratios
@pytest.mark.parametrize("warm,then", [((0,), (2,)), ((2, 3), (0, 1)), ((0, 2, 3), (1, 2, 3))])
def test_one_call_warms_up_the_grid(own, lmax, warm, then):
    """A call with as many windows on the same grid is enough before a capture, whatever its spins."""
    from powerspectra_gpu import Context
    ctx, s = own
    Call(ctx, warm, lmax, "chosen").direct()
    b = Call(ctx, then, lmax, "chosen", seed=5)
    g = b.record(s)
    got = b.replayed(g).clone()
    assert bool((got == b.direct()).all())
    assert bool((b.replayed(g) == got).all())
    Call(ctx, (2, 3), lmax + 100, "chosen").direct()  # its own, larger table
    ref = Context(0)
    ref.set_stream(s.cuda_stream)
    c = Call(ref, then, lmax, "chosen", seed=5)
    assert bool((c.direct() == got).all())
    ref.close()


@pytest.mark.parametrize("larger,lmax", [(1300, 1000), (2000, 1100), (300, 20)])
def test_window_spectrum_after_a_larger_one(own, larger, lmax):
    """The scratch of a larger call is enough for a smaller one, whose sums are cut finer."""
    ctx, s = own

    def call(lm, seed):
        a = torch.tensor(np.random.default_rng(seed).normal(size=(lm + 1) * (lm + 2)), device="cuda")
        out = torch.zeros(lm + 1, dtype=torch.float64, device="cuda")
        return a, out, lambda: ctx.window_W_device([a.data_ptr()], [a.data_ptr()], lm, lm, lm, out.data_ptr())

    *keep, big = call(larger, 1)
    big()
    a, out, run = call(lmax, 2)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        run()
    g.replay()
    torch.cuda.synchronize()
    got = out.clone()
    run()
    torch.cuda.synchronize()
    assert bool((got == out).all()) and bool((got > 0).all())


def test_warm_calls_beside_another_threads_capture(own):
    """Calls of a warmed-up context never end a capture that another thread has begun, also when a table is made or
    replaced by one of them."""
    import threading
    from powerspectra_gpu import Context
    ctx, s = own
    a = Call(ctx, (0,), 80, "chosen")
    want = a.direct()
    other = Context(0)  # its own stream
    b, c = Call(other, (2, 3), 600, "chosen"), Call(other, (2, 3), 640, "chosen")
    torch.cuda.synchronize()
    for x in (c, b):
        x()
        other.synchronize()
    errors = []

    def work():
        try:
            for _ in range(50):  # enqueued only: waiting is not allowed during another thread's capture
                b()
        except BaseException as e:  # reported by the test's own thread
            errors.append(repr(e))

    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            a()
            t = threading.Thread(target=work)
            t.start()
            t.join()
        other.synchronize()
        assert not errors, errors
        assert bool((a.replayed(g) == want).all())
        b = c  # a larger table in the second capture
        b()
        other.synchronize()
    other.close()
