"""The tables that only save time: not made where they would cost more than they save, and given back before a call is
refused for lack of device memory.  The results are the same bits with and without them.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _hold(leave):
    """Takes the device's memory but for `leave` bytes."""
    torch.cuda.empty_cache()
    return torch.empty(_free() - leave, dtype=torch.uint8, device="cuda")


def _ratios(lmax):  # bytes of the table: 3.5 lmax^2 entries of 16 bytes and its margins
    return 56 * lmax * lmax


class Pair:
    """++ and -- of one window, device matrices."""

    def __init__(self, ctx, lmax):
        from powerspectra_gpu import synthetic as syn
        self.ctx, self.lmax, self.n, self.nW = ctx, lmax, lmax + 1, lmax + 1
        self.W = torch.tensor(syn.mask_spectrum(self.nW, 0.5, self.nW / 3.0, seed=3), device="cuda")
        self.M = torch.zeros((2, self.n, self.n), dtype=torch.float64, device="cuda")

    def __call__(self):
        torch.cuda.synchronize()  # the context has a stream of its own
        self.ctx.mcm_multi_device({2: self.W.data_ptr(), 3: self.W.data_ptr()}, self.nW, 0, self.lmax,
                                  {2: self.M[0].data_ptr(), 3: self.M[1].data_ptr()}, self.n, mode="chosen")
        torch.cuda.synchronize()
        return self.M.clone()


def _context():
    from powerspectra_gpu import Context
    return Context(0)


def test_no_table_for_one_call():
    ctx = _context()
    a = Pair(ctx, 600)
    want = a()
    before = _free()
    assert bool((a() == want).all())
    assert before - _free() < _ratios(600)  # nor for the second call of a size
    for _ in range(40):
        assert bool((a() == want).all())
    assert before - _free() >= _ratios(600)
    ctx.close()


@pytest.mark.parametrize("then", ["matrix", "solve"])
def test_table_given_back(then):
    ctx = _context()
    a = Pair(ctx, 3000)
    want = a()  # 504 MB of ratios, made at once
    x = np.linspace(1.0, 2.0, 4400)
    hold = _hold(400 << 20)
    if then == "matrix":
        lmax = 7399  # 438 MB on the device
        assert np.all(np.isfinite(ctx.mcm(0, x, 7000, lmax, mode="chosen")))
        got = ctx.mcm(0, x, 0, lmax, mode="chosen")
        assert got.shape == (lmax + 1, lmax + 1) and got[1, 1] != 0.0
    else:
        assert np.allclose(ctx.solve(2.0 * np.eye(4400), x), 0.5 * x)  # three matrices of 155 MB
    assert bool((a() == want).all())
    del hold
    torch.cuda.empty_cache()
    assert bool((a() == want).all())
    ctx.close()


def test_no_room_for_a_table():
    ctx = _context()
    a, b = Pair(ctx, 2000), Pair(ctx, 2600)
    want = a(), b()  # 224 MB, then 378 MB in its place
    ctx.close()
    ctx = _context()
    a.ctx = b.ctx = ctx
    assert bool((a() == want[0]).all())
    hold = _hold(300 << 20)
    assert bool((b() == want[1]).all())  # without a table: the smaller one stays
    before = _free()
    for _ in range(3):
        assert bool((b() == want[1]).all())
        assert bool((a() == want[0]).all())
    assert _free() == before
    del hold
    torch.cuda.empty_cache()
    ctx.close()


class Batch:
    """TT, TE, ++ and -- of one window each on uneven grids."""

    def __init__(self, ctx, sizes):
        from powerspectra_gpu import synthetic as syn
        self.ctx, self.probs, self.keep = ctx, [], []
        for i, lmax in enumerate(sizes):
            n = lmax + 1
            W = torch.tensor(syn.mask_spectrum(n, 0.5, n / 3.0, seed=i), device="cuda")
            M = torch.zeros((4, n, n), dtype=torch.float64, device="cuda")
            self.keep.append((W, M))
            self.probs.append({"lmin": 0, "lmax": lmax, "cases": 0xF, "nW": n, "ldm": n, "W": [W.data_ptr()],
                               "M": [M[s].data_ptr() for s in range(4)]})

    def prepare(self, **kw):
        self.ctx.batch_prepare(self.probs, **kw)

    def run(self, how):
        for _, M in self.keep:
            M.zero_()
        torch.cuda.synchronize()  # the context has a stream of its own
        how()
        torch.cuda.synchronize()

    def matrices(self):
        return [M.clone() for _, M in self.keep]

    def equal(self, want):
        return all(bool((M == w).all()) for (_, M), w in zip(self.keep, want))


@pytest.mark.parametrize("form", [0, -1])
def test_batch_with_little_room(form):
    ctx = _context()
    b = Batch(ctx, range(900, 964))  # 131 MB of slices and 55 of ratios; 20 MB of what it needs
    b.prepare(blocks_per_sm=form)
    b.run(ctx.batch_run)
    want = b.matrices()
    for leave in range(230, 30, -20):
        ctx2 = _context()
        b.ctx = ctx2
        hold = _hold(leave << 20)
        b.prepare(blocks_per_sm=form)
        b.run(ctx2.batch_run)
        del hold
        torch.cuda.empty_cache()
        ctx2.close()
        assert b.equal(want), leave
    ctx.close()


@pytest.mark.parametrize("form", [0, -1])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_tables_given_back(form, graph):
    ctx = _context()
    b = Batch(ctx, range(900, 964))
    b.prepare(blocks_per_sm=form)
    b.run(ctx.batch_graph_launch)
    want = b.matrices()
    hold = _hold(64 << 20)
    x = np.linspace(1.0, 2.0, 3800)
    lmax = 3799 if form == 0 else 3199  # 115 MB, or 82 where the ratios alone come back
    assert np.all(np.isfinite(ctx.mcm(0, x, 0, lmax, mode="chosen")))
    b.run(ctx.batch_graph_launch if graph else ctx.batch_run)
    del hold
    torch.cuda.empty_cache()
    assert b.equal(want)
    ctx.close()


def test_blocks_stage_two_matrices():
    """[++ -(--); -(--) ++] needs no more on the device than ++ and --."""
    import powerspectra_gpu as pg
    lmax = 3599
    n = lmax + 1
    x = np.linspace(2.0, 1.0, n)
    ctx = _context()
    want = pg.mcm(("EE_BB", "EB_BE"), x, lmax=lmax, mode="chosen", ctx=ctx)
    assert np.array_equal(want[0].parent[:n], np.hstack([want[1].parent[:n, :n], -want[1].parent[:n, n:]]))
    ctx.close()
    ctx = _context()
    hold = _hold(280 << 20)  # two of 104 MB and the slices; three do not fit
    got = pg.mcm("EB_BE", x, lmax=lmax, mode="chosen", ctx=ctx)
    del hold
    torch.cuda.empty_cache()
    assert np.array_equal(got.parent, want[1].parent)
    ctx.close()
