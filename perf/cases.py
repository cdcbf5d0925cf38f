"""The work that users of this library have it do, as cases whose passes can be timed and compared.

A case names one kind of call and its sizes.  `listed()` holds the calls a program makes in earnest, at
the sizes of this repository's configurations and tests; `draw(rng)` gives more of the same kinds over
their whole ranges (odd sizes, lmin > 0, short windows, both arithmetics).  `prepare` makes what such a
program has in hand, `run` makes the call through the public entry points, `work` counts the bytes and
operations the call cannot do without, and `exact` restates its result in 64-bit torch.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "powerspectra.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import powerspectra_gpu as pg  # noqa: E402
from powerspectra_gpu import covariance as pgcov  # noqa: E402
from powerspectra_gpu import synthetic as syn  # noqa: E402

SPIN_OF = {"TT": (0,), "TE": (1,), "M++": (2,), "M--": (3,), "EE_BB": (2, 3), "EB_BE": (2, 3)}


def listed():
    return [
        # Host calls with the default arithmetic (FP64), as a program ported from the reference makes them.
        # The smallest: a quick look at one mask at low resolution, where latency and launches count.
        {"name": "mcm_tt_95", "kind": "mcm", "spec": "TT", "lmin": 0, "lmax": 95, "mode": "plain"},
        # The reference test suite's grid: the EE/BB block matrix of one mask.
        {"name": "mcm_eebb_767", "kind": "mcm", "spec": "EE_BB", "lmin": 0, "lmax": 767, "mode": "plain"},
        # One temperature matrix on device arrays in the fast arithmetic (one call per mask in a loop).
        {"name": "tt_767_chosen", "kind": "multi", "cases": 0x1, "lmin": 0, "lmax": 767, "nW": 1535,
         "mode": "chosen"},
        # Every spin case of one analysis grid, fast arithmetic.
        {"name": "all_spins_3071_chosen", "kind": "multi", "cases": 0xF, "lmin": 0, "lmax": 3071, "nW": 6143,
         "mode": "chosen"},
        # The same in FP64 on a grid that starts at l = 2 (the check of the fast arithmetic, and production
        # where FP64 is asked for).
        {"name": "all_spins_1999_plain", "kind": "multi", "cases": 0xF, "lmin": 2, "lmax": 1999, "nW": 3999,
         "mode": "plain"},
        # The largest: 20 mask spectra at lmax 8191 (7 TT, 7 EE and 6 BB matrices), fast arithmetic.
        {"name": "large_8191_set", "kind": "set", "cases": 0xD, "K": 20, "one_each": True, "lmin": 0, "lmax": 8191,
         "nW": 16383, "mode": "chosen"},
        # One covariance block through the host call with the default arithmetic.
        {"name": "cov_eeee_1001", "kind": "cov", "ch1": "EE", "ch2": "EE", "lmin": 0, "lmax": 1001, "mode": "plain"},
        # The six covariance blocks of a Planck-like analysis (31 windows) in one device call.
        {"name": "cov_set_2508", "kind": "covset", "nblk": 6, "lmin": 0, "lmax": 2508, "mode": "chosen"},
        # Many small uneven problems replayed as one graph (simulation loops over masks).
        {"name": "batch_small_256", "kind": "batch", "n": 256, "lo": 64, "hi": 1023, "kmax": 4},
        # A window spectrum of the covariance workspace: the PP x PP mean of four terms over coefficient sets.
        {"name": "window_pp_2508", "kind": "window", "nterms": 4, "auto": False, "lmax": 2508, "mmax": 2508,
         "lout": 2508},
        # The QuickPol beam coupling of the reference's notebook (1000 x 1000, band 100), default arithmetic.
        {"name": "quickpol_999", "kind": "quickpol", "nu1": 0, "nu2": 0, "s1": 2, "s2": 2, "lmax": 999, "bl": 100,
         "bu": 100, "nW": 1999, "mode": "plain"},
        # The decoupling step of master: the 2 x 2 EE/BB block matrix against one pseudo-spectrum.
        {"name": "solve_1532", "kind": "solve", "n": 1532, "nrhs": 1},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mcm", "multi", "multi", "set", "cov", "covset", "batch", "window", "quickpol", "solve"])
    lmin = rng.choice([0, 0, 2, 3, 30])
    mode = rng.choice(["plain", "chosen"])
    if kind == "mcm":
        return {"kind": kind, "spec": rng.choice(sorted(SPIN_OF)), "lmin": lmin, "lmax": _logint(rng, 63, 1535),
                "mode": mode}
    if kind == "multi":
        lmax = _logint(rng, 127, 2600 if mode == "plain" else 4000)
        return {"kind": kind, "cases": rng.randrange(1, 16), "lmin": lmin, "lmax": lmax,
                "nW": rng.choice([lmax + 1, 2 * lmax + 1, lmax + 1 + lmax // 3]), "mode": mode}
    if kind == "set":
        lmax = _logint(rng, 255, 4100)
        return {"kind": kind, "cases": rng.choice([0x1, 0xC, 0xD, 0xF]), "K": rng.randrange(2, 13),
                "one_each": rng.random() < 0.5, "lmin": lmin, "lmax": lmax,
                "nW": rng.choice([lmax + 1, 2 * lmax + 1]), "mode": "chosen"}
    if kind == "cov":
        ch1, ch2 = rng.choice(syn.COV_BLOCKS)
        return {"kind": kind, "ch1": ch1, "ch2": ch2, "lmin": lmin, "lmax": _logint(rng, 95, 1600), "mode": mode}
    if kind == "covset":
        return {"kind": kind, "nblk": rng.randrange(2, 7), "lmin": lmin, "lmax": _logint(rng, 255, 2700),
                "mode": "chosen"}
    if kind == "batch":
        lo = _logint(rng, 48, 256)
        return {"kind": kind, "n": _logint(rng, 16, 256), "lo": lo, "hi": _logint(rng, lo, 1023),
                "kmax": rng.randrange(1, 5)}
    if kind == "window":
        lmax = _logint(rng, 383, 8191)
        return {"kind": kind, "nterms": rng.choice([1, 1, 2, 4]), "auto": rng.random() < 0.3, "lmax": lmax,
                "mmax": rng.choice([lmax, lmax, lmax - lmax // 5]), "lout": rng.choice([lmax, lmax - lmax // 7])}
    if kind == "quickpol":
        lmax = _logint(rng, 200, 2000)
        nu, s = rng.choice([(0, 0), (0, 0), (1, 1), (-1, 2), (0, 3)]), rng.choice([(2, 2), (2, 2), (0, 2), (-2, 2)])
        band = _logint(rng, 10, 120)
        return {"kind": kind, "nu1": nu[0], "nu2": nu[1], "s1": s[0], "s2": s[1], "lmax": lmax, "bl": band,
                "bu": rng.choice([band, band // 2]), "nW": 2 * lmax + 1, "mode": mode}
    return {"kind": "solve", "n": _logint(rng, 96, 3000), "nrhs": rng.choice([1, 1, 3])}


# ---- inputs -------------------------------------------------------------------------------------

def _masks(n, nW, seed):
    """n mask spectra (f_sky 0.4 - 0.8, cutoffs 400 - 1200): the values every coupling call meets."""
    rng = np.random.default_rng(seed)
    return [syn.mask_spectrum(nW, float(rng.uniform(0.4, 0.8)), float(rng.uniform(400, 1200)),
                              seed=int(rng.integers(2 ** 31))) for _ in range(n)]


def _dev(x):
    return torch.tensor(np.ascontiguousarray(x), device="cuda")


def _spins(cases):
    return [s for s in range(4) if cases >> s & 1]


def _slots(c):
    """The (window, spin case) slots of a set: every case of every window, or one case per window in turn."""
    sp = _spins(c["cases"])
    return [(k, s) for k in range(c["K"]) for s in ([sp[k % len(sp)]] if c["one_each"] else sp)]


def _cov_workspace(lmax, seed):
    made = {}

    def window(*key):
        if key not in made:
            rng = np.random.default_rng([seed, syn._key_seed(key) % (1 << 62)])
            made[key] = syn.mask_spectrum(lmax + 1, float(rng.uniform(0.4, 0.8)), float(rng.uniform(500, 900)),
                                          seed=int(rng.integers(2 ** 31)))
        return made[key]

    spectra, noise = syn.signal_spectra(lmax, seed=seed)
    return pgcov.WindowWorkspace(syn.FIELDS, lmax, window), spectra, noise


def _batch_problems(c, seed):
    """[(lmax, K, cases, spectra)]: uneven problems (the case gives their sizes), spin 0 (TT) or spin 2
    (++ and --)."""
    size = np.random.default_rng([c["n"], c["lo"], c["hi"], c["kmax"]])
    rng = np.random.default_rng([seed, 4])
    out = []
    for _ in range(c["n"]):
        lmax = int(round(math.exp(size.uniform(math.log(c["lo"]), math.log(c["hi"])))))
        K, cases = int(size.integers(1, c["kmax"] + 1)), int(size.choice([0x1, 0xC]))
        out.append((lmax, K, cases, _masks(K, lmax + 1, int(rng.integers(2 ** 31)))))
    return out


def _n_alms(lmax, mmax):
    return (mmax + 1) * (mmax + 2) // 2 + (mmax + 1) * (lmax - mmax)


def _window_sets(c, seed):
    """Coefficient sets (HEALPix m-major order) with a mask-like envelope, two per term (one if auto)."""
    lmax, mmax = c["lmax"], c["mmax"]
    ls = torch.cat([torch.arange(m, lmax + 1, device="cuda", dtype=torch.float64) for m in range(mmax + 1)])
    env = (torch.exp(-ls / 3000.0) / (ls + 1.0))[:, None]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    sets = []
    for _ in range(c["nterms"] * (1 if c["auto"] else 2)):
        a = torch.randn((len(ls), 2), dtype=torch.float64, device="cuda", generator=gen) * env
        a[:lmax + 1, 1] = 0.0  # the m = 0 coefficients of a real field are real
        sets.append(a)
    A = sets[:c["nterms"]]
    return A, A if c["auto"] else sets[c["nterms"]:]


def _solve_inputs(c, seed):
    """A matrix with a coupling matrix's shape (a falling kernel around a dominant diagonal) and spectra."""
    n = c["n"]
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    M = 0.05 / (1.0 + (i[:, None] - i[None, :]).abs()) ** 1.5
    M *= 1.0 + 0.05 * torch.randn((n, n), dtype=torch.float64, device="cuda", generator=gen)
    M += torch.diag(0.5 + 0.1 * torch.rand(n, dtype=torch.float64, device="cuda", generator=gen))
    b = (1.0 + torch.rand((n, c["nrhs"]), dtype=torch.float64, device="cuda", generator=gen)) / (i[:, None] + 10.0)
    return M, b


def prepare(case, seed):
    c, k = case, case["kind"]
    st = {"case": c}
    if k == "mcm":
        st["W"] = _masks(1, c["lmax"] + 1, seed)[0]
        pg.default_context()
    elif k == "multi":
        n = c["lmax"] - c["lmin"] + 1
        Ws = _masks(4, c["nW"], seed)
        st["W"] = {s: _dev(Ws[s]) for s in _spins(c["cases"])}
        st["M"] = {s: torch.empty((n, n), dtype=torch.float64, device="cuda") for s in _spins(c["cases"])}
        st["ctx"] = pg.default_context()
    elif k == "set":
        n = c["lmax"] - c["lmin"] + 1
        st["W"] = [_dev(w) for w in _masks(c["K"], c["nW"], seed)]
        st["M"] = {q: torch.empty((n, n), dtype=torch.float64, device="cuda") for q in _slots(c)}
        st["ctx"] = pg.default_context()
    elif k == "cov":
        ws, spectra, noise = _cov_workspace(c["lmax"], seed)
        pgcov.gather(c["ch1"], c["ch2"], ws, spectra, noise)  # the workspace holds its windows
        st.update(ws=ws, spectra=spectra, noise=noise)
        pg.default_context()
    elif k == "covset":
        n = c["lmax"] - c["lmin"] + 1
        ws, spectra, noise = _cov_workspace(c["lmax"], seed)
        st["blocks"] = []
        for a, b in syn.COV_BLOCKS[:c["nblk"]]:
            kind, S, R, Ws = pgcov.gather(a, b, ws, spectra, noise)
            st["blocks"].append((kind, [_dev(x) for x in S], [_dev(x) for x in R], [_dev(x) for x in Ws],
                                 torch.empty((n, n), dtype=torch.float64, device="cuda")))
        st["ctx"] = pg.default_context()
    elif k == "batch":
        probs = _batch_problems(c, seed)
        sizes = [(p[0] + 1) ** 2 * p[1] * len(_spins(p[2])) for p in probs]
        out = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
        desc, keep, off = [], [], 0
        for lmax, K, cases, Ws in probs:
            n2 = (lmax + 1) ** 2
            dW = [_dev(w) for w in Ws]
            keep.append(dW)
            M = [0] * (4 * K)
            for q in range(K):
                for s in _spins(cases):
                    M[4 * q + s] = out.data_ptr() + 8 * off
                    off += n2
            desc.append({"lmin": 0, "lmax": lmax, "cases": cases, "nW": lmax + 1, "ldm": lmax + 1,
                         "W": [w.data_ptr() for w in dW], "M": M})
        st["ctx"] = pg.Context(0)  # the batch lives in its context
        st["ctx"].batch_prepare(desc)
        st.update(out=out, keep=keep)
    elif k == "window":
        st["A"], st["B"] = _window_sets(c, seed)
        st["out"] = torch.empty(c["lout"] + 1, dtype=torch.float64, device="cuda")
        st["ctx"] = pg.default_context()
    elif k == "quickpol":
        st["W"] = _masks(1, c["nW"], seed)[0]
        st["ctx"] = pg.default_context()
    else:
        M, b = _solve_inputs(c, seed)
        st["M"], st["b"] = np.asfortranarray(M.cpu().numpy()), np.asfortranarray(b.cpu().numpy())
        st["ctx"] = pg.default_context()
    return st


def run(st):
    c, k = st["case"], st["case"]["kind"]
    if k == "mcm":
        return pg.mcm(c["spec"], st["W"], lmin=c["lmin"], lmax=c["lmax"], mode=c["mode"]).parent
    if k == "multi":
        st["ctx"].mcm_multi_device({s: w.data_ptr() for s, w in st["W"].items()}, c["nW"], c["lmin"], c["lmax"],
                                   {s: m.data_ptr() for s, m in st["M"].items()}, c["lmax"] - c["lmin"] + 1,
                                   mode=c["mode"])
        return list(st["M"].values())
    if k == "set":
        ptr = [0] * (4 * c["K"])
        for (q, s), m in st["M"].items():
            ptr[4 * q + s] = m.data_ptr()
        st["ctx"].mcm_set_device(c["cases"], [w.data_ptr() for w in st["W"]], c["nW"], c["lmin"], c["lmax"], ptr,
                                 c["lmax"] - c["lmin"] + 1, mode=c["mode"])
        return list(st["M"].values())
    if k == "cov":
        return pg.coupledcov(c["ch1"], c["ch2"], st["ws"], st["spectra"], st["noise"], lmin=c["lmin"],
                             lmax=c["lmax"], mode=c["mode"]).parent
    if k == "covset":
        st["ctx"].coupledcov_set_device(
            [(kind, [x.data_ptr() for x in S], [x.data_ptr() for x in R], [x.data_ptr() for x in W], C.data_ptr())
             for kind, S, R, W, C in st["blocks"]], c["lmax"] + 1, c["lmin"], c["lmax"], c["lmax"] - c["lmin"] + 1,
            mode=c["mode"])
        return [b[4] for b in st["blocks"]]
    if k == "batch":
        st["ctx"].batch_graph_launch()
        return st["out"]
    if k == "window":
        st["ctx"].window_W_device([a.data_ptr() for a in st["A"]], [b.data_ptr() for b in st["B"]], c["lmax"],
                                  c["mmax"], c["lout"], st["out"].data_ptr())
        return st["out"]
    if k == "quickpol":
        return st["ctx"].quickpol_xi(c["nu1"], c["nu2"], c["s1"], c["s2"], st["W"], c["lmax"], c["bl"], c["bu"],
                                     mode=c["mode"])
    return st["ctx"].solve(st["M"], st["b"] if c["nrhs"] > 1 else st["b"][:, 0])


# ---- work ---------------------------------------------------------------------------------------

def _terms(lmin, lmax, nW):
    """l3-terms of one family over the pairs lmin <= l1 <= l2 <= lmax, l3 <= nW - 1."""
    tot = 0
    for l1 in range(lmin, lmax + 1):
        l2 = np.arange(l1, lmax + 1)
        tot += int(np.clip(np.minimum(l1 + l2, nW - 1) - (l2 - l1) + 1, 0, None).sum())
    return tot


def _pair_flops(terms, spins, spectra):
    """Recurrences (9 flops per term for spin 0, 16 for spin 2) and 3 per spectrum contracted."""
    return terms * (9 * bool(spins & {0, 1}) + 16 * bool(spins & {1, 2, 3}) + 3 * spectra)


_COV_SPINS = {"TTTT": {0}, "EEEE": {2}, "TTTE": {0}, "TETE": {0, 1}, "TEEE": {1}, "TEEE_PLANCK": {2}, "TTEE": {0}}
_COV_NW = {"TTTT": 8, "EEEE": 8, "TTTE": 4, "TETE": 5, "TEEE": 4, "TEEE_PLANCK": 4, "TTEE": 2}


def work(case):
    c, k = case, case["kind"]
    n = c["lmax"] - c["lmin"] + 1 if "lmin" in c else 0
    if k == "mcm":
        spins = set(SPIN_OF[c["spec"]])
        t = _terms(c["lmin"], c["lmax"], c["lmax"] + 1)
        return {"bytes": 8 * (c["lmax"] + 1 + (4 if len(spins) > 1 else 1) * n * n), "flops": _pair_flops(t, spins, 1)}
    if k == "multi":
        sp = _spins(c["cases"])
        t = _terms(c["lmin"], c["lmax"], c["nW"])
        return {"bytes": 8 * len(sp) * (c["nW"] + n * n), "flops": _pair_flops(t, set(sp), len(sp))}
    if k == "set":
        sl = _slots(c)
        t = _terms(c["lmin"], c["lmax"], c["nW"])
        return {"bytes": 8 * (c["K"] * c["nW"] + len(sl) * n * n), "flops": _pair_flops(t, {s for _, s in sl}, c["K"])}
    if k in ("cov", "covset"):
        t = _terms(c["lmin"], c["lmax"], c["lmax"] + 1)
        names = {("TT", "TT"): "TTTT", ("EE", "EE"): "EEEE", ("TE", "TE"): "TETE", ("TT", "TE"): "TTTE",
                 ("TT", "EE"): "TTEE", ("TE", "EE"): "TEEE_PLANCK"}
        kinds = [names[c["ch1"], c["ch2"]]] if k == "cov" else [names[b] for b in syn.COV_BLOCKS[:c["nblk"]]]
        nw = sum(_COV_NW[x] for x in kinds)
        return {"bytes": 8 * ((nw + 8 * len(kinds)) * (c["lmax"] + 1) + len(kinds) * n * n),
                "flops": _pair_flops(t, set().union(*[_COV_SPINS[x] for x in kinds]), nw)}
    if k == "batch":
        b = f = 0
        for lmax, K, cases, _ in _batch_problems(c, 1):
            b += 8 * K * (lmax + 1 + len(_spins(cases)) * (lmax + 1) ** 2)
            f += _pair_flops(_terms(0, lmax, lmax + 1), set(_spins(cases)), K)
        return {"bytes": b, "flops": f}
    if k == "window":
        na = _n_alms(c["lmax"], c["mmax"])
        return {"bytes": 16 * na * c["nterms"] * (1 if c["auto"] else 2) + 8 * (c["lout"] + 1),
                "flops": 4 * na * c["nterms"]}
    if k == "quickpol":
        lpp = np.arange(2, c["lmax"] + 1)
        t = sum(int((2 * np.minimum(lpp, l) + 1).sum()) for l, lpp in
                ((l, lpp[(lpp >= l - c["bu"]) & (lpp <= l + c["bl"])]) for l in range(2, c["lmax"] + 1)))
        fams = 1 if (c["nu1"], c["s1"]) == (c["nu2"], c["s2"]) else 2
        return {"bytes": 8 * (c["nW"] + (c["lmax"] + 1) ** 2), "flops": t * (22 * fams + 3)}
    return {"bytes": 8 * (c["n"] ** 2 + 2 * c["n"] * c["nrhs"]),
            "flops": 2 * c["n"] ** 3 // 3 + 2 * c["n"] ** 2 * c["nrhs"]}


# ---- the results in 64-bit torch ----------------------------------------------------------------

def _couple(l1, l2, wins):
    """Xi of the pairs (l1 <= l2; sorted by l1, largest first) for windows (family product, parity, values
    laid end to end, each pair's first index and length): sum over l3 of (2 l3 + 1) W x / 4 pi with x the product
    "00", "22" or "02" of the families (l1 l2 l3; 0 0 0) and (l1 l2 l3; -2 2 0).

    Each family runs by the three-term relation a(j+1) f(j+1) + c (2j+1) f(j) + a(j) f(j-1) = 0 forward from
    |l1 - l2| and backward from l1 + l2, matched at l2 and normalised by sum (2j+1) f^2 = 1."""
    dev = l1.device
    need2 = any(w[0] != "00" for w in wins)
    need0 = any(w[0] != "22" for w in wins)
    a1, b2 = l1.double(), l2.double()
    count = torch.flip(torch.cumsum(torch.flip(torch.bincount(l1), [0]), 0), [0]).tolist()  # pairs with l1 >= t
    n0 = count[1] if len(count) > 1 else 0  # pairs with l1 >= 1
    z = lambda v: torch.full((n0,), v, dtype=torch.float64, device=dev)  # noqa: E731
    sides = []
    for fwd in (True, False):
        f, fo, a, g = z(1.0), z(0.0), z(0.0), z(1.0)
        N2, N0, S = z(0.0), z(0.0), [z(0.0) for _ in wins]
        for t in range(0, len(count) if fwd else len(count) - 1):
            m = n0 if t == 0 else (count[t] if fwd else count[t + 1])  # forward l1 >= t, backward l1 > t
            if fwd and t > 0:
                m = min(m, n0)
            p, q = a1[:m], b2[:m]
            j = (l2[:m] - l1[:m] + t) if fwd else (l1[:m] + l2[:m] - t)
            w = 2.0 * j.double() + 1.0
            even = t % 2 == 0
            x22 = f[:m] * f[:m]
            if need2:
                N2[:m] += w * x22
            if even and need0:
                N0[:m] += w * g[:m] * g[:m]
            for k, (prod, par, flat, base, length) in enumerate(wins):
                if (par == "even" and not even) or (par == "odd" and even) or (prod != "22" and not even):
                    continue
                ww = torch.where(j < length[:m], flat[base[:m] + torch.minimum(j, length[:m] - 1)], 0.0) * w
                x = x22 if prod == "22" else (g[:m] * g[:m] if prod == "00" else g[:m] * f[:m])
                S[k][:m] += ww * x
            if fwd:
                P = (t + 1.0) * (2 * (q - p) + t + 1) * (2 * p - t) * (2 * q + t + 2)
            else:
                P = (2 * p - t) * (2 * q - t) * (1.0 + t) * (2 * p + 2 * q + 1 - t)
            an = torch.sqrt(P)
            if need2:
                nf = -(4.0 * w * f[:m] + a[:m] * fo[:m]) / an
                fo[:m] = f[:m]
                f[:m] = nf
            if need0 and not even:
                g[:m] *= -a[:m] / an
            a[:m] = an
        sides.append((f, fo, g, N2, N0, S))
    (f, fo, g, FN2, FN0, FS), (h, ho, hg, BN2, BN0, BS) = sides
    lam2 = (fo * h + f * ho) / (h * h + ho * ho)
    lam0 = g / hg
    N2, N0 = FN2 + lam2 ** 2 * BN2, FN0 + lam0 ** 2 * BN0
    big = a1[:n0] >= 2
    out = []
    for k, (prod, par, flat, base, length) in enumerate(wins):
        X = torch.zeros(len(l1), dtype=torch.float64, device=dev)
        if prod == "00":
            X[:n0] = (FS[k] + lam0 ** 2 * BS[k]) / N0
            X[n0:] = torch.where(l2[n0:] < length[n0:], flat[base[n0:] + torch.minimum(l2[n0:], length[n0:] - 1)], 0.0)
        elif prod == "22":
            X[:n0] = torch.where(big, (FS[k] + lam2 ** 2 * BS[k]) / N2, 0.0)
        else:
            X[:n0] = torch.where(big, (FS[k] + lam0 * lam2 * BS[k]) * torch.sign(lam0 * lam2) / torch.sqrt(N0 * N2), 0.0)
        out.append(X / (4.0 * math.pi))
    return out


_SPIN_WIN = {0: ("00", "all"), 1: ("02", "even"), 2: ("22", "even"), 3: ("22", "odd")}


def _pairs(lmin, lmax):
    l1, l2 = torch.triu_indices(lmax - lmin + 1, lmax - lmin + 1, device="cuda") + lmin
    o = torch.argsort(l1, descending=True, stable=True)
    return l1[o], l2[o]


def _grid_xi(lmin, lmax, wins):
    """Symmetric n x n Xi matrices for windows (product, parity, spectrum)."""
    l1, l2 = _pairs(lmin, lmax)
    base = torch.zeros_like(l1)
    out = []
    for X in _couple(l1, l2, [(a, b, _dev(W), base, base + len(W)) for a, b, W in wins]):
        M = torch.empty((lmax - lmin + 1,) * 2, dtype=torch.float64, device="cuda")
        M[l1 - lmin, l2 - lmin] = X
        M[l2 - lmin, l1 - lmin] = X
        out.append(M)
    return out


def _weight(lmin, lmax):
    return 2.0 * torch.arange(lmin, lmax + 1, dtype=torch.float64, device="cuda") + 1.0


_COV_WIN = {"TTTT": ("00", "all"), "EEEE": ("22", "even"), "TTTE": ("00", "all"), "TETE": ("02", "even"),
            "TEEE": ("02", "even"), "TEEE_PLANCK": ("22", "even"), "TTEE": ("00", "all")}


def _cov_element(kind, S, R, X, lmin, lmax):
    """The analytic covariance element of each kind from its windows' Xi (symmetric in l1, l2)."""
    col = [_dev(s[lmin:lmax + 1])[:, None] for s in S]
    row = [x.reshape(1, -1) for x in col]
    rc = [_dev(r[lmin:lmax + 1])[:, None] for r in R]
    rr = [x.reshape(1, -1) for x in rc]
    g = [torch.sqrt(a * b) for a, b in zip(col, row)]   # geometric means over the two l
    p = [a * b for a, b in zip(rc, rr)]                 # noise ratio products over the two l
    add = [a + b for a, b in zip(col, row)]
    if kind in ("TTTT", "EEEE"):
        return (g[0] * g[1] * X[0] + g[2] * g[3] * X[1] + g[0] * X[2] * p[1] + g[1] * X[3] * p[0]
                + g[2] * X[4] * p[3] + g[3] * X[5] * p[2] + X[6] * p[0] * p[1] + X[7] * p[2] * p[3])
    if kind == "TTTE":
        return (g[0] * add[3] * X[0] + g[1] * add[2] * X[1] + add[3] * X[2] * p[0] + add[2] * X[3] * p[1]) / 2
    if kind == "TETE":
        return (g[0] * g[1] * X[0] + 0.5 * (col[2] * row[3] + col[3] * row[2]) * X[1] + g[0] * X[2] * p[1]
                + g[1] * X[3] * p[0] + X[4] * p[0] * p[1])
    if kind in ("TEEE", "TEEE_PLANCK"):
        return (g[0] * add[2] * X[0] + g[1] * add[3] * X[1] + add[2] * X[2] * p[0] + add[3] * X[3] * p[1]) / 2
    return ((col[0] * row[2] + col[2] * row[0]) * X[0] + (col[1] * row[3] + col[3] * row[1]) * X[1]) / 2


def _exact_cov(blocks, lmin, lmax):
    wins = []
    for kind, S, R, Ws in blocks:
        wins += [(("00", "all") if kind == "TETE" and k == 1 else _COV_WIN[kind]) + (W,) for k, W in enumerate(Ws)]
    X = _grid_xi(lmin, lmax, wins)
    out, at = [], 0
    for kind, S, R, Ws in blocks:
        out.append(_cov_element(kind, S, R, X[at:at + len(Ws)], lmin, lmax))
        at += len(Ws)
    return out


def _family(lo, hi, m3, dm, l1, l2):
    """(2 hi.max + 1) x elements values of the families (l1 l2 j; m1 m2 m3), m2 - m1 = dm, by the three-term
    relation j A(j+1) f(j+1) + B(j) f(j) + (j+1) A(j) f(j-1) = 0 from both ends of lo..hi, unit norm and the
    Condon-Shortley sign (-1)^(l1 - l2 - m3) at hi."""
    top = int(hi.max())
    a, b, lod, hid = l1.double(), l2.double(), lo, hi
    s, d = a + b + 1, a - b

    def A(j):
        return torch.sqrt(torch.clamp((j * j - d * d) * (s * s - j * j) * (j * j - m3 * m3), min=0.0))

    def B(j):
        return -(2 * j + 1) * ((a * (a + 1) - b * (b + 1)) * m3 - j * (j + 1) * dm)

    mid = (lod + hid) // 2
    up = torch.zeros((top + 2, len(a)), dtype=torch.float64, device=a.device)
    f, fp = torch.zeros_like(a), torch.zeros_like(a)
    for j in range(int(lod.min()), int(mid.max()) + 1):
        f = torch.where(lod == j, 1.0, f)
        fp = torch.where(lod == j, 0.0, fp)
        on = (lod <= j) & (j <= mid)
        up[j] = torch.where(on, f, up[j])
        if j == 0:
            n = -dm * f / A(1.0)
        else:
            n = -(B(float(j)) * f + (j + 1.0) * A(float(j)) * fp) / (j * A(j + 1.0))
        up[j + 1] = torch.where(on, n, up[j + 1])  # mid + 1 kept for the match
        f, fp = torch.where(on, n, f), torch.where(on, f, fp)
    i = torch.arange(len(a), device=a.device)
    u0, u1 = up[mid, i], up[mid + 1, i]
    h, hn = torch.zeros_like(a), torch.zeros_like(a)
    d0, d1 = torch.zeros_like(a), torch.zeros_like(a)
    dn = up
    for j in range(top, int(mid.min()), -1):
        h = torch.where(hid == j, 1.0, h)
        hn = torch.where(hid == j, 0.0, hn)
        on = (mid < j) & (j <= hid)
        dn[j] = torch.where(on, h, dn[j])
        n = -(B(float(j)) * h + j * A(j + 1.0) * hn) / ((j + 1.0) * A(float(j)))
        last = mid + 1 == j
        d1, d0 = torch.where(last, h, d1), torch.where(last, n, d0)
        h, hn = torch.where(on, n, h), torch.where(on, h, hn)
    lam = (u0 * d0 + u1 * d1) / (d0 * d0 + d1 * d1)
    jj = torch.arange(top + 2, device=a.device)[:, None]
    dn *= torch.where(jj > mid, lam, 1.0)
    norm = ((2.0 * jj + 1.0) * dn * dn).sum(0)
    sign = torch.where((l1 - l2 - m3) % 2 != 0, -1.0, 1.0) * torch.sign(lam)
    return dn * (sign / torch.sqrt(norm))


def _exact_quickpol(c, seed):
    lmax = c["lmax"]
    W = _dev(_masks(1, c["nW"], seed)[0])
    X = torch.zeros((lmax + 1, lmax + 1), dtype=torch.float64, device="cuda")
    ll = torch.arange(2, lmax + 1, device="cuda")
    lpp, l = torch.meshgrid(ll, ll, indexing="ij")
    on = (l >= lpp - c["bl"]) & (l <= lpp + c["bu"])
    P, L = lpp[on], l[on]
    for at in range(0, len(P), 1 << 17):  # elements at a time: two families of 2 lmax + 2 values each
        p, q = P[at:at + (1 << 17)], L[at:at + (1 << 17)]
        fam = []
        for nu, s in ((c["nu1"], c["s1"]), (c["nu2"], c["s2"])):
            m1, m2, m3 = -s, -nu, s + nu
            F = _family(torch.clamp((q - p).abs(), min=abs(m3)), q + p, m3, float(m2 - m1), q, p)
            F[:, (q < abs(m1)) | (p < abs(m2))] = 0.0
            fam.append(F)
        n = min(len(W), len(fam[0]))
        X[p, q] = (W[:n, None] * fam[0][:n] * fam[1][:n]).sum(0)
    return X * (-1.0) ** ((c["s1"] + c["s2"] + c["nu1"] + c["nu2"]) % 2)


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("mcm", "multi", "set"):
        lmin, lmax = c["lmin"], c["lmax"]
        nslot = len(_slots(c)) if k == "set" else 4
        if (lmax / 3071.0) ** 3 * (10 + 3 * nslot) > 200:  # over about 20 s of torch
            return None
        w = _weight(lmin, lmax)
        if k == "mcm":
            W = _masks(1, lmax + 1, seed)[0]
            M = [X * w[None, :] for X in _grid_xi(lmin, lmax, [_SPIN_WIN[s] + (W,) for s in SPIN_OF[c["spec"]]])]
            if len(M) == 1:
                return M[0]
            m = M[1] if c["spec"] == "EE_BB" else -M[1]
            return torch.cat([torch.cat([M[0], m], 1), torch.cat([m, M[0]], 1)], 0)
        if k == "multi":
            Ws = _masks(4, c["nW"], seed)
            wins = [_SPIN_WIN[s] + (Ws[s],) for s in _spins(c["cases"])]
        else:
            Ws = _masks(c["K"], c["nW"], seed)
            wins = [_SPIN_WIN[s] + (Ws[q],) for q, s in _slots(c)]
        return [X * w[:, None] for X in _grid_xi(lmin, lmax, wins)]  # column-major, as the call writes it
    if k == "cov":
        ws, spectra, noise = _cov_workspace(c["lmax"], seed)
        return _exact_cov([pgcov.gather(c["ch1"], c["ch2"], ws, spectra, noise)], c["lmin"], c["lmax"])[0]
    if k == "covset":
        ws, spectra, noise = _cov_workspace(c["lmax"], seed)
        return _exact_cov([pgcov.gather(a, b, ws, spectra, noise) for a, b in syn.COV_BLOCKS[:c["nblk"]]],
                          c["lmin"], c["lmax"])
    if k == "batch":
        probs = _batch_problems(c, seed)
        out = [None] * len(probs)
        for key in sorted({(p[1], p[2]) for p in probs}):  # the problems with one K and one spin together
            mine = [i for i, p in enumerate(probs) if (p[1], p[2]) == key]
            pr = [_pairs(0, probs[i][0]) for i in mine]
            l1, l2 = torch.cat([x for x, _ in pr]), torch.cat([y for _, y in pr])
            which = torch.repeat_interleave(torch.arange(len(mine), device="cuda"),
                                            torch.tensor([len(x) for x, _ in pr], device="cuda"))
            length = torch.tensor([probs[i][0] + 1 for i in mine], device="cuda")
            base = torch.cumsum(length, 0) - length
            o = torch.argsort(l1, descending=True, stable=True)
            flat = [_dev(np.concatenate([probs[i][3][q] for i in mine])) for q in range(key[0])]
            slots = [(q, s) for q in range(key[0]) for s in _spins(key[1])]
            X = _couple(l1[o], l2[o], [_SPIN_WIN[s] + (flat[q], base[which[o]], length[which[o]]) for q, s in slots])
            back = torch.empty_like(o)
            back[o] = torch.arange(len(o), device="cuda")
            at = 0
            for i, (x, y) in zip(mine, pr):
                n = probs[i][0] + 1
                w = _weight(0, n - 1)[:, None]
                mats = []
                for v in X:
                    v = v[back[at:at + len(x)]]
                    M = torch.empty((n, n), dtype=torch.float64, device="cuda")
                    M[x, y] = v
                    M[y, x] = v
                    mats.append((M * w).reshape(-1))
                out[i] = torch.cat(mats)
                at += len(x)
        return torch.cat(out)
    if k == "window":
        A, B = _window_sets(c, seed)
        W = torch.zeros(c["lmax"] + 1, dtype=torch.float64, device="cuda")
        for a, b in zip(A, B):
            v = (a * b).sum(1)
            at = 0
            for m in range(c["mmax"] + 1):
                W[m:] += (1.0 if m == 0 else 2.0) * v[at:at + c["lmax"] + 1 - m]
                at += c["lmax"] + 1 - m
        return (W / _weight(0, c["lmax"]) / c["nterms"])[:c["lout"] + 1]
    if k == "quickpol":
        return _exact_quickpol(c, seed)
    M, b = _solve_inputs(c, seed)
    x = torch.linalg.solve(M, b)
    return x if c["nrhs"] > 1 else x[:, 0]
