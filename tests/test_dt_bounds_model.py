"""Host model of the third stage's skip rule (dt_skip, step_begin): on oracle states, in float32 as
the kernel forms it, every skipped cell has its CFL, conduction and viscosity limits above the
thresholds and its Mach term below (src/step.cpp:125-196), so the fold over the others is exact
whenever the check at the step's end passes; most cells are skipped; and hostile values (non-finite,
beyond float, zero, negative T) are never skipped.  FP32-bulk forms rho and T as background + deviation:
the same with values that nearly cancel their background."""
import numpy as np
import pytest

import r3d_b200 as R
from oracle import Oracle

MARGIN, WIDE = 1.0 / 64.0, 1.0 + 2.0 ** -10
MAG = ["--lmag", "1", "--beta", "10", "--rm", "1", "--ampb", "0.1", "--bfh", "2", "--bzp", "20"]
f = np.float32


def state(o, p, s=(slice(2, -2), slice(1, -1), slice(1, -1))):
    x = {n: o.field(n)[s] for n in ("ru", "rv", "rw", "ro", "tt") + (("bx", "by", "bz") if p.lmag else ())}
    a, b, c = (o.line(n) for n in ("ddx", "ddy", "ddz"))
    dd = np.minimum(np.minimum(a[None, None, 1:-1], b[None, 1:-1, None]), c[2:-2, None, None])
    return x, dd, o.line("rkapa")[2:-2, None, None] + 0.0 * dd


def limits(x, dd, rk, p, c):
    r = 1.0 / x["ro"]
    uu = (x["ru"] ** 2 + x["rv"] ** 2 + x["rw"] ** 2) * r * r
    um = (1.0 / p.gamma) * uu / x["tt"]
    s = p.gamma * x["tt"]
    if p.lmag:
        s = s + (x["bx"] ** 2 + x["by"] ** 2 + x["bz"] ** 2) * c["obeta"] / x["ro"]
    w1 = dd / np.sqrt(uu + s + 2.0 * np.sqrt(uu * s))
    w2 = 0.5 * dd * dd * c["repr"] * c["cv"] * x["ro"] / rk
    return w1, w2, 0.375 * dd * dd * p.re * x["ro"], um


def skip(x, dd, rk, p, c, t, tu, bg=None, share=2.0 ** -8):
    """bg: rho and T of the FP32-bulk background, whose deviations are the stored floats; its estimates are
    sums, trusted from share of the background on."""
    s = np.sqrt(tu)
    u, a1, a2, a3 = (f(v) for v in (tu * p.gamma / WIDE, t[0] ** 2 * WIDE * (1 + 1 / s),
                                    t[0] ** 2 * WIDE * (1 + s) * p.gamma, t[0] ** 2 * WIDE * (1 + s) * c["obeta"]))
    q2, q3 = f(t[1] * WIDE / (0.5 * c["repr"] * c["cv"])), f(t[2] * WIDE / (0.375 * p.re))
    ru, rv, rw, ro, tt = (x[n].astype(f) for n in ("ru", "rv", "rw", "ro", "tt"))
    low = {n: f(2.0 ** -30) for n in ("ro", "tt")}
    if bg is not None:
        ro, tt = (bg[n].astype(f) + (x[n] - bg[n]).astype(f) for n in ("ro", "tt"))
        low = {n: np.maximum(low[n], f(share) * bg[n].astype(f)) for n in ("ro", "tt")}
    d = dd.astype(f)
    dd2, msq, r2 = d * d, ru * ru + rv * rv + rw * rw, ro * ro
    tr2, bc = tt * r2, f(0)
    if p.lmag:
        bc = a3 * ((x["bx"] ** 2 + x["by"] ** 2 + x["bz"] ** 2).astype(f) * ro)
    inside = (ro >= low["ro"]) & (ro < f(2.0 ** 30)) & (tt >= low["tt"]) & (tt < f(2.0 ** 30))
    return inside & (msq < u * tr2) & (dd2 * r2 > a1 * msq + a2 * tr2 + bc) & \
        (dd2 * ro > np.maximum(q2 * rk.astype(f), q3))


@pytest.mark.parametrize("flags,seed", [
    (["--npx", "32", "--npy", "32", "--npz", "64"], 1),
    (["--npx", "20", "--npy", "16", "--npz", "40", "--pzp", "0.5", "--sigma", "0.1", "--polys", "1.5"], 5),
    (["--npx", "20", "--npy", "16", "--npz", "32"] + MAG, 7),
], ids=["hydro", "variable_kappa", "mhd"])
def test_skipped_cells_cannot_matter(flags, seed):
    p = R.parse(flags)
    c = {n: R.derived(p, n) for n in ("obeta", "repr", "cv")}
    o = Oracle(flags).init(seed)
    prev, seen = None, 0
    with np.errstate(all="ignore"):
        for _ in range(6):
            x, dd, rk = state(o, p)
            w = limits(x, dd, rk, p, c)
            if prev is not None and prev[3] > 0:
                t, tu = [v * (1 + MARGIN) for v in prev[:3]], prev[3] * (1 - MARGIN)
                sk = skip(x, dd, rk, p, c, t, tu)
                assert all((w[q][sk] > t[q]).all() for q in range(3)) and (w[3][sk] < tu).all()
                keep = ~sk
                if keep.any() and all(np.nanmin(w[q][keep]) <= t[q] for q in range(3)) and np.nanmax(w[3][keep]) >= tu:
                    assert all(np.nanmin(w[q][keep]) == np.nanmin(w[q]) for q in range(3))
                    assert np.nanmax(w[3][keep]) == np.nanmax(w[3])
                seen = max(seen, sk.mean())
                for n, v in (("tt", -1.0), ("tt", np.nan), ("ro", 0.0), ("ro", np.inf), ("ru", 1e30), ("ru", np.nan),
                             ("rw", np.inf), ("tt", 1e300)):
                    y = {k: a.copy() for k, a in x.items()}
                    y[n][...] = v
                    assert not skip(y, dd, rk, p, c, t, tu).any(), (n, v)
            prev = [np.nanmin(v) for v in w[:3]] + [np.nanmax(w[3])]
            o.step(3)
    assert seen > 0.8, seen


def test_fp32bulk_sums_that_cancel():
    """rho and T from 2^-24 of their background up, every cell's limits close to the thresholds: no cell whose
    limits matter is skipped (with the window of correctly rounded inputs, 2^-30, some are)."""
    p = R.parse(["--npx", "8", "--npy", "8", "--npz", "8"])
    c = {n: R.derived(p, n) for n in ("obeta", "repr", "cv")}
    rng = np.random.default_rng(1)
    n = 400000
    bg = {q: 1.0 + 9.0 * rng.random(n) for q in ("ro", "tt")}
    # deviations are floats: the state is background + float
    x = {q: bg[q] + (bg[q] * (2.0 ** rng.uniform(-24, 1, n) - 1.0)).astype(f) for q in bg}
    ok = (x["ro"] > 0) & (x["tt"] > 0)
    x, bg = {q: a[ok] for q, a in x.items()}, {q: a[ok] for q, a in bg.items()}
    n = ok.sum()
    tu = 0.04
    um = tu * rng.uniform(0.98, 1.02, n)
    m = np.sqrt(um * p.gamma * x["tt"] * x["ro"] ** 2 / 3.0).astype(f).astype(float)
    x.update(ru=m, rv=m, rw=m)
    rk = np.ones(n)
    # spacings that put a cell's CFL limit, conduction limit or viscosity limit near its threshold of 1
    w = limits(x, np.ones(n), rk, p, c)
    need = np.maximum(1.0 / w[0], np.minimum(w[1], w[2]) ** -0.5)
    dd = need * rng.uniform(0.99, 1.03, n)
    w = limits(x, dd, rk, p, c)
    t = [1.0, 1.0, 1.0]

    def wrong(share):
        sk = skip(x, dd, rk, p, c, t, tu, bg, share)
        bad = sk & ~((w[0] > t[0]) & (w[1] > t[1]) & (w[2] > t[2]) & (w[3] < tu))
        return int(bad.sum()), int(sk.sum())

    assert wrong(0.0)[0] > 0
    bad, skipped = wrong(2.0 ** -8)
    assert bad == 0 and skipped > n // 100, (bad, skipped)
