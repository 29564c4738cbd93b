"""The workloads whose speed is followed, through the framework's Python interface.

Five kinds of work, each as a simulation program has it do:

  run      N steps in one call (GpuSim.run), then the state copied to the host, as between two
           dumps of a production run (the default interval is 100 steps)
  steps    the time loop of the command line driver: one GpuSim.step per step, each returning its
           scalars (dt, Mach number, times), then the state copied to the host
  adjoint  a start state uploaded, N steps recorded with checkpoints, the final state copied to
           the host, and the reverse sweep from a cotangent of it to the gradient of the start
           state: one iteration of an optimisation over initial states
  vjp      the one-step vector-Jacobian product at the current state (GpuSim.adjoint_step)
  fluxes   the right-hand sides of the current state as host arrays (GpuSim.fluxes)

The initial states are the framework's own: the static polytrope with the seeded temperature
perturbation (and the magnetic layer with MHD), default physics with the plume at the top.  Host
buffers are page-locked, as in a program that dumps often.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rast-3dmhd_b200", "python"))
import r3d_b200 as R  # noqa: E402

HYDRO = ["ru", "rv", "rw", "ro", "tt"]
MHD = HYDRO + ["bx", "by", "bz"]
PRESTEPS = 5  # steps a vjp or fluxes state has behind it, so that it is in motion


def _case(name, kind, nx, ny, nz, steps, mhd=False, fp32=False, rotation=False, kappa=False, ngrid=1, every=0):
    return {"name": name, "kind": kind, "npx": nx, "npy": ny, "npz": nz, "steps": steps, "mhd": mhd, "fp32": fp32,
            "rotation": rotation, "kappa": kappa, "ngrid": ngrid, "every": every}


def listed():
    return [
        # the parity grid, whose whole state fits in L2: launches and the host round trip per step count
        _case("hydro 32x32x64 steps", "steps", 32, 32, 64, 100),
        # a mid-size production cut; the benchmark grid of the notes on small launches
        _case("hydro 128x128x256 run", "run", 128, 128, 256, 100),
        # ragged tiles in x, y and z, rotation, a conductivity that varies with depth, two-arctan grid
        _case("hydro 250x131x187 rot kappa", "run", 250, 131, 187, 100, rotation=True, kappa=True, ngrid=2),
        # the headline benchmark grid (the largest ones with fewer steps, to keep a pass below a second)
        _case("hydro 504x504x512 run", "run", 504, 504, 512, 40),
        # the MHD grid of the adjoint case stepped forward by the driver's loop
        _case("mhd 64x64x128 steps", "steps", 64, 64, 128, 100, mhd=True),
        # the MHD benchmark grid
        _case("mhd 126x126x256 run", "run", 126, 126, 256, 100, mhd=True),
        # MHD that fills the GPU many times over
        _case("mhd 252x252x256 run", "run", 252, 252, 256, 40, mhd=True),
        # the reduced-precision form, a small grid and the benchmark's horizontal extent
        _case("fp32 126x126x256 run", "run", 126, 126, 256, 100, fp32=True),
        _case("fp32 504x504x256 run", "run", 504, 504, 256, 40, fp32=True),
        # the adjoint benchmark grid: a tenth of its trajectory, its checkpoint spacing halved
        _case("adjoint mhd 64x64x128", "adjoint", 64, 64, 128, 20, mhd=True, every=10),
        # one vector-Jacobian product of a larger hydro state (Newton-Krylov, sensitivities)
        _case("vjp hydro 128x128x128", "vjp", 128, 128, 128, 1),
        # the FLUXES entry point, as analysis and dumps call it
        _case("fluxes mhd 126x126x128", "fluxes", 126, 126, 128, 0, mhd=True),
    ]


def draw(rng):
    def extent(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "steps", "adjoint", "vjp", "fluxes"])
    mhd = rng.random() < 0.4
    fp32 = not mhd and kind in ("run", "steps") and rng.random() < 0.4
    rotation, kappa = rng.random() < 0.3, rng.random() < 0.3
    ngrid = rng.choice([0, 1, 1, 2])
    if kind in ("run", "steps"):
        nx, ny, nz, steps, every = extent(24, 504), extent(24, 504), extent(32, 512), rng.choice([20, 50, 100]), 0
        most = (800_000_000 if kind == "run" else 100_000_000) // steps
    else:
        nx, ny, nz = extent(24, 160), extent(24, 160), extent(32, 192)
        steps = rng.choice([4, 10]) if kind == "adjoint" else (1 if kind == "vjp" else 0)
        every = rng.choice([2, 4, 5]) if kind == "adjoint" else 0
        most = 1_000_000
    while nx * ny * nz > most:
        nx, ny, nz = max(24, nx * 3 // 4), max(24, ny * 3 // 4), max(32, nz * 3 // 4)
    c = _case("", kind, nx, ny, nz, steps, mhd, fp32, rotation, kappa, ngrid, every)
    del c["name"]
    return c


def _params(c, seed):
    a = ["--npx", c["npx"], "--npy", c["npy"], "--npz", c["npz"], "--ngrid", c["ngrid"], "--seed", 1 + seed % 700000]
    if c["mhd"]:
        a += ["--lmag", 1, "--beta", 10, "--rm", 1, "--ampb", 0.1, "--bfh", 2, "--bzp", 20]
    if c["rotation"]:
        a += ["--lrot", 1, "--ry", 2, "--ang", 0.3]
    if c["kappa"]:
        a += ["--pzp", 0.5, "--sigma", 0.1, "--polys", 1.5]
    if c["fp32"]:
        a += ["--precision", "fp32bulk"]
    return R.parse([str(v) for v in a])


def _names(c):
    return MHD if c["mhd"] else HYDRO


def _shape(p):
    nx, ny, nz = R.dims(p)
    return nz, ny, nx


def _host_fields(c, p):
    """Page-locked host arrays for the state's fields (the metric lines are not downloaded)."""
    f = {n: torch.empty(_shape(p), dtype=torch.float64, pin_memory=torch.cuda.is_available()) for n in _names(c)}
    return R.HostState({n: t.numpy() for n, t in f.items()}, R.HostState.empty_slab(p, 4).lines, {})


def _cotangent(c, p, seed):
    """A cotangent of the final state: noise of unit size on the interior (a misfit against data)."""
    rng = np.random.default_rng(seed)
    lam = {}
    for n in _names(c):
        lam[n] = np.zeros(_shape(p))
        lam[n][1:-1, 1:-1, 1:-1] = rng.standard_normal((p.npz, p.npy, p.npx))
    return lam


def prepare(case, seed):
    p = _params(case, seed)
    s = {"case": case, "sim": R.GpuSim(p)}
    if case["kind"] == "adjoint":
        st = R.HostState.setup(p)
        s["start"] = _host_fields(case, p)
        for n in _names(case):
            s["start"].fields[n][...] = st.fields[n]
        s["start"].lines, s["start"].scalars = st.lines, st.scalars
        s["lam"] = _cotangent(case, p, seed)
    else:
        s["sim"].setup()
    if case["kind"] in ("run", "steps", "adjoint"):
        s["host"] = _host_fields(case, p)
    else:
        s["sim"].run(PRESTEPS)
    if case["kind"] == "vjp":
        s["lam"] = _cotangent(case, p, seed)
    return s


def run(state):
    c, sim = state["case"], state["sim"]
    if c["kind"] == "fluxes":
        return sim.fluxes()
    if c["kind"] == "vjp":
        return sim.adjoint_step(state["lam"])
    if c["kind"] == "adjoint":
        sim.upload(state["start"])
        sc = sim.adjoint_record(c["steps"], c["every"])
        sim.download(state["host"])
        grad = sim.adjoint_backward(state["lam"])
        return {"state": state["host"].fields, "grad": grad, "dt": sc["dt"], "timc": sc["timc"]}
    if c["kind"] == "steps":
        for _ in range(c["steps"]):
            sc = sim.step()
    else:
        sc = sim.run(c["steps"])
    sim.download(state["host"])
    return {"state": state["host"].fields, "dt": sc["dt"], "timc": sc["timc"], "umach": sc["umach"]}


def work(case):
    """Bytes: per step, each of the three stages of the low-storage scheme reads the state and its
    accumulator once and writes them once (15, 20 and 15 field passes for five fields: a stage needs
    its neighbours' results of the one before); the copies to and from the host once.  A reverse
    step reads each stage's state and the cotangent and writes the cotangent.  Operations: the
    flux terms and the update of a cell, about 340 (hydro) and 700 (MHD) per stage; twice that for
    the reverse of a stage."""
    nf = 8 if case["mhd"] else 5
    cells = case["npx"] * case["npy"] * case["npz"]
    word = 4 if case["fp32"] else 8
    ops = 700 if case["mhd"] else 340
    host = nf * cells * 8
    step_b, step_f = 10 * nf * word * cells, 3 * ops * cells
    back_b, back_f = 9 * nf * word * cells, 6 * ops * cells
    n = case["steps"]
    if case["kind"] in ("run", "steps"):
        return {"bytes": n * step_b + host, "flops": n * step_f}
    if case["kind"] == "adjoint":
        return {"bytes": n * (step_b + back_b) + 4 * host, "flops": n * (step_f + back_f)}
    if case["kind"] == "vjp":
        return {"bytes": step_b + back_b + 2 * host, "flops": step_f + back_f}
    return {"bytes": 3 * host, "flops": ops * cells}


def tolerance(case):
    """Stepping and fluxes in FP64 are defined to the last bit (the order of every sum is part of
    the method), so they stay the same.  The reduced-precision form rounds its deviations to 32
    bits per stage (3e-7 off the 64-bit result after 100 steps, the same again between two such
    runs); the reverse sweep's sums may be taken in another order (1.2e-16 off plain torch's)."""
    if case["fp32"]:
        return {"rel": 1.2e-6}
    if case["kind"] in ("adjoint", "vjp"):
        return {"rel": 2e-15, "max": 1e-12}
    return "exact"


# ------------------------------------------------------------------ the same work in plain torch, in 64 bits


class _Plain:
    """One step of the scheme on tensors of the whole z range (ghost planes included) and the
    periodic interior in x and y."""

    def __init__(self, c, p, st):
        self.c, self.p = c, p
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        f32 = lambda v: float(np.float32(v))  # noqa: E731  (the scheme's constants are single-precision literals)
        L = st.lines
        x = {n: self.t(L[n][1:-1])[None, None, :] for n in ("exx", "dxxdx", "d2xxdx2", "ddx")}
        y = {n: self.t(L[n][1:-1])[None, :, None] for n in ("wyy", "dyydy", "d2yydy2", "ddy")}
        z = {n: self.t(L[n][1:-1])[:, None, None] for n in ("dzzdz", "d2zzdz2", "ddz", "rkapa", "dkapa")}
        h = {a: f32(0.5 * (n - 1)) for a, n in (("x", p.npx), ("y", p.npy), ("z", p.npz))}
        h2 = {a: f32((n - 1) * (n - 1)) for a, n in (("x", p.npx), ("y", p.npy), ("z", p.npz))}
        self.first = {"x": h["x"] * x["dxxdx"], "y": h["y"] * y["dyydy"], "z": h["z"] * z["dzzdz"]}
        self.second = {"x": (h["x"] * x["d2xxdx2"], h2["x"] * x["dxxdx"] ** 2),
                       "y": (h["y"] * y["d2yydy2"], h2["y"] * y["dyydy"] ** 2),
                       "z": (h["z"] * z["d2zzdz2"], h2["z"] * z["dzzdz"] ** 2)}
        self.rk, self.dk = z["rkapa"], z["dkapa"]
        self.dd = torch.minimum(torch.minimum(x["ddx"], y["ddy"]), z["ddz"])
        self.c13 = f32(1.0 / 3.0)
        self.c43 = 4.0 * self.c13
        self.cv = 1.0 / (p.gamma - 1.0)
        self.repr = p.re * p.pr
        self.obeta, self.orm = (2.0 / p.beta, 1.0 / p.rm) if p.lmag else (0.0, 0.0)
        self.omx, self.omz = (math.sin(p.ang) / p.r_y, math.cos(p.ang) / p.r_y) if p.lrot else (0.0, 0.0)
        self.gam = [f32(8 / 15), f32(5 / 12), f32(3 / 4)]
        self.zeta = [0.0, f32(-17 / 60), f32(-5 / 12)]
        self.tb = st.scalars["tb"]
        cln = f32(np.float32(-4.0) * np.log(np.float32(2.0))) / (p.hh * p.hh)
        plume = torch.exp(cln * (x["exx"] - p.xp) ** 2) / p.hh * torch.exp(cln * (y["wyy"] - p.yp) ** 2) / p.hh
        self.top = 2.0 * self.c13 * f32(1.0 / (p.npz - 1)) / L["dzzdz"][1] * (p.theta - (p.theta - p.tp) * plume[0])
        self.X = {n: self.t(st.fields[n][:, 1:-1, 1:-1]) for n in _names(c)}

    def d(self, f, a):
        """First derivative along a: x and y on every plane given, z on the inner planes."""
        if a == "z":
            return (f[2:] - f[:-2]) * self.first["z"]
        return (torch.roll(f, -1, "yx".index(a) + 1) - torch.roll(f, 1, "yx".index(a) + 1)) * self.first[a]

    def dd2(self, f, a):
        s, l = self.second[a]
        if a == "z":
            return (f[2:] - f[:-2]) * s + (f[2:] - 2.0 * f[1:-1] + f[:-2]) * l
        up, dn = torch.roll(f, -1, "yx".index(a) + 1), torch.roll(f, 1, "yx".index(a) + 1)
        return (up - dn) * s + (up - 2.0 * f + dn) * l

    def one_sided(self, inner, f):
        """The first z derivative with the one-sided forms on the first and last plane."""
        z = self.first["z"]
        top = (4.0 * f[2] - f[3]) * z[0]
        bot = (f[-4] - 4.0 * f[-3]) * z[-1]
        return torch.cat([top[None], inner[1:-1], bot[None]])

    def one_sided2(self, f):
        inner, (s, l) = self.dd2(f, "z"), self.second["z"]
        top = (-3.0 * f[1] + 4.0 * f[2] - f[3]) * s[0] + (2.0 * f[1] - 5.0 * f[2] + 4.0 * f[3] - f[4]) * l[0]
        bot = (3.0 * f[-2] - 4.0 * f[-3] + f[-4]) * s[-1] + (2.0 * f[-2] - 5.0 * f[-3] + 4.0 * f[-4] - f[-5]) * l[-1]
        return torch.cat([top[None], inner[1:-1], bot[None]])

    def fluxes(self, X):
        p, d, q = self.p, self.d, lambda f: f[1:-1]
        ore, ocv, c13, c43 = 1.0 / p.re, 1.0 / self.cv, self.c13, self.c43
        r = 1.0 / X["ro"]
        m = [X["ru"], X["rv"], X["rw"]]
        v = [a * r for a in m]
        T, ri, P = q(X["tt"]), q(r), X["ro"] * X["tt"]
        F = {"ro": -d(q(m[0]), "x") - d(q(m[1]), "y") - self.one_sided(d(m[2], "z"), m[2])}
        g = {}
        for a, f in zip("uvw", v):
            g[a, "x"], g[a, "y"], g[a, "z"] = d(q(f), "x"), d(q(f), "y"), d(f, "z")
        div = g["u", "x"] + g["v", "y"] + g["w", "z"]
        dP = [d(q(P), "x"), d(q(P), "y"), d(P, "z")]
        for a, (n, mom, f) in enumerate(zip(("ru", "rv", "rw"), m, v)):
            e = "xyz"[a]
            adv = d(q(mom * v[0]), "x") + d(q(mom * v[1]), "y") + d(mom * v[2], "z")
            lap = sum((c43 if b == e else 1.0) * self.dd2(f if b == "z" else q(f), b) for b in "xyz")
            # the cross differences d/de of the other velocities' own derivatives
            cross = sum(self.d_of(v[b], "xyz"[b], e) for b in range(3) if b != a)
            F[n] = -dP[a] - adv + ore * lap + c13 * ore * cross
        F["rw"] = F["rw"] + p.grav * q(X["ro"])
        dT = [d(q(X["tt"]), "x"), d(q(X["tt"]), "y"), d(X["tt"], "z")]
        lapT = sum(self.dd2(X["tt"] if b == "z" else q(X["tt"]), b) for b in "xyz")
        heat = (c43 * g["u", "x"] ** 2 + g["v", "x"] ** 2 + g["w", "x"] ** 2 + g["u", "y"] ** 2 + 2.0 * g["u", "y"] * g["v", "x"]
                + g["u", "z"] ** 2 + g["v", "z"] ** 2 + g["w", "y"] ** 2 + 2.0 * g["v", "z"] * g["w", "y"]
                + 2.0 * g["u", "z"] * g["w", "x"]
                + c43 * (g["v", "y"] ** 2 + g["w", "z"] ** 2 - g["u", "x"] * g["w", "z"] - g["u", "x"] * g["v", "y"]
                         - g["v", "y"] * g["w", "z"]))
        F["tt"] = (-sum(q(v[a]) * dT[a] for a in range(3)) + ocv / self.repr * ri * (lapT * self.rk + dT[2] * self.dk)
                   + ocv * ore * ri * heat - ocv * div * T)
        if p.lrot:
            ru, rv, rw = (q(a) for a in m)
            F["ru"] = F["ru"] + self.omz * rv
            F["rv"] = F["rv"] - self.omz * ru + self.omx * rw
            F["rw"] = F["rw"] - self.omx * rv
        if not self.c["mhd"]:
            return F
        B = [X["bx"], X["by"], X["bz"]]
        b = [q(f) for f in B]
        u, w = [q(f) for f in v], self.one_sided(g["w", "z"], v[2])
        D = {(a, e): d(B[a] if e == "z" else q(B[a]), e) for a in range(3) for e in "xyz"}
        J = [D[2, "y"] - D[1, "z"], D[0, "z"] - D[2, "x"], D[1, "x"] - D[0, "y"]]
        for a, n in enumerate(("ru", "rv", "rw")):
            i, j = (a + 1) % 3, (a + 2) % 3
            F[n] = F[n] + self.obeta * (J[i] * b[j] - J[j] * b[i])
        F["tt"] = F["tt"] + self.obeta * self.orm * ocv * ri * (J[0] ** 2 + J[1] ** 2 + J[2] ** 2)
        adv = [sum(u[e] * D[a, "xyz"[e]] for e in range(3)) for a in range(3)]
        # dw/dz is one-sided on the first and last plane in the Bx and By equations
        F["bx"] = (b[1] * g["u", "y"] - b[0] * g["v", "y"] + b[2] * g["u", "z"] - b[0] * w - adv[0]
                   + self.orm * (self.dd2(b[0], "x") + self.dd2(b[0], "y") + self.one_sided2(B[0])))
        F["by"] = (b[0] * g["v", "x"] - b[1] * g["u", "x"] + b[2] * g["v", "z"] - b[1] * w - adv[1]
                   + self.orm * (self.dd2(b[1], "x") + self.dd2(b[1], "y") + self.one_sided2(B[1])))
        F["bz"] = (b[0] * g["w", "x"] - b[2] * g["u", "x"] + b[1] * g["w", "y"] - b[2] * g["v", "y"] - adv[2]
                   + self.orm * (self.dd2(b[2], "x") + self.dd2(b[2], "y") + self.dd2(B[2], "z")))
        return F

    def d_of(self, f, inner, outer):
        """d/d(outer) of d f/d(inner), the inner difference with its own metric at each cell."""
        if outer == "z":  # d/dz is the inner one (the metric of the output plane), then x or y
            return self.d(self.d(f, "z"), inner)
        g = self.d(f, "z") if inner == "z" else self.d(f[1:-1], inner)
        return self.d(g, outer)

    def boundary(self, X):
        """The first and last plane from the two inside them."""
        c13, c43, p, new = self.c13, self.c43, self.p, {}
        for n, f in X.items():
            top, bot = f[1], f[-2]
            if n in ("ru", "rv"):
                ro = X["ro"]
                top = ro[1] * (c43 * f[2] / ro[2] - c13 * f[3] / ro[3])
                bot = ro[-2] * (c43 * f[-3] / ro[-3] - c13 * f[-4] / ro[-4])
            elif n in ("rw", "bz"):
                top, bot = torch.zeros_like(top), torch.zeros_like(bot)
            elif n == "tt":
                top = c43 * f[2] - c13 * f[3] - self.top
                bot = torch.full_like(bot, self.tb)
            new[n] = torch.cat([f[:1], top[None], f[2:-2], bot[None], f[-1:]])
        return new

    def limits(self, X):
        p, q, dd = self.p, {n: f[1:-1] for n, f in X.items()}, self.dd
        uu = (q["ru"] ** 2 + q["rv"] ** 2 + q["rw"] ** 2) / q["ro"] ** 2
        um = (uu / (p.gamma * q["tt"])).max()
        s = p.gamma * q["tt"]
        if self.c["mhd"]:
            s = s + (q["bx"] ** 2 + q["by"] ** 2 + q["bz"] ** 2) * self.obeta / q["ro"]
        moving = uu > 0  # at rest the mixed term and its derivative are 0
        mixed = torch.where(moving, torch.sqrt(torch.where(moving, uu * s, torch.ones_like(s))), torch.zeros_like(s))
        w = [dd / torch.sqrt(uu + s + 2.0 * mixed), 0.5 * dd * dd * self.repr * self.cv * q["ro"] / self.rk,
             0.375 * dd * dd * p.re * q["ro"]]
        best = None
        for f in w:
            low = torch.nan_to_num(f.detach(), nan=math.inf).min()  # a cell without a limit (T < 0 in the plume) sets none
            if best is None or low < best.detach():
                best = f[tuple((f.detach() == low).nonzero()[0])]  # the first of equal cells
        if self.c["mhd"] and (0.5 * dd * dd * p.rm).min() < best.detach():
            best = (0.5 * dd * dd * p.rm).min()
        return p.sf * best, torch.sqrt(um.detach())

    def step(self, X):
        dt, mach = self.limits(X)
        Z = {n: f[1:-1] for n, f in X.items()}
        for s in range(3):
            F = self.fluxes(X)
            inner = {n: Z[n] + self.gam[s] * dt * F[n] for n in X}
            if s < 2:
                full = {n: torch.cat([X[n][:1], inner[n], X[n][-1:]]) for n in X}
                full = self.boundary(full)
                # the accumulator of the next stage restarts from the state the boundary left
                Z = {n: full[n][1:-1] + self.zeta[s + 1] * dt * F[n] for n in X}
                # on the boundary planes the framework's fluxes of what is rewritten there do not count
                X = full
            else:
                X = self.boundary({n: torch.cat([X[n][:1], inner[n], X[n][-1:]]) for n in X})
        return X, dt, mach

    def whole(self, X):
        """Tensors of the periodic interior as host arrays with their x and y ghost cells."""
        return {n: torch.nn.functional.pad(f.detach()[None], (1, 1, 1, 1), mode="circular")[0].cpu().numpy() for n, f in X.items()}

    def alone(self, X):
        """Tensors of interior planes as host arrays whose ghost cells are zero."""
        return {n: torch.nn.functional.pad(f.detach(), (1, 1, 1, 1, 1, 1)).cpu().numpy() for n, f in X.items()}


def exact(case, seed):
    cells = case["npx"] * case["npy"] * case["npz"]
    if cells * max(1, case["steps"]) > 420_000_000:
        return None
    p = _params(case, seed)
    S = _Plain(case, p, R.HostState.setup(p))
    X, time = S.X, 0.0
    if case["kind"] in ("vjp", "fluxes"):
        for _ in range(PRESTEPS):
            X, _, _ = S.step(X)
    if case["kind"] == "fluxes":
        F = S.fluxes(X)
        for n in ("ru", "rv", "rw", "tt"):  # the boundary rewrites these there: no flux is formed
            F[n] = torch.cat([0.0 * F[n][:1], F[n][1:-1], 0.0 * F[n][-1:]])
        names = dict(zip(MHD, ("fu", "fv", "fw", "fr", "ft", "w1", "w2", "w3")))
        return {names[n]: a for n, a in S.alone(F).items()}
    states = [X]
    for _ in range(case["steps"]):
        X, dt, mach = S.step(X)
        time += float(dt)
        states = states + [X] if case["kind"] in ("adjoint", "vjp") else [X]
    out = {"state": S.whole(X), "dt": float(dt), "timc": time, "umach": float(mach)}
    if case["kind"] in ("run", "steps"):
        return out
    lam = {n: S.t(a[:, 1:-1, 1:-1]) for n, a in _cotangent(case, p, seed).items()}
    for X in reversed(states[:-1]):
        X = {n: f.detach().requires_grad_() for n, f in X.items()}
        Y, _, _ = S.step(X)
        names = list(X)
        lam = dict(zip(names, torch.autograd.grad([Y[n] for n in names], [X[n] for n in names], [lam[n] for n in names])))
        lam = {n: torch.cat([0.0 * f[:1], f[1:-1], 0.0 * f[-1:]]) for n, f in lam.items()}  # ghost planes are constants
    grad = S.alone({n: f[1:-1] for n, f in lam.items()})
    del out["umach"]
    return grad if case["kind"] == "vjp" else {**out, "grad": grad}
