"""Launch forms of the FP64 step and its host transfers at the sizes where they change.

* Single-wave launches run BCON and the bookkeeping inside the stages, with the planes BCON reads
  in one, two or three chunks; larger launches cut the planned chunks: bit for bit the oracle's.
* The reverse sweep's BCON transpose takes one side per thread from npz = 6 on, both in turn below;
  its tiles are 32 x 8: dot products against the exact tangent.
* Host arrays are copied directly when page-locked or below 4 MB and through page-locked buffers in
  8 MB chunks when pageable: the same arrays either way.
"""
import numpy as np
import pytest

import r3d_b200 as R
from oracle import Oracle, interior
from tangent_np import NumpyStep

MAG = ["--lmag", "1", "--beta", "10", "--rm", "1", "--ampb", "0.1", "--bfh", "2", "--bzp", "20"]
I3 = (slice(1, -1),) * 3


def grid(nx, ny, nz, *extra):
    # fewer than 8 planes resolve the static column of a shallow domain only
    shallow = ["--zmax", "2"] if nz < 8 else []
    return ["--npx", str(nx), "--npy", str(ny), "--npz", str(nz), *shallow, *extra]


@pytest.mark.gpu
@pytest.mark.parametrize("flags,steps", [
    (grid(3, 3, 5), 3),                                   # every plane an edge plane's neighbour
    (grid(33, 9, 6, "--izcon", "1", "--itcon", "0"), 3),  # ragged tiles, flux bottom
    (grid(40, 30, 64, "--tp", "0"), 4),                   # one-plane chunks
    (grid(100, 61, 87), 3),                               # one wave of seven-plane chunks
    (grid(160, 96, 100), 2),                              # several waves, cut chunks
    (grid(33, 17, 5, *MAG), 3),
    (grid(64, 64, 40, *MAG), 2),
], ids=["3x3x5", "33x9x6", "40x30x64", "100x61x87", "160x96x100", "mhd33x17x5", "mhd64x64x40"])
def test_forward_bitexact(flags, steps):
    p = R.parse(flags + ["--seed", "8"])
    st = R.HostState.setup(p)
    with R.GpuSim(p) as sim:
        sim.upload(st)
        for _ in range(steps - 1):
            sim.step()
        sc = sim.step()
        sim.download(st)
    o = Oracle(flags).init(8)
    for _ in range(steps):
        o.step(3)
    for n in st.fields:
        assert np.array_equal(interior(st.fields[n]), interior(o.field(n))), n
    osc = o.scalars()
    for k in ("dt", "timc", "umach"):
        assert sc[k] == osc[k], k


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [
    grid(3, 3, 5), grid(33, 9, 6), grid(32, 8, 7, "--lrot", "1", "--ry", "2", "--ang", "0.4"),
    grid(5, 17, 5, *MAG), grid(34, 7, 8, *MAG),
    grid(12, 9, 9, "--pzp", "0.5", "--sigma", "0.1", "--polys", "1.5", *MAG),
], ids=["3x3x5", "33x9x6", "rotation", "mhd5x17x5", "mhd34x7x8", "mhd_kappa"])
def test_adjoint_step_dot_product(flags):
    p = R.parse(flags + ["--seed", "3"])
    names = R.FIELDS3D if p.lmag else R.FIELDS3D[:5]
    st = R.HostState.setup(p)
    rng = np.random.default_rng(7)
    ns = NumpyStep(Oracle(flags).init(3))
    with R.GpuSim(p) as sim:
        sim.upload(st)
        sim.run(2)
        sim.download(st)
        V, lam = {}, {}
        for n in names:
            V[n] = np.zeros_like(st.fields[n])
            V[n][I3] = rng.standard_normal(V[n][I3].shape)
            ns.ghost_fill(V[n])
            lam[n] = np.zeros_like(V[n])
            lam[n][I3] = rng.standard_normal(V[n][I3].shape)
        g = sim.adjoint_step(lam)
    h = 1e-30  # complex step: the exact tangent
    Y, _ = ns.run({n: st.fields[n] + 1j * h * V[n] for n in names}, 1)
    left = [lam[n][I3] * Y[n][I3].imag / h for n in names]
    right = [g[n][I3] * V[n][I3] for n in names]
    lhs, rhs = (sum(float(t.sum()) for t in s) for s in (left, right))
    # a value of either side is a sum of some 200 products in each of three stages, every one
    # rounded: 600 eps of the summed sizes
    size = sum(float(np.abs(t).sum()) for t in left + right)
    assert abs(lhs - rhs) <= 600 * 2.0 ** -53 * size, (lhs, rhs)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(20, 20, 30), (64, 64, 120), (64, 64, 300)],
                         ids=["direct", "one_chunk", "chunks"])  # 0.12, 4.3 and 10.5 MB per field
@pytest.mark.parametrize("precision", ["fp64", "fp32bulk"])
def test_pageable_and_page_locked_arrays(shape, precision):
    import torch

    p = R.parse(grid(*shape, "--seed", "5", "--precision", precision))
    st = R.HostState.setup(p)

    def locked(a):
        t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
        t.numpy()[...] = a
        return t.numpy()

    out = {}
    for kind in ("pageable", "locked"):
        src = st.copy()
        if kind == "locked":
            src.fields = {n: locked(a) for n, a in src.fields.items()}
        with R.GpuSim(p) as sim:
            sim.upload(src)
            sim.run(2)
            acc = sim.accumulators()
            sim.download(src)
            out[kind] = dict(src.fields, **acc)
            if precision == "fp64":
                out[kind].update(sim.work())
                out[kind].update({"F" + n: a for n, a in sim.fluxes().items()})
    for n, a in out["pageable"].items():
        assert np.array_equal(a, out["locked"][n]), n
    for n in out["pageable"]:
        assert np.isfinite(out["pageable"][n]).all(), n


@pytest.mark.gpu
@pytest.mark.parametrize("value,launches", [(None, 9), ("sixteen", 9), ("0", 9), ("16", 4)])
def test_depth_override(value, launches, monkeypatch):
    """160x96x100: the planned 16 planes per CTA are one wave (4 launches a step), which a handle cuts into several
    (9).  R3D_KCHUNK is taken as it is; what is ignored leaves the cut."""
    monkeypatch.delenv("R3D_KCHUNK", raising=False)
    if value is not None:
        monkeypatch.setenv("R3D_KCHUNK", value)
    p = R.parse(grid(160, 96, 100))
    with R.GpuSim(p) as sim:
        sim.setup()
        assert sim.run_timed(1)[1]["total_launches"] == launches
