"""FP32-bulk: the forms a stage launch can take give the same bits.

BCON runs inside the stages of a single-wave launch and in a kernel of its own after the others; which one a
handle takes follows from its planes per CTA and its slab, so a slab, a domain and an R3D_KCHUNK setting meet both.
"""
import numpy as np
import pytest

import r3d_b200 as R

BC = {
    "plume_constant": ["--itcon", "0"],
    "plume_flux": ["--itcon", "1", "--hh", "0.7"],
    "constant": ["--itcon", "0", "--tp", "0", "--izcon", "1"],
    "half": ["--itcon", "4"],
    "kappa": ["--pzp", "0.5", "--sigma", "0.1", "--polys", "1.5", "--izcon", "1"],
}


def params(shape, extra):
    flags = [f for n, v in zip(("--npx", "--npy", "--npz"), shape) for f in (n, str(v))]
    return R.parse(flags + ["--seed", "4", "--precision", "fp32bulk", *extra])


def domain(p, launches):
    st = R.HostState.setup(p)
    with R.GpuSim(p) as sim:
        sim.upload(st)
        assert sim.run_timed(1)[1]["total_launches"] == launches
        sc = [sim.step() for _ in range(5)]
        sim.download(st)
    return st, sc


@pytest.mark.gpu
@pytest.mark.parametrize("bc", BC)
@pytest.mark.parametrize("shape", [(256, 128, 64), (61, 37, 300)], ids=["even", "ragged"])
def test_single_wave_equals_several_waves(shape, bc, monkeypatch):
    p = params(shape, BC[bc])
    monkeypatch.setenv("R3D_KCHUNK", "16")
    one, a = domain(p, 4)
    monkeypatch.setenv("R3D_KCHUNK", "1")
    many, b = domain(p, 9)
    assert a == b
    for n in one.fields:
        assert np.array_equal(one.fields[n], many.fields[n]), n


@pytest.mark.gpu
def test_single_wave_slabs_equal_a_domain_of_several_waves(monkeypatch):
    p = params((256, 256, 64), BC["plume_flux"])
    one, sc = domain(p, 9)
    monkeypatch.setenv("R3D_KCHUNK", "16")  # 128 CTAs a slab
    st = R.HostState.setup(p)
    with R.GpuMesh(p, 4) as m:
        m.upload(st)
        for _ in range(6):
            last = m.step()
        m.download(st)
    assert last == sc[-1]
    for n in st.fields:
        assert np.array_equal(st.fields[n][1:-1, 1:-1, 1:-1], one.fields[n][1:-1, 1:-1, 1:-1]), n
