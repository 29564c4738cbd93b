"""The reverse sweep where its time step or its recompute is degenerate."""
import numpy as np
import pytest

import r3d_b200 as R
from oracle import Oracle
from tangent_np import NumpyStep

MAG = ["--lmag", "1", "--beta", "10", "--rm", "1", "--ampb", "0.1", "--bfh", "2", "--bzp", "20"]
I3 = (slice(1, -1),) * 3


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [[], MAG], ids=["hydro", "mhd"])
def test_zero_safety_factor(extra):
    """--sff 0: dt is 0 whatever the state, a step is BCON alone and the sweep its transpose."""
    flags = ["--npx", "33", "--npy", "9", "--npz", "7", "--zmax", "2", "--sff", "0", *extra]
    p = R.parse(flags + ["--seed", "3"])
    names = R.FIELDS3D if p.lmag else R.FIELDS3D[:5]
    st = R.HostState.setup(p)
    rng = np.random.default_rng(11)
    ns = NumpyStep(Oracle(flags).init(3))
    with R.GpuSim(p) as sim:
        sim.upload(st)
        V, lam = {}, {}
        for n in names:
            V[n] = np.zeros_like(st.fields[n])
            V[n][I3] = rng.standard_normal(V[n][I3].shape)
            ns.ghost_fill(V[n])
            lam[n] = np.zeros_like(V[n])
            lam[n][I3] = rng.standard_normal(V[n][I3].shape)
        assert sim.adjoint_record(3, 2)["dt"] == 0.0
        many = sim.adjoint_backward(lam)
        sim.upload(st)
        one = sim.adjoint_step(lam)
    h = 1e-30  # complex step: the exact tangent
    for grad, steps in ((one, 1), (many, 3)):
        Y, _ = ns.run({n: st.fields[n] + 1j * h * V[n] for n in names}, steps)
        left = [lam[n][I3] * Y[n][I3].imag / h for n in names]
        right = [grad[n][I3] * V[n][I3] for n in names]
        lhs, rhs = (sum(float(t.sum()) for t in s) for s in (left, right))
        # a value of either side passes BCON or its transpose three times a step, some ten products
        # each, every one rounded: 30 eps of the summed sizes a step
        size = sum(float(np.abs(t).sum()) for t in left + right)
        assert abs(lhs - rhs) <= 30 * steps * 2.0 ** -53 * size, (lhs, rhs)


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [["--npx", "32", "--npy", "32", "--npz", "64"],
                                   ["--npx", "24", "--npy", "20", "--npz", "40", *MAG]], ids=["hydro", "mhd"])
def test_abandoned_recompute_leaves_nothing_behind(extra):
    """The recompute's bounded waits run out (single-wave stages, BCON planes in several chunks for hydro): the
    sweep reports it, and the forward steps, the sweeps and the trajectory after it are as without it."""
    p = R.parse(extra + ["--seed", "3"])
    st = R.HostState.setup(p)
    rng = np.random.default_rng(2)
    lam = {n: rng.standard_normal(a.shape) for n, a in st.fields.items()}

    def session(fail):
        out = []
        with R.GpuSim(p) as sim:
            sim.upload(st)
            sim.adjoint_record(4, 3)
            for call in (sim.adjoint_backward, sim.adjoint_step) if fail else ():
                sim.debug_tma_extra(16)
                with pytest.raises(R.R3dError) as e:
                    call(lam)
                assert e.value.code == R.R3D_ECUDA and "bounded TMA wait" in str(e.value)
                sim.debug_tma_extra(0)
            dts = [sim.step()["dt"] for _ in range(3)]
            got = st.copy()
            sim.download(got)
            out = [got.fields, sim.adjoint_step(lam), sim.adjoint_backward(lam)]
        return dts, out

    ref, got = session(False), session(True)
    assert got[0] == ref[0]
    for a, b in zip(got[1], ref[1]):
        for n in a:
            assert np.array_equal(a[n], b[n]), n


@pytest.mark.gpu
def test_diverged_recompute_is_reported_once():
    """A recompute that differs from the recorded trajectory (here: another conductivity profile uploaded in
    between) is an error of that sweep, not of the next."""
    p = R.parse(["--npx", "24", "--npy", "20", "--npz", "36", "--seed", "3"])
    st = R.HostState.setup(p)
    other = st.copy()
    other.lines["rkapa"] = 1.0 + 0.1 * np.linspace(0.0, 1.0, p.npz + 2)
    lam = {n: np.ones_like(a) for n, a in st.fields.items()}
    with R.GpuSim(p) as sim:
        sim.upload(other)
        ref = sim.adjoint_step(lam)
    with R.GpuSim(p) as sim:
        sim.upload(st)
        sim.adjoint_record(2, 1)
        sim.upload(other)
        with pytest.raises(R.R3dError) as e:
            sim.adjoint_backward(lam)
        assert e.value.code == R.R3D_ENUMERIC
        got = sim.adjoint_step(lam)
    for n in ref:
        assert np.array_equal(got[n], ref[n]), n


@pytest.mark.gpu
def test_memory_counts_the_recorded_limits():
    p = R.parse(["--npx", "16", "--npy", "12", "--npz", "16", "--seed", "3"])
    got = []
    for steps in (4, 40):
        with R.GpuSim(p) as sim:
            sim.setup()
            sim.adjoint_record(steps, steps)  # two checkpoints
            got.append(sim.adjoint_memory_bytes)
    assert got[1] - got[0] == 36 * 32
