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
