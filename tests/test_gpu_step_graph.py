"""r3d_gpu_step replays one step and its read-back as a graph; the graphs of a handle follow its uploads."""
import numpy as np
import pytest

import r3d_b200 as R


def same(a, b):
    return all(np.array_equal(a.fields[n], b.fields[n]) for n in a.fields)


@pytest.mark.gpu
@pytest.mark.parametrize("flags", [
    ["--npx", "24", "--npy", "20", "--npz", "36"],                               # single-wave stages
    ["--npx", "24", "--npy", "20", "--npz", "36", "--precision", "fp32bulk"],
    ["--npx", "130", "--npy", "70", "--npz", "120"],                             # several waves
], ids=["tail", "fp32", "plain"])
def test_steps_graphs_and_reuploads(flags):
    p = R.parse(flags + ["--seed", "4"])
    st = R.HostState.setup(p)
    other = st.copy()  # another bottom temperature and another conductivity profile
    other.scalars["tb"] = st.scalars["tb"] * 1.01
    other.lines["rkapa"] = 1.0 + 0.1 * np.linspace(0.0, 1.0, p.npz + 2)

    def run(sim, start, how):
        sim.upload(start)
        if how == "step":
            sc = [sim.step() for _ in range(5)][-1]
        elif how == "mixed":  # graphs of both parities, a partial step between whole ones
            sim.step()
            sim.run(3)
            sc = sim.step()
        else:
            sc = sim.run(5)
        got = st.copy()
        sim.download(got)
        return got, sc

    ref = {}
    for name, start in (("st", st), ("other", other)):
        with R.GpuSim(p) as sim:
            ref[name] = run(sim, start, "run")
    assert not same(ref["st"][0], ref["other"][0])
    with R.GpuSim(p) as sim:  # one handle through all of them
        for how in ("step", "mixed", "run", "step"):
            for name, start in (("st", st), ("other", other)):
                got, sc = run(sim, start, how)
                assert same(got, ref[name][0]) and sc == ref[name][1], (how, name)
