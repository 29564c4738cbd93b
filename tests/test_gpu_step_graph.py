"""r3d_gpu_step replays one step and its read-back as a graph; the graphs of a handle follow its uploads."""
import numpy as np
import pytest

import r3d_b200 as R

# whole steps by r3d_gpu_step (the first four are eager), by r3d_gpu_run, and partial steps of one or two stages
OPS = {
    "step": [("step", 20)],
    "mixed": [("step", 18), ("run", 3), ("partial", 2), ("step", 3), ("partial", 1), ("step", 3), ("run", 4)],
    "run": [("run", 5)],
    "few": [("step", 2)],
}


def same(a, b):
    return all(np.array_equal(a.fields[n], b.fields[n]) for n in a.fields)


def session(sim, start, ops, eager=False):
    sim.upload(start)
    for kind, n in ops:
        if kind == "partial":
            sc = sim.step(n)
        elif eager:  # a timed step is never a graph
            sc = [sim.run_timed(1)[0] for _ in range(n)][-1]
        elif kind == "step":
            sc = [sim.step() for _ in range(n)][-1]
        else:
            sc = sim.run(n)
    got = start.copy()
    sim.download(got)
    return got, sc


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
    starts = {"st": st, "other": other}
    ref = {}
    for how in OPS:
        for name, start in starts.items():
            with R.GpuSim(p) as sim:
                ref[how, name] = session(sim, start, OPS[how], eager=True)
        assert not same(ref[how, "st"][0], ref[how, "other"][0])
    with R.GpuSim(p) as sim:  # one handle through all of them
        for how in ("step", "mixed", "run", "few", "step"):
            for name in ("st", "other", "other"):
                got, sc = session(sim, starts[name], OPS[how])
                assert same(got, ref[how, name][0]) and sc == ref[how, name][1], (how, name)
