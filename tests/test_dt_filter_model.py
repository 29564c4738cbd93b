"""Host model of the check behind the third stage's filtered dt fold (step_begin, step_end), on oracle states:
whenever it passes, the limits folded over the cells that are not skipped equal those of every interior cell
(src/step.cpp:125-196), and a negative margin never passes it.

The thresholds are the previous step's CFL, conduction and viscosity limits, widened by the margin, and its
Mach term, narrowed; the check accepts the folded minima <= their thresholds and the maximum >= its own, and
otherwise every cell is evaluated.  The skip rule is test_dt_bounds_model's.
"""
import numpy as np
import pytest

import r3d_b200 as R
from oracle import Oracle
from test_dt_bounds_model import MARGIN, limits, skip, state


def folded(w, keep):
    if not keep.any():
        return [1e300] * 3 + [0.0]
    return [np.nanmin(v[keep]) for v in w[:3]] + [np.nanmax(w[3][keep])]


def accepted(got, t, tu):
    return all(g <= v for g, v in zip(got, t)) and got[3] >= tu


@pytest.mark.parametrize("flags,seed", [
    (["--npx", "32", "--npy", "32", "--npz", "64"], 1),
    (["--npx", "24", "--npy", "20", "--npz", "48", "--ngrid", "2", "--izcon", "1", "--itcon", "0"], 5),
])
def test_filter_exact_on_trajectory(flags, seed):
    p = R.parse(flags)
    c = {n: R.derived(p, n) for n in ("obeta", "repr", "cv")}
    o = Oracle(flags).init(seed)
    prev, passed, skipped = None, 0, 0
    with np.errstate(all="ignore"):
        for _ in range(8):
            x, dd, rk = state(o, p)
            w = limits(x, dd, rk, p, c)
            exact = folded(w, np.ones(dd.shape, bool))
            if prev is not None and prev[3] > 0:
                for margin in (MARGIN, -0.5):
                    t, tu = [v * (1 + margin) for v in prev[:3]], prev[3] * (1 - margin)
                    sk = skip(x, dd, rk, p, c, t, tu)
                    got = folded(w, ~sk)
                    if margin > 0 and accepted(got, t, tu):
                        assert got == exact
                        passed += 1
                        skipped += int(sk.sum())
                    elif margin < 0:
                        assert not accepted(got, t, tu)
            prev = exact
            o.step(3)
    assert passed >= 4 and skipped > 0, (passed, skipped)
