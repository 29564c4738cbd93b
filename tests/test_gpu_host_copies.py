"""Transfers of pageable arrays on a host short of memory."""
import os
import subprocess
import sys

import pytest

NO_MEMORY = """
import resource
import numpy as np
import r3d_b200 as R

p = R.parse(["--npx", "64", "--npy", "64", "--npz", "120", "--seed", "5"])  # 4.3 MB per field
st = R.HostState.setup(p)
a, b = st.copy(), st.copy()
with R.GpuSim(p) as sim:
    sim.setup()  # on the device: no host array has been copied yet
    sim.run(2)
    pages = int(open("/proc/self/statm").read().split()[0])
    old = resource.getrlimit(resource.RLIMIT_AS)
    resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + (1 << 20), old[1]))
    sim.download(a)
    sim.upload(a)
    resource.setrlimit(resource.RLIMIT_AS, old)
    sim.download(b)
assert a.scalars["nit"] == 2
for n in a.fields:
    assert np.abs(a.fields[n]).max() > 0 and np.array_equal(a.fields[n], b.fields[n]), n
print("COPIED")
"""


def child(code, **env):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    path = os.path.join(root, "rast-3dmhd_b200", "python")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, PYTHONPATH=path, **env), text=True,
                       capture_output=True, timeout=300)
    return r.returncode, r.stdout + r.stderr


@pytest.mark.gpu
def test_copies_without_page_locked_buffers():
    """No address space is left for the buffers: the copies go through the driver's staging instead."""
    rc, out = child(NO_MEMORY)
    assert rc == 0 and "COPIED" in out, out


FORKED = """
import os, signal
import numpy as np
import r3d_b200 as R

p = R.parse(["--npx", "64", "--npy", "64", "--npz", "120", "--seed", "5"])
st = R.HostState.setup(p)  # OpenMP loops; CUDA not yet in use
pid = os.fork()
if pid == 0:
    signal.alarm(120)
    got = st.copy()
    with R.GpuSim(p) as sim:
        sim.upload(st)
        sim.download(got)
    os._exit(0 if all(np.array_equal(got.fields[n], st.fields[n]) for n in st.fields) else 1)
assert os.waitpid(pid, 0)[1] == 0
print("COPIED")
"""


@pytest.mark.gpu
def test_copies_in_a_worker_forked_after_the_set_up():
    rc, out = child(FORKED)
    assert rc == 0 and "COPIED" in out, out


CHILDREN = """
import os, time
import numpy as np
import r3d_b200 as R

p = R.parse(["--npx", "64", "--npy", "64", "--npz", "300", "--seed", "5"])  # 10.5 MB per field: both buffers
st = R.HostState.setup(p)
got = st.copy()
with R.GpuSim(p) as sim:
    for turn in range(3):
        for n in st.fields:
            st.fields[n] += 1.0
        sim.upload(st)
        pid = os.fork()  # alive through the next copies, which rewrite the buffers
        if pid == 0:
            time.sleep(0.5)
            os._exit(0)
        sim.download(got)
        assert all(np.array_equal(got.fields[n], st.fields[n]) for n in st.fields), turn
        os.waitpid(pid, 0)
print("COPIED")
"""


@pytest.mark.gpu
def test_copies_beside_a_forked_child():
    rc, out = child(CHILDREN)
    assert rc == 0 and "COPIED" in out, out
