"""fm_problem_get_state in a process that cannot have any more threads: the work
it shares out to host threads is done on the calling one.  A default thread
stack of 128 TB makes every new thread fail; the call runs in a child process,
after CUDA's own threads have started."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, sys, threading
import numpy as np
from femorph_b200 import api, mesh

def no_more_threads():
    libc = ctypes.CDLL(None)
    attr = (ctypes.c_char * 256)()
    assert libc.pthread_attr_init(attr) == 0
    assert libc.pthread_attr_setstacksize(attr, ctypes.c_size_t(1 << 47)) == 0
    assert libc.pthread_setattr_default_np(attr) == 0
    try:
        threading.Thread(target=print).start()
    except RuntimeError:
        return
    sys.exit(3)

p = mesh.cavity(56, seed=1, noise=1e-2)   # 4.4 MB of velocities, 101 MB of subscales
g = api.GpuProblem(p)
b = api.Batch([g])
b.step(2)
b.sync()
u = g.state(elements=False)[0]
no_more_threads()
state = g.state()
assert np.array_equal(state[0], u) and np.isfinite(state[3]).all()
print("done")
"""


def test_read_back_without_threads():
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=300)
    if r.returncode == 3:
        pytest.skip("threads start whatever their stack")
    assert r.returncode == 0 and "done" in r.stdout, r.stderr[-2000:]
