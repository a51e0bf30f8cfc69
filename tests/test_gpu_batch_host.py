"""A batch whose driving thread is kept off its core while the members iterate:
they go on when it is back.  Stand-ins for two calls, preloaded into a process
of its own, make the thread sleep where it would look for a stopped member."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# the 16th yield (of 256 looks each) without a launch in between comes right
# before the driver asks whether a member's stream has stopped
SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <time.h>
static __thread int yields, naps;
int cudaGraphLaunch(void *exec, void *stream)
{
    yields = 0;
    return ((int (*)(void *, void *))dlsym(RTLD_NEXT, "cudaGraphLaunch"))(exec, stream);
}
int sched_yield(void)
{
    if (++yields == 16 && naps < 20) {
        struct timespec t = {0, 20000000};
        naps++;
        nanosleep(&t, 0);
    }
    return 0;
}
int test_naps(void) { return naps; }
"""

CHILD = r"""
import ctypes
import os
import numpy as np
from hmfem_b200 import gpu
from hmfem_b200.problem import make_problem
shapes = [(128, 128, 128), (96, 80, 64)][:%(members)d]
probs = [make_problem(*s, log10k=(-14.0, 1.0, 2.0), seed=3 + i) for i, s in enumerate(shapes)]
def solver(p):
    s = gpu.Solver(tol=1e-10)
    s.assemble(p)
    s.setup()
    return s
xs = [np.zeros(p.n) for p in probs]
sts = gpu.batch_solve([solver(p) for p in probs], xs)
naps = ctypes.CDLL(os.environ["LD_PRELOAD"]).test_naps()
assert naps > 0, "the stand-in never slept"
for p, x, st in zip(probs, xs, sts):
    y, want = solver(p).solve()
    assert st["status"] == gpu.OK and st["iterations"] == want["iterations"]
    assert np.array_equal(x, y)
print("solved after", naps, "naps")
"""


@pytest.mark.parametrize("members", [1, 2])
def test_members_go_on_after_the_host_was_away(members, tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", CHILD % dict(members=members)], env=env, cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "solved after" in out.stdout, out.stdout + out.stderr
