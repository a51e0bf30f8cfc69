"""A solve whose iteration graph cannot be instantiated fails with a status,
and the next solve captures it again.  The failure comes from a stand-in for
the runtime's call, preloaded into a process of its own."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
typedef int (*fn_t)(void **, void *, unsigned long long);
int cudaGraphInstantiate(void **exec, void *graph, unsigned long long flags)
{
    static int calls = 0;
    const char *e = getenv("FAIL_AT");
    if (e && ++calls == atoi(e)) return 2;  /* cudaErrorMemoryAllocation */
    return ((fn_t)dlsym(RTLD_NEXT, "cudaGraphInstantiate"))(exec, graph, flags);
}
"""

CHILD = r"""
import numpy as np
from hmfem_b200 import gpu
from hmfem_b200.problem import make_problem
p = make_problem(20, 18, 16, log10k=(-14.0, 1.0, 2.0), seed=1)
q = make_problem(9, 8, 7, log10k=(-14.0, 1.0, 2.0), seed=2)
s = gpu.Solver(tol=1e-10)
if %(before)d:                      # an executable graph of other levels first
    s.assemble(q); s.setup(); s.solve()
s.assemble(p)
s.setup()
try:
    s.solve()
    raise SystemExit("the stand-in did not fail")
except gpu.HmfemError as e:
    assert e.code == gpu.E_CUDA, e
x, st = s.solve()
assert st["status"] == gpu.OK
r = gpu.Solver(tol=1e-10)
r.assemble(p)
r.setup()
y, _ = r.solve()
assert np.array_equal(x, y)
print("retried")
"""


@pytest.mark.parametrize("before", [0, 1])
def test_a_failed_instantiation_is_tried_again(before, tmp_path):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", str(so), str(src), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so), FAIL_AT=str(1 + before), PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", CHILD % dict(before=before)], env=env, cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "retried" in out.stdout, out.stdout + out.stderr
