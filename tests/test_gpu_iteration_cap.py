"""The iteration cap at the ends of its range: one iteration, and the largest
integer (no cap), for a solve on its own and for a batch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402


@pytest.mark.parametrize("check_every", [1, 2, 16])
@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("max_iter", [1, 2147483646, 2147483647])
def test_cap(max_iter, batch, check_every):
    p = make_problem(20, 18, 16, log10k=(-14.0, 1.0, 2.0), seed=4)

    def solver(**opt):
        s = gpu.Solver(tol=1e-10, **opt)
        s.assemble(p)
        s.setup()
        return s

    want, ref = solver().solve()
    s = solver(max_iter=max_iter, check_every=check_every)
    x = np.zeros(p.n)
    if batch:
        (st,) = gpu.batch_solve([s], [x], allow_notconv=True)
    else:
        x, st = s.solve(x=x, allow_notconv=True)
    if max_iter == 1:
        assert st["status"] == gpu.E_NOTCONV and st["iterations"] == 1
    else:
        assert st["status"] == gpu.OK and st["iterations"] == ref["iterations"]
        assert np.array_equal(x, want)
    s.close()
