"""hmfem_time_kernel 12 (a V-cycle from level l on) runs the kernels a solve
runs: from the first level of the one-launch form on, that launch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402


@pytest.mark.parametrize("opt", [dict(), dict(precision=1, bf16_from=1, schur0=1)],
                         ids=["fp64", "fast"])
def test_a_cycle_from_a_small_level_is_the_cluster_launch(opt, monkeypatch):
    def launches(on):
        monkeypatch.setenv("HMFEM_SMALL_CYCLE", on)
        s = gpu.Solver(tol=1e-9, **opt)
        s.assemble(make_problem(32, 32, 32, log10k=(-14.0, 1.0, 2.0), seed=1))
        s.setup()
        out = []
        for l in range(s.num_levels()):
            a = gpu.launch_count()
            s.time_kernel(12, l, reps=1)
            b = gpu.launch_count()
            s.time_kernel(12, l, reps=3)
            out.append((gpu.launch_count() - b - (b - a)) // 2)   # one repetition's
        s.close()
        return out

    one, many = launches("1"), launches("0")
    # the first level whose cycle is one launch (and its right-hand side's seed)
    first = next(l for l, (o, m) in enumerate(zip(one, many)) if o != m and o == 2)
    # every level above it saves the same launches, those below are as they were
    assert {m - o for m, o in zip(many[:first], one[:first])} == {many[first] - 2}
    assert one[first + 1:] == many[first + 1:]
