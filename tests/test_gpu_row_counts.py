"""Row counts that do not describe a matrix are refused as bad arguments, also
when their sum is negative or another matrix was set before: the solver then
holds no matrix to solve."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402


def _line(n):
    i = np.arange(n)
    col = np.stack([i - 1, i, i + 1], 1)
    keep = (col >= 0) & (col < n)
    ele = np.tile([-1.0, 2.5, -1.0], (n, 1))
    return keep.sum(1).astype(np.int32), col[keep].astype(np.int32), ele[keep]


@pytest.mark.parametrize("earlier", [False, True], ids=["first", "after_another"])
@pytest.mark.parametrize("what", ["all_negative", "one_very_negative", "one_negative", "too_few"])
def test_counts_that_are_no_matrix(what, earlier):
    n = 300
    cnt, col, ele = _line(n)
    s = gpu.Solver(reuse_setup=1, tol=1e-10)
    if earlier:
        s.set_matrix(cnt, col, ele, np.ones(n))
        s.setup()
        s.solve()
    bad = cnt.copy()
    if what == "all_negative":
        bad[:] = -1
    elif what == "one_very_negative":
        bad[7] = -2000000000
    elif what == "one_negative":
        bad[7], bad[8] = -1, 7
    else:
        bad[7] -= 1
    with pytest.raises(gpu.HmfemError) as e:
        s.set_matrix(bad, col, ele, np.ones(n))
    assert e.value.code == gpu.E_ARG
    assert ("add up" if what == "too_few" else "negative row count") in str(e.value)
    for call in (s.setup, s.solve):     # the refused matrix, and not the one before
        with pytest.raises(gpu.HmfemError) as e:
            call()
        assert e.value.code == gpu.E_ARG
    s.set_matrix(cnt, col, ele, np.ones(n))
    s.setup()
    x, st = s.solve()
    assert st["status"] == gpu.OK and st["relres"] <= 1e-10
    s.close()
