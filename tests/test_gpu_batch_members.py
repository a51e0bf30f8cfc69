"""hmfem_batch_solve with members that differ: one that runs out of iterations,
one that breaks down, initial guesses, members not yet set up, members on one
stream, more members than the host can keep busy -- each gives what it gives
solved alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402

SHAPES = [(20, 18, 16), (12, 9, 15), (24, 10, 9), (33, 31, 17), (7, 11, 5)]
FAST = dict(precision=1, bf16_from=1, schur0=1)


def _problem(i):
    return make_problem(*SHAPES[i % len(SHAPES)], log10k=(-14.0, 1.0, 2.0), seed=90 + i)


def _solver(i, setup=True, **opt):
    s = gpu.Solver(tol=1e-10, **opt)
    s.assemble(_problem(i))
    if setup:
        s.setup()
    return s


def _alone(i, x0=None, **opt):
    s = _solver(i, **opt)
    x, st = s.solve(x=None if x0 is None else x0.copy(), allow_notconv=True)
    s.close()
    return x, st["iterations"]


def _check(members, xs, sts, starts, opts):
    for i, (x, st) in enumerate(zip(xs, sts)):
        want, its = _alone(i, starts[i], **opts[i])
        assert st["iterations"] == its, i
        assert np.array_equal(x, want), i
    for s in members:
        s.close()


@pytest.mark.parametrize("opt", [dict(), FAST], ids=["fp64", "fast"])
@pytest.mark.parametrize("case", ["plain", "not_set_up", "guess", "one_stream", "out_of_iterations"])
def test_members_give_what_they_give_alone(case, opt, monkeypatch):
    m = len(SHAPES)
    opts = [dict(opt) for _ in range(m)]
    if case == "out_of_iterations":
        opts[1]["max_iter"] = 4
        opts[3]["max_iter"] = 5
    starts = [None] * m
    if case == "guess":
        starts = [np.cos(np.arange(_problem(i).n)) if i % 2 else np.zeros(_problem(i).n)
                  for i in range(m)]
    members = [_solver(i, setup=case != "not_set_up" or i % 2 == 0, **opts[i]) for i in range(m)]
    stream = torch.cuda.Stream()
    if case == "one_stream":
        for s in members[1:4]:
            s.set_stream(stream.cuda_stream)
    xs = [np.zeros(_problem(i).n) if starts[i] is None else starts[i].copy() for i in range(m)]
    sts = gpu.batch_solve(members, xs, allow_notconv=case == "out_of_iterations")
    for i in range(m):
        ok = case != "out_of_iterations" or i not in (1, 3)
        assert sts[i]["status"] == (gpu.OK if ok else gpu.E_NOTCONV), i
    _check(members, xs, sts, starts, opts)


def test_a_member_that_breaks_down_leaves_the_others_alone():
    m = len(SHAPES)
    members = [_solver(i) for i in range(m)]
    xs = [np.zeros(_problem(i).n) for i in range(m)]
    xs[2][7] = np.nan
    with pytest.raises(gpu.HmfemError) as e:
        gpu.batch_solve(members, xs)
    assert e.value.code == gpu.E_BREAKDOWN
    for i in range(m):
        if i != 2:
            assert np.array_equal(xs[i], _alone(i)[0]), i
    # and all of them solve again, the failed one too
    xs = [np.zeros(_problem(i).n) for i in range(m)]
    sts = gpu.batch_solve(members, xs)
    _check(members, xs, sts, [None] * m, [dict()] * m)


def test_more_members_than_one_thread_keeps_busy():
    m = 60
    members = [_solver(i, **FAST) for i in range(m)]
    xs = [np.zeros(_problem(i).n) for i in range(m)]
    sts = gpu.batch_solve(members, xs)
    _check(members, xs, sts, [None] * m, [FAST] * m)
