"""The coarse end of the V-cycle in one cluster launch (small_cycle.cu)
against the level kernels, which HMFEM_SMALL_CYCLE=0 selects: the same bits,
over row counts around a CTA's share, both precisions and every value form,
several Chebyshev degrees, and standing alone (hmfem_vcycle)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402

FORMS = {"fp64": dict(), "fp32": dict(precision=1), "bf16": dict(precision=1, bf16_from=1),
         "schur": dict(precision=1, bf16_from=1, schur0=1)}


def _run(p, monkeypatch, on, team="1", **opt):
    monkeypatch.setenv("HMFEM_SMALL_CYCLE", on)
    monkeypatch.setenv("HMFEM_TEAM", team)
    s = gpu.Solver(tol=1e-9, **opt)
    s.assemble(p)
    s.setup()
    x, st = s.solve()
    u = s.vcycle(np.sin(np.arange(p.n)))
    names = {k["kernel"] for k in s.profile_iteration(1)}
    s.close()
    return x, u, st["iterations"], any("small_cycle" in k for k in names)


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("shape", [(14, 12, 10), (33, 31, 17), (40, 40, 40), (64, 33, 50),
                                   (210, 42, 20)])
def test_one_launch_gives_the_level_kernels_bits(shape, form, monkeypatch):
    p = make_problem(*shape, log10k=(-14.0, 1.0, 2.0), seed=shape[0])
    a = _run(p, monkeypatch, "1", **FORMS[form])
    b = _run(p, monkeypatch, "0", **FORMS[form])
    assert not b[3]
    if shape[0] > 20:
        assert a[3]
    assert a[2] == b[2]
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1], b[1])


@pytest.mark.parametrize("degree,cheb_from,direct", [(2, 2, 512), (3, 2, 100), (5, 1, 512),
                                                     (9, 2, 40)])
def test_degrees_and_level_ranges(degree, cheb_from, direct, monkeypatch):
    p = make_problem(30, 29, 28, log10k=(-14.0, 1.0, 2.0), seed=degree)
    opt = dict(cheb_degree=degree, cheb_from=cheb_from, coarse_direct=direct)
    for prec in (dict(), dict(precision=1)):
        a = _run(p, monkeypatch, "1", **opt, **prec)
        b = _run(p, monkeypatch, "0", **opt, **prec)
        assert a[3] and not b[3]
        assert a[2] == b[2] and np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("shape", [(17, 9, 7), (48, 48, 48), (91, 61, 63), (120, 96, 80)])
def test_teams_give_the_row_kernels_bits(shape, form, monkeypatch):
    """Warps sharing a slice's loads (levels of up to ~38000 rows) against a
    row per thread, with the one-launch form off so that every level has its
    kernels."""
    p = make_problem(*shape, log10k=(-14.0, 1.0, 2.0), seed=shape[1])
    a = _run(p, monkeypatch, "0", team="1", **FORMS[form])
    b = _run(p, monkeypatch, "0", team="0", **FORMS[form])
    assert a[2] == b[2]
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_threads_with_different_grids():
    """Solvers whose cluster launches take different amounts of shared
    memory, captured and launched from eight threads at once."""
    from hmfem_b200 import batch

    shapes = [(14, 12, 10), (24, 20, 16), (33, 31, 17), (40, 36, 30)]
    probs = [make_problem(*shapes[i % 4], log10k=(-14.0, 1.0, 2.0), seed=i) for i in range(64)]
    out = batch.solve_batch(probs, precision=1, tol=1e-9, workers=8)
    for i in (0, 1, 2, 3):
        s = gpu.Solver(precision=1, tol=1e-9)
        s.assemble(probs[i])
        s.setup()
        x, st = s.solve()
        s.close()
        assert st["iterations"] == out[i][1]["iterations"]
        assert np.array_equal(x, out[i][0])
