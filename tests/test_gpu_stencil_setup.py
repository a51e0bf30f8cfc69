"""hmfem_set_stencil on a grid's own rows takes the structured setup (FP64
cycle); rows that are not a grid's and the reduced-precision cycle take the
general one.  Both against generic_setup=1: the same
hierarchy and the same V-cycle, bit for bit (the CG's dot products are grouped
by kernel, so its iterates are not compared)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402

# field positions in perm (u, d, l, r, c, t, b) and indcol (c, u, d, l, r, t, b)
E = {f: i for i, f in enumerate("udlrctb")}
I = {f: i for i, f in enumerate("cudlrtb")}


def _rows(port, p):
    perm, ind, b = port.assemble(p)
    return (np.array(perm, dtype=np.float64).reshape(-1, 7),
            np.array(ind, dtype=np.int32).reshape(-1, 7), np.array(b))


def _change(kind, perm, ind, p):
    """One pair of rows that the grid's pattern does not have."""
    q = p.n // 2 // p.nx * p.nx + p.nx // 2  # inside its x row
    if kind == "cut":           # a coupling left out on both sides
        ind[q, I["r"]] = ind[q + 1, I["l"]] = -1
    elif kind == "cut_last":    # the last row keeps its diagonal only
        s = p.n - 1
        for f, g, o in (("l", "r", 1), ("d", "u", p.nx), ("b", "t", p.nx * p.ny)):
            if ind[s, I[f]] >= 0:
                ind[s, I[f]] = -1
                ind[s - o, I[g]] = -1
    elif kind == "order":       # the same matrix with two entries exchanged
        for t, at in ((perm, E), (ind, I)):
            t[q, at["l"]], t[q, at["r"]] = t[q, at["r"]], t[q, at["l"]]
    elif kind == "unsymmetric":  # one side a bit larger
        perm[q, E["r"]] = np.nextafter(perm[q, E["r"]], np.inf)


@pytest.mark.parametrize("opt", [dict(), dict(precision=1), dict(precision=1, bf16_from=1),
                                 dict(precision=1, schur0=1)], ids=str)
@pytest.mark.parametrize("kind", ["grid", "cut", "cut_last", "order", "unsymmetric"])
@pytest.mark.parametrize("shape", [(16, 12, 10), (17, 9, 7), (40, 33, 20), (8, 8, 1), (1, 1, 40)])
def test_same_bits_as_the_general_setup(shape, kind, opt, port):
    p = make_problem(*shape, log10k=(-14.0, 1.0, 2.0), seed=sum(shape))
    perm, ind, b = _rows(port, p)
    if kind != "grid" and shape[0] > 1:
        _change(kind, perm, ind, p)
    got = []
    for generic in (0, 1):
        s = gpu.Solver(tol=1e-8, generic_setup=generic, **opt)
        s.set_stencil(*shape, perm, ind, b)
        s.setup()
        u = s.vcycle(np.sin(np.arange(p.n)))
        levels = [s.level(k) for k in range(s.num_levels())]
        forms = {k["kernel"] for k in s.profile_iteration(1)}
        got.append((u, levels, any("g7" in f for f in forms)))
        s.close()
    (u, la, structured), (v, lb, _) = got
    assert structured == (not opt and (kind == "grid" or shape[0] == 1))
    assert np.array_equal(u, v)
    assert len(la) == len(lb)
    for a, c in zip(la, lb):
        for key in ("cnt", "col", "ele", "sel", "pcnt", "pcol"):
            assert np.array_equal(a[key], c[key])
