"""The small end of the hierarchy (one launch for every level of at most 512
rows, amg_tail.cu) and the coarse inverse, against the oracle's hierarchy and
V-cycle, around the sizes where the forms change."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402
from oracle.oracle import Port  # noqa: E402


def _matrix(nx, ny, nz, seed):
    p = make_problem(nx, ny, nz, log10k=(-14.0, 1.5, 2.0), seed=seed)
    port = Port()
    perm, ind, b = port.assemble(p)
    return port, port.pack(perm, ind), b


# level 1 of an n-row 7-point matrix has about n / 2 rows: 512 and 513 among
# them; one row, a line, a slab
@pytest.mark.parametrize("shape", [(2, 1, 1), (3, 3, 3), (64, 1, 1), (16, 8, 8), (19, 9, 6),
                                   (27, 19, 2), (41, 25, 1), (32, 32, 1)])
@pytest.mark.parametrize("max_levels,min_coarse", [(16, 1), (3, 1), (16, 20)])
def test_small_levels_match_the_oracle(shape, max_levels, min_coarse):
    port, (cnt, col, ele), b = _matrix(*shape, seed=sum(shape))
    H = port.amg(cnt, col, ele)
    s = gpu.Solver(max_levels=max_levels, min_coarse=min_coarse)
    s.set_matrix(cnt, col, ele, b)
    s.setup()
    n = s.num_levels()
    want = 1
    while want < H.nlevels and want < max_levels and H.level(want - 1)["n"] > min_coarse:
        want += 1
    assert n == want
    for l in range(n):
        g, o = s.level(l), H.level(l)
        for k in ("cnt", "col", "ele", "dinv"):
            assert np.array_equal(g[k], o[k]), (l, k)
        if l < n - 1:
            for k in ("sel", "pcnt", "pcol"):
                assert np.array_equal(g[k], o[k]), (l, k)
    s.close()


@pytest.mark.parametrize("n", [1, 15, 16, 17, 128, 129, 255, 256, 257, 384, 385, 511, 512])
def test_coarse_inverse_solves(n):
    """A level of n rows solved directly: the V-cycle is the inverse."""
    rng = np.random.default_rng(n)
    k = 0.5 + rng.random(n + 1)
    cnt, col, ele = [], [], []
    for i in range(n):
        row = [(j, v) for j, v in ((i - 1, -k[i]), (i, k[i] + k[i + 1]), (i + 1, -k[i + 1]))
               if 0 <= j < n]
        cnt.append(len(row))
        col += [j for j, _ in row]
        ele += [v for _, v in row]
    s = gpu.Solver()
    s.set_matrix(np.array(cnt, np.int32), np.array(col, np.int32), np.array(ele))
    s.setup()
    f = rng.standard_normal(n)
    u = s.vcycle(f)
    A = np.zeros((n, n))
    q = 0
    for i, c in enumerate(cnt):
        A[i, col[q:q + c]] = ele[q:q + c]
        q += c
    # Gauss-Jordan on a matrix of condition ~n^2: n^2 ulps, and a margin
    ref = np.linalg.solve(A, f)
    assert np.abs(u - ref).max() <= 1e-13 * (n * n + 10) * np.abs(ref).max()
    s.close()


@pytest.mark.parametrize("n,band", [(1023, 3), (1024, 40), (1025, 90), (2500, 70), (3000, 200)])
def test_greedy_split_of_banded_matrices(n, band):
    """The general split around its 1024-row tiles, with rows shorter and
    longer than the 64 entries its masks cover: every level the oracle's."""
    rng = np.random.default_rng(n + band)
    up = [np.unique(i + 1 + rng.integers(0, 2 * band, band)) for i in range(n)]
    rows = [dict() for _ in range(n)]
    for i, js in enumerate(up):
        for j in js[js < n]:
            rows[i][int(j)] = rows[int(j)][i] = -float(rng.random() + 0.1)
    cnt, col, ele = np.zeros(n, np.int32), [], []
    for i, r in enumerate(rows):
        r[i] = 1.0 - sum(r.values())
        cnt[i] = len(r)
        for j in sorted(r):
            col.append(j)
            ele.append(r[j])
    col, ele = np.array(col, np.int32), np.array(ele)
    H = Port().amg(cnt, col, ele)
    s = gpu.Solver()
    s.set_matrix(cnt, col, ele)
    s.setup()
    assert s.num_levels() == H.nlevels
    for l in range(H.nlevels):
        g, o = s.level(l), H.level(l)
        for k in ("cnt", "col", "ele", "sel", "pcnt", "pcol")[:3 if l == H.nlevels - 1 else 6]:
            assert np.array_equal(g[k], o[k]), (l, k)
    s.close()
