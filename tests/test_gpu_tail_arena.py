"""The small levels' arena running out of room (HMFEM_TEST_TAIL_ARENA makes it
small): the general path makes the next level, the one-launch form may take
over again below it, and the levels made before keep their place -- every
level the oracle's, whatever the room."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402
from oracle.oracle import Port  # noqa: E402


@pytest.mark.parametrize("shape", [(19, 9, 6), (64, 1, 1), (41, 25, 1)])
def test_levels_stay_the_oracles_when_the_arena_is_full(shape, monkeypatch):
    port = Port()
    p = make_problem(*shape, log10k=(-14.0, 1.5, 2.0), seed=sum(shape))
    perm, ind, b = port.assemble(p)
    cnt, col, ele = port.pack(perm, ind)
    H = port.amg(cnt, col, ele)
    s = gpu.Solver(tol=1e-10)
    x0 = None
    for room in [1 << 21, 0, 1000] + list(range(2000, 90000, 2500)):
        monkeypatch.setenv("HMFEM_TEST_TAIL_ARENA", str(room))
        s.set_matrix(cnt, col, ele, b)
        s.setup()
        assert s.num_levels() == H.nlevels
        for l in range(H.nlevels):
            g, o = s.level(l), H.level(l)
            keys = ("cnt", "col", "ele", "dinv") + (("sel", "pcnt", "pcol")
                                                    if l < H.nlevels - 1 else ())
            for k in keys:
                assert np.array_equal(g[k], o[k]), (room, l, k)
        x, st = s.solve()
        x0 = x if x0 is None else x0
        assert np.array_equal(x, x0), room
    s.close()
