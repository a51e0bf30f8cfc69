"""The general split's bounded wait: rows that only wait for a neighbour of
their own tile poll fast, and must not give up sooner than a row that waits on
an earlier tile while a long chain of decisions runs before them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402


def test_a_fast_poller_waits_as_long_as_a_slow_one(monkeypatch):
    # Tiles of 1024 rows, one per SM.  147 tiles of a line ordered along itself
    # (one decision after another, ~0.16 s); in the last tile row a continues
    # the line, a + 512 (another warp) hangs on a, the others are alone and
    # leave at once.
    a, n = 147 * 1024, 148 * 1024
    edges = [(i, i + 1) for i in range(a)] + [(a, a + 512)]
    lo = np.array([e[0] for e in edges])
    up = np.array([e[1] for e in edges])
    row = np.concatenate([lo, up, np.arange(n)])
    col = np.concatenate([up, lo, np.arange(n)])
    ele = np.concatenate([np.full(2 * len(edges), -1.0), np.full(n, 3.5)])
    order = np.lexsort((col, row))
    cnt = np.bincount(row, minlength=n)
    # 220000 polls of an earlier tile take ~0.27 s
    monkeypatch.setenv("HMFEM_TEST_POLL_LIMIT", "220000")
    s = gpu.Solver()
    s.set_matrix(cnt.astype(np.int32), col[order].astype(np.int32), ele[order])
    s.setup()
    sel = s.level(0)["sel"]
    want = np.ones(n, sel.dtype)
    want[1:a + 1:2] = 2
    want[a + 512] = 2 if want[a] == 1 else 1
    assert np.array_equal(sel, want)
    s.close()
