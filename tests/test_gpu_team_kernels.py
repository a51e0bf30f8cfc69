"""Which levels the warp teams take (k_team): the kernels that ran are named,
so a dispatch that never chose them would show."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("no CUDA device", allow_module_level=True)

from hmfem_b200 import gpu  # noqa: E402
from hmfem_b200.problem import make_problem  # noqa: E402


def _teams(shape, team, monkeypatch, **opt):
    """Warps per slice of every level above the coarse solve (0: a row per
    thread), from the kernels of one iteration; the levels' rows."""
    monkeypatch.setenv("HMFEM_SMALL_CYCLE", "0")
    monkeypatch.setenv("HMFEM_TEAM", team)
    s = gpu.Solver(tol=1e-9, **opt)
    s.assemble(make_problem(*shape, log10k=(-14.0, 1.0, 2.0), seed=shape[1]))
    s.setup()
    s.solve()
    rows = [s.level(l)["n"] for l in range(s.num_levels())]
    warps = {}
    for k in s.profile_iteration(1):
        name = k["kernel"]
        if "k_team" in name or "k_cheb" in name:
            w = 4 if ", 4," in name else 2 if ", 2," in name else 0
            warps.setdefault(k["level"], set()).add(w if "k_team" in name else 0)
    s.close()
    return warps, rows


@pytest.mark.parametrize("opt", [dict(), dict(precision=1), dict(precision=1, bf16_from=1)],
                         ids=["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("shape", [(91, 61, 63), (120, 96, 80)])
def test_teams_run_where_the_rule_says(shape, opt, monkeypatch):
    seen = set()
    warps, rows = _teams(shape, "1", monkeypatch, **opt)
    assert warps
    for l, w in warps.items():
        slices = -(-rows[l] // 32)
        want = 4 if slices * 4 <= 148 * 16 else 2 if slices * 2 <= 148 * 16 else 0
        assert w == {want}, (l, rows[l], w)
        seen |= w
    assert seen & {2, 4}
    off, _ = _teams(shape, "0", monkeypatch, **opt)
    assert set(off) == set(warps) and all(w == {0} for w in off.values())
