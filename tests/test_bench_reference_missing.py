"""`bench.py --impl reference` where the reference's library was not built: one
JSON line that says so, and a clean exit."""
import json
from types import SimpleNamespace

import bench
from oracle import oracle


def test_a_missing_reference_is_reported(monkeypatch, tmp_path, capsys):
    monkeypatch.setattr(oracle, "REF_SO", str(tmp_path / "libhmfem_ref.so"))
    monkeypatch.delenv("RANK", raising=False)
    bench.run_reference(SimpleNamespace(size=256, tol=1e-10, steps=2, warmup=1, gpus=1))
    (line,) = capsys.readouterr().out.strip().splitlines()
    d = json.loads(line)
    assert d["impl"] == "reference" and "libhmfem_ref.so" in d["unavailable"]
