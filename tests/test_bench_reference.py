"""bench.py's reference arm times the reference's own program or says that there is none."""
import json
import os
import sys
import types

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def test_no_stand_in_for_a_missing_reference_program(monkeypatch, capsys, tmp_path):
    import bench
    from oracle import pyoracle, refscene
    monkeypatch.setattr(refscene, "REF_BIN", str(tmp_path / "ref_render"))
    monkeypatch.setattr(pyoracle, "Oracle", None)             # the CPU restatement is not asked
    bench.run_reference(types.SimpleNamespace(gpus=1, steps=1, warmup=0), 0, 1)
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
    assert "value" not in line and "e2e" not in line
