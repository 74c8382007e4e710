"""bench.py --impl reference where the reference's library is not built: one JSON line that says so, and exit 0."""
import json
import pathlib
import sys

ROOT = pathlib.Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))
sys.path.insert(0, str(ROOT / "luminagi-cudaref_b200"))


def test_says_that_it_is_unavailable(monkeypatch, capsys):
    import bench
    import oracle as O
    monkeypatch.setattr(O, "ref_available", lambda: False)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--scene", "box", "--steps", "1"])
    bench.main()
    line, = capsys.readouterr().out.strip().splitlines()
    got = json.loads(line)
    assert got["impl"] == "reference" and got["unavailable"]
