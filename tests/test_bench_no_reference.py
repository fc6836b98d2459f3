"""bench.py --impl reference where the reference's library is not built: one
line that says so, and a clean exit."""
import argparse
import json

import bench


def test_the_line_says_so(monkeypatch, capsys):
    monkeypatch.setattr(bench, "reference_built", lambda: False)
    args = argparse.Namespace(qubits=16, depth=4, terms=2, shots=100, steps=1, warmup=3, validate_cpu=False,
                              no_reference_gpu=True)
    bench.main_reference(args, 0, 1)
    (line,) = [json.loads(x) for x in capsys.readouterr().out.splitlines()]
    assert line["impl"] == "reference" and "not built" in line["unavailable"]
    bench.main_reference(args, 1, 2)  # other ranks print nothing
    assert capsys.readouterr().out == ""
