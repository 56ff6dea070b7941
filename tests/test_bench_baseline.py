"""The benchmark's GPU line keeps its measurements where the reference package is missing or fails."""
import argparse
import json
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("error", [ImportError("reference package not installed"), RuntimeError("two\nlines"), None])
def test_line_without_the_reference(monkeypatch, error):
    monkeypatch.syspath_prepend(ROOT)
    import bench
    from oracle import ref_step

    def time_steps(*a, **k):
        if error is not None:
            raise error
        return 7.0, {"threads": 1, "steps": 1, "warmup": 1, "seconds": 1.0}

    monkeypatch.setattr(ref_step, "time_steps", time_steps)
    monkeypatch.setattr(bench, "cpu_baseline_port", lambda args: {"value": 2.0})
    args = argparse.Namespace(L=8, rank=2, batch=4, ref_batch=2, seed=0, width=6)
    line = json.loads(json.dumps(bench.cpu_baselines(args)))
    assert line["cpu_baseline_es_port"] == {"value": 2.0}
    assert line["cpu_baseline"]["value"] == (7.0 if error is None else None)
    if error is not None:
        assert line["cpu_baseline"]["unavailable"] == f"{type(error).__name__}: {error}".splitlines()[0]
