"""bench.py where the compiled reference cannot be had: the reference arm says
so in its one line and ends, and worker processes that fail to start end the
step with an error instead of being started again for ever."""
import concurrent.futures.process
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402
from oracle import pyoracle as po  # noqa: E402


@pytest.mark.parametrize("workload", ["pt1080p", "raycast", "batch", "adjoint", "cornell"])
def test_reference_arm_without_the_reference(monkeypatch, capsys, workload):
    monkeypatch.setattr(po, "REF_SO", os.path.join(ROOT, "oracle", "no_such_library.so"))
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--workload", workload])
    bench.main()
    out = json.loads(capsys.readouterr().out)
    assert out["impl"] == "reference" and out["unavailable"]


@pytest.mark.timeout(120)
def test_workers_that_fail_to_start_end_the_step():
    with bench.ref_pt_pool(2, init=int, initargs=("not a number",)) as pool:
        with pytest.raises(concurrent.futures.process.BrokenProcessPool):
            bench.ref_pt_step(pool, 2, 0)
