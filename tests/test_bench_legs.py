"""bench.py's extra legs: one that fails does not take the line with it, the batched leg leaves room for the work
buffers of all its volumes, and profile figures of another kernel are not reported."""
import json
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
bench = pytest.importorskip("bench")


def test_failing_leg_is_reported_in_its_place():
    def leg(x):
        raise RuntimeError("CUDA out of memory" + "." * 1000)

    r = bench.extra(leg, 1)
    assert r["error"].startswith("RuntimeError: CUDA out of memory") and len(r["error"]) < 400
    assert bench.extra(lambda a: {"v": a}, 3) == {"v": 3}


@pytest.mark.parametrize("free_gb", [277, 200, 60])
def test_batched_volumes_leave_room(free_gb):
    """Byte ledger of the 48 volumes: 1.6 KB a sample for the tables at J = 6, taken while the buffers still fit."""
    vols = bench.uneven_volumes()
    work = sum(bench.batch_work_bytes(N, om.size // 3, nc) for om, N, nc, _ in vols)
    free, tables = free_gb << 30, 0
    for om, N, nc, _ in vols:
        m = om.size // 3
        if bench.table_options(m, free - work - (12 << 30)) == {}:
            free -= 1600 * m
            tables += 1
    assert free >= work or tables == 0
    if free_gb == 277:
        assert work < free and 10 < tables <= 48


def test_profile_figures_belong_to_the_kernel(tmp_path, monkeypatch):
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    assert bench.ncu_figure("gather", "traffic") is None
    (tmp_path / "profiles").mkdir()
    p = tmp_path / "profiles" / "interp_traffic_N128.json"
    p.write_text(json.dumps({"gather": {"kernel": "k_gather_tab", "traffic": 1}, "spread": 5}))
    assert bench.ncu_figure("gather", "traffic") is None and bench.ncu_figure("spread", "traffic") is None
    p.write_text(json.dumps({"gather": {"kernel": "k_gather_rows", "traffic": 7}}))
    assert bench.ncu_figure("gather", "traffic") == 7 and bench.ncu_figure("gather", "sm_side") is None
