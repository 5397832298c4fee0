"""Columns-per-lane choice per length bucket (ragged.cols_table, bucket_of):
host logic, on CPU."""

import json
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def test_buckets():
    from orihime_b200 import ragged

    assert ragged.bucket_of(32, 32) == "0:0"
    assert ragged.bucket_of(300, 63) == "0:256"
    assert ragged.bucket_of(255, 64) == "64:0"
    assert ragged.bucket_of(2048, 2048) == "1024:256"
    assert ragged.bucket_of(256, 1023) == "512:256"
    # every bucket has a default
    for a2 in ragged.L2_EDGES:
        for a1 in ragged.L1_EDGES:
            assert ragged.DEFAULT_COLS[f"{a2}:{a1}"] in (2, 4, 8)


def test_table_overrides(monkeypatch, tmp_path):
    from orihime_b200 import ragged

    monkeypatch.setenv("ORIHIME_B200_CACHE", str(tmp_path))
    monkeypatch.delenv("ORIHIME_B200_COLS", raising=False)
    assert ragged.cols_table() == ragged.DEFAULT_COLS
    monkeypatch.setenv("ORIHIME_B200_COLS", "0:0=4,1024:256=2")
    t = ragged.cols_table()
    assert t["0:0"] == 4 and t["1024:256"] == 2 and t["512:0"] == ragged.DEFAULT_COLS["512:0"]
    monkeypatch.setenv("ORIHIME_B200_COLS", json.dumps({"64:0": 8}))
    assert ragged.cols_table()["64:0"] == 8
    p = tmp_path / "t.json"
    p.write_text(json.dumps({"128:256": 4}))
    monkeypatch.setenv("ORIHIME_B200_COLS", str(p))
    assert ragged.cols_table()["128:256"] == 4


def test_bench_batch_computed_cells_reported():
    """Cells the bands compute per useful cell on the bench batch (dead
    columns of each pair's last band, 31 fill and drain steps per band) at 4
    columns per lane for all pairs and with the bucket table.  The table is
    chosen for time, not for this count: 8 columns per lane computes more
    dead cells on wide pairs but halves the per-step work of the bands."""
    import bench
    from orihime_b200 import ragged

    ln = bench.workload_lengths(3)
    useful = float((ln[:, 0] * ln[:, 1]).sum())
    r4 = ragged.pair_cost(ln, 4).sum() / useful
    cols = np.array([ragged.DEFAULT_COLS[ragged.bucket_of(int(a), int(b))] for a, b in ln])
    w = 32 * cols
    nb = np.maximum(1, (ln[:, 1] + w - 1) // w)
    mixed = (nb * (ln[:, 0] + 31) * w).sum() / useful
    print(f"  computed / useful cells: 4 columns per lane {r4:.3f}, bucket table {mixed:.3f}")
    assert 1.0 < r4 < 1.3 and 1.0 < mixed < 1.4


def test_bench_traffic_profile_per_cols():
    """The bench's roofline traffic comes from the committed DRAM capture of
    the adjoint it launched: one per columns-per-lane choice."""
    import bench

    for cols in (4, 8):
        v, src = bench.profile_traffic(cols)
        assert v is not None and 8.0 <= v <= 20.0, (cols, v)
        assert os.path.exists(os.path.join(ROOT, src))
    assert bench.profile_traffic(2) == (None, None)


def test_columns_do_not_depend_on_the_batch_and_fall_with_the_temperature(monkeypatch, tmp_path):
    from orihime_b200 import _lib, ragged

    q = _lib.load().swb_cols_per_lane
    for fam in (1, 3):
        for L2 in (1, 64):
            assert q(fam, L2, -2.0, -0.5, 1.0) == 2
        for L2 in (65, 255, 256, 300, 4096):
            for T, want in ((1.0, 4), (0.35, 4), (0.34, 2), (0.25, 2)):
                assert q(fam, L2, -2.0, -0.5, T) == want, (fam, L2, T)
            assert q(fam, L2, 1.0, -0.5, 0.25) == 4   # the log domain
    for fam in (2, 4, 5):
        assert q(fam, 300, -2.0, -0.5, 0.25) == 4
    assert [ragged.cols_limit(T) for T in (1.0, 0.5, 0.49, 0.35, 0.34)] == [8, 8, 4, 4, 2]
    assert [ragged.cols_limit(1.0, s) for s in (6.0, 8.5, 10.0)] == [8, 4, 2]

    # autotune_plan offers no candidate above the limit, whatever an earlier call cached
    monkeypatch.setenv("ORIHIME_B200_CACHE", str(tmp_path))
    monkeypatch.delenv("ORIHIME_B200_COLS", raising=False)
    made = []

    class Fake:
        def __init__(self, ln, off, family, device, cols_per_lane=0, table=None):
            made.append(("mixed", max(table.values())) if table else ("R", cols_per_lane))

    monkeypatch.setattr(ragged, "Plan", Fake)
    monkeypatch.setattr(ragged, "MixedPlan", Fake)
    ln = np.array([[300, 400], [50, 60]])
    off, ln32 = ragged.layout(ln)
    for temp, sig in ((1.0, ""), (0.35, "|c4"), (0.25, "|c2")):
        path = tmp_path / "plans_cpu.json"
        monkeypatch.setattr(ragged, "_cache_path", lambda dev: str(tmp_path / "cols_cpu.json"))
        base = ragged._signature(ln32, "affine")
        path.write_text(json.dumps({base + s: {"choice": c} for s, c in (("", "R8"), ("|c4", "mixed"), ("|c2", "R2"))}))
        made.clear()
        _, report = ragged.autotune_plan(ln32, off, device="cpu", gap_open=-2.0, gap_ext=-0.5, temp=temp)
        assert report["cached"]
        assert made == {"": [("R", 8)], "|c4": [("mixed", 4)], "|c2": [("R", 2)]}[sig]
