"""The profiling harness the profiles/ summaries cite parses its arguments on
the CPU, and its byte counts agree with the ones bench.py reports."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_profile_cases_help_lists_every_case():
    out = subprocess.run([sys.executable, "-m", "kg_b200.profile_cases", "--help"], cwd=ROOT, capture_output=True,
                         text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    for case in ("pirk", "mixed", "proj", "configured", "batch", "refine", "diag", "steppers"):
        assert case in out.stdout


def test_stage_bytes_agree_with_bench():
    sys.path.insert(0, ROOT)
    import bench
    from kg_b200.profile_cases import STAGE_BYTES
    for k, v in bench.ALG_BYTES.items():
        assert STAGE_BYTES[k] == v


def test_stage_points_leave_out_what_the_fill_writes():
    """The launch that the committed counters belong to moves at least the bytes that
    the roofline counts for it."""
    sys.path.insert(0, ROOT)
    import bench
    from kg_b200.profile_cases import STAGE_BYTES, WHOLE_GRID, stage_points
    w = bench.WORKLOAD
    grid = (w["Nx"], w["Ny"], w["Nz"])
    for k in STAGE_BYTES:
        n = stage_points(k, *grid)
        assert n == (bench.stored_points(w) if k in WHOLE_GRID else 2053 * 128 * 257)
    counted = bench.ALG_BYTES["stage_pirk2_s2"] * stage_points("stage_pirk2_s2", *grid)
    assert 1.0 <= bench.profile_traffic("stage_pirk2_s2") / counted < 1.1
