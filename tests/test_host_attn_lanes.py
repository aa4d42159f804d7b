"""Attention of few queries on the CPU: the value columns that each lane reads.  CPU only."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_lane_reads_behind_a_value_row(tmp_path):
    """A block of columns that is not full: its lanes must not read what lies behind the row, which for the last row is behind the tensor.  The numbers would be thrown
    away, so that no result can show it."""
    exe = str(tmp_path / "lanes")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(ROOT, "tests", "host", "attn_lanes_check.cpp"), "-o", exe], check=True, capture_output=True, timeout=300)
    sizes = [*range(1, 140), 256, 511, 512, 513, 576, 640, 1000, *range(1020, 1036), 1500, 2047, 2048, 2049, 2052, 5000]
    out = subprocess.run([exe, *map(str, sizes)], check=True, capture_output=True, text=True, timeout=300).stdout.split("\n")
    rows = [tuple(map(int, r.split())) for r in out if r]
    assert len(rows) == 5 * len(sizes)
    assert [r for r in rows if r[2] or r[3]] == []
