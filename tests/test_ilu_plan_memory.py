"""The record plan of the ILU is filled by several threads; one that cannot be
started for want of memory must not end the process (the C entry points return
an error instead)."""
import subprocess
from pathlib import Path

HERE = Path(__file__).resolve().parent


def test_plan_survives_a_failed_allocation(tmp_path):
    exe = tmp_path / "ilu_plan_memory_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-o", str(exe), str(HERE / "ilu_plan_memory_check.cpp")],
                   check=True)
    assert subprocess.run([str(exe)]).returncode == 0
