"""The record plan of the subdomain ILU apply (rdst_records.h), walked on the
CPU as the kernel walks it: offsets, row ids, columns, group ranges and the
result of both sweeps against the plain substitution (same order of the same
FP64 operations up to the row order inside a task: 1e-12)."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("rec") / "ilu_records_check.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-o", str(so),
                    str(HERE / "ilu_records_check.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("n,nparts,wide,reach,sms", [
    (1, 1, 2, 1, 148),          # one row
    (7, 3, 2, 3, 148),          # subdomains of two or three rows
    (700, 5, 2, 9, 148),        # levels of a few rows: warps taking turns
    (3000, 4, 3, 400, 148),     # levels of hundreds of rows: full and partial tasks
    (3001, 7, 4, 60, 2),        # four subdomains an SM
    (2500, 8, 7, 150, 1),       # more blocks than the registers hold, six subdomains an SM
    (900, 2, 16, 80, 148),      # the widest rows
    (9000, 1, 2, 8000, 148),    # levels wider than the level buffers: columns in the global vector
])
@pytest.mark.parametrize("elem", [2, 4, 8])
def test_records_reproduce_the_substitution(lib, n, nparts, wide, reach, sms, elem):
    for gauss_seidel in (0, 1):
        assert lib.check_records(n, nparts, wide, reach, elem, sms, gauss_seidel, 7) == 0
