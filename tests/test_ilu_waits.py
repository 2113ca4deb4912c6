"""A bounded wait of the record apply that expires leaves no warp in a level
barrier: the compute warps' walk of rdst_records.h on the CPU, every group of
both sweeps lost by one warp, by all but one and by random ones."""
import ctypes
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("waits") / "ilu_waits_check.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-o", str(so),
                    str(HERE / "ilu_waits_check.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("nlev,wide,nparts", [
    (1, 4, 1),          # no level barrier at all
    (3, 5, 1),          # fewer tasks than warps
    (40, 6, 1),         # a task a level: warps taking turns
    (23, 60, 1),        # several tasks a level
    (50, 70, 1),        # several groups a sweep
    (40, 60, 4),        # four subdomains an SM
    (40, 60, 6),        # six: the tight instance
])
@pytest.mark.parametrize("elem", [4, 8])
def test_expired_waits_leave_no_warp_behind(lib, nlev, wide, nparts, elem):
    assert lib.check_waits(nlev, wide, elem, nparts, 11) == 0
