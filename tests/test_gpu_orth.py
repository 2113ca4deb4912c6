"""The GMRES orthogonalisation kernel by itself: the basis stays orthogonal to
rounding however close a vector lies to it, and a CTA a "block" (SPLIT) and two
"blocks" a CTA give the same bits.

Two classical passes leave |V^T V - I| at the rounding of the second pass's
update, one unit a basis vector and a few for the norm: (m + 4) 2^-52.  (With
the second pass's coefficients taken from the Gram matrix 4e-14 is left at a
ratio |w| / |w - V h| of 86.)  A basis stored in FP32 adds the rounding of both
vectors of a product and of the norm: 4 2^-24."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from rhodst_b200 import build

HERE = Path(__file__).resolve().parent

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("orth") / "orth_check.so"
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-Xcompiler", "-fvisibility=default", "-o", str(so),
                    str(HERE / "orth_check.cu")], check=True)
    return ctypes.CDLL(str(so))


def _vectors(n, m, ratio, seed):
    """Vectors with |w| / |w - V h| = ratio against the basis of those before."""
    rng = np.random.default_rng(seed)
    W, V = np.empty((m + 1, n)), np.empty((m + 1, n))
    for i in range(m + 1):
        w = rng.standard_normal(n)
        for _ in range(2):
            w -= V[:i].T @ (V[:i] @ w)
        V[i] = w / np.linalg.norm(w)
        c = rng.standard_normal(i)
        W[i] = V[i] + (ratio ** 2 - 1) ** 0.5 * (c / max(np.linalg.norm(c), 1e-300)) @ V[:i]
    return W * rng.uniform(0.1, 10.0, m + 1)[:, None]


def _run(lib, W, fp32, split):
    out = np.zeros_like(W)
    rc = lib.orth_run(ctypes.c_long(W.shape[1]), W.shape[0] - 1, fp32, split, W.ctypes.data_as(ctypes.c_void_p),
                      out.ctypes.data_as(ctypes.c_void_p))
    assert rc == 0
    return out


# entries of one cell, a ragged piece, 4 k cells, the last size with a CTA a
# block (148 x 1024) and the first without, several pieces a thread
@pytest.mark.parametrize("n,m", [(5, 3), (1501, 33), (1500, 64), (20160, 20), (151552, 17), (151555, 17), (700005, 5)])
@pytest.mark.parametrize("ratio", [1.5, 86.0, 1e4])
@pytest.mark.parametrize("fp32", [0, 1])
def test_basis_is_orthogonal(lib, n, m, ratio, fp32):
    W = _vectors(n, m, ratio, 5)
    V = _run(lib, W, fp32, 0)
    G = V.astype(np.longdouble) @ V.T.astype(np.longdouble)
    loss = float(np.abs(G - np.eye(m + 1)).max())
    assert loss <= (4 * 2.0 ** -24 if fp32 else (m + 4) * 2.0 ** -52), loss
    if n <= 151552:
        assert np.array_equal(_run(lib, W, fp32, 1), V)


def test_barrier_gives_up(lib):
    out = np.zeros(3)
    for wait_ms in (0, 30):
        flags = lib.lonely_run(wait_ms, out.ctypes.data_as(ctypes.c_void_p))
        assert flags == 4 and out[0] == 0 and out[1] == 0
        assert wait_ms <= out[2] < wait_ms + 1000
