"""GMRES basis sizes around the orthogonalisation kernel's edges: one vector,
a full set of 16 and one more, 32 and one more, the 64 allowed, and a Krylov
space that is nearly exhausted (a small mesh, many directions: the Arnoldi
vectors come close to the basis and take the second pass).

The oracle orthogonalises by modified Gram-Schmidt; in exact arithmetic both
are the same, and one restart cycle's step agrees to 1e-9 relative as in the
other GMRES step tests.  With FP32 storage of the Jacobian and the basis the
step is compared with the FP64 one at 1e-5 of the update (FP32 rounding of the
matrix, 6e-8, times the condition of the few directions taken)."""
import numpy as np
import pytest

import rhodst_b200
from rhodst_b200 import cases
from tests.oracle_lib import OracleSolver

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("precon", ["diagonal", "ILUC0"])
def test_directions_match_oracle(m, precon):
    case = cases.forward_step_c1(preconditioner=precon, n_directions=m).with_options(**{"ilu.parts": 1})
    gpu = rhodst_b200.Solver(case.mesh, case.bcs, case.options)
    ora = OracleSolver(case.mesh, case.bcs, case.options)
    for s in (gpu, ora):
        s.set_primitive(case.p, case.U, case.T)
    rg, ro = gpu.step(3), ora.step(3)
    for a, b in zip(rg, ro):
        assert abs(a["res_mag"] - b["res_mag"]) <= 1e-9 * abs(b["res_mag"])
    for a, b in zip(gpu.conservative(), ora.conservative()):
        assert rel(a, b) < 1e-9


@pytest.mark.parametrize("m", [5, 17, 33])
def test_fp32_basis_step(m):
    case = cases.forward_step_c1(n_directions=m)
    W, W0 = {}, None
    for prec in ("fp64", "fp32"):
        s = rhodst_b200.solver_for(case.with_options(precision=prec))
        if W0 is None:
            W0 = s.conservative()
        s.step(1)
        W[prec] = s.conservative()
    for w0, a, b in zip(W0, W["fp32"], W["fp64"]):
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b - w0).max()
