"""A bounded device wait that runs out: the call reports RDST_ERR_TIMEOUT, the
context says so until a state is set, and then works as a new one does (the
same numbers to the bit).  The limit is set to zero, so that every wait gives
up at once and nothing is waited for."""
import numpy as np
import pytest

import rhodst_b200
from rhodst_b200 import cases
from rhodst_b200._abi import RdstError

pytestmark = pytest.mark.gpu

RDST_ERR_TIMEOUT, RDST_ERR_ARG = 5, 7


def _set(s, case):
    s.set_primitive(case.p, case.U, case.T)


def _times_out(call):
    with pytest.raises(RdstError) as e:
        call()
    assert e.value.status == RDST_ERR_TIMEOUT
    assert "expired" in str(e.value)


CASES = {
    # the grid barrier of the orthogonalisation, with both storages of the basis
    "gmres_fp64": lambda: cases.forward_step_c1(),
    "gmres_fp32": lambda: cases.forward_step_c1().with_options(precision="fp32"),
    # that of BiCGStab, launched ahead of the check
    "bicgstab": lambda: cases.forward_step_c1(solver="BiCGStab"),
    # the ILU apply's alone
    "ilu": lambda: cases.forward_step_c1(solver="ILU", preconditioner="ILUC0", max_iter=4).with_options(
        **{"solvers.W.minIter": 4, "ilu.parts": 8}),
    "ilu_tight": lambda: cases.swept_wing_c3(n_around=36, n_normal=12, n_span=9, n_tip=5, precision="fp32",
                                             n_directions=8, ilu_parts=900),
}


@pytest.mark.parametrize("name", CASES)
def test_step_reports_and_recovers(name):
    case = CASES[name]()
    s = rhodst_b200.Solver(case.mesh, case.bcs, case.options)
    _set(s, case)
    s.step(2)
    want = s.conservative()
    _set(s, case)
    s.set_wait_limit(0.0)
    _times_out(lambda: s.step(2))
    s.set_wait_limit(2.0)
    _times_out(lambda: s.step(1))          # until a state is set
    _set(s, case)
    s.step(2)
    for a, b in zip(s.conservative(), want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("solver", ["GMRES", "BiCGStab"])
def test_adjoint_reports_and_recovers(solver):
    case = cases.naca0012_inviscid(65, 17).with_options(**{"solvers.W.solver": solver, "ilu.parts": 4})
    s = rhodst_b200.Solver(case.mesh, case.bcs, case.options)
    _set(s, case)
    s.step(3)
    W = s.conservative()

    def adjoint():
        return s.adjoint(case.force_patch, case.force_dirs["drag"], rel_tol=1e-12, max_cycles=2, n_directions=12,
                         want_psi=True)

    want, psi = adjoint()
    s.set_wait_limit(0.0)
    _times_out(adjoint)
    s.set_wait_limit(2.0)
    got, psi2 = adjoint()                  # the state is as it was
    assert np.array_equal(psi, psi2) and got["residual"] == want["residual"]
    for a, b in zip(s.conservative(), W):
        assert np.array_equal(a, b)
    s.step(1)
    # a step's expired wait is not cleared by an adjoint call
    s.set_wait_limit(0.0)
    _times_out(lambda: s.step(1))
    s.set_wait_limit(2.0)
    _times_out(adjoint)


def test_limit_range():
    case = cases.forward_step_c1()
    s = rhodst_b200.Solver(case.mesh, case.bcs, case.options)
    for bad in (-1.0, 3601.0, float("nan")):
        with pytest.raises(RdstError) as e:
            s.set_wait_limit(bad)
        assert e.value.status == RDST_ERR_ARG
