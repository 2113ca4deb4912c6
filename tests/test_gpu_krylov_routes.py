"""The routes a context can take through the subdomain ILU, BiCGStab and the
field exchange, each against the route beside it.

* Factorisation and apply on the records' tasks against gather + factorisation
  + register apply (ilu.bulk false), from one subdomain to several an SM
  (the instances for five and six CTAs an SM).  FP64: the same blocks summed in
  another order, 1e-12 relative per step; FP32 and BF16 factors are applied in
  FP32 by one and in FP64 by the other, 1e-6 after two steps (the tolerances
  of the bulk-against-register tests).
* BiCGStab launching an iteration ahead (graphs) against one that waits for
  every check (no graphs): the same kernels, so bit for bit.
* Primitive fields in and out through the reordered numbering: the same values."""
import numpy as np
import pytest

import rhodst_b200
from rhodst_b200 import cases

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-6), ("bf16", 1e-6)])
@pytest.mark.parametrize("parts", [1, 7, 148, 500, 700, 900])
def test_ilu_routes_agree(parts, prec, tol):
    base = cases.swept_wing_c3(n_around=36, n_normal=12, n_span=9, n_tip=5, precision=prec, n_directions=8,
                               ilu_parts=parts)
    out = []
    for bulk in (True, False):
        s = rhodst_b200.solver_for(base.with_options(**{"ilu.bulk": bulk}))
        s.step(2)
        out.append(s.conservative())
    for a, b in zip(*out):
        assert rel(a, b) < tol


@pytest.mark.parametrize("precon", ["ILUC0", "diagonal"])
def test_bicgstab_ahead_matches_waiting(precon):
    case = cases.forward_step_c1(solver="BiCGStab", preconditioner=precon, max_iter=60).with_options(
        **{"solvers.W.tolerance": 1e-9, "solvers.W.minIter": 1, "ilu.parts": 8})
    out = []
    for graphs in (True, False):
        s = rhodst_b200.solver_for(case.with_options(graphs=graphs))
        reps = s.step(3)
        out.append(([r["lin_iterations"] for r in reps], [r["flags"] for r in reps], s.conservative()))
    assert out[0][0] == out[1][0] and out[0][1] == out[1][1]
    assert max(out[0][0]) < 60
    for a, b in zip(out[0][2], out[1][2]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("turb", [False, True])
def test_primitive_fields_round_trip(turb):
    case = cases.naca0012_turbulent(97, 25) if turb else cases.naca0012_inviscid(65, 17)
    case = case.with_options(**{"ilu.parts": 5})
    rng = np.random.default_rng(3)
    N = case.mesh.n_cells
    p, T = 1.0 + 0.1 * rng.random(N), 1.0 + 0.1 * rng.random(N)
    U = case.U * (1.0 + 0.1 * rng.random(N))[:, None]
    nut = case.nuTilda * (1.0 + rng.random(N)) if turb else None
    s = rhodst_b200.Solver(case.mesh, case.bcs, case.options)
    s.set_primitive(p, U, T, nut)
    p1, U1, T1, nut1 = s.primitive()
    assert np.array_equal(p, p1) and np.array_equal(T, T1) and np.array_equal(U, U1)
    assert np.array_equal(nut1, nut if turb else np.zeros(N))
