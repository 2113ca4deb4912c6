"""The record route of the subdomain ILU against gather + factorisation +
register apply on prisms and tetrahedra, whose breadth-first order gives rows of
up to four blocks a side: one more than the record kernels hold in registers, in
the record layout of each storage.  From one subdomain to six an SM, and one
whose levels (up to 1,053 rows) are too wide for the factorisation's level
buffers.

Same blocks, summed in another order: a relative 2^-53 an operation along a
chain of 200 levels is 2e-14 in an application, ten times that in a step at the
most; FP32 and BF16 factors are applied in FP32 by one and in FP64 by the other,
2^-24 likewise.  1e-11 and 1e-5 of the state after two steps."""
import numpy as np
import pytest

import rhodst_b200
from rhodst_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("fp32", 1e-5), ("bf16", 1e-5)])
@pytest.mark.parametrize("dims,parts", [((24, 10, 8), 1), ((24, 10, 8), 7), ((24, 10, 8), 148), ((24, 10, 8), 700),
                                        ((24, 10, 8), 900), ((28, 30, 30), 1)])
def test_routes_agree_on_prisms_and_tetrahedra(dims, parts, prec, tol):
    base = cases.forward_step_3d_hybrid_c5(*dims, precision=prec).with_options(
        **{"ilu.parts": parts, "ilu.order": "bfs", "solvers.W.nDirections": 8})
    out = []
    for bulk in (True, False):
        s = rhodst_b200.solver_for(base.with_options(**{"ilu.bulk": bulk}))
        s.step(2)
        out.append(s.conservative())
        s.close()
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-11), ("fp32", 1e-5), ("bf16", 1e-5)])
@pytest.mark.parametrize("fill,parts", [(1, 1), (1, 8), (2, 8)])
def test_routes_agree_with_fill(fill, parts, prec, tol):
    """Fill of one and two faces more (up to 6 and 12 blocks a side on quads):
    rows that update blocks of their own, so the factorisations beside the record
    one, their L and U packed into the records; chains of up to 160 levels."""
    base = cases.forward_step_c1(preconditioner="ILUCp", n_directions=8).with_options(
        **{"precision": prec, "ilu.parts": parts, "solvers.W.fillInLevel": fill})
    out = []
    for bulk in (True, False):
        s = rhodst_b200.solver_for(base.with_options(**{"ilu.bulk": bulk}))
        s.step(2)
        out.append(s.conservative())
        s.close()
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= tol * np.abs(b).max()
