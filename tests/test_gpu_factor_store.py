"""Device memory of the ILU: a context whose factorisation writes the apply's
records (hexahedra) holds those, not the sliced factor store beside them.

The records hold the blocks of the store and the pivot inverses, with headers
and columns (an eighth more at the most: 32 bytes a block of 200), so against a
context with the store and the register apply at most the records of the
inverses and that eighth come on top: a store that is kept too is another six
blocks a row."""
import gc

import pytest

import rhodst_b200
from rhodst_b200 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,size", [("fp64", 8), ("fp32", 4)])
def test_no_store_beside_the_records(prec, size):
    import torch
    case = cases.swept_wing_c3(128, 40, 32, 16, precision=prec)
    used = {}
    for bulk in (False, True, False, True):     # the second pair: with the library's own memory in place
        gc.collect()                            # contexts of earlier tests
        free = torch.cuda.mem_get_info()[0]
        s = rhodst_b200.solver_for(case.with_options(**{"ilu.bulk": bulk}))
        used[bulk] = free - torch.cuda.mem_get_info()[0]
        s.close()
    N, Fi = case.mesh.n_cells, case.mesh.n_internal_faces
    block = 25 * size
    records = N * block + (N + 2 * Fi) * block // 8
    lists = 16 * N + 20 * Fi                    # descriptors and task lists; 16 MB: rounding of eight allocations
    assert used[True] - used[False] <= records + lists + (16 << 20), (used, records)
    assert records + lists + (16 << 20) < 2 * Fi * block * 2 // 3      # the store itself would show
