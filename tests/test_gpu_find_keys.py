"""Enclosing coarse elements searched by 64-bit keys against the search by
coordinates (where the keys need 128 bits): the same P."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W
from tests.test_gpu_balance_paths import _brick, _cells, _union

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("gap", [1, 0])
def test_rows_by_keys_equal_rows_by_coordinates(gpu_lib, dim, order, gap):
    # gap 0: the other forest refined elsewhere, finer in places than this one
    from tmr_gb300 import TMR
    base = _brick(dim, 2, 2, 2)
    if dim == 3:
        base = W.rotate_blocks(base, 3)
    depth = 17 if dim == 3 else 27

    def refined(conn, seed):
        f = (TMR.OctForest if dim == 3 else TMR.QuadForest)(order=order)
        f.setConnectivity(conn)
        f.createTrees(1)
        for p in range(depth - 1):
            c = _cells(f)
            mine = np.flatnonzero(c[:, 0] < len(base))
            pick = np.zeros(len(c), np.intc)
            pick[mine] = W.uniform(seed, p, len(mine)) < (0.2 if p < 2 else 0.0)
            pick[mine[-1 if seed % 2 else 0]] = 1
            f.refine(pick, 0, depth)
            f.balance(1)
        f.createNodes()
        return f

    got = []
    for conn in (base, _union([base, _brick(dim, 40, 30, 1)])):
        fine = refined(conn, 5)
        if gap:
            coarse = fine.coarsen()
            coarse.balance(1)
            coarse.createNodes()
        else:
            coarse = refined(conn, 6)
        rows = 1 + max(int(m[m >= 0].max()) for m in
                       (fine.getMeshConn()[_cells(fine)[:, 0] < len(base)],))
        P = TMR.VecInterp()
        fine.createInterpolation(coarse, P)
        ptr, cols, w = P.getCSR()
        got.append((ptr[:rows + 1], cols[:ptr[rows]], w[:ptr[rows]]))
        assert _cells(fine)[:, 4 if dim == 3 else 3].max() == depth
    for a, b in zip(*got):
        assert np.array_equal(a, b)
