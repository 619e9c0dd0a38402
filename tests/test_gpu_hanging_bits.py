"""Hanging faces and edges found through the octants' bitmap and by families
against octant by octant."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W
from tests.test_gpu_balance_paths import _cells, _forest, _union

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("corner", [0, 1])
@pytest.mark.parametrize("prob,depth", [(0.3, 5), (0.9, 4), (0.02, 17)])
def test_hanging_nodes_beside_many_octants(gpu_lib, corner, prob, depth):
    # a small forest alone is looked up octant by octant; beside 76,800 more
    # octants through the bitmap: whole families (refined nearly everywhere),
    # scattered siblings, and (17 levels) keys of 128 bits
    from tmr_gb300 import TMR
    base = W.rotate_blocks(W.brick(2, 2, 1), 8)
    got = []
    for conn in (base, _union([base, W.brick(40, 30, 1)])):
        f = _forest(TMR, 3, conn, 2)
        for p in range(depth - 2):
            c = _cells(f)
            mine = np.flatnonzero(c[:, 0] < len(base))
            flags = np.zeros(len(c), np.intc)
            flags[mine] = W.uniform(17, p, len(mine)) < (prob if p < 3 else 0.0)
            flags[mine[0]] = 1  # the first octant always, down to `depth`
            f.refine(flags, 0, depth)
            f.balance(corner)
        f.createNodes()
        c = _cells(f)
        n = int((c[:, 0] < len(base)).sum())
        mesh = f.getMeshConn()[:n]
        ptr, dc, dw = f.getDepNodeConn()
        nd = int(max(0, -mesh.min()))
        got.append((n, len(c), c[:n, 4].max(), mesh, ptr[:nd + 1], dc[:ptr[nd]], dw[:ptr[nd]]))
    assert got[0][1] < 16384 <= got[1][1] and got[0][2] == depth and len(got[0][4]) > 10
    for a, b in zip(got[0][3:], got[1][3:]):
        assert np.array_equal(a, b)
