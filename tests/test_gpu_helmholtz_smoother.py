"""The smoother a Helmholtz filter chooses: on meshes with elements much larger
than r (where the mass matrix rules) as on those without, few iterations and the
same field as with the longer smoother."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [3, 7])
@pytest.mark.parametrize("dim", [3, 2])
def test_chosen_smoother_takes_few_iterations(gpu_lib, dim, depth):
    # refined towards a corner down to `depth`, with r of the finest elements
    from tmr_gb300 import TMR
    conn = W.brick(3, 2, 2) if dim == 3 else W.brick2d(6, 5)
    nb = len(conn)
    f = (TMR.OctForest if dim == 3 else TMR.QuadForest)(order=2)
    f.setConnectivity(conn)
    f.createTrees(2)
    for p in range(depth - 2):
        a = f.getOctantsArray() if dim == 3 else f.getQuadrantsArray()
        flags = np.zeros(len(a), np.intc)
        flags[a[:, 0] == 0] = 1 if p == 0 else 0
        flags[0] = 1
        f.refine(flags, 0, depth)
        f.balance(1)
    forests = [f]
    for _ in range(2):
        c = forests[-1].coarsen()
        c.balance(1)
        forests.append(c)
    for c in forests:
        c.createNodes()
        if dim == 3:
            c.setBlockBoxes(np.array([[b % 3, b // 3 % 2, b // 6, 1, 1, 1] for b in range(nb)],
                                     np.float64))
        else:
            c.setFaceBoxes(np.array([[b % 6, b // 6, 1, 1] for b in range(nb)], np.float64))
    n = int(f.getNodeRange()[1])
    x = W.uniform(5, 0, n)
    H = TMR.HelmholtzFilter(2.0 / 2.0 ** depth, None, forests)
    y, z = np.empty(n), np.empty(n)
    H.applyFilter(x, y)
    its = H.lastSolve()[0]
    H.setSmoother(5, 6, 0.05, 0.1, 1.1)
    H.applyFilter(x, z)
    assert its <= 12 and H.lastSolve()[0] <= 12
    # both solves end at a residual of 1e-12 |b|
    np.testing.assert_allclose(y, z, rtol=0, atol=1e-9)


@pytest.mark.parametrize("dim,levels", [(3, 1), (3, 2), (2, 1), (2, 2)])
@pytest.mark.parametrize("r", [0.25, 2.0])
def test_large_radius_on_few_levels(gpu_lib, dim, levels, r):
    # a coarsest level of more than 2048 nodes, solved by sweeps, and r of many of
    # its elements: about the iterations of the longer smoother on every level (1.8
    # times as many with the shorter one there)
    from tmr_gb300 import TMR
    conn = W.brick(3, 2, 2) if dim == 3 else W.brick2d(8, 6)
    nb = len(conn)
    f = (TMR.OctForest if dim == 3 else TMR.QuadForest)(order=2)
    f.setConnectivity(conn)
    f.createTrees(4 if dim == 3 else 6)
    forests = [f]
    for _ in range(levels - 1):
        c = forests[-1].coarsen()
        c.balance(1)
        forests.append(c)
    for c in forests:
        c.createNodes()
        if dim == 3:
            c.setBlockBoxes(np.array([[b % 3, b // 3 % 2, b // 6, 1, 1, 1] for b in range(nb)],
                                     np.float64))
        else:
            c.setFaceBoxes(np.array([[b % 8, b // 8, 1, 1] for b in range(nb)], np.float64))
    assert int(forests[-1].getNodeRange()[1]) > 2048
    n = int(f.getNodeRange()[1])
    x = W.uniform(5, 0, n)
    H = TMR.HelmholtzFilter(r, None, forests)
    y, z = np.empty(n), np.empty(n)
    H.applyFilter(x, y)
    its = H.lastSolve()[0]
    H.setSmoother(5, 6, 0.05, 0.1, 1.1)
    H.applyFilter(x, z)
    assert its <= 1.3 * H.lastSolve()[0] + 1
    np.testing.assert_allclose(y, z, rtol=0, atol=1e-9)
