"""Quadtree rows of P from the direction-state table and outside it."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 3])
@pytest.mark.parametrize("gap", [1, 2, 0])
def test_quad_rows_reproduce_polynomials(gpu_lib, order, gap):
    # P takes the nodal values of a polynomial that the coarse elements hold
    # to those on the fine nodes.  gap: coarsenings between the forests (2:
    # levels too far apart for the table); 0: two forests refined at random,
    # each finer than the other in places
    from tmr_gb300 import TMR
    nx, ny = 5, 3
    conn = W.brick2d(nx, ny)
    box = np.array([[b % nx, b // nx, 1, 1] for b in range(nx * ny)], np.float64)

    def refined(seed):
        f = TMR.QuadForest(order=order, interp=TMR.GAUSS_LOBATTO_POINTS)
        f.setConnectivity(conn)
        f.createTrees(2)
        for p in range(3):
            f.refine(W.random_indicator(f.getNumQuadrants(), seed, p, 0.3), 0, 6)
            f.balance(1)
        f.createNodes()
        return f

    fine = refined(3)
    coarse = refined(4) if gap == 0 else fine
    for _ in range(gap):
        coarse = coarse.coarsen()
        coarse.balance(1)
    coarse.createNodes()
    P = TMR.VecInterp()
    fine.createInterpolation(coarse, P)
    vals = []
    for f in (fine, coarse):
        f.setFaceBoxes(box)
        X = f.getPoints()[int(f.getExtPreOffset()):]
        x, y = X[:, 0] / nx, X[:, 1] / ny
        vals.append(np.stack([1.0 + x - 2.0 * y + 0.5 * x * y,
                              (x * x - x * y + y * y * x) if order == 3 else y], 1).copy())
    rows, cols, _ = P.sizes()
    assert vals[0].shape == (rows, 2) and vals[1].shape == (cols, 2)
    y = np.empty(rows * 2)
    P.mult(vals[1].reshape(-1), y)
    # at most 27 products a row; values up to 4, weights sum up to 1.25^4 in size
    np.testing.assert_allclose(y.reshape(rows, 2), vals[0], rtol=0, atol=2e-13)
