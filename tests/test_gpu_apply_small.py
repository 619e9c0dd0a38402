"""P and P^T of many vectors on matrices with fewer tiles than SMs and on one
with more, against 64-bit products of the same P."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [2, 3, 4])
@pytest.mark.parametrize("nvec", [9, 14, 15, 16, 17])
def test_many_vectors_on_either_side_of_the_line(gpu_lib, depth, nvec):
    from tmr_gb300 import TMR
    f = TMR.OctForest(order=2)
    f.setConnectivity(W.brick(3, 2, 2))
    f.createTrees(depth)
    f.refine(W.random_indicator(f.getNumOctants(), 3, 0, 0.3), 0, 6)
    f.balance(1)
    f.createNodes()
    c = f.coarsen()
    c.balance(1)
    c.createNodes()
    I = TMR.VecInterp()
    f.createInterpolation(c, I)
    rows, cols, _ = I.sizes()
    assert (rows < 152 * 256) == (depth < 4)
    ptr, ci, w = I.getCSR()
    ri = np.repeat(np.arange(rows), np.diff(ptr))
    xc = W.uniform(1, 0, cols * nvec).reshape(cols, nvec) - 0.5
    xf = W.uniform(2, 0, rows * nvec).reshape(rows, nvec) - 0.5
    up, down = np.zeros((rows, nvec)), np.zeros((cols, nvec))
    np.add.at(up, ri, w[:, None] * xc[ci])
    np.add.at(down, ci, w[:, None] * xf[ri])
    s = np.zeros(cols)
    np.add.at(s, ci, w)
    y, z, m = np.empty(rows * nvec), np.empty(cols * nvec), np.empty(cols * nvec)
    I.mult(xc.reshape(-1), y)
    I.multTranspose(xf.reshape(-1), z)
    I.multWeightTranspose(xf.reshape(-1), m)
    # the applies' stated error is 3e-14 of the largest value; sums of |w| up to 8
    np.testing.assert_allclose(y.reshape(rows, nvec), up, rtol=0, atol=1e-13)
    np.testing.assert_allclose(z.reshape(cols, nvec), down, rtol=0, atol=4e-13)
    np.testing.assert_allclose(m.reshape(cols, nvec), down / s[:, None], rtol=0, atol=1e-13)
