"""P and P^T built and applied by tiles of rows: ragged last tiles, matrices whose
tiles need the larger table or do not fit, more (tile, column) pairs than rows,
vector counts around the lanes' groups, against FP64 products of P's entries."""
import numpy as np
import pytest

from tests import pipeline

pytestmark = pytest.mark.gpu


def _operator(order, coarse_order):
    import scipy.sparse as sp

    import bench
    from tmr_gb300 import TMR
    case = dict(bench.cpu_sample_case(), coarse_levels=1, order=order)
    if coarse_order == order:
        case["passes"] += {2: 1, 3: 0, 4: -1, 5: -1}[order]
    g = pipeline.run_gpu(case)
    fine, I = g["forests"][0], g["levels"][0]["I"]
    if coarse_order != order:
        coarse = g["forests"][1].duplicate()
        coarse.setMeshOrder(coarse_order)
        coarse.createNodes()
        I = TMR.VecInterp()
        fine.createInterpolation(coarse, I)
    rp, c, w = I.getCSR()
    rows, cols, _ = I.sizes()
    P = sp.csr_matrix((w, c, rp), shape=(rows, cols))
    # the applies leave out P's numerically-zero weights
    P.data[abs(P.data) < 2.0 ** -40] = 0.0
    P.eliminate_zeros()
    assert I.applyNnz() in (P.nnz, len(w))
    return I, P


@pytest.fixture(scope="module", params=[(2, 2), (3, 3), (4, 4), (5, 5), (2, 4)],
                ids=lambda o: "order%d_from%d" % o)
def operator(request, gpu_lib):
    return _operator(*request.param)


def _bound(A, x):
    # a row of n entries: 2^-48 of each product from the parts left out and the
    # split, and 2^-46 of the running sum for each addition in (hi, lo)
    n = np.diff(A.indptr)[:, None]
    return (n + 4) * 2.0 ** -46 * (abs(A) @ abs(x)) + 1e-300


@pytest.mark.parametrize("nvec", [2, 3, 4, 5, 8, 9, 16, 17])
def test_tile_applies(operator, nvec):
    import torch
    I, P = operator
    rows, cols = P.shape
    if I.applyNnz() * nvec <= 1_000_000:
        pytest.skip("few entries: one FP64 kernel")
    T = P.T.tocsr()
    rng = np.random.default_rng(nvec)
    one = np.asarray(T @ np.ones(rows))[:, None]
    one[one == 0.0] = np.inf  # a column of no weight gives 0
    for fn, A, scale in ((I.mult, P, 1.0), (I.multTranspose, T, 1.0),
                         (I.multWeightTranspose, T, one)):
        x = rng.standard_normal((A.shape[1], nvec))
        y = torch.full((A.shape[0] * nvec + 1,), float("nan"), dtype=torch.float64, device="cuda")
        xd = torch.from_numpy(x.reshape(-1)).cuda()
        for shift in (0, 1):  # on and off the 16-byte grid
            out = y[shift:shift + A.shape[0] * nvec]
            fn(xd, out)
            got = out.cpu().numpy().reshape(-1, nvec)
            assert np.all(abs(got - (A @ x) / scale) <= _bound(A, x) / abs(scale))


def test_tile_applies_outside_the_window(operator):
    # one input the pairs do not hold, in the middle: the FP64 kernels
    import torch
    I, P = operator
    for fn, A in ((I.mult, P), (I.multTranspose, P.T.tocsr())):
        x = np.random.default_rng(5).standard_normal((A.shape[1], 16))
        x[A.shape[1] // 2, 7] = 1e30
        y = torch.empty(A.shape[0] * 16, dtype=torch.float64, device="cuda")
        xd = torch.from_numpy(x.reshape(-1)).cuda()
        fn(xd, y)
        assert np.all(abs(y.cpu().numpy().reshape(-1, 16) - A @ x) <= _bound(A, x))


def test_host_buffers_equal_device_buffers(operator):
    import torch
    I, P = operator
    if P.nnz > 20 * P.shape[0]:
        pytest.skip("tiles that do not fit: row kernels, whose shape is tuned by call")
    for fn, nin, nout in ((I.mult, P.shape[1], P.shape[0]), (I.multTranspose, *P.shape)):
        x = np.random.default_rng(6).standard_normal(nin * 16)
        yh = np.zeros(nout * 16)
        fn(x, yh)
        y = torch.empty(nout * 16, dtype=torch.float64, device="cuda")
        xd = torch.from_numpy(x).cuda()
        fn(xd, y)
        np.testing.assert_array_equal(yh, y.cpu().numpy())
