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


@pytest.mark.parametrize("nvec", [2, 5, 17])
@pytest.mark.parametrize("where", ["all", "first", "last", "inf"])
def test_values_outside_the_window_at_the_ends(operator, nvec, where):
    # values the (hi, lo) pairs do not hold everywhere, at the first or the last
    # input that is read, or one infinity: the whole result in FP64, infinite
    # where a row reads it
    import torch
    I, P = operator
    if P.nnz > 20 * P.shape[0]:
        pytest.skip("tiles that do not fit")
    rows, cols = P.shape
    T = P.T.tocsr()
    rng = np.random.default_rng(80 + nvec)
    one = np.asarray(T @ np.ones(rows))[:, None]
    # the column sums' own rounding and that of the weights in them
    sums = (np.diff(T.indptr)[:, None] + 4) * 2.0 ** -48 * np.asarray(abs(T) @ np.ones(rows))[:, None]
    sums = np.where(one == 0.0, 0.0, sums / np.where(one == 0.0, 1.0, abs(one)))
    one[one == 0.0] = np.inf
    for fn, A, scale, den in ((I.mult, P, 1.0, 0.0), (I.multTranspose, T, 1.0, 0.0),
                              (I.multWeightTranspose, T, one, sums)):
        x = rng.standard_normal((A.shape[1], nvec))
        read = np.unique(A.indices)
        if where == "all":
            x *= 1e-30
        else:
            i = (read[0], 0) if where == "first" else (read[-1], nvec - 1)
            x[i] = np.inf if where == "inf" else 1e-30
        want = (A @ np.where(np.isinf(x), 0.0, x)) / scale
        bound = (abs(A) @ np.where(np.isinf(x), 0.0, abs(x))) / abs(scale)
        # rounding of a row's products, its sum and the weights (2^-48 each)
        n = np.diff(A.indptr)[:, None]
        bound = bound * ((n + 4) * 2.0 ** -52 + 2.0 ** -47 + den) + 1e-300
        for shift in (0, 1):
            xd = torch.empty(x.size + shift, dtype=torch.float64, device="cuda")[shift:]
            xd.copy_(torch.from_numpy(x.reshape(-1)))
            y = torch.full((A.shape[0] * nvec + shift,), float("nan"), dtype=torch.float64,
                           device="cuda")[shift:]
            fn(xd, y)
            got = y.cpu().numpy().reshape(-1, nvec)
            fin = np.ones(got.shape, bool)
            if where == "inf":
                fin[:, nvec - 1] = np.asarray(A[:, read[-1]].todense())[:, 0] == 0.0
                if fn != I.multWeightTranspose:  # (a column of no weight gives 0)
                    assert not fin.all() and not np.isfinite(got[~fin]).any()
            assert np.all(np.abs(got - want)[fin] <= bound[fin])


def test_tile_applies_outside_the_window_take_no_second_apply(gpu_lib):
    # small values everywhere: a few times the double-float apply (2 to 4; 12
    # where it ran in full before a thread per row and vector)
    import time

    import torch

    from tmr_gb300 import TMR
    from tmr_gb300 import workloads as W
    f = TMR.OctForest(order=3)
    f.setConnectivity(W.brick(4, 4, 2))
    f.createTrees(2)
    for p in range(3):
        f.refine(W.random_indicator(f.getNumOctants(), 7, p, 0.3), 0, 9)
        f.balance(1)
    f.createNodes()
    c = f.coarsen()
    c.balance(1)
    c.createNodes()
    I = TMR.VecInterp()
    f.createInterpolation(c, I)
    rows, cols, _ = I.sizes()

    def best(fn, x, y):
        t = []
        for _ in range(7):
            torch.cuda.synchronize()
            a = time.perf_counter()
            for _ in range(10):
                fn(x, y)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - a)
        return min(t[2:])

    for nvec in (4, 16):
        for fn, nin, nout in ((I.mult, cols, rows), (I.multTranspose, rows, cols)):
            x = torch.randn(nin * nvec, dtype=torch.float64, device="cuda")
            y = torch.empty(nout * nvec, dtype=torch.float64, device="cuda")
            assert best(fn, x * 1e-20, y) <= 7 * best(fn, x, y)


def _refined(TMR, order, grid, depth, passes):
    from tmr_gb300 import workloads as W
    f = TMR.OctForest(order=order)
    f.setConnectivity(W.brick(*grid))
    f.createTrees(depth)
    for p in range(passes):
        f.refine(W.random_indicator(f.getNumOctants(), 7, p, 0.3), 0, 9)
        f.balance(1)
    f.createNodes()
    c = f.coarsen()
    c.balance(1)
    c.createNodes()
    I = TMR.VecInterp()
    f.createInterpolation(c, I)
    return I


@pytest.mark.parametrize("grid", [(2, 2, 2), (4, 3, 2), (4, 4, 4)])
def test_host_buffers_of_any_count_equal_device_buffers(gpu_lib, grid):
    # one, two and more pieces; pageable and page-locked buffers; and values
    # that send the apply to FP64, from the first or the last piece on
    import torch

    from tmr_gb300 import TMR
    I = _refined(TMR, 2, grid, 3, 2)
    rows, cols, _ = I.sizes()
    for nvec in (2, 3, 4, 9, 16, 17, 18):
        for fn, nin, nout in ((I.mult, cols, rows), (I.multTranspose, rows, cols),
                              (I.multWeightTranspose, rows, cols)):
            for where in (None, 0, -1):
                x = np.random.default_rng(nvec).standard_normal(nin * nvec)
                if where is not None:
                    x[where] = 1e-30
                y = torch.empty(nout * nvec, dtype=torch.float64, device="cuda")
                fn(torch.from_numpy(x).cuda(), y)
                want = y.cpu().numpy()
                got = np.full(nout * nvec, np.nan)
                fn(x, got)
                pin = torch.full((nout * nvec,), float("nan"), dtype=torch.float64).pin_memory()
                fn(torch.from_numpy(x).pin_memory().numpy(), pin.numpy())
                for a in (got, pin.numpy()):
                    if where is None:
                        np.testing.assert_array_equal(a, want)
                    else:
                        # pieces before the value stay double-float
                        np.testing.assert_allclose(a, want, rtol=1e-13, atol=1e-13)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("grid", [(6, 4, 4), (8, 8, 4)])
def test_host_buffers_in_pieces(gpu_lib, grid, pinned):
    # two and seven pieces: input and output apart, and the output over the
    # input, from the buffer's start or to its end
    import torch

    from tmr_gb300 import TMR
    I = _refined(TMR, 2, grid, 3, 2)
    rows, cols, _ = I.sizes()
    assert rows >= 2 * 4 * 152 * 256

    def host(n):
        a = torch.zeros(n, dtype=torch.float64)
        return (a.pin_memory() if pinned else a).numpy()

    for nvec in (2, 16):
        for fn, nin, nout in ((I.mult, cols, rows), (I.multTranspose, rows, cols),
                              (I.multWeightTranspose, rows, cols)):
            x = np.random.default_rng(nvec).standard_normal(nin * nvec)
            for where in (None, 0, -1):
                if where is not None:
                    x[where] = 1e-30
                y = torch.empty(nout * nvec, dtype=torch.float64, device="cuda")
                fn(torch.from_numpy(x).cuda(), y)
                want = y.cpu().numpy()
                n = max(nin, nout) * nvec
                for at in (n, 0, n - nout * nvec):
                    both = host(n + (nout * nvec if at == n else 0))
                    both[:nin * nvec] = x
                    got = both[at:at + nout * nvec]
                    fn(both[:nin * nvec], got)
                    if where is None:
                        np.testing.assert_array_equal(got, want)
                    else:
                        # pieces before the value stay double-float
                        np.testing.assert_allclose(got, want, rtol=1e-13, atol=1e-13)


def test_page_locked_odd_counts_cost_what_even_ones_do(gpu_lib):
    # 3 vectors into page-locked memory: no more than 4 (twice as much where the
    # rows went over the link in order of length)
    import time

    import torch

    from tmr_gb300 import TMR
    I = _refined(TMR, 2, (4, 4, 4), 3, 3)
    rows, cols, _ = I.sizes()
    t = {}
    for nvec in (3, 4):
        x = torch.randn(cols * nvec, dtype=torch.float64).pin_memory().numpy()
        y = torch.empty(rows * nvec, dtype=torch.float64).pin_memory().numpy()
        best = []
        for _ in range(12):
            a = time.perf_counter()
            I.mult(x, y)
            best.append(time.perf_counter() - a)
        t[nvec] = min(best[4:])
    assert t[3] <= 1.3 * t[4]


def test_rows_too_long_for_any_tile_are_sorted_at_once(gpu_lib):
    # quartic elements: over 32 entries a row, which no tile holds; the tiles
    # are not tried
    import ctypes
    import json

    from tmr_gb300 import TMR
    from tmr_gb300 import workloads as W
    f = TMR.OctForest(order=4)
    f.setConnectivity(W.brick(3, 2, 2))
    f.createTrees(1)
    for p in range(2):
        f.refine(W.random_indicator(f.getNumOctants(), 7, p, 0.3), 0, 9)
        f.balance(1)
    f.createNodes()
    c = f.coarsen()
    c.balance(1)
    c.createNodes()
    I = TMR.VecInterp()
    lib = TMR.lib()
    lib.tmrg_profile_begin()
    f.createInterpolation(c, I)
    buf = ctypes.create_string_buffer(1 << 20)
    assert lib.tmrg_profile_end(buf, len(buf)) == 0
    rows, cols, nnz = I.sizes()
    assert I.applyNnz() > 32 * rows
    assert not [k for k in json.loads(buf.value.decode()) if "k_tb_build" in k]
