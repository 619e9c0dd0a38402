"""P, P^T and the weight-normalised P^T for the vector counts whose kernels
differ (one vector, few on a small matrix, odd counts, buffers off the
16-byte grid), against FP64 products of P's own entries."""
import numpy as np
import pytest

from tests import pipeline

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def operators(gpu_lib):
    import bench
    from tmr_gb300 import TMR  # noqa: F401
    small = pipeline.run_gpu(dict(pipeline.cases()["rot_o2"], coarse_levels=1))
    large = pipeline.run_gpu(dict(bench.cpu_sample_case(), coarse_levels=1))
    out = {}
    for name, g in (("small", small), ("large", large)):
        I = g["levels"][0]["I"]
        import scipy.sparse as sp
        rp, c, w = I.getCSR()
        rows, cols, _ = I.sizes()
        out[name] = (I, sp.csr_matrix((w, c, rp), shape=(rows, cols)))
    assert out["small"][0].applyNnz() * 8 < 1_000_000 < out["large"][0].applyNnz()
    return out


def _on_device(a, shift):
    """a in a CUDA buffer that starts `shift` doubles past an aligned one."""
    import torch
    t = torch.empty(a.size + shift, dtype=torch.float64, device="cuda")[shift:]
    t.copy_(torch.from_numpy(a.reshape(-1)))
    return t


@pytest.mark.parametrize("size,nvec,shift", [
    ("large", 1, 0), ("large", 1, 1), ("small", 1, 0), ("small", 2, 0), ("small", 2, 1),
    ("small", 3, 0), ("small", 4, 1), ("small", 5, 0), ("small", 7, 0), ("small", 8, 0)])
def test_applies_match_fp64_products(operators, size, nvec, shift):
    import torch
    I, P = operators[size]
    rows, cols = P.shape
    rng = np.random.default_rng(nvec)
    xc, xf = rng.standard_normal((cols, nvec)), rng.standard_normal((rows, nvec))
    one = np.asarray(P.T @ np.ones(rows))[:, None]
    want = (P @ xc, P.T @ xf, (P.T @ xf) / one)
    xcd, xfd = _on_device(xc, shift), _on_device(xf, shift)
    for fn, x, ref in ((I.mult, xcd, want[0]), (I.multTranspose, xfd, want[1]),
                       (I.multWeightTranspose, xfd, want[2])):
        y = torch.empty(ref.size + shift, dtype=torch.float64, device="cuda")[shift:]
        y.fill_(float("nan"))
        fn(x, y)
        # the applies' bar: 1e-13 of max(1, |y|)
        np.testing.assert_allclose(y.cpu().numpy(), ref.reshape(-1), rtol=1e-13, atol=1e-13)


@pytest.mark.parametrize("nvec,shift", [(2, 1), (3, 0), (3, 1), (5, 0), (7, 0), (9, 0), (15, 0),
                                        (16, 1), (17, 0)])
@pytest.mark.parametrize("shape", [0, 1, 4, 6])
def test_odd_and_unaligned_vectors_equal_whole_pairs(operators, nvec, shift, shape):
    # the same vectors with a zero one beside them, on the 16-byte grid, at
    # the same forced launch shape: the same bits
    import torch

    from tmr_gb300 import TMR
    I, P = operators["large"]
    rows, cols = P.shape
    even = nvec + nvec % 2
    if even // 2 < 8 and shape > 1:
        pytest.skip("shapes of 8 or more pairs")
    if shape == 6 and even == 16:
        shape = 4  # the staged kernel is for aligned pairs and equals shape 4
    rng = np.random.default_rng(nvec)
    lib = TMR.lib()
    try:
        assert lib.tmrg_tune_force(1, shape) == 0 and lib.tmrg_tune_force(2, shape) == 0
        for fn, nin, nout in ((I.mult, cols, rows), (I.multTranspose, rows, cols),
                              (I.multWeightTranspose, rows, cols)):
            x = rng.standard_normal((nin, nvec))
            y = torch.empty(nout * nvec + shift, dtype=torch.float64, device="cuda")[shift:]
            fn(_on_device(x, shift), y)
            xe = np.zeros((nin, even))
            xe[:, :nvec] = x
            ye = torch.empty(nout * even, dtype=torch.float64, device="cuda")
            fn(_on_device(xe, 0), ye)
            assert torch.equal(y.reshape(nout, nvec), ye.reshape(nout, even)[:, :nvec])
    finally:
        lib.tmrg_tune_force(1, -1)
        lib.tmrg_tune_force(2, -1)


@pytest.mark.parametrize("size", ["small", "large"])
@pytest.mark.parametrize("nvec", [1, 3, 9])
def test_applies_outside_the_window(operators, size, nvec):
    # values the double-float pairs do not hold: the FP64 branches
    import torch
    I, P = operators[size]
    rows, cols = P.shape
    rng = np.random.default_rng(40 + nvec)
    for scale in (1e-30, 1e25):
        for fn, A in ((I.mult, P), (I.multTranspose, P.T)):
            x = rng.standard_normal((A.shape[1], nvec)) * scale
            y = torch.empty(A.shape[0] * nvec, dtype=torch.float64, device="cuda")
            fn(_on_device(x, 0), y)
            np.testing.assert_allclose(y.cpu().numpy().reshape(-1, nvec) / scale,
                                       (A @ x) / scale, rtol=1e-13, atol=1e-13)


@pytest.mark.parametrize("size", ["small", "large"])
@pytest.mark.parametrize("nvec", [1, 2, 3, 8, 9, 16])
@pytest.mark.parametrize("shift", [0, 3])
def test_input_and_output_in_one_buffer(operators, size, nvec, shift):
    # the output written over the input, from its start or a few values on
    import torch
    I, P = operators[size]
    rows, cols = P.shape
    rng = np.random.default_rng(60 + nvec)
    for scale in (1.0, 1e-30):
        for fn, nin, nout in ((I.mult, cols, rows), (I.multTranspose, rows, cols),
                              (I.multWeightTranspose, rows, cols)):
            x = _on_device(rng.standard_normal(nin * nvec) * scale, 0)
            want = torch.empty(nout * nvec, dtype=torch.float64, device="cuda")
            fn(x, want)
            both = torch.zeros(max(nin, nout) * nvec + shift, dtype=torch.float64, device="cuda")
            both[:nin * nvec] = x
            got = both[shift:shift + nout * nvec]
            fn(both[:nin * nvec], got)
            # an unaligned output may take another launch shape
            assert torch.equal(got, want) if shift == 0 else torch.allclose(
                got, want, rtol=0, atol=1e-13 * scale * 8)


def test_unaligned_vectors_are_tuned_by_themselves(operators):
    # vectors off the 16-byte grid run other kernels: a class of their own
    import ctypes
    import json

    import torch

    from tmr_gb300 import TMR
    I, P = operators["large"]
    rows, cols = P.shape
    lib = TMR.lib()
    assert lib.tmrg_tune_reset(1) == 0
    try:
        x = np.random.default_rng(3).standard_normal(rows * 2)
        for shift in (1, 0, 1):
            y = torch.empty(cols * 2 + shift, dtype=torch.float64, device="cuda")[shift:]
            I.multTranspose(_on_device(x, shift), y)
        buf = ctypes.create_string_buffer(1 << 16)
        assert lib.tmrg_tune_report(buf, len(buf)) == 0
        keys = [tuple(e["key"]) for e in json.loads(buf.value.decode()) if e["kind"] == 2]
        assert len(keys) == 2 and len({k[:2] for k in keys}) == 1
    finally:
        lib.tmrg_tune_reset(1)


def _applied(P):
    """P without the numerically-zero weights, which the applies leave out."""
    P = P.copy()
    P.data[abs(P.data) < 2.0 ** -40] = 0.0
    P.eliminate_zeros()
    return P


@pytest.mark.parametrize("nvec", [2, 3, 4, 5, 6, 7, 8, 9, 14])
@pytest.mark.parametrize("shape", [0, 1, 2, 3])
def test_narrow_launch_shapes(operators, nvec, shape):
    # one to seven pairs, all at once in one to eight groups of lanes
    import torch

    from tests.test_gpu_apply_tiles import _bound
    from tmr_gb300 import TMR
    I, P = operators["large"]
    P = _applied(P)
    rng = np.random.default_rng(70 + nvec)
    lib = TMR.lib()
    try:
        assert lib.tmrg_tune_force(1, shape) == 0 and lib.tmrg_tune_force(2, shape) == 0
        for fn, A in ((I.mult, P), (I.multTranspose, P.T.tocsr())):
            x = rng.standard_normal((A.shape[1], nvec))
            for shift in (0, 1):
                y = torch.full((A.shape[0] * nvec + shift,), float("nan"), dtype=torch.float64,
                               device="cuda")[shift:]
                fn(_on_device(x, shift), y)
                assert np.all(abs(y.cpu().numpy().reshape(-1, nvec) - A @ x) <= _bound(A, x))
    finally:
        lib.tmrg_tune_force(1, -1)
        lib.tmrg_tune_force(2, -1)


@pytest.mark.parametrize("size", ["small", "large"])
@pytest.mark.parametrize("nvec", [9, 15, 16, 17, 24, 31, 33])
def test_counts_beyond_eight(operators, size, nvec):
    # the FP64 rows in parts, and nine or more pairs at once
    import torch

    from tests.test_gpu_apply_tiles import _bound
    I, P = operators[size]
    P = _applied(P)
    rng = np.random.default_rng(90 + nvec)
    one = np.asarray(P.T @ np.ones(P.shape[0]))[:, None]
    for fn, A, s in ((I.mult, P, 1.0), (I.multTranspose, P.T.tocsr(), 1.0),
                     (I.multWeightTranspose, P.T.tocsr(), one)):
        x = rng.standard_normal((A.shape[1], nvec))
        y = torch.full((A.shape[0] * nvec,), float("nan"), dtype=torch.float64, device="cuda")
        fn(_on_device(x, 0), y)
        assert np.all(abs(y.cpu().numpy().reshape(-1, nvec) - (A @ x) / s) <= _bound(A, x) / s)


def test_few_long_rows_cost_no_more_for_odd_counts(gpu_lib):
    # P^T of quartic elements, 160 entries a row: 5 vectors within twice 4 (2.3
    # times where the pairs were taken two at a time by two lanes)
    import time

    import torch

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
    f.createInterpolation(c, I)
    rows, cols, _ = I.sizes()
    t = {}
    for nvec in (4, 5):
        x = torch.randn(rows * nvec, dtype=torch.float64, device="cuda")
        y = torch.empty(cols * nvec, dtype=torch.float64, device="cuda")
        best = []
        for _ in range(8):
            torch.cuda.synchronize()
            a = time.perf_counter()
            for _ in range(20):
                I.multTranspose(x, y)
            torch.cuda.synchronize()
            best.append(time.perf_counter() - a)
        t[nvec] = min(best[2:])
    assert t[5] <= 2 * t[4] and t[5] < 20 * 250e-6
