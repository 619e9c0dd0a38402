"""The Helmholtz filter's solver with K on tiles: vector counts, smoother
degrees, a coarsest level too large for the dense inverse, and one filter used
with changing vector counts.  K and M themselves are checked against the
oracle in test_gpu_helmholtz.py; here the solutions' residuals are."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _filter(TMR, dim, levels, depth=2, passes=2):
    if dim == 3:
        f = TMR.OctForest(order=2)
        f.setConnectivity(W.rotate_blocks(W.brick(3, 2, 2), 6))
        boxes = np.array([[i, j, k, 1.0, 1.0, 1.0] for k in range(2) for j in range(2)
                          for i in range(3)])
    else:
        f = TMR.QuadForest(order=2)
        f.setConnectivity(W.brick2d(4, 3))
        boxes = np.array([[i, j, 1.0, 1.0] for j in range(3) for i in range(4)])
    f.createTrees(depth)
    for p in range(passes):
        n = f.getNumOctants() if dim == 3 else f.getNumQuadrants()
        f.refine(W.random_indicator(n, 9, p, 0.25), 0, 6)
        f.balance(1)
    f.createNodes()
    fs = [f]
    for _ in range(levels - 1):
        c = fs[-1].coarsen()
        c.balance(1)
        c.createNodes()
        fs.append(c)
    for c in fs:
        (c.setBlockBoxes if dim == 3 else c.setFaceBoxes)(boxes)
    return TMR.HelmholtzFilter(0.15, None, fs)


def _solves(H, vpn, seed):
    """|K y - M x| / |M x| of the filter and, for the adjoint y = M psi, the
    solve's residual through the symmetry <K^-1 M x, w> = <x, M K^-1 w>."""
    import torch
    n = int(H.sizes()[0][0])
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(n * vpn, dtype=torch.float64, device="cuda", generator=g)
    w = torch.randn(n * vpn, dtype=torch.float64, device="cuda", generator=g)
    y, a = torch.empty_like(x), torch.empty_like(x)
    H.applyFilter(x, y, vpn)
    H.applyTranspose(w, a, vpn)
    Ky, Mx = torch.empty_like(x), torch.empty_like(x)
    H.mult(0, 0, y, Ky, vpn)
    H.mult(0, 1, x, Mx, vpn)
    r = (Ky - Mx).reshape(n, vpn).norm(dim=0) / Mx.reshape(n, vpn).norm(dim=0)
    dots = torch.stack([(y * w).reshape(n, vpn).sum(0), (x * a).reshape(n, vpn).sum(0)])
    scale = y.reshape(n, vpn).norm(dim=0) * w.reshape(n, vpn).norm(dim=0)
    return float(r.max()), float(((dots[0] - dots[1]).abs() / scale).max())


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("vpn", [1, 2, 4, 5, 9])
def test_vector_counts(gpu_lib, dim, vpn):
    from tmr_gb300 import TMR
    r, s = _solves(_filter(TMR, dim, 3), vpn, 3)
    # the solver stops at a residual of 1e-12 |b|; K is applied again here
    assert r <= 2e-12 and s <= 1e-11


@pytest.mark.parametrize("degree", [1, 2, 3, 6])
@pytest.mark.parametrize("levels", [1, 2, 3])
def test_degrees_and_coarsest_levels(gpu_lib, degree, levels):
    # 1 level: no smoother but the coarsest solve, of more than 2048 nodes
    from tmr_gb300 import TMR
    H = _filter(TMR, 3, levels, depth=3, passes=1)
    assert int(H.sizes()[0][0]) > 2048 and int(H.sizes()[0][0]) % 256 != 0
    H.setSmoother(degree_order2=degree, lower_order2=0.2)
    r, s = _solves(H, 2, 4)
    assert r <= 2e-12 and s <= 1e-11


def test_vector_counts_in_turn(gpu_lib):
    # the work vectors grow and shrink in use between the calls
    from tmr_gb300 import TMR
    H = _filter(TMR, 3, 3)
    first = {}
    for vpn in (1, 3, 2, 5, 1, 4, 3):
        r, s = _solves(H, vpn, 10 + vpn)
        assert r <= 2e-12 and s <= 1e-11
        assert first.setdefault(vpn, (r, s)) == (r, s)  # the same bits again


@pytest.mark.parametrize("vpn,k", [(1, 1533), (1, 1534), (1, 1535), (2, 766), (2, 767), (2, 768)])
def test_largest_tile_about_the_shared_memory_limit(gpu_lib, vpn, k):
    # k blocks around an edge: every node is a column of the first tile, and
    # its FP64 inputs with the sums beside them end just below, at and above
    # 48 KB (4 k + 2 columns of 8 vpn bytes, and 64 bytes)
    from tests.test_gpu_filter_rows import _fan
    from tmr_gb300 import TMR
    f = TMR.OctForest(order=2)
    f.setConnectivity(_fan(k))
    f.createTrees(0)
    f.createNodes()
    n = int(f.getNodeRange()[1])
    assert n == 4 * k + 2 and abs(8 * vpn * n + 64 - 48 * 1024) < 150
    f.setBlockBoxes(np.tile([0.0, 0.0, 0.0, 1.0, 1.0, 1.0], (k, 1)))
    r, s = _solves(TMR.HelmholtzFilter(0.3, None, [f]), vpn, 6)
    assert r <= 2e-12 and s <= 1e-11


@pytest.mark.parametrize("vpn", [1, 3])
@pytest.mark.parametrize("level", [0, 1])
def test_operators_in_place(gpu_lib, vpn, level):
    # K x and M x written over x
    import torch

    from tmr_gb300 import TMR
    H = _filter(TMR, 3, 2)
    n = int(H.sizes()[level][0])
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(n * vpn, dtype=torch.float64, device="cuda", generator=g)
    for which in (0, 1):
        want = torch.empty_like(x)
        H.mult(level, which, x, want, vpn)
        same = x.clone()
        H.mult(level, which, same, same, vpn)
        assert torch.equal(same, want)
