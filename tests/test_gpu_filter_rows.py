"""The mass matrix assembled row by row, against a dense assembly from the
forest's own connectivity: a node shared by many blocks (rows larger than
the tables of the first attempts), hanging nodes, and a block size so small
that no entry is taken from the unit block's."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _fan(k):
    """k hexahedra around one edge: node 0 (and 0 + layer) on the axis, then
    2k nodes of the rim per layer."""
    layer = 2 * k + 1
    conn = []
    for i in range(k):
        a, b, c = 1 + 2 * i, 2 + 2 * i, 1 + (2 * i + 2) % (2 * k)
        conn.append([0, a, c, b, layer, layer + a, layer + c, layer + b])
    return np.array(conn, np.intc)


def _mass(f, dim, n, block_len):
    """Dense M, element by element, dependent nodes through their rows."""
    conn = f.getMeshConn()
    ptr, dc, dw = f.getDepNodeConn()
    lev = f.getOctantsArray()[:, 5] if dim == 3 else f.getQuadrantsArray()[:, 4]
    m1 = np.array([[2.0, 1.0], [1.0, 2.0]]) / 6.0
    ref = m1
    for _ in range(dim - 1):
        ref = np.kron(m1, ref)
    M = np.zeros((n, n))
    for e, c in enumerate(conn):
        S = np.zeros((len(c), n))
        for a, g in enumerate(c):
            if g >= 0:
                S[a, g] = 1.0
            else:
                r = slice(ptr[-g - 1], ptr[-g])
                np.add.at(S[a], dc[r], dw[r])
        M += (block_len * 0.5 ** lev[e]) ** dim * (S.T @ ref @ S)
    return M


def _check(F, M):
    rp, c, v, _, _, _ = F.getMatrix()
    n = len(rp) - 1
    got = np.zeros((n, n))
    for i in range(n):
        cols = c[rp[i]:rp[i + 1]]
        assert np.all(np.diff(cols) > 0)
        got[i, cols] = v[rp[i]:rp[i + 1]]
    # sums of at most a few thousand products
    np.testing.assert_allclose(got, M, rtol=1e-12, atol=1e-15 * np.abs(M).max())


@pytest.mark.parametrize("k", [7, 100, 300])
def test_rows_of_a_node_in_many_blocks(gpu_lib, k):
    from tmr_gb300 import TMR
    f = TMR.OctForest(order=2)
    f.setConnectivity(_fan(k))
    f.createTrees(0)
    f.createNodes()
    n = int(f.getNodeRange()[1])
    assert n == 2 * (2 * k + 1)
    F = TMR.MatrixFilter(0.5, 3, None, [f])
    _check(F, _mass(f, 3, n, 1.0))


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("block_len", [1.0, 0.7, 1e-60, 1e-98])
def test_rows_with_hanging_nodes(gpu_lib, dim, block_len):
    from tmr_gb300 import TMR
    if dim == 3:
        f = TMR.OctForest(order=2)
        f.setConnectivity(W.rotate_blocks(W.brick(2, 2, 1), 4))
    else:
        f = TMR.QuadForest(order=2)
        f.setConnectivity(W.brick2d(3, 2))
    f.createTrees(1)
    for p in range(3):
        n = f.getNumOctants() if dim == 3 else f.getNumQuadrants()
        f.refine(W.random_indicator(n, 5, p, 0.25), 0, 5)
        f.balance(1)
    f.createNodes()
    n = int(f.getNodeRange()[1])
    F = TMR.MatrixFilter(0.1 * block_len, 3, None, [f], block_len=block_len)
    _check(F, _mass(f, dim, n, block_len))


def _horner(F, N, x, transpose):
    import scipy.sparse as sp
    rp, c, v, A, B, T = F.getMatrix()
    n = len(rp) - 1
    M = sp.csr_matrix((v, c, rp), shape=(n, n))
    A, B, T = A[:, None], B[:, None], T[:, None]
    if not transpose:
        t1 = A * x
        y = t1
        for _ in range(N):
            y = B * (M @ y) + t1
        return T * y
    t1 = T * x
    y = t1
    for _ in range(N):
        y = M @ (B * y) + t1
    return A * y


def _random_filter(TMR, N):
    f = TMR.OctForest(order=2)
    f.setConnectivity(W.rotate_blocks(W.brick(2, 2, 1), 4))
    f.createTrees(1)
    for p in range(3):
        f.refine(W.random_indicator(f.getNumOctants(), 5, p, 0.25), 0, 5)
        f.balance(1)
    f.createNodes()
    return TMR.MatrixFilter(0.1, N, None, [f])


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("N,vpn", [(0, 2), (1, 1), (2, 3), (3, 2), (4, 4), (5, 5), (3, 7), (10, 3)])
def test_terms_of_tiles_match_horner(gpu_lib, dtype, N, vpn):
    # apart, in place and overlapping by one row; rounding of N + 1 terms of
    # about 30 products each
    import torch

    from tmr_gb300 import TMR
    F = _random_filter(TMR, N)
    n = F.size()[0]
    assert n % 256 != 0 and n > 512
    rng = np.random.default_rng(N)
    tol = (1e-13 if dtype == "float64" else 4e-6)
    for transpose in (False, True):
        x = rng.uniform(0.0, 1.0, (n, vpn))
        want = _horner(F, N, x.astype(dtype).astype(np.float64), transpose)
        xd = torch.from_numpy(x.reshape(-1)).cuda().to(getattr(torch, dtype))
        apply = F.applyTranspose if transpose else F.applyFilter
        y = torch.empty_like(xd)
        apply(xd, y, vpn)
        got = y.cpu().numpy().astype(np.float64).reshape(n, vpn)
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
        same = xd.clone()
        apply(same, same, vpn)
        assert torch.equal(same, y)
        both = torch.zeros((n + 1) * vpn, dtype=xd.dtype, device="cuda")
        both[: n * vpn] = xd
        apply(both[: n * vpn], both[vpn:], vpn)
        assert torch.equal(both[vpn:], y)


def test_terms_of_a_tile_with_too_many_columns(gpu_lib):
    # a node in 2000 blocks: its row alone has 8002 columns, more than a tile
    # may have, and the sliced copy runs
    import torch

    from tmr_gb300 import TMR
    f = TMR.OctForest(order=2)
    f.setConnectivity(_fan(2000))
    f.createTrees(0)
    f.createNodes()
    F = TMR.MatrixFilter(0.5, 4, None, [f])
    n = F.size()[0]
    rng = np.random.default_rng(2)
    for vpn in (1, 3):
        for transpose in (False, True):
            x = rng.uniform(0.0, 1.0, (n, vpn))
            want = _horner(F, 4, x, transpose)
            y = torch.empty(n * vpn, dtype=torch.float64, device="cuda")
            (F.applyTranspose if transpose else F.applyFilter)(
                torch.from_numpy(x.reshape(-1)).cuda(), y, vpn)
            assert np.abs(y.cpu().numpy().reshape(n, vpn) - want).max() <= (
                1e-12 * np.abs(want).max())


def _fan_forest(TMR, k, extra):
    """k blocks around an edge, and `extra` beside them: 8 uniform blocks of
    4096 octants, which take the matrix over the line to the row assembly."""
    from tests.test_gpu_balance_paths import _union
    f = TMR.OctForest(order=2)
    f.setConnectivity(_union([_fan(k), W.brick(2, 2, 2)]) if extra else _fan(k))
    f.createTrees(0)
    for _ in range(4 if extra else 0):
        f.refine((f.getOctantsArray()[:, 0] >= k).astype(np.intc), 0, 4)
        f.balance(1)
    f.createNodes()
    assert (f.getNumOctants() * 64 > 2_000_000) == extra
    return f


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("k", [7, 100, 300, 2040, 2047, 2048, 2100])
def test_rows_of_more_columns_than_any_table(gpu_lib, k, extra):
    # a node in k blocks has 4 k + 2 columns; above 8192 the entries are
    # sorted.  M 1 is the volume around each node
    from tmr_gb300 import TMR
    f = _fan_forest(TMR, k, extra)
    n = 4 * k + 2
    F = TMR.MatrixFilter(0.5, 3, None, [f])
    rp, c, v, _, _, _ = F.getMatrix()
    assert rp[1] - rp[0] == n
    assert all(np.all(np.diff(c[rp[i]:rp[i + 1]]) > 0) for i in range(0, n, 97))
    D = np.add.reduceat(v, rp[:-1])
    conn = f.getMeshConn()
    lev = f.getOctantsArray()[:, 5]
    vol = np.bincount(conn.reshape(-1), np.repeat(0.125 ** lev, 8), minlength=len(D)) / 8.0
    # sums of at most 8 k + 4 products of positive numbers
    np.testing.assert_allclose(D, vol, rtol=1e-12)
    # the entry of the axis with itself: k corners of 1/27
    np.testing.assert_allclose(v[rp[0]], k / 27.0, rtol=1e-12)


def test_filter_of_many_quadrants(gpu_lib):
    # 2^27 quadrants: one more than the row assembly's places take
    import torch

    from tmr_gb300 import TMR
    if torch.cuda.mem_get_info()[0] < (200 << 30):
        pytest.skip("needs 200 GB of device memory")
    f = TMR.QuadForest(order=2)
    f.setConnectivity(W.brick2d(2, 1))
    f.createTrees(13)
    assert f.getNumQuadrants() == 1 << 27
    f.createNodes()
    F = TMR.MatrixFilter(1e-4, 1, None, [f])
    n, nnz = F.size()
    side = 1 << 13
    assert n == (2 * side + 1) * (side + 1)
    assert nnz == (3 * (2 * side + 1) - 2) * (3 * (side + 1) - 2)
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    y = torch.empty_like(x)
    F.applyFilter(x, y)
    # the filter keeps constants: rounding of a two-term sum
    assert float((y - 1).abs().max()) < 1e-12


@pytest.mark.parametrize("dim", [3, 2])
def test_sorted_and_row_assembly_agree(gpu_lib, dim):
    # a small mesh, whose entries are sorted, beside uniform blocks that take
    # the matrix over the line to the rows: the same bits
    from tests.test_gpu_balance_paths import _union
    from tmr_gb300 import TMR
    base = W.rotate_blocks(W.brick(2, 2, 1), 4) if dim == 3 else W.brick2d(3, 2)
    extra = W.brick(2, 2, 2) if dim == 3 else W.brick2d(3, 3)
    depth = 4 if dim == 3 else 7
    got = []
    for conn in (base, _union([base, extra])):
        f = (TMR.OctForest if dim == 3 else TMR.QuadForest)(order=2)
        f.setConnectivity(conn)
        f.createTrees(1)
        for p in range(depth - 1):
            a = f.getOctantsArray() if dim == 3 else f.getQuadrantsArray()
            mine = a[:, 0] < len(base)
            flags = np.zeros(len(a), np.intc)
            flags[mine] = W.uniform(21, p, int(mine.sum())) < (0.3 if p < 3 else 0.0)
            flags[~mine] = 1
            f.refine(flags, 0, depth)
            f.balance(1)
        f.createNodes()
        a = f.getOctantsArray() if dim == 3 else f.getQuadrantsArray()
        ne = len(a)
        n = int(f.getMeshConn()[a[:, 0] < len(base)].max()) + 1
        rp, c, v, A, B, T = TMR.MatrixFilter(0.1, 3, None, [f]).getMatrix()
        got.append((ne, rp[:n + 1], c[:rp[n]], v[:rp[n]]))
    line = 2_000_000 // (64 if dim == 3 else 16)
    assert got[0][0] < line < got[1][0]
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.array_equal(a, b)
