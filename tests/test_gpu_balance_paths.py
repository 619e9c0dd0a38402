"""The paths of refine and balance against each other: an in-place refine
against the sorting one, and the balance over a hash set of families against
the sorting one (128-bit keys, and a set that outgrew its list)."""
import numpy as np
import pytest

from tmr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _union(conns):
    """Disjoint bricks as one connectivity."""
    out, off = [], 0
    for c in conns:
        out.append(c + off)
        off += int(c.max()) + 1
    return np.vstack(out)


def _forest(TMR, dim, conn, depth):
    f = (TMR.OctForest if dim == 3 else TMR.QuadForest)(order=2)
    f.setConnectivity(conn)
    f.createTrees(depth)
    return f


def _cells(f):
    if hasattr(f, "getOctantsArray"):
        a = f.getOctantsArray()
        return a[:, [0, 1, 2, 3, 5, 6]]
    a = f.getQuadrantsArray()
    return a[:, [0, 1, 2, 4, 5]]


def _brick(dim, *n):
    return W.brick(*n) if dim == 3 else W.brick2d(*n[:2])


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("other", [-1, 2])
def test_refine_in_place_equals_sorted(gpu_lib, dim, other):
    # the second brick's flags decide the path: zeros leave every octant at
    # its anchor, a coarsening or a refinement by two levels does not
    from tmr_gb300 import TMR
    conn = _union([_brick(dim, 3, 2, 1), _brick(dim, 1, 1, 1)])
    nb = len(conn) - 1
    got = []
    for last in (0, other):
        f = _forest(TMR, dim, conn, 2)
        for p in range(3):
            c = _cells(f)
            flags = W.random_indicator(len(c), 11, p, 0.4)
            flags[c[:, 0] == nb] = last if p == 1 else 0
            f.refine(flags, 0, 5)
            c = _cells(f)
            got.append(c[c[:, 0] < nb])
            f.balance(1)
    for a, b in zip(got[:3], got[3:]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dim", [3, 2])
@pytest.mark.parametrize("corner", [0, 1])
def test_hashed_balance_equals_sorted(gpu_lib, dim, corner):
    # 64-bit keys alone; with many more trees the same levels need 128-bit
    # keys, which take the sorting path
    from tmr_gb300 import TMR
    base = _brick(dim, 2, 2, 2)
    if dim == 3:
        base = W.rotate_blocks(base, 3)
    depth = 17 if dim == 3 else 27
    extra = _brick(dim, 40, 30, 1)
    got = []
    for conn in (base, _union([base, extra])):
        f = _forest(TMR, dim, conn, 1)
        for p in range(depth - 1):
            c = _cells(f)
            pick = np.zeros(len(c), np.intc)
            mine = np.flatnonzero(c[:, 0] < len(base))
            # the octants next to a point off the grid, and a few at random
            h = (1 << (30 - c[mine, 4 if dim == 3 else 3].astype(np.int64)))
            pt = np.int64(0.3141592 * (1 << 30))
            inside = np.ones(len(mine), bool)
            for k in range(dim):
                x = c[mine, 1 + k].astype(np.int64)
                inside &= (x <= pt) & (pt < x + h)
            pick[mine] = (inside & (c[mine, 0] % 3 == 1)) | (
                W.uniform(5, p, len(mine)) < (0.1 if p < 4 else 0.0))
            f.refine(pick, 0, depth)
            f.balance(corner)
        c = _cells(f)
        got.append(c[c[:, 0] < len(base)])
    assert got[0][:, 4 if dim == 3 else 3].max() == depth
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("dim", [3, 2])
def test_balance_of_a_set_that_outgrows_its_list(gpu_lib, dim):
    # deep seeds far apart: their closure has many more families than the
    # octants given, so the hash set gives up and the sorting path runs; one
    # balanced forest balanced again (which fits the set) must not change
    from tmr_gb300 import TMR
    f = _forest(TMR, dim, _brick(dim, 2, 1, 1), 0)
    f.createRandomTrees(600 if dim == 3 else 3000, 9, 10, 4)
    n0 = len(_cells(f))
    f.balance(1)
    a = _cells(f)
    assert len(a) > (8 if dim == 3 else 4) * (n0 + n0 // 4 + 4096)
    # a complete cover of both trees, in element order
    lev = a[:, 4 if dim == 3 else 3].astype(np.float64)
    assert abs((2.0 ** (-dim * lev)).sum() - 2.0) < 1e-9
    f.balance(1)
    assert np.array_equal(_cells(f), a)


@pytest.mark.parametrize("order,interp", [(2, 1), (3, 1), (4, 1), (3, 2)])
def test_nodes_of_tiles_equal_nodes_of_entries(gpu_lib, order, interp):
    # a small forest emits every (element, object); with uniform bricks
    # beside it the same elements go through tiles, the last one ragged, and
    # keep their numbers (nodes are numbered in block order)
    from tmr_gb300 import TMR
    base = W.rotate_blocks(W.brick(2, 2, 1), 8)
    got = []
    for extra in (0, 4):
        conn = base if not extra else _union([base, W.brick(extra, 2, 1)])
        f = TMR.OctForest(order=order, interp=interp)
        f.setConnectivity(conn)
        f.createTrees(1)
        for p in range(4):
            c = _cells(f)
            flags = np.zeros(len(c), np.intc)
            mine = c[:, 0] < len(base)
            flags[mine] = W.uniform(13, p, int(mine.sum())) < (0.45 if p < 3 else 0.0)
            flags[~mine] = p < 3
            f.refine(flags, 0, 5)
            f.balance(1)
        f.createNodes()
        c = _cells(f)
        n = int((c[:, 0] < len(base)).sum())
        conn = f.getMeshConn()[:n]
        ptr, dc, dw = f.getDepNodeConn()
        nd = int(-conn.min())
        got.append((n, len(c), conn, ptr[:nd + 1], dc[:ptr[nd]], dw[:ptr[nd]]))
    assert got[0][1] < 16384 <= got[1][1] and got[1][1] % 256 != 0
    for a, b in zip(got[0][2:], got[1][2:]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("dim,blocks,nrand,lo,hi", [(3, (8, 8, 4), 2000, 5, 7), (3, (4, 4, 2), 3000, 6, 9),
                                                    (2, (8, 8), 20000, 6, 12)])
def test_a_set_that_outgrows_its_list_is_given_up_early(gpu_lib, dim, blocks, nrand, lo, hi):
    # the balance that gave its set up takes no more than a few times the
    # balance of its result, which fits one (1 to 2 times; 10 where every
    # level goes on adding to the full table)
    import time

    import torch

    from tmr_gb300 import TMR
    f = _forest(TMR, dim, _brick(dim, *blocks), 0)
    f.createRandomTrees(nrand, lo, hi, 4)

    def best(g):
        out, t = None, []
        for _ in range(4):
            out = g.duplicate()
            torch.cuda.synchronize()
            a = time.perf_counter()
            out.balance(1)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - a)
        return out, min(t)

    a, ta = best(f)
    b, tb = best(a)
    num = (lambda g: g.getNumOctants()) if dim == 3 else (lambda g: g.getNumQuadrants())
    n0 = num(f)
    assert num(a) > (8 if dim == 3 else 4) * (n0 + n0 // 4 + 4096) and num(b) == num(a)
    assert ta <= 5 * tb + 1e-3
