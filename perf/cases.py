"""What a user of the framework has it do, one case per entry of ``listed()``.

Every case goes through the package's public entry points (``tmr_gb300.TMR``).
The kinds, each over a range of sizes:

``step``      one adaptive step of an analysis forest: refine by an
              indicator, 2:1 balance, number the nodes, read the mesh
``pipeline``  the whole adaptation: trees, refinement passes, a hierarchy of
              coarser forests, the prolongations between them, and one
              restriction / prolongation of a block of vectors
``quad``      the same on a forest of quadtrees
``setup``     building the density filter of a new design mesh and filtering
              and restricting the design variables through it
``transfer``  P, P^T and the weight-normalised P^T of one prolongation
``mfilter``   the matrix density filter and its adjoint
``helmholtz`` the Helmholtz PDE filter and its adjoint
``stl``       the iso-surface of a design field

Forest sizes follow the configurations of the benchmark and of the tests: bricks
of blocks (their corners relabelled by rotations where the neighbours are to
meet in every orientation), refined at random or towards bumps.  A case's
``mesh`` number fixes which octants refine; the seed of ``prepare`` gives the
blocks the order a mesher happened to number them in (the same mesh, so sizes
do not change, with every octant, node and row at another place) and the
values of the vectors.
"""
import math

import numpy as np
import torch

from tmr_gb300 import TMR
from tmr_gb300 import workloads as W

HMAX = float(1 << 30)


def listed():
    return [
        # a few small trees, as in a unit problem or the first steps of an
        # adaptive run: launches and waits count, not bandwidth
        dict(name="step_small_o2", kind="step", order=2, nx=2, ny=2, nz=1, rot=0, shape="random",
             mesh=7, L0=2, passes=2, prob=0.3, max_level=6, corner=1),
        # blocks of a general hexahedral mesh meeting in every orientation
        dict(name="step_rot_o3", kind="step", order=3, nx=3, ny=3, nz=2, rot=1, shape="random",
             mesh=7, L0=1, passes=5, prob=0.3, max_level=7, corner=1),
        # a large linear mesh refined around features
        dict(name="step_bump_o2", kind="step", order=2, nx=16, ny=8, nz=8, rot=0, shape="bump",
             mesh=3, L0=2, target=6_000_000, max_level=9, corner=1),
        # the benchmark's multi-tree configuration, whole
        dict(name="pipeline_brick_o3", kind="pipeline", order=3, nx=8, ny=4, nz=4, rot=0,
             shape="random", mesh=7, L0=2, passes=5, prob=0.3, max_level=9, corner=1,
             levels=4, nvec=16),
        # the quadtree configuration of the benchmark, one pass less
        dict(name="quad_o3", kind="quad", order=3, nx=64, ny=64, mesh=7, L0=3, passes=4, prob=0.3,
             max_level=11, corner=1, levels=4, nvec=16),
        # a new design mesh: filter matrix and restriction operators
        dict(name="setup_bump_o2", kind="setup", order=2, nx=16, ny=8, nz=8, rot=0, shape="bump",
             mesh=3, L0=2, target=2_600_000, max_level=9, levels=3, N=10, vpn=3),
        # multigrid transfers of a block of vectors, quadratic elements
        dict(name="transfer_brick_o3_v16", kind="transfer", order=3, nx=8, ny=4, nz=4, rot=0,
             shape="random", mesh=7, L0=2, passes=4, prob=0.3, max_level=9, nvec=16),
        # one vector on a small linear mesh, as a solver's coarse levels see
        dict(name="transfer_rot_o2_v1", kind="transfer", order=2, nx=3, ny=2, nz=2, rot=1,
             shape="random", mesh=7, L0=2, passes=2, prob=0.3, max_level=6, nvec=1),
        # three design components per node through the filter and its
        # adjoint, in the two precisions it takes
        dict(name="mfilter_bump_f64_v3", kind="mfilter", order=2, nx=16, ny=8, nz=8, rot=0,
             shape="bump", mesh=3, L0=2, target=2_600_000, max_level=9,
             N=10, vpn=3, dtype="float64"),
        dict(name="mfilter_bump_f32_v3", kind="mfilter", order=2, nx=16, ny=8, nz=8, rot=0,
             shape="bump", mesh=3, L0=2, target=2_600_000, max_level=9,
             N=10, vpn=3, dtype="float32"),
        # one density field through the PDE filter and its adjoint
        dict(name="helmholtz_bump_o2", kind="helmholtz", order=2, nx=16, ny=8, nz=8, rot=0,
             shape="bump", mesh=3, L0=2, target=2_600_000, max_level=9, levels=5, vpn=1),
        # the surface of a design for export
        dict(name="stl_bump_o2", kind="stl", order=2, nx=16, ny=8, nz=8, rot=0, shape="bump",
             mesh=3, L0=2, target=2_600_000, max_level=9),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_forest(rng, lo, hi, order):
    """A brick refined to about log-uniform(lo, hi) octants."""
    if hi > 20_000 and rng.random() < 0.4:
        return dict(order=order, nx=rng.randint(2, 12), ny=rng.randint(2, 7),
                    nz=rng.randint(1, 7), rot=rng.randint(0, 1), shape="bump",
                    mesh=rng.randint(1, 999), L0=2,
                    target=_log_int(rng, max(lo, 20_000), hi), max_level=9)
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    while True:
        c = dict(order=order, nx=rng.randint(2, 8), ny=rng.randint(2, 5), nz=rng.randint(1, 4),
                 rot=rng.randint(0, 1), shape="random", mesh=rng.randint(1, 999),
                 L0=rng.randint(1, 3), passes=rng.randint(1, 5), prob=round(rng.uniform(0.15, 0.4), 3), max_level=9)
        # a pass makes 1 + 7 p octants of one, and the balance adds some
        n = c["nx"] * c["ny"] * c["nz"] * 8.0 ** c["L0"] * min(
            8.0, (1 + 7 * c["prob"]) * 1.35) ** c["passes"]
        if target / 1.6 < n < min(target * 1.6, hi):
            return c


def draw(rng):
    kind = rng.choice(["step", "step", "pipeline", "quad", "setup", "transfer", "transfer",
                       "mfilter", "mfilter", "helmholtz", "stl"])
    if kind == "step":
        order = rng.choice([2, 2, 3, 3, 4])
        c = _draw_forest(rng, 1_000, {2: 6_000_000, 3: 2_000_000, 4: 600_000}[order], order)
        c["corner"] = rng.choice([0, 1, 1])
    elif kind == "pipeline":
        order = rng.choice([2, 3])
        c = _draw_forest(rng, 3_000, 4_000_000, order)
        c.update(corner=1, levels=rng.randint(2, 4), nvec=rng.choice([1, 2, 3, 6, 16]))
    elif kind == "quad":
        c = dict(order=rng.choice([2, 3]), nx=rng.randint(3, 64), ny=rng.randint(3, 64),
                 mesh=rng.randint(1, 999), L0=rng.randint(1, 3), passes=rng.randint(1, 4),
                 prob=round(rng.uniform(0.15, 0.3), 3), max_level=11, corner=rng.choice([0, 1]),
                 levels=rng.randint(2, 4), nvec=rng.choice([1, 2, 3, 6, 16]))
    elif kind == "setup":
        c = _draw_forest(rng, 5_000, 2_600_000, 2)
        c.update(levels=rng.randint(1, 4), N=rng.randint(5, 15), vpn=rng.choice([1, 2, 3]))
    elif kind == "transfer":
        order = rng.choice([2, 3])
        c = _draw_forest(rng, 1_000, {2: 4_000_000, 3: 1_500_000}[order], order)
        c["nvec"] = rng.choice([1, 2, 3, 4, 6, 7, 16])
    elif kind == "mfilter":
        c = _draw_forest(rng, 2_000, 2_600_000, 2)
        c.update(N=rng.randint(5, 15), vpn=rng.choice([1, 2, 3, 3, 5]),
                 dtype=rng.choice(["float64", "float32"]))
    elif kind == "helmholtz":
        c = _draw_forest(rng, 20_000, 2_000_000, 2)
        c.update(levels=rng.randint(4, 5), vpn=rng.choice([1, 2, 3]))
    else:
        c = _draw_forest(rng, 5_000, 2_600_000, rng.choice([2, 2, 3]))
        c["rot"] = 0  # a block's box has the axes of its corners
    c["kind"] = kind
    return c


# ---------------------------------------------------------------------------
# Forests.
def _order(nblocks, seed):
    """The brick's block (its place counted x fastest) at every number."""
    return np.random.default_rng(seed).permutation(nblocks)


def _conn(case, seed):
    conn = W.brick(case["nx"], case["ny"], case["nz"])
    conn = W.rotate_blocks(conn, 5) if case["rot"] else conn
    return conn[_order(len(conn), seed)]


def _boxes(case, seed):
    """Unit cubes at the blocks' places in the brick."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    b = _order(nx * ny * nz, seed)
    box = np.ones((len(b), 6))
    box[:, 0], box[:, 1], box[:, 2] = b % nx, (b // nx) % ny, b // (nx * ny)
    return box


def _random_flags(case, p, place):
    """Pass p's random refinement array, drawn in the order of the brick's
    places: `place` is the place of every element's block."""
    n = place.numel()
    flags = torch.empty(n, dtype=torch.int32, device="cuda")
    flags[torch.argsort(place, stable=True)] = TMR.random_refinement(n, case["mesh"], p,
                                                                    case["prob"])
    return flags


def _bump_flags(case, f, place):
    """The octants nearest 16 Gaussian bumps, as many as take the forest to
    about the target size (the balance adds about 30%)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    L = torch.tensor([nx, ny, nz], dtype=torch.float64, device="cuda")
    cen = torch.tensor(W.uniform(case["mesh"], 0, 48).reshape(-1, 3), device="cuda") * L
    sig = 0.05 * L
    o = f.getOctantsDevice()
    lev = o["level"].long()
    org = torch.stack([place % nx, (place // nx) % ny, place // (nx * ny)], 1).double()
    xyz = torch.stack([o["x"], o["y"], o["z"]], 1).double()
    c = org + (xyz + 0.5 * torch.pow(2.0, (30 - lev).double())[:, None]) / HMAX
    val = torch.zeros(c.shape[0], dtype=torch.float64, device="cuda")
    for k in range(16):
        val += torch.exp(-0.5 * (((c - cen[k]) / sig) ** 2).sum(1))
    val[lev >= case["max_level"]] = -1.0
    n = val.numel()
    k = int(min(n, max(1, (case["target"] - n) / 7 / 1.3)))
    thr = torch.topk(val, k).values[-1]
    return ((val >= thr) & (val > 0)).int()


def _adapt(case, seed, last=True):
    """The forest of a case after its refinement passes (last=False: before
    the last one) and the refinement array of every pass."""
    conn = _conn(case, seed)
    order = torch.from_numpy(_order(len(conn), seed)).cuda()
    f = TMR.OctForest(order=case["order"], interp=TMR.GAUSS_LOBATTO_POINTS)
    f.setConnectivity(conn)
    f.createTrees(case["L0"])
    passes = 12 if case["shape"] == "bump" else case["passes"]
    flags = []
    for p in range(passes):
        place = order[f.getOctantsDevice()["block"].long()]
        if case["shape"] == "bump":
            flags.append(_bump_flags(case, f, place))
        else:
            flags.append(_random_flags(case, p, place))
        done = p == passes - 1 or (
            case["shape"] == "bump" and
            place.numel() + 7 * 1.3 * int(flags[-1].sum()) >= 0.95 * case["target"])
        if done and not last:
            break
        f.refine(flags[-1], 0, case["max_level"])
        f.balance(case.get("corner", 1))
        if done:
            break
    return f, flags


def _numbered(case, seed):
    f = _adapt(case, seed)[0]
    f.createNodes()
    return f


def _coarser(f, corner=1):
    c = f.coarsen()
    c.balance(corner)
    c.createNodes()
    return c


def _hierarchy(f, levels, corner=1):
    out = [f]
    for _ in range(levels - 1):
        out.append(_coarser(out[-1], corner))
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _octants(f):
    o = f.getOctantsDevice()
    return {k: o[k] for k in ("block", "x", "y", "z", "level")}


def _filter_radius(f):
    return 2.0 / 2.0 ** int(f.getOctantsDevice()["level"].max().item())


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": seed}
    g = _gen(seed)
    if kind == "step":
        s["forest"], flags = _adapt(case, seed, last=False)
        s["flags"] = flags[-1]
    elif kind == "pipeline":
        s["conn"] = _conn(case, seed)
        f, s["flags"] = _adapt(case, seed)
        f.createNodes()
        n = int(f.getNodeRange()[1])
        s["x"] = torch.randn(n * case["nvec"], dtype=torch.float64, device="cuda", generator=g)
    elif kind == "quad":
        s["conn"], f, s["flags"] = _quad_forest(case, seed)
        n = int(f.getNodeRange()[1])
        s["x"] = torch.randn(n * case["nvec"], dtype=torch.float64, device="cuda", generator=g)
    elif kind == "transfer":
        f = _numbered(case, seed)
        s["I"] = TMR.VecInterp()
        f.createInterpolation(_coarser(f), s["I"])
        rows, cols, _ = s["I"].sizes()
        nv = case["nvec"]
        s["xc"] = torch.randn(cols * nv, dtype=torch.float64, device="cuda", generator=g)
        s["xf"] = torch.randn(rows * nv, dtype=torch.float64, device="cuda", generator=g)
    else:
        f = _numbered(case, seed)
        n = int(f.getNodeRange()[1])
        if kind == "stl":
            f.setBlockBoxes(_boxes(case, seed))
            # a few waves across the domain
            ph = W.uniform(case["mesh"], 1, 3) * 2 * np.pi
            X = torch.from_numpy(f.getPoints()[int(f.getExtPreOffset()):]).cuda()
            s["forest"] = f
            s["x"] = 0.5 + 0.2 * (torch.sin(2.0 * X[:, 0] + ph[0]) +
                                  torch.sin(2.5 * X[:, 1] + ph[1]) +
                                  torch.sin(3.0 * X[:, 2] + ph[2]))
            return s
        vpn = case["vpn"]
        dt = torch.float32 if case.get("dtype") == "float32" else torch.float64
        # densities in [0, 1] and a sensitivity of either sign
        s["x"] = torch.rand(n * vpn, dtype=dt, device="cuda", generator=g)
        s["w"] = torch.randn(n * vpn, dtype=dt, device="cuda", generator=g)
        s["r"] = _filter_radius(f)
        if kind == "setup":
            s["forests"] = _hierarchy(f, case["levels"])
        elif kind == "mfilter":
            s["forest"] = f
            s["F"] = TMR.MatrixFilter(s["r"], case["N"], None, [f], vpn=vpn)
        else:
            s["forests"] = _hierarchy(f, case["levels"])
            for c in s["forests"]:
                c.setBlockBoxes(_boxes(case, seed))
            s["F"] = TMR.HelmholtzFilter(s["r"], None, s["forests"], vpn=vpn)
    return s


def _quad_forest(case, seed):
    conn = W.brick2d(case["nx"], case["ny"])
    order = _order(len(conn), seed)
    conn = conn[order]
    f = TMR.QuadForest(order=case["order"], interp=TMR.GAUSS_LOBATTO_POINTS)
    f.setConnectivity(conn)
    f.createTrees(case["L0"])
    flags = []
    for p in range(case["passes"]):
        place = torch.from_numpy(order[f.getQuadrantsArray()[:, 0]]).cuda()
        flags.append(_random_flags(case, p, place))
        f.refine(flags[-1], 0, case["max_level"])
        f.balance(case["corner"])
    f.createNodes()
    return conn, f, flags


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        f = s["forest"].duplicate()
        f.refine(s["flags"], 0, case["max_level"])
        f.balance(case["corner"])
        f.createNodes()
        s["kept"] = f  # the outputs are views of the forest's own arrays
        return {"octants": _octants(f), "conn": f.getMeshConn(copy=False),
                "dep": f.getDepNodeConn(copy=False)}
    if kind in ("pipeline", "quad"):
        s["kept"] = None
        cls = TMR.OctForest if kind == "pipeline" else TMR.QuadForest
        f = cls(order=case["order"], interp=TMR.GAUSS_LOBATTO_POINTS)
        f.setConnectivity(s["conn"])
        f.createTrees(case["L0"])
        for flags in s["flags"]:
            f.refine(flags, 0, case["max_level"])
            f.balance(case["corner"])
        f.createNodes()
        forests = _hierarchy(f, case["levels"], case["corner"])
        interps = []
        for fine, coarse in zip(forests, forests[1:]):
            interps.append(TMR.VecInterp())
            fine.createInterpolation(coarse, interps[-1])
        nv, x, restricted = case["nvec"], s["x"], []
        for I in interps:
            y = torch.empty(I.sizes()[1] * nv, dtype=torch.float64, device="cuda")
            x = I.multTranspose(x, y)
            restricted.append(x)
        for I in reversed(interps):
            y = torch.empty(I.sizes()[0] * nv, dtype=torch.float64, device="cuda")
            x = I.mult(x, y)
        s["kept"] = forests
        out = {"restricted": restricted, "prolonged": x}
        if kind == "pipeline":
            out["octants"] = [_octants(c) for c in forests]
        else:
            out["quadrants"] = [c.getNumQuadrants() for c in forests]
            # the coarsest mesh is what a direct solver is set up with
            out["coarsest"] = [forests[-1].getQuadrantsArray(), forests[-1].getMeshConn()]
        return out
    if kind == "transfer":
        I, nv = s["I"], case["nvec"]
        rows, cols, _ = I.sizes()
        up = torch.empty(rows * nv, dtype=torch.float64, device="cuda")
        down = torch.empty(cols * nv, dtype=torch.float64, device="cuda")
        mean = torch.empty_like(down)
        return {"P": I.mult(s["xc"], up), "Pt": I.multTranspose(s["xf"], down),
                "Pwt": I.multWeightTranspose(s["xf"], mean)}
    if kind == "setup":
        F = TMR.MatrixFilter(s["r"], case["N"], None, s["forests"], vpn=case["vpn"])
        return F.setDesignVars(s["x"])
    if kind == "stl":
        return TMR.getSTLTriangles(s["forest"], s["x"], cutoff=0.5)
    # mfilter, helmholtz
    rho, gx = torch.empty_like(s["x"]), torch.empty_like(s["w"])
    return {"filtered": s["F"].applyFilter(s["x"], rho),
            "adjoint": s["F"].applyTranspose(s["w"], gx)}


# ---------------------------------------------------------------------------
def _nbytes(v):
    if isinstance(v, dict):
        return sum(_nbytes(x) for x in v.values())
    if isinstance(v, (list, tuple)):
        return sum(_nbytes(x) for x in v)
    return getattr(v, "nbytes", 8)


def _mesh_bytes(f, order, dim=3):
    """Connectivity and dependent rows of a numbered forest."""
    z = f._sizes()
    return 4 * int(z[4]) * order ** dim + 4 * int(z[2]) + 12 * int(z[5])


def work(case):
    """Bytes and operations of one pass: inputs and outputs once, and the
    operators that are built or applied (12 bytes an entry) once each."""
    s = prepare(case, 1)
    out = run(s)
    kind, order = case["kind"], case["order"]
    b, fl = float(_nbytes(out)), 0.0
    if kind == "step":
        b += _nbytes(s["flags"]) + 18.0 * s["forest"].getNumOctants()
    elif kind in ("pipeline", "quad"):
        b += _nbytes(s["x"]) + _nbytes(s["flags"])
        dim = 3 if kind == "pipeline" else 2
        for f in s["kept"]:
            b += _mesh_bytes(f, order, dim)
        for fine, coarse in zip(s["kept"], s["kept"][1:]):
            I = TMR.VecInterp()
            fine.createInterpolation(coarse, I)
            b += 12.0 * I.sizes()[2] + 2 * 12.0 * I.applyNnz()
            fl += 2 * 2.0 * I.applyNnz() * case["nvec"]
    elif kind == "transfer":
        nnz = s["I"].applyNnz()
        b += 12.0 * nnz * 3 + _nbytes([s["xc"], s["xf"], s["xf"]])
        fl = 3 * 2.0 * nnz * case["nvec"]
    elif kind == "setup":
        n, nnz = TMR.MatrixFilter(s["r"], case["N"], None, s["forests"][:1]).size()
        b += _nbytes(s["x"]) + 12.0 * nnz + sum(_mesh_bytes(f, order) for f in s["forests"])
        fl = 2.0 * nnz * case["vpn"] * case["N"]
    elif kind == "mfilter":
        n, nnz = s["F"].size()
        word = 4 if case["dtype"] == "float32" else 8
        # every Horner term needs the whole matrix and the previous term
        b += _nbytes([s["x"], s["w"]]) + 2.0 * case["N"] * ((word + 4) * nnz + 2 * word * n *
                                                          case["vpn"])
        fl = 2 * 2.0 * nnz * case["vpn"] * case["N"]
    elif kind == "helmholtz":
        b += _nbytes([s["x"], s["w"]]) + 2.0 * _mesh_bytes(s["forests"][0], order)
        fl = 2 * 2.0 * 64 * s["forests"][0].getNumOctants() * case["vpn"]
    else:
        b += _nbytes(s["x"]) + _mesh_bytes(s["forest"], order) + 18.0 * s["forest"].getNumOctants()
    return {"bytes": b, "flops": fl}


# ---------------------------------------------------------------------------
# 64-bit values, in plain torch.
class _Mesh:
    """A linear octree mesh's nodes and elements as torch arrays: values on
    the element corners (dependent nodes through their weights) and back."""

    def __init__(self, f):
        self.n = int(f.getNodeRange()[1])
        ptr, dconn, dw = f.getDepNodeConn()
        nd = len(ptr) - 1
        self.nd = nd
        self.drow = torch.repeat_interleave(
            torch.arange(nd, device="cuda"), torch.from_numpy(np.diff(ptr)).cuda().long())
        self.dcol = torch.from_numpy(dconn).cuda().long()
        self.dw = torch.from_numpy(dw).cuda()
        c = torch.from_numpy(f.getMeshConn()).cuda().long()
        # independent nodes first, then the dependent ones
        self.conn = torch.where(c >= 0, c, self.n - c - 1)
        lev = f.getOctantsDevice()["level"].double()
        self.h = torch.pow(2.0, -lev)

    def gather(self, x):
        """x (n, v) -> corner values (elements, 8, v)."""
        d = torch.zeros(self.nd, x.shape[1], dtype=torch.float64, device="cuda")
        d.index_add_(0, self.drow, self.dw[:, None] * x[self.dcol])
        return torch.cat([x, d])[self.conn]

    def scatter(self, u):
        y = torch.zeros(self.n + self.nd, u.shape[2], dtype=torch.float64, device="cuda")
        y.index_add_(0, self.conn.reshape(-1), u.reshape(-1, u.shape[2]))
        out = y[: self.n].clone()
        out.index_add_(0, self.dcol, self.dw[:, None] * y[self.n:][self.drow])
        return out


def _kron3(a, b, c):
    """Corner matrix of a product of 1-D matrices, x fastest."""
    return torch.kron(c, torch.kron(b, a))


_M1 = torch.tensor([[2.0, 1.0], [1.0, 2.0]], dtype=torch.float64) / 6.0
_K1 = torch.tensor([[1.0, -1.0], [-1.0, 1.0]], dtype=torch.float64)


def _corner(mesh, A, scale, x):
    u = torch.einsum("ab,ebv->eav", A.cuda(), mesh.gather(x))
    return mesh.scatter(u * scale[:, None, None])


def _mass(mesh, x):
    return _corner(mesh, _kron3(_M1, _M1, _M1), mesh.h ** 3, x)


def _helmholtz_matrix(mesh, r, x):
    lap = _kron3(_K1, _M1, _M1) + _kron3(_M1, _K1, _M1) + _kron3(_M1, _M1, _K1)
    return _mass(mesh, x) + r * r * _corner(mesh, lap, mesh.h, x)


def _solve(apply, diag, b):
    """Conjugate gradients to rounding, one component at a time."""
    out = torch.zeros_like(b)
    for v in range(b.shape[1]):
        x, res = torch.zeros_like(b[:, v: v + 1]), b[:, v: v + 1].clone()
        z = res / diag
        p, rz = z.clone(), float((res * z).sum())
        stop = 1e-15 * float(b[:, v].norm())
        for _ in range(600):
            q = apply(p)
            a = rz / float((p * q).sum())
            x += a * p
            res -= a * q
            if float(res.norm()) <= stop:
                break
            z = res / diag
            new = float((res * z).sum())
            p, rz = z + (new / rz) * p, new
        out[:, v: v + 1] = x
    return out


def _horner(mesh, r, N, x, transpose):
    """The matrix filter: N + 1 terms of the Neumann series of the
    Helmholtz operator, scaled to keep constants."""
    one = torch.ones(mesh.n, 1, dtype=torch.float64, device="cuda")
    D = _mass(mesh, one)
    t = D ** (2.0 / 3.0)
    A = 1.0 / (1.0 + r * r / t)
    B = A * r * r / (t * D)

    def forward(x):
        t1 = A * x
        y = t1
        for _ in range(N):
            y = B * _mass(mesh, y) + t1
        return y

    T = 1.0 / forward(one)
    if not transpose:
        return T * forward(x)
    t1 = T * x
    y = t1
    for _ in range(N):
        y = _mass(mesh, B * y) + t1
    return A * y


def _product(rows, cols, w, x, nout):
    """y[rows] += w x[cols] in pieces."""
    y = torch.zeros(nout, x.shape[1], dtype=torch.float64, device="cuda")
    for a in range(0, len(w), 8_000_000):
        k = slice(a, a + 8_000_000)
        y.index_add_(0, rows[k], w[k, None] * x[cols[k].long()])
    return y


def exact(case, seed):
    """The filters and the transfers of a given P; the forests themselves
    and what is interpolated between them have no closed form (None)."""
    kind = case["kind"]
    if kind not in ("transfer", "mfilter", "helmholtz", "setup"):
        return None
    s = prepare(case, seed)
    if kind == "transfer":
        nv = case["nvec"]
        ptr, cols, w = s["I"].getCSR()
        n, nc, _ = s["I"].sizes()
        cols, w = torch.from_numpy(cols).cuda(), torch.from_numpy(w).cuda()
        rows = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32),
                                       torch.from_numpy(np.diff(ptr)).cuda())
        xc, xf = s["xc"].reshape(-1, nv), s["xf"].reshape(-1, nv)
        down = _product(cols, rows, w, xf, nc)
        one = torch.ones(n, 1, dtype=torch.float64, device="cuda")
        norm = _product(cols, rows, w, one, nc)
        return {"P": _product(rows, cols, w, xc, n).reshape(-1), "Pt": down.reshape(-1),
                "Pwt": torch.where(norm != 0, down / norm, 0.0).reshape(-1)}
    forest = s["forest"] if kind == "mfilter" else s["forests"][0]
    mesh, vpn, r = _Mesh(forest), case["vpn"], s["r"]
    x, w = s["x"].double().reshape(-1, vpn), s["w"].double().reshape(-1, vpn)
    if kind == "setup":
        first = _horner(mesh, r, case["N"], x, False).reshape(-1)
        return [first] + [None] * (case["levels"] - 1)
    if kind == "mfilter":
        return {"filtered": _horner(mesh, r, case["N"], x, False).reshape(-1),
                "adjoint": _horner(mesh, r, case["N"], w, True).reshape(-1)}
    # the diagonal only speeds the solve up: the mass matrix's row sums do
    diag = _mass(mesh, torch.ones(mesh.n, 1, dtype=torch.float64, device="cuda"))
    K = lambda v: _helmholtz_matrix(mesh, r, v)  # noqa: E731
    return {"filtered": _solve(K, diag, _mass(mesh, x)).reshape(-1),
            "adjoint": _mass(mesh, _solve(K, diag, w)).reshape(-1)}
