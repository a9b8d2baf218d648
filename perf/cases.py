"""The work that is timed: what programs have this library do, through its public calls.

Structures come from the library's own generator (value noise of period 8, the bottom layer
held; a case's `world` is the generator's seed), or, for the calls that take any lattice,
from the same structures laid out as the reference's `build` does
(statics/src/lattice.rs:76-163). The stiffnesses, materials and loads come from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parallax-world_b200"))
import statics_cuda as sc  # noqa: E402

UNIT = 0.125  # a level-0 cell's edge, metres
SECTION = 0.336
G_OVER_E = 0.4
FACES = np.array([(-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)])
PRECISION = {"fp64": sc.FP64, "mixed": sc.MIXED}
EDGES = (16, 24, 32, 48, 64)
MATERIALS = ["masonry", "stone", "wood"]
DENSITY = np.array([2000.0, 2500.0, 600.0])


def listed():
    return [
        # The smallest structure an edit leaves behind, at the defaults of the drop-in call: all
        # latency and launches.
        dict(name="piece 8 fp64", kind="solve", world=1, nx=8, ny=8, nz=8, k="uniform", precision="fp64", tol=1e-6, host=False),
        # The plain FP64 solve of the benchmark's small configuration.
        dict(name="piece 32 fp64", kind="solve", world=1, nx=32, ny=32, nz=32, k="uniform", precision="fp64", tol=1e-8,
             host=False),
        # A ragged building-sized piece in host arrays, as a caller without device buffers has it.
        dict(name="piece 61x45x37 mixed", kind="solve", world=1, nx=61, ny=45, nz=37, k="lognormal", precision="mixed",
             tol=1e-8, host=True),
        # The headline piece in each precision, inputs and motions in device memory.
        dict(name="piece 128 fp64", kind="solve", world=1, nx=128, ny=128, nz=128, k="uniform", precision="fp64", tol=1e-8,
             host=False),
        dict(name="piece 128 mixed", kind="solve", world=1, nx=128, ny=128, nz=128, k="uniform", precision="mixed", tol=1e-8,
             host=False),
        # The largest piece of the range, edges that are no powers of two.
        dict(name="piece 167x160x150 mixed", kind="solve", world=1, nx=167, ny=160, nz=150, k="lognormal", precision="mixed",
             tol=1e-8, host=False),
        # Many uneven pieces in one call, sized as the benchmark's batch draws them.
        dict(name="batch 64 mixed", kind="batch", world=1, pieces=64, most=64, precision="mixed", tol=1e-8),
        # Forward and backward: the compliance and its gradient by every cell's stiffness.
        dict(name="adjoint 96 fp64", kind="adjoint", world=1, nx=96, ny=96, nz=96, k="uniform", precision="fp64", tol=1e-8),
        # The drop-in call for any lattice, at the reference's tolerance.
        dict(name="lattice 28", kind="motions", world=1, nx=28, ny=28, nz=28, tol=1e-6),
        # The reference's caller of it: rounds of solving and breaking until nothing breaks.
        dict(name="settle 20", kind="settle", world=1, nx=20, ny=20, nz=20),
        # A coarser level measured from a finer one.
        dict(name="gather 28", kind="gather", world=1, nx=28, ny=28, nz=28),
        # One step of the engine's solver, at the engine's tolerance.
        dict(name="mechanics 40", kind="mech", world=1, nx=40, ny=40, nz=40, tol=1e-3),
    ]


def draw(rng):
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "solve", "batch", "adjoint", "motions", "settle", "gather", "mech"])
    if kind == "batch":
        return dict(kind=kind, world=rng.randrange(1 << 30), pieces=edge(4, 64), most=rng.choice(EDGES[1:]), precision=rng.choice(["mixed", "mixed", "fp64"]),
                    tol=1e-8)
    most = {"solve": 144, "adjoint": 96, "motions": 30, "settle": 20, "gather": 30, "mech": 40}[kind]
    case = dict(kind=kind)
    case.update({a: edge(9, most) for a in ("nx", "ny", "nz")})
    while True:  # a world that has something standing on its support
        case["world"] = rng.randrange(1 << 30)
        if (structure(case) == sc.CELL_FREE).sum() * 20 >= case["nx"] * case["ny"] * case["nz"]:
            break
    if kind in ("solve", "adjoint"):
        case.update(k=rng.choice(["uniform", "lognormal"]), precision=rng.choice(["fp64", "mixed"]), tol=1e-8)
    if kind == "solve":
        case["host"] = rng.random() < 0.25
    if kind == "motions":
        case["tol"] = rng.choice([1e-6, 1e-8])
    if kind == "mech":
        case["tol"] = rng.choice([1e-3, 1e-8])
    return case


# ---- inputs -------------------------------------------------------------------------
_solver = None


def solver():
    """The one context a program keeps."""
    global _solver
    if _solver is None:
        _solver = sc.Solver(0)
    return _solver


def structure(case, shape=None, more=0):
    shape = shape or (case["nx"], case["ny"], case["nz"])
    return sc.generate_piece(*shape, case["world"] + more, sc.K_UNIFORM)[0]


def stiffness(state, dist, seed):
    """Each cell's stiffness: uniform in [0.5, 2], or lognormal clipped to [0.1, 10]."""
    rng = np.random.default_rng(seed)
    k = rng.random(state.shape, np.float32) * np.float32(1.5) + np.float32(0.5) if dist == "uniform" else \
        np.clip(np.exp(0.5 * rng.standard_normal(state.shape, np.float32)), 0.1, 10.0)
    return np.where(state != sc.CELL_EMPTY, k, np.float32(0.0)).astype(np.float32)


def batch_pieces(case, seed):
    rng = np.random.default_rng(case["world"])
    edges = [e for e in EDGES if e <= case["most"]]
    pieces = []
    for i in range(case["pieces"]):
        state = structure(case, tuple(int(v) for v in rng.choice(edges, 3)), i)
        pieces.append((state, stiffness(state, "uniform", seed * 64 + i)))
    return pieces


def upright(case, seed):
    """A structure whose held layer is y = 0 (the lattice calls' gravity points down y), and each
    cell's material."""
    state = sc.generate_piece(case["nx"], case["nz"], case["ny"], case["world"], sc.K_UNIFORM)[0]
    state = np.ascontiguousarray(state.transpose(0, 2, 1))
    return state, np.random.default_rng(seed).integers(0, len(MATERIALS), state.shape)


def materials(case, seed):
    """The materials by name; for a gather, whose result's sizes hang on the materials' ratios,
    the structure's own materials with values that the seed scales."""
    if case["kind"] != "gather":
        return MATERIALS
    return [tuple(v * (0.5 + np.random.default_rng(seed).random()) for v in sc.MATERIALS[m]) for m in MATERIALS]


def cells_of(state):
    """The free cells, in order, each one's six nodes (numbered by first touch), each node's key
    (axis and the greater of the two cells it lies between) and whether it is held."""
    shape = np.array(state.shape)
    cells = np.argwhere(state == sc.CELL_FREE)
    big = shape + 1
    keys = np.empty((len(cells), 6), np.int64)
    for f, d in enumerate(FACES):
        at = cells + np.maximum(d, 0)  # the greater cell of the face
        keys[:, f] = (((f // 2) * big[0] + at[:, 0]) * big[1] + at[:, 1]) * big[2] + at[:, 2]
    uniq, first, back = np.unique(keys.ravel(), return_index=True, return_inverse=True)
    order = np.argsort(first, kind="stable")
    rank = np.empty_like(order)
    rank[order] = np.arange(len(order))
    ends = rank[back.ravel()].reshape(-1, 6)
    key = uniq[order]
    z, key = key % big[2], key // big[2]
    y, key = key % big[1], key // big[1]
    x, axis = key % big[0], key // big[0]
    hi = np.stack([x, y, z], 1)
    lo = hi - np.eye(3, dtype=np.int64)[axis]

    def is_held(c):
        inside = ((c >= 0) & (c < shape)).all(1)
        at = np.where(inside[:, None], c, 0)
        return inside & (state[at[:, 0], at[:, 1], at[:, 2]] == sc.CELL_HELD)

    return cells, ends, np.stack([lo, hi], 1), is_held(lo) | is_held(hi)


def beams():
    """The 15 beams of a unit cell: ends, direction, length, and the four bonds' points from
    the cell's centre."""
    out = []
    for a in range(6):
        for b in range(a + 1, 6):
            xa, xb = 0.5 * FACES[a], 0.5 * FACES[b]
            d = float(np.linalg.norm(xb - xa))
            n = (xb - xa) / d
            e1 = np.cross(n, [1.0, 0.0, 0.0] if abs(n[0]) < 0.9 else [0.0, 1.0, 0.0])
            e1 /= np.linalg.norm(e1)
            e2 = np.cross(n, e1)
            r = math.sqrt(SECTION / (2.0 * math.pi))
            out.append((a, b, n, d, 0.5 * (xa + xb) + r * np.stack([e1, -e1, e2, -e2])))
    return out


def lattice(state, mat, names=MATERIALS):
    """The piece as a lattice: nodes on every face of a free cell, four bonds a beam."""
    cells, ends, around, held = cells_of(state)
    of = mat[cells[:, 0], cells[:, 1], cells[:, 2]]
    table = np.array([sc.MATERIALS[m] if isinstance(m, str) else m for m in names])
    n_nodes = len(around)
    mass = np.zeros(n_nodes)
    np.add.at(mass, ends.ravel(), np.repeat(DENSITY[of] * UNIT ** 3 / 6.0, 6))
    node_mat = np.full(n_nodes, -1, np.int64)
    for m in np.argsort(DENSITY):  # the densest of the cells at a node
        node_mat[ends[of == m].ravel()] = m
    cols = {k: [] for k in ("bi", "bj", "p", "n")}
    keep, d, c = [], [], (cells + 0.5) * UNIT
    for a, b, n, length, p in beams():
        keep.append(np.repeat(~(held[ends[:, a]] & held[ends[:, b]])[:, None], 4, 1))
        cols["bi"].append(np.repeat(ends[:, a:a + 1], 4, 1))
        cols["bj"].append(np.repeat(ends[:, b:b + 1], 4, 1))
        cols["p"].append(c[:, None, :] + UNIT * p)
        cols["n"].append(np.broadcast_to(n, (len(cells), 4, 3)))
        d.append(np.full((len(cells), 4), UNIT * length))
    keep = np.stack(keep, 1).reshape(-1)
    out = {k: np.ascontiguousarray(np.stack(v, 1).reshape((-1, 3) if k in "pn" else -1)[keep]) for k, v in cols.items()}
    rows = table[np.repeat(of, 60)[keep]]
    for i, k in enumerate(("e", "g", "ft", "fc", "fs")):
        out[k] = np.ascontiguousarray(rows[:, i])
    out.update(x=(around + 0.5).sum(1) * 0.5 * UNIT, held=held.astype(np.uint8), around=around, level=0, m=mass,
               mat=node_mat.astype(np.int32), a=np.full(len(rows), SECTION * UNIT ** 2 / 4.0),
               d=np.stack(d, 1).reshape(-1)[keep])
    return out


def weights(lat):
    loads = np.zeros((len(lat["m"]), 6))
    loads[:, 1] = -9.81 * lat["m"]
    return loads


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, solver=solver())
    if kind in ("solve", "batch", "adjoint"):
        s["opt"] = sc.options(tol=case["tol"], precision=PRECISION[case["precision"]])
    if kind == "batch":
        s["pieces"] = batch_pieces(case, seed)
    elif kind in ("solve", "adjoint"):
        state = structure(case)
        k = stiffness(state, case["k"], seed)
        n_nodes = max(1, sc.grid_count(state)[0])
        if kind == "solve" and not case["host"]:
            state, k = torch.from_numpy(state).cuda(), torch.from_numpy(k).cuda()
            g = sc.Grid()
            g.nx, g.ny, g.nz = case["nx"], case["ny"], case["nz"]
            g.state, g.k, g.on_device = state.data_ptr(), k.data_ptr(), 1
            g.g_over_e, g.rho, g.gravity[2] = G_OVER_E, 512.0, -1.0
            s.update(grid=g, motions=torch.zeros(n_nodes, 6, dtype=torch.float64, device="cuda"))
        elif kind == "solve":
            s["motions"] = np.zeros((n_nodes, 6))
        s.update(state=state, k=k)
    elif kind == "mech":
        state = structure(case)
        k = stiffness(state, "uniform", seed)
        s.update(system=sc.mech_voxel_system(state, np.float32(1e9) * k), tol=case["tol"])
    else:
        names = materials(case, seed)
        s.update(lattice=lattice(*upright(case, case["world"] if kind == "gather" else seed), names), materials=names)
        if kind == "motions":
            s.update(loads=weights(s["lattice"]), opt=sc.options(tol=case["tol"]))
    return s


def run(s):
    kind, solver = s["kind"], s["solver"]
    if kind == "solve" and "grid" in s:
        solver.solve_grid_device(s["grid"], s["opt"], s["motions"].data_ptr(), s["motions"].numel())
        return {"motions": s["motions"]}
    if kind == "solve":
        return {"motions": solver.solve_grid(s["state"], s["k"], s["opt"], out=s["motions"])[0]}
    if kind == "batch":
        return {"motions": solver.solve_grid_batch(s["pieces"], s["opt"])[0]}
    if kind == "adjoint":
        c, grad, motions, _ = solver.compliance_grad(s["state"], s["k"], s["opt"])
        return {"compliance": c, "gradient": grad, "motions": motions}
    if kind == "motions":
        return {"motions": solver.motions(s["lattice"], loads=s["loads"], opt=s["opt"])}
    if kind == "settle":
        fell, _, gone, _ = solver.settle(s["lattice"])
        return {"fell": fell, "gone": gone}
    if kind == "gather":
        return solver.gather(s["lattice"], s["materials"])
    x, _, _ = solver.mech_solve(s["system"], tol=s["tol"])
    return {"x": x}


# ---- what a pass cannot do without ----------------------------------------------------
def work(case):
    """The inputs read and the outputs written once, and the operator's arithmetic: a cell's
    36 x 36 template has 552 entries that are not zero, the V-cycle and the conjugate
    gradients apply it six times an iteration, and the iterations to the tolerance grow about as
    the cube root of the piece's edge (36 at 16 cubed, 59 at 48 cubed, 92 at 128 cubed to 1e-8)."""
    kind = case["kind"]
    if kind == "batch":
        edges = [e for e in EDGES if e <= case["most"]]
        shapes = [(sum(edges) / len(edges),) * 3] * case["pieces"]
    else:
        shapes = [(case["nx"], case["ny"], case["nz"])]
    total = {"bytes": 0.0, "flops": 0.0}
    for shape in shapes:
        cells = float(np.prod(shape))
        free = cells * 0.5 + 1
        nodes = 3.3 * free
        if kind in ("motions", "settle", "gather"):
            in_out = nodes * (24 + 1 + 48 + 8) + 60 * free * 112
            in_out += {"motions": nodes * 96, "settle": nodes, "gather": (nodes * 100 + 60 * free * 150) / 7}[kind]
        elif kind == "mech":
            in_out = 1.2 * free * (24 + 24 + 72 + 24 + 24) + 1.2 * free * 11 * 80
        else:
            in_out = cells * 5 + nodes * 48 + (cells * 8 if kind == "adjoint" else 0)
        tol = case.get("tol", 1e-6)
        iterations = 0 if kind == "gather" else 16.5 * cells ** (1 / 9) * -math.log10(tol) / 8
        flops = iterations * free * (2 * 24 * 24 * 3 if kind == "mech" else 6 * 2 * 552)
        if kind == "gather":
            flops = free / 8 * 2 * 72 * 72 * 90 / 3
        total["bytes"] += in_out
        total["flops"] += flops
    return total


# ---- the same answers in 64 bits, by other means ----------------------------------------
def cell_stiffness(s):
    """A free cell's 36 x 36 stiffness for E = 1 (statics/src/model.rs:139-149)."""
    K = np.zeros((36, 36))
    for a, b, n, d, points in beams():
        S = (np.outer(n, n) + G_OVER_E * (np.eye(3) - np.outer(n, n))) * (SECTION / 4.0 * s / d)

        def moved(r):
            return np.array([[1, 0, 0, 0, r[2], -r[1]], [0, 1, 0, -r[2], 0, r[0]], [0, 0, 1, r[1], -r[0], 0]])

        for p in points:
            B = np.zeros((3, 36))
            B[:, 6 * a:6 * a + 6] = moved(s * (p - 0.5 * FACES[a]))
            B[:, 6 * b:6 * b + 6] = -moved(s * (p - 0.5 * FACES[b]))
            K += B.T @ S @ B
    return K


def pcg(apply, precondition, b):
    """Conjugate gradients to rounding, restarted twice from the true residual."""
    x = torch.zeros_like(b)
    norm = float(b.norm())
    for _ in range(3):
        r = b - apply(x)
        z = precondition(r)
        p, rz = z.clone(), (r * z).sum()
        for i in range(40000):
            q = apply(p)
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            z = precondition(r)
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
            if i % 50 == 49 and float(r.norm()) <= 1e-14 * norm:
                break
    return x


def solve_cells(state, stiff, loads_of):
    """Motions of a piece's nodes, the free cells' stiffness and nodes, and the loads."""
    cells, ends, _, held = cells_of(state)
    dev = "cuda"
    K = torch.from_numpy(cell_stiffness(UNIT)).to(dev)
    k = torch.from_numpy(np.ascontiguousarray(stiff[cells[:, 0], cells[:, 1], cells[:, 2]].astype(np.float64))).to(dev)
    ends = torch.from_numpy(ends).to(dev)
    free = torch.from_numpy(~held).to(dev).double()[:, None]
    n = len(held)
    loads = loads_of(cells, ends, n) * free
    diag = torch.zeros(n, 6, 6, dtype=torch.float64, device=dev)
    for f in range(6):
        diag.index_add_(0, ends[:, f], k[:, None, None] * K[6 * f:6 * f + 6, 6 * f:6 * f + 6])
    inv = torch.linalg.inv(diag)
    flat = ends.reshape(-1)

    def apply(x):
        y = k[:, None] * (x[flat].reshape(-1, 36) @ K)
        return torch.zeros_like(x).index_add_(0, flat, y.reshape(-1, 6)) * free

    u = pcg(apply, lambda r: (inv @ r[:, :, None])[:, :, 0] * free, loads)
    return u, k, K, ends, loads


def down_z(cells, ends, n):
    """The generator's loads: a mass of 1 a cell, a sixth of it on each face, gravity -z."""
    loads = torch.zeros(n, 6, dtype=torch.float64, device="cuda")
    loads[:, 2] = -torch.bincount(ends.reshape(-1), minlength=n).double() / 6.0
    return loads


def exact(case, seed):
    kind = case["kind"]
    cells = case["pieces"] * case["most"] ** 3 / 4 if kind == "batch" else case["nx"] * case["ny"] * case["nz"]
    if kind in ("settle", "gather") or cells > 130000:
        return None
    if kind == "mech":
        state = structure(case)
        system = sc.mech_voxel_system(state, np.float32(1e9) * stiffness(state, "uniform", seed))
        t = {a: torch.from_numpy(system[a].astype(np.int64) if a in ("pi", "pj") else system[a]).cuda()
             for a in ("diag", "pi", "pj", "pb", "b")}
        inv = torch.linalg.inv(t["diag"])

        def apply(x):
            y = (t["diag"] @ x[:, :, None])[:, :, 0]
            y.index_add_(0, t["pi"], (t["pb"] @ x[t["pj"]][:, :, None])[:, :, 0])
            return y.index_add_(0, t["pj"], (t["pb"].transpose(1, 2) @ x[t["pi"]][:, :, None])[:, :, 0])

        return {"x": pcg(apply, lambda r: (inv @ r[:, :, None])[:, :, 0], t["b"])}
    if kind == "batch":
        return {"motions": [solve_cells(state, k, down_z)[0] for state, k in batch_pieces(case, seed)]}
    if kind == "motions":
        state, mat = upright(case, seed)
        lat = lattice(state, mat)
        e = np.array([sc.MATERIALS[m][0] for m in MATERIALS])[mat]
        return {"motions": solve_cells(state, e, lambda c, ends, n: torch.from_numpy(weights(lat)).cuda())[0]}
    state = structure(case)
    stiff = stiffness(state, case["k"], seed)
    u, k, K, ends, loads = solve_cells(state, stiff, down_z)
    if kind == "solve":
        return {"motions": u}
    x = u[ends.reshape(-1)].reshape(-1, 36)
    grad = torch.zeros(state.shape, dtype=torch.float64, device="cuda")
    grad[torch.from_numpy(state == sc.CELL_FREE).cuda()] = -((x @ K) * x).sum(1)
    return {"compliance": float((loads * u).sum()), "gradient": grad, "motions": u}
