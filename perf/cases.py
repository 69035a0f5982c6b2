"""Workloads of the T-matrix solve path, run through the package's public entry points.

Two sources of the operator, as hosts use them:

* "host": the program owns the operator in the reference's arrays (projector columns S, Sx, Sy, Sz with indS,
  near-zone blocks sp_mat with sp_ind) and hands it over with set_projectors and set_nearzone.  These arrays are
  synthetic: basis functions at random places of an ellipsoid's projection boxes, quadratic interpolation weights
  and their derivatives as projectors, near-zone blocks that fall off with distance around a unit diagonal.
* "mesh": seeded meshes of the shapes the benchmark and the tests use (jittered cube lattices clipped to a body),
  with the operator built on the device.

Paths ("path"):

* "matvec"   compute_Ax2 on host vectors: a host that keeps its own Krylov loop calls this once per iteration
* "gmres"    one right-hand side solved to the reference's tolerance, where the host keeps its column loop
* "columns"  solve_columns on an incident matrix the host owns
* "T"        compute_T_matrix: incident columns, solve and T assembly on the device
* "sweep"    solve_sweep: several wavelengths of one particle in one batched solve
* "particle" everything one new particle needs: context, Green spectrum, projectors, near zone, T
* "served"   requests of different particles submitted together to a server that keeps their operators resident

Mixed-precision solves refine to 1e-10: the T-matrix to FP64 quality, three refinement steps.  Their step counts are
diagnostics of the inner complex64 solves and are not returned; those of FP64 solves are.
"""
import math

import numpy as np
import torch

from scadyn_b200 import api, meshgen
from scadyn_b200.server import Server

FP64, MIXED = "fp64", "mixed"
AXES = {"sphere": (1.0, 1.0, 1.0), "ellipsoid": (1.0, 0.8, 0.6)}


def listed():
    return [
        # the tests' 1,680-tet size handed over by the host: one matvec, where launches and copies count
        {"name": "matvec host 1.7k", "path": "matvec", "source": "host", "tets": 1680, "N": 14, "storage": 32},
        # a host that keeps its near zone in complex128, a ragged size
        {"name": "matvec host 7k c128", "path": "matvec", "source": "host", "tets": 7013, "N": 22, "storage": 64},
        # the linear basis: 12 unknowns per tet, 12x12 near-zone blocks
        {"name": "matvec linear 3k", "path": "matvec", "source": "mesh", "body": "sphere", "n": 5.0, "cell": 2.6,
         "ka": 1.5, "order": 1},
        # the benchmark's 150k-tet ellipsoid: one iteration of a large solve
        {"name": "matvec 150k", "path": "matvec", "source": "mesh", "body": "ellipsoid", "n": 23.2, "cell": 2.7183,
         "ka": 8.0, "order": 0},
        # the benchmark's 43k-tet sphere at ka 2: one column in the reference's FP64 GMRES
        {"name": "gmres 43k", "path": "gmres", "source": "mesh", "body": "sphere", "n": 12.0, "cell": 2.9567, "ka": 2.0},
        # host-owned operator and incident matrix, all columns of Nmax 3 in FP64
        {"name": "columns host 3k fp64", "path": "columns", "source": "host", "tets": 3000, "N": 18, "storage": 32,
         "ncol": 30, "precision": FP64, "block": 16},
        # the same hand-over in mixed precision, an odd column count
        {"name": "columns host 6k mixed", "path": "columns", "source": "host", "tets": 6144, "N": 22, "storage": 32,
         "ncol": 47, "precision": MIXED, "block": 32},
        # whole T-matrix of a 12k-tet sphere in FP64, batched
        {"name": "T sphere 12k fp64", "path": "T", "source": "mesh", "body": "sphere", "n": 8.0, "cell": 2.7, "ka": 2.0,
         "Nmax": 4, "ncol": 48, "precision": FP64, "block": 16},
        # the sweep's 60k-tet ellipsoid at the middle of its ka range: columns of the benchmark's form
        {"name": "T ellipsoid 60k mixed", "path": "T", "source": "mesh", "body": "ellipsoid", "n": 17.05, "cell": 2.7,
         "ka": 4.0, "Nmax": 9, "ncol": 32, "precision": MIXED, "block": 32},
        # three wavelengths of a small ellipsoid in one solve
        {"name": "sweep 3 x 6k", "path": "sweep", "source": "mesh", "body": "ellipsoid", "n": 8.0, "cell": 2.6,
         "ka": 1.2, "nw": 3, "Nmax": 3, "precision": MIXED, "block": 32},
        # one new 8k-tet particle from mesh to T
        {"name": "particle 8k", "path": "particle", "source": "mesh", "body": "sphere", "n": 7.0, "cell": 2.6, "ka": 1.5,
         "Nmax": 3, "precision": MIXED, "block": 32},
        # three requests of the served stream's small sizes, together
        {"name": "served 3 requests", "path": "served", "source": "mesh", "body": "sphere", "n": 6.0, "cell": 2.6,
         "ka": 1.5, "Nmax": 4, "requests": 3, "precision": MIXED, "block": 32},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _even(v):
    return 2 * int(round(v / 2))


def draw(rng):
    path = rng.choice(["matvec", "matvec", "gmres", "columns", "T", "T", "sweep", "particle", "served"])
    precision = rng.choice([FP64, MIXED])
    few = path in ("columns", "T")      # a host may solve a few columns in small blocks; whole T-matrices go in large ones
    block = rng.choice(([1, 7] if few else []) + [16, 32, 48]) if precision == MIXED else \
        rng.choice(([1, 4] if few else []) + [16, 32])
    body = rng.choice(["sphere", "ellipsoid"])
    fill = 1.0 if body == "sphere" else 0.48 ** (1 / 3)
    cell = round(rng.uniform(1.8, 3.0), 2)
    n_of = lambda tets: round((tets / (8 * math.pi)) ** (1 / 3) / fill, 2)  # noqa: E731
    if path in ("matvec", "columns") and rng.random() < 0.5:
        tets = int(_log(rng, 300, 7500 if path == "matvec" else 4000))
        case = {"path": path, "source": "host", "tets": tets, "storage": rng.choice([32, 32, 64]),
                "N": max(8, _even(2.2 * (tets / rng.uniform(12, 22) * 1.9) ** (1 / 3) + 3))}
        if path == "columns":
            case.update(ncol=rng.randint(1, min(48, 8 * block)), precision=precision, block=block)
        return case
    case = {"path": path, "source": "mesh", "body": body, "cell": cell}
    if path == "matvec":
        order = rng.choice([0, 0, 1])
        case.update(order=order, n=n_of(_log(rng, 400, 4000 if order else 60000)), ka=round(rng.uniform(0.5, 8.0), 3))
    elif path == "gmres":
        case.update(n=n_of(_log(rng, 400, 45000)), ka=round(rng.uniform(0.5, 4.0), 3))
    elif path in ("columns", "T"):
        nmax = rng.randint(2, 6)
        case.update(n=n_of(_log(rng, 400, 20000)), ka=round(rng.uniform(0.5, 4.0), 3), Nmax=nmax,
                    ncol=rng.randint(1, min(48, 8 * block, 2 * ((nmax + 1) ** 2 - 1))), precision=precision, block=block)
        case["path"] = "T"
    elif path == "sweep":
        case.update(n=n_of(_log(rng, 400, 8000)), ka=round(rng.uniform(0.8, 1.6), 3), nw=rng.randint(2, 4),
                    Nmax=rng.randint(2, 3), precision=precision, block=block)
    elif path == "particle":
        case.update(n=n_of(_log(rng, 400, 12000)), ka=round(rng.uniform(0.5, 2.5), 3), Nmax=rng.randint(2, 4),
                    precision=precision, block=block)
    else:
        case.update(n=n_of(_log(rng, 400, 5000)), ka=round(rng.uniform(0.8, 2.0), 3), Nmax=rng.randint(2, 4),
                    requests=rng.randint(2, 4), precision=precision, block=block)
    return case


def _opts(case):
    if case["precision"] == MIXED:
        return dict(tol=1e-10, m=30, cycles=60, block=case["block"], precision=api.PREC_MIXED, inner_tol=3e-4,
                    max_outer=10)
    return dict(tol=1e-6, m=50, cycles=12, block=case["block"], precision=api.PREC_FP64)


# ---- operators from a mesh ------------------------------------------------


def _mesh(case, seed, n=None):
    mesh = meshgen.lattice_body(n or case["n"], AXES[case["body"]], seed=seed, eps=2.25 + 0.01j)
    if case["body"] == "ellipsoid":
        mesh.param = meshgen.uniform_eps_sampler()(np.random.default_rng(seed + 1), mesh.n_tet)
    return mesh


def _mesh_solver(mesh, ka, cell, order=0):
    s = api.Solver.from_desc(api.grid_from_mesh(mesh.coord, mesh.etopol, grid_size=cell, order=order))
    s.set_wavenumber(ka / mesh.a)
    s.set_mesh(mesh.coord, mesh.etopol, mesh.param)
    s.build_G()
    # the C call behind pfft_projection_const / _lin, without their copy back to the host
    rc = s.lib.scd_build_projectors(s.ctx)
    if rc:
        raise api.ScadynError(rc, "scd_build_projectors")
    s.compute_near_zone_interactions_const(api.STORE_C64)
    return s


# ---- operators a host owns ------------------------------------------------

KD = 0.3        # wavenumber times node spacing


def _host_operator(case, seed):
    """The arrays of a host's operator, from the seed: S*, indS, sp_mat, sp_ind, the grid and k (node spacing 1)."""
    rng = np.random.default_rng(seed)
    T, N = case["tets"], case["N"]
    n = np.array([N, max(8, _even(0.9 * N)), max(8, _even(0.8 * N))])
    nc = (n - 2) // 2
    x, y, z = np.meshgrid(*[np.arange(c) for c in nc], indexing="ij")
    cubes = np.stack([x, y, z], -1).reshape(-1, 3)
    body = cubes[(((cubes + 0.5 - nc / 2) / (nc / 2)) ** 2).sum(1) < 1.0]
    cube = body[rng.integers(0, len(body), T)]
    frac = rng.uniform(0.0, 2.0, (T, 3))                    # place in the box, in node spacings
    pos = 2.0 * cube + frac
    # projectors: quadratic interpolation onto the box's 3 x 3 x 3 nodes
    t = frac[:, :, None]
    L = np.concatenate([(t - 1) * (t - 2) / 2, t * (2 - t), t * (t - 1) / 2], 2)
    D = np.concatenate([t - 1.5, 2 - 2 * t, t - 0.5], 2)
    density = T / (8.0 * len(body))
    amp = np.sqrt((rng.uniform(0.1, 0.3, T) + 1j * rng.uniform(0.0, 0.05, T)) / density)[:, None]

    def weights(ax, ay, az):
        return amp * np.einsum("ti,tj,tk->tkji", ax, ay, az).reshape(T, 27)

    S = weights(L[:, 0], L[:, 1], L[:, 2])
    P = [weights(*[(D if e == d else L)[:, e] for e in range(3)]) for d in range(3)]
    j = np.arange(27)
    first = 2 * cube[:, 0] + n[0] * (2 * cube[:, 1] + n[1] * 2 * cube[:, 2])
    indS = (first[:, None] + j % 3 + n[0] * (j // 3 % 3 + n[1] * (j // 9)) + 1).astype(np.int32)
    # near-zone pairs: every pair of neighbouring boxes, each pair of tets once
    cid = (cube * [1, nc[0], nc[0] * nc[1]]).sum(1)
    order = np.argsort(cid, kind="stable")
    start = np.searchsorted(cid[order], np.arange(nc.prod() + 1))
    pairs = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                other = cube + [dx, dy, dz]
                ok = ((other >= 0) & (other < nc)).all(1)
                oc = np.where(ok, (other * [1, nc[0], nc[0] * nc[1]]).sum(1), 0)
                cnt = np.where(ok, start[oc + 1] - start[oc], 0)
                a = np.repeat(np.arange(T), cnt)
                at = np.arange(len(a)) - np.repeat(np.cumsum(cnt) - cnt, cnt)
                b = order[np.repeat(start[oc], cnt) + at]
                pairs.append(np.stack([a, b], 1)[b >= a])
    pairs = np.concatenate(pairs)
    a, b = pairs[:, 0], pairs[:, 1]
    r2 = ((pos[a] - pos[b]) ** 2).sum(1) + 0.4
    size = 0.05 / density * r2 ** -1.5
    sp = rng.standard_normal((len(a), 9), np.float32) + 1j * rng.standard_normal((len(a), 9), np.float32)
    sp = (sp.reshape(-1, 3, 3) * size[:, None, None]).astype(np.complex64 if case["storage"] == 32 else np.complex128)
    sp[a == b] = sp[a == b] * 0.2 + np.eye(3, dtype=sp.dtype)
    return {"n": [int(v) for v in n], "S": [S] + P, "indS": indS, "sp_mat": sp,
            "sp_ind": np.ascontiguousarray(pairs + 1, dtype=np.int32), "pos": pos}


def _incident(case, op, seed):
    """Plane waves of seeded directions and polarisations at the tets, (ncol, 3T)."""
    rng = np.random.default_rng([seed, 7])
    d = rng.standard_normal((case["ncol"], 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    pol = rng.standard_normal((case["ncol"], 3)) + 1j * rng.standard_normal((case["ncol"], 3))
    phase = np.exp(1j * KD * d @ op["pos"].T)
    return (phase[:, :, None] * pol[:, None, :]).reshape(case["ncol"], -1)


def _vector(n, seed):
    rng = np.random.default_rng([seed, 3])
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


# ---- prepare and run --------------------------------------------------------


def prepare(case, seed):
    path = case["path"]
    if case["source"] == "host":
        op = _host_operator(case, seed)
        s = api.Solver(*op["n"], 1.0, (0.0, 0.0, 0.0), case["tets"])
        s.set_wavenumber(KD)
        s.set_projectors(*op["S"], op["indS"])
        s.build_G()
        s.set_nearzone(op["sp_mat"], op["sp_ind"])
        if path == "matvec":
            return {"case": case, "solver": s, "x": _vector(s.n, seed)}
        return {"case": case, "solver": s, "mat": _incident(case, op, seed)}
    if path == "served":
        meshes = [_mesh(case, seed + 10 * r, case["n"] * (1 - 0.12 * r)) for r in range(case["requests"])]
        return {"case": case, "server": Server(), "meshes": meshes}
    mesh = _mesh(case, seed)
    if path == "particle":
        return {"case": case, "mesh": mesh}
    if path == "sweep":
        kas = [case["ka"] * 1.4 ** w for w in range(case["nw"])]
        return {"case": case, "solvers": [_mesh_solver(mesh, ka, case["cell"]) for ka in kas],
                "Nmax": [case["Nmax"] + w for w in range(case["nw"])]}
    s = _mesh_solver(mesh, case["ka"], case["cell"], case.get("order", 0))
    state = {"case": case, "solver": s}
    if path in ("matvec", "gmres"):
        state["x"] = _vector(s.n, seed)
    return state


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "matvec":
        return state["solver"].compute_Ax2(state["x"])
    if path == "gmres":
        x, info = state["solver"].gmres(state["x"], tol=1e-6, m=50, cycles=4)
        return {"x": x, "iters": info["iters"]}
    opts = _opts(case)
    if path == "columns":
        T, iters, X, _ = state["solver"].solve_columns(state["mat"], want_x=True, **opts)
    elif path == "T":
        T, iters = state["solver"].compute_T_matrix(case["Nmax"], ncol=case["ncol"], **opts)
    elif path == "sweep":
        T, iters, _, _ = api.solve_sweep(state["solvers"], state["Nmax"], **opts)
    elif path == "particle":
        s = _mesh_solver(state["mesh"], case["ka"], case["cell"])
        T, iters = s.compute_T_matrix(case["Nmax"], **opts)
        s.close()
    else:
        srv = state["server"]
        ids = [srv.submit(m, case["ka"] / m.a, case["cell"], case["Nmax"], **opts) for m in state["meshes"]]
        for i in ids:
            srv.wait(i)
        done = [srv.result(i) for i in ids]
        T, iters = [d[0] for d in done], [d[1] for d in done]
    out = {"T": T}
    if path == "columns":
        out["X"] = X
    if case["precision"] == FP64:
        out["iters"] = iters
    return out


# ---- work ---------------------------------------------------------------------


def _tets(case, n):
    return case["tets"] if case["source"] == "host" else 8 * math.pi * n ** 3 * math.prod(AXES[case["body"]])


def _operator_work(case, n):
    """(bytes of the operator, flops of one application to one vector, unknowns), estimated from the sizes."""
    T = _tets(case, n)
    if case["source"] == "host":
        grid = case["N"] ** 3 * 0.72
        boxes = 0.52 * (case["N"] / 2 - 1) ** 3 * 0.72
    else:
        boxes = T / (6 * (case["cell"] / 6 ** (1 / 3)) ** 3)
        grid = 8 * (2 * n * 6 ** (1 / 3) / case["cell"] + 2) ** 3 * math.prod(AXES[case["body"]])
    per_box = max(1.0, T / boxes)
    pairs = T * 13.5 * per_box * max(0.3, 1 - 1.6 / max(2.0, boxes ** (1 / 3)))
    nb = 4 if case.get("order") else 1
    pairs, cols = pairs * nb * nb, T * nb
    el = 16 if case.get("storage") == 64 else 8
    fft = 8 * 8 * grid * 5 * math.log2(max(2.0, 8 * grid))
    return pairs * 9 * el + 4 * 27 * cols * 16 + grid * 16, pairs * 9 * 16 + 4 * 2 * 27 * cols * 8 + fft, 3 * cols


def work(case):
    path = case["path"]
    n0 = case.get("n", 0.0)
    if path == "matvec":
        by, fl, unk = _operator_work(case, n0)
        return {"bytes": by + 2 * 16 * unk, "flops": fl}
    ka = case.get("ka", 1.0)
    mixed = case.get("precision") == MIXED
    if path == "served":
        parts = [(n0 * (1 - 0.12 * r), ka, 2 * ((case["Nmax"] + 1) ** 2 - 1)) for r in range(case["requests"])]
    elif path == "sweep":
        parts = [(n0, ka * 1.4 ** w, 2 * ((case["Nmax"] + w + 1) ** 2 - 1)) for w in range(case["nw"])]
    else:
        ncol = 1 if path == "gmres" else case["ncol"] if "ncol" in case else 2 * ((case["Nmax"] + 1) ** 2 - 1)
        parts = [(n0, ka, ncol)]
    bytes_, flops = 0.0, 0.0
    for n, k, ncol in parts:
        by, fl, unk = _operator_work(case, n)
        steps = (8 + 3 * k) * (1.7 if mixed else 1.0)
        together = min(ncol, case.get("block", 1))
        el = 8 if mixed else 16
        # per step of a block of columns: the operator once, and each column's new basis vector written and read
        bytes_ += steps * (math.ceil(ncol / together) * by + ncol * 2 * el * unk) + ncol * 2 * 16 * unk
        flops += steps * ncol * (fl + steps * 8 * unk)
        if path == "particle":
            bytes_ += 2 * by
            flops += 12 * 24 * 60 * _tets(case, n) * 200
    return {"bytes": bytes_, "flops": flops}


# ---- exact ----------------------------------------------------------------------


class _Dense64:
    """The host operator applied in complex128 with plain torch: near-zone blocks, interpolation and FFT convolution."""

    def __init__(self, op):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        put = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(dev)  # noqa: E731
        self.n, self.dev = op["n"], dev
        self.P = [put(p) for p in op["S"]]
        self.node = put(op["indS"].astype(np.int64) - 1)
        self.V = put(op["sp_mat"].astype(np.complex128)).transpose(1, 2)      # sp_mat[b, c, r] -> V[b, r, c]
        ind = put(op["sp_ind"].astype(np.int64) - 1)
        self.a, self.b = ind[:, 0], ind[:, 1]
        self.off = self.a != self.b
        nx, ny, nz = self.n
        ax = [torch.cat([torch.arange(v), v - torch.arange(v)]).to(dev).double() for v in self.n]
        R = (ax[2][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2).sqrt()
        G = torch.exp(1j * KD * R) / (4 * math.pi * R.clamp(min=1.0))
        G[0, 0, 0] = 0
        G[nz], G[:, ny], G[:, :, nx] = 0, 0, 0
        self.F = torch.fft.fftn(G)

    def _grid(self, g):
        nx, ny, nz = self.n
        f = torch.fft.fftn(g.reshape(-1, nz, ny, nx), s=(2 * nz, 2 * ny, 2 * nx), dim=(1, 2, 3)) * self.F
        return torch.fft.ifftn(f, dim=(1, 2, 3))[:, :nz, :ny, :nx].reshape(len(g), -1)

    def one(self, x):
        X = x.reshape(-1, 3)
        ngrid = math.prod(self.n)
        src = torch.zeros(4, ngrid, dtype=torch.complex128, device=self.dev)
        for d in range(3):
            src[d].index_add_(0, self.node.reshape(-1), (self.P[0] * X[:, d:d + 1]).reshape(-1))
            src[3].index_add_(0, self.node.reshape(-1), (self.P[1 + d] * X[:, d:d + 1]).reshape(-1))
        g = self._grid(src)
        out = torch.zeros_like(X)
        for d in range(3):
            out[:, d] = (self.P[1 + d] * g[3][self.node]).sum(1) - KD ** 2 * (self.P[0] * g[d][self.node]).sum(1)
        out.index_add_(0, self.a, torch.einsum("brc,bc->br", self.V, X[self.b]))
        V, a, b = self.V[self.off], self.a[self.off], self.b[self.off]
        out.index_add_(0, b, torch.einsum("brc,br->bc", V, X[a]))
        return out.reshape(-1)

    def solve(self, rhs):
        """GMRES to rounding."""
        x = torch.zeros_like(rhs)
        for _ in range(6):
            r = rhs - self.one(x)
            beta = torch.linalg.vector_norm(r)
            if beta < 3e-14 * torch.linalg.vector_norm(rhs):
                break
            Q, m = [r / beta], 40
            H = torch.zeros(m + 1, m, dtype=torch.complex128, device=self.dev)
            for i in range(m):
                w = self.one(Q[i])
                B = torch.stack(Q)
                for _twice in range(2):
                    h = B.conj() @ w
                    w = w - h @ B
                    H[:i + 1, i] += h
                H[i + 1, i] = torch.linalg.vector_norm(w)
                Q.append(w / H[i + 1, i])
                if i % 8 == 7 or i == m - 1:
                    e = torch.zeros(i + 2, 1, dtype=torch.complex128, device=self.dev)
                    e[0] = beta
                    y = torch.linalg.lstsq(H[:i + 2, :i + 1].cpu(), e.cpu()).solution.to(self.dev)
                    if torch.linalg.vector_norm(H[:i + 2, :i + 1] @ y - e) < 1e-11 * beta:
                        break
            x = x + (torch.stack(Q[:len(y)]).T @ y)[:, 0]
        return x


def exact(case, seed):
    if case["source"] != "host":
        return None             # the mesh's singular integrals in 64 bits take minutes
    op = _host_operator(case, seed)
    A = _Dense64(op)
    if case["path"] == "matvec":
        return A.one(torch.from_numpy(_vector(3 * case["tets"], seed)).to(A.dev)).cpu().numpy()
    mat = torch.from_numpy(_incident(case, op, seed)).to(A.dev)
    X = torch.stack([A.solve(m) for m in mat])
    out = {"T": (X @ mat.conj().T).cpu().numpy(), "X": X.cpu().numpy()}
    if case["precision"] == FP64:
        out["iters"] = None
    return out
