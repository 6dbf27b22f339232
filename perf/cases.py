"""The work a user of this library has it do, as timed cases.

Each case is one pass through the public entry points, on the seeded
synthetic systems of the benchmarks: jittered hex meshes (also one cell
deep, the 2-d convention), cells permuted and then renumbered by the
framework, the pressure-correction and the momentum matrix.  As in the
SIMPLE loop, a program keeps one solver per mesh (the structure is handed
over once) and every pass brings new coefficients and right-hand sides.

kinds
  cg     solv_cg on a pressure system (FP64, or FP32 inner iterations)
  host   the same through the host-array call, as a Fortran caller makes it
  bicg   solv_bicg on a momentum system, n_vc components from a given field
  batch  solv_cg_batch: uneven pressure systems solved together
  fcg    solv_fcg, the learned + mixed-precision pressure solve
  fv     the assembly, gradient, flux and correction steps of one outer
         iteration of the SIMPLE loop
  train  one gradient of the learned preconditioner's training loss
"""
import math

import numpy as np
import torch

from programs_b200.cases import batch_sizes
from programs_b200.fv import GpuFv
from programs_b200.learn import DEFAULT_WEIGHTS, load_params
from programs_b200.mesh import Mesh
from programs_b200.solver import OPT_GNN_LOSS, OPT_PERSISTENT, OPT_PRECISION, GpuSolver

ORDERS = {"rcm": Mesh.RCM, "sfc": Mesh.SFC, "color": Mesh.COLOR, "none": 0}
CAP = 100000  # iteration cap of a solve that runs to its tolerance
RHO, MU, URF_U, URF_P = 1.0, 1e-3, 0.7, 0.3


def _case(name, kind, nx, ny, nz, **more):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, **more}


def listed():
    return [
        # the reference's own pressure solve (DIC-PCG to a 0.1 drop in at most 20
        # iterations) on a mesh the size of its 3-d cavity, from a host program
        _case("host_dic_6", "host", 6, 5, 6, order="rcm", imat=1, reduc=0.1, n_iter=20),
        # its two-component momentum solve on a 2-d channel (0.1 in at most 5)
        _case("momentum_2d_dilu", "bicg", 37, 42, 1, order="rcm", n_vc=2, precision=0, reduc=0.1,
              n_iter=5),
        # a small pressure system to the benchmarks' tolerance, plain Jacobi-PCG
        _case("jacobi_32", "cg", 32, 32, 32, order="rcm", imat=0, precision=0, persistent=0,
              reduc=1e-10, n_iter=CAP),
        # the reference's pressure solve at an ordinary size, odd edges
        _case("dic_63", "cg", 63, 64, 67, order="rcm", imat=1, precision=0, persistent=0, reduc=0.1,
              n_iter=20),
        # u, v, w of an outer iteration: BiCGSTAB + DILU, three components of one matrix
        _case("momentum_uvw_96", "bicg", 96, 96, 96, order="rcm", n_vc=3, precision=0, reduc=0.1,
              n_iter=5),
        # one momentum component to full accuracy, FP32 inner iterations, multicolour order
        _case("momentum_mixed_128", "bicg", 128, 128, 128, order="color", n_vc=1, precision=1,
              reduc=1e-12, n_iter=CAP),
        # the plain run of a reordered SIMPLE loop: DIC-PCG in multicolour order
        _case("dic_color_101", "cg", 101, 96, 100, order="color", imat=1, precision=0,
              persistent=0, reduc=1e-10, n_iter=CAP),
        # many uneven systems at once (per-block meshes)
        _case("batch_24", "batch", 0, 0, 0, n_sys=24, lo=2000, hi=100000, imat=0, precision=0,
              reduc=1e-10, n_iter=CAP),
        # the learned solve at the SIMPLE loop's ordinary size and near the benchmark's
        _case("learned_64", "fcg", 64, 64, 64, order="rcm", reduc=1e-12, n_iter=CAP),
        _case("learned_160", "fcg", 160, 160, 160, order="rcm", reduc=1e-12, n_iter=CAP),
        # everything of an outer iteration that is not a linear solve
        _case("outer_fv_80", "fv", 80, 80, 80, order="rcm"),
        # a training step at half the training size
        _case("train_33", "train", 33, 32, 31, order="rcm", loss=2, samples=4),
    ]


def _edges(rng, cells, flat):
    """Edge lengths of a mesh of about `cells` cells, uneven, one deep if flat."""
    n = cells ** (1.0 / (2 if flat else 3))
    e = [max(3, int(round(n * math.exp(rng.uniform(-0.25, 0.25))))) for _ in range(3)]
    return e[0], e[1], 1 if flat else e[2]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["cg", "cg", "cg", "host", "bicg", "bicg", "batch", "fcg", "fcg", "fv",
                       "train"])

    def cells(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    simple = rng.random() < 0.5  # the SIMPLE loop's tolerance, or full accuracy
    if kind in ("cg", "host"):
        top = 30000 if kind == "host" else 1000000
        nx, ny, nz = _edges(rng, cells(100, top), rng.random() < 0.2)
        c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz,
             "order": rng.choice(["rcm", "rcm", "sfc", "color", "none"]),
             "imat": rng.choice([0, 1, 1, 2]), "reduc": 0.1 if simple else 1e-10,
             "n_iter": 20 if simple else CAP}
        if kind == "cg":
            c["precision"] = 0
            c["persistent"] = int(c["imat"] == 0 and nx * ny * nz < 40000 and rng.random() < 0.5)
        return c
    if kind == "bicg":
        nx, ny, nz = _edges(rng, cells(200, 800000), rng.random() < 0.25)
        mixed = int(not simple and rng.random() < 0.5)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz,
                "order": rng.choice(["rcm", "rcm", "color", "none"]),
                "n_vc": rng.choice([1, 2, 3, 3, 4]), "precision": mixed,
                "reduc": 0.1 if simple else 1e-12 if mixed else 1e-10,
                "n_iter": 5 if simple else CAP}
    if kind == "batch":
        lo = int(cells(300, 4000))
        return {"kind": kind, "nx": 0, "ny": 0, "nz": 0, "n_sys": rng.randint(3, 40), "lo": lo,
                "hi": lo * rng.randint(3, 20), "imat": rng.choice([0, 0, 1]), "precision": 0,
                "reduc": 1e-10, "n_iter": CAP}
    if kind == "fcg":
        nx, ny, nz = _edges(rng, cells(4000, 2500000), False)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "order": rng.choice(["rcm", "color"]),
                "reduc": 1e-12, "n_iter": CAP}
    if kind == "fv":
        nx, ny, nz = _edges(rng, cells(1000, 800000), rng.random() < 0.2)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz,
                "order": rng.choice(["rcm", "color", "none"])}
    nx, ny, nz = _edges(rng, cells(8000, 60000), False)
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "order": "rcm",
            "loss": rng.choice([1, 2, 2]), "samples": rng.randint(1, 4)}


# ---- meshes and what a program keeps for one -------------------------------------------
def _mesh(nx, ny, nz, order, seed=0):
    m = Mesh.hex(nx, ny, nz, jitter=0.15, seed=seed, permute=True)
    if ORDERS[order]:
        m.renumber(ORDERS[order])
    return m


class _Kept:
    """One mesh's structure, base coefficients, solver (or geometry) and stream."""

    def __init__(self, case):
        self.kind = case["kind"]
        self.stream = torch.cuda.Stream()
        self.fv = self.solver = None
        if self.kind == "batch":
            sizes = batch_sizes(case["n_sys"], case["lo"], case["hi"])
            meshes = [_mesh(n, n, n, "rcm", 1000 + k) for k, n in enumerate(sizes)]
        else:
            meshes = [_mesh(case["nx"], case["ny"], case["nz"], case["order"])]
        if self.kind == "fv":
            self.fv = GpuFv(meshes[0])
            self.fv._lib.fv_gpu_set_stream(self.fv._h, self.stream.cuda_stream)
            self.geom = _geometry(meshes[0])
            self.n_cell = meshes[0].n_cell
            return
        if self.kind == "bicg":
            self.mats = [meshes[0].momentum()[0]]
        else:
            self.mats = [m.pressure(pin=0) for m in meshes]
            for A in self.mats:  # cell 1 pinned by zeroing its faces' coefficients
                A.p[(A.ip == 1) | (A.inb == 1)] = 0.0
                A.n[:] = A.p
        start = np.cumsum([0] + [A.n_cell for A in self.mats])
        self.n_cell = int(start[-1])
        self.ip = np.concatenate([A.ip - 1 + s for A, s in zip(self.mats, start)])
        self.inb = np.concatenate([np.where(A.inb > 0, A.inb - 1 + s, -1)
                                   for A, s in zip(self.mats, start)])
        self.p, self.n, self.pl = (np.concatenate([getattr(A, k) for A in self.mats])
                                   for k in ("p", "n", "pl"))
        self.sys = np.repeat(np.arange(len(self.mats)), np.diff(start))
        s = self.solver = GpuSolver()
        s.set_stream(self.stream.cuda_stream)
        s.set_option(OPT_PRECISION, case.get("precision", 0))
        s.set_option(OPT_PERSISTENT, case.get("persistent", 0))
        if self.kind == "batch":
            s.matrix_set_batch(self.mats)
        else:
            s.matrix_set(self.mats[0])
        if self.kind in ("fcg", "train"):
            s.gnn_set_params(load_params(DEFAULT_WEIGHTS))
            s.set_option(OPT_GNN_LOSS, case.get("loss", 1))
            s.mg_aggregates(1, self.n_cell)  # the hierarchy, built once per structure
        self.mats = None


_KEPT = {}


def _kept(case):
    key = tuple(sorted((k, v) for k, v in case.items()
                       if k not in ("name", "reduc", "n_iter", "samples", "n_vc", "imat")))
    if key not in _KEPT:
        while len(_KEPT) >= 2:
            _KEPT.pop(next(iter(_KEPT)))
        _KEPT[key] = _Kept(case)
    return _KEPT[key]


def _coefficients(k, rng):
    """New coefficients on a kept structure: every cell's own factor (the
    a_P of its velocity) taken to the faces; a new momentum flux."""
    inner = k.inb >= 0
    if k.kind == "bicg":
        f = rng.uniform(0.8, 1.0, k.p.size)
        return k.p * f, k.n * f, k.pl * rng.uniform(1.0, 1.1, k.n_cell)
    g = np.exp(rng.uniform(-0.3, 0.3, k.n_cell))
    f = np.zeros(k.p.size)
    f[inner] = 0.5 * (g[k.ip[inner]] + g[k.inb[inner]])
    p = k.p * f
    # the diagonal: minus the off-diagonals, and the pinned faces' share of the base
    kept = k.pl + np.bincount(k.ip, k.p, k.n_cell) + np.bincount(
        k.inb[inner], k.n[inner], k.n_cell)
    pl = (np.abs(kept) > 1e-9 * k.pl) * kept - np.bincount(k.ip, p, k.n_cell) - np.bincount(
        k.inb[inner], p[inner], k.n_cell)
    return p, p.copy(), pl


def _host_inputs(case, seed):
    """Everything a pass is given, as numpy arrays, and the kept structure."""
    k = _kept(case)
    rng = np.random.default_rng([int(seed), 12345])
    N = k.n_cell
    x = {}
    if k.kind == "fv":
        F = k.geom["ip"].size
        x["u"] = rng.uniform(-1, 1, (N, 3))
        x["pr"] = rng.uniform(-1, 1, N)
        x["pp"] = rng.uniform(-0.1, 0.1, N)
        x["wall"] = np.zeros((F, 3))
        x["wall"][k.geom["lid"], 0] = 1.0
        return k, x
    x["p"], x["n"], x["pl"] = _coefficients(k, rng)
    V = case.get("n_vc", 1)
    b = rng.uniform(-1, 1, (V, N))
    if k.kind != "bicg":  # a mass imbalance: each system's sum is zero, its first cell pinned
        n_of = np.bincount(k.sys)
        b[0] -= (np.bincount(k.sys, b[0]) / n_of)[k.sys]
        b[0, np.concatenate([[0], np.cumsum(n_of)[:-1]])] = 0.0
    x["b"] = b
    x["phi"] = rng.uniform(-1, 1, (N, V)) if k.kind == "bicg" else np.zeros((N, V))
    if k.kind == "train":
        x["samples"] = rng.uniform(-1, 1, (case["samples"], N))
        x["samples"][0] = b[0]
    return k, x


class _State:
    pass


def prepare(case, seed):
    k, x = _host_inputs(case, seed)
    s = _State()
    s.case, s.k = case, k
    if case["kind"] == "host":
        s.x = x
        s.phi = np.zeros((k.n_cell, 1))
        s.res = np.zeros((k.n_cell, 1), order="F")
        s.res_n = np.zeros(1)
        return s
    with torch.cuda.stream(k.stream):
        s.x = {name: torch.from_numpy(np.ascontiguousarray(a)).cuda() for name, a in x.items()}
        if case["kind"] not in ("fv", "train"):
            s.phi = torch.empty_like(s.x["phi"])
            s.res = torch.empty_like(s.x["b"])
        if case["kind"] == "fv":
            s.vol = torch.from_numpy(k.geom["vol"]).cuda()
            s.u, s.pr = torch.empty_like(s.x["u"]), torch.empty_like(s.x["pr"])
    k.stream.synchronize()
    return s


def run(s):
    c, k, x = s.case, s.k, s.x
    kind, g = c["kind"], k.solver
    if kind == "host":
        s.phi[:] = x["phi"]
        s.res[:, 0] = x["b"][0]
        g.matrix_values(x["p"], x["n"], x["pl"])
        g.solv_cg(c["imat"], c["reduc"], c["n_iter"], s.phi, s.res, s.res_n)
        return {"phi": s.phi, "res0": s.res, "res0_n": s.res_n}
    if kind == "fv":
        return _outer(s)
    with torch.cuda.stream(k.stream):
        g.matrix_values_dev(x["p"].data_ptr(), x["n"].data_ptr(), x["pl"].data_ptr())
        if kind == "train":
            loss = g.gnn_grad_dev(x["b"].data_ptr(), x["samples"].data_ptr(), c["samples"])
            return {"loss": loss, "grad": g.gnn_get_grad()}
        s.phi.copy_(x["phi"])
        s.res.copy_(x["b"])
        at = (s.phi.data_ptr(), s.res.data_ptr())
        if kind == "fcg":
            rn, _ = g.solv_fcg_dev(c["reduc"], c["n_iter"], *at)
        elif kind == "bicg":
            rn, _ = g.solv_bicg_dev(2, c["reduc"], c["n_iter"], c["n_vc"], *at)
        elif kind == "batch":
            rn = g.solv_batch_dev("cg", c["imat"], c["reduc"], c["n_iter"], 1, *at)["res0_n"]
        else:
            rn, _ = g.solv_cg_dev(c["imat"], c["reduc"], c["n_iter"], 1, *at)
    return {"phi": s.phi, "res0": s.res, "res0_n": rn}


def _outer(s):
    """One outer iteration's pieces, with the reference's explicit terms; the
    pressure correction is given instead of solved for."""
    k, x, fv = s.k, s.x, s.k.fv
    with torch.cuda.stream(k.stream):
        s.u.copy_(x["u"])
        s.pr.copy_(x["pr"])
        u, pr = s.u, s.pr
        gp = fv.gradient_sweeps(pr, 2, 2)
        p, n, pl, rhs, flux = fv.momentum_field(u, rho=RHO, mu=MU, u_lid=1.0, urf=URF_U)
        rhs -= gp * s.vol[:, None]
        gu = fv.gradient_sweeps(u, 2, 0, x["wall"])
        fv.momentum_deferred(u, gu, flux, MU, rhs)
        face = fv.face_flux(u, pr, gp, pl, RHO, aux=True)
        pc, _, pcl = fv.pressure_correction(pl, rho=RHO, pin=1)
        b, total = fv.mass_imbalance(face, pin=1)
        gpp = fv.gradient_sweeps(x["pp"], 2, 2)
        fv.simple_correct(x["pp"], gpp, pl, RHO, URF_P, u, pr, face)
    return {"p": p, "n": n, "pl": pl, "rhs": rhs, "pc": pc, "pcl": pcl, "b": b, "total": total,
            "u": u, "pr": pr, "flux": face}


# ---- the work a pass cannot do without ----------------------------------------------------
def _iterations(case, n):
    """Krylov iterations of a solve to its tolerance, from its order, its
    preconditioner and its longest edge."""
    if case["n_iter"] < CAP:
        return case["n_iter"]
    digits = -math.log10(case["reduc"]) / 10.0
    if case["kind"] == "fcg":
        return 35 * digits
    if case["kind"] == "bicg":
        return (25 if case["order"] == "color" else 9) * digits
    per_edge = 10.5 if case["imat"] == 0 else 6.0 if case.get("order") == "color" else 3.5
    return per_edge * n * digits


def work(case):
    """Per Krylov iteration the matrix once and each vector of the recurrence
    once; a pass's inputs and outputs once."""
    kind = case["kind"]
    if kind == "batch":
        sizes = [n ** 3 for n in batch_sizes(case["n_sys"], case["lo"], case["hi"])]
        parts = [(c, round(c ** (1 / 3))) for c in sizes]
    else:
        parts = [(case["nx"] * case["ny"] * case["nz"], max(case["nx"], case["ny"], case["nz"]))]
    total = flops = 0.0
    for N, edge in parts:
        F = 3 * N if case["nz"] != 1 else 2 * N  # interior faces
        if kind == "fv":  # geometry once per face and cell, every field once in and once out
            total += F * (8 + 80) + N * (32 + 8 * 3) + 8 * (N * 40 + F * 12)
            flops += 400.0 * F
            continue
        if kind == "train":  # network forward and backward, operator applications per sample
            total += 8 * (2 * F + N) + N * 32 * 4 * 20.0 + case["samples"] * 12 * (12 * F + 16 * N)
            flops += N * 3 * 2 * 2 * 32 * 32 * 3.0
            continue
        V = case.get("n_vc", 1)
        it = _iterations(case, edge)
        k = 2 if kind == "bicg" else 1
        fp = 4 if kind == "fcg" or case.get("precision") == 1 else 8
        mat = F * (8 + fp * k) + fp * N
        passes = 4 if kind == "fcg" else 2 if kind == "bicg" else 1
        sweeps = 0 if kind == "fcg" or (kind != "bicg" and case["imat"] == 0) else passes
        vec = {"fcg": 20, "bicg": 14}.get(kind, 9) * fp * N * V
        total += it * (passes * mat + sweeps * (mat + 2 * fp * N + 4 * fp * N * V) + vec)
        total += 8 * (F * k + N + 4 * N * V)
        flops += it * V * (passes + sweeps) * 4.0 * F
    return {"bytes": total, "flops": flops}


# ---- the same in plain 64-bit torch --------------------------------------------------------
def _csr(N, ip, inb, p, n, pl):
    """The face matrix as a sparse CSR tensor on the GPU, from its faces."""
    inner = inb >= 0
    a, b = ip[inner], inb[inner]
    d = np.arange(N)
    row = torch.from_numpy(np.concatenate([a, b, d]).astype(np.int64)).cuda()
    col = torch.from_numpy(np.concatenate([b, a, d]).astype(np.int64)).cuda()
    val = torch.from_numpy(np.concatenate([p[inner], n[inner], pl])).cuda()
    at = torch.argsort(row * N + col)
    ptr = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=N), 0)
    return torch.sparse_csr_tensor(ptr, col[at], val[at], (N, N), check_invariants=False)


def _solution(A, dinv, b, sys, n_sys):
    """Jacobi-PCG far past the cases' tolerances, each system its own scalars
    (BiCGSTAB is not needed: see _momentum_solution)."""
    def dot(u, v):
        return torch.zeros(n_sys, dtype=u.dtype, device=u.device).index_add_(0, sys, u * v)[sys] \
            if n_sys > 1 else (u * v).sum()
    x = torch.zeros_like(b)
    for _ in range(3):  # restarted on the true residual
        r = b - A @ x
        z = dinv * r
        p, rz = z.clone(), dot(r, z)
        r0 = r.abs().sum()
        for it in range(20000):
            q = A @ p
            al = rz / (dot(p, q) + 1e-300)
            x += al * p
            r -= al * q
            z = dinv * r
            new = dot(r, z)
            p = z + new / (rz + 1e-300) * p
            rz = new
            if it % 50 == 49 and float(r.abs().sum()) < 1e-13 * float(r0):
                break
    return x


def _momentum_solution(A, dinv, b):
    """Damped Jacobi: the momentum matrix is strictly diagonally dominant."""
    x = torch.zeros_like(b)
    r0 = float(b.abs().sum())
    for it in range(4000):
        r = b - A @ x
        x += dinv * r
        if it % 20 == 19 and float(r.abs().sum()) < 1e-15 * r0:
            break
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None  # the gradient of the bfloat16 network has no 64-bit counterpart
    k, x = _host_inputs(case, seed)
    if kind == "fv":
        return _exact_outer(k.geom, x)
    b, phi = (torch.from_numpy(x[n]).cuda() for n in ("b", "phi"))
    A = _csr(k.n_cell, k.ip, k.inb, x["p"], x["n"], x["pl"])
    r0 = (b - (A @ phi).t()).contiguous()
    n_sys = int(k.sys[-1]) + 1
    sys = torch.from_numpy(k.sys).cuda()
    rn = torch.stack([torch.zeros(n_sys, dtype=torch.float64, device="cuda").index_add_(
        0, sys, r.abs()) for r in r0], 1)
    sol = None
    if case["n_iter"] >= CAP:  # a solve to its tolerance has a solution to be near
        dinv = 1.0 / torch.from_numpy(x["pl"]).cuda()
        sol = torch.stack([_momentum_solution(A, dinv, v) if kind == "bicg" else
                           _solution(A, dinv, v, sys, n_sys) for v in b], 1)
    return {"phi": sol, "res0": r0.t() if kind == "host" else r0,
            "res0_n": rn if kind == "batch" else rn[0]}


def _geometry(m):
    ip, inb = m.faces()
    s, nrm, xf, l_pn, w = m.face_geom()
    xc, vol = m.cell_geom()
    lid = (inb == 0) & (nrm[:, 1] > 0.9) & (xf[:, 1] > 1.0 - 1e-9)
    return {"ip": ip - 1, "inb": inb - 1, "s": s, "nrm": nrm, "xf": xf, "l": l_pn, "w": w,
            "xc": xc, "vol": vol, "lid": lid}


def _exact_outer(geom, x):
    """_outer, from the finite-volume formulas."""
    G = {n: torch.from_numpy(np.ascontiguousarray(a)).cuda() for n, a in geom.items()}
    u, pr, pp, wall = (torch.from_numpy(x[n]).cuda() for n in ("u", "pr", "pp", "wall"))
    a, b = G["ip"].long(), G["inb"].long()
    I = torch.nonzero(b >= 0)[:, 0]
    a_i, b_i = a[I], b[I]
    w, s, l, nrm, vol, xc = G["w"], G["s"], G["l"], G["nrm"], G["vol"], G["xc"]
    N, F = vol.numel(), s.numel()
    zero = torch.zeros

    def new(*n):
        return zero(*n, dtype=torch.float64, device="cuda")

    def face(q):  # interpolated to the interior faces
        wi = w[I].reshape(-1, *[1] * (q.dim() - 1))
        return wi * q[b_i] + (1 - wi) * q[a_i]

    def scatter(out, f):  # + to the owner, - to the neighbour
        return out.index_add_(0, a_i, f).index_add_(0, b_i, -f)

    def aux(c, f):  # cell centre to its auxiliary point on the face
        t = ((G["xf"][f] - xc[c]) * nrm[f]).sum(1, keepdim=True)
        return G["xf"][f] - nrm[f] * t - xc[c]

    xa, xb = aux(a_i, I), aux(b_i, I)
    B = torch.nonzero(b < 0)[:, 0]

    def gradient(q, neu, bval=None):
        q2 = q.reshape(N, -1)
        g = None
        for _ in range(2):
            fi = face(q2)
            fb = q2[a[B]] if neu else bval[B]
            if g is not None:
                qa = q2[a_i] + (g[a_i] * xa[:, None]).sum(2)
                qb = q2[b_i] + (g[b_i] * xb[:, None]).sum(2)
                fi = w[I][:, None] * qb + (1 - w[I][:, None]) * qa
                if neu == 2:
                    fb = fb + (g[a[B]] * (G["xf"][B] - xc[a[B]])[:, None]).sum(2)
            t = scatter(new(N, q2.shape[1], 3), (fi * s[I][:, None])[:, :, None] * nrm[I][:, None])
            t.index_add_(0, a[B], (fb * s[B][:, None])[:, :, None] * nrm[B][:, None])
            g = t / vol[:, None, None]
        return g

    gp, gu, gpp = gradient(pr, 2), gradient(u, 0, wall), gradient(pp, 2)
    d = MU * s / l
    flux = RHO * s[I] * (face(u) * nrm[I]).sum(1)
    p, n = -d.clone(), new(F)
    p[I] += torch.clamp(flux, max=0.0)
    n[I] = -d[I] - torch.clamp(flux, min=0.0)
    pl = new(N).index_add_(0, a[B], d[B]).index_add_(0, a_i, -p[I]).index_add_(0, b_i, -n[I])
    pl /= URF_U
    rhs = (1 - URF_U) * pl[:, None] * u - gp[:, 0] * vol[:, None]
    lid = torch.nonzero(G["lid"])[:, 0]
    rhs[:, 0].index_add_(0, a[lid], d[lid])
    ua = u[a_i] + (gu[a_i] * xa[:, None]).sum(2)
    ub = u[b_i] + (gu[b_i] * xb[:, None]).sum(2)
    wi = w[I][:, None]
    up = torch.where(flux[:, None] > 0, u[a_i], u[b_i])
    cor = flux[:, None] * (up - (wi * ub + (1 - wi) * ua)) + d[I][:, None] * (
        (ub - ua) - (u[b_i] - u[a_i]))
    scatter(rhs, cor)
    dc = RHO * (w[I] / pl[b_i] + (1 - w[I]) / pl[a_i]) * s[I] * face(vol) / l[I]
    pa = pr[a_i] + (gp[a_i, 0] * xa).sum(1)
    pb = pr[b_i] + (gp[b_i, 0] * xb).sum(1)
    dp = pb - pa - (face(gp[:, 0]) * (xc[b_i] - xc[a_i])).sum(1)
    mass = flux - dc * dp
    bvec = -scatter(new(N), mass)
    bvec[0] = 0.0
    pc = new(F)
    pc[I] = -dc * ((a_i != 0) & (b_i != 0))
    out = new(F)
    out[I] = mass - dc * (pp[b_i] - pp[a_i])
    return {"p": p, "n": n, "pl": pl, "rhs": rhs, "pc": pc,
            "pcl": new(N).index_add_(0, a_i, dc).index_add_(0, b_i, dc), "b": bvec,
            "total": float(bvec.abs().sum()), "u": u - (vol / pl)[:, None] * gpp[:, 0],
            "pr": pr + URF_P * pp, "flux": out}
