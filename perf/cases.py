"""Performance cases of the SIMPLE solver and its linear solvers, driven through the Python
interface and the C entry points a program on this library calls.

kind "flow": a flow advanced by one outer iteration (NavierStokesSolver.iterate), the fields
going in from and coming back to page-locked host memory as in a coupled or restarted run.
Meshes are the repository's own: uniform hex cavities, cavities of jittered tets and the
conjugate-heat-transfer channel with k-epsilon; they are written once per machine into the
temporary directory.  The flow comes from the seed: a divergence-free velocity (the curl of
a vector potential that vanishes with its gradient on the walls), its face mass fluxes, a
smooth pressure and, in the channel, k, epsilon and temperatures.  Every pass starts from it.
Solver forms (the option sets that the benchmark and the tests use):
  fp64       the drop-in form, every recurrence in FP64; relative tolerance 1e-8, the p'
             solve capped at the reference's 1000 iterations
  mixed      FP32 recurrences with FP64 residuals in every equation, p' by Jacobi-CG
  multigrid  as mixed, p' by the aggregation-multigrid flexible CG
  learned    as multigrid, with a trained message-passing network on the second coarse level
The last three solve to 1e-11, where the FP32 recurrences no longer show in the fields.

kind "batch": hex cavities advanced together as one CUDA graph (CaseBatch).
kind "csr": a host CSR system solved on the GPU (csr_solve, the LASPack-style call).
kind "device": a CSR system in the caller's device memory (sysu_csr_cg_noalloc).
kind "train": Adam steps of the learned preconditioner (forward, backward, update).
The systems of the last three are 7-point operators with random face coefficients, as the
p' and momentum matrices of a hex mesh have.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from sysu_cfd_heat_gb300 import meshgen as mg
from sysu_cfd_heat_gb300._lib import LIB_PATH, Case, pinned_empty
from sysu_cfd_heat_gb300.batch import CaseBatch
from sysu_cfd_heat_gb300.learned import LearnedPreconditioner
from sysu_cfd_heat_gb300.solver import NavierStokesSolver, csr_solve

MIXED = {"p.mixed": 1, "mom.mixed": 1, "ke.mixed": 1, "t.mixed": 1, "ts.mixed": 1}
MULTIGRID = {**MIXED, "p.mixed": 0, "p.precond": 4}
FORMS = {
    "fp64": {"rtc": 1e-8, "p.maxit": 1000},
    "mixed": {"rtc": 1e-11, "p.maxit": 100000, **MIXED},
    "multigrid": {"rtc": 1e-11, "p.maxit": 100000, **MULTIGRID},
    "learned": {"rtc": 1e-11, "p.maxit": 100000, **MULTIGRID, "p.learned": 1, "p.learn_level": 2, "p.learn_iters": 2},
}
TRAIN_ITERS = 2   # outer iterations that train the network of the learned form
CHANNEL = dict(lx=2.0, ly_fluid=0.5, ly_solid=0.1, lz=0.5)
METHODS = {"CG": 1e-8, "BiCGSTAB": 1e-10}  # csr systems: relative tolerance
ADAM_STEPS = 4


def _flow_case(mesh, nx, ny, nz, form, ns=0):
    return dict(kind="flow", mesh=mesh, nx=nx, ny=ny, nz=nz, ns=ns, form=form)


def listed():
    return [
        # the smallest call: a caller's own device system of some 1,700 rows (a 12^3 cavity's p')
        dict(name="device CG 13x11x12", kind="device", nx=13, ny=11, nz=12),
        # LASPack's BiCGSTABIter on a host system of ordinary size, odd edges
        dict(name="csr BiCGSTAB 41x37x40", kind="csr", method="BiCGSTAB", nx=41, ny=37, nz=40),
        # the 24^3 lid-driven cavity (Re 100), the drop-in form: latency counts
        dict(name="cavity 24 fp64", **_flow_case("hex", 24, 24, 24, "fp64")),
        # the largest cavity of the many-cavity batch, on its own
        dict(name="cavity 64 mixed", **_flow_case("hex", 64, 64, 64, "mixed")),
        # the k-epsilon conjugate-heat-transfer channel: every equation of the iteration
        dict(name="channel fp64", **_flow_case("channel", 160, 40, 40, "fp64", 8)),
        dict(name="channel multigrid", **_flow_case("channel", 160, 40, 40, "multigrid", 8)),
        # the benchmark's mesh, 1,996,800 jittered tets: the drop-in form and the fast ones
        dict(name="tets 2M fp64", **_flow_case("tet", 80, 80, 52, "fp64")),
        dict(name="tets 2M mixed", **_flow_case("tet", 80, 80, 52, "mixed")),
        dict(name="tets 2M multigrid", **_flow_case("tet", 80, 80, 52, "multigrid")),
        # the learned form on an odd-sized mesh of 263,958 tets
        dict(name="tets 41x37x29 learned", **_flow_case("tet", 41, 37, 29, "learned")),
        # cavities of mixed size in one graph
        dict(name="batch 8 cavities", kind="batch", e0=40, e1=33, e2=28, e3=24, e4=21, e5=18, e6=14, e7=12),
        # the network's training step on a p' graph
        dict(name="train 60x48x44", kind="train", nx=60, ny=48, nz=44),
    ]


def draw(rng):
    def edges(lo, hi):
        """Three edges whose product is about a log-uniform size in [lo, hi]."""
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        e = cells ** (1 / 3)
        nx, ny = (max(4, round(e * rng.uniform(0.8, 1.25))) for _ in range(2))
        return dict(nx=nx, ny=ny, nz=max(4, round(cells / (nx * ny))))

    what = rng.choice(["flow", "flow", "flow", "flow", "flow", "batch", "csr", "device", "train"])
    if what == "flow":
        mesh, form = rng.choice(["hex", "tet", "channel"]), rng.choice(["fp64", "mixed", "multigrid"])
        if mesh == "channel":
            c = edges(8000, 500000)
            ny = max(6, c["ny"] // 2)
            return _flow_case(mesh, 2 * c["nx"], ny, c["nz"], form, max(2, ny // 5))
        e = edges(1728, 1000000) if mesh == "hex" else edges(500, 250000)  # tets: 6 a hex
        return _flow_case(mesh, e["nx"], e["ny"], e["nz"], rng.choice([form, "learned"]) if mesh == "tet" and e["nx"] > 15 else form)
    if what == "batch":
        return dict(kind="batch", **{"e%d" % k: rng.randint(12, 44) for k in range(8)})
    if what == "csr":
        return dict(kind="csr", method=rng.choice(list(METHODS)), **edges(1000, 300000))
    if what == "device":
        return dict(kind="device", **edges(500, 240000))
    return dict(kind="train", **edges(4000, 300000))


# --- meshes and flows ---------------------------------------------------------------------
def _param(case):
    """The case's param.in, its mesh written once per machine."""
    kind, nx, ny, nz, ns = (case[k] for k in ("mesh", "nx", "ny", "nz", "ns"))
    d = os.path.join(tempfile.gettempdir(), f"sysu_perf_{kind}_{nx}x{ny}x{nz}_{ns}")
    p = os.path.join(d, "param.in")
    if not os.path.exists(p):
        lid = {"y1": mg.INLET_ID}
        if kind == "hex":
            mesh, rows = mg.box_hex(nx, ny, nz, side_ids=lid), mg.cavity_param("x", 100000, mu=0.01)
        elif kind == "tet":
            mesh, rows = mg.lid_cavity_tet(nx, ny, nz), mg.cavity_param("x", 100000, mu=0.0025)
        else:
            mesh, rows = mg.cht_channel(nx, ny, ns, nz, **CHANNEL), mg.cht_param("x", 100000, nu=1e-5, k_solid=15.0)
        tmp = d + ".tmp%d" % os.getpid()
        mg.write_case(tmp, mesh, rows)
        try:
            os.rename(tmp, d)
        except OSError:
            pass  # another process was first
    return p


_geometry = {}


def _geom(param):
    """Cell centroids, face centroids and face area vectors of a mesh (host arrays)."""
    if param not in _geometry:
        c = Case(param)
        _geometry.clear()
        _geometry[param] = {k: c.array(k).reshape(-1, 3) for k in ("cell_x", "face_x", "face_n")}
        if c.info()["has_solid"]:
            _geometry[param]["solid_cell_x"] = c.array("solid_cell_x").reshape(-1, 3)
        c.close()
    return _geometry[param]


def _bump(s, n):
    """g and g' of g(s) = s^2 (1-s)^2 cos(n pi s): zero with its slope on both walls."""
    q, c, d = s * (1 - s), torch.cos(n * math.pi * s), torch.sin(n * math.pi * s)
    return q * q * c, 2 * q * (1 - 2 * s) * c - n * math.pi * q * q * d


def _velocity(x, lengths, origin, amp):
    """curl of psi_j = sum_m amp[j, m] g_a(s0) g_b(s1) g_c(s2), s the coordinates scaled to the box."""
    s = [(x[:, k] - origin[k]) / lengths[k] for k in range(3)]
    u = [torch.zeros_like(s[0]) for _ in range(3)]
    modes = [(0, 0, 0), (1, 0, 1), (0, 1, 2), (2, 1, 0), (1, 2, 1), (3, 0, 2)]
    for m, nm in enumerate(modes):
        g = [_bump(s[k], nm[k]) for k in range(3)]
        grad = []
        for k in range(3):
            t = [g[i][0] for i in range(3)]
            t[k] = g[k][1] / lengths[k]
            grad.append(t[0] * t[1] * t[2])
        for j in range(3):  # psi along axis j: u_{j+1} += d psi / d x_{j+2}, u_{j+2} -= d psi / d x_{j+1}
            a, b = (j + 1) % 3, (j + 2) % 3
            u[a] = u[a] + amp[j, m] * grad[b]
            u[b] = u[b] - amp[j, m] * grad[a]
    return u


def _scalar(x, lengths, origin, amp):
    """A smooth field: sum of cosine modes with the given amplitudes."""
    s = [(x[:, k] - origin[k]) / lengths[k] for k in range(3)]
    f = torch.zeros_like(s[0])
    for m, (a, b, c) in enumerate([(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (2, 0, 1), (1, 2, 1)]):
        f = f + amp[m] * torch.cos(a * math.pi * s[0]) * torch.cos(b * math.pi * s[1]) * torch.cos(c * math.pi * s[2])
    return f


def _flow(case, param, seed):
    """The starting fields by member name, as host arrays."""
    rng = np.random.default_rng(seed)
    G = _geom(param)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, xf, nf = (torch.from_numpy(G[k]).to(dev) for k in ("cell_x", "face_x", "face_n"))
    channel = case["mesh"] == "channel"
    L = (CHANNEL["lx"], CHANNEL["ly_fluid"], CHANNEL["lz"]) if channel else (1.0, 1.0, 1.0)
    o = (0.0, 0.0, 0.0)
    # a few tenths of the lid or inlet velocity
    amp = torch.from_numpy(rng.uniform(-1.0, 1.0, (3, 6))) * (1.0 if channel else 6.0)
    u, uf = _velocity(x, L, o, amp), _velocity(xf, L, o, amp)
    base = 1.0 if channel else 0.0
    out = {"U": u[0] + base, "V": u[1], "W": u[2],
           "P": _scalar(x, L, o, rng.uniform(-0.05, 0.05, 6)),
           "RUFace": (uf[0] + base) * nf[:, 0] + uf[1] * nf[:, 1] + uf[2] * nf[:, 2]}
    if channel:
        k0 = 1.5 * 0.05 ** 2
        e0 = 0.09 ** 0.75 * k0 ** 1.5 / 0.05
        a = rng.uniform(-0.1, 0.1, (4, 6))
        out["TE"] = k0 * torch.exp(_scalar(x, L, o, a[0]))
        out["ED"] = e0 * torch.exp(_scalar(x, L, o, a[1]))
        out["VisTur"] = 0.09 * out["TE"] ** 2 / out["ED"]
        out["T"] = 300.0 + 20.0 * torch.exp(_scalar(x, L, o, a[2])) * (1.0 - x[:, 1] / L[1])
        xs = torch.from_numpy(G["solid_cell_x"]).to(dev)
        out["solid_T"] = 350.0 + 20.0 * _scalar(xs, (L[0], CHANNEL["ly_solid"], L[2]), (0.0, -CHANNEL["ly_solid"], 0.0), a[3])
    return {k: v.cpu().numpy() for k, v in out.items()}


def _state_arrays(case, seed):
    """The starting fields and room for the results, in page-locked memory."""
    start, back = {}, {}
    for k, v in _flow(case, _param(case), seed).items():
        start[k] = pinned_empty(v.size)
        start[k][:] = v
        back[k] = pinned_empty(v.size)
    return start, back


# --- linear systems -----------------------------------------------------------------------
def _system(case, seed, skew=0.0):
    """(rowptr, col, val, x, b) of a 7-point operator with random face coefficients, a
    fixed value on one side and, with skew, an upwind part; b = A x in 64 bits."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    rng = np.random.default_rng(seed)
    idx = np.arange(n).reshape(nz, ny, nx)
    diag = np.zeros(n)
    rows, cols, vals = [], [], []
    for ax in range(3):
        a = np.take(idx, range(idx.shape[ax] - 1), axis=ax).ravel()
        b = np.take(idx, range(1, idx.shape[ax]), axis=ax).ravel()
        d, f = rng.uniform(0.5, 1.5, a.size), skew * rng.uniform(-1.0, 1.0, a.size)
        lo, up = -(d + np.maximum(f, 0.0)), -(d + np.maximum(-f, 0.0))
        rows += [a, b]
        cols += [b, a]
        vals += [up, lo]
        np.add.at(diag, a, -up)
        np.add.at(diag, b, -lo)
    first = idx[0].ravel()
    diag[first] += 2.0 * rng.uniform(0.5, 1.5, first.size)
    r = np.concatenate([np.arange(n)] + rows)
    c = np.concatenate([np.arange(n)] + cols)
    v = np.concatenate([diag] + vals)
    order = np.lexsort((c, r))
    r, c, v = r[order], c[order].astype(np.int32), v[order]
    rowptr = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    k = np.arange(n)
    x = np.sin(0.5 + 3.0 * rng.uniform() * k / n * math.pi) + 0.1 * rng.standard_normal(n)
    b = np.add.reduceat(v * x[c], rowptr[:-1])
    return rowptr, c, v, x, b


def _batch_edges(case):
    return [case["e%d" % k] for k in range(8)]


def _hex(n):
    return dict(mesh="hex", nx=n, ny=n, nz=n, ns=0)


# --- the interface ------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "flow":
        opts = dict(FORMS[case["form"]])
        s = NavierStokesSolver(_param(case), opts)
        if case["form"] == "learned":
            s.iterate(TRAIN_ITERS)
        start, back = _state_arrays(case, seed)
        return {"kind": kind, "solver": s, "start": start, "back": back}
    if kind == "batch":
        edges = _batch_edges(case)
        batch = CaseBatch([_param(_hex(e)) for e in edges], FORMS["mixed"])
        # SM shares by the cells of each case, as a program without time to tune them sets them
        total = sum(e ** 3 for e in edges)
        batch.set_caps([max(4, min(152, round(2 * 152 * e ** 3 / total))) for e in edges])
        batch.capture()
        both = [_state_arrays(_hex(e), seed + 1000 * k) for k, e in enumerate(edges)]
        return {"kind": kind, "batch": batch, "start": [a for a, _ in both], "back": [b for _, b in both]}
    if kind == "csr":
        rp, c, v, _, b = _system(case, seed, skew=1.0 if case["method"] == "BiCGSTAB" else 0.0)
        return {"kind": kind, "method": case["method"], "system": (rp, c, v, b)}
    rp, c, v, x, b = _system(case, seed)
    if kind == "device":
        fn = ctypes.CDLL(LIB_PATH).sysu_csr_cg_noalloc
        p = ctypes.c_void_p
        fn.argtypes = [ctypes.c_int, p, p, p, p, p, ctypes.c_int, ctypes.c_double, ctypes.c_double, p, p, p, p]
        d = [torch.from_numpy(a).cuda() for a in (rp, c, v, b)]
        return {"kind": kind, "call": fn, "rows": len(rp) - 1, "system": d, "x": torch.zeros_like(d[3])}
    net = LearnedPreconditioner(rp, c, v)
    net.init_params(seed)
    net.add_pair(b, x)
    return {"kind": kind, "net": net}


def run(state):
    kind = state["kind"]
    if kind == "flow":
        s, back = state["solver"], state["back"]
        for k, v in state["start"].items():
            s.set(k, v)
        s.iterate(1)
        for k, v in back.items():
            s.get(k, v)
        return back
    if kind == "batch":
        b = state["batch"]
        for s, start in zip(b.cases, state["start"]):
            for k, v in start.items():
                s.set(k, v)
        b.replay(1)
        b.check()
        for s, back in zip(b.cases, state["back"]):
            for k, v in back.items():
                s.get(k, v)
        return state["back"]
    if kind == "csr":
        rp, c, v, b = state["system"]
        x, _, _, _ = csr_solve(rp, c, v, b, method=state["method"], maxit=2000, eps=METHODS[state["method"]])
        return x
    if kind == "device":
        x, (rp, c, v, b) = state["x"].zero_(), state["system"]
        it, res, status = ctypes.c_int(), ctypes.c_double(), ctypes.c_int()
        code = state["call"](state["rows"], rp.data_ptr(), c.data_ptr(), v.data_ptr(), b.data_ptr(), x.data_ptr(), 2000,
                             1e-10, 1.0, torch.cuda.current_stream().cuda_stream, ctypes.addressof(it),
                             ctypes.addressof(res), ctypes.addressof(status))
        if code or status.value:
            raise RuntimeError("sysu_csr_cg_noalloc: code %d, status %d" % (code, status.value))
        return x
    state["net"].train(ADAM_STEPS, lr=1e-3, loss_kind=1)
    return state["net"].params


def exact(case, seed):
    """The linear systems have the solution that their right-hand side was made from; an
    outer iteration and a training step have no short one in plain numpy."""
    if case["kind"] == "csr":
        return _system(case, seed, skew=1.0 if case["method"] == "BiCGSTAB" else 0.0)[3]
    if case["kind"] == "device":
        return torch.from_numpy(_system(case, seed)[3])
    return None


def work(case):
    """Each input read once and each output written once, however many iterations the
    solves take: fields in and out, the mesh's geometry and the matrix of every equation."""
    kind = case["kind"]
    if kind in ("csr", "device", "train"):
        n = case["nx"] * case["ny"] * case["nz"]
        nnz = 7 * n - 2 * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nz"] * case["nx"])
        if kind == "train":  # four layers of width 32: forward, backward and weight gradients
            return {"bytes": ADAM_STEPS * (8.0 * nnz + 8 * 64.0 * n), "flops": ADAM_STEPS * 3.0 * 4 * 2 * 64 * 32 * n}
        return {"bytes": 12.0 * nnz + 16.0 * n, "flops": 2.0 * nnz}
    if kind == "batch":
        parts = [work(dict(kind="flow", form="mixed", **_hex(e))) for e in _batch_edges(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    hexes = case["nx"] * case["ny"] * case["nz"]
    cells, faces = (6 * hexes, 12 * hexes) if case["mesh"] == "tet" else (hexes, 3 * hexes)
    fields, equations = (9, 6) if case["mesh"] == "channel" else (4, 2)
    nnz = cells + 2 * faces
    return {"bytes": 16.0 * (fields * cells + faces) + 16 * 8.0 * faces + 12.0 * nnz * equations,
            "flops": 2.0 * nnz * (equations + 2) + 300.0 * faces}
