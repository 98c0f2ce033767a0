"""Timed cases of the framework's public entry points on one GPU.

Each case is one call that a finite-element program makes over and over (an assembly per
Newton iteration or load case, a recovery, a sensitivity, a solve), with the plan and the
buffers such a program keeps. `listed` holds the fixed cases, `draw` more of the same
ranges; `exact` gives the same outputs in plain 64-bit torch.
"""
import functools
import math

import numpy as np
import torch

from calculixpp_b200 import Batch, Material, Model, Plan, ThermalPlan, assemble_linear_static
from calculixpp_b200 import meshgen as mg

C3D4, C3D10, C3D8, C3D8R, C3D20, C3D20R, C3D6, C3D15 = range(8)
NAMES = ("C3D4", "C3D10", "C3D8", "C3D8R", "C3D20", "C3D20R", "C3D6", "C3D15")
PER_CELL = (6, 6, 1, 1, 1, 1, 2, 2)  # elements per hexahedral cell of a box mesh
E0, NU = 210000.0, 0.3


def listed():
    return [
        # the 320-hex cantilever, one assembly: the smallest model, where launches count
        _case("linear_c3d8_fp64_320", "linear", "C3D8", 20, 4, 4, "fp64"),
        # a model handed over once: mesh and loads on the host, CSR system back on the GPU
        _case("one_shot_c3d10_fp64", "one_shot", "C3D10", 23, 21, 17, "fp64"),
        # linear statics of an ordinary part with odd cell counts, FP64
        _case("linear_c3d20_fp64_odd", "linear", "C3D20", 41, 37, 33, "fp64"),
        # the benchmark's block: 262,144 quadratic hexes, mixed precision
        _case("linear_c3d20_mixed_64", "linear", "C3D20", 64, 64, 64, "mixed"),
        # one Newton iteration of the largest plasticity model, FP64
        _case("newton_c3d8_fp64_128", "newton", "C3D8", 128, 128, 128, "fp64"),
        # a Newton iteration of a mid-sized part, mixed, its history read back for output
        _case("newton_c3d8_mixed_history", "newton", "C3D8", 63, 47, 53, "mixed", history=True),
        # many small models of five element types in one graph
        dict(name="batch_mixed_24", kind="batch", models=24, low=1000, high=40000, order=3, precision="mixed"),
        # consistent mass matrix of a tetrahedral mesh (dynamics, eigenvalues)
        _case("mass_c3d10", "mass", "C3D10", 31, 25, 19, "fp64"),
        # heat conduction with prescribed temperatures and nodal flux, wedges and odd sizes
        _case("conduction_c3d15", "conduction", "C3D15", 45, 35, 27, "fp64"),
        # stresses, strains and reactions after a solve
        _case("recover_c3d20r", "recover", "C3D20R", 49, 41, 37, "fp64"),
        # design sensitivities of the 96 x 96 x 48 cantilever
        _case("adjoint_c3d8", "adjoint", "C3D8", 96, 96, 48, "fp64"),
        # iterative solve of an assembled block
        _case("solve_cg_c3d8", "solve", "C3D8", 45, 40, 35, "fp64"),
    ]


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "newton", "newton", "batch", "mass", "conduction", "recover",
                       "adjoint", "solve", "one_shot"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return dict(kind="batch", models=rng.randint(3, 24), low=300, high=rng.randint(2000, 30000),
                    order=rng.randint(0, 10**6), precision=precision)
    if kind in ("mass", "conduction", "solve", "recover", "adjoint"):
        precision = "fp64"
    types = {"recover": [C3D4, C3D8, C3D20, C3D20R, C3D6, C3D15], "adjoint": [C3D8, C3D20, C3D20R, C3D6, C3D15],
             "solve": [C3D8, C3D20R, C3D6]}.get(kind, list(range(8)))
    t = rng.choice(types)
    # elements over the range's logarithm; the box's sides apart by up to a factor of about two
    top = 20000 if kind == "solve" else 60000 if t in (C3D20, C3D15, C3D10) else 200000
    cells = math.exp(rng.uniform(math.log(300), math.log(top))) / PER_CELL[t]
    side = cells ** (1.0 / 3.0)
    nx, ny = (max(2, round(side * math.exp(rng.uniform(-0.35, 0.35)))) for _ in range(2))
    nz = max(2, round(cells / (nx * ny)))
    return _case(None, kind, NAMES[t], nx, ny, nz, precision, history=kind == "newton" and rng.random() < 0.5)


def _case(name, kind, elem, nx, ny, nz, precision, history=False):
    c = dict(kind=kind, elem=elem, nx=nx, ny=ny, nz=nz, precision=precision)
    if kind == "newton":
        c["history"] = history
    if name:
        c["name"] = name
    return c


# ---- inputs -----------------------------------------------------------------------------

@functools.lru_cache(maxsize=2)
def _box(t, nx, ny, nz):
    return mg.box_mesh(t, nx, ny, nz, float(nx), float(ny), float(nz))


def _mesh(t, nx, ny, nz, rng):
    """A box of unit cells, its inner nodes moved at random."""
    b = _box(t, nx, ny, nz)
    amount = 0.05 if t in (C3D8, C3D8R, C3D20, C3D20R, C3D6) else 0.015
    x = b.coords
    inner = np.all((x > 1e-9) & (x < np.array([nx, ny, nz]) - 1e-9), axis=1)
    x = x + rng.uniform(-amount, amount, x.shape) * inner[:, None]
    return mg.Mesh(coords=x, conn=b.conn, etype=t)


def _inputs(case, seed):
    """The model and what goes with it, on the host, from the seed alone."""
    rng = np.random.default_rng([seed, 17])
    t = NAMES.index(case["elem"])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = _mesh(t, nx, ny, nz, rng)
    kind = case["kind"]
    out = {}
    if kind == "newton":
        m.coords = m.coords / np.array([nx, ny, nz])
        m.young, m.poisson = np.full(m.n_elems, E0), np.full(m.n_elems, NU)
        eps = 0.005 * rng.uniform(0.95, 1.05)
        x = m.coords
        sn = np.concatenate([np.flatnonzero(x[:, 0] < 1e-9), np.flatnonzero(x[:, 0] > 1 - 1e-9), [0, 0]])
        sc = np.zeros(sn.size, np.int64)
        sc[-2:] = 1, 2
        out["u_last"] = mg.graded_uniaxial_field(x, 0.9 * eps)
        out["u"] = mg.graded_uniaxial_field(x, eps)
        out["model"] = Model(m, [Material(E0, NU, mg.j2_table())], None, (sn, sc, out["u"][3 * sn + sc]), None)
        return out
    m.young = E0 * np.exp(0.3 * rng.standard_normal(m.n_elems))
    m.poisson = rng.uniform(0.25, 0.35, m.n_elems)
    bottom = np.flatnonzero(m.coords[:, 2] < 1e-9)
    top = np.flatnonzero(m.coords[:, 2] > nz - 1e-9)
    if kind == "conduction":
        out["mesh"] = m
        out["tbc"] = (bottom, rng.uniform(280.0, 320.0, bottom.size))
        out["k"] = rng.uniform(10.0, 50.0, m.n_elems)
        out["flux"] = rng.uniform(0.0, 5.0, m.n_nodes)
        return out
    sn, sc = np.repeat(bottom, 3), np.tile(np.arange(3), bottom.size)
    sv = rng.uniform(-1e-3, 1e-3, sn.size) if kind in ("linear", "one_shot") else np.zeros(sn.size)
    load = (top, np.zeros(top.size, np.int64), rng.uniform(0.5, 1.5, top.size) / top.size)
    out["model"] = Model(m, [Material(E0, NU)], None, (sn, sc, sv), load)
    out["density"] = rng.uniform(2.0e-9, 8.0e-9, m.n_elems)
    out["u_field"] = rng.standard_normal(3 * m.n_nodes) * 1e-3
    return out


def _batch_inputs(case, seed):
    shape = np.random.default_rng(case["order"])  # types and sizes belong to the case
    rng = np.random.default_rng([seed, 23])
    models = []
    for _ in range(case["models"]):
        t = int(shape.choice([C3D8, C3D8R, C3D20R, C3D6, C3D15]))
        cells = math.exp(shape.uniform(math.log(case["low"]), math.log(case["high"]))) / PER_CELL[t]
        nx = max(1, round(cells ** (1.0 / 3.0)))
        nz = max(1, round(cells / nx**2))
        b = mg.box_mesh(t, nx, nx, nz, float(nx), float(nx), float(nz))
        x = b.coords
        inner = np.all((x > 1e-9) & (x < np.array([nx, nx, nz]) - 1e-9), axis=1)
        m = mg.Mesh(coords=x + rng.uniform(-0.02, 0.02, x.shape) * inner[:, None], conn=b.conn, etype=t)
        E, nu = float(rng.uniform(70000.0, 210000.0)), float(rng.uniform(0.25, 0.35))
        m.young, m.poisson = np.full(m.n_elems, E), np.full(m.n_elems, nu)
        top = np.flatnonzero(x[:, 2] > nz - 1e-9)
        models.append(Model(m, [Material(E, nu)], None, mg.clamp_face_spc(m, 2, 0.0),
                            (top, np.zeros(top.size, np.int64), np.full(top.size, 1.0 / top.size))))
    return models


def _on_gpu(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = Batch(_batch_inputs(case, seed), case["precision"])
        vals, rhs = b.buffers()
        return dict(kind=kind, batch=b, f=_on_gpu(b.load_vector()), vals=vals, rhs=rhs)
    i = _inputs(case, seed)
    s = dict(kind=kind)
    if kind == "one_shot":
        s.update(model=i["model"], precision=case["precision"])
        return s
    if kind == "conduction":
        p = ThermalPlan(i["mesh"], *i["tbc"])
        s.update(plan=p, k=_on_gpu(i["k"]), flux=_on_gpu(i["flux"]))
    else:
        p = s["plan"] = Plan(i["model"], case["precision"])
    s["vals"] = torch.empty(p.nnz, dtype=torch.float64, device="cuda")
    s["rhs"] = torch.empty(p.n_free, dtype=torch.float64, device="cuda")
    if kind == "linear":
        s["f"] = _on_gpu(i["model"].external_load_vector())
    elif kind == "newton":
        s["f_int"] = torch.empty(3 * i["model"].mesh.n_nodes, dtype=torch.float64, device="cuda")
        s["u"], s["history"] = _on_gpu(i["u"]), case["history"]
        p.assemble_tangent(_on_gpu(i["u_last"]), vals=s["vals"], f_int=s["f_int"], rhs=s["rhs"])
        p.commit()
    elif kind == "mass":
        s["density"] = _on_gpu(i["density"])
    elif kind in ("recover", "adjoint"):
        s["u"], s["f"] = _on_gpu(i["u_field"]), _on_gpu(i["model"].external_load_vector())
    elif kind == "solve":
        p.assemble_linear(_on_gpu(i["model"].external_load_vector()), vals=s["vals"], rhs=s["rhs"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "linear":
        return s["plan"].assemble_linear(s["f"], vals=s["vals"], rhs=s["rhs"], check=False)
    if kind == "one_shot":
        r = assemble_linear_static(s["model"], s["precision"])
        return r.row_ptr, r.col_idx, r.vals, r.rhs
    if kind == "newton":
        out = s["plan"].assemble_tangent(s["u"], vals=s["vals"], f_int=s["f_int"], rhs=s["rhs"], check=False)
        return out + (s["plan"].state(committed=False),) if s["history"] else out
    if kind == "batch":
        return s["batch"].graph_launch(s["f"], s["vals"], s["rhs"])
    if kind == "mass":
        return s["plan"].assemble_mass(s["density"], vals=s["vals"], check=False)
    if kind == "conduction":
        return s["plan"].assemble_conduction(s["k"], s["flux"], vals=s["vals"], rhs=s["rhs"], check=False)
    if kind == "recover":
        return s["plan"].recover_fields(s["u"], s["f"])
    if kind == "adjoint":
        return s["plan"].adjoint_compliance(s["u"])
    return s["plan"].solve_cg(s["vals"], s["rhs"], rtol=1e-12, max_iter=5000)[0]


# ---- the work a pass cannot do without ------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _small(t, nx, ny, nz):
    m = mg.box_mesh(t, nx, ny, nz)
    n = m.conn.shape[1]
    keys = m.conn.astype(np.int64)[:, :, None] * m.n_nodes + m.conn[:, None, :]
    return m.n_nodes, np.unique(keys.reshape(-1)).size, n


def _counts(t, nx, ny, nz):
    """(nodes, node pairs, elements, nodes per element): both counts are linear in each of
    the box's three cell counts, so eight small boxes give them for all."""
    total = np.zeros(2)
    for c in range(8):
        pick = [(c >> d) & 1 for d in range(3)]
        w = math.prod((v - 1) if hi else (2 - v) for v, hi in zip((nx, ny, nz), pick))
        total += w * np.array(_small(t, 1 + pick[0], 1 + pick[1], 1 + pick[2])[:2])
    return int(total[0]), int(total[1]), PER_CELL[t] * nx * ny * nz, _small(t, 1, 1, 1)[2]


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = dict(bytes=0, flops=0)
        shape = np.random.default_rng(case["order"])
        for _ in range(case["models"]):
            t = int(shape.choice([C3D8, C3D8R, C3D20R, C3D6, C3D15]))
            cells = math.exp(shape.uniform(math.log(case["low"]), math.log(case["high"]))) / PER_CELL[t]
            nx = max(1, round(cells ** (1.0 / 3.0)))
            w = work(_case(None, "linear", NAMES[t], nx, nx, max(1, round(cells / nx**2)), "mixed"))
            total = {k: total[k] + w[k] for k in total}
        return total
    t = NAMES.index(case["elem"])
    N, pairs, E, n = _counts(t, case["nx"], case["ny"], case["nz"])
    q = mg.NGP[t]
    grad = E * q * (36 * n + 60)           # Jacobian, inverse and gradients
    block = E * q * n * (n + 1) // 2 * 18  # 3x3 blocks of the upper triangle
    mesh = 4 * n * E + 24 * N
    if kind == "linear":
        return dict(bytes=mesh + 16 * E + 24 * N + 72 * pairs + 24 * N, flops=grad + block)
    if kind == "one_shot":  # values, column indices and row pointers written, the mesh read
        return dict(bytes=mesh + 16 * E + 36 * N + 108 * pairs + 48 * N, flops=grad + block)
    if kind == "newton":
        history = 104 * E * q if case["history"] else 0
        return dict(bytes=mesh + 16 * E + 24 * N + 72 * pairs + 48 * N + 112 * E * q + history,
                    flops=grad + 18 * n * E * q + 2 * block)
    if kind == "mass":
        return dict(bytes=mesh + 8 * E + 72 * pairs, flops=grad + E * q * n * (n + 1) * 2)
    if kind == "conduction":
        return dict(bytes=mesh + 8 * E + 16 * N + 8 * pairs, flops=grad + E * q * n * (n + 1) * 3)
    if kind == "recover":
        return dict(bytes=mesh + 16 * E + 48 * N + 120 * N, flops=grad + E * q * n * 36)
    if kind == "adjoint":
        return dict(bytes=mesh + 24 * E + 48 * N, flops=grad + E * q * n * 36)
    # about 100 + 6 sides iterations, each of which reads the matrix and its columns once
    it = 100 + 6 * max(case["nx"], case["ny"], case["nz"])
    return dict(bytes=it * (108 * pairs + 250 * N), flops=it * (18 * pairs + 30 * N))


# ---- the same outputs in 64 bits ---------------------------------------------------------------

_CORNERS = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]
_EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]


def _shape(t, r):
    """Shape functions of family t at the natural point r (a 3-vector)."""
    x, y, z = r
    if t in (C3D8, C3D8R):
        return torch.stack([(1 + a * x) * (1 + b * y) * (1 + c * z) / 8 for a, b, c in _CORNERS])
    if t in (C3D20, C3D20R):
        N = [(1 + a * x) * (1 + b * y) * (1 + c * z) * (a * x + b * y + c * z - 2) / 8 for a, b, c in _CORNERS]
        for i, j in _EDGES:
            f = 0.25
            for d in range(3):
                p = (_CORNERS[i][d] + _CORNERS[j][d]) // 2
                f = f * ((1 + p * r[d]) if p else (1 - r[d] * r[d]))
            N.append(f)
        return torch.stack(N)
    if t in (C3D4, C3D10):
        L = [1 - x - y - z, x, y, z]
        if t == C3D4:
            return torch.stack(L)
        return torch.stack([v * (2 * v - 1) for v in L]
                           + [4 * L[i] * L[j] for i, j in ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))])
    L = [1 - x - y, x, y]
    if t == C3D6:
        return torch.stack([v * (1 + s * z) / 2 for s in (-1, 1) for v in L])
    N = [v * (1 + s * z) * (2 * v + s * z - 2) / 2 for s in (-1, 1) for v in L]
    N += [2 * L[i] * L[j] * (1 + s * z) for s in (-1, 1) for i, j in ((0, 1), (1, 2), (2, 0))]
    return torch.stack(N + [v * (1 - z * z) for v in L])


def _rule(t):
    a, b = 1 / math.sqrt(3.0), math.sqrt(0.6)
    if t in (C3D8, C3D20R):
        return [(x, y, z, 1.0) for z in (-a, a) for y in (-a, a) for x in (-a, a)]
    if t == C3D8R:
        return [(0.0, 0.0, 0.0, 8.0)]
    if t == C3D20:
        line = ((-b, 5 / 9), (0.0, 8 / 9), (b, 5 / 9))
        return [(x, y, z, u * v * w) for z, w in line for y, v in line for x, u in line]
    if t == C3D4:
        return [(0.25, 0.25, 0.25, 1 / 6)]
    if t == C3D10:
        p, q = (5 - math.sqrt(5.0)) / 20, (5 + 3 * math.sqrt(5.0)) / 20
        return [(p, p, p, 1 / 24), (q, p, p, 1 / 24), (p, q, p, 1 / 24), (p, p, q, 1 / 24)]
    if t == C3D6:
        return [(1 / 3, 1 / 3, z, 0.5) for z in (-a, a)]
    return [(x, y, z, 1 / 6) for z in (-a, a) for x, y in ((1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3))]


@functools.lru_cache(maxsize=None)
def _tables(t):
    """(weights [q], values [q, n], natural derivatives [q, n, 3]) of family t."""
    w, N, dN = [], [], []
    for *r, v in _rule(t):
        r = torch.tensor(r, dtype=torch.float64)
        w.append(v)
        N.append(_shape(t, r))
        dN.append(torch.autograd.functional.jacobian(lambda y: _shape(t, y), r))
    return torch.tensor(w, dtype=torch.float64), torch.stack(N), torch.stack(dN)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, kind=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=_device()).to(kind)


def _gradients(t, x):
    """s = det J w [e, q] and the physical gradients [e, q, n, 3] of elements x [e, n, 3]."""
    w, _, dN = (v.to(x.device) for v in _tables(t))
    J = torch.einsum("eni,qnj->eqij", x, dN)
    return torch.linalg.det(J) * w, torch.einsum("qnj,eqji->eqni", dN, torch.linalg.inv(J))


def _lame(E, nu):
    return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))


def _gram(g, s):
    """sum_q s g_a (x) g_b as [e, a, i, b, j]."""
    e, q, n, _ = g.shape
    V = g.reshape(e, q, 3 * n)
    return torch.bmm((V * s[:, :, None]).transpose(1, 2), V).reshape(e, n, 3, n, 3)


def _blocks(G_lam, G_mu):
    K = G_lam + G_mu.transpose(2, 4)
    tr = torch.einsum("eaibi->eab", G_mu)
    for i in range(3):
        K[:, :, i, :, i] += tr
    return K


def _stiffness(t, x, E, nu):
    s, g = _gradients(t, x)
    lam, mu = _lame(E, nu)
    G = _gram(g, s)
    K = _blocks(G * lam[:, None, None, None, None], G * mu[:, None, None, None, None])
    if t == C3D8R:
        h = torch.tensor([[1, 1, -1, -1, -1, -1, 1, 1], [1, -1, -1, 1, -1, 1, 1, -1], [1, -1, 1, -1, 1, -1, 1, -1],
                          [-1, 1, -1, 1, 1, -1, 1, -1]], dtype=torch.float64, device=x.device)
        gam = h - torch.einsum("aj,ejd,ekd->eak", h, x, g[:, 0])
        kappa = 0.05 * mu * s[:, 0] * (g[:, 0] ** 2).sum((1, 2))
        H = torch.einsum("e,eka,ekb->eab", kappa, gam, gam)
        for i in range(3):
            K[:, :, i, :, i] += H
    return K


def _return_mapping(eps, state, lam, mu):
    """Radial return with linear isotropic hardening (engineering shear strains)."""
    h, sy = mg.J2_H, mg.J2_SY
    el = eps - state[..., :6]
    tr = el[..., :3].sum(-1, keepdim=True)
    sig = torch.cat([lam * tr + 2 * mu * el[..., :3], mu * el[..., 3:]], -1)
    p = sig[..., :3].mean(-1, keepdim=True)
    dev = torch.cat([sig[..., :3] - p, sig[..., 3:]], -1)
    norm = torch.sqrt((dev[..., :3] ** 2).sum(-1) + 2 * (dev[..., 3:] ** 2).sum(-1))
    f = math.sqrt(1.5) * norm - (sy + h * state[..., 6])
    pl = f > 0
    dg = torch.where(pl, f / (3 * mu + h), torch.zeros_like(f))
    N = dev / torch.where(norm > 0, norm, torch.ones_like(norm))[..., None]
    out = state.clone()
    out[..., :3] += math.sqrt(1.5) * dg[..., None] * N[..., :3]
    out[..., 3:6] += 2 * math.sqrt(1.5) * dg[..., None] * N[..., 3:]
    out[..., 6] += dg
    sig = sig - 2 * mu * math.sqrt(1.5) * dg[..., None] * N
    shrink = torch.where(pl, 2 * mu * math.sqrt(1.5) * dg / torch.where(norm > 0, norm, torch.ones_like(norm)),
                         torch.zeros_like(dg))
    c = torch.where(pl, 2 * mu * (1 / (1 + h / (3 * mu)) - shrink), torch.zeros_like(dg))
    return sig, out, lam + 2 / 3 * shrink * mu, mu * (1 - shrink), c, N


def _sym(v):
    """Voigt xx, yy, zz, xy, xz, yz as 3 x 3."""
    return v[..., [0, 3, 4, 3, 1, 5, 4, 5, 2]].reshape(v.shape[:-1] + (3, 3))


def _voigt_strain(H):
    return torch.stack([H[..., 0, 0], H[..., 1, 1], H[..., 2, 2], H[..., 0, 1] + H[..., 1, 0],
                        H[..., 0, 2] + H[..., 2, 0], H[..., 1, 2] + H[..., 2, 1]], -1)


def _tangent(s, g, u, state, lam, mu):
    """(K_e, f_e, new history) of elements with the return mapping above."""
    eps = _voigt_strain(torch.einsum("eni,eqnj->eqij", u, g))
    sig, new, lt, mt, c, N = _return_mapping(eps, state, lam, mu)
    m = torch.einsum("eqij,eqnj->eqni", _sym(N), g)
    K = _blocks(_gram(g, s * lt) - _gram(m, s * c), _gram(g, s * mt))
    f = torch.einsum("eq,eqij,eqnj->eni", s, _sym(sig), g)
    return K, f, new


def _system(conn, N, free, pre, element_blocks, step):
    """Reduced CSR system of 3 x 3 element blocks: row_ptr, col_idx, vals, K_fc u_c."""
    conn = _t(conn, torch.int64)
    E, n = conn.shape
    keys = (conn[:, :, None] * N + conn[:, None, :]).reshape(-1)
    pair, where = torch.unique(keys, return_inverse=True)
    B = torch.zeros(pair.numel(), 9, dtype=torch.float64, device=conn.device)
    for e in range(0, E, step):
        K = element_blocks(slice(e, e + step))  # [e, a, i, b, j]
        k = K.permute(0, 1, 3, 2, 4).reshape(-1, 9)
        B.index_add_(0, where[e * n * n:e * n * n + k.shape[0]], k)
    del keys, where
    B = B.view(-1, 3, 3)
    a, b = pair // N, pair % N
    free = _t(free, torch.bool)
    nf = free.sum(1)
    length = torch.zeros(N, dtype=torch.int64, device=a.device).index_add_(0, a, nf[b])
    size = nf * length
    base = torch.cumsum(size, 0) - size
    width = torch.cumsum(nf[b], 0) - nf[b]
    first = torch.cumsum(length, 0) - length
    off = width - first[a]
    rank = torch.cumsum(free.long(), 1) - free.long()
    eq = torch.cumsum(nf, 0) - nf
    nnz = int(size.sum())
    vals = torch.empty(nnz, dtype=torch.float64, device=a.device)
    cols = torch.empty(nnz, dtype=torch.int32, device=a.device)
    for i in range(3):
        for j in range(3):
            on = free[a, i] & free[b, j]
            at = (base[a] + rank[a, i] * length[a] + off + rank[b, j])[on]
            vals[at] = B[on, i, j]
            cols[at] = (eq[b] + rank[b, j])[on].to(torch.int32)
    rows = length[:, None].expand(N, 3)[free]
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=a.device), torch.cumsum(rows, 0)])
    moved = torch.zeros(N, 3, dtype=torch.float64, device=a.device)
    moved.index_add_(0, a, torch.einsum("mij,mj->mi", B, _t(pre).reshape(N, 3)[b]))
    return ptr, cols, vals, moved[free]


def _model_system(model, element_blocks=None):
    m = model.mesh
    t = m.etype
    deq, pre, _ = model.dof_map()
    free = deq.reshape(-1, 3) >= 0
    x, conn = _t(m.coords), _t(m.conn, torch.int64)
    E, nu = _t(m.young), _t(m.poisson)
    blocks = element_blocks or (lambda c: _stiffness(t, x[conn[c]], E[c], nu[c]))
    ptr, cols, vals, moved = _system(m.conn, m.n_nodes, free, pre, blocks, 8192)
    return ptr, cols, vals, _t(model.external_load_vector()).reshape(-1, 3)[_t(free, torch.bool)] - moved


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        models = _batch_inputs(case, seed)
        parts = [_model_system(m) for m in sorted(models, key=lambda m: m.mesh.etype)]
        return torch.cat([p[2] for p in parts]), torch.cat([p[3] for p in parts])
    i = _inputs(case, seed)
    if kind == "conduction":
        return _conduction(i)
    model = i["model"]
    m = model.mesh
    t = m.etype
    x, conn = _t(m.coords), _t(m.conn, torch.int64)
    E, nu = _t(m.young), _t(m.poisson)
    if kind == "linear":
        return _model_system(model)[2:]
    if kind == "one_shot":
        return _model_system(model)
    if kind == "newton":
        return _newton(case, i, model, x, conn)
    if kind == "mass":
        return _mass(i, model, x, conn)
    if kind == "solve":
        return _solve(*_model_system(model))
    u = _t(i["u_field"]).reshape(-1, 3)
    lam, mu = _lame(E, nu)
    node_sum = [torch.zeros(m.n_nodes, k, dtype=torch.float64, device=x.device) for k in (6, 6, 3)]
    dE, dX = torch.empty_like(E), torch.zeros_like(x)
    for e in range(0, m.n_elems, 16384):
        c = slice(e, e + 16384)
        s, g = _gradients(t, x[conn[c]])
        H = torch.einsum("eni,eqnj->eqij", u[conn[c]], g)
        eps = _voigt_strain(H)
        l, w = lam[c, None, None], mu[c, None, None]
        sig = torch.cat([l * eps[..., :3].sum(-1, keepdim=True) + 2 * w * eps[..., :3], w * eps[..., 3:]], -1)
        at = conn[c].reshape(-1)
        if kind == "recover":
            n = conn.shape[1]
            f = torch.einsum("eq,eqij,eqnj->eni", s, _sym(sig), g)
            for total, v in zip(node_sum, (eps.mean(1), sig.mean(1))):
                total.index_add_(0, at, v[:, None].expand(-1, n, -1).reshape(-1, 6))
            node_sum[2].index_add_(0, at, f.reshape(-1, 3))
        else:
            W = (sig * eps).sum(-1)
            dE[c] = -(s * W).sum(1) / E[c]
            M = W[..., None, None] * torch.eye(3, dtype=torch.float64, device=x.device)
            M = s[..., None, None] * (M - 2 * torch.einsum("eqia,eqib->eqab", H, _sym(sig)))
            dX.index_add_(0, at, -torch.einsum("eqab,eqnb->ena", M, g).reshape(-1, 3))
    if kind == "adjoint":
        return dE, dX
    count = torch.bincount(conn.reshape(-1), minlength=m.n_nodes)[:, None].double()
    return (node_sum[0] / count, node_sum[1] / count,
            node_sum[2] - _t(model.external_load_vector()).reshape(-1, 3))


def _newton(case, i, model, x, conn):
    m, t = model.mesh, model.mesh.etype
    if t == C3D8R:
        return None  # the hourglass terms follow the last point's tangent modulus
    q = mg.NGP[t]
    lam, mu = _lame(E0, NU)
    u0, u1 = (_t(i[k]).reshape(-1, 3) for k in ("u_last", "u"))
    f_int = torch.zeros(m.n_nodes, 3, dtype=torch.float64, device=x.device)
    history = torch.empty(m.n_elems, q, 13, dtype=torch.float64, device=x.device) if case["history"] else None

    def blocks(c):
        s, g = _gradients(t, x[conn[c]])
        zero = torch.zeros(g.shape[0], q, 13, dtype=torch.float64, device=x.device)
        state = _tangent(s, g, u0[conn[c]], zero, lam, mu)[2]
        K, f, new = _tangent(s, g, u1[conn[c]], state, lam, mu)
        f_int.index_add_(0, conn[c].reshape(-1), f.reshape(-1, 3))
        if history is not None:
            history[c] = new
        return K

    _, _, vals, rhs = _model_system(model, blocks)
    out = (vals, f_int.reshape(-1), rhs)
    return out + (history.reshape(-1, 13),) if history is not None else out


def _mass(i, model, x, conn):
    t = model.mesh.etype
    N, rho = _tables(t)[1].to(x.device), _t(i["density"])

    def blocks(c):
        s, _ = _gradients(t, x[conn[c]])
        M = torch.einsum("e,eq,qa,qb->eab", rho[c], s, N, N)
        K = torch.zeros(M.shape[0], M.shape[1], 3, M.shape[2], 3, dtype=torch.float64, device=x.device)
        for d in range(3):
            K[:, :, d, :, d] = M
        return K

    return _model_system(model, blocks)[2]


def _conduction(i):
    m = i["mesh"]
    t, N = m.etype, m.n_nodes
    x, conn, k = _t(m.coords), _t(m.conn, torch.int64), _t(i["k"])
    free, pre = np.zeros((N, 3), bool), np.zeros((N, 3))
    free[:, 0] = True
    free[i["tbc"][0], 0] = False
    pre[i["tbc"][0], 0] = i["tbc"][1]

    def blocks(c):
        s, g = _gradients(t, x[conn[c]])
        K = torch.zeros(s.shape[0], conn.shape[1], 3, conn.shape[1], 3, dtype=torch.float64, device=x.device)
        K[:, :, 0, :, 0] = torch.einsum("e,eq,eqai,eqbi->eab", k[c], s, g, g)
        return K

    _, _, vals, moved = _system(m.conn, N, free, pre, blocks, 8192)
    return vals, _t(i["flux"])[_t(free[:, 0], torch.bool)] - moved


def _solve(ptr, cols, vals, rhs):
    n = rhs.numel()
    A = torch.sparse_csr_tensor(ptr, cols.long(), vals, size=(n, n))
    row = torch.repeat_interleave(torch.arange(n, device=ptr.device), ptr[1:] - ptr[:-1])
    inv = torch.empty_like(rhs)
    on = row == cols
    inv[row[on]] = 1.0 / vals[on]
    best = torch.zeros_like(rhs)
    for _ in range(3):  # restarted from the true residual, so the last digits are right
        r = rhs - A @ best
        x, z = torch.zeros_like(rhs), inv * r
        p, rz, stop = z.clone(), torch.dot(r, z), 1e-13 * float(torch.linalg.norm(r))
        for k in range(4000):
            q = A @ p
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            if k % 25 == 0 and float(torch.linalg.norm(r)) <= stop:
                break
            z = inv * r
            rz, old = torch.dot(r, z), rz
            p = z + (rz / old) * p
        best += x
    return best
