"""The work that a user of this library has it do, as timed cases.

Six forms, each through the entry point that a program calls:

* ``solve``    one elastic model from host arrays to displacements, reactions and stresses
               (``Model.solve``): what the host program does once per model;
* ``loads``    several load cases on one kept analysis and factor, loads and displacements in
               device memory (``maille_gpu_solve_device``);
* ``design``   one step of a material optimisation on a kept handle: new moduli, refactorisation,
               solve, adjoint gradient (``SolverHandle.refactor / solve / backward``);
* ``batch``    many models of uneven size with several load cases each (``BatchSolver``), on a kept
               handle or from host arrays to results;
* ``thermal``  a transient heat conduction step (``thermal.solve_problem``);
* ``large``    a neo-Hookean large-strain run and the adjoint of its reactions
               (``LargeStrainSolver.run / backward``).

The meshes are boxes of Kuhn tetrahedra (``maille_b200.meshgen``); the materials, loads and initial
fields are drawn from the seed. ``exact`` solves the same models in 64 bits with plain torch: element
matrices by batched products, element-by-element conjugate gradients with a diagonal preconditioner.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import maille_b200 as mb
from maille_b200 import _lib
from maille_b200 import meshgen as mg
from maille_b200 import thermal as th

FP64, MIXED = _lib.MAILLE_FP64, _lib.MAILLE_MIXED
E0, NU = 210000.0, 0.3
LAMBDA, MU_RANGE = 120000.0, (60000.0, 100000.0)  # the large-strain block's Lame constants


# ---- the cases -----------------------------------------------------------------------------------

def listed():
    return [
        # a part of a few hundred nodes: launches, synchronisations and the analysis are the time
        dict(name="solve_tet4_6", form="solve", nx=6, ny=6, nz=6, tet10=False, mixed=False, tol=1e-12),
        # the plain FP64 benchmark configuration, at the reference's default tolerance
        dict(name="solve_tet4_20", form="solve", nx=20, ny=20, nz=20, tet10=False, mixed=False, tol=1e-12),
        # an ordinary quadratic model of uneven sides in FP64
        dict(name="solve_tet10_27x19x23", form="solve", nx=27, ny=19, nz=23, tet10=True, mixed=False, tol=1e-12),
        # the mixed benchmark configuration: 1.57 M free DOF
        dict(name="solve_tet10_40_mixed", form="solve", nx=40, ny=40, nz=40, tet10=True, mixed=True, tol=1e-10),
        # load cases on one factor: a quadratic model in the mixed form, a small linear one in FP64
        dict(name="loads_tet10_21x24x18_mixed", form="loads", nx=21, ny=24, nz=18, tet10=True, mixed=True, tol=1e-10,
             count=4),
        dict(name="loads_tet4_13x11x12", form="loads", nx=13, ny=11, nz=12, tet10=False, mixed=False, tol=1e-12,
             count=3),
        # the SIMP benchmark configuration: refactorisation, forward and adjoint solve
        dict(name="design_tet4_48", form="design", nx=48, ny=48, nz=48, tet10=False, mixed=False, tol=1e-10),
        # many models of the batched configuration's sizes on a kept handle; a few small ones, once
        dict(name="batch_48x8", form="batch", count=48, lo=6, hi=24, rhs=8, mixed=False, kept=True, tol=1e-10),
        dict(name="batch_once_24x3_mixed", form="batch", count=24, lo=3, hi=12, rhs=3, mixed=True, kept=False,
             tol=1e-10),
        # the transient benchmark configuration (backward Euler); a linear Crank-Nicolson step with
        # fluxes
        dict(name="thermal_tet10_40", form="thermal", nx=40, ny=40, nz=40, tet10=True, mixed=False, theta=1.0,
             increments=10, fluxes=False, tol=1e-12),
        dict(name="thermal_tet4_23x30x17", form="thermal", nx=23, ny=30, nz=17, tet10=False, mixed=False, theta=0.5,
             increments=12, fluxes=True, tol=1e-12),
        # the large-strain benchmark configuration with its reverse pass
        dict(name="large_64x16x16", form="large", nx=64, ny=16, nz=16, increments=10, tol=1e-12),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """Three sides around one size: a part is rarely a cube."""
    m = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return [max(2, min(hi, int(round(m * rng.uniform(0.75, 1.3))))) for _ in range(3)]


def draw(rng):
    form = rng.choice(["solve", "solve", "solve", "loads", "design", "batch", "thermal", "large"])
    mixed = rng.random() < 0.5
    tol = 1e-10 if mixed else rng.choice([1e-10, 1e-12])
    if form == "batch":
        lo = rng.randint(2, 8)
        return dict(form=form, count=_log_int(rng, 2, 48), lo=lo, hi=lo + rng.randint(2, 16), rhs=rng.randint(1, 8),
                    mixed=mixed, kept=rng.random() < 0.7, tol=tol)
    if form == "large":
        nx, ny, nz = _sides(rng, 4, 16)
        return dict(form=form, nx=2 * nx, ny=ny, nz=nz, increments=rng.randint(2, 8), tol=1e-12)
    tet10 = form != "design" and rng.random() < 0.5
    nx, ny, nz = _sides(rng, 3, 40 if form == "solve" or not tet10 else 28)
    case = dict(form=form, nx=nx, ny=ny, nz=nz, tet10=tet10, mixed=mixed, tol=tol)
    if form == "loads":
        case["count"] = rng.randint(1, 6)
    if form == "thermal":
        case.update(theta=rng.choice([1.0, 0.5, 0.75]), increments=rng.randint(1, 12), fluxes=rng.random() < 0.5,
                    mixed=rng.random() < 0.3, tol=1e-12)
    return case


# ---- inputs --------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _box(nx, ny, nz, tet10, size):
    """Nodes, connectivity, the faces on the top (z = size z) as (element, node) arrays and areas."""
    nodes, conn = mg.box_grid((nx, ny, nz), size)
    if tet10:
        nodes, conn = mg.to_quadratic_tet(nodes, conn)
    e, f = mg.faces_on(nodes, conn, 2, size[2])
    tri = conn[e][np.arange(e.size)[:, None], mg.TET_FACES[f]]
    p = nodes[tri]
    area = 0.5 * np.linalg.norm(np.cross(p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]), axis=1)
    if tet10:  # the mid-edge nodes of each face, in the order 0-1, 1-2, 2-0
        mid = {frozenset(v): 4 + k for k, v in enumerate(mg.TET10_EDGES.tolist())}
        local = np.array([[mid[frozenset((a[i], a[(i + 1) % 3]))] for i in range(3)] for a in mg.TET_FACES.tolist()])
        tri = np.concatenate([tri, conn[e][np.arange(e.size)[:, None], local[f]]], axis=1)
    return nodes, conn, e, f, tri, area


def _mesh(case):
    if case["form"] == "large":
        return _box(case["nx"], case["ny"], case["nz"], False, (4.0, 1.0, 1.0))
    n = max(case["nx"], case["ny"], case["nz"])
    return _box(case["nx"], case["ny"], case["nz"], case["tet10"], (case["nx"] / n, case["ny"] / n, case["nz"] / n))


def _face_share(n, tri, area):
    """The integral of N over the faces: area / 3 at each vertex (linear) or mid-edge node (quadratic)."""
    share = np.zeros(n)
    np.add.at(share, tri[:, -3:].ravel(), np.repeat(area / 3.0, 3))
    return share


def _elastic_inputs(case, seed, stream=0):
    """(nodes, conn, young, fixed, list of load vectors) of a box clamped at z = 0 under tractions on
    its top: moduli lognormal for Tet10, E0 rho^3 for a design step, uniform in [50, 250] GPa else."""
    nodes, conn, _, _, tri, area = _mesh(case)
    rng = np.random.default_rng([seed, stream])
    ne, n = conn.shape[0], nodes.shape[0]
    if case["form"] == "design":
        young = E0 * (0.01 + 0.99 * rng.random(ne)) ** 3
    elif case["tet10"]:
        young = E0 * np.exp(0.5 * rng.standard_normal(ne))
    else:
        young = 50000.0 + 200000.0 * rng.random(ne)
    fixed = np.repeat((np.abs(nodes[:, 2]) < 1e-12).astype(np.uint8), 3)
    share = _face_share(n, tri, area)
    loads = []
    for _ in range(case.get("rhs", case.get("count", 1))):
        t = rng.standard_normal(3)
        t *= rng.uniform(1.0, 20.0) / np.linalg.norm(t)
        loads.append((share[:, None] * t).ravel())
    return nodes, conn, young, fixed, loads


def _batch_inputs(case, seed):
    sides = np.random.default_rng(12345).integers(case["lo"], case["hi"] + 1, case["count"])
    out = []
    for k, m in enumerate(sides):
        one = dict(form="solve", nx=int(m), ny=int(m), nz=int(m), tet10=False, rhs=case["rhs"])
        out.append(_elastic_inputs(one, seed, k))
    return out


def _thermal_inputs(case, seed):
    """meshgen's heated cube on this box: T = 100 below, convection on top, a source, lognormal
    conductivities and an uneven initial field."""
    nodes, conn, e, f, tri, area = _mesh(case)
    rng = np.random.default_rng([seed, 7])
    n, ne = nodes.shape[0], conn.shape[0]
    fixed = (np.abs(nodes[:, 2]) < 1e-12).astype(np.uint8)
    film, sink, source = 10.0, 20.0, 50.0
    vol = np.abs(np.linalg.det(nodes[conn[:, 1:4]] - nodes[conn[:, :1]])) / 6.0
    loads = film * sink * _face_share(n, tri, area)
    for local, w in [(slice(0, 4), -0.05), (slice(4, 10), 0.2)] if case["tet10"] else [(slice(0, 4), 0.25)]:
        ids = conn[:, local]
        loads += np.bincount(ids.ravel(), np.repeat(w * source * vol, ids.shape[1]), n)
    prob = mg.ThermalProblem(
        coords=nodes, conn=conn, conductivity=np.exp(0.5 * rng.standard_normal(ne)), rho_c=np.ones(ne), fixed=fixed,
        imposed=np.where(fixed != 0, 100.0, 0.0), loads=loads, initial=20.0 + 5.0 * rng.random() * nodes[:, 0],
        time_period=0.01 * case["increments"], increments=case["increments"], theta=case["theta"], c_elem=e, c_face=f,
        c_film=np.full(e.size, film), c_sink=np.full(e.size, sink))
    return prob, tri, area


def _large_inputs(case, seed):
    """meshgen's bending block: mu uniform per element, the end face's z displacement imposed; and the
    weights of the reactions that the reverse pass differentiates (the end face's, last increment)."""
    nodes, conn, _, _, _, _ = _mesh(case)
    rng = np.random.default_rng([seed, 6])
    ne, n = conn.shape[0], nodes.shape[0]
    mu = MU_RANGE[0] + (MU_RANGE[1] - MU_RANGE[0]) * rng.random(ne)
    fixed = np.repeat((np.abs(nodes[:, 0]) < 1e-12).astype(np.uint8), 3)
    end = np.nonzero(np.abs(nodes[:, 0] - 4.0) < 1e-12)[0]
    fixed[3 * end + 2] = 1
    imposed = np.zeros(3 * n)
    imposed[3 * end + 2] = -0.04 * case["increments"]
    weights = np.zeros((case["increments"], 3 * n))
    weights[-1, 3 * end + 2] = rng.uniform(0.5, 1.5)
    return nodes, conn, mu, fixed, imposed, weights


def _model(case, nodes, conn, young, fixed, f):
    m = mb.Model.from_arrays(nodes, conn, young, NU, fixed, None, f)
    return m.with_solver(mb.SolverKind.ITERATIVE).with_tolerance(case["tol"]).with_precision(
        MIXED if case["mixed"] else FP64)


def prepare(case, seed):
    form = case["form"]
    if form in ("solve", "loads", "design"):
        nodes, conn, young, fixed, loads = _elastic_inputs(case, seed)
        model = _model(case, nodes, conn, young, fixed, loads[0])
        if form == "solve":
            return dict(form=form, model=model)
        if form == "design":
            model.mesh.young = np.full(conn.shape[0], E0)  # the handle starts from the full design
            return dict(form=form, handle=mb.SolverHandle(model), young=young, load=loads[0])
        dev = [torch.from_numpy(f).cuda() for f in loads]
        return dict(form=form, handle=mb.SolverHandle(model), loads=dev, out=[torch.zeros_like(f) for f in dev])
    if form == "batch":
        inputs = _batch_inputs(case, seed)
        probs = [mg.Problem(coords=x, conn=c, young=y, poisson=np.full(y.size, NU), fixed=fx,
                            imposed=np.zeros(fx.size), loads=np.zeros(fx.size)) for x, c, y, fx, _ in inputs]
        state = dict(form=form, loads=[np.stack(l, axis=1) for *_, l in inputs], probs=probs,
                     args=dict(tol=case["tol"], precision=MIXED if case["mixed"] else FP64))
        if case["kept"]:
            state["solver"] = mb.BatchSolver(probs, state["loads"], **state["args"])
        return state
    if form == "thermal":
        prob, _, _ = _thermal_inputs(case, seed)
        s, n = prob.increments, prob.n_nodes
        pinned = lambda *shape: torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy()  # noqa: E731
        out = dict(temps=pinned(s + 1, n), reactions=pinned(s + 1, n), iterations=np.zeros(s, np.int32),
                   fluxes=pinned(s + 1, prob.n_elems, 4 if case["tet10"] else 1, 6) if case["fluxes"] else None)
        return dict(form=form, prob=prob, out=out, tol=case["tol"], precision=MIXED if case["mixed"] else FP64)
    nodes, conn, mu, fixed, imposed, weights = _large_inputs(case, seed)
    young, poisson = mb.large_strain.from_lame(LAMBDA, mu)
    prob = mg.Problem(coords=nodes, conn=conn, young=young, poisson=poisson, fixed=fixed, imposed=imposed,
                      loads=np.zeros(fixed.size))
    return dict(form=form, weights=weights,
                solver=mb.LargeStrainSolver(prob, increments=case["increments"], tol=case["tol"]))


def run(state):
    form = state["form"]
    if form == "solve":
        f = state["model"].solve()
        return dict(u=f.displacements, reactions=f.reactions, stresses=f.stresses, von_mises=f.von_mises)
    if form == "loads":
        lib, h = _lib.load(), state["handle"]
        for f, u in zip(state["loads"], state["out"]):
            if lib.maille_gpu_solve_device(h._h, f.data_ptr(), u.data_ptr()) != _lib.MAILLE_OK:
                raise RuntimeError(_lib.last_error())
        return dict(u=list(state["out"]))
    if form == "design":
        h = state["handle"]
        h.refactor(young=state["young"])
        f = h.solve()
        grad, lam = h.backward(state["load"])
        return dict(u=f.displacements, von_mises=f.von_mises, grad=grad, adjoint=lam)
    if form == "batch":
        if "solver" in state:
            return dict(u=state["solver"].solve(state["loads"]).displacements)
        with mb.BatchSolver(state["probs"], state["loads"], **state["args"]) as b:
            return dict(u=b.solve().displacements)
    if form == "thermal":
        prob, out = state["prob"], state["out"]
        status, got = th.solve_problem(prob, f=prob.loads, tol=state["tol"], fluxes=out["fluxes"] is not None, out=out,
                                       precision=state["precision"])
        if status != _lib.MAILLE_OK:
            raise RuntimeError(_lib.last_error())
        return dict(temps=got["temps"], reactions=got["reactions"], fluxes=got["fluxes"])
    h = state["solver"].run()
    gm, gl = state["solver"].backward(state["weights"])
    return dict(u=h.displacements, reactions=h.reactions, dmu=gm, dlambda=gl)


def work(case):
    """Bytes: the inputs once, the element data of the operator once per pass over it, the results
    once. A pass over the operator cannot be left out, the number of passes is the method's: one pass
    per right-hand side is counted. Flops: the element matrices and those passes."""
    form = case["form"]
    if form == "batch":
        sides = np.random.default_rng(12345).integers(case["lo"], case["hi"] + 1, case["count"])
        ne, n = float((6 * sides ** 3).sum()), float(((sides + 1) ** 3).sum())
        rhs, dof, npe, width = case["rhs"], 3, 4, 4 if case["mixed"] else 8
    else:
        tet10 = case.get("tet10", False)
        cells = case["nx"] * case["ny"] * case["nz"]
        k = 2 if tet10 else 1
        n = float((k * case["nx"] + 1) * (k * case["ny"] + 1) * (k * case["nz"] + 1))
        ne, npe, dof = 6.0 * cells, 10 if tet10 else 4, 1 if form == "thermal" else 3
        rhs = {"loads": case.get("count", 1), "design": 2, "thermal": case.get("increments", 1),
               "large": 3 * case.get("increments", 1)}.get(form, 1)
        width = 4 if case.get("mixed") else 8
    # blocks of the assembled pattern: 15 neighbours of a Tet4 node, about 28 of a Tet10 node
    blocks = n * (28.0 if npe == 10 else 15.0)
    ng = 4 if npe == 10 else 1
    inputs = n * (24.0 + 9.0 * dof) + ne * (8.0 * npe + 16.0)
    results = 8.0 * dof * n * max(1, rhs if form in ("loads", "batch", "thermal") else 1)
    if form == "solve":
        results += 8.0 * dof * n + 80.0 * ng * ne
    kept = form in ("loads",) or (form == "batch" and case["kept"])
    matrix = blocks * (dof * dof * width + 4.0)
    bytes_ = (0.0 if kept else inputs) + results + matrix * (1 if form == "batch" else rhs) + 16.0 * dof * n * rhs
    integration = 0.0 if kept else ne * ng * npe * (npe + 1) / 2 * (40.0 if dof == 3 else 8.0)
    return dict(bytes=bytes_, flops=integration + 2.0 * blocks * dof * dof * rhs)


# ---- 64-bit values with plain torch --------------------------------------------------------------

_A, _B = 0.5854101966249685, 0.1381966011250105
_TETRA_4 = [(_A, _B, _B, _B), (_B, _A, _B, _B), (_B, _B, _A, _B), (_B, _B, _B, _A)]  # (l0, l1, l2, l3), weight 1/4
_EDGES = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev())


def _barycentric(x):
    """Gradients (E, 4, 3) of the barycentric coordinates of straight tetrahedra, and volumes."""
    edges = x[:, 1:4] - x[:, :1]
    g = torch.linalg.inv(edges).transpose(1, 2)
    return torch.cat([-g.sum(1, keepdim=True), g], 1), torch.linalg.det(edges).abs() / 6.0


def _points(npe):
    """Gauss points as barycentric tuples, in the order the results list them, and their weight."""
    return ([(0.25,) * 4], 1.0) if npe == 4 else (_TETRA_4, 0.25)


def _gradients(dl, l, npe):
    """dN/dx (E, npe, 3) at barycentric l."""
    if npe == 4:
        return dl
    g = [(4.0 * l[a] - 1.0) * dl[:, a] for a in range(4)]
    g += [4.0 * (l[p] * dl[:, q] + l[q] * dl[:, p]) for p, q in _EDGES]
    return torch.stack(g, 1)


def _shape(l, npe):
    if npe == 4:
        return list(l)
    return [l[a] * (2.0 * l[a] - 1.0) for a in range(4)] + [4.0 * l[p] * l[q] for p, q in _EDGES]


class _Operator:
    """Element matrices (E, m, m) on dof ids (E, m) of a vector of n entries."""

    def __init__(self, ke, dofs, n):
        self.ke, self.dofs, self.n = ke, dofs, n
        self.diag = torch.zeros(n, dtype=torch.float64, device=ke.device).index_add_(
            0, dofs.reshape(-1), torch.diagonal(ke, dim1=1, dim2=2).reshape(-1))

    def __call__(self, x):
        y = torch.bmm(self.ke, x[self.dofs])
        return torch.zeros_like(x).index_add_(0, self.dofs.reshape(-1), y.reshape(-1, x.shape[1]))


def _cg(op, free, b, tol=1e-14, limit=20000):
    """Columns of x with op x = b on the free entries, x = 0 elsewhere: conjugate gradients with the
    diagonal as preconditioner, restarted on the true residual until it stops falling."""
    free = free[:, None]
    inv = torch.where(free, 1.0 / op.diag[:, None], 0.0)
    b = torch.where(free, b, 0.0)
    bb = b.square().sum(0)
    x = torch.zeros_like(b)
    for _ in range(3):
        r = torch.where(free, b - op(x), 0.0)
        z = inv * r
        p, rz = z.clone(), (r * z).sum(0)
        d = torch.zeros_like(x)
        for k in range(limit):
            ap = torch.where(free, op(p), 0.0)
            pap = (p * ap).sum(0)
            alpha = torch.where(pap > 0, rz / pap, 0.0)
            d += alpha * p
            r -= alpha * ap
            z = inv * r
            new = (r * z).sum(0)
            p = z + torch.where(rz > 0, new / rz, 0.0) * p
            rz = new
            if k % 50 == 49 and bool((r.square().sum(0) <= tol * tol * bb).all()):
                break
        x = x + d
    return x


def _dofs3(conn):
    return (3 * _t(conn, torch.int64)[:, :, None] + torch.arange(3, device=_dev())).reshape(conn.shape[0], -1)


def _elastic_operator(nodes, conn, young):
    """The isotropic stiffness at Poisson ratio NU, summed over the Gauss points."""
    x, e, npe = _t(nodes)[_t(conn, torch.int64)[:, :4]], _t(young), conn.shape[1]
    lam, mu = e * NU / ((1 + NU) * (1 - 2 * NU)), e / (2 * (1 + NU))
    dl, vol = _barycentric(x)
    pts, w = _points(npe)
    ke = torch.zeros(len(e), npe, 3, npe, 3, dtype=torch.float64, device=_dev())
    eye = torch.eye(3, dtype=torch.float64, device=_dev())
    for l in pts:
        g = _gradients(dl, l, npe)
        gg = torch.einsum("eai,ebj->eaibj", g, g)
        ke += (w * vol * lam)[:, None, None, None, None] * gg
        ke += (w * vol * mu)[:, None, None, None, None] * gg.transpose(2, 4)
        ke += torch.einsum("e,eab,ij->eaibj", w * vol * mu, torch.einsum("eak,ebk->eab", g, g), eye)
    m = 3 * npe
    return _Operator(ke.reshape(-1, m, m), _dofs3(conn), 3 * nodes.shape[0])


def _stresses(nodes, conn, young, u):
    """Per Gauss point x, y, z, sxx, syy, szz, txy, tyz, txz and the von Mises value."""
    ids, npe = _t(conn, torch.int64), conn.shape[1]
    x, ue, e = _t(nodes)[ids], u.reshape(-1, 3)[ids], _t(young)
    lam, mu = (e * NU / ((1 + NU) * (1 - 2 * NU)))[:, None, None], (e / (2 * (1 + NU)))[:, None, None]
    dl, _ = _barycentric(x[:, :4])
    eye, out = torch.eye(3, dtype=torch.float64, device=_dev()), []
    for l in _points(npe)[0]:
        grad = torch.einsum("eai,eaj->eij", ue, _gradients(dl, l, npe))
        eps = 0.5 * (grad + grad.transpose(1, 2))
        s = lam * torch.diagonal(eps, dim1=1, dim2=2).sum(1)[:, None, None] * eye + 2 * mu * eps
        at = torch.einsum("a,eai->ei", _t(_shape(l, npe)), x)
        out.append(torch.cat([at, torch.stack([s[:, 0, 0], s[:, 1, 1], s[:, 2, 2], s[:, 0, 1], s[:, 1, 2], s[:, 0, 2]],
                                              1)], 1))
    out = torch.stack(out, 1)
    sx, sy, sz, xy, yz, xz = (out[..., k] for k in range(3, 9))
    vm = torch.sqrt(0.5 * ((sx - sy) ** 2 + (sy - sz) ** 2 + (sz - sx) ** 2) + 3 * (xy ** 2 + yz ** 2 + xz ** 2))
    return out, vm


def _cpu(x):
    return x.cpu().numpy()


def _exact_elastic(case, seed):
    nodes, conn, young, fixed, loads = _elastic_inputs(case, seed)
    op, free, f = _elastic_operator(nodes, conn, young), _t(fixed) == 0, _t(np.stack(loads, 1))
    u = _cg(op, free, f)
    if case["form"] == "loads":
        return dict(u=[_cpu(u[:, k]) for k in range(u.shape[1])])
    stresses, vm = _stresses(nodes, conn, young, u[:, 0])
    if case["form"] == "design":  # compliance is self-adjoint: lambda = u on the free entries
        ue = u[:, 0][op.dofs]
        grad = -torch.einsum("ei,eij,ej->e", ue, op.ke, ue) / _t(young)
        return dict(u=_cpu(u[:, 0]), von_mises=_cpu(vm), grad=_cpu(grad), adjoint=_cpu(u[:, 0]))
    reactions = torch.where(free, 0.0, (op(u) - f)[:, 0])
    return dict(u=_cpu(u[:, 0]), reactions=_cpu(reactions), stresses=_cpu(stresses), von_mises=_cpu(vm))


def _exact_batch(case, seed):
    inputs = _batch_inputs(case, seed)
    off = np.concatenate([[0], np.cumsum([x.shape[0] for x, *_ in inputs])])
    op = _elastic_operator(np.concatenate([x for x, *_ in inputs]),
                           np.concatenate([c + o for (_, c, *_), o in zip(inputs, off)]),
                           np.concatenate([y for _, _, y, *_ in inputs]))
    f = _t(np.concatenate([np.stack(l, 1) for *_, l in inputs]))
    u = _cg(op, _t(np.concatenate([fx for *_, fx, _ in inputs])) == 0, f)
    return dict(u=[_cpu(u[3 * a:3 * b]) for a, b in zip(off[:-1], off[1:])])


def _monomial(powers):
    """6 V times this is the integral of l0^i l1^j l2^k l3^m over a tetrahedron of volume V."""
    return math.prod(math.factorial(p) for p in powers) / math.factorial(sum(powers) + 3)


def _mass(npe):
    """(npe, npe) integral of N N^T over a tetrahedron of unit volume."""
    one = lambda *at: tuple(sum(1 for a in at if a == i) for i in range(4))  # noqa: E731
    if npe == 4:
        shapes = [{one(a): 1.0} for a in range(4)]
    else:  # l (2 l - 1) = 2 l^2 - l
        shapes = [{one(a, a): 2.0, one(a): -1.0} for a in range(4)] + [{one(p, q): 4.0} for p, q in _EDGES]
    return np.array([[sum(6.0 * cp * cq * _monomial([i + j for i, j in zip(p, q)]) for p, cp in s.items()
                          for q, cq in t.items()) for t in shapes] for s in shapes])


def _exact_thermal(case, seed):
    p, tri, area = _thermal_inputs(case, seed)
    ids, npe, n = _t(p.conn, torch.int64), p.npe, p.n_nodes
    x, k = _t(p.coords)[ids], _t(p.conductivity)
    dl, vol = _barycentric(x[:, :4])
    pts, w = _points(npe)
    ke = sum((w * vol * k)[:, None, None] * torch.einsum("eai,ebi->eab", _gradients(dl, l, npe), _gradients(dl, l, npe))
             for l in pts)
    ce = (vol * _t(p.rho_c))[:, None, None] * _t(_mass(npe))
    # convection: h times the integral of N N^T over each face, closed form
    if npe == 4:
        fm = (np.ones((3, 3)) + np.eye(3)) / 12.0
    else:
        fm = np.array([[6, -1, -1, 0, -4, 0], [-1, 6, -1, 0, 0, -4], [-1, -1, 6, -4, 0, 0], [0, 0, -4, 32, 16, 16],
                       [-4, 0, 0, 16, 32, 16], [0, -4, 0, 16, 16, 32]]) / 180.0
    he = _t(p.c_film * area)[:, None, None] * _t(fm)
    face = _Operator(he, _t(tri, torch.int64), n)
    dt, theta = p.time_step, p.theta
    left = _Operator(ce / dt + theta * ke, ids, n)
    right = _Operator(ce / dt - (1 - theta) * ke, ids, n)
    both = _Sum(left, face, theta)
    free, f = _t(p.fixed) == 0, _t(p.loads)[:, None]
    t = torch.where(free, _t(p.initial), _t(p.imposed))[:, None]
    temps, reactions = [t], [torch.zeros_like(t)]
    fixed = torch.where(free[:, None], 0.0, t)
    for _ in range(p.increments):
        b = right(t) - (1 - theta) * face(t) + f
        new = fixed + _cg(both, free, b - both(fixed))
        reactions.append(torch.where(free[:, None], 0.0, both(new) - b))
        temps.append(new)
        t = new
    fluxes = None
    if case["fluxes"]:
        fluxes = []
        for t in temps:
            at = []
            for l in _points(npe)[0]:
                grad = torch.einsum("ea,eai->ei", t[:, 0][ids], _gradients(dl, l, npe))
                at.append(torch.cat([torch.einsum("a,eai->ei", _t(_shape(l, npe)), x), -k[:, None] * grad], 1))
            fluxes.append(torch.stack(at, 1))
        fluxes = _cpu(torch.stack(fluxes))
    return dict(temps=_cpu(torch.cat(temps, 1).T), reactions=_cpu(torch.cat(reactions, 1).T), fluxes=fluxes)


class _Sum:
    """a + scale b of two operators on the same entries."""

    def __init__(self, a, b, scale):
        self.a, self.b, self.scale, self.diag = a, b, scale, a.diag + scale * b.diag

    def __call__(self, x):
        return self.a(x) + self.scale * self.b(x)


def _neo_hookean(dl, vol, lam, mu, ue, tangent):
    """Internal forces (E, 12) of P = mu (F - F^-T) + lambda ln J F^-T, and the tangents or the forces'
    derivatives with respect to mu and lambda."""
    f = torch.eye(3, dtype=torch.float64, device=ue.device) + torch.einsum("eai,eaj->eij", ue, dl)
    fi, lj = torch.linalg.inv(f), torch.log(torch.linalg.det(f))
    h = torch.einsum("eaj,eji->eai", dl, fi)  # F^-T dN/dX
    v = vol[:, None, None]
    d_mu, d_lam = v * (torch.einsum("eij,eaj->eai", f, dl) - h), v * lj[:, None, None] * h
    forces = mu[:, None, None] * d_mu + lam * d_lam
    if not tangent:
        return forces.reshape(-1, 12), d_mu.reshape(-1, 12), d_lam.reshape(-1, 12)
    eye = torch.eye(3, dtype=torch.float64, device=ue.device)
    ke = torch.einsum("e,eab,ij->eaibj", vol * mu, torch.einsum("eak,ebk->eab", dl, dl), eye)
    ke += torch.einsum("e,eai,ebj->eaibj", vol * lam, h, h)
    ke += torch.einsum("e,eaj,ebi->eaibj", vol * (mu - lam * lj), h, h)
    return forces.reshape(-1, 12), ke.reshape(-1, 12, 12)


def _exact_large(case, seed):
    if case["nx"] * case["ny"] * case["nz"] * case["increments"] > 8000:
        return None  # the Newton iterations' plain conjugate gradients take too long
    nodes, conn, mu, fixed, imposed, weights = _large_inputs(case, seed)
    dl, vol = _barycentric(_t(nodes)[_t(conn, torch.int64)])
    dofs, n, mu, free = _dofs3(conn), fixed.size, _t(mu), _t(fixed) == 0
    total = lambda fe: torch.zeros(n, dtype=torch.float64, device=fe.device).index_add_(  # noqa: E731
        0, dofs.reshape(-1), fe.reshape(-1))
    u, us, rs = torch.zeros(n, dtype=torch.float64, device=_dev()), [], []
    for k in range(case["increments"]):
        target = _t(imposed) * ((k + 1) / case["increments"])
        step = torch.where(free, 0.0, target - u)
        for _ in range(12):
            fe, ke = _neo_hookean(dl, vol, LAMBDA, mu, u[dofs].reshape(-1, 4, 3), True)
            op = _Operator(ke, dofs, n)
            du = step + _cg(op, free, -(total(fe)[:, None] + op(step[:, None])), 1e-12)[:, 0]
            u, step = u + du, torch.zeros_like(u)
            if float(du.norm()) <= 1e-13 * float(u.norm()):
                break
        fe, d_mu, d_lam = _neo_hookean(dl, vol, LAMBDA, mu, u[dofs].reshape(-1, 4, 3), False)
        us.append(u)
        rs.append(torch.where(free, 0.0, total(fe)))
    # the weights are those of the last increment: w = (g, m) with K_ff m = -K_fc g
    _, ke = _neo_hookean(dl, vol, LAMBDA, mu, u[dofs].reshape(-1, 4, 3), True)
    op, g = _Operator(ke, dofs, n), _t(weights[-1])[:, None]
    w = (g + _cg(op, free, -op(g)))[:, 0][dofs]
    return dict(u=_cpu(torch.stack(us)), reactions=_cpu(torch.stack(rs)), dmu=_cpu((w * d_mu).sum(1)),
                dlambda=_cpu((w * d_lam).sum(1)))


def exact(case, seed):
    form = case["form"]
    if form == "batch":
        return _exact_batch(case, seed)
    if form == "thermal":
        return _exact_thermal(case, seed)
    if form == "large":
        return _exact_large(case, seed)
    return _exact_elastic(case, seed)
