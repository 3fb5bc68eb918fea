"""The work a user of this package has it do, as measurable cases.

Each case is one call sequence through the public entry points: residual
evaluations of the ideal-gas set in both arithmetics, whole Newton steps, the
reacting set's per-node and per-edge calls, and a training gradient of the
learned preconditioner.  ``exact`` restates the computed outputs in plain
64-bit torch from the mesh arrays and the input state alone.
"""
import ctypes as C
import functools
import math
from pathlib import Path

import numpy as np
import torch

from proteuscfd_gb300 import Mesh, SolutionSpace, cases
from proteuscfd_gb300 import _native as N
from proteuscfd_gb300.chem import ChemModel, load_mechanism

MECHANISM = Path(__file__).resolve().parent.parent / "tests" / "golden" / "chem_5species_air.json"
NS = 5                      # species of that mechanism
NREC = 6 + 3 * NS           # reacting node record: rho_i, u, v, w, T, P, rho, cv_i, concentrations
REF_TIME = 2.5e-4
CHEM_RE = 1.0e4
GAMMA = 1.4


def listed():
    return [
        # a unit-test-sized flat plate: what a user sees while setting a case up; latency and launches count
        dict(name="residual_tiny", kind="residual", flow="ns", nx=10, ny=8, nz=8, sorder=2, limiter=3, arith=0,
             state="perturbed"),
        # an odd-sized plate with the plain Venkatakrishnan limiter, boundary-layer state
        dict(name="residual_ragged", kind="residual", flow="ns", nx=53, ny=37, nz=29, sorder=2, limiter=2, arith=0,
             state="layer"),
        # the benchmark's 128x96x96 plate in FP64, the reference's arithmetic
        dict(name="residual_plate", kind="residual", flow="ns", nx=128, ny=96, nz=96, sorder=2, limiter=3, arith=0,
             state="perturbed"),
        # the same physics in the optional double-float arithmetic
        dict(name="residual_double_float", kind="residual", flow="ns", nx=96, ny=72, nz=64, sorder=2, limiter=3,
             arith=1, state="layer"),
        # the Mach 2 ramp with its shock, first order, slip walls
        dict(name="residual_ramp", kind="residual", flow="ramp", nx=161, ny=65, nz=63, sorder=1, limiter=0, arith=0,
             state="shock"),
        # a Newton step of the reference's method: FP64 Jacobian, ten SGS sweeps
        dict(name="newton_sgs", kind="newton", nx=64, ny=48, nz=48, jac_precision=0, linear_solver=0, nsgs=10,
             cfl=20.0),
        # a Newton step of the mixed-precision solver: FP32 Jacobian, FGMRES(30) preconditioned by two sweeps
        dict(name="newton_mixed", kind="newton", nx=64, ny=48, nz=48, jac_precision=1, linear_solver=1, nsgs=2,
             cfl=50.0),
        # finite-rate chemistry of a field of nodes from host arrays
        dict(name="chem_rates", kind="chem_rates", n=1000003),
        # the implicit chemistry blocks of a field of device-resident records
        dict(name="chem_jacobian", kind="chem_jacobian", n=250007),
        # the reacting first-order residual with its source, device-resident records
        dict(name="chem_first_order", kind="chem_first_order", nx=96, ny=64, nz=64),
        # the reacting second-order Navier-Stokes residual stage by stage from host arrays
        dict(name="chem_second_order", kind="chem_second_order", nx=41, ny=33, nz=29),
        # forward and backward pass of the learned preconditioner (training)
        dict(name="learned_gradient", kind="learned", nx=40, ny=32, nz=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """Grid sizes with about lo..hi nodes (log-uniform), flat-plate-like proportions."""
    n = _log_int(rng, lo, hi)
    a, b = rng.uniform(1.0, 1.8), rng.uniform(0.8, 1.2)
    nz = max(6, int((n / (a * b)) ** (1.0 / 3.0)))
    return max(8, int(a * nz)), max(7, int(b * nz)), nz


def draw(rng):
    kind = rng.choice(["residual", "residual", "residual", "newton", "newton", "chem_rates", "chem_jacobian",
                       "chem_first_order", "chem_second_order", "learned"])
    if kind == "residual":
        flow = rng.choice(["ns", "ns", "ramp"])
        nx, ny, nz = _box(rng, 600, 700000)
        if flow == "ns":
            return dict(kind=kind, flow=flow, nx=nx, ny=ny, nz=nz, sorder=2, limiter=rng.choice([1, 2, 3, 3, 3]),
                        arith=rng.choice([0, 0, 1]), state=rng.choice(["perturbed", "layer"]))
        sorder = rng.choice([1, 2])
        return dict(kind=kind, flow=flow, nx=nx, ny=ny, nz=nz, sorder=sorder, limiter=3 if sorder == 2 else 0,
                    arith=rng.choice([0, 0, 1]), state=rng.choice(["perturbed", "shock"]))
    if kind == "newton":
        nx, ny, nz = _box(rng, 600, 140000)
        mixed = rng.choice([False, True])
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, jac_precision=int(mixed), linear_solver=int(mixed),
                    nsgs=2 if mixed else rng.choice([5, 10, 20]), cfl=rng.choice([5.0, 20.0, 50.0]))
    if kind == "chem_rates":
        return dict(kind=kind, n=_log_int(rng, 500, 1000000))
    if kind == "chem_jacobian":
        return dict(kind=kind, n=_log_int(rng, 500, 250000))
    nx, ny, nz = _box(rng, 600, 300000 if kind == "chem_first_order" else 40000)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz)


# ---- inputs ----------------------------------------------------------------

@functools.lru_cache(maxsize=6)
def _grid(flow, nx, ny, nz):
    """The mesh of a case: one grid per size, as a user's program has."""
    c = cases.ns_flatplate(nx, ny, nz) if flow == "ns" else cases.euler_ramp(nx, ny, nz)
    return cases.build_mesh(c), c


def _flow_case(case):
    """(mesh, parameters) of an ideal-gas case."""
    flow = case.get("flow", "ns")
    mesh, c = _grid(flow, case["nx"], case["ny"], case["nz"])
    c = cases.ns_flatplate(case["nx"], case["ny"], case["nz"]) if flow == "ns" else cases.euler_ramp(
        case["nx"], case["ny"], case["nz"])
    p = c.param
    p.sorder, p.limiter = case.get("sorder", 2), case.get("limiter", 3)
    return mesh, p


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _state(mesh, p, kind, seed):
    """Start state [nnode + nbedge][10] in pinned memory.  perturbed: the
    benchmark's freestream with +-1 % noise; layer: a boundary-layer profile
    over the wall with +-0.05 % noise, as a run under way has; shock: the
    attached oblique shock of the ramp with +-0.5 % noise."""
    rng = np.random.default_rng(seed)
    rows = mesh.nnode + mesh.nbedge
    xyz = np.concatenate([mesh.xyz, mesh.xyz[mesh.bedges[:, 0]]])
    rho = np.full(rows, GAMMA)
    vel = np.zeros((rows, 3))
    vel[:, 0] = p.mach
    pr = np.ones(rows)
    amp = {"perturbed": 0.01, "layer": 0.0005, "shock": 0.005}[kind]
    if kind == "layer":
        on = 1.0 / (1.0 + np.exp(-40.0 * (xyz[:, 0] - (xyz[:, 0].max() - 1.0))))
        prof = np.tanh(xyz[:, 1] / 0.06)
        vel[:, 0] *= 1.0 - on * (1.0 - prof)
        vel[:, 1] += 0.004 * p.mach * on * prof * (1.0 - prof)
        temp = 1.0 + 0.17 * p.mach ** 2 * (1.0 - (vel[:, 0] / p.mach) ** 2)
        rho = GAMMA / temp
    elif kind == "shock":
        beta, th = math.radians(45.344), math.radians(15.0)
        behind = xyz[:, 1] < (xyz[:, 0] - 0.5) * math.tan(beta)
        behind &= xyz[:, 0] > 0.5
        mach2 = 1.446
        rho[behind] *= 1.7289
        pr[behind] = 2.1947
        speed2 = mach2 * math.sqrt(2.1947 / 1.7289)
        vel[behind, 0], vel[behind, 1] = speed2 * math.cos(th), speed2 * math.sin(th)
    q = _pinned((rows, 10))
    q[:, 0] = rho
    q[:, 1:4] = rho[:, None] * vel
    q[:, 4] = pr / (GAMMA - 1.0) + 0.5 * rho * (vel ** 2).sum(axis=1)
    q[:, :5] *= 1.0 + rng.uniform(-amp, amp, size=(rows, 5))
    u = q[:, 1:4] / q[:, :1]
    q[:, 6] = (GAMMA - 1.0) * (q[:, 4] - 0.5 * q[:, 0] * (u * u).sum(axis=1))
    q[:, 5] = GAMMA * q[:, 6] / q[:, 0]
    q[:, 7:] = u
    return q


@functools.lru_cache(maxsize=1)
def _mechanism():
    return load_mechanism(MECHANISM)


def _chem_ref():
    """Air at 300 K and 101325 Pa in the reference's style of scales."""
    v = (1.4 * 287.0 * 300.0) ** 0.5
    return ChemModel.ref(101325.0 / v ** 2, 101325.0, 300.0 / 1.4, v * v, v)


def _chem_full_ref():
    r = _chem_ref()
    r.viscosity = r.density * r.velocity
    r.conductivity = r.density * r.velocity ** 3 / r.temperature
    return r


def _aux(ref, rhoi, vel, T):
    """Reacting node records completed from species densities, velocity and
    temperature (ideal mixture; NASA-7 curves)."""
    spec = _mechanism()["species"]
    mw = np.array([s["MW"] for s in spec])
    R = 8.31447215 / mw
    td = T * ref.temperature
    P = (rhoi * ref.density * R).sum(axis=1) * td / ref.pressure
    cp = np.empty_like(rhoi)
    for k, s in enumerate(spec):
        lo, hi = np.polyval(s["lo"][4::-1], td), np.polyval(s["hi"][4::-1], td)
        cp[:, k] = np.where(td > 1000.0, hi, lo) * R[k]
    cvi = (cp - R) / (ref.velocity ** 2 / ref.temperature)
    return np.ascontiguousarray(np.c_[rhoi, vel, T, P, rhoi.sum(axis=1), cvi, rhoi / mw / 1000.0])


def _chem_field(xyz, seed):
    """A hypersonic shock-layer-like field: air partly dissociated behind a
    smooth front, 300 to 4500 K, with +-2 % noise."""
    ref = _chem_ref()
    rng = np.random.default_rng(seed)
    n = len(xyz)
    x = (xyz[:, 0] - xyz[:, 0].min()) / max(np.ptp(xyz[:, 0]), 1e-30)
    y = (xyz[:, 1] - xyz[:, 1].min()) / max(np.ptp(xyz[:, 1]), 1e-30)
    s = 1.0 / (1.0 + np.exp(-18.0 * (x - 0.35 - 0.4 * y)))
    cold = np.array([0.233, 1e-6, 1e-6, 0.766, 1e-6])
    hot = np.array([0.11, 0.09, 0.02, 0.74, 0.04])
    Y = cold + s[:, None] * (hot - cold)
    rho = (0.02 + 0.08 * s) / ref.density
    T = (300.0 + 4200.0 * s) / ref.temperature
    vel = np.stack([4.0 - 3.0 * s, 0.6 * s, 0.1 * np.sin(6.0 * x)], axis=1)
    noise = rng.uniform(0.98, 1.02, size=(n, NS + 4))
    return _aux(ref, rho[:, None] * Y * noise[:, :NS], vel * noise[:, NS:NS + 3], T * noise[:, NS + 3])


def _chem_points(n, seed):
    """Unordered reacting states over the mechanism's range (one node's state
    says nothing of the next's)."""
    rng = np.random.default_rng(seed)
    Y = rng.dirichlet(np.array([2.0, 0.6, 0.3, 6.0, 0.4]), size=n) + 1e-9
    rho = 10.0 ** rng.uniform(-3.0, 0.0, size=n)
    return rho[:, None] * Y, rng.uniform(300.0, 7000.0, size=n)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "residual":
        mesh, p = _flow_case(case)
        S = SolutionSpace(mesh, p)
        S.set_residual_arithmetic(case["arith"])
        return dict(kind=kind, S=S, q=_state(mesh, p, case["state"], seed), b=_pinned((mesh.nnode, 5)))
    if kind == "newton":
        mesh, p = _flow_case(case)
        S = SolutionSpace(mesh, p)
        S.set_jacobian_precision(case["jac_precision"])
        q = _state(mesh, p, "layer", seed)
        opts = dict(cfl=case["cfl"], nsgs=case["nsgs"], jac_precision=case["jac_precision"],
                    linear_solver=case["linear_solver"], fgmres_m=30, fgmres_rtol=0.1)
        return dict(kind=kind, S=S, q=q, out=_pinned(q.shape), opts=opts)
    if kind == "learned":
        mesh, p = _flow_case(case)
        S = SolutionSpace(mesh, p)
        S.lp_init(1)
        rng = np.random.default_rng(seed)
        S.lp_set_params(_lp_params(rng))
        x = rng.normal(size=(mesh.nnode, N.LP_NIN)).astype(np.float32)
        t = rng.normal(size=(mesh.nnode, N.LP_NOUT)).astype(np.float32)
        return dict(kind=kind, S=S, x=x, t=t)
    model = ChemModel(_mechanism())
    ref = _chem_full_ref()
    if kind == "chem_rates":
        rho, T = _chem_points(case["n"], seed)
        hr, ht, hw = _pinned(rho.shape), _pinned(T.shape), _pinned(rho.shape)
        hr[:], ht[:] = rho, T
        return dict(kind=kind, model=model, rho=hr, T=ht, w=hw)
    if kind == "chem_jacobian":
        rho, T = _chem_points(case["n"], seed)
        rng = np.random.default_rng(seed + 1)
        rec = _aux(ref, rho / ref.density, rng.normal(size=(len(T), 3)) * 0.5, T / ref.temperature)
        n = len(T)
        return dict(kind=kind, model=model, ref=ref, n=n, q=_dev(rec), vol=_dev(rng.uniform(0.5, 2.0, n)),
                    dtau=_dev(rng.uniform(0.01, 0.1, n)), beta=_dev(rng.uniform(0.3, 1.0, n)),
                    A=torch.empty((n, NS + 4, NS + 4), dtype=torch.float64, device="cuda"))
    mesh = _grid("ns", case["nx"], case["ny"], case["nz"])[0]
    model.attach_mesh(mesh)
    rec = _chem_field(np.concatenate([mesh.xyz, mesh.xyz[mesh.bedges[:, 0]]]), seed)
    if kind == "chem_first_order":
        return dict(kind=kind, model=model, ref=ref, q=_dev(rec),
                    b=torch.empty((mesh.nnode, NS + 4), dtype=torch.float64, device="cuda"))
    return dict(kind=kind, model=model, ref=ref, q=rec)


def _lp_params(rng):
    """A trained-looking network: Kaiming-sized matrices and a live decoder."""
    w = rng.uniform(-0.2, 0.2, size=N.LP_NPARAM).astype(np.float32)
    return w


# ---- one pass --------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "residual":
        S = state["S"]
        S.set_state(state["q"])
        norms = S.residual_full()
        S.get_residual(out=state["b"])
        return {"b": state["b"], "norms": norms}
    if kind == "newton":
        S, out = state["S"], state["out"]
        S.set_state(state["q"])
        rep = S.newton_iterate(5, **state["opts"])
        # the C interface's read of the updated state into the program's own buffer
        N.check(N.load().pcfd_get_state(S.handle, N.dptr(out), 10, S.nrows), "pcfd_get_state")
        return {"q": out, "res": np.array(rep["res"])}
    if kind == "learned":
        loss, grad = state["S"].lp_loss_grad(state["x"], state["t"])
        return {"loss": np.float32(loss), "grad": grad}
    m = state["model"]
    if kind == "chem_rates":
        return {"w": m.production_rates(state["rho"], state["T"], out=state["w"])}
    ref, q = state["ref"], state["q"]
    if kind == "chem_jacobian":
        A = state["A"]
        m.source_jacobian_dev(ref, REF_TIME, state["n"], q.data_ptr(), state["vol"].data_ptr(), A.data_ptr())
        m.temporal_terms_dev(ref, state["n"], q.data_ptr(), state["vol"].data_ptr(), state["dtau"].data_ptr(),
                             state["beta"].data_ptr(), 1.0, 0.0, 0, A.data_ptr())
        return {"A": A}
    opts = ChemModel.flux_opts()
    if kind == "chem_first_order":
        norms = m.residual_dev(ref, opts, REF_TIME, 1, q.data_ptr(), state["b"].data_ptr())
        return {"b": state["b"], "norms": norms}
    grad = m.gradient(q, sym_tags=(5, 6, 7))
    lim = m.limiter(0.0, q, grad)
    b, norms = m.residual_ho(ref, opts, 0.0, REF_TIME, 1, q, grad, lim)
    bv = m.viscous_residual(ref, opts, CHEM_RE, 1, q, grad)
    return {"grad": grad, "lim": lim, "b": b, "norms": norms, "bv": bv}


# ---- work ------------------------------------------------------------------

def _sizes(case):
    """(nodes, edges, boundary half-edges) of the box (six tetrahedra a cell)."""
    a, b, c = case["nx"], case["ny"], case["nz"]
    n = a * b * c
    faces = 2 * ((a - 1) * (b - 1) + (b - 1) * (c - 1) + (a - 1) * (c - 1))
    cells = (a - 1) * (b - 1) * (c - 1)
    return n, n + 6 * cells + faces - 1, 6 * faces


def work(case):
    kind = case["kind"]
    if kind == "chem_rates":
        return {"bytes": 88.0 * case["n"], "flops": 900.0 * case["n"]}
    if kind == "chem_jacobian":
        return {"bytes": (8.0 * 14 + 8.0 * 81) * case["n"], "flops": 3000.0 * case["n"]}
    n, e, h = _sizes(case)
    if kind == "residual":
        ns = case["flow"] == "ns"
        per_edge = 200.0 + (160.0 if case["sorder"] > 1 else 0.0) + (130.0 if ns else 0.0)
        return {"bytes": 40.0 * e + 200.0 * n + 84.0 * h, "flops": per_edge * e + 100.0 * n + 2500.0 * h}
    if kind == "newton":
        s = 4.0 if case["jac_precision"] else 8.0
        sweeps = case["nsgs"] * (8.0 if case["linear_solver"] else 1.0)
        blocks = n + 2.0 * e
        return {"bytes": 40.0 * e + 200.0 * n + (1.0 + 2.0 * sweeps) * 25.0 * s * blocks,
                "flops": (1500.0 + 500.0) * e + 2.0 * sweeps * 50.0 * blocks}
    if kind == "learned":
        return {"bytes": 64.0 * n + 16.0 * 2 * e, "flops": 6.0 * 26821 * n + 3 * 3 * 2.0 * 640 * e}
    if kind == "chem_first_order":
        return {"bytes": 40.0 * e + (88.0 + 72.0) * n + 84.0 * h, "flops": 250.0 * e + 900.0 * n}
    return {"bytes": 40.0 * e + (8.0 * (2 * NREC + 42 + 27)) * n + 84.0 * h, "flops": 1500.0 * e + 900.0 * n}


# ---- 64-bit restatement ------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind == "residual":
        return _exact_residual(case, seed)
    if kind == "chem_rates":
        rho, T = _chem_points(case["n"], seed)
        return {"w": _rates(torch.from_numpy(rho), torch.from_numpy(T))}
    if kind == "chem_first_order":
        return _exact_chem(case, seed, 1)
    if kind == "chem_second_order":
        return _exact_chem(case, seed, 2)
    # a Newton step and the source Jacobian rest on one-sided differences with
    # h = 1e-8, whose rounding noise has no exact value; the network's
    # activations are rounded to bfloat16 between layers
    return None


def _col(mesh):
    """The mesh arrays as tensors."""
    t = lambda a: torch.from_numpy(np.array(a)).cuda()  # noqa: E731
    e, b = t(mesh.edges).long(), t(mesh.bedges).long()
    return dict(L=e[:, 0], R=e[:, 1], a=t(mesh.edge_area), bL=b[:, 0], bR=b[:, 1], ba=t(mesh.bedge_area),
                tag=t(mesh.bfactag).long(), xyz=t(mesh.xyz), vol=t(mesh.vol), sw=t(mesh.sw), n=mesh.nnode)


def _ranked(m, which):
    """The chosen half-edges grouped by their rank within their node."""
    ids = torch.nonzero(which).flatten()
    node = m["bL"][ids]
    order = torch.argsort(node, stable=True)
    ids, node = ids[order], node[order]
    k = torch.arange(len(ids), device=ids.device)
    first = torch.ones_like(node, dtype=torch.bool)
    first[1:] = node[1:] != node[:-1]
    rank = k - torch.cummax(torch.where(first, k, torch.zeros_like(k)), 0).values if len(ids) else k
    return [ids[rank == r] for r in range(int(rank.max()) + 1 if len(ids) else 0)]


def _complete(q):
    """The auxiliary variables of ideal-gas rows."""
    u = q[:, 1:4] / q[:, :1]
    P = (GAMMA - 1.0) * (q[:, 4] - 0.5 * q[:, 0] * (u * u).sum(1))
    return torch.cat([q[:, :5], (GAMMA * P / q[:, 0])[:, None], P[:, None], u], 1)


def _pressure(q):
    return (GAMMA - 1.0) * (q[:, 4] - 0.5 * (q[:, 1:4] ** 2).sum(1) / q[:, 0])


def _farfield(QL, QR, nrm, qinf):
    """Ten sub-iterations of the characteristic far-field condition."""
    QR = QR.clone()
    done = torch.zeros(len(QR), dtype=torch.bool, device=QR.device)
    pi, ui = QL[:, 6], QL[:, 1:4] / QL[:, :1]
    pinf, uinf = qinf[6], qinf[1:4] / qinf[0]
    for _ in range(10):
        t = 0.5 * (QL[:, :5] + QR[:, :5])
        th = ((t[:, 1:4] / t[:, :1]) * nrm).sum(1)
        pa = _pressure(t)
        c2 = GAMMA * pa / t[:, 0]
        c = c2.sqrt()
        done |= ~((th > 0) | (th < 0))
        out, sup = th > 0, (th / c).abs() >= 1.0
        po = pinf.expand_as(pi)
        pin = 0.5 * (pinf + pi + t[:, 0] * c * (nrm * (uinf - ui)).sum(1))
        pb = torch.where(out, po, pin)
        base_p = torch.where(out, pi, pinf)
        rb = torch.where(out, QL[:, 0], qinf[0]) + (pb - base_p) / c2
        k = (pb - base_p) / (t[:, 0] * c)
        ub = torch.where(out[:, None], ui - nrm * k[:, None], uinf + nrm * k[:, None])
        new = torch.cat([rb[:, None], rb[:, None] * ub,
                         (pb / (GAMMA - 1.0) + 0.5 * rb * (ub * ub).sum(1))[:, None]], 1)
        new = torch.where(sup[:, None], torch.where(out[:, None], QL[:, :5], qinf[None, :5]), new)
        QR[:, :5] = torch.where(done[:, None], QR[:, :5], new)
    return _complete(QR)


def _slip(QL, QR, nrm):
    """Ten sub-iterations of the characteristic slip wall (and symmetry)."""
    QR = QR.clone()
    pi, ui = QL[:, 6], QL[:, 1:4] / QL[:, :1]
    th = (ui * nrm).sum(1)
    for _ in range(10):
        t = 0.5 * (QL[:, :5] + QR[:, :5])
        c2 = GAMMA * _pressure(t) / t[:, 0]
        rc = t[:, 0] * c2.sqrt()
        pb = pi + rc * th
        rb = QL[:, 0] + (pb - pi) / c2
        ub = ui - nrm * ((pb - pi) / rc)[:, None]
        QR[:, :5] = torch.cat([rb[:, None], rb[:, None] * ub,
                               (pb / (GAMMA - 1.0) + 0.5 * rb * (ub * ub).sum(1))[:, None]], 1)
    return _complete(QR)


def _normal_nodes(mesh, ids):
    """The neighbour of each wall half-edge's node most along its normal."""
    ids = ids.cpu().numpy()
    node = mesh.bedges[ids, 0].astype(np.int64)
    cnt = mesh.ipsp[node + 1] - mesh.ipsp[node]
    rep = np.repeat(np.arange(len(ids)), cnt)
    off = np.arange(len(rep)) - np.repeat(np.cumsum(cnt) - cnt, cnt)
    nb = mesh.psp[mesh.ipsp[node][rep] + off]
    d = mesh.xyz[nb] - mesh.xyz[node[rep]]
    d /= np.sqrt((d * d).sum(1))[:, None]
    dot = -(d * mesh.bedge_area[ids][rep, :3]).sum(1)
    order = np.lexsort((off, dot, rep))
    last = np.append(rep[order][1:] != rep[order][:-1], True)
    return torch.from_numpy(nb[order][last].astype(np.int64)).cuda()


def _boundary(mesh, m, p, q):
    """The boundary update of every half-edge."""
    types = torch.tensor([p.bc_type.get(t, -1) for t in range(max(p.bc_type) + 1)], device="cuda")[m["tag"]]
    qinf = torch.zeros(10, dtype=torch.float64, device="cuda")
    qinf[0], qinf[1] = GAMMA, GAMMA * p.mach
    qinf[4] = 1.0 / (GAMMA - 1.0) + 0.5 * GAMMA * p.mach ** 2
    qinf = _complete(qinf[None])[0]
    hard = torch.zeros(m["n"], dtype=torch.bool, device="cuda")
    is_hard = (types == N.BC_NOSLIP) | (types == N.BC_SONIC_INFLOW)
    hard[m["bL"][is_hard]] = True
    normal = torch.full_like(m["bL"], -1)
    ns = torch.nonzero(types == N.BC_NOSLIP).flatten()
    if len(ns):
        normal[ns] = _normal_nodes(mesh, ns)
    old = q.clone()

    def apply(ids):
        L, R, nrm = m["bL"][ids], m["bR"][ids], m["ba"][ids, :3]
        bt = types[ids]
        for t, f in ((N.BC_FARFIELD, lambda a, b, c: _farfield(a, b, c, qinf)), (N.BC_IMPERMEABLE_WALL, _slip),
                     (N.BC_SYMMETRY, _slip)):
            w = bt == t
            q[R[w]] = f(q[L[w]], q[R[w]], nrm[w])
        w = bt == N.BC_SONIC_OUTFLOW
        q[R[w]] = _complete(q[L[w]])
        w = bt == N.BC_SONIC_INFLOW
        q[R[w]] = qinf
        q[L[w]] = qinf
        w = bt == N.BC_NOSLIP
        if w.any():
            nq = old[normal[ids[w]]]
            z = torch.zeros_like(nq[:, :1])
            row = _complete(torch.cat([nq[:, :1], z, z, z, nq[:, 4:5]], 1))
            q[R[w]] = row
            q[L[w]] = row

    apply(torch.nonzero(~hard[m["bL"]]).flatten())
    for ids in _ranked(m, hard[m["bL"]]):
        apply(ids)
    return types


def _lsq(m, f):
    """Inverse-distance weighted least-squares gradient of the columns of f."""
    s11, s12, s13, s22, s23, s33 = [c[:, None] for c in m["sw"].T]
    r12, r13 = s12 / s11, s13 / s11
    r22 = s22 - s12 * r12
    r23 = s23 - r12 * s13
    r33 = s33 - s13 * r13 - r23 * (r23 / r22)
    g = torch.zeros((m["n"], f.shape[1], 3), dtype=torch.float64, device=f.device)
    d = m["xyz"][m["R"]] - m["xyz"][m["L"]]
    w = 1.0 / (d * d).sum(1, keepdim=True).sqrt()
    d = d * w
    for me, sgn, other in ((m["L"], 1.0, m["R"]), (m["R"], -1.0, m["L"])):
        x = sgn * d
        y = x[:, 1:2] - r12[me] * x[:, :1]
        c2 = (x[:, 2:] - r13[me] * x[:, :1] - (r23 / r22)[me] * y) / r33[me]
        c1 = (y - r23[me] * c2) / r22[me]
        c0 = (x[:, :1] - s12[me] * c1 - s13[me] * c2) / s11[me]
        c = torch.cat([c0, c1, c2], 1) * w
        g.index_add_(0, me, (f[other] - f[me])[:, :, None] * c[:, None, :])
    return g


def _symmetric(m, g, on):
    """The normal part of the gradient removed on symmetry half-edges, in order."""
    for ids in _ranked(m, on):
        nrm = m["ba"][ids, :3]
        gl = g[m["bL"][ids]]
        g[m["bL"][ids]] = gl - (gl * nrm[:, None, :]).sum(2, keepdim=True) * nrm[:, None, :]
    return g


def _limit(m, f, g, kind):
    """The limiter of the columns of f before the clamp to zero, and each
    edge end's gradient extrapolation to the midpoint."""
    h = 0.5 * (m["xyz"][m["R"]] - m["xyz"][m["L"]])
    lo, hi = torch.zeros_like(f[:m["n"]]), torch.zeros_like(f[:m["n"]])
    lim = torch.ones_like(lo)
    ext = []
    for me, other in ((m["L"], m["R"]), (m["R"], m["L"])):
        idx = me[:, None].expand(-1, f.shape[1])
        lo.scatter_reduce_(0, idx, f[other], "amin")
        hi.scatter_reduce_(0, idx, f[other], "amax")
    ep2 = 6.0 * math.pi * m["vol"][:, None]
    for me, x in ((m["L"], h), (m["R"], -h)):
        own = f[me]
        e = g[me, :f.shape[1], 0] * x[:, :1] + g[me, :f.shape[1], 1] * x[:, 1:2] + g[me, :f.shape[1], 2] * x[:, 2:]
        ext.append(e)
        dm = (own + e) - own
        dp = torch.where(dm > 0, hi[me] - own, lo[me] - own)
        if kind == 3:
            t = (dp * dp + ep2[me] + 2 * dm * dp) / (dp * dp + 2 * dm * dm + dm * dp + ep2[me])
        else:
            t = torch.where(dm == 0, torch.ones_like(dm), dp / torch.where(dm == 0, torch.ones_like(dm), dm))
            t = t.clamp(0.0, 1.0) if kind == 1 else (t * t + 2 * t) / (t * t + t + 2)
        lim.scatter_reduce_(0, me[:, None].expand(-1, f.shape[1]), t, "amin")
    return lim, ext


def _roe_average(a, b):
    ha, hb = (a[:, 4] + _pressure(a)) / a[:, 0], (b[:, 4] + _pressure(b)) / b[:, 0]
    rho = (a[:, 0] * b[:, 0]).sqrt()
    s = (rho / (a[:, 0] + rho))[:, None]
    ua, ub = a[:, 1:4] / a[:, :1], b[:, 1:4] / b[:, :1]
    u = ua + s * (ub - ua)
    h = ha + s[:, 0] * (hb - ha)
    k = 0.5 * (u * u).sum(1)
    E = rho / GAMMA * (h + (GAMMA - 1.0) * k)
    return torch.cat([rho[:, None], rho[:, None] * u, E[:, None]], 1), u, h, k


def _unphysical(q):
    return (_pressure(q) < 1e-10) | (q[:, 0] < 0) | (q[:, 4] < 1e-10)


def _clip(m, q, ext, raw):
    """Nodes whose limited extrapolation, or its Roe average with a neighbour's, is not physical."""
    a, b = q[m["L"], :5] + ext[0] * raw[m["L"]], q[m["R"], :5] + ext[1] * raw[m["R"]]
    both = _unphysical(_roe_average(a, b)[0])
    bad = torch.zeros(m["n"], dtype=torch.bool, device=q.device)
    bad[m["L"][_unphysical(a) | both]] = True
    bad[m["R"][_unphysical(b) | both]] = True
    return bad


def _roe(a, b, area):
    """Roe's flux with the Harten-Hyman entropy fix, out of the left state."""
    nrm, A = area[:, :3], area[:, 3:]
    ua, ub = a[:, 1:4] / a[:, :1], b[:, 1:4] / b[:, :1]
    pa, pb = _pressure(a), _pressure(b)
    ta, tb = (ua * nrm).sum(1), (ub * nrm).sum(1)
    ca, cb = (GAMMA * pa / a[:, 0]).sqrt(), (GAMMA * pb / b[:, 0]).sqrt()
    _, u, h, k = _roe_average(a, b)
    c2 = (GAMMA - 1.0) * (h - k)
    c = c2.sqrt()
    th = (u * nrm).sum(1)

    def fixed(x, xa, xb):
        eps = torch.maximum(x - xa, xb - x).clamp(min=0.0)
        return torch.where(x.abs() < eps, 0.5 * (x * x / torch.where(eps > 0, eps, torch.ones_like(eps)) + eps),
                           x.abs())

    l0, l1, l2 = fixed(th, ta, tb), fixed(th + c, ta + ca, tb + cb), fixed(th - c, ta - ca, tb - cb)
    d = b - a
    rdv = (nrm * d[:, 1:4]).sum(1) - th * d[:, 0]
    dp = (GAMMA - 1.0) * (d[:, 4] - (u * d[:, 1:4]).sum(1) + k * d[:, 0])
    ap, am = (l1 - l0) * (dp + c * rdv) / (2 * c2), (l2 - l0) * (dp - c * rdv) / (2 * c2)
    rp = lambda s: torch.cat([torch.ones_like(c)[:, None], u + (s * c)[:, None] * nrm,  # noqa: E731
                              (h + s * c * th)[:, None]], 1)
    diss = l0[:, None] * d + ap[:, None] * rp(1.0) + am[:, None] * rp(-1.0)

    def physical(q, p, t):
        return torch.cat([(q[:, 0] * t)[:, None], q[:, 1:4] * t[:, None] + p[:, None] * nrm,
                          ((q[:, 4] + p) * t)[:, None]], 1)

    return 0.5 * A * (physical(a, pa, ta) + physical(b, pb, tb) - diss)


def _viscous(p, Q, g, area):
    """Laminar viscous flux from a face state [.][5] and the face gradients of T, u, v, w [.][4][3]."""
    nrm = area[:, :3]
    u = Q[:, 1:4] / Q[:, :1]
    T = GAMMA * _pressure(Q) / Q[:, 0]
    S = 110.4 / p.ref_temperature
    mu = (1.0 + S) * T ** 1.5 / (T + S)
    du = g[:, 1:4]
    div = du.diagonal(dim1=1, dim2=2).sum(1)
    tau = du + du.transpose(1, 2) - (2.0 / 3.0) * div[:, None, None] * torch.eye(3, dtype=Q.dtype, device=Q.device)
    tn = (tau * nrm[:, None, :]).sum(2)
    k = (area[:, 3] * p.mach / p.Re * mu)[:, None]
    heat = (g[:, 0] * nrm).sum(1, keepdim=True) / ((GAMMA - 1.0) * p.Pr)
    return torch.cat([torch.zeros_like(k), -k * tn, -k * ((tn * u).sum(1, keepdim=True) + heat)], 1)


def _assemble(m, f, fb):
    b = torch.zeros((m["n"], f.shape[1]), dtype=torch.float64, device=f.device)
    b.index_add_(0, m["L"], -f)
    b.index_add_(0, m["R"], f)
    b.index_add_(0, m["bL"], -fb)
    return b


def _norms(b):
    per = b.square().sum(0)
    return torch.cat([(per.sum().sqrt() / b.numel())[None], per.sqrt() / b.shape[0]])


def _exact_residual(case, seed):
    mesh, p = _flow_case(case)
    m = _col(mesh)
    q = torch.from_numpy(np.array(_state(mesh, p, case["state"], seed))).cuda()
    start = q[:m["n"], :5].clone()
    types = _boundary(mesh, m, p, q)
    a, b = q[m["L"], :5], q[m["R"], :5]
    if p.sorder > 1:
        cols = q[:, [0, 1, 2, 3, 4, 5, 7, 8, 9]]
        g = _symmetric(m, _lsq(m, cols), types == N.BC_SYMMETRY)
        raw, ext = _limit(m, q[:, :5], g, p.limiter)
        lim = torch.where(_clip(m, q, ext, raw)[:, None], torch.zeros_like(raw), raw.clamp(min=0.0))
        a, b = a + ext[0] * lim[m["L"]], b + ext[1] * lim[m["R"]]
    f = _roe(a, b, m["a"])
    fb = _roe(q[m["bL"], :5], q[m["bR"], :5], m["ba"])
    if p.viscous:
        dx = m["xyz"][m["R"]] - m["xyz"][m["L"]]
        gf = 0.5 * (g[m["L"], 5:] + g[m["R"], 5:])
        dq = cols[m["R"], 5:] - cols[m["L"], 5:]
        gf = gf + ((dq - (gf * dx[:, None, :]).sum(2)) / (dx * dx).sum(1, keepdim=True))[:, :, None] * dx[:, None, :]
        f = f + _viscous(p, 0.5 * (q[m["L"], :5] + q[m["R"], :5]), gf, m["a"])
        fb = fb + _viscous(p, 0.5 * (q[m["bL"], :5] + q[m["bR"], :5]), g[m["bL"], 5:], m["ba"])
    r = _assemble(m, f, fb)
    r = r + m["vol"][:, None] * (q[:m["n"], :5] - start)   # steady temporal term, dt = -1
    r[m["bL"][types == N.BC_NOSLIP]] = 0.0                 # adiabatic no-slip rows
    return {"b": r, "norms": _norms(r)}


# reacting set

def _curves(T, dev):
    """Per species cp/R, h/(RT)*T and the curve coefficients in force at T [K]."""
    spec = _mechanism()["species"]
    lo = torch.tensor([s["lo"] for s in spec], dtype=torch.float64, device=dev)
    hi = torch.tensor([s["hi"] for s in spec], dtype=torch.float64, device=dev)
    return torch.where((T > 1000.0)[:, None, None], hi, lo)


def _gas(dev):
    mw = torch.tensor([s["MW"] for s in _mechanism()["species"]], dtype=torch.float64, device=dev)
    return mw, 8.31447215 / mw


def _cp_h(T):
    mw, R = _gas(T.device)
    a, t = _curves(T, T.device), T[:, None]
    cp = R * (a[..., 0] + t * (a[..., 1] + t * (a[..., 2] + t * (a[..., 3] + t * a[..., 4]))))
    h = R * (a[..., 5] + t * (a[..., 0] + t * (a[..., 1] / 2 + t * (a[..., 2] / 3 + t * (a[..., 3] / 4 + t * a[..., 4] / 5)))))
    return cp, h


def _rates(rho, T):
    """Mass production rates [kg/(m^3 s)] of the mechanism."""
    mw, _ = _gas(rho.device)
    X = rho / mw
    a = _curves(T, rho.device)
    w = torch.zeros_like(rho)
    for r in _mechanism()["reactions"]:
        kf = r["A"] * T ** r["n"] * torch.exp(-r["EA"] / T)   # this mechanism's form (activation temperature)
        d = torch.zeros((len(T), 7), dtype=torch.float64, device=rho.device)
        form, dest, nu = torch.ones_like(T), torch.ones_like(T), 0.0
        for g, up, upp in zip(r["global"], r["nup"], r["nupp"]):
            d += (upp - up) * a[:, g]
            nu += upp - up
            form, dest = form * X[:, g] ** up, dest * X[:, g] ** upp
        kp = torch.exp(d[:, 0] * (T.log() - 1) + T * (d[:, 1] / 2 + T * (d[:, 2] / 6 + T * (d[:, 3] / 12 + d[:, 4] / 20 * T)))
                       - d[:, 5] / T + d[:, 6])
        net = kf * form - kf / (kp * (101325.0 / (8.31447215 * T)) ** nu) * dest
        if r["third_bodies"]:
            M = X.sum(1)
            for g, e in zip(r["global"], r["tbeff"]):
                M = M + (e - 1.0) * X[:, g]
            net = net * M
        for g, up, upp in zip(r["global"], r["nup"], r["nupp"]):
            w[:, g] += (upp - up) * net * mw[g]
    return w


def _sound2(ref, rhoi, T):
    """Frozen speed of sound squared, non-dimensional."""
    _, R = _gas(T.device)
    td = T * ref.temperature
    cp, _ = _cp_h(td)
    Y = rhoi / rhoi.sum(1, keepdim=True)
    cpm, Rm = (Y * cp).sum(1), (Y * R).sum(1)
    return cpm / (cpm - Rm) * Rm * td / ref.velocity ** 2


def _hllc(ref, a, b, area):
    """HLLC flux of reacting states [.][rho_i, u, v, w, T] (beta = 1, no gauge pressure)."""
    nrm, A = area[:, :3], area[:, 3:]
    _, Rg = _gas(a.device)
    side = []
    for q in (a, b):
        rho, u, T = q[:, :NS].sum(1), q[:, NS:NS + 3], q[:, NS + 3]
        P = (q[:, :NS] * ref.density * Rg).sum(1) * T * ref.temperature / ref.pressure
        h = (q[:, :NS] * _cp_h(T * ref.temperature)[1]).sum(1) / ref.specific_enthalpy
        side.append((rho, u, P, h + 0.5 * rho * (u * u).sum(1) - P, (u * nrm).sum(1), _sound2(ref, q[:, :NS], T).sqrt()))
    (ra, ua, pa, Ea, ta, ca), (rb, ub, pb, Eb, tb, cb) = side
    s = (ra * rb).sqrt()
    s = (s / (ra + s))[:, None]
    roe = a + s * (b - a)
    c, th = _sound2(ref, roe[:, :NS], roe[:, NS + 3]).sqrt(), (roe[:, NS:NS + 3] * nrm).sum(1)
    SL, SR = torch.minimum(ta - ca, th - c), torch.maximum(tb + cb, th + c)
    SM = (pb - pa + ra * ta * (SL - ta) - rb * tb * (SR - tb)) / (ra * (SL - ta) - rb * (SR - tb))
    left = SM >= 0
    pick = lambda x, y: torch.where(left if x.dim() == 1 else left[:, None], x, y)  # noqa: E731
    q, rho, u, P, E, t, S = (pick(x, y) for x, y in zip((a, ra, ua, pa, Ea, ta, SL), (b, rb, ub, pb, Eb, tb, SR)))
    ps = P + rho * (t - S) * (t - SM)
    om, k = 1.0 / (S - SM), S - t
    sup_l, sup_r = SL >= 0, SR <= 0
    sup = sup_l | sup_r
    out = []
    star = torch.cat([(om * k)[:, None] * q[:, :NS], om[:, None] * ((k * rho)[:, None] * u + (ps - P)[:, None] * nrm),
                      (om * (k * E - P * t + ps * SM))[:, None]], 1)
    fs = torch.cat([star[:, :NS] * SM[:, None], star[:, NS:NS + 3] * SM[:, None] + ps[:, None] * nrm,
                    ((star[:, NS + 3] + ps) * SM)[:, None]], 1)
    for qq, r_, u_, p_, e_, t_ in ((a, ra, ua, pa, Ea, ta), (b, rb, ub, pb, Eb, tb)):
        out.append(torch.cat([qq[:, :NS] * t_[:, None], (r_ * t_)[:, None] * u_ + p_[:, None] * nrm,
                              ((e_ + p_) * t_)[:, None]], 1))
    return A * torch.where(sup[:, None], torch.where(sup_l[:, None], out[0], out[1]), fs)


def _transport(ref, rhoi, T):
    """Wilke's mixture viscosity and conductivity, non-dimensional."""
    mw, _ = _gas(T.device)
    td = T * ref.temperature
    X = rhoi / rhoi.sum(1, keepdim=True) / mw
    X = X / X.sum(1, keepdim=True)
    mu, k = torch.empty_like(rhoi), torch.empty_like(rhoi)
    for s, sp in enumerate(_mechanism()["species"]):
        for out, key, conv, ref_val, sut in ((mu, "mu", 1e-7, 1.716e-5, 111.0), (k, "k", 1e-4, 0.0241, 194.0)):
            v = ref_val * (td / 273.0) ** 1.5 * (273.0 + sut) / (td + sut)
            for lo, hi, c0, c1, c2, c3 in sp[key]:
                fit = torch.exp(c0 * td.log() + c1 / td + c2 / (td * td) + c3) * conv
                v = torch.where((td > 1000.0) & (td >= lo) & (td <= hi), fit, v)
            out[:, s] = v
    wsum = torch.zeros_like(mu)
    for i in range(NS):
        for j in range(NS):
            t = 1.0 + (mu[:, i] / mu[:, j]).sqrt() * (mw[j] / mw[i]) ** 0.25
            wsum[:, i] += X[:, j] * t * t / (8.0 * (1.0 + mw[i] / mw[j])).sqrt()
    return (X / wsum * mu).sum(1) / ref.viscosity, (X / wsum * k).sum(1) / ref.conductivity


def _chem_viscous(ref, Q, g, area):
    """Laminar viscous flux of the reacting set; g: face gradients of u, v, w, T [.][4][3]."""
    nrm = area[:, :3]
    mu, kc = _transport(ref, Q[:, :NS], Q[:, NS + 3])
    du = g[:, :3]
    div = du.diagonal(dim1=1, dim2=2).sum(1)
    off = du + du.transpose(1, 2)
    # diagonal 4/3 of the own derivative less 2/3 of the others; off-diagonal the plain sum
    tau = off - (2.0 / 3.0) * div[:, None, None] * torch.eye(3, dtype=Q.dtype, device=Q.device)
    tn = -(tau * nrm[:, None, :]).sum(2)
    rk = (area[:, 3] / CHEM_RE)[:, None]
    e = rk * mu[:, None] * (tn * Q[:, NS:NS + 3]).sum(1, keepdim=True) - rk * kc[:, None] * (g[:, 3] * nrm).sum(1, keepdim=True)
    return torch.cat([torch.zeros_like(Q[:, :NS]), rk * mu[:, None] * tn, e], 1)


def _exact_chem(case, seed, order):
    mesh = _grid("ns", case["nx"], case["ny"], case["nz"])[0]
    m, ref = _col(mesh), _chem_full_ref()
    q = torch.from_numpy(_chem_field(np.concatenate([mesh.xyz, mesh.xyz[mesh.bedges[:, 0]]]), seed)).cuda()
    nat = q[:, :NS + 4]
    a, b = nat[m["L"]], nat[m["R"]]
    out = {}
    if order == 2:
        cols = torch.cat([nat, q[:, 2 * NS + 6:]], 1)
        on = torch.zeros_like(m["tag"], dtype=torch.bool)
        for t in (5, 6, 7):
            on |= m["tag"] == t
        g = _symmetric(m, _lsq(m, cols), on)
        raw, ext = _limit(m, nat, g, 3)
        lim = raw.clamp(min=0.0)
        a, b = a + ext[0] * lim[m["L"]], b + ext[1] * lim[m["R"]]
        out["grad"], out["lim"] = g, lim
    src = _rates(nat[:m["n"], :NS] * ref.density, nat[:m["n"], NS + 3] * ref.temperature) / (ref.density / REF_TIME)
    r = _assemble(m, _hllc(ref, a, b, m["a"]), _hllc(ref, nat[m["bL"]], nat[m["bR"]], m["ba"]))
    r[:, :NS] += m["vol"][:, None] * src
    out["b"], out["norms"] = r, _norms(r)
    if order == 2:
        dx = m["xyz"][m["R"]] - m["xyz"][m["L"]]
        gf = 0.5 * (g[m["L"], NS:NS + 4] + g[m["R"], NS:NS + 4])
        dq = (nat[m["R"]] - nat[m["L"]])[:, NS:]
        gf = gf + ((dq - (gf * dx[:, None, :]).sum(2)) / (dx * dx).sum(1, keepdim=True))[:, :, None] * dx[:, None, :]
        fv = _chem_viscous(ref, 0.5 * (nat[m["L"]] + nat[m["R"]]), gf, m["a"])
        fb = _chem_viscous(ref, 0.5 * (nat[m["bL"]] + nat[m["bR"]]), g[m["bL"], NS:NS + 4], m["ba"])
        out["bv"] = _assemble(m, fv, fb)
    return out
