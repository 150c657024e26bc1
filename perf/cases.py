"""The work that users of the forward-path library have it do, as timed cases.

A case is one call sequence through the public entry points on one mesh:

* request   tg_forward_path: Reset, forward and adjoint solves, projections and
            the nodal Jacobian of a new parameter set (a Gauss-Newton step);
* fields    Reset and CalcFields with one of the solvers a user can select;
* jacobian  the nodal Jacobian from fields in hand;
* grid      the Jacobian on a pixel raster from fields in hand;
* element   the element-basis Jacobian from fields in hand;
* gradient  Reset and the data gradient on a pixel raster.

Meshes are the package's seeded workloads (2D disc, 3D cylinder, 3D box) and
are kept with their solver between passes, as a user's program keeps them; the
optical parameters, optode positions, sources, fields and data come from the
seed.  All arrays are device memory.
"""
import functools
import math

import numpy as np
import torch

from toastpp_gb300 import capi, workloads

DEV = "cuda"
WIDTH = 2.0      # Gaussian optode width [mm]
NREF = 1.4
RADIUS = 25.0    # disc and cylinder [mm]
BOX = (80.0, 80.0, 60.0)


def listed():
    return [
        # the smallest request: a coarse 2D slice, few optodes; launches and host reads count
        dict(name="request_disc217_fd", kind="request", mesh="disc", a=8, b=0, nq=4, nm=4, mhz=100.0,
             solver="BICGSTAB", fp32=0),
        # the 2D CW benchmark configuration (3.2k nodes, 16 + 16 optodes, CG)
        dict(name="request_disc3k_cw", kind="request", mesh="disc", a=32, b=0, nq=16, nm=16, mhz=0.0, solver="CG",
             fp32=0),
        # the headline configuration: 30k-node cylinder, 100 MHz, 80 + 80 optodes, FP64 Jacobian
        dict(name="request_cyl30k_fd", kind="request", mesh="cylinder", a=18, b=30, nq=80, nm=80, mhz=100.0,
             solver="BICGSTAB", fp32=0),
        # fields on a large box for an odd number of sources (a user without Jacobian needs)
        dict(name="fields_box106k_fd", kind="fields", mesh="box", a=48, b=46, k=37, mhz=100.0, solver="BICGSTAB",
             precision="mixed"),
        # the reference's own recursion in FP64 on the 2D 100 MHz configuration
        dict(name="fields_disc13k_fp64", kind="fields", mesh="disc", a=64, b=0, k=32, mhz=100.0, solver="BICGSTAB",
             precision="fp64"),
        # LSOLVER_DIRECT: factor and solve at every parameter update
        dict(name="fields_disc3k_direct", kind="fields", mesh="disc", a=32, b=0, k=32, mhz=100.0, solver="DIRECT",
             precision="fp64"),
        # CW reconstruction in 3D: FP64 nodal Jacobian of real fields
        dict(name="jacobian_cyl30k_cw", kind="jacobian", mesh="cylinder", a=18, b=30, nq=80, nm=80, mhz=0.0, fp32=0),
        # the request server's default: FP32 nodal Jacobian of complex fields
        dict(name="jacobian_cyl30k_fp32", kind="jacobian", mesh="cylinder", a=18, b=30, nq=80, nm=80, mhz=100.0,
             fp32=1),
        # toast.Raster Jacobian on a 32^3 raster, the benchmark's grid workload
        dict(name="grid_cyl30k_32", kind="grid", mesh="cylinder", a=18, b=30, nq=80, nm=80, mhz=100.0, g=32, fp32=1),
        # element basis on the small cylinder, FP32 storage
        dict(name="element_cyl7k", kind="element", mesh="cylinder", a=12, b=16, nq=80, nm=80, mhz=100.0, fp32=1),
        # CW element basis in FP64 in 2D, ragged sizes
        dict(name="element_disc11k_cw", kind="element", mesh="disc", a=61, b=0, nq=31, nm=33, mhz=0.0, fp32=0),
        # a nonlinear conjugate-gradient step in 2D: data gradient on a 64 x 64 raster
        dict(name="gradient_disc13k", kind="gradient", mesh="disc", a=64, b=0, nq=32, nm=32, mhz=100.0, g=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["request", "request", "fields", "fields", "jacobian", "grid", "element", "gradient"])
    two_d = rng.random() < 0.5
    mhz = 0.0 if rng.random() < 0.4 else 100.0
    if two_d:
        c = dict(kind=kind, mesh="disc", a=_log_int(rng, 8, 64), b=0)
    elif kind == "fields" and rng.random() < 0.4:
        c = dict(kind=kind, mesh="box", a=_log_int(rng, 8, 40), b=_log_int(rng, 8, 40))
    else:
        c = dict(kind=kind, mesh="cylinder", a=_log_int(rng, 6, 16), b=_log_int(rng, 8, 28))
    if kind == "fields":
        c.update(k=_log_int(rng, 1, 64), mhz=mhz)
        how = rng.random()
        if how < 0.6:
            c.update(solver="BICGSTAB" if mhz or rng.random() < 0.5 else "CG", precision="mixed")
        elif how < 0.8 or not two_d:
            c.update(solver="BICGSTAB" if mhz else "CG", precision="fp64", k=min(c["k"], 32))
        elif how < 0.9:
            c.update(solver="DIRECT", precision="fp64", a=min(c["a"], 40))
        else:
            c.update(solver="GMRES", precision="fp64", a=min(c["a"], 32), k=min(c["k"], 16))
        return c
    c.update(nq=_log_int(rng, 3, 64), nm=_log_int(rng, 3, 64), mhz=mhz)
    if kind == "request":
        c.update(solver="BICGSTAB" if mhz or rng.random() < 0.5 else "CG", fp32=int(rng.random() < 0.4))
    elif kind == "jacobian":
        c.update(fp32=int(rng.random() < 0.4))
    elif kind == "grid":
        c.update(g=_log_int(rng, 12, 80 if two_d else 40), fp32=int(rng.random() < 0.6))
    elif kind == "element":
        c.update(fp32=int(rng.random() < 0.6))
        if not two_d:
            c.update(b=min(c["b"], 16), a=min(c["a"], 12))
    else:
        c.update(mhz=100.0, g=_log_int(rng, 12, 80 if two_d else 32))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _geometry(mesh, a, b):
    """coords, elements and the boundary-node mask of a workload mesh."""
    if mesh == "disc":
        p = workloads.disc(a, 0, 0.0, 4)
    elif mesh == "cylinder":
        p = workloads.cylinder(a, b, 0)
    else:
        p = workloads.box(a, a, b, seed=0, nq=16)
    dim = p.coords.shape[1]
    sides = _sides(p.elems)
    key = np.sort(sides, 1).astype(np.int64)
    code = key[:, 0]
    for d in range(1, dim):
        code = code * p.n + key[:, d]
    _, inv, cnt = np.unique(code, return_inverse=True, return_counts=True)
    faces = sides[cnt[inv] == 1]
    bnd = np.zeros(p.n, bool)
    bnd[faces] = True
    return p.coords, p.elems, bnd, faces


def _sides(el):
    nn = el.shape[1]
    return np.concatenate([np.delete(el, i, 1) for i in range(nn)])


def _optodes(case, count, rng, detectors):
    """count positions on the mesh's boundary; detectors sit between the sources."""
    i = np.arange(count)
    turn = rng.uniform(0, 2 * np.pi) + (0.5 if detectors else 0.0) * 2 * np.pi / max(count, 1)
    if case["mesh"] == "disc":
        t = turn + 2 * np.pi * i / count
        return np.stack([RADIUS * np.cos(t), RADIUS * np.sin(t)], 1)
    if case["mesh"] == "cylinder":
        rings = 5 if count >= 10 else 1
        per = -(-count // rings)
        t = turn + 2 * np.pi * (i // rings) / per
        z = np.linspace(-20.0, 20.0, rings)[i % rings] if rings > 1 else np.zeros(count)
        return np.stack([RADIUS * np.cos(t), RADIUS * np.sin(t), z], 1)
    side = math.ceil(math.sqrt(count))
    g = np.linspace(12.0, 68.0, max(side, 2))
    sh = rng.uniform(-2, 2, 2)
    return np.stack([g[i % side] + sh[0], g[i // side] + sh[1], np.full(count, BOX[2] if detectors else 0.0)], 1)


def _parameters(case, seed):
    """mua, mus, nref: the configurations' background with three seeded inclusions."""
    coords = _geometry(case["mesh"], case["a"], case["b"])[0]
    rng = np.random.default_rng([seed, 1])
    base = (0.025, 2.0) if case["mesh"] == "disc" else (0.01, 1.0)
    mua, mus = np.full(len(coords), base[0]), np.full(len(coords), base[1])
    lo, hi = coords.min(0), coords.max(0)
    for _ in range(3):
        c = lo + (0.25 + 0.5 * rng.random(coords.shape[1])) * (hi - lo)
        g = np.exp(-((coords - c) ** 2).sum(1) / (2 * 4.0 ** 2))
        f = 1 + rng.uniform(0.5, 2.0) * g
        mua, mus = mua * f, mus * f
    return mua, mus, np.full(len(coords), NREF)


def _coefficients(mua, mus, nref):
    """c mua, c kappa and c / 2A (Keijzer's boundary parameter), c = 0.3 mm/ps."""
    c0 = 0.3
    co = np.cos(np.arcsin(1.0 / nref))
    r0 = ((nref - 1.0) / (nref + 1.0)) ** 2
    big = (2.0 / (1.0 - r0) - 1.0 + np.abs(co) ** 3) / (1.0 - co ** 2)
    return mua * c0 / nref, c0 / (3.0 * nref * (mua + mus)), c0 / (2.0 * nref * big)


def _spots(case, pos, scale=None):
    """One Gaussian boundary source per position, on the device (npos x n)."""
    coords, _, bnd, _ = _geometry(case["mesh"], case["a"], case["b"])
    x = torch.as_tensor(coords, device=DEV)
    d2 = ((torch.as_tensor(pos, device=DEV)[:, None, :] - x[None]) ** 2).sum(-1)
    v = torch.exp(-d2 / (2 * WIDTH ** 2)) * torch.as_tensor(bnd, device=DEV)
    v = v / v.sum(1, keepdim=True)
    if scale is not None:
        v = v * torch.as_tensor(scale, device=DEV)
    return (v.to(torch.complex128) if case["mhz"] else v).contiguous()


def _decay(case):
    mua, mus = (0.025, 2.0) if case["mesh"] == "disc" else (0.01, 1.0)
    k = math.sqrt(3 * mua * (mua + mus))
    return k * (1 + 0.15j) if case["mhz"] else k


def _wave(case, points, pos, rng):
    """Diffusion-like fields of sources at pos, at the points: exp(-k r) / r with a smooth modulation."""
    x, p = torch.as_tensor(points, device=DEV), torch.as_tensor(pos, device=DEV)
    r = (((p[:, None, :] - x[None]) ** 2).sum(-1) + 1.0).sqrt()
    g = torch.as_tensor(rng.uniform(-0.2, 0.2, x.shape[1]), device=DEV)
    mod = 1 + 0.1 * torch.sin(x @ g)
    return (torch.exp(-_decay(case) * r) / r * mod).contiguous()


def _links(case):
    nq, nm = case["nq"], case["nm"]
    return np.arange(nq + 1, dtype=np.int32) * nm, np.tile(np.arange(nm, dtype=np.int32), nq)


def _inputs(case, seed):
    """What the case's call takes, from the seed alone."""
    rng = np.random.default_rng([seed, 2])
    coords = _geometry(case["mesh"], case["a"], case["b"])[0]
    out = {}
    kind = case["kind"]
    if kind in ("request", "fields", "gradient"):
        mua, mus, nref = _parameters(case, seed)
        out["coef"] = [torch.as_tensor(v, device=DEV) for v in _coefficients(mua, mus, nref)]
        nq = case["k"] if kind == "fields" else case["nq"]
        q = _optodes(case, nq, rng, False)
        out["qvec"] = _spots(case, q)
        if kind != "fields":
            m = _optodes(case, case["nm"], rng, True)
            out["mvec"] = _spots(case, m, out["coef"][2])
        if kind == "gradient":
            y = _wave(case, m, q, rng).reshape(-1)
            noise = torch.as_tensor(rng.normal(1.0, 0.05, (2, len(y))), device=DEV)
            d = torch.stack([y.abs().log(), y.angle()]) * noise
            out["data"] = d.reshape(-1).contiguous()
            out["sd"] = (0.05 * d.abs() + 0.01).reshape(-1).contiguous()
        return out
    q, m = _optodes(case, case["nq"], rng, False), _optodes(case, case["nm"], rng, True)
    out["dphi"] = _wave(case, coords, q, rng)
    out["aphi"] = _wave(case, coords, m, rng)
    out["proj"] = _wave(case, m, q, rng).reshape(-1).contiguous()
    return out


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
class _Kit:
    """What a user's program keeps: the mesh, the solver on its stream, the raster and the link list."""

    def __init__(self, case):
        coords, elems, _, _ = _geometry(case["mesh"], case["a"], case["b"])
        self.mesh = capi.Mesh(coords, elems)
        cplx = case["mhz"] != 0.0
        solver = case.get("solver") or ("BICGSTAB" if cplx else "CG")
        precision = case.get("precision", "mixed")
        self.solver = capi.FwdSolver(self.mesh, solver, 1e-12, "ICH", cplx, precision=precision)
        self.stream = torch.cuda.Stream()
        self.solver.set_stream(self.stream.cuda_stream)
        self.raster = None
        if "g" in case:
            self.raster = capi.Raster(self.mesh, [case["g"]] * self.mesh.dim)
        self.links = capi.Links(*_links(case)) if "nq" in case else None


@functools.lru_cache(maxsize=1)
def _kit(items):
    return _Kit(dict(items))


def prepare(case, seed):
    case = {k: v for k, v in case.items() if k != "name"}
    kit = _kit(tuple(sorted(case.items())))
    x = _inputs(case, seed)
    n, ne = kit.mesh.n, kit.mesh.ne
    cplx = case["mhz"] != 0.0
    dt = torch.complex128 if cplx else torch.float64
    jt = torch.float32 if case.get("fp32") else torch.float64
    kind = case["kind"]
    if kind == "fields":
        x["phi"] = torch.empty((case["k"], n), dtype=dt, device=DEV)
    elif kind == "request":
        x["dphi"] = torch.empty((case["nq"], n), dtype=dt, device=DEV)
        x["aphi"] = torch.empty((case["nm"], n), dtype=dt, device=DEV)
        x["proj"] = torch.empty(kit.links.nqm, dtype=dt, device=DEV)
        x["logproj"] = torch.empty(kit.links.nqm, dtype=dt, device=DEV)
    elif kind == "gradient":
        x["grad"] = torch.empty(2 * kit.raster.slen, dtype=torch.float64, device=DEV)
    if kind not in ("fields", "gradient"):
        cols = ne if kind == "element" else kit.raster.slen if kind == "grid" else n
        x["J"] = torch.empty((2 * kit.links.nqm, 2 * cols if cplx else cols), dtype=jt, device=DEV)
    torch.cuda.synchronize()
    return case, kit, x


def run(state):
    case, kit, x = state
    s, mem = kit.solver, capi.MEM_DEVICE
    omega = capi.omega_of(case["mhz"])
    kind = case["kind"]
    if kind == "request":
        cm, ck, ca = x["coef"]
        s.forward_path_raw(cm, ck, ca, omega, case["nq"], x["qvec"], case["nm"], x["mvec"], kit.links, x["dphi"],
                           x["aphi"], x["proj"], x["logproj"], x["J"], case["fp32"], mem)
        return {k: x[k] for k in ("dphi", "aphi", "proj", "logproj", "J")}
    if kind == "fields":
        s.reset(*x["coef"], omega, mem=mem)
        with torch.cuda.stream(kit.stream):
            x["phi"].zero_()
        s.calc_fields_raw(case["k"], x["qvec"], x["phi"], mem)
        return x["phi"]
    if kind == "gradient":
        s.reset(*x["coef"], omega, mem=mem)
        with torch.cuda.stream(kit.stream):
            x["grad"].zero_()
        L, p = kit.links, capi._ptr
        capi._check(capi.lib().tg_gradient(s._h, kit.raster._h, case["nq"], p(x["qvec"]), case["nm"], p(x["mvec"]),
                                           p(L.ofs), p(L.m), p(x["data"]), p(x["sd"]), p(x["grad"]), mem, None))
        return x["grad"]
    args = (case["nq"], x["dphi"], case["nm"], x["aphi"], x["proj"], kit.links, capi.DATA_LOG, x["J"], case["fp32"],
            mem)
    if kind == "grid":
        s.jacobian_grid_raw(kit.raster, *args)
    elif kind == "element":
        s.jacobian_el_raw(*args)
    else:
        L, p = kit.links, capi._ptr
        capi._check(capi.lib().tg_jacobian(s._h, case["nq"], p(x["dphi"]), case["nm"], p(x["aphi"]), p(x["proj"]),
                                           p(L.ofs), p(L.m), capi.DATA_LOG, p(x["J"]), case["fp32"], mem))
    return x["J"]


def work(case):
    """Inputs read once and outputs written once; operations of the products that form the outputs."""
    a, b = case["a"], case["b"]
    n2, e2 = 1 + 3 * a * (a + 1), 6 * a * a
    if case["mesh"] == "disc":
        n, ne, deg, nn = n2, e2, 7, 3
    elif case["mesh"] == "cylinder":
        n, ne, deg, nn = n2 * b, 3 * e2 * (b - 1), 14, 4
    else:
        n, ne, deg, nn = a * a * b, 6 * (a - 1) * (a - 1) * (b - 1), 14, 4
    v, mul = (16, 8) if case["mhz"] else (8, 2)
    kind = case["kind"]
    if kind == "fields":  # the right-hand sides and fields, the matrix, and one product with it
        k = case["k"]
        return dict(bytes=2 * v * n * k + 24 * n + v * n * deg, flops=mul * n * deg * k)
    nq, nm = case["nq"], case["nm"]
    links = nq * nm
    if kind == "gradient":
        gl = case["g"] ** (2 if case["mesh"] == "disc" else 3)
        return dict(bytes=v * n * (nq + nm) + 24 * n + 16 * gl + 32 * links, flops=mul * n * deg * 2 * nq)
    cols = ne if kind == "element" else (case["g"] ** (2 if nn == 3 else 3) * 3 // 4) if kind == "grid" else n
    per = nn if kind == "element" else nn if kind == "grid" else deg
    jb = 2 * links * cols * (2 if case["mhz"] else 1) * (4 if case["fp32"] else 8)
    fl = mul * links * cols * 2 * per
    fb = v * n * (nq + nm)
    if kind == "request":
        return dict(bytes=jb + 2 * fb + 24 * n + v * n * deg, flops=fl + mul * n * deg * (nq + nm))
    return dict(bytes=jb + fb + v * links, flops=fl)


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, with plain torch
# ---------------------------------------------------------------------------
def _elements(case):
    """vol (ne), gradients of the shape functions (ne x nn x dim), nodes, barycentric rows (ne x nn x (dim + 1))."""
    coords, el, _, faces = _geometry(case["mesh"], case["a"], case["b"])
    x = torch.as_tensor(coords, device=DEV)
    e = torch.as_tensor(el.astype(np.int64), device=DEV)
    p = x[e]
    m = torch.cat([torch.ones_like(p[..., :1]), p], -1)            # ne x nn x (dim + 1)
    bary = torch.linalg.inv(m).transpose(1, 2).contiguous()        # rows: constant and gradient of each shape function
    vol = torch.linalg.det(m).abs() / math.factorial(p.shape[2])
    return vol, bary[..., 1:], e, bary, x, torch.as_tensor(faces.astype(np.int64), device=DEV)


def _triple(nn):
    """IntFFF / size: 2 or 6 x multiplicities / (dim + 3)!."""
    t = torch.ones(nn, nn, nn, dtype=torch.float64, device=DEV)
    for i in range(nn):
        for j in range(nn):
            for k in range(nn):
                t[i, j, k] = {3: 1.0, 2: 2.0, 1: 6.0}[len({i, j, k})]
    return t / (60.0 if nn == 3 else 120.0)


def _solve(case, coef, rhs):
    """F phi = rhs for every row of rhs, by a dense factorisation with one refinement step."""
    vol, grad, e, _, x, faces = _elements(case)
    cm, ck, ca = (torch.as_tensor(v, device=DEV) for v in coef)
    nn, n = e.shape[1], len(x)
    ff = _triple(nn)
    k = torch.einsum("eid,ejd->eij", grad, grad) * (vol * ck[e].mean(1))[:, None, None]
    k = k + torch.einsum("el,lij->eij", cm[e], ff) * vol[:, None, None]
    dt = torch.complex128 if case["mhz"] else torch.float64
    a = torch.zeros(n, n, dtype=dt, device=DEV)
    mass = (torch.ones(nn, nn, dtype=torch.float64, device=DEV) + torch.eye(nn, dtype=torch.float64, device=DEV)) / (
        nn * (nn + 1))
    k = k.to(dt)
    if case["mhz"]:
        k = k + 1j * (2 * math.pi * case["mhz"] * 1e-6) * mass * vol[:, None, None]
    a.index_put_((e[:, :, None].expand(-1, nn, nn), e[:, None, :].expand(-1, nn, nn)), k, accumulate=True)
    q, nf = x[faces], faces.shape[1]
    size = (q[:, 1] - q[:, 0]).norm(dim=1) if nf == 2 else 0.5 * torch.linalg.cross(q[:, 1] - q[:, 0],
                                                                                   q[:, 2] - q[:, 0]).norm(dim=1)
    fm = (torch.ones(nf, nf, dtype=torch.float64, device=DEV) + torch.eye(nf, dtype=torch.float64, device=DEV)) / (
        nf * (nf + 1))
    fb = fm * (size * ca[faces].mean(1))[:, None, None]            # c / 2A is constant here
    a.index_put_((faces[:, :, None].expand(-1, nf, nf), faces[:, None, :].expand(-1, nf, nf)), fb.to(dt),
                 accumulate=True)
    lu, piv = torch.linalg.lu_factor(a)
    b = rhs.T.contiguous()
    phi = torch.linalg.lu_solve(lu, piv, b)
    phi = phi + torch.linalg.lu_solve(lu, piv, b - a @ phi)
    return phi.T.contiguous()


def _stack(pm, pk, y, cplx):
    """J rows [Re; Im] x [mua | kappa] (complex) or [mua; kappa] of -PMDF / y; pm, pk: links x columns."""
    pm, pk = pm.div_(-y[:, None]), pk.div_(-y[:, None])
    if not cplx:
        return torch.cat([pm, pk])
    j = torch.empty(2 * pm.shape[0], 2 * pm.shape[1], dtype=torch.float64, device=DEV)
    for c, p in enumerate((pm, pk)):
        j[: len(p), c * p.shape[1]:(c + 1) * p.shape[1]] = p.real
        j[len(p):, c * p.shape[1]:(c + 1) * p.shape[1]] = p.imag if p.is_complex() else 0
    return j


def _nodal(case, f, g, y):
    """Nodal Jacobian: per node its element integrals as a dense block over its neighbours."""
    vol, grad, e, _, x, _ = _elements(case)
    n, (ne, nn) = len(x), e.shape
    pairs = torch.unique((e[:, :, None] * n + e[:, None, :]).reshape(-1))      # sorted (row, column)
    row, col = pairs // n, pairs % n
    first = torch.searchsorted(row, torch.arange(n, device=DEV))
    slot = torch.arange(len(row), device=DEV) - first[row]
    deg = int(slot.max()) + 1
    nbr = torch.zeros(n, deg, dtype=torch.int64, device=DEV)
    nbr[row, slot] = col
    at = slot[torch.searchsorted(pairs, e[:, :, None] * n + e[:, None, :])]    # ne x nn (node) x nn (neighbour)
    fff = _triple(nn)
    stiff = torch.einsum("eid,ejd->eij", grad, grad) * (vol / nn)[:, None, None]
    w = [torch.zeros(n * deg * deg, dtype=torch.float64, device=DEV) for _ in range(2)]
    for i in range(nn):
        idx = (e[:, i, None, None] * deg + at[:, i, :, None]) * deg + at[:, i, None, :]
        w[0].index_put_((idx,), fff[i] * vol[:, None, None], accumulate=True)
        w[1].index_put_((idx,), stiff, accumulate=True)
    nq, nm = len(f), len(g)
    dt = f.dtype
    out = [torch.empty(nq * nm, n, dtype=dt, device=DEV) for _ in range(2)]
    step = max(1, (1 << 28) // (nq * nm))
    for s in range(0, n, step):
        t = min(n, s + step)
        fn, gn = f[:, nbr[s:t]].permute(1, 0, 2), g[:, nbr[s:t]].permute(1, 2, 0)
        for o, ww in zip(out, w):
            h = torch.bmm(ww.view(n, deg, deg)[s:t].to(dt), gn)
            o[:, s:t] = torch.bmm(fn, h).reshape(t - s, nq * nm).T
    return _stack(out[0], out[1], y, bool(case["mhz"]))


def _element(case, f, g, y):
    vol, grad, e, _, _, _ = _elements(case)
    nn = e.shape[1]
    mass = (torch.ones(nn, nn, dtype=torch.float64, device=DEV) + torch.eye(nn, dtype=torch.float64, device=DEV)) / (
        nn * (nn + 1)) * vol[:, None, None]
    stiff = torch.einsum("eid,ejd->eij", grad, grad) * vol[:, None, None]
    fe, ge = f[:, e], g[:, e]                                                   # n? x ne x nn
    out = []
    for w in (mass, stiff):
        h = torch.einsum("eij,mej->mei", w.to(f.dtype), ge)
        out.append(torch.cat([torch.einsum("ei,mei->me", fq, h) for fq in fe]))
    return _stack(out[0], out[1], y, bool(case["mhz"]))


def _raster(case):
    """Element and shape functions at every grid point: inside mask, nodes and weights."""
    _, _, e, bary, x, _ = _elements(case)
    dim, g = x.shape[1], case["g"]
    lo, hi = x.min(0).values, x.max(0).values
    ax = [lo[d] + (hi[d] - lo[d]) / (g - 1) * torch.arange(g, dtype=torch.float64, device=DEV) for d in range(dim)]
    p = torch.stack(torch.meshgrid(*ax[::-1], indexing="ij")[::-1], -1).reshape(-1, dim)   # x fastest
    ph = torch.cat([torch.ones_like(p[:, :1]), p], 1).T.contiguous()
    best = torch.full((len(p),), -1e300, dtype=torch.float64, device=DEV)
    who = torch.zeros(len(p), dtype=torch.int64, device=DEV)
    step = max(1, (1 << 27) // len(p))
    for s in range(0, len(e), step):
        lam = (bary[s:s + step].reshape(-1, dim + 1) @ ph).view(-1, dim + 1, len(p)).amin(1)
        v, i = lam.max(0)
        better = v > best
        best = torch.where(better, v, best)
        who = torch.where(better, i + s, who)
    inside = best >= -1e-8
    w = torch.einsum("pid,dp->pi", bary[who], ph) * inside[:, None]
    return inside, e[who], w, (hi - lo)


def _planes(case, f, masked):
    """Value and difference gradient of the fields at the grid points inside the mesh: (1 + dim) x fields x points."""
    inside, nodes, w, size = _raster(case)
    g, dim = case["g"], len(size)
    v = (f[:, nodes] * w).sum(-1)
    out = [v[:, inside]]
    shape = (len(f),) + (g,) * dim
    vg, ins = v.view(shape), inside.view((g,) * dim)
    for d in range(dim):
        axis = dim - 1 - d                                                      # x is the last axis
        ok = ins if masked else torch.ones_like(ins)
        has_lo, has_hi = torch.zeros_like(ins), torch.zeros_like(ins)
        up, down = [slice(None)] * dim, [slice(None)] * dim
        up[axis], down[axis] = slice(1, None), slice(None, -1)
        has_lo[tuple(up)], has_hi[tuple(down)] = ok[tuple(down)], ok[tuple(up)]
        lo, hi = vg.clone(), vg.clone()
        lo[(slice(None), *up)] = torch.where(has_lo[tuple(up)], vg[(slice(None), *down)], vg[(slice(None), *up)])
        hi[(slice(None), *down)] = torch.where(has_hi[tuple(down)], vg[(slice(None), *up)], vg[(slice(None), *down)])
        ih = g / size[d]
        gr = (hi - lo) * torch.where(has_lo & has_hi, 0.5 * ih, ih)
        out.append(gr.reshape(len(f), -1)[:, inside])
    return torch.stack(out), size


def _grid(case, f, g, y):
    pf, size = _planes(case, f, True)
    pa, _ = _planes(case, g, bool(case["mhz"]))
    vox = float(torch.prod(size / (case["g"] - 1.0)))
    pm = (pf[0][:, None] * pa[0][None]).flatten(0, 1) * vox
    pk = sum((pf[d][:, None] * pa[d][None]).flatten(0, 1) for d in range(1, len(pf))) * vox
    return _stack(pm, pk, y, bool(case["mhz"]))


def exact(case, seed):
    case = {k: v for k, v in case.items() if k != "name"}
    n = len(_geometry(case["mesh"], case["a"], case["b"])[0])
    kind = case["kind"]
    if kind in ("request", "fields", "gradient") and n > 13000:
        return None                                                             # the dense factorisation takes too long
    x = _inputs(case, seed)
    if kind == "fields":
        return _solve(case, x["coef"], x["qvec"])
    if kind in ("jacobian", "element", "grid"):
        return {"jacobian": _nodal, "element": _element, "grid": _grid}[kind](case, x["dphi"], x["aphi"], x["proj"])
    nq, nm = case["nq"], case["nm"]
    if kind == "request":
        phi = _solve(case, x["coef"], torch.cat([x["qvec"], x["mvec"]]))
        dphi, aphi = phi[:nq].contiguous(), phi[nq:].contiguous()
        y = (dphi @ x["mvec"].T).reshape(-1)
        return {"dphi": dphi, "aphi": aphi, "proj": y, "logproj": y.log(), "J": _nodal(case, dphi, aphi, y)}
    phi = _solve(case, x["coef"], x["qvec"])
    y = phi @ x["mvec"].T                                                       # nq x nm
    lg = y.log()
    d, sd = x["data"].view(2, nq, nm), x["sd"].view(2, nq, nm)
    a = -2 * (d[0] - lg.real) / sd[0] ** 2
    b = -2 * (d[1] - lg.imag) / sd[1] ** 2
    inv = 1.0 / (y.real ** 2 + y.imag ** 2)
    c = torch.complex(a * y.real * inv, -a * y.imag * inv) + torch.complex(-b * y.imag * inv, -b * y.real * inv)
    adj = _solve(case, x["coef"], c @ x["mvec"])
    pf, pa = _planes(case, phi, True)[0], _planes(case, adj, True)[0]
    return torch.cat([-(pf[0] * pa[0]).real.sum(0), -(pf[1:] * pa[1:]).sum(0).real.sum(0)])
