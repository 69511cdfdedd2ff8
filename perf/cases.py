"""What a user has this framework do, as cases to be measured.

A case is one call (or the few calls a program makes in a row) through the
public entry points: a steady-state transport solve on a resident context
(Context.solve and the results), the same with the problem handed over anew,
one CSR system through the BiCGSTAB boundary, or one gradient of the
accelerator's network.  Sizes are those of the repository's configurations
(synth.make_problem, the regression cases, bench.py) and what lies between
them; meshes are jittered triangulations of the unit square and Kuhn
subdivisions of the unit cube, made from the seed.
"""
import ctypes
import math

import numpy as np
import torch

import staticbtesolver_gb300 as sbte
from staticbtesolver_gb300 import learned, synth

FORMS = {"plain": sbte.FORM_PLAIN, "mixed": sbte.FORM_MIXED, "sweep": sbte.FORM_SWEEP}


def _solve(name, dim, n, bands, side, walls, form, outer, tol, **kw):
    """A transport solve: n cells per side (2 n^2 triangles or 6 n^3 tetrahedra), `outer` outer
    iterations (the limit where tol is 0, else what the solve typically takes to margin <= tol)."""
    return dict(name=name, kind="solve", dim=dim, n=n, bands=bands, side=side, walls=walls, form=form, outer=outer,
                tol=tol, anderson=0, dsa=False, anew=False, inner=1) | kw


def listed():
    return [
        # the size of the reference's regression cases (gray band, specular walls), default form, to its stop
        _solve("plain_578_gray", 2, 17, 1, 1e-8, 31, "plain", 40, 1e-5, inner=44),
        _solve("plain_cube_750_gray", 3, 5, 1, 1e-8, 33, "plain", 126, 1e-5, inner=25),
        # the default form on the ballistic square with several bands
        _solve("plain_20k_b8", 2, 100, 8, 1e-7, 2, "plain", 2, 0.0, inner=205),
        # mixed precision on an odd mesh size
        _solve("mixed_10k_b8", 2, 71, 8, 1e-7, 2, "mixed", 3, 0.0, inner=216),
        # the sweep form on a small mesh: the latency of an outer iteration
        _solve("sweep_1k_b5", 2, 23, 5, 1e-7, 31, "sweep", 274, 1e-5),
        # the ballistic benchmark: 40 bands, Anderson mixing to the reference's stop
        _solve("sweep_20k_b40_anderson", 2, 100, 40, 1e-7, 2, "sweep", 29, 1e-5, anderson=8),
        # the diffusive benchmark: 20 bands, diffusion-synthetic correction, resident inputs
        _solve("sweep_100k_b20_dsa", 2, 224, 20, 1e-4, 2, "sweep", 9, 1e-5, dsa=True),
        # a new problem each time, end to end: host arrays in, set-up, solve, fields out
        _solve("anew_25k_b20_dsa", 2, 112, 20, 1e-4, 2, "sweep", 9, 1e-5, dsa=True, anew=True),
        # cubes with specular walls: a middling one and the largest
        _solve("sweep_cube_48k_b7", 3, 20, 7, 1e-8, 33, "sweep", 6, 0.0),
        _solve("sweep_cube_132k_b20", 3, 28, 20, 1e-8, 33, "sweep", 4, 0.0),
        # the reference's inner-solver boundary: one upwind system of a 9,800-triangle mesh
        dict(name="csr_10k", kind="csr", n=70, tol=1e-12, inner=180),
        # one full-batch gradient of the accelerator's network at its training batch
        dict(name="mlp_gradient_4k", kind="mlp", rows=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain2", "plain3", "plain", "mixed", "sweep", "anderson", "dsa", "anew", "cube", "cube", "csr",
                       "mlp"])
    case = None
    if kind == "plain2":
        case = _solve("", 2, rng.randint(9, 32), rng.choice([1, 1, 2, 3]), 1e-8, rng.choice([2, 31]), "plain", 40,
                      1e-5, inner=44)
    elif kind == "plain3":
        case = _solve("", 3, rng.randint(3, 7), 1, 1e-8, rng.choice([2, 33]), "plain", 126, 1e-5, inner=25)
    elif kind == "plain":
        case = _solve("", 2, _log(rng, 33, 100), rng.randint(1, 8), 1e-7, rng.choice([2, 31]), "plain", 2, 0.0,
                      inner=100)
    elif kind == "mixed":
        case = _solve("", 2, _log(rng, 17, 80), rng.randint(1, 8), 1e-7, rng.choice([2, 31]), "mixed", 3, 0.0,
                      inner=80)
    elif kind == "sweep":
        case = _solve("", 2, _log(rng, 12, 140), rng.randint(1, 24), 1e-7, rng.choice([2, 31]), "sweep", 20, 0.0)
    elif kind == "anderson":
        case = _solve("", 2, _log(rng, 30, 110), rng.randint(8, 40), 1e-7, 2, "sweep", 34, 1e-5, anderson=8)
    elif kind == "dsa":
        case = _solve("", 2, _log(rng, 60, 224), rng.randint(4, 20), 1e-4, 2, "sweep", 9, 1e-5, dsa=True)
    elif kind == "anew":
        case = _solve("", 2, _log(rng, 40, 130), rng.randint(4, 20), 1e-4, 2, "sweep", 9, 1e-5, dsa=True, anew=True)
    elif kind == "cube":
        case = _solve("", 3, rng.randint(8, 27), rng.randint(3, 20), 1e-8, rng.choice([2, 33]), "sweep", 4, 0.0)
    elif kind == "csr":
        case = dict(kind="csr", n=_log(rng, 12, 150), tol=1e-12, inner=180)
    else:
        case = dict(kind="mlp", rows=_log(rng, 500, 20000))
    case.pop("name", None)
    return case


# ---------------------------------------------------------------------------
# Inputs


def _morton(xyz, bits=12):
    q = (xyz * ((1 << bits) - 1)).astype(np.int64)
    code = np.zeros(len(q), np.int64)
    for b in range(bits):
        for k in range(q.shape[1]):
            code |= ((q[:, k] >> b) & 1) << (q.shape[1] * b + k)
    return np.argsort(code, kind="stable")


def _square(n, rng):
    """Points and triangles of a jittered n x n grid, each quad cut along its Delaunay diagonal."""
    i, j = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
    P = np.stack([i.ravel(), j.ravel()], 1) / n
    J = rng.uniform(-0.2, 0.2, P.shape) / n
    J[(P == 0) | (P == 1)] = 0
    P = P + J
    a = (np.arange(n)[:, None] * (n + 1) + np.arange(n)).ravel()
    b, c, d = a + n + 1, a + n + 2, a + 1
    ang = lambda p, q, r: np.arccos(np.sum((P[q] - P[p]) * (P[r] - P[p]), 1) / np.linalg.norm(P[q] - P[p], axis=1) /
                                    np.linalg.norm(P[r] - P[p], axis=1))
    ac = (ang(b, a, c) + ang(d, c, a) <= math.pi)[:, None]  # the diagonal a-c is locally Delaunay
    T = np.concatenate([np.where(ac, np.stack([a, b, c], 1), np.stack([a, b, d], 1)),
                        np.where(ac, np.stack([a, c, d], 1), np.stack([b, c, d], 1))])
    return P, T


def _cube(n, rng):
    """Points and tetrahedra of a jittered n^3 lattice, six Kuhn tetrahedra per cube."""
    g = np.stack(np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
    P = g / n
    J = rng.uniform(-0.1, 0.1, P.shape) / n
    J[(P == 0) | (P == 1)] = 0
    o = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    at = lambda v: (v[:, 0] * (n + 1) + v[:, 1]) * (n + 1) + v[:, 2]
    T = []
    for perm in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        v = o.copy()
        tet = [at(v)]
        for k in perm:
            v[:, k] += 1
            tet.append(at(v))
        T.append(np.stack(tet, 1))
    return P + J, np.concatenate(T)


def _quadrature(dim):
    """The direction sets of the configurations: 32 azimuths in 2D (DM 2), 8 x 16 angles in 3D (DM 3)."""
    if dim == 2:
        nt = nphi = 8
        phi = (np.arange(4 * nphi) + 0.5) * 0.5 * math.pi / nphi
        s = np.stack([np.sin(phi), np.cos(phi), 0 * phi], 1)
        w = np.full(len(phi), 4 * math.pi / len(phi))
        return dict(DM=2, num_theta=nt, num_phi=nphi, s=s, S=s * w[:, None], omega=w)
    nt = nphi = 4
    dth, dphi = 0.5 * math.pi / nt, 0.5 * math.pi / nphi
    th, phi = np.meshgrid((np.arange(2 * nt) + 0.5) * dth, (np.arange(4 * nphi) + 0.5) * dphi, indexing="ij")
    th, phi = th.ravel(), phi.ravel()
    s = np.stack([np.sin(th) * np.sin(phi), np.sin(th) * np.cos(phi), np.cos(th)], 1)
    lat = math.sin(0.5 * dphi) * (dth - np.cos(2 * th) * math.sin(dth))
    S = np.stack([np.sin(phi) * lat, np.cos(phi) * lat, 0.5 * dphi * np.sin(2 * th) * math.sin(dth)], 1)
    return dict(DM=3, num_theta=nt, num_phi=nphi, s=s, S=S, omega=2 * np.sin(th) * math.sin(0.5 * dth) * dphi)


def _problem(case, seed):
    """Host arrays of a transport problem, as Context.set_arrays takes them."""
    rng = np.random.default_rng(seed)
    dim, n, side = case["dim"], case["n"], case["side"]
    P, T = (_square if dim == 2 else _cube)(n, rng)
    T = T[_morton(P[T].mean(1))]
    X = P[T] * side  # [cell][vertex][xyz]
    cells, F = T.shape
    area, normal, key = np.zeros((cells, F)), np.zeros((cells, F, 3)), np.zeros((cells, F), np.int64)
    code = np.zeros((cells, F), np.int64)
    walls = [(k, hi) for k in range(dim) for hi in (0, 1)]  # entity 2k: coordinate k = 0, 2k + 1: = 1
    for f in range(F):
        face = [v for v in range(F) if v != f]
        q = [X[:, v] for v in face]
        if dim == 2:
            e = q[1] - q[0]
            nv = np.stack([e[:, 1], -e[:, 0], 0 * e[:, 0]], 1)
            area[:, f] = np.linalg.norm(nv, axis=1)
        else:
            nv = np.cross(q[1] - q[0], q[2] - q[0])
            area[:, f] = 0.5 * np.linalg.norm(nv, axis=1)
        nv /= np.linalg.norm(nv, axis=1)[:, None]
        back = np.sum(nv[:, :dim] * (X[:, f] - q[0]), 1) > 0
        normal[:, f] = np.where(back[:, None], -nv, nv)
        v = np.sort(T[:, face], 1)
        for k in range(dim):
            key[:, f] = key[:, f] * len(P) + v[:, k]
        for w, (k, hi) in enumerate(walls):
            code[(P[T[:, face], k] == hi).all(1), f] = -w - 1
    order = np.argsort(key.ravel(), kind="stable")
    ks = key.ravel()[order]
    twin = np.flatnonzero(ks[1:] == ks[:-1])
    nbr = code.ravel()
    nbr[order[twin]], nbr[order[twin + 1]] = order[twin + 1] // F, order[twin] // F
    E = X[:, 1:] - X[:, :1]
    volume = np.abs(np.linalg.det(E)) / (2 if dim == 2 else 6)
    centroid = np.zeros((cells, 3))
    centroid[:, :dim] = X.mean(1)
    hot = rng.uniform(300.5, 302.0)
    # x walls isothermal; the others diffuse, or the specular type that mirrors their axis
    y, z = (2, 2) if case["walls"] == 2 else (31, None) if dim == 2 else (32, 33)
    types = [1, 1, y, y] + ([z, z] if dim == 3 else [])
    bands = synth.debye_bands(case["bands"]) if case["bands"] > 1 else dict(
        vg=np.array([6400.0]), tau=np.array([4e-11]), C=np.array([synth.C_TOTAL]), Lr=np.array([1.0]))
    return dict(dim=dim, n_cell=cells, n_face=F, nbr=nbr.reshape(cells, F).astype(np.int32), area=area, normal=normal,
                volume=volume, centroid=centroid, n_dir=32 if dim == 2 else 128, solid_angle=4 * math.pi, T_ref=300.0,
                bands=bands,
                bcs=dict(index=-np.arange(len(types), dtype=np.int32) - 1, type=np.array(types, np.int32),
                         T=np.array([hot, 600.0 - hot] + [300.0] * (len(types) - 2))), **_quadrature(dim))


def _upwind_csr(case, seed):
    """One (band, direction) system of a square mesh in CSR form, and a right-hand side."""
    rng = np.random.default_rng(seed + 1)
    a = _problem(dict(dim=2, n=case["n"], side=1e-7, walls=2, bands=1), seed)
    d = int(rng.integers(a["n_dir"]))
    g = a["area"] * (a["normal"] @ a["S"][d])
    k = float(a["bands"]["vg"][0] * 4e-11)
    inflow = (g < 0) & (a["nbr"] >= 0)
    diag = k * np.where(g > 0, g, 0).sum(1) + a["volume"] * a["omega"][d]
    rows = np.concatenate([np.arange(len(diag)), np.nonzero(inflow)[0]])
    cols = np.concatenate([np.arange(len(diag)), a["nbr"][inflow]])
    vals = np.concatenate([diag, k * g[inflow]]) / diag.mean()
    o = np.lexsort((cols, rows))
    ptr = np.searchsorted(rows[o], np.arange(len(diag) + 1)).astype(np.int32)
    return ptr, cols[o].astype(np.int32), vals[o], rng.uniform(0.0, 1.0, len(diag))


def _mlp_data(case, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(0, 1, (case["rows"], 8)).astype(np.float32)
    X[:, :3] /= np.abs(X[:, :3]).sum(1, keepdims=True)
    X[:, 3:6] = rng.uniform(0, 1, (case["rows"], 3))
    Y = (2 * X[:, 0] - X[:, 1] + 0.5 * np.tanh(X[:, 6])).astype(np.float32)
    return X, Y, learned.init_params(seed % 1000)


def prepare(case, seed):
    if case["kind"] == "csr":
        return dict(case=case, system=_upwind_csr(case, seed))
    if case["kind"] == "mlp":
        return dict(case=case, data=_mlp_data(case, seed))
    a = _problem(case, seed)
    ctx = sbte.Context(0)
    if not case["anew"]:
        ctx.set_arrays(a)
    opt = dict(max_iter=case["outer"] if case["tol"] == 0 else 1000, tol=case["tol"], form=FORMS[case["form"]])
    if case["anderson"]:
        opt |= dict(accel=3, accel_every=case["anderson"])
    if case["dsa"]:
        opt |= dict(dsa=True)
    return dict(case=case, ctx=ctx, arrays=a if case["anew"] else None, opt=opt)


def run(state):
    case = state["case"]
    if case["kind"] == "csr":
        x, _, _ = sbte.bicgstab_csr(*state["system"], maxit=2000, tol=case["tol"])
        return x
    if case["kind"] == "mlp":
        X, Y, p = state["data"]
        L, _ = sbte._load()
        grad, loss = np.zeros(learned.NPARAM, np.float32), ctypes.c_double(0)
        ptr = lambda v: v.ctypes.data_as(ctypes.c_void_p)
        st = L.bte_mlp_gradient(ptr(X), ptr(Y), len(Y), ptr(p), ptr(grad), ctypes.byref(loss))
        if st != 0:
            raise sbte.BteError(st)
        return dict(grad=grad, loss=np.float32(loss.value))
    ctx = state["ctx"]
    if state["arrays"] is not None:
        ctx.set_arrays(state["arrays"])
    ctx.solve(**state["opt"])
    return dict(T=ctx.temperature(), q=ctx.heat_flux()[0])


def work(case):
    """Bytes and operations of one pass.  Transport: per outer iteration every intensity read and written
    once, the mesh once per direction; the Krylov forms per BiCGSTAB iteration (`inner` of them typically)
    ten vector reads and writes (the update of x, r, p and the two products) in the form's precision."""
    if case["kind"] == "mlp":
        weights = 8 * 128 + 2 * 128 * 128 + 128
        return dict(bytes=case["rows"] * 36 + 8 * learned.NPARAM, flops=6.0 * weights * case["rows"])
    if case["kind"] == "csr":
        n = 2 * case["n"] ** 2
        return dict(bytes=n * (8 + 8 + 2.5 * 12 + case["inner"] * 10 * 8.0), flops=n * case["inner"] * 24.0)
    dim, n = case["dim"], case["n"]
    cells, dirs, faces = (2 * n ** 2, 32, 3) if dim == 2 else (6 * n ** 3, 128, 4)
    values = float(cells) * dirs * case["bands"]
    mesh = float(cells) * dirs * (8 * (faces + 2))
    if case["form"] == "sweep":
        return dict(bytes=case["outer"] * (16 * values + mesh), flops=case["outer"] * values * (faces + 8))
    word = 4 if case["form"] == "mixed" else 8
    return dict(bytes=case["outer"] * (16 * values + case["inner"] * 10 * word * values),
                flops=case["outer"] * case["inner"] * values * (2 * faces + 18))


# ---------------------------------------------------------------------------
# The same in 64 bits, with torch and numpy alone


def _waves(nbr, fc):
    """Kahn's waves of all directions' upwind graphs at once: flat (direction, cell) indices."""
    D, n, F = fc.shape
    into = (fc != 0) & (nbr >= 0)[None]
    left = into.sum(2).reshape(-1)
    twin = torch.zeros_like(nbr)
    for f in range(F):
        for g in range(F):
            ok = (nbr[:, f] >= 0) & (nbr[nbr[:, f].clamp(min=0), g] == torch.arange(n, device=nbr.device))
            twin[ok, f] = g
    free = torch.nonzero(left == 0).flatten()
    waves = []
    while len(free):
        waves.append(free)
        d, c = free // n, free % n
        o = nbr[c]  # [m][F]
        oc = o.clamp(min=0)
        hit = (o >= 0) & into[d[:, None], oc, twin[c]]
        t = (d[:, None] * n + oc)[hit]
        left.index_add_(0, t, torch.full_like(t, -1))
        free = torch.unique(t[left[t] == 0])
    return waves


def _exact_solve(case, seed):
    dim, n = case["dim"], case["n"]
    values = (2 * n ** 2 * 32 if dim == 2 else 6 * n ** 3 * 128) * case["bands"]
    if case["anderson"] or case["dsa"] or values > 3e8:
        return None  # (the accelerated iterations' limits take minutes this way)
    a = _problem(case, seed)
    dev = torch.device("cuda")
    f64 = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=dev)
    nbr = torch.as_tensor(a["nbr"], device=dev).long()
    cells, F = nbr.shape
    s, S, om = f64(a["s"]), f64(a["S"]), f64(a["omega"])
    nrm, area, vol = f64(a["normal"]), f64(a["area"]), f64(a["volume"])
    b = {k: f64(v) for k, v in a["bands"].items()}
    kb, NB, D = b["vg"] * b["tau"], len(b["vg"]), len(om)
    sn = torch.einsum("dx,cfx->dcf", s, nrm)
    ag = torch.einsum("dx,cfx->dcf", S, nrm) * area
    dg = torch.where(sn >= 0, ag, 0 * ag).sum(2)
    fc = torch.where((sn < 0) & (nbr >= 0), ag, 0 * ag)
    vo = vol[None] * om[:, None]
    diag = (kb[:, None, None] * dg + vo).reshape(NB, -1)
    waves = _waves(nbr, fc)
    up = (torch.arange(D, device=dev)[:, None, None] * cells + nbr.clamp(min=0)).reshape(-1, F)
    fcf = fc.reshape(-1, F)
    plan = [(w, up[w], fcf[w], diag[:, w]) for w in waves]
    # boundary faces by wall, the directions that enter there
    types, temps, Omega, Tr = a["bcs"]["type"], a["bcs"]["T"], a["solid_angle"], a["T_ref"]
    faces = []
    for w, t in enumerate(types):
        c, f = torch.nonzero(nbr == -w - 1, as_tuple=True)
        mirror = None
        if t in (31, 32, 33):
            axis = int(np.flatnonzero(np.abs(a["normal"][int(c[0]), int(f[0])]) > 0.5)[0])
            r = s.clone()
            r[:, axis] *= -1
            mirror = torch.cdist(s, r).argmin(0)
        faces.append((int(t), float(temps[w]), c, f, mirror))
    e = torch.zeros(NB, D, cells, dtype=torch.float64, device=dev)
    T = torch.full((cells,), Tr, dtype=torch.float64, device=dev)
    limit = case["outer"] if case["tol"] == 0 else 1000
    for _ in range(limit):
        R = (b["C"] / Omega)[:, None, None] * (T - Tr) * vo
        for t, temp, c, f, mirror in faces:
            out, g = sn[:, c, f], ag[:, c, f]
            if t == 1:
                wall = ((b["C"] / Omega) * (temp - Tr))[:, None, None].expand(NB, D, len(c))
            elif t == 2:
                Sn = torch.einsum("dx,mx->dm", S, nrm[c, f]) * (om[:, None] if dim == 3 else 1.0)
                Sn = torch.where(out > 0, Sn, 0 * Sn)
                wall = ((e[:, :, c] * Sn).sum(1) / Sn.sum(0))[:, None].expand(NB, D, len(c))
            else:
                wall = e[:, mirror][:, :, c]
            add = torch.where(out < 0, -wall * kb[:, None, None] * g, 0 * wall)
            R.view(NB * D, cells).index_add_(1, c, add.reshape(NB * D, len(c)))
        R = R.reshape(NB, -1)
        x = torch.zeros(NB, D * cells, dtype=torch.float64, device=dev)
        for w, u, q, dd in plan:
            x[:, w] = (R[:, w] - kb[:, None] * (x[:, u] * q).sum(2)) / dd
        x = x.reshape(NB, D, cells)
        margin = float(((x - e) ** 2).sum() / (NB * cells))
        e = x
        Tb = (e * om[:, None]).sum(1) / b["C"][:, None] + Tr
        T = (b["Lr"][:, None] * Tb).sum(0) / b["Lr"].sum()
        if margin <= case["tol"]:
            break
    q = []
    for t, temp, c, f, _ in faces:
        hw = sn[:, c, f] * area[c, f] * om[:, None] if dim == 3 else ag[:, c, f]
        q.append((((e[:, :, c] * hw).sum((1, 2)) / area[c, f].sum()) * b["vg"]).sum())
    return dict(T=T, q=torch.stack(q))


def _exact_csr(case, seed):
    """Forward substitution in an order in which every row follows the rows it couples to."""
    ptr, col, val, rhs = _upwind_csr(case, seed)
    n = len(rhs)
    rows = np.repeat(np.arange(n), np.diff(ptr))
    off = rows != col
    left = np.bincount(rows[off], minlength=n)
    diag, x = np.zeros(n), np.zeros(n)
    diag[rows[~off]] = val[~off]
    r_off, c_off, v_off = rows[off], col[off], val[off]
    by_col = np.argsort(c_off, kind="stable")
    start = np.searchsorted(c_off[by_col], np.arange(n + 1))
    acc = rhs.astype(np.longdouble)
    free = list(np.flatnonzero(left == 0))
    while free:
        c = free.pop()
        x[c] = acc[c] / diag[c]
        for k in by_col[start[c]:start[c + 1]]:
            r = r_off[k]
            acc[r] -= np.longdouble(v_off[k]) * x[c]
            left[r] -= 1
            if left[r] == 0:
                free.append(r)
    return x


def _exact_mlp(case, seed):
    X, Y, p = _mlp_data(case, seed)
    p = torch.tensor(p, dtype=torch.float64, requires_grad=True)
    h, o = torch.as_tensor(X, dtype=torch.float64), 0
    for fan_in, fan_out in ((8, 128), (128, 128), (128, 128), (128, 1)):
        h = h @ p[o:o + fan_in * fan_out].view(fan_in, fan_out) + p[o + fan_in * fan_out:][:fan_out]
        o += fan_in * fan_out + fan_out
        if fan_out > 1:
            h = torch.relu(h)
    loss = 0.5 * ((h[:, 0] - torch.as_tensor(Y, dtype=torch.float64)) ** 2).mean()
    loss.backward()
    return dict(grad=p.grad, loss=loss.detach())


def exact(case, seed):
    return {"csr": _exact_csr, "mlp": _exact_mlp, "solve": _exact_solve}[case["kind"]](case, seed)
