"""The work that a user of the framework has it do, as timed cases.

Every case goes through the host mirror of the reference's API (``solve``,
``solve_batch``, ``calcfield_*``, ``Uind``, the autograd functions) with host
arrays in and host arrays out, as a user's program calls it: meshing is the
program's own preparation; normals, control points, the upload of the geometry,
assembly, factorisation, solve and download are part of a pass.

``exact`` restates the panel method in plain torch, in 64 bits: the influence
of a vortex ring, of a semi-infinite wake filament and of a constant source,
dense solves by ``torch.linalg``, the Kutta averages and the forces.
"""
import math

import numpy as np
import torch

import __graft_entry__

fp = __graft_entry__.load_package()

OFFSET, CUTOFF2 = 1e-8, 1e-28   # the bodies' default kerneloffset and kernelcutoff ** 2


def listed():
    return [
        # A first wing: the coarse mesh of the tests and the tutorials, default FP64 solver. Latency and host work count.
        {"name": "wing_fp64_480", "kind": "wing", "nc": 20, "ns": 24, "method": "ludiv", "precision": "fp64"},
        # The non-lifting body of the reference's sphere example: constant sources, FP64.
        {"name": "sphere_fp64_1800", "kind": "sphere", "nt": 30, "np": 60},
        # The iterative solver (the reference's Krylov option), to a residual near the one that the direct forms refine to.
        {"name": "wing_gmres_3828", "kind": "wing", "nc": 58, "ns": 66, "method": "gmres", "precision": "fp64"},
        # The headline wing, mixed precision: FP32 factors refined in FP64.
        {"name": "wing_mixed_12000", "kind": "wing", "nc": 100, "ns": 120, "method": "ludiv", "precision": "mixed"},
        # The same wing with the default solver, plain FP64.
        {"name": "wing_fp64_12000", "kind": "wing", "nc": 100, "ns": 120, "method": "ludiv", "precision": "fp64"},
        # The largest body: fuselage and wing, 36,600 panels (triangles and quadrilaterals mixed).
        {"name": "wingbody_mixed_36600", "kind": "wingbody", "fx": 120, "ft": 80, "wc": 150, "ws": 180, "precision": "mixed"},
        # A polar: 21 angles of attack on one factorisation.
        {"name": "polar_mixed_12000x21", "kind": "polar", "nc": 100, "ns": 120, "precision": "mixed", "k": 21},
        # A design step: forward solve and the gradients by vertex, freestream and wake direction; a ragged size, FP64.
        {"name": "gradient_fp64_6300", "kind": "gradient", "nc": 70, "ns": 90, "precision": "fp64"},
        # Post-processing of a solved body on triangles: surface velocity off the surface, Cp, forces, lift and drag.
        {"name": "loads_12000", "kind": "loads", "nc": 100, "ns": 60},
        # Off-body field of the wing-body at probes, single precision (kept in single, as a field file holds it).
        {"name": "probes_fp32_36600x100000", "kind": "probes", "fx": 120, "ft": 80, "wc": 150, "ws": 180, "m": 100000},
        # A design study: wings of uneven sizes (2,000 to 8,000 panels) solved together, mixed precision.
        {"name": "batch_mixed_16", "kind": "batch", "count": 16, "wings": 0, "pmin": 2000, "pmax": 8000},
        # A watertight body: the duct of the reference's tests, least squares, FP64.
        {"name": "duct_ls_7200", "kind": "duct", "nq": 60, "nt": 60},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """A case of the same kinds: sizes over the whole of each range, ragged ones among them."""
    kind = rng.choice(["wing", "wing", "wing", "wing", "sphere", "wingbody", "polar", "gradient", "loads", "probes", "batch", "duct"])
    if kind in ("wing", "polar", "gradient"):
        n = _log(rng, *{"wing": (200, 12000), "polar": (1000, 12000), "gradient": (300, 6300)}[kind])
        nc = 2 * max(5, round(math.sqrt(n / rng.uniform(0.6, 1.6)) / 2))
        ns = 2 * max(4, int(n / nc / 2))
        case = {"kind": kind, "nc": nc, "ns": ns, "precision": rng.choice(["fp64", "mixed"])}
        if kind == "wing":
            case["method"] = rng.choice(["ludiv", "ludiv", "gmres"]) if 800 < n < 4000 else "ludiv"
            if case["method"] == "gmres":
                case["precision"] = "fp64"
        if kind == "polar":
            case["k"] = rng.randint(3, 21)
        return case
    if kind == "sphere":
        nt = round(_log(rng, 10, 45))
        return {"kind": kind, "nt": nt, "np": 2 * nt + rng.choice([-5, -3, -1, 1, 3, 5, 7, 9])}
    if kind in ("wingbody", "probes"):
        s = _log(rng, 0.25, 0.85)
        case = {"kind": kind, "fx": round(120 * s), "ft": round(80 * s), "wc": 2 * round(75 * s), "ws": 2 * round(90 * s)}
        return {**case, "precision": "mixed"} if kind == "wingbody" else {**case, "m": round(_log(rng, 1000, 100000))}
    if kind == "loads":
        nc = 2 * rng.randint(8, 50)
        return {"kind": kind, "nc": nc, "ns": 2 * rng.randint(4, 30)}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 16), "wings": rng.randint(1, 1000), "pmin": 2000, "pmax": rng.randint(4000, 8000)}
    return {"kind": "duct", "nq": 2 * rng.randint(8, 30), "nt": rng.randint(12, 60)}


# ----------------------------------------------------------------------------- problems
def _problem(case, seed):
    """The mesh and the host arrays of a case: what a program has before it calls the framework."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    aoa = np.deg2rad(rng.uniform(2.0, 6.0))
    p = {"V": np.array([np.cos(aoa), 0.0, np.sin(aoa)])}
    if kind in ("wing", "polar", "gradient", "loads"):
        m = fp.meshes.swept_wing("0012", case["nc"], case["ns"], 1.0, rng.uniform(4.5, 5.5), rng.uniform(40.0, 45.0),
                                 rng.uniform(0.8, 1.0), 0.0, rng.uniform(-2.0, 0.0))
        p["mesh"] = fp.meshes.triangulate(m) if kind == "loads" else m
    elif kind in ("wingbody", "probes"):
        p["mesh"] = fp.meshes.wing_body(case["fx"], case["ft"], case["wc"], case["ws"], sweep=rng.uniform(38.0, 42.0))
    elif kind == "sphere":
        p["mesh"] = fp.meshes.sphere(rng.uniform(0.8, 1.2), case["nt"], case["np"])
        p["V"] = np.array([1.0, 0.0, 0.0])
    elif kind == "duct":
        chord, d = 1.002, 1.67
        profile = fp.meshes.naca4_contour("0015", case["nq"] // 2) * chord * rng.uniform(0.95, 1.05)
        profile[:, 1] += d / 2
        p["mesh"] = fp.meshes.revolution_liftbody(profile, case["nt"], name="duct", CPoffset=1e-14)
    if kind == "batch":
        p["meshes"] = fp.meshes.random_wings(case["count"], case["wings"], case["pmin"], case["pmax"])[0]
        for m in p["meshes"]:   # the same planforms, stretched
            m.nodes = m.nodes * np.array([1.0, rng.uniform(0.9, 1.1), rng.uniform(0.95, 1.05)])
        return p
    m = p["mesh"]
    p["U"] = np.tile(p["V"], (m.npanels, 1))
    p["D"] = np.tile(p["V"], (m.nsheddings, 1))
    if kind == "polar":
        a = np.deg2rad(np.linspace(-10.0, 10.0, case["k"]))
        w = np.stack([np.cos(a), np.zeros_like(a), np.sin(a)], axis=1)
        p["U"] = np.repeat(w[:, None, :], m.npanels, axis=1)
    if kind == "gradient":
        p["w"] = rng.standard_normal(m.npanels)
    if kind == "probes":
        p["X"] = fp.meshes.probe_box(m, case["m"], seed=seed)
    return p


def prepare(case, seed):
    s = _problem(case, seed)
    kind = case["kind"]
    s["kind"] = kind
    if kind == "batch":
        s["bodies"] = [fp.RigidWakeBody(m) for m in s["meshes"]]
        s["Us"] = [np.tile(s["V"], (m.npanels, 1)) for m in s["meshes"]]
        s["Ds"] = [np.tile(s["V"], (m.nsheddings, 1)) for m in s["meshes"]]
        s["batch"] = fp._capi.Batch(0, 8)
        return s
    if kind == "sphere":
        s["body"] = fp.NonLiftingBody(s["mesh"])
    else:
        s["body"] = fp.RigidWakeBody(s["mesh"], watertight=kind == "duct")
    if case.get("method") == "gmres":
        s["solver"] = fp.B200Solver("gmres", atol=1e-11, rtol=1e-11)
    else:
        s["solver"] = fp.B200Solver("ludiv", case.get("precision", "mixed" if kind in ("loads", "probes") else "fp64"))
    if kind == "gradient":
        s["geom"] = fp.adjoint._Geom(s["mesh"])
        for k in ("U", "D", "w"):
            s[k] = torch.from_numpy(s[k])
        s["nodes"] = torch.from_numpy(s["mesh"].nodes.copy())
    if kind in ("loads", "probes"):   # the field is taken of a solved body
        fp.solve(s["body"], s["U"], s["D"], s["D"], solver=s["solver"])
        s["L"] = np.cross(s["V"], [0.0, 1.0, 0.0])
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        fp.solve_batch(s["bodies"], s["Us"], s["Ds"], s["Ds"], precision="mixed", batch=s["batch"])
        return [b.strength for b in s["bodies"]]
    body, solver = s["body"], s["solver"]
    if kind == "sphere":
        return fp.solve(body, s["U"], solver=solver).strength
    if kind == "polar":
        solver.load(body)
        solver.ctx.set_wake(s["mesh"].shedding, s["D"], s["D"])
        return solver.ctx.solve_body(body.element, s["U"], opts=solver.opts)[0]
    if kind == "gradient":
        nodes, U, D = (s[k].clone().requires_grad_() for k in ("nodes", "U", "D"))
        normals, cps, _, _ = fp.adjoint.geometry(s["geom"], nodes)
        gamma = fp.adjoint.PanelSolve.apply(solver, s["geom"], nodes, cps, normals, U, D, D, 1e-8, 1e-14)
        return {"gamma": gamma.detach(), "grads": torch.autograd.grad(gamma, (nodes, U, D), s["w"])}
    if kind == "loads":
        fp.calcfield_U(body, body, offset=0.02, solver=solver)
        fp.calcfield_Cp(body, 1.0, solver=solver)
        fp.calcfield_F(body, 1.0, 1.225, solver=solver)
        lds = fp.calcfield_LDS(body, s["L"], s["V"], np.array([0.0, 1.0, 0.0]), solver=solver)
        return {"lds": lds, **{k: np.asarray(body.get_field(k)["field_data"]) for k in ("U", "Cp", "F")}}
    if kind == "probes":
        out = fp.Uind(body, s["X"], np.tile(s["V"], (len(s["X"]), 1)), solver, precision="fp32")
        return out.astype(np.float32)
    return fp.solve(body, s["U"], s["D"], s["D"], solver=solver).strength   # wing, wingbody, duct


# ----------------------------------------------------------------------------- work
def _sizes(case):
    """(panels, edges of a panel, shedding edges) of a case's mesh."""
    kind = case["kind"]
    if kind == "sphere":
        return case["nt"] * case["np"], 4, 0
    if kind in ("wingbody", "probes"):
        return case["fx"] * case["ft"] + case["wc"] * case["ws"], 4, case["ws"]
    if kind == "duct":
        return 2 * case["nq"] * case["nt"], 3, case["nt"]
    return case["nc"] * case["ns"] * (2 if kind == "loads" else 1), 3 if kind == "loads" else 4, case["ns"]


def work(case):
    """Arithmetic of the influence coefficients (62 operations an edge, 290 a horseshoe, 534 a source panel), of the
    factorisation, the solves and the reverse pass; the bytes are those of the host's arrays and the matrix, once."""
    kind = case["kind"]
    if kind == "batch":
        n = 0.5 * (case["pmin"] + case["pmax"])
        one = work({"kind": "wing", "nc": round(math.sqrt(n)), "ns": round(math.sqrt(n)), "method": "ludiv"})
        return {k: v * case["count"] for k, v in one.items()}
    n, edges, nsh = _sizes(case)
    pair = 534 if kind == "sphere" else 62 * edges
    if kind in ("loads", "probes"):
        m = case.get("m", n)
        return {"bytes": 128 * n + 48 * m, "flops": m * (n * pair + 580 * nsh)}
    flops = n * (n * pair + 580 * nsh)
    if case.get("method") == "gmres":
        flops += 2.0 * n * n * 250   # about the steps it takes
    else:
        flops += 2.0 * n ** 3 / 3 + 2.0 * n * n * case.get("k", 1)
    if kind == "duct":
        flops += n ** 3
    if kind == "gradient":
        flops += 2 * n * n + 3 * n * (n * pair + 580 * nsh)
    return {"bytes": 16 * n * n + 200 * n * case.get("k", 1), "flops": flops}


# ----------------------------------------------------------------------------- in 64 bits
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_device())


def _corners(m):
    """Node indices (N, 4) of the panels, a triangle's first node again as its fourth, and the nodes of each."""
    nn = np.diff(m.panel_offsets)
    first = m.panel_offsets[:-1]
    idx = np.stack([m.panel_nodes[first + np.where(nn > k, k, 0)] for k in range(4)], axis=1).astype(np.int64)
    return _t(idx), _t(nn.astype(np.int64))


def _geometry(nodes, idx, nn, off=1e-14):
    """Normals, control points (vertex mean with the in-plane centroid step, off the surface) and areas."""
    P = nodes[idx]
    t = P[:, 1] - P[:, 0]
    t = t / t.norm(dim=1, keepdim=True)
    c = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    n = c / c.norm(dim=1, keepdim=True)
    o = torch.linalg.cross(n, t)
    use = (torch.arange(4, device=P.device)[None] < nn[:, None]).to(P.dtype)[:, :, None]
    mean = (P * use).sum(1) / nn[:, None]
    d = (P - mean[:, None]) * use
    x, y = (d * t[:, None]).sum(2).sum(1) / nn, (d * o[:, None]).sum(2).sum(1) / nn
    area = 0.5 * c.norm(dim=1)
    quad = nn == 4
    more = torch.linalg.cross(P[:, 2] - P[:, 0], P[:, 3] - P[:, 0])[quad]
    area = area.index_add(0, torch.nonzero(quad)[:, 0], 0.5 * more.norm(dim=1)) if bool(quad.any()) else area
    return n, mean + x[:, None] * t + y[:, None] * o + off * n, area


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])


def _col(a):
    return tuple(a[:, i][:, None] for i in range(3))


def _row(a):
    return tuple(a[:, i][None, :] for i in range(3))


def _sub(a, b):
    return tuple(x - y for x, y in zip(a, b))


def _add(u, s, c):
    return tuple(x + s * y for x, y in zip(u, c))


def _bound(u, X, a, b):
    """u + the velocity at X of unit filaments a -> b (Biot-Savart with the core offset and the cutoff)."""
    ra, rb, e = _sub(X, a), _sub(X, b), _sub(b, a)
    ia, ib = ((_dot(r, r).clamp_min(1e-300).sqrt() + OFFSET).reciprocal() for r in (ra, rb))
    c = _cross(ra, rb)
    cc = _dot(c, c)
    f = (_dot(e, ra) * ia - _dot(e, rb) * ib) / (4 * math.pi * (cc + OFFSET ** 2))
    return _add(u, torch.where(cc > CUTOFF2, f, torch.zeros_like(f)), c)


def _semi(u, X, p, d, sign):
    """u + sign times the velocity at X of unit semi-infinite filaments from p along d."""
    r = _sub(X, p)
    s = _dot(r, d)
    foot = tuple(x + s * y for x, y in zip(p, d))
    zero = tuple(torch.zeros_like(s) for _ in range(3))
    near = _bound(zero, X, p, foot)
    h = _sub(X, foot)
    hh = _dot(h, h)
    f = torch.where(hh > CUTOFF2, 1 / (4 * math.pi * (hh + OFFSET ** 2)), torch.zeros_like(hh))
    return tuple(x + sign * (torch.where(s * s > OFFSET ** 2, y, torch.zeros_like(y)) + f * z)
                 for x, y, z in zip(u, near, _cross(d, h)))


class _Wake:
    """The shedding rows: upper and lower panels and the nodes of their trailing edges."""

    def __init__(self, m, idx):
        sh = _t(m.shedding.astype(np.int64)).reshape(-1, 6)
        self.sides = [(sh[:, 0], idx[sh[:, 0], sh[:, 1]], idx[sh[:, 0], sh[:, 2]], False),
                      (sh[:, 3], idx[sh[:, 3], sh[:, 4]], idx[sh[:, 3], sh[:, 5]], True)]   # every row has a lower panel here

    def add(self, X, nodes, D, use):
        """use(panels, velocity) for both sides; the lower one has the directions in turn (one direction here)."""
        for panels, a, b, _ in self.sides:
            pa, pb, d = _row(nodes[a]), _row(nodes[b]), _row(D)
            zero = tuple(torch.zeros_like(x - y) for x, y in zip(X, pa))
            use(panels, _semi(_bound(_semi(zero, X, pa, d, -1.0), X, pa, pb), X, pb, d, 1.0))


def _rings(X, nodes, idx):
    P = [_row(nodes[idx[:, k]]) for k in range(4)]
    u = tuple(torch.zeros_like(x - y) for x, y in zip(X, P[0]))
    for k in range(4):
        u = _bound(u, X, P[k], P[(k + 1) % 4])
    return u


def _sources(X, nodes, idx, nn):
    """Velocity at X of unit constant-source panels (Hess and Smith), the panel's frame with its normal turned."""
    P = nodes[idx]
    t = P[:, 1] - P[:, 0]
    t = t / t.norm(dim=1, keepdim=True)
    c = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
    n = c / c.norm(dim=1, keepdim=True)
    ax = (torch.linalg.cross(n, t), t, -n)
    r = _sub(X, _row(P[:, 0]))
    x, y, z = (_dot(r, _row(a)) for a in ax)
    V1, V2, V3 = (torch.zeros_like(x) for _ in range(3))
    inside, zeros = torch.ones_like(x), torch.zeros_like(x)
    for i in range(4):
        for count in (3, 4):
            on = (nn == count) & (i < count)
            if not bool(on.any()):
                continue
            k, j = torch.nonzero(on)[:, 0], (i + 1) % count
            (xi, yi, zi), (xj, yj, zj) = (tuple((a[k] * (P[k, q] - P[k, 0])).sum(1)[None] for a in ax) for q in (i, j))
            X_, Y_, Z_ = x[:, k], y[:, k], z[:, k]
            d = ((xj - xi) ** 2 + (yj - yi) ** 2 + (zj - zi) ** 2).sqrt()
            S, C = (yj - yi) / d, (xj - xi) / d
            ri, rj = (((X_ - a) ** 2 + (Y_ - b) ** 2 + (Z_ - e) ** 2).sqrt() for a, b, e in ((xi, yi, zi), (xj, yj, zj)))
            Q = ((ri + rj + d) / (ri + rj - d + OFFSET)).log()
            si, sj = (xi - X_) * C + (yi - Y_) * S, (xj - X_) * C + (yj - Y_) * S
            R = (X_ - xi) * S - (Y_ - yi) * C
            J = torch.atan2(R * Z_.abs() * (ri * sj - rj * si), ri * rj * R * R + Z_ * Z_ * sj * si)
            V1[:, k] -= S * Q
            V2[:, k] += C * Q
            V3[:, k] -= J
            inside[:, k] *= (R >= 0).to(R.dtype)
            zeros[:, k] += (R == 0).to(R.dtype)
    V3 = (V3 + 2 * math.pi * inside) * z.sign() * (zeros <= 1)
    return tuple((V1 * _row(ax[0])[q] + V2 * _row(ax[1])[q] + V3 * _row(ax[2])[q]) / (4 * math.pi) for q in range(3))


def _step(n):
    return max(16, int(6e7 / n))


def _matrix(m, D, normals, cps, idx, nn, nodes):
    """Unit-strength normal velocity of every panel (column) at every control point (row)."""
    N = cps.shape[0]
    G = torch.empty(N, N, dtype=torch.float64, device=cps.device)
    wake = _Wake(m, idx) if len(D) else None
    for i in range(0, N, _step(N)):
        j = min(N, i + _step(N))
        X, n = _col(cps[i:j]), _col(normals[i:j])
        G[i:j] = _dot(_rings(X, nodes, idx) if m.bodies[0].kind != "source" else _sources(X, nodes, idx, nn), n)
        if wake:
            wake.add(X, nodes, D, lambda panels, u: G[i:j].index_add_(1, panels, _dot(u, n)))
    return G


def _field(m, D, gamma, targets, idx, nodes):
    """Velocity induced at the targets by the solved body and its wake."""
    out, wake = torch.zeros_like(targets), _Wake(m, idx)
    for i in range(0, len(targets), _step(len(gamma))):
        j = min(len(targets), i + _step(len(gamma)))
        X = _col(targets[i:j])
        out[i:j] += torch.stack([u @ gamma for u in _rings(X, nodes, idx)], dim=1)
        wake.add(X, nodes, D, lambda panels, u: out[i:j].add_(torch.stack([v @ gamma[panels] for v in u], dim=1)))
    return out


def _gradient(m, D, U, gamma, lam, idx, nn, nodes):
    """Gradients of lam^T (b - A gamma) by vertex, freestream and wake direction, lam and gamma held."""
    nodes, D, U = (a.clone().requires_grad_() for a in (nodes, D, U))
    wake, sums = _Wake(m, idx), [torch.zeros_like(a) for a in (nodes, U, D)]
    step = max(8, _step(len(gamma)) // 16)
    for i in range(0, len(gamma), step):
        j = min(len(gamma), i + step)
        normals, cps, _ = _geometry(nodes, idx, nn)
        X, n = _col(cps[i:j]), _col(normals[i:j])
        parts = [-(U[i:j] * normals[i:j]).sum(1) - _dot(_rings(X, nodes, idx), n) @ gamma]
        wake.add(X, nodes, D, lambda panels, u: parts.append(-(_dot(u, n) @ gamma[panels])))
        for a, g in zip(sums, torch.autograd.grad((lam[i:j] * sum(parts)).sum(), (nodes, U, D))):
            a += g
    return sums


def exact(case, seed):
    p = _problem(case, seed)
    kind = case["kind"]
    if kind == "batch":
        return [_strengths(m, _t(np.tile(p["V"], (m.nsheddings, 1))), _t(np.tile(p["V"], (m.npanels, 1)))).cpu() for m in p["meshes"]]
    m, D, U = p["mesh"], _t(p["D"]), _t(p["U"])
    if kind == "duct":
        return _least_squares(m, D, U).cpu()
    if kind == "gradient":
        nodes, (idx, nn) = _t(m.nodes), _corners(m)
        normals, cps, _ = _geometry(nodes, idx, nn)
        G = _matrix(m, D, normals, cps, idx, nn, nodes)
        gamma = torch.linalg.solve(G, -(U * normals).sum(1))
        lam = torch.linalg.solve(G.T, _t(p["w"]))
        return {"gamma": gamma.cpu(), "grads": tuple(g.cpu() for g in _gradient(m, D, U, gamma, lam, idx, nn, nodes))}
    gamma = _strengths(m, D, U)
    if kind not in ("loads", "probes"):
        return gamma.cpu()
    nodes, (idx, nn) = _t(m.nodes), _corners(m)
    if kind == "probes":
        return (_t(p["V"])[None] + _field(m, D, gamma, _t(p["X"]), idx, nodes)).cpu()
    normals, cps, area = _geometry(nodes, idx, nn, 0.02)
    vel = U + _field(m, D, gamma, cps, idx, nodes)
    Cp = (1 - (vel * vel).sum(1)).cpu().numpy()
    normals, area = normals.cpu().numpy(), area.cpu().numpy()
    rows = [(r[0], r[0] + 1, r[3], r[3] - 1) for r in m.shedding]
    for r in rows:
        Cp[list(r)] = Cp[list(r)].mean()
    F = -0.5 * 1.225 * (Cp * area)[:, None] * normals
    for r in rows:
        ave = Cp[list(r)].mean()
        for i in r:
            F[i] = -0.5 * 1.225 * ave * area[i] * normals[i]
    S = np.array([0.0, 1.0, 0.0])
    lds = np.stack([e * F.sum(0).dot(e) for e in (np.cross(p["V"], S), p["V"], S)], axis=1)
    return {"lds": lds, "U": vel.cpu(), "Cp": Cp, "F": F}


def _strengths(m, D, U):
    """The strengths for one freestream (N, 3) or several (k, N, 3)."""
    nodes, (idx, nn) = _t(m.nodes), _corners(m)
    normals, cps, _ = _geometry(nodes, idx, nn)
    b = -(U * normals).sum(-1)
    x = torch.linalg.solve(_matrix(m, D, normals, cps, idx, nn, nodes), b.T if b.dim() == 2 else b)
    return x.T.contiguous() if b.dim() == 2 else x


def _least_squares(m, D, U):
    """The watertight body's strengths: the first panel's is zero, the others the least-squares solution (by QR)."""
    nodes, (idx, nn) = _t(m.nodes), _corners(m)
    normals, cps, _ = _geometry(nodes, idx, nn)
    G = _matrix(m, D, normals, cps, idx, nn, nodes)
    Q, R = torch.linalg.qr(G[:, 1:])
    x = torch.linalg.solve_triangular(R, (Q.T @ -(U * normals).sum(1))[:, None], upper=True)
    return torch.cat([torch.zeros_like(x[:1, 0]), x[:, 0]])
