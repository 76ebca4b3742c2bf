"""Timed cases of the library: the work a finite-element user has it do, through the public
entry points of ``adfem_gpu``.

Meshes are unit squares of m x n cells, each cell split into two triangles, interior nodes
jittered by up to 0.2 cells; coefficients are random Fourier fields at the Gauss points.
Kinds of case:

    ops      summed P1 operators on the device (matrix values and load vector)
    coo      the graph-op arm: unsummed COO values and load, forward and backward, P1 or P2
    stiff    the elasticity operators: material, summed and COO stiffness, their backward ops
    p2ops    P2 operators: Laplace, mass, load, interpolation and its transpose
    array    the host Array arm: numpy fields in, sparse matrix, Dirichlet, K\\F, numpy out
    solve    a resident Poisson system: assembly and one forward solve
    grad     the same with the misfit's adjoint solve and the kappa-gradient, P1 or P2
    elastic  a resident elasticity system: assembly, forward, adjoint, E-gradient
    serve    a batch of requests of uneven sizes through the request server
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "adfem.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)


def listed():
    return [
        # the smallest operator calls: 64 x 64 cells, where latency and launches count
        {"name": "ops_64", "kind": "ops", "m": 64, "n": 64},
        # the graph-op arm of a large inverse problem (2M elements, forward and backward)
        {"name": "coo_p1_1000x990", "kind": "coo", "m": 1000, "n": 990, "degree": 1},
        # the same on a medium P2 mesh of odd sizes
        {"name": "coo_p2_161x120", "kind": "coo", "m": 161, "n": 120, "degree": 2},
        # every elasticity operator of a medium mesh, both directions
        {"name": "stiff_401x400", "kind": "stiff", "m": 401, "n": 400},
        # P2 operators and interpolation, forward and transpose
        {"name": "p2ops_400", "kind": "p2ops", "m": 400, "n": 400},
        # the README's host pipeline at 64 x 64: matrix, load, Dirichlet, K\F on numpy arrays
        {"name": "array_64", "kind": "array", "m": 64, "n": 64},
        # a small resident system at the default precision: assembly and solve
        {"name": "solve_fp64_64", "kind": "solve", "m": 64, "n": 64, "precision": "fp64", "rtol": 1e-12,
         "contrast": 10.0},
        # inverse Poisson at 1M DOF: forward, adjoint, gradient of 6M coefficients
        {"name": "grad_mixed_1000", "kind": "grad", "m": 1000, "n": 1000, "degree": 1, "precision": "mixed",
         "rtol": 1e-11, "contrast": 30.0},
        # the headline solve: 4M DOF, coefficient contrast 1e3
        {"name": "solve_mixed_2000", "kind": "solve", "m": 2000, "n": 2000, "precision": "mixed", "rtol": 1e-11,
         "contrast": 1e3},
        # elasticity with a gradient, 320k DOF, odd sizes
        {"name": "elastic_mixed_399x401", "kind": "elastic", "m": 399, "n": 401, "precision": "mixed",
         "rtol": 1e-11},
        # a resident P2 system with its gradient, 240k DOF
        {"name": "grad_p2_251x241", "kind": "grad", "m": 251, "n": 241, "degree": 2, "precision": "mixed",
         "rtol": 1e-11, "contrast": 30.0},
        # the serving mix: small and medium requests of both kinds, half with gradients
        {"name": "serve_24", "kind": "serve", "requests": 24, "lo": 16, "hi": 160, "rtol": 1e-12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ops", "coo", "stiff", "p2ops", "array", "solve", "grad", "elastic", "serve"])
    if kind == "serve":
        lo = _log(rng, 12, 24)
        return {"kind": kind, "requests": rng.randint(4, 24), "lo": lo, "hi": _log(rng, 2 * lo, 160), "rtol": 1e-12}
    degree = rng.choice([1, 1, 2]) if kind in ("coo", "grad") else 1
    hi = {"ops": 1400, "coo": 900 if degree == 1 else 400, "stiff": 400, "p2ops": 500, "array": 100, "solve": 900,
          "grad": 700 if degree == 1 else 240, "elastic": 300}[kind]
    lo = {"array": 16}.get(kind, 24)
    m = _log(rng, lo, hi)
    n = max(8, min(hi, int(m * rng.uniform(0.6, 1.4))))
    case = {"kind": kind, "m": m, "n": n}
    if kind in ("coo", "grad"):
        case["degree"] = degree
    if kind in ("solve", "grad", "elastic"):
        case["precision"] = rng.choice(["mixed", "mixed", "fp64"]) if m * n <= 250000 else "mixed"
        case["rtol"] = 1e-12 if case["precision"] == "fp64" else 1e-11
    if kind in ("solve", "grad"):
        case["contrast"] = rng.choice([3.0, 30.0, 1e3])
    return case


# ------------------------------------------------------------------ inputs
def _square(m, n, seed):
    """Coordinates (nodes numbered x-fastest) and 0-based counterclockwise triangles."""
    rng = np.random.default_rng(seed)
    jj, ii = np.meshgrid(np.arange(m + 1), np.arange(n + 1))
    jj, ii = jj.ravel(), ii.ravel()
    inner = (jj > 0) & (jj < m) & (ii > 0) & (ii < n)
    d = rng.uniform(-0.2, 0.2, (jj.size, 2)) * inner[:, None]
    xy = np.stack([(jj + d[:, 0]) / m, (ii + d[:, 1]) / n], axis=1)
    a = (np.arange(n)[:, None] * (m + 1) + np.arange(m)[None, :]).ravel()
    el = np.empty((2 * m * n, 3), np.int64)
    el[0::2] = np.stack([a, a + 1, a + m + 1], 1)
    el[1::2] = np.stack([a + 1, a + m + 2, a + m + 1], 1)
    return xy, el


_A1, _A2 = 0.091576213509770743460, 0.44594849091596488632
_RULE = {
    1: (np.array([[1 / 6, 1 / 6], [1 / 6, 2 / 3], [2 / 3, 1 / 6]]), np.full(3, 1 / 6)),
    2: (np.array([[_A1, _A1], [_A1, 1 - 2 * _A1], [1 - 2 * _A1, _A1], [_A2, _A2], [_A2, 1 - 2 * _A2],
                  [1 - 2 * _A2, _A2]]),
        np.array([0.054975871827660933819] * 3 + [0.11169079483900573285] * 3)),
}


def _dev(a):
    return torch.as_tensor(a, device="cuda")


def _points(xy, el, degree):
    """Gauss points (element-major) on the device."""
    p = _dev(xy)[_dev(el)]
    q = _dev(_RULE[degree][0])
    lam = torch.stack([1 - q[:, 0] - q[:, 1], q[:, 0], q[:, 1]], 1)
    g = torch.einsum("kc,ecd->ekd", lam, p).reshape(-1, 2)
    return g[:, 0].contiguous(), g[:, 1].contiguous()


def _field(x, y, seed):
    """Unit-variance random Fourier field (64 modes, wavenumbers up to 16 pi)."""
    rng = np.random.default_rng(seed)
    r, th = 16 * math.pi * np.sqrt(rng.random(64)), 2 * math.pi * rng.random(64)
    kx, ky, ph = r * np.cos(th), r * np.sin(th), 2 * math.pi * rng.random(64)
    out = torch.zeros_like(x)
    for j in range(64):
        out += torch.cos(kx[j] * x + (ky[j] * y + ph[j]))
    return math.sqrt(2 / 64) * out


def _kappa(x, y, seed, contrast):
    """1 + exp(s G), s such that max / min is `contrast`."""
    g = _field(x, y, seed)
    hi, lo = float(g.max()), float(g.min())
    a, b = 0.0, 64.0
    for _ in range(100):
        s = 0.5 * (a + b)
        if math.log1p(math.exp(s * hi)) - math.log1p(math.exp(s * lo)) < math.log(contrast):
            a = s
        else:
            b = s
    return 1 + torch.exp(a * g)


def _rand(n, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)


def _sub(seed, k):
    return (1000003 * seed + 7919 * k + 1) % (1 << 31)


def _boundary(m, n):
    """1-based boundary vertices."""
    j, i = np.meshgrid(np.arange(m + 1), np.arange(n + 1))
    on = (i == 0) | (i == n) | (j == 0) | (j == m)
    return np.flatnonzero(on.ravel()) + 1


def _edges(el, nv):
    """Edge ids of each element's local edges (0,1), (1,2), (2,0), numbered by first
    appearance, and the endpoints of each edge."""
    a = np.stack([el[:, 0], el[:, 1], el[:, 2]], 1).ravel()
    b = np.stack([el[:, 1], el[:, 2], el[:, 0]], 1).ravel()
    key = np.minimum(a, b) * nv + np.maximum(a, b)
    uniq, first, inv = np.unique(key, return_index=True, return_inverse=True)
    rank = np.empty(uniq.size, np.int64)
    order = np.argsort(first, kind="stable")
    rank[order] = np.arange(uniq.size)
    ends = np.stack([uniq // nv, uniq % nv], 1)[order]
    return rank[inv.ravel()].reshape(-1, 3), ends


def _dofs(case, xy, el):
    """DOFs of each element, DOF count, 1-based boundary DOFs, grid row of each DOF."""
    m, n = case["m"], case["n"]
    nv = xy.shape[0]
    row = np.arange(nv) // (m + 1)
    bd = _boundary(m, n)
    if case.get("degree", 1) == 1:
        return el, nv, bd, row
    ee, ends = _edges(el, nv)
    cnt = np.bincount(ee.ravel(), minlength=ends.shape[0])
    bd = np.concatenate([bd, nv + np.flatnonzero(cnt == 1) + 1])
    return np.concatenate([el, nv + ee], 1), nv + ends.shape[0], bd, np.concatenate([row, row[ends].min(axis=1)])


def _obs(ndof, seed):
    """1% of the DOFs (0-based, ascending) and noise of the observations there."""
    rng = np.random.default_rng(seed)
    k = np.sort(rng.choice(ndof, max(1, ndof // 100), replace=False))
    return k, 1e-3 * rng.standard_normal(k.size)


def _poisson_fields(case, xy, el, seed):
    x, y = _points(xy, el, case.get("degree", 1))
    return _kappa(x, y, _sub(seed, 1), case.get("contrast", 10.0)), 1e5 * (x + y + 0.1 * _field(x, y, _sub(seed, 2)))


def _elastic_fields(xy, el, seed):
    x, y = _points(xy, el, 1)
    E = 1e9 * torch.exp(0.3 * _field(x, y, _sub(seed, 1)))
    nu = 0.3 + 0.02 * torch.tanh(_field(x, y, _sub(seed, 2)))
    return E, nu, torch.zeros_like(E), -1e6 * (1 + 0.1 * _field(x, y, _sub(seed, 3)))


def _clamped(m, n):
    """1-based DOFs of the clamped left edge, both components."""
    left = np.arange(n + 1) * (m + 1) + 1
    return np.concatenate([left, left + (m + 1) * (n + 1)])


def _requests(case, seed):
    """Sizes and kinds come from the case (the same meshes stay in service), fields from the seed."""
    rng = np.random.default_rng(4242 + case["requests"])
    out = []
    for k in range(case["requests"]):
        m = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append({"m": m, "n": m, "elastic": k % 5 == 4, "grad": k % 2 == 0, "contrast": 30.0,
                    "seed": _sub(seed, 100 + k)})
    return out


def _request_inputs(r):
    xy, el = _square(r["m"], r["n"], r["seed"])
    if r["elastic"]:
        fields, bd, ndof = _elastic_fields(xy, el, r["seed"]), _clamped(r["m"], r["n"]), 2 * xy.shape[0]
    else:
        fields, bd, ndof = _poisson_fields(r, xy, el, r["seed"]), _boundary(r["m"], r["n"]), xy.shape[0]
    obs, noise = _obs(ndof, _sub(r["seed"], 5))
    return xy, el, fields, bd, obs, noise


# ------------------------------------------------------------------ one pass
def prepare(case, seed):
    import adfem_gpu as A
    from adfem_gpu import _lib, system

    kind = case["kind"]
    s = {"kind": kind, "A": A, "S": system, "case": case}
    if kind == "serve":
        s["server"] = A.Server(workers=8, precision="mixed", rtol=case["rtol"])
        s["requests"] = []
        for r in _requests(case, seed):
            xy, el, fields, bd, obs, noise = _request_inputs(r)
            args = [A.Mesh(xy, el + 1), _lib.SYS_ELASTICITY if r["elastic"] else _lib.SYS_POISSON,
                    tuple(f.cpu().numpy() for f in fields), bd]
            s["requests"].append((args, {"obs": obs + 1, "uobs": noise} if r["grad"] else {}))
        return s
    m, n, degree = case["m"], case["n"], case.get("degree", 2 if kind == "p2ops" else 1)
    xy, el = _square(m, n, _sub(seed, 0))
    mesh = s["mesh"] = A.Mesh(xy, el + 1, degree=degree)
    ng, nd2 = A.get_ngauss(mesh), mesh.elem_ndof ** 2
    if kind in ("ops", "coo", "p2ops"):
        s["kappa"], s["f"] = _poisson_fields({**case, "degree": degree}, xy, el, seed)
        if kind == "coo":
            s["gvv"], s["grhs"] = _rand(nd2 * ng, _sub(seed, 3)), _rand(mesh.ndof, _sub(seed, 4))
        if kind == "p2ops":
            s["u"], s["gout"] = _rand(mesh.ndof, _sub(seed, 3)), _rand(ng, _sub(seed, 4))
            s["grhs"] = _rand(mesh.ndof, _sub(seed, 5))
        mesh.pattern()
    elif kind == "stiff":
        s["E"], s["nu"] = _elastic_fields(xy, el, seed)[:2]
        s["gvv"] = _rand(4 * nd2 * ng, _sub(seed, 3))
        mesh.pattern_elasticity()
    elif kind == "array":
        s["kappa"], s["f"] = (t.cpu().numpy() for t in _poisson_fields(case, xy, el, seed))
        s["bd"] = A.bcnode(mesh)
        s["bdval"] = np.zeros(s["bd"].size)
        mesh.pattern()
    elif kind in ("solve", "grad"):
        s["kappa"], s["f"] = _poisson_fields(case, xy, el, seed)
        s["sys"] = A.PoissonSystem(mesh)
        s["sys"].set_dirichlet(A.bcnode(mesh))
    else:
        s["E"], s["nu"], s["fx"], s["fy"] = _elastic_fields(xy, el, seed)
        s["sys"] = A.ElasticitySystem(mesh)
        s["sys"].set_dirichlet(_clamped(m, n))
    if kind in ("grad", "elastic"):
        k, noise = _obs(s["sys"].ndof, _sub(seed, 5))
        s["obs"], s["uobs"] = _dev(k), _dev(noise)
    return s


def run(s):
    A, S, kind = s["A"], s["S"], s["kind"]
    if kind == "serve":
        tickets = [s["server"].submit(*a, **kw) for a, kw in s["requests"]]
        done = [s["server"].wait(t) for t in tickets]
        if any(r["status"] for r, _, _ in done):
            raise RuntimeError("a request failed")
        return {"u": [u for _, u, _ in done], "grad": [g for _, _, g in done if g is not None]}
    mesh, case = s["mesh"], s["case"]
    if kind == "ops":
        return {"K": S.laplace_csr(mesh, s["kappa"]), "F": S.source(mesh, s["f"])}
    if kind == "coo":
        idx, vv = S.laplace_coo(mesh, s["kappa"])
        return {"idx": idx, "vv": vv, "F": S.source(mesh, s["f"]),
                "gkappa": S.laplace_coo_backward(mesh, s["gvv"]), "gf": S.source_backward(mesh, s["grhs"])}
    if kind == "stiff":
        D = S.plane_strain(s["E"], s["nu"])
        idx, vv = S.stiffness_coo(mesh, D)
        gD = S.stiffness_coo_backward(mesh, s["gvv"])
        gE, gnu = S.plane_strain_backward(gD, s["E"], s["nu"])
        return {"D": D, "K": S.stiffness_csr(mesh, D), "idx": idx, "vv": vv, "gD": gD, "gE": gE, "gnu": gnu}
    if kind == "p2ops":
        return {"K": S.laplace_csr(mesh, s["kappa"]), "M": S.mass_csr(mesh, s["kappa"]), "F": S.source(mesh, s["f"]),
                "gf": S.source_backward(mesh, s["grhs"]), "ug": S.dof_to_gauss(mesh, s["u"]),
                "gu": S.dof_to_gauss_backward(mesh, s["gout"])}
    if kind == "array":
        K = A.compute_fem_laplace_matrix1(s["kappa"], mesh)
        F = A.compute_fem_source_term1(s["f"], mesh)
        B, r = A.impose_Dirichlet_boundary_conditions(K, F, s["bd"], s["bdval"])
        return {"K": K.data, "B": B.data, "r": r, "u": A.solve(B, r)}
    sysm, o = s["sys"], {"precision": case["precision"], "rtol": case["rtol"]}
    if kind == "elastic":
        sysm.assemble(s["E"], s["nu"], s["fx"], s["fy"])
    else:
        sysm.assemble(s["kappa"], s["f"])
    u = sysm.solve(**o)
    if kind == "solve":
        return {"u": u}
    g = torch.zeros_like(u)
    g[s["obs"]] = 2 * (u[s["obs"]] - s["uobs"])
    lam = sysm.adjoint(g, **o)
    grad = sysm.grad_E(u, lam, s["E"], s["nu"]) if kind == "elastic" else sysm.grad_kappa(u, lam)
    return {"u": u, "lam": lam, "grad": grad}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "serve":
        total = {"bytes": 0, "flops": 0}
        for r in _requests(case, 0):
            w = work({"kind": "elastic" if r["elastic"] else "grad", "m": r["m"], "n": r["n"], "degree": 1})
            total["bytes"] += w["bytes"]
            total["flops"] += w["flops"]
        return total
    m, n = case["m"], case["n"]
    nv, ne = (m + 1) * (n + 1), 2 * m * n
    nedge = 3 * m * n + m + n
    degree = case.get("degree", 2 if kind == "p2ops" else 1)
    nd, ng = (3, 3 * ne) if degree == 1 else (6, 6 * ne)
    ndof = nv if degree == 1 else nv + nedge
    # entries of the DOF graph: the diagonal and both directions of every coupled pair (15 pairs
    # a P2 element, 3 of them shared across each inner edge)
    nnz = nv + 2 * nedge if degree == 1 else ndof + 2 * (15 * ne - 3 * (nedge - 2 * m - 2 * n))
    mesh = 16 * nv + 12 * ne
    field = 8 * ng
    if kind == "ops":
        return {"bytes": mesh + 2 * field + 8 * nnz + 8 * ndof, "flops": 20 * ne}
    if kind == "coo":
        return {"bytes": mesh + (24 + 8) * nd * nd * ng + 4 * field + 16 * ndof, "flops": 6 * nd * nd * ng}
    if kind == "stiff":
        return {"bytes": mesh + 4 * field + 3 * 9 * field + 8 * 4 * nnz + (24 + 8) * 36 * ng,
                "flops": 36 * 10 * ng}
    if kind == "p2ops":
        return {"bytes": mesh + 5 * field + 16 * nnz + 32 * ndof, "flops": 400 * ng}
    if kind == "array":
        return {"bytes": mesh + 2 * field + 3 * 8 * nnz + 16 * ndof, "flops": 60 * nnz}
    if kind == "elastic":
        return {"bytes": mesh + 6 * field + 16 * 4 * nnz + 3 * 16 * ndof, "flops": 2 * 60 * 4 * nnz}
    solves = 2 if kind == "grad" else 1
    return {"bytes": mesh + (2 + (solves - 1)) * field + 8 * (1 + solves) * nnz + 16 * solves * ndof,
            "flops": 60 * solves * nnz}


# ------------------------------------------------------------------ plain 64-bit results
class _Elements:
    """Gradients, weights and basis tables of every element, 64 bits, on the device."""

    def __init__(self, xy, el, dof, degree):
        p = _dev(xy)[_dev(el)]
        e1, e2 = p[:, 1] - p[:, 0], p[:, 2] - p[:, 0]
        det = e1[:, 0] * e2[:, 1] - e1[:, 1] * e2[:, 0]
        l1 = torch.stack([e2[:, 1], -e2[:, 0]], 1) / det[:, None]
        l2 = torch.stack([-e1[:, 1], e1[:, 0]], 1) / det[:, None]
        gl = torch.stack([-(l1 + l2), l1, l2], 1)  # gradients of the barycentric coordinates
        q, w = _RULE[degree]
        lam = np.stack([1 - q[:, 0] - q[:, 1], q[:, 0], q[:, 1]], 1)
        if degree == 1:
            h, t = lam, np.broadcast_to(np.eye(3), (3, 3, 3))
        else:
            k = lam.shape[0]
            h, t = np.zeros((k, 6)), np.zeros((k, 6, 3))
            for a in range(3):
                b = (a + 1) % 3
                h[:, a], t[:, a, a] = lam[:, a] * (2 * lam[:, a] - 1), 4 * lam[:, a] - 1
                h[:, 3 + a], t[:, 3 + a, a], t[:, 3 + a, b] = 4 * lam[:, a] * lam[:, b], 4 * lam[:, b], 4 * lam[:, a]
        self.h = _dev(np.ascontiguousarray(h))
        self.w = det[:, None] * _dev(w)[None, :]                                      # (e, k)
        self.g = torch.einsum("krc,ecd->ekrd", _dev(np.ascontiguousarray(t)), gl)      # (e, k, r, d)
        self.dof = _dev(dof)
        self.ndof = int(dof.max()) + 1

    def laplace(self, kappa):
        kw = kappa.reshape(self.w.shape) * self.w
        return torch.einsum("ekrd,eksd->ekrs", self.g, self.g) * kw[:, :, None, None]

    def mass(self, rho):
        return torch.einsum("kr,ks->krs", self.h, self.h)[None] * (rho.reshape(self.w.shape) * self.w)[:, :, None, None]

    def pairs(self, shape):
        d = self.dof
        r, c = torch.broadcast_tensors(d[:, None, :, None], d[:, None, None, :])
        return r.expand(shape).reshape(-1), c.expand(shape).reshape(-1)

    def load(self, f):
        v = torch.einsum("ek,kr->er", f.reshape(self.w.shape) * self.w, self.h)
        return torch.zeros(self.ndof, dtype=torch.float64, device="cuda").index_add_(0, self.dof.reshape(-1),
                                                                                    v.reshape(-1))

    def b(self):
        """Strain matrices (e, k, 3, 2 nd), columns [x; y]."""
        gx, gy = self.g[..., 0], self.g[..., 1]
        z = torch.zeros_like(gx)
        return torch.stack([torch.cat([gx, z], -1), torch.cat([z, gy], -1), torch.cat([gy, gx], -1)], -2)


def _summed(r, c, v, n):
    """Values of the summed matrix in row-major order of its entries, and the entries."""
    key, inv = torch.unique(r * n + c, return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_add_(0, inv, v)
    return key // n, key % n, val


def _dmat(E, nu):
    s = E * (1 - nu) / (1 + nu) / (1 - 2 * nu)
    a = s * nu / (1 - nu)
    D = a[:, None, None].expand(-1, 3, 3).clone()
    for j in range(3):
        D[:, j, j] = s
    return D


def _dmat_d(E, nu):
    """Derivatives of the diagonal and off-diagonal entries with respect to E and nu."""
    q = (1 + nu) * (1 - 2 * nu)
    return (1 - nu) / q, nu / q, E * 2 * nu * (2 - nu) / q ** 2, E * (1 + 2 * nu ** 2) / q ** 2


class _Direct:
    """Block tridiagonal Cholesky over the grid rows, with one step of refinement."""

    def __init__(self, r, c, v, row):
        self.r, self.c, self.v, self.n = r, c, v, row.size
        order = np.argsort(row, kind="stable")
        self.start = np.concatenate([[0], np.cumsum(np.bincount(row))])
        pos = np.empty(row.size, np.int64)
        pos[order] = np.arange(row.size)
        self.order = _dev(order)
        pr, pc, rr, rc = _dev(pos)[r], _dev(pos)[c], _dev(row)[r], _dev(row)[c]
        nb = self.start.size - 1
        srt = torch.argsort(rr * 2 + (rc > rr).long() + 2 * nb * (rc < rr).long(), stable=True)
        tag = (rr * 2 + (rc > rr).long() + 2 * nb * (rc < rr).long())[srt]
        cut = torch.searchsorted(tag, torch.arange(2 * nb + 1, device="cuda")).cpu().numpy()
        pr, pc, vv = pr[srt], pc[srt], v[srt]
        st = self.start

        def block(tagno, i, j):
            B = torch.zeros(int(st[i + 1] - st[i]), int(st[j + 1] - st[j]), dtype=torch.float64, device="cuda")
            a, b = int(cut[tagno]), int(cut[tagno + 1])
            return B.index_put_((pr[a:b] - int(st[i]), pc[a:b] - int(st[j])), vv[a:b])

        self.L, self.W = [], []
        D = block(0, 0, 0)
        for i in range(nb):
            L = torch.linalg.cholesky_ex(D)[0]
            self.L.append(L)
            if i + 1 < nb:
                Y = torch.linalg.solve_triangular(L, block(2 * i + 1, i, i + 1), upper=False)
                self.W.append(Y)
                D = block(2 * i + 2, i + 1, i + 1) - Y.T @ Y

    def _once(self, b):
        b = b[self.order]
        st, nb, y = self.start, len(self.L), []
        for i in range(nb):
            x = b[int(st[i]):int(st[i + 1])]
            if i:
                x = x - self.W[i - 1].T @ y[-1]
            y.append(torch.linalg.solve_triangular(self.L[i], x[:, None], upper=False)[:, 0])
        out = [None] * nb
        for i in reversed(range(nb)):
            x = y[i] - self.W[i] @ out[i + 1] if i + 1 < nb else y[i]
            out[i] = torch.linalg.solve_triangular(self.L[i].T, x[:, None], upper=True)[:, 0]
        u = torch.empty_like(b)
        u[self.order] = torch.cat(out)
        return u

    def solve(self, b):
        u = self._once(b)
        res = b - torch.zeros_like(b).index_add_(0, self.r, self.v * u[self.c])
        return u + self._once(res)


def _dirichlet0(r, c, v, F, bd1):
    """Homogeneous Dirichlet conditions: identity rows and columns, zero loads."""
    on = torch.zeros(F.numel(), dtype=torch.bool, device="cuda")
    on[_dev(bd1 - 1)] = True
    v = torch.where(on[r] | on[c], (r == c).double(), v)
    return v, torch.where(on, torch.zeros_like(F), F), on


def _exact_solve(case, xy, el, fields, obs, noise, grad):
    dof, ndof, bd, row = _dofs(case, xy, el)
    kappa, f = fields
    X = _Elements(xy, el, dof, case.get("degree", 1))
    N = X.laplace(kappa).sum(1)[:, None]
    r, c, v = _summed(*X.pairs(N.shape), N.reshape(-1), ndof)
    v, F, on = _dirichlet0(r, c, v, X.load(f), bd)
    K = _Direct(r, c, v, row)
    u = K.solve(F)
    if not grad:
        return u, None, None
    g = torch.zeros_like(u)
    g[_dev(obs)] = 2 * (u[_dev(obs)] - _dev(noise))
    lam = torch.where(on, torch.zeros_like(u), K.solve(torch.where(on, torch.zeros_like(g), g)))
    gu = torch.einsum("ekrd,er->ekd", X.g, u[X.dof])
    gl = torch.einsum("ekrd,er->ekd", X.g, lam[X.dof])
    return u, lam, (-X.w * (gu * gl).sum(-1)).reshape(-1)


def _exact_elastic(case, xy, el, fields, obs, noise, grad):
    E, nu, fx, fy = fields
    nv = xy.shape[0]
    X = _Elements(xy, el, el, 1)
    B = X.b()
    D = _dmat(E, nu).reshape(-1, 3, 3, 3)
    N = torch.einsum("ekps,ekpq,ekqt->est", B, D * X.w[:, :, None, None], B)
    d2 = torch.cat([X.dof, X.dof + nv], 1)
    r, c = (t.reshape(-1) for t in torch.broadcast_tensors(d2[:, :, None], d2[:, None, :]))
    r, c, v = _summed(r, c, N.reshape(-1), 2 * nv)
    v, F, on = _dirichlet0(r, c, v, torch.cat([X.load(fx), X.load(fy)]), _clamped(case["m"], case["n"]))
    K = _Direct(r, c, v, np.tile(np.arange(nv) // (case["m"] + 1), 2))
    u = K.solve(F)
    if not grad:
        return u, None, None
    g = torch.zeros_like(u)
    g[_dev(obs)] = 2 * (u[_dev(obs)] - _dev(noise))
    lam = torch.where(on, torch.zeros_like(u), K.solve(torch.where(on, torch.zeros_like(g), g)))
    eu = torch.einsum("ekpc,ec->ekp", B, u[d2])
    ev = torch.einsum("ekpc,ec->ekp", B, lam[d2])
    dd = (eu * ev).sum(-1)
    off = eu.sum(-1) * ev.sum(-1) - dd
    sd, so = _dmat_d(E, nu)[:2]
    return u, lam, (-X.w * (sd.reshape(X.w.shape) * dd + so.reshape(X.w.shape) * off)).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        us, gs = [], []
        for q in _requests(case, seed):
            xy, el, fields, _, obs, noise = _request_inputs(q)
            u, _, g = (_exact_elastic if q["elastic"] else _exact_solve)(q, xy, el, fields, obs, noise, q["grad"])
            us.append(u)
            gs += [g] if g is not None else []
        return {"u": us, "grad": gs}
    m, n = case["m"], case["n"]
    if kind in ("solve", "grad", "elastic") and min(m, n) > 1100:
        return None  # the direct solve would take minutes
    xy, el = _square(m, n, _sub(seed, 0))
    degree = case.get("degree", 2 if kind == "p2ops" else 1)
    cased = {**case, "degree": degree}
    dof, ndof, bd, row = _dofs(cased, xy, el)
    if kind == "stiff":
        E, nu = _elastic_fields(xy, el, seed)[:2]
        X = _Elements(xy, el, dof, 1)
        B, D = X.b(), _dmat(E, nu).reshape(-1, 3, 3, 3)
        N = torch.einsum("ekps,ekpq,ekqt->ekst", B, D, B) * X.w[:, :, None, None]
        d2 = torch.cat([X.dof, X.dof + ndof], 1)
        r, c = (t.expand(N.shape).reshape(-1) for t in torch.broadcast_tensors(d2[:, None, :, None],
                                                                              d2[:, None, None, :]))
        G = _rand(N.numel(), _sub(seed, 3)).reshape(N.shape)
        gD = torch.einsum("ekps,ekst,ekqt->ekpq", B, G, B) * X.w[:, :, None, None]
        gD = gD.reshape(-1, 3, 3)
        gd = gD.diagonal(dim1=1, dim2=2).sum(1)
        go = gD.sum((1, 2)) - gd
        sd, so, nd_, no = _dmat_d(E, nu)
        return {"D": D.reshape(-1), "K": _summed(r, c, N.reshape(-1), 2 * ndof)[2], "idx": torch.stack([r, c], 1),
                "vv": N.reshape(-1), "gD": gD.reshape(-1), "gE": gd * sd + go * so, "gnu": gd * nd_ + go * no}
    if kind == "elastic":
        obs, noise = _obs(2 * xy.shape[0], _sub(seed, 5))
        u, lam, g = _exact_elastic(case, xy, el, _elastic_fields(xy, el, seed), obs, noise, True)
        return {"u": u, "lam": lam, "grad": g}
    kappa, f = _poisson_fields(cased, xy, el, seed)
    if kind in ("solve", "grad"):
        obs, noise = _obs(ndof, _sub(seed, 5))
        u, lam, g = _exact_solve(cased, xy, el, (kappa, f), obs, noise, kind == "grad")
        return {"u": u} if kind == "solve" else {"u": u, "lam": lam, "grad": g}
    X = _Elements(xy, el, dof, degree)
    N = X.laplace(kappa)
    r, c = X.pairs(N.shape)
    if kind == "coo":
        ng, nd = X.w.numel(), dof.shape[1]
        G = _rand(nd * nd * ng, _sub(seed, 3)).reshape(N.shape)
        grhs = _rand(ndof, _sub(seed, 4))
        gk = (G * X.laplace(torch.ones_like(kappa))).sum((2, 3)).reshape(-1)
        gf = (torch.einsum("kr,er->ek", X.h, grhs[X.dof]) * X.w).reshape(-1)
        return {"idx": torch.stack([r, c], 1), "vv": N.reshape(-1), "F": X.load(f), "gkappa": gk, "gf": gf}
    kr, kc, kv = _summed(r, c, N.reshape(-1), ndof)
    if kind == "ops":
        return {"K": kv, "F": X.load(f)}
    if kind == "p2ops":
        M = X.mass(kappa)
        u, gout, grhs = _rand(ndof, _sub(seed, 3)), _rand(X.w.numel(), _sub(seed, 4)), _rand(ndof, _sub(seed, 5))
        gu = torch.einsum("ek,kr->er", gout.reshape(X.w.shape), X.h)
        return {"K": kv, "M": _summed(r, c, M.reshape(-1), ndof)[2], "F": X.load(f),
                "gf": (torch.einsum("kr,er->ek", X.h, grhs[X.dof]) * X.w).reshape(-1),
                "ug": torch.einsum("kr,er->ek", X.h, u[X.dof]).reshape(-1),
                "gu": torch.zeros(ndof, dtype=torch.float64, device="cuda").index_add_(0, X.dof.reshape(-1),
                                                                                       gu.reshape(-1))}
    v, F, on = _dirichlet0(kr, kc, kv, X.load(f), bd)
    keep = ~(on[kr] | on[kc]) | (kr == kc)
    return {"K": kv, "B": None if bool((v[keep] == 0).any()) else v[keep], "r": F,
            "u": _Direct(kr, kc, v, row).solve(F)}
