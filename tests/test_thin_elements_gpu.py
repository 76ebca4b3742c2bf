"""COO entries in thin oblique triangles (height 2^-13 of the width) in every numbering of the vertices, entry by
entry: each is a product of the gradients of its own two basis functions, whatever the gradients of the
element's other vertices are.

Reference: the same sums in extended precision.  The coordinates make the gradients of the vertices exact;
the element's area, a factor of all its entries, is fitted to the output.  Bar: an entry is at most 32
roundings (of 2^-53) off, relative to the product of the lengths that its factors have before any
cancellation (basis factors, products and weights are some 12; the fit is better than one), and an output
of the backward operators, a sum over an element's 36 entries, at most 64.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from adfem_gpu import synth

pytestmark = pytest.mark.gpu
LD = np.longdouble
EPS = 2.0 ** -53


def thin_mesh():
    m, n = 9, 7
    coords, elems = synth.jittered_square(m, n=n, jitter=0.0)
    i, j = np.round(coords * [m, n]).T
    coords = np.stack([i + j * 2.0 ** -13, j * 2.0 ** -13], axis=1)
    e = np.arange(len(elems))
    elems = np.stack([elems[e, (e // 2 + k) % 3] for k in range(3)], axis=1)
    x, y = np.moveaxis(coords[elems - 1], 2, 0)
    neg = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) < (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
    elems[neg, :2] = elems[neg, 1::-1]  # (as the mesh itself orders them: counterclockwise)
    return coords, elems


def gradients(coords, elems):
    """gradients (ne, 3, 2) of the barycentric coordinates and areas"""
    p = coords.astype(LD)[elems - 1]
    x, y = p[..., 0], p[..., 1]
    det = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
    j, k = [1, 2, 0], [2, 0, 1]
    g = np.stack([y[:, j] - y[:, k], x[:, k] - x[:, j]], axis=-1) / det[:, None, None]
    return g, abs(det) / 2


def p2_points(g):
    """gradients at the six points of the order-4 rule (ne, 6 points, 6 functions, 2), their lengths
    before cancellation, and the weights (of an area of 1)"""
    r = LD(8) - np.sqrt(LD(10))
    s = np.sqrt(LD(38) - 44 * np.sqrt(LD(2) / 5))
    a = [(r - s) / 18, (r + s) / 18]
    w = [(620 - np.sqrt(LD(213125) - 53320 * np.sqrt(LD(10)))) / 3720,
         (620 + np.sqrt(LD(213125) - 53320 * np.sqrt(LD(10)))) / 3720]
    out, mag, ws = [], [], []
    for o in range(2):
        for xi, eta in ((a[o], a[o]), (a[o], 1 - 2 * a[o]), (1 - 2 * a[o], a[o])):
            l = [1 - xi - eta, xi, eta]
            T = np.zeros((6, 3), LD)
            for i in range(3):
                T[i, i] = 4 * l[i] - 1
                T[3 + i, i], T[3 + i, (i + 1) % 3] = 4 * l[(i + 1) % 3], 4 * l[i]
            out.append(np.einsum("fc,ecd->efd", T, g))
            mag.append(np.einsum("fc,ec->ef", abs(T), np.sqrt((g * g).sum(-1))))
            ws.append(w[o])
    return np.stack(out, 1), np.stack(mag, 1), np.array(ws)


def worst(got, want, scale, area=None):
    """largest error in roundings, and the factors by which the elements' areas differ"""
    got = got.cpu().numpy() if hasattr(got, "cpu") else got
    got, ne = got.reshape(want.shape).astype(LD), len(want)
    if area is None:
        area = (got * want).reshape(ne, -1).sum(1) / (want * want).reshape(ne, -1).sum(1)
    f = area.reshape((ne,) + (1,) * (want.ndim - 1))
    return float(np.max(np.abs(got - f * want) / scale)) / EPS, area


def test_elasticity(gpulib):
    from adfem_gpu import system as S

    coords, elems = thin_mesh()
    g, area = gradients(coords, elems)
    ne = len(elems)
    M = gpulib.Mesh(coords, elems)
    rng = np.random.default_rng(5)
    D = rng.standard_normal((ne, 3, 3, 3))
    G = rng.standard_normal((ne, 3, 6, 6))
    B = np.zeros((ne, 3, 6), LD)
    B[:, 0, :3], B[:, 1, 3:], B[:, 2, :3], B[:, 2, 3:] = g[..., 0], g[..., 1], g[..., 1], g[..., 0]
    w = (area / 3)[:, None, None, None]
    h = np.sqrt((g * g).sum(-1))
    hh = np.concatenate([h, h], 1)
    _, vv = S.stiffness_coo(M, torch.tensor(D.reshape(-1), device="cuda"))
    want = np.einsum("epl,ekpq,eqc->eklc", B, D.astype(LD), B) * w
    scale = hh[:, None, :, None] * hh[:, None, None, :] * abs(D).sum((2, 3))[..., None, None] * w
    err, area = worst(vv, want, scale)
    assert err < 32
    gD = S.stiffness_coo_backward(M, torch.tensor(G.reshape(-1), device="cuda"))
    want = np.einsum("epl,eklc,eqc->ekpq", B, G.astype(LD), B) * w
    scale = np.einsum("epl,eklc,eqc->ekpq", abs(B), abs(G).astype(LD), abs(B)) * w
    assert worst(gD, want, scale, area)[0] < 64


def test_p2_laplace_coo(gpulib):
    from adfem_gpu import system as S

    coords, elems = thin_mesh()
    g, area = gradients(coords, elems)
    N, mag, ws = p2_points(g)
    w = ws[None, :] * area[:, None]
    M = gpulib.Mesh(coords, elems, degree=2)
    ne = len(N)
    rng = np.random.default_rng(6)
    kappa = 1 + rng.random((ne, 6))
    G = rng.standard_normal((ne, 6, 6, 6))
    _, vv = S.laplace_coo(M, torch.tensor(kappa.reshape(-1), device="cuda"))
    want = np.einsum("ekpd,ekqd->ekpq", N, N) * (w * kappa)[..., None, None]
    scale = mag[..., :, None] * mag[..., None, :] * (w * kappa)[..., None, None]
    err, area = worst(vv, want, scale)
    assert err < 32
    gk = S.laplace_coo_backward(M, torch.tensor(G.reshape(-1), device="cuda"))
    want = np.einsum("ekpd,ekpq,ekqd->ek", N, G.astype(LD), N) * w
    scale = np.einsum("ekp,ekpq,ekq->ek", mag, abs(G).astype(LD), mag) * w
    assert worst(gk, want, scale, area)[0] < 64
