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
