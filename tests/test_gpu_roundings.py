"""Roundings that the kernels write out, against the same operations in exact
rational arithmetic, each rounded once: every kernel form (L2 prefetch, run
form, plain) then gives these bits.
"""
from fractions import Fraction as Q

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Q(a) * Q(b) + Q(c))   # a quotient of integers rounds to nearest even


def _mesh(cg, kind, order):
    """A mesh, and its geometry and incidences in the internal numbering."""
    mesh = cg.Mesh.jittered(7, 5, 4, jitter=0.25, seed=6, permute=True, order=order) if kind == "jitter" else \
        cg.Mesh.structgen(34, 3, 2, order=order)
    cells, faces = mesh.numbering()
    geo = mesh.geometry()
    g = {k: geo[k][cells if k.startswith("cell") else faces] for k in
         ("faceNorm", "faceLambda", "faceCenter", "cellCenter", "cellVolume")}
    xadj, code, other = (a.tolist() for a in mesh.incidences())
    g["inc"] = [[(f >> 1, f & 1, o) for f, o in zip(code[xadj[c]:xadj[c + 1]], other[xadj[c]:xadj[c + 1]])]
                for c in range(mesh.nCells)]
    return mesh, g


MESHES = [("jitter", 0), ("jitter", 1), ("struct", 2)]   # plain kernels, full lists, run form


@pytest.mark.parametrize("sign", [0, 1])
@pytest.mark.parametrize("f64", [True, False])
@pytest.mark.parametrize("kind,order", MESHES)
def test_gradient_adjoint_roundings(cg, gpu, kind, order, f64, sign):
    """dev_gradient_adjoint: gbar . S summed y, x, z by FMAs; with the
    reference's sign the other cell's share joins this cell's in one FMA with
    1 / V, with the switched sign it rounds by itself; FP64 throughout."""
    import torch
    mesh, geo = _mesh(cg, kind, order)
    t = np.float64 if f64 else np.float32
    nC, nB = mesh.nCells, mesh.nBoundaries
    gbar = np.random.default_rng(1).standard_normal((3, nC)).astype(t)
    S, lam = geo["faceNorm"].astype(t).astype(float).tolist(), geo["faceLambda"].astype(t).astype(float).tolist()
    iv = (1.0 / geo["cellVolume"]).tolist()
    g = gbar.astype(float).T.tolist()
    dot = lambda a, s: fma(a[2], s[2], fma(a[0], s[0], a[1] * s[1]))
    want, wantB = np.empty(nC, t), np.empty(nB, t)
    for c in range(nC):
        h, pb = [x * iv[c] for x in g[c]], 0.0
        for f, isN, o in geo["inc"][c]:
            own = dot(h, S[f])
            if o < 0:
                wantB[-1 - o] = own
                continue
            gS = dot(g[o], S[f])
            both = fma(gS, iv[o], own) if sign == 0 else gS * iv[o] - own if isN else own - gS * iv[o]
            pb = fma(lam[f] if isN else 1.0 - lam[f], both, pb)
        want[c] = pb
    dev = lambda a: torch.from_numpy(a).to(gpu)
    phi, phiB = dev(np.full(nC, np.nan, t)), dev(np.full(nB, np.nan, t))
    cg.dev_gradient_adjoint(mesh, cg.PREC_F64 if f64 else cg.PREC_F32C, dev(gbar), phi, phiB, sign_mode=sign,
                            stream=torch.cuda.current_stream())
    assert np.array_equal(phi.cpu().numpy(), want)
    assert np.array_equal(phiB.cpu().numpy(), wantB)


def f32(q):
    """The float nearest to a rational, ties to even."""
    x = np.float32(float(q))
    return min((np.nextafter(x, np.float32(-np.inf)), x, np.nextafter(x, np.float32(np.inf))),
               key=lambda y: (abs(Q(float(y)) - q), int(y.view(np.int32)) & 1))


def fmaf(a, b, c):
    return f32(Q(float(a)) * Q(float(b)) + Q(float(c)))


class Sum:
    """A compensated sum of products as the FP32 kernels keep it."""
    def __init__(self):
        self.s = self.e = np.float32(0)

    def add(self, a, b):
        t = self.s + fmaf(a, b, 0)
        nbp = self.s - t
        ar = self.s - (t + nbp)
        self.e = self.e + (ar + fmaf(a, b, nbp))
        self.s = t


@pytest.mark.parametrize("sign", [0, 1])
@pytest.mark.parametrize("kind,order", MESHES[:2])
def test_corrected_gradient_roundings_f32(cg, gpu, kind, order, sign):
    """dev_gradient in FP32 with one non-orthogonal correction: the three
    products of gradient and distance summed y, x, z by FMAs, then added to
    the interpolated value."""
    import torch
    mesh, geo = _mesh(cg, kind, order)
    nC, nB = mesh.nCells, mesh.nBoundaries
    r = np.random.default_rng(2)
    phi, phiB = r.standard_normal(nC).astype(np.float32), r.standard_normal(nB).astype(np.float32)
    S, lam, xf, xc = (geo[k].astype(np.float32) for k in ("faceNorm", "faceLambda", "faceCenter", "cellCenter"))
    fact = 1.0 / geo["cellVolume"]
    one, grad = np.float32(1), None
    for _ in range(2):
        to = np.empty((nC, 3), np.float32)
        for c in range(nC):
            sums = [Sum() for _ in range(3)]
            for f, isN, o in geo["inc"][c]:
                if o < 0:
                    phif = phiB[-1 - o]
                else:
                    n, p = lam[f], one - lam[f]
                    N, P = (c, o) if isN else (o, c)
                    wc, wo = (n, p) if isN else (p, n)
                    phif = fmaf(wc, phi[c], wo * phi[o])
                    if grad is not None:
                        d = [xf[f, k] - fmaf(n, xc[N, k], p * xc[P, k]) for k in range(3)]
                        a = [fmaf(n, grad[N, k], p * grad[P, k]) for k in range(3)]
                        phif = phif + fmaf(a[2], d[2], fmaf(a[0], d[0], a[1] * d[1]))
                for k in range(3):
                    sums[k].add(-phif if sign and isN else phif, S[f, k])
            to[c] = [np.float32((float(x.s) + float(x.e)) * fact[c]) for x in sums]
        grad = to
    dev = lambda a: torch.from_numpy(a).to(gpu)
    g = torch.empty(3, nC, device=gpu)
    cg.dev_gradient(mesh, cg.PREC_F32C, dev(phi), dev(phiB), g, nGradient=2, sign_mode=sign,
                    stream=torch.cuda.current_stream())
    assert np.array_equal(g.cpu().numpy().T, grad)
