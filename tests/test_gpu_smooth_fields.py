"""Products and assembled vectors on smooth fields far from zero, against extended precision.

The operator annihilates constants, so its rounding has to follow the variation of the field
over an element and not its value: with a field of 1000 + O(1) on elements of edge 1/64 a
derivative that carried the rounding of the values would be wrong by 1e4 of the bound below.
The bound of a node is eps times 64 (the roundings on the way from a nodal value to an
assembled sum: one difference, 12 in the interpolation, 6 in derivative and weight, 27 + 15 in
the sums back, 3 more with their constants) times the sum of |weights| over its elements with
every gradient replaced by its largest possible value, 8 max |x_a - x_centre| / h.  GPU."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

K = 64.0
LD = np.longdouble
# several layers a tile; several tiles along every axis; odd and even rows
SIZES = [(3, 2, 9), (17, 12, 20), (30, 26, 28)]


def _tables():
    q = [LD(1) / 2 - np.sqrt(LD(15)) / 10, LD(1) / 2, LD(1) / 2 + np.sqrt(LD(15)) / 10]
    B = np.array([[(1 - t) * (1 - 2 * t), 4 * t * (1 - t), t * (2 * t - 1)] for t in q])
    G = np.array([[4 * t - 3, 4 - 8 * t, 4 * t - 1] for t in q])
    w = np.array([LD(5) / 18, LD(8) / 18, LD(5) / 18])
    return B, G, w


def _to_points(M, x):
    """(ne, z, y, x) with one table an axis (x, y, z)."""
    for ax, t in ((3, M[0]), (2, M[1]), (1, M[2])):
        x = np.moveaxis(np.tensordot(x, t, axes=([ax], [1])), -1, ax)
    return x


def _to_nodes(M, x):
    return _to_points([t.T for t in M], x)


class _Exact:
    def __init__(self, n, L, m, u, p):
        self.n, self.h = n, [LD(s) / v for s, v in zip(L, n)]
        self.N = [2 * v + 1 for v in n]
        B, G, w = _tables()
        self.B, self.G = B, G
        vol = self.h[0] * self.h[1] * self.h[2]
        W = vol * w[:, None, None] * w[None, :, None] * w[None, None, :]
        self.D = W[None] * np.exp(_to_points([B] * 3, self.elements(m)))
        self.u, self.p = (self.elements(v) for v in (u, p))

    def elements(self, v):
        a = np.asarray(v, dtype=LD).reshape(self.N[2], self.N[1], self.N[0])
        out = np.empty((self.n[2], self.n[1], self.n[0], 3, 3, 3), dtype=LD)
        for k in range(3):
            for j in range(3):
                for i in range(3):
                    out[..., k, j, i] = a[k:k + 2 * self.n[2] - 1:2, j:j + 2 * self.n[1] - 1:2,
                                          i:i + 2 * self.n[0] - 1:2]
        return out.reshape(-1, 3, 3, 3)

    def assemble(self, y):
        y = y.reshape(self.n[2], self.n[1], self.n[0], 3, 3, 3)
        out = np.zeros((self.N[2], self.N[1], self.N[0]), dtype=LD)
        for k in range(3):
            for j in range(3):
                for i in range(3):
                    out[k:k + 2 * self.n[2] - 1:2, j:j + 2 * self.n[1] - 1:2,
                        i:i + 2 * self.n[0] - 1:2] += y[..., k, j, i]
        return out.reshape(-1)

    def _axes(self):
        for ax in range(3):
            M = [self.B] * 3
            M[ax] = self.G / self.h[ax]
            yield M

    def gradient(self, x):
        return [_to_points(M, x) for M in self._axes()]

    def product(self, x):
        return self.assemble(sum(_to_nodes(M, self.D * g) for M, g in zip(self._axes(), self.gradient(x))))

    def most(self, x):
        """The largest gradient component an element's values allow."""
        return 8 * np.abs(x - x[:, 1:2, 1:2, 1:2]).max(axis=(1, 2, 3), keepdims=True) / min(self.h)

    def product_bound(self, x):
        return self.assemble(sum(_to_nodes([np.abs(t) for t in M], self.D * self.most(x)) for M in self._axes()))

    def parameter(self):
        g, r = self.gradient(self.u), self.gradient(self.p)
        return self.assemble(_to_nodes([self.B] * 3, self.D * sum(a * b for a, b in zip(g, r))))

    def parameter_bound(self):
        return self.assemble(_to_nodes([np.abs(self.B)] * 3, 3 * self.D * self.most(self.u) * self.most(self.p)))


def _case(n):
    import hippymfem_b200 as hm

    L = tuple(v / 64.0 for v in n)
    mesh = hm.BoxMesh(n, L)
    x, y, z = mesh.node_coords().T
    u = 1000.0 + np.sin(3 * x + 1) * np.cos(2 * y) * np.exp(z)
    p = -700.0 + np.cos(2 * x + y) * np.sin(3 * z + 0.4)
    u, p = (v.astype(np.float32).astype(np.float64) for v in (u, p))   # exact in both precisions
    m = 0.3 * np.cos(4 * x + 3 * y - 2 * z)
    return mesh, _Exact(n, L, m, u, p), u, m, p


@pytest.mark.parametrize("n", SIZES)
def test_products(cuda, n):
    from hippymfem_b200 import _lib
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr
    from hippymfem_b200.sparse import MatrixFreeJacobian

    mesh, ex, u, m, p = _case(n)
    want, bound = ex.product(ex.u), ex.product_bound(ex.u)
    U, M = torch.as_tensor(u, device=cuda), torch.as_tensor(m, device=cuda)
    quad = torch.empty(mesh.quad_bytes() // 8 + 1, dtype=torch.float64, device=cuda)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    check(lib.hm_lattice_quadrature(mesh.handle, ptr(U), ptr(M), ptr(U), _lib.HM_FP64, ptr(quad),
                                    ptr(status), stream_ptr()))
    for prec, eps in ((_lib.HM_FP64, 2.0 ** -53), (_lib.HM_FP32, 2.0 ** -24)):
        A = MatrixFreeJacobian(mesh, quad, None, prec, quad_precision=_lib.HM_FP64)
        y = torch.full_like(U, 7.0)
        A.mult(U, y)
        err = np.abs(y.cpu().numpy().astype(LD) - want)
        assert (err <= K * eps * bound).all(), (prec, float((err / (eps * bound)).max()))


@pytest.mark.parametrize("n", SIZES)
def test_vectors(cuda, n):
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    mesh, ex, u, m, p = _case(n)
    want = [ex.product(ex.p), ex.parameter(), ex.product(ex.u)]
    bound = [ex.product_bound(ex.p), ex.parameter_bound(), ex.product_bound(ex.u)]
    f = [torch.as_tensor(v, device=cuda) for v in (u, m, p)]
    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, 3)
    work = torch.empty(nbytes // 8, dtype=torch.float64, device=cuda)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    out = [torch.empty_like(f[0]) for _ in range(3)]
    check(lib.hm_lattice_vectors(mesh.handle, *(ptr(v) for v in f), None, 0.0, None,
                                 *(ptr(v) for v in out), 0, ptr(work), ptr(status), stream_ptr()))
    for s in range(3):
        err = np.abs(out[s].cpu().numpy().astype(LD) - want[s])
        assert (err <= K * 2.0 ** -53 * bound[s]).all(), (s, float((err / (2.0 ** -53 * bound[s])).max()))
