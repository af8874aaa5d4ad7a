"""The tile-marching passes give the same bits every time they run: the product, the smoothing
passes inside a solve at degrees 1 and 2 and the assembled vectors, on a mesh with several
tiles along every axis that start in the interior and several layers a tile.  (A slot of the
ring of node planes overwritten before a slow thread has read it, or an exchange read before it
is complete, shows as a result that varies.)  One run of each is compared with the assembled
operator and vectors.  GPU."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N = (48, 40, 56)
RUNS = 60


def _point():
    import hippymfem_b200 as hm

    mesh = hm.BoxMesh(N, (1.0, 0.8, 1.2))
    V = hm.Q2Space(mesh)
    bc = hm.DirichletBC(V)
    rng = np.random.default_rng(8)
    f = [torch.as_tensor(0.3 * rng.standard_normal(mesh.ndof), device=mesh.device) for _ in range(3)]
    prob = hm.PDEVariationalProblem([V, V, V], f=1.0, bc=bc, matrix_free_solves=True)
    quad = prob._quadrature([None, f[1], None], "jacobian")
    return hm, mesh, V, bc, f, quad


def _same_every_time(run, outs):
    run()
    first = [o.clone() for o in outs]
    for _ in range(RUNS):
        for o in outs:
            o.fill_(7.0)
        run()
        for o, w in zip(outs, first):
            assert torch.equal(o, w)
    return first


@pytest.mark.parametrize("prec,tol", [("HM_FP64", 1000 * 2.0 ** -53), ("HM_FP32", 1000 * 2.0 ** -24)])
def test_products(cuda, prec, tol):
    """Against the assembled block within 1000 roundings of |A| |x| (a bound of it: the largest
    row sum of |A| times the largest |x|)."""
    from hippymfem_b200 import MatrixFreeJacobian, _lib

    hm, mesh, V, bc, f, quad = _point()
    A = MatrixFreeJacobian(mesh, quad, bc.marker, getattr(_lib, prec), quad_precision=_lib.HM_FP64)
    y = V.vector()
    got = _same_every_time(lambda: A.mult(f[0], y), [y])[0]
    full = hm.PDEVariationalProblem([V, V, V], f=1.0, bc=bc)
    B, _ = full._jacobian([None, f[1], None])
    want = B.mult(f[0], V.vector())
    B.values.abs_()
    scale = B.mult(f[0].abs(), V.vector())
    assert bool(((got - want).abs() <= tol * scale).all())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("degree", [1, 2])
def test_smoothing_passes(cuda, degree, precision):
    from hippymfem_b200 import MatrixFreeJacobian, _lib
    from hippymfem_b200._lib import lib, ptr, stream_ptr
    from hippymfem_b200.sparse import Multigrid

    hm, mesh, V, bc, f, quad = _point()
    A = MatrixFreeJacobian(mesh, quad, bc.marker)
    mg = Multigrid(mesh, degree=degree, precision=precision).setup(A.jac, A.ess, A._diag)
    b = f[0].clone()
    bc.zero(b)
    x = V.vector()
    work = torch.empty(lib.hm_pcg_workspace_bytes(mesh.ndof) // 8 + 1, dtype=torch.float64, device=cuda)
    it, rr = ctypes.c_int(), ctypes.c_double()

    def run():
        x.zero_()
        rc = lib.hm_pcg_mg(mg._mg, ptr(b), ptr(x), 1e-30, 2, 2, ptr(work), ctypes.byref(it),
                           ctypes.byref(rr), stream_ptr())
        assert rc == _lib.HM_ERR_NOCONV

    _same_every_time(run, [x])


@pytest.mark.parametrize("slots", [(0, 1, 2), (1,), (2,)])
def test_vectors(cuda, slots):
    from hippymfem_b200 import _lib
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    hm, mesh, V, bc, f, quad = _point()
    out = {s: V.vector() for s in slots}
    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, len(slots))
    work = torch.empty(nbytes // 8, dtype=torch.float64, device=cuda)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)

    def run():
        check(lib.hm_lattice_vectors(mesh.handle, *(ptr(v) for v in f), None, 1.0, None,
                                     ptr(out.get(0)), ptr(out.get(1)), ptr(out.get(2)), 0, ptr(work),
                                     ptr(status), stream_ptr()))

    got = _same_every_time(run, [out[s] for s in slots])
    data = torch.empty(mesh.quad_bytes() // 8, dtype=torch.float64, device=cuda)
    check(lib.hm_lattice_quadrature(mesh.handle, *(ptr(v) for v in f), _lib.HM_FP64, ptr(data),
                                    ptr(status), stream_ptr()))
    want = [V.vector() for _ in range(3)]
    check(lib.hm_lattice_assemble(mesh.handle, ptr(data), _lib.HM_FP64, None, None, 1.0, None, None,
                                  None, None, *(ptr(v) for v in want), 0, stream_ptr()))
    assert int(status) == 0
    for s, g in zip(slots, got):
        assert float((g - want[s]).abs().max()) <= 1e-12 * float(want[s].abs().max())
