"""A tile-marching pass that gives up waiting for its staged data is reported: by the caller's
status word (vectors), by the return code (every kind of solve) and by the library's own
status word (the product alone).  The waits are counted as run out on request; the copies
themselves land.  GPU."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# one tile; several along every axis; several layers a tile
SIZES = [(4, 4, 4), (20, 16, 24), (40, 12, 32)]


def _device_status():
    from hippymfem_b200._lib import check, lib

    st = np.zeros(1, np.uint32)
    check(lib.hm_device_status(st.ctypes.data, 1))
    return int(st[0])


def _lib_timeout():
    from hippymfem_b200 import _lib

    return _lib.HM_STATUS_TIMEOUT


class _GivingUp:
    """The lattice's waits count as run out inside the block."""

    def __init__(self, mesh):
        self.mesh = mesh

    def __enter__(self):
        from hippymfem_b200._lib import check, lib

        check(lib.hm_lattice_fail_waits(self.mesh.handle, 1))

    def __exit__(self, *a):
        from hippymfem_b200._lib import check, lib

        check(lib.hm_lattice_fail_waits(self.mesh.handle, 0))


def _setup(n):
    import hippymfem_b200 as hm

    mesh = hm.BoxMesh(n)
    V = hm.Q2Space(mesh)
    bc = hm.DirichletBC(V)
    rng = np.random.default_rng(3)
    fields = [torch.as_tensor(0.3 * rng.standard_normal(mesh.ndof), device=mesh.device) for _ in range(3)]
    return hm, mesh, V, bc, fields


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("slots", [(0,), (1,), (2,), (0, 1, 2)])
def test_vectors_set_the_callers_status(cuda, n, slots):
    from hippymfem_b200 import _lib
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    hm, mesh, V, bc, f = _setup(n)
    check(lib.hm_lattice_set_slab(mesh.handle, 1))       # the tile-marching passes at every size
    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, 3)
    work = torch.empty(nbytes // 8, dtype=torch.float64, device=cuda)
    status = torch.zeros(1, dtype=torch.int32, device=cuda)
    out = {s: V.vector() for s in slots}

    def call():
        check(lib.hm_lattice_vectors(mesh.handle, *(ptr(v) for v in f), None, 1.0, None,
                                     ptr(out.get(0)), ptr(out.get(1)), ptr(out.get(2)), 0, ptr(work),
                                     ptr(status), stream_ptr()))

    _device_status()
    call()
    assert int(status) == 0 and _device_status() == 0
    want = {s: v.clone() for s, v in out.items()}
    prob = hm.PDEVariationalProblem([V, V, V], f=1.0, bc=bc)
    with _GivingUp(mesh):
        call()
        assert int(status) == _lib.HM_STATUS_TIMEOUT
        assert _device_status() & _lib.HM_STATUS_TIMEOUT
        with pytest.raises(RuntimeError, match="gave up"):
            prob.evalGradientParameter(f, V.vector())
    _device_status()
    status.zero_()
    call()
    assert int(status) == 0 and _device_status() == 0
    assert all(torch.equal(out[s], want[s]) for s in slots)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("prec", ["HM_FP64", "HM_FP32"])
def test_a_product_alone_sets_the_librarys_status(cuda, n, prec):
    from hippymfem_b200 import _lib
    from hippymfem_b200.sparse import MatrixFreeJacobian

    hm, mesh, V, bc, f = _setup(n)
    prob = hm.PDEVariationalProblem([V, V, V], f=1.0, bc=bc, matrix_free_solves=True)
    quad = prob._quadrature([None, f[1], None], "jacobian")
    A = MatrixFreeJacobian(mesh, quad, bc.marker, getattr(_lib, prec), quad_precision=_lib.HM_FP64)
    y, z = V.vector(), V.vector()
    _device_status()
    A.mult(f[0], y)
    assert _device_status() == 0
    with _GivingUp(mesh):
        A.mult(f[0], z)
        assert _device_status() & _lib.HM_STATUS_TIMEOUT
    A.mult(f[0], z)
    assert _device_status() == 0 and torch.equal(y, z)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["jacobi", "mixed", "mg", "mg-fp32", "plan", "plan-mixed", "group"])
def test_a_solve_whose_operator_gave_up_is_an_error(cuda, n, kind):
    """Captured batches included (a stream of its own); a solver made before answers as before
    afterwards."""
    from hippymfem_b200.sparse import (MatrixFreeJacobian, MGPCGSolver, MixedPCGSolver, PCGSolver,
                                       SolveGroup, SolvePlan)

    hm, mesh, V, bc, f = _setup(n)
    prob = hm.PDEVariationalProblem([V, V, V], f=1.0, bc=bc, matrix_free_solves=True)
    quad = prob._quadrature([None, f[1], None], "jacobian")
    A = MatrixFreeJacobian(mesh, quad, bc.marker)
    b = f[0].clone()
    bc.zero(b)
    tol = dict(rel_tolerance=1e-8)

    def make():
        if kind == "jacobi":
            return PCGSolver(A, **tol)
        if kind == "mixed":
            return MixedPCGSolver(A, quad, **tol)
        if kind == "plan":
            return SolvePlan(mesh, bc.marker, multigrid=True, **tol).set_point(quad)
        if kind == "plan-mixed":
            return SolvePlan(mesh, bc.marker, precision="mixed", **tol).set_point(quad)
        if kind == "group":
            return SolveGroup([SolvePlan(mesh, bc.marker, multigrid=k == 0, **tol).set_point(quad)
                               for k in range(2)])
        return MGPCGSolver(A, mg_precision="fp32" if kind == "mg-fp32" else "fp64", **tol)

    def solve(s):
        out = [V.vector(), V.vector()]
        torch.cuda.synchronize()
        with torch.cuda.stream(torch.cuda.Stream()):
            if kind == "group":
                s.solve(out, [b, b])
            else:
                s.solve(out[0], b)
        torch.cuda.synchronize()
        return out

    good = make()
    want = solve(good)
    assert _device_status() == 0
    with _GivingUp(mesh):
        bad = make()
        with pytest.raises(RuntimeError, match="CUDA"):
            solve(bad)
    assert _device_status() & _lib_timeout()
    got = solve(good)
    assert _device_status() == 0
    assert all(torch.equal(a, w) for a, w in zip(got, want))
