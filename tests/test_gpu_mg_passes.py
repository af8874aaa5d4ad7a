"""The multigrid cycle's fused passes and its one-launch coarse levels against the
step-by-step, level-by-level cycle, at every smoothing degree and on meshes that coarsen
well, partly or not at all.  GPU."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-13, "fp32": 2e-5}      # rounding through one cycle, relative to its norm

MESHES = [((4, 4, 4), (1.0, 1.0, 1.0)), ((6, 5, 7), (1.0, 0.8, 1.1)), ((10, 10, 14), (0.7, 0.7, 1.0)),
          ((24, 16, 20), (1.0, 0.6, 0.9)), ((2, 2, 40), (0.1, 0.1, 1.5)), ((40, 36, 44), (1.0, 1.0, 1.0))]


def _point(n, L, degree, precision, coarse_degree=24):
    from hippymfem_b200 import BoxMesh, DirichletBC, PDEVariationalProblem, Q2Space
    from hippymfem_b200.sparse import Multigrid
    from hippymfem_b200.synthetic import log_conductivity

    mesh = BoxMesh(n, L)
    V = Q2Space(mesh)
    prob = PDEVariationalProblem([V, V, V], bc=DirichletBC(V), matrix_free_solves=True)
    m = V.project(lambda x: log_conductivity(x, seed=2, sigma=0.4))
    A, _ = prob._jacobian([None, m, None])
    mg = Multigrid(mesh, degree, coarse_degree, precision=precision).setup(A.jac, A.ess, A._diag)
    r = torch.as_tensor(np.random.default_rng(9).standard_normal(mesh.ndof), device=mesh.device)
    return mesh, V, prob, A, mg, r.masked_fill_(prob.bc0.mask, 0.0)


def _one_iteration(mesh, V, mg, r):
    """One CG iteration from zero: x = alpha V(r), through the cycle the solves use."""
    from hippymfem_b200._lib import lib, ptr, stream_ptr

    work = torch.empty(lib.hm_pcg_workspace_bytes(mesh.ndof) // 8 + 1, dtype=torch.float64,
                       device=mesh.device)
    x = V.vector()
    it, rr = ctypes.c_int(), ctypes.c_double()
    rc = lib.hm_pcg_mg(mg._mg, ptr(r), ptr(x), 1e-300, 1, 1, ptr(work), ctypes.byref(it),
                       ctypes.byref(rr), stream_ptr())
    assert rc in (0, 5) and it.value == 1
    return x


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("n,L", MESHES)
def test_fused_passes_are_the_step_by_step_cycle(cuda, n, L, degree, precision):
    mesh, V, prob, A, mg, r = _point(n, L, degree, precision)
    mg.set_tail_nodes(0).set_fused(False)
    ref_x, ref_z = _one_iteration(mesh, V, mg, r), mg.apply(r, V.vector())
    for tail in (0, 150, 5000, 10 ** 9):
        for fused in (True, False):
            mg.set_tail_nodes(tail).set_fused(fused)
            x, z = _one_iteration(mesh, V, mg, r), mg.apply(r, V.vector())
            assert float((x - ref_x).norm()) <= TOL[precision] * float(ref_x.norm()), (tail, fused)
            assert float((z - ref_z).norm()) <= TOL[precision] * float(ref_z.norm()), (tail, fused)


@pytest.mark.parametrize("coarse_degree", [1, 2, 5])
def test_coarse_solves_of_small_degree(cuda, coarse_degree):
    """A coarsest level without an exact solve (5 x 5 x 7 elements), whatever its degree."""
    mesh, V, prob, A, mg, r = _point((10, 10, 14), (0.7, 0.7, 1.0), 1, "fp64", coarse_degree)
    ref = mg.set_tail_nodes(0).set_fused(False).apply(r, V.vector())
    for tail, fused in ((0, True), (5000, True), (5000, False)):
        z = mg.set_tail_nodes(tail).set_fused(fused).apply(r, V.vector())
        assert float((z - ref).norm()) <= TOL["fp64"] * float(ref.norm())
