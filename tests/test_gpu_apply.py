"""The matrix-free Jacobian apply (``hm_lattice_apply_A``) against the oracle's assembled
block, at the edges of its tiling: meshes of one element, thinner and longer than a tile,
several tiles and layers in every direction, storage and vectors that are only 8-byte
aligned (4-byte in FP32), with and without Dirichlet nodes; and independent of how the
mesh is cut.  GPU."""

import numpy as np
import pytest
import torch

from oracle import q2

pytestmark = pytest.mark.gpu

# an entry is a sum of at most 125 products formed in under 1000 roundings
TOL64 = 1000 * 2.0 ** -53      # relative to (|A| |x|) per node
TOL32 = 1000 * 2.0 ** -24

SIZES = [(1, 1, 1), (1, 5, 2), (2, 1, 1), (3, 4, 5), (1, 1, 19), (34, 2, 3), (66, 3, 1),
         (3, 70, 2), (13, 9, 11), (16, 17, 6), (26, 5, 24)]


def _operator(n, L, seed, precision, offset, ess):
    """The operator's storage, `offset` entries into its allocation, and the oracle's
    matrix."""
    from hippymfem_b200 import BoxMesh, _lib
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    mesh = BoxMesh(n, L)
    mo = q2.Lattice(n, L)
    rng = np.random.default_rng(seed)
    m = 0.4 * rng.standard_normal(mo.ndof)
    z = np.zeros(mo.ndof)
    mask = np.zeros(mo.ndof, bool)
    if ess:
        mask[mo.boundary_dofs()] = True
    E = mo.edofs()
    pat = q2.build_tables(E, E, mo.ndof, mo.ndof, True)
    A = q2.csr(pat, q2.assemble_block("A", pat, q2.element_blocks(mo, E, z, m, z, ("A",))["A"],
                                      mask), (mo.ndof,) * 2)
    dev = mesh.device
    dm, dz = torch.as_tensor(m, device=dev), torch.zeros(mo.ndof, dtype=torch.float64, device=dev)
    quad = torch.empty(mesh.quad_bytes() // 8, dtype=torch.float64, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    check(lib.hm_lattice_quadrature(mesh.handle, ptr(dz), ptr(dm), ptr(dz), _lib.HM_FP64, ptr(quad),
                                    ptr(status), stream_ptr()))
    size = 4 if precision == _lib.HM_FP32 else 8
    nbytes = lib.hm_lattice_jacobian_bytes(mesh.handle, precision)
    store = torch.full((nbytes // size + 8,), float("nan"),
                       dtype=torch.float32 if size == 4 else torch.float64, device=dev)
    jac = store[offset:offset + nbytes // size]
    check(lib.hm_lattice_jacobian_prepare(mesh.handle, ptr(quad), _lib.HM_FP64, ptr(jac), precision,
                                          stream_ptr()))
    return mesh, A, jac, mask


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_apply_matches_the_oracle(cuda, n, precision):
    from hippymfem_b200 import _lib
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    assert (_lib.HM_FP64, _lib.HM_FP32) == (0, 1)
    L = tuple(0.1 * v * s for v, s in zip(n, (1.0, 0.8, 1.3)))
    for offset, ess in ((0, True), (1, True), (0, False)):
        mesh, A, jac, mask = _operator(n, L, 3, precision, offset, ess)
        rng = np.random.default_rng(4)
        x = rng.standard_normal(mesh.ndof)           # not zero on the Dirichlet nodes
        store = torch.full((mesh.ndof + 2,), float("nan"), dtype=torch.float64, device=cuda)
        dx = store[offset:offset + mesh.ndof]
        dx.copy_(torch.as_tensor(x))
        y = torch.full((mesh.ndof + 2,), 7.0, dtype=torch.float64, device=cuda)
        marker = torch.as_tensor(mask.astype(np.uint8), device=cuda) if ess else None
        check(lib.hm_lattice_apply_A(mesh.handle, ptr(jac), precision, ptr(marker), ptr(dx),
                                     ptr(y[1:-1]), stream_ptr()))
        got = y.cpu().numpy()
        assert got[0] == 7.0 and got[-1] == 7.0      # nothing written beside y
        ref, scale = A @ x, abs(A) @ np.abs(x)
        tol = TOL32 if precision else TOL64
        assert np.all(np.abs(got[1:-1] - ref) <= tol * scale), (offset, ess)


def test_apply_does_not_depend_on_the_cut(cuda):
    """The owned planes of z-slabs (one element layer of halo below) equal the whole
    lattice's rows bit for bit, whatever tiling each lattice takes."""
    from hippymfem_b200 import BoxMesh, MatrixFreeJacobian, _lib
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    n = (9, 14, 23)
    h = 0.125
    rng = np.random.default_rng(5)

    def product(mesh, m, x):
        quad = torch.empty(mesh.quad_bytes() // 8, dtype=torch.float64, device=cuda)
        status = torch.zeros(1, dtype=torch.int32, device=cuda)
        z = torch.zeros_like(m)
        check(lib.hm_lattice_quadrature(mesh.handle, ptr(z), ptr(m), ptr(z), _lib.HM_FP64,
                                        ptr(quad), ptr(status), stream_ptr()))
        y = torch.empty_like(x)
        return MatrixFreeJacobian(mesh, quad, None).mult(x, y)

    mesh = BoxMesh(n, tuple(v * h for v in n))
    m = torch.as_tensor(0.3 * rng.standard_normal(mesh.ndof), device=cuda)
    x = torch.as_tensor(rng.standard_normal(mesh.ndof), device=cuda)
    y = product(mesh, m, x)
    plane = mesh.N[0] * mesh.N[1]
    for e0, e1 in ((0, 5), (4, 13), (12, 23)):       # elements, the halo layer included
        part = BoxMesh((n[0], n[1], e1 - e0), (n[0] * h, n[1] * h, (e1 - e0) * h))
        s = slice(2 * e0 * plane, (2 * e1 + 1) * plane)
        yp = product(part, m[s].clone(), x[s].clone())
        lo = 0 if e0 == 0 else 2 * plane             # planes whose elements are all here
        hi = part.ndof if e1 == n[2] else part.ndof - plane
        assert torch.equal(yp[lo:hi], y[s][lo:hi])
