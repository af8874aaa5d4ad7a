"""The two routes of ``hm_lattice_vectors`` on either side of the sizes where the choice changes
(14^3 elements for one vector, 12^3 for two): the same vectors, and on a lattice declared a slab
the same bits whatever the cut.  GPU."""

import itertools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-12      # relative to the largest entry, as the other FP64 parity tests


def _vectors(mesh, f, slots, mhat=None, marker=None, zero=0):
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, len(slots))
    work = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=mesh.device)
    status = torch.zeros(1, dtype=torch.int32, device=mesh.device)
    out = {s: torch.full_like(f[0], 7.0) for s in slots}
    check(lib.hm_lattice_vectors(mesh.handle, *(ptr(v) for v in f), ptr(mhat), 1.3, ptr(marker),
                                 ptr(out.get(0)), ptr(out.get(1)), ptr(out.get(2)), zero, ptr(work),
                                 ptr(status), stream_ptr()))
    assert int(status) == 0
    return out


def _fields(mesh, seed):
    rng = np.random.default_rng(seed)
    return [torch.as_tensor(0.4 * rng.standard_normal(mesh.ndof), device=mesh.device) for _ in range(4)]


@pytest.mark.parametrize("n", [(1, 1, 1), (12, 12, 12), (19, 7, 13), (14, 14, 14), (61, 5, 9), (15, 14, 14)])
def test_the_routes_agree(cuda, n):
    import hippymfem_b200 as hm
    from hippymfem_b200._lib import check, lib

    L = tuple(0.1 * v for v in n)
    mesh, slab = hm.BoxMesh(n, L), hm.BoxMesh(n, L)
    check(lib.hm_lattice_set_slab(slab.handle, 1))
    marker = hm.DirichletBC(hm.Q2Space(mesh)).marker
    f = _fields(mesh, 1)
    for k in (1, 2, 3):
        for slots in itertools.combinations((0, 1, 2), k):
            for mhat, mark, zero in ((None, None, 0), (None, marker, 1), (f[3], marker, 1)):
                a = _vectors(mesh, f[:3], slots, mhat, mark, zero)
                b = _vectors(slab, f[:3], slots, mhat, mark, zero)
                for s in slots:
                    err = float((a[s] - b[s]).abs().max())
                    assert err <= TOL * float(b[s].abs().max()), (slots, s, err)


@pytest.mark.parametrize("slots", [(0,), (1,), (2,), (0, 2), (0, 1, 2)])
def test_slabs_give_the_bits_of_the_mesh(cuda, slots):
    """Element layers 0-13, 6-19 and 11-29 of a mesh of 30 (edges that are powers of two, so that
    every lattice has the same ones): the nodes whose elements all lie in the slab."""
    import hippymfem_b200 as hm
    from hippymfem_b200._lib import check, lib

    nx, ny, nz, h = 9, 10, 30, 0.0625
    mesh = hm.BoxMesh((nx, ny, nz), (nx * h, ny * h, nz * h))
    f = _fields(mesh, 2)
    check(lib.hm_lattice_set_slab(mesh.handle, 1))
    whole = _vectors(mesh, f[:3], slots)
    plane = (2 * nx + 1) * (2 * ny + 1)
    for z0, z1 in ((0, 14), (6, 20), (11, 30)):
        part = hm.BoxMesh((nx, ny, z1 - z0), (nx * h, ny * h, (z1 - z0) * h))
        check(lib.hm_lattice_set_slab(part.handle, 1))
        g = [v[2 * z0 * plane:(2 * z1 + 1) * plane].contiguous() for v in f[:3]]
        got = _vectors(part, g, slots)
        a, b = (0 if z0 == 0 else 2 * z0 + 1), (2 * nz + 1 if z1 == nz else 2 * z1)
        for s in slots:
            assert torch.equal(got[s][(a - 2 * z0) * plane:(b - 2 * z0) * plane],
                               whole[s][a * plane:b * plane]), (z0, s)
