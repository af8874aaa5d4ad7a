"""``hm_lattice_vectors`` and ``hm_lattice_vectors_at`` with an output that is, or overlaps,
one of the fields it is made of: the vectors are those of the fields as they were when the
call was made.  GPU."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = 1e-12      # relative to the largest entry, as the other FP64 parity tests

# one element; one tile; several tiles along every axis, even and odd rows
SIZES = [(1, 1, 1), (5, 4, 6), (26, 23, 31), (40, 32, 36)]


def _fields(mesh, seed, extra=0):
    """u, m, p, mhat side by side in one array, ``extra`` entries behind each."""
    rng = np.random.default_rng(seed)
    n = mesh.ndof + extra
    a = torch.as_tensor(rng.standard_normal(4 * n) * 0.4, device=mesh.device)
    return a, [a[k * n:k * n + mesh.ndof] for k in range(4)]


def _call(mesh, fields, mhat, outs, marker=None, zero=0):
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, len(outs))
    work = torch.full((nbytes // 8,), float("nan"), dtype=torch.float64, device=mesh.device)
    status = torch.zeros(1, dtype=torch.int32, device=mesh.device)
    u, m, p = fields
    check(lib.hm_lattice_vectors(mesh.handle, ptr(u), ptr(m), ptr(p), ptr(mhat), 1.3, ptr(marker),
                                 ptr(outs.get(0)), ptr(outs.get(1)), ptr(outs.get(2)), zero,
                                 ptr(work), ptr(status), stream_ptr()))
    return int(status.item())


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("targets", [{0: 0}, {0: 2}, {1: 0}, {1: 2}, {2: 0}, {2: 2}, {1: 1}, {2: 3},
                                     {0: 2, 2: 0}, {0: 0, 1: 2}, {0: 2, 1: 1, 2: 0}])
def test_outputs_that_are_inputs(cuda, n, targets):
    """``targets``: slot -> the field (u, m, p, mhat) its vector overwrites."""
    from hippymfem_b200 import BoxMesh, DirichletBC, Q2Space

    mesh = BoxMesh(n, tuple(0.1 * v for v in n))
    marker = DirichletBC(Q2Space(mesh)).marker
    for with_mhat in (False, True):
        _, f = _fields(mesh, 5)
        mhat = f[3] if with_mhat else None
        want = {s: torch.empty_like(f[0]) for s in targets}
        assert _call(mesh, f[:3], mhat, want, marker, 1) == 0
        assert _call(mesh, f[:3], mhat, {s: f[k] for s, k in targets.items()}, marker, 1) == 0
        for s, k in targets.items():
            err = float((f[k] - want[s]).abs().max())
            assert err <= TOL * float(want[s].abs().max()), (with_mhat, s, err)


def test_outputs_that_overlap_inputs_in_part(cuda):
    """dR/du in place of p's first half and what lies before it; the gradient over the end of u."""
    from hippymfem_b200 import BoxMesh

    mesh = BoxMesh((18, 21, 16), (1.0, 1.2, 0.9))
    nd = mesh.ndof
    for slot, field, shift in ((0, 2, -(nd // 2)), (1, 0, nd // 3), (2, 0, 1)):
        a, f = _fields(mesh, 7, extra=nd)
        want = {slot: torch.empty_like(f[0])}
        assert _call(mesh, f[:3], None, want) == 0
        at = field * 2 * nd + shift
        assert _call(mesh, f[:3], None, {slot: a[at:at + nd]}) == 0
        err = float((a[at:at + nd] - want[slot]).abs().max())
        assert err <= TOL * float(want[slot].abs().max()), (slot, err)


@pytest.mark.parametrize("same", [False, True])
def test_vectors_at_in_place(cuda, same):
    from hippymfem_b200 import BoxMesh
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    mesh = BoxMesh((26, 23, 31))
    _, f = _fields(mesh, 9)
    want = {0: torch.empty_like(f[0]), 2: torch.empty_like(f[0])}
    assert _call(mesh, f[:3], None, want) == 0
    kept = [torch.full_like(f[0], 3.0), torch.full_like(f[0], 4.0)]
    point = [v.clone() for v in f[:3]]
    if not same:
        point[1][11] += 1.0
    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, 2)
    work = torch.empty(nbytes // 8, dtype=torch.float64, device=cuda)
    word, status = (torch.zeros(1, dtype=torch.int32, device=cuda) for _ in range(2))
    u, m, p = f[:3]
    check(lib.hm_lattice_vectors_at(mesh.handle, ptr(u), ptr(m), ptr(p), *(ptr(v) for v in point),
                                    ptr(kept[0]), None, ptr(kept[1]), 1.3, ptr(p), None, ptr(u),
                                    ptr(work), ptr(word), ptr(status), stream_ptr()))
    for got, k, w in ((p, kept[0], want[0]), (u, kept[1], want[2])):
        if same:
            assert torch.equal(got, k)
        else:
            assert float((got - w).abs().max()) <= TOL * float(w.abs().max())
