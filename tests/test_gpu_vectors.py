"""``hm_lattice_vectors`` at the edges of its tiling and of its finiteness check: every subset
of the three vectors against the oracle, odd and even rows (with one vector an odd row's
pointwise data has no 16-byte pitch), directional products, and non-finite or overflowing
values reported whichever vectors are asked for.  GPU."""

import numpy as np
import pytest
import torch

from oracle import q2

pytestmark = pytest.mark.gpu

TOL = 1e-12      # relative to the largest entry, as the other FP64 parity tests

SIZES = [(1, 1, 1), (2, 1, 3), (1, 7, 2), (5, 4, 6), (35, 2, 3), (4, 33, 2), (14, 9, 12), (27, 6, 23)]


def _call(mesh, fields, slots, mhat=None, f=1.3, marker=None, zero=0, offset=0):
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    dev = mesh.device
    nbytes = lib.hm_lattice_vectors_workspace_bytes(mesh.handle, len(slots))
    work = torch.full((nbytes // 8 + offset,), float("nan"), dtype=torch.float64, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    out = {s: torch.full((mesh.ndof,), 7.0, dtype=torch.float64, device=dev) for s in slots}
    u, m, p = (torch.as_tensor(v, device=dev) for v in fields)
    h = None if mhat is None else torch.as_tensor(mhat, device=dev)
    check(lib.hm_lattice_vectors(mesh.handle, ptr(u), ptr(m), ptr(p), ptr(h), f, ptr(marker),
                                 ptr(out.get(0)), ptr(out.get(1)), ptr(out.get(2)), zero,
                                 ptr(work[offset:]), ptr(status), stream_ptr()))
    return {s: v.cpu().numpy() for s, v in out.items()}, int(status.item())


def _setup(n, seed=0):
    from hippymfem_b200 import BoxMesh

    L = tuple(0.1 * v * s for v, s in zip(n, (1.0, 0.8, 1.3)))
    mesh, mo = BoxMesh(n, L), q2.Lattice(n, L)
    rng = np.random.default_rng(seed)
    u, p, h = (rng.standard_normal(mo.ndof) for _ in range(3))
    return mesh, mo, u, 0.4 * rng.standard_normal(mo.ndof), p, h


@pytest.mark.parametrize("n", SIZES)
def test_every_subset_matches_the_oracle(cuda, n):
    mesh, mo, u, m, p, h = _setup(n)
    E = mo.edofs()
    ref = {s: q2.assemble_vector(E, v, mo.ndof) for s, v in
           q2.element_vectors(mo, E, u, m, p, f=1.3).items()}
    blk = q2.element_blocks(mo, E, u, m, p, ("C", "Wum", "Wmm"))
    name = {q2.ADJOINT: "C", q2.STATE: "Wum", q2.PARAMETER: "Wmm"}
    dref = {s: q2.assemble_vector(E, np.einsum("eab,eb->ea", blk[k], h[E]), mo.ndof)
            for s, k in name.items()}
    ess = np.zeros(mo.ndof, np.uint8)
    ess[mo.boundary_dofs()] = 1
    marker = torch.as_tensor(ess, device=cuda)
    for slots in ((0,), (1,), (2,), (0, 1), (0, 2), (1, 2), (0, 1, 2)):
        for offset in (0, 1):
            got, status = _call(mesh, (u, m, p), slots, offset=offset)
            assert status == 0
            for s in slots:
                assert np.abs(got[s] - ref[s]).max() <= TOL * np.abs(ref[s]).max(), (slots, s)
        got, status = _call(mesh, (u, m, p), slots, mhat=h, marker=marker, zero=1)
        assert status == 0
        for s in slots:
            want = np.where(ess != 0, 0.0, dref[s]) if s != q2.PARAMETER else dref[s]
            assert np.abs(got[s] - want).max() <= TOL * np.abs(dref[s]).max(), (slots, s)


@pytest.mark.parametrize("slots", [(0,), (1,), (2,), (0, 1, 2)])
def test_non_finite_values_are_reported_whatever_is_asked_for(cuda, slots):
    n = (5, 3, 4)
    mesh, mo, u, m, p, h = _setup(n, 1)
    node = mo.ndof // 2 + 3
    for which in range(3):
        for bad in (np.nan, np.inf, -np.inf if which != 1 else np.inf):
            f = [u.copy(), m.copy(), p.copy()]
            f[which][node] = bad
            assert _call(mesh, f, slots)[1] != 0, (which, bad)
    # e^m overflows; E = D grad u overflows with every node finite; D h does
    f = [u, m.copy(), p]
    f[1][node] = 2000.0
    assert _call(mesh, f, slots)[1] != 0
    f = [1e200 * u, m + 300.0, p]
    assert _call(mesh, f, slots)[1] != 0
    assert _call(mesh, (u, m + 300.0, p), slots, mhat=1e200 * h)[1] != 0
    # large but finite throughout: not reported
    assert _call(mesh, (1e60 * u, m + 100.0, 1e-60 * p), slots)[1] == 0
    assert _call(mesh, (u, m - 1000.0, p), slots)[1] == 0
