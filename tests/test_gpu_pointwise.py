"""The pointwise data of an assembly point and the operator's diagonal against their direct
sums, at element counts around a block's, meshes around a tile's edge, both precisions, the
directional form, a buffer on an 8-byte boundary, and non-finite fields.  GPU."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import q2

pytestmark = pytest.mark.gpu

EPS = {0: 2.0 ** -52, 1: 2.0 ** -23}          # HM_FP64, HM_FP32
MESHES = [(1, 1, 1), (3, 1, 1), (31, 1, 1), (32, 1, 1), (33, 1, 1), (8, 4, 4), (9, 5, 5), (7, 3, 9), (16, 4, 3)]


def _fields(mesh, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal(mesh.ndof) for _ in range(4)]


def _reference(lat, u, m, p, mhat):
    """quad (ne, 8, 27) and, for each value, the sum of the absolute terms behind it."""
    ed = lat.edofs()
    N, G, _ = q2.basis_tables()
    h = np.asarray(lat.h)
    mv = m[ed] @ N.T
    D = lat.wdet()[None] * np.exp(mv)
    # relative size of D's error: the exponent's absolute error, and a direction's
    rel = np.abs(m)[ed] @ np.abs(N).T
    if mhat is not None:
        D, Dabs = D * (mhat[ed] @ N.T), D * (np.abs(mhat)[ed] @ np.abs(N).T)
    else:
        Dabs = D
    out, mag = [D], [Dabs * (1 + rel)]
    g, ga = [], []
    for f in (u, p):
        g.append(np.einsum("qak,ea->ekq", G, f[ed]) / h[None, :, None])
        ga.append(np.einsum("qak,ea->ekq", np.abs(G), np.abs(f)[ed]) / h[None, :, None])
    for f in range(2):
        for k in range(3):
            out.append(D * g[f][:, k])
            mag.append(mag[0] * ga[f][:, k])
    out.append(D * (g[0] * g[1]).sum(1))
    mag.append(mag[0] * (ga[0] * ga[1]).sum(1))
    return np.stack(out, 1), np.stack(mag, 1)


def _quad(mesh, fields, precision, direction, offset=0):
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    d = [torch.as_tensor(f, device=mesh.device) for f in fields]
    item = 8 if precision == 0 else 4
    n = mesh.ne * 216
    buf = torch.full((n * item // 8 + 4,), -7.0, dtype=torch.float64, device=mesh.device)
    status = torch.zeros(1, dtype=torch.int32, device=mesh.device)
    at = ctypes.c_void_p(buf.data_ptr() + offset)
    if direction:
        check(lib.hm_lattice_quadrature_dir(mesh.handle, *(ptr(v) for v in d), precision, at, ptr(status),
                                            stream_ptr()))
    else:
        check(lib.hm_lattice_quadrature(mesh.handle, *(ptr(v) for v in d[:3]), precision, at, ptr(status),
                                        stream_ptr()))
    torch.cuda.synchronize()
    raw = buf.cpu().numpy().tobytes()
    out = np.frombuffer(raw[offset:offset + n * item], np.float64 if precision == 0 else np.float32)
    assert set(np.frombuffer(raw[offset + n * item:], np.float64)) <= {-7.0}
    return out.reshape(mesh.ne, 8, 27).astype(np.float64), int(status.item()), buf


@pytest.mark.parametrize("direction", [False, True])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", MESHES)
def test_pointwise_data_matches_the_direct_sums(cuda, n, precision, direction):
    """Each value within 64 eps of the sum of its absolute terms: three contractions of at
    most three terms a field (9 roundings with the table's), the exponential and the weight
    (4), two or three products and W's sum, for up to four fields."""
    from hippymfem_b200 import BoxMesh

    L = (1.0, 0.7, 1.3)
    mesh, lat = BoxMesh(n, L), q2.Lattice(n, L)
    f = _fields(mesh, 3)
    want, mag = _reference(lat, *f[:3], f[3] if direction else None)
    for offset in (0, 8):
        out, status, _ = _quad(mesh, f, precision, direction, offset)
        assert status == 0
        assert np.all(np.abs(out - want) <= 64 * EPS[precision] * mag)


def test_non_finite_fields_set_the_status(cuda):
    from hippymfem_b200 import BoxMesh

    mesh = BoxMesh((9, 5, 5))
    for k in range(3):
        for bad in (np.nan, np.inf):
            f = _fields(mesh, 4)
            f[k][mesh.ndof - 1] = bad              # the last element's last node
            assert _quad(mesh, f, 0, False)[1] & 1


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", MESHES)
def test_diagonal_matches_the_direct_sum(cuda, n, precision):
    """All terms are positive: within 64 eps (27 D's in three contractions, the squared
    tables, eight elements), of the sum over the data as stored; 1 on the marked nodes."""
    from hippymfem_b200 import BoxMesh
    from hippymfem_b200._lib import check, lib, ptr, stream_ptr

    L = (1.0, 0.7, 1.3)
    mesh, lat = BoxMesh(n, L), q2.Lattice(n, L)
    quad, _, buf = _quad(mesh, _fields(mesh, 5), precision, False)
    _, G, _ = q2.basis_tables()
    local = np.einsum("eq,qak->ea", quad[:, 0], (G / np.asarray(lat.h)) ** 2)
    want = np.zeros(mesh.ndof)
    np.add.at(want, lat.edofs(), local)
    marker = np.zeros(mesh.ndof, np.uint8)
    marker[::7] = 1
    ess = torch.as_tensor(marker, device=cuda)
    for e in (None, ess):
        diag = torch.empty(mesh.ndof, dtype=torch.float64, device=cuda)
        check(lib.hm_lattice_diag_A(mesh.handle, ptr(buf), precision, None if e is None else ptr(e), ptr(diag),
                                    stream_ptr()))
        ref = want if e is None else np.where(marker, 1.0, want)
        assert np.all(np.abs(diag.cpu().numpy() - ref) <= 64 * EPS[0] * ref)
