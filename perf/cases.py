"""What a user of this package has it do, as cases that can be timed and checked.

Every case goes through the package's public entry points with the inputs such a program
meets: log-conductivity fields that are sums of 32 cosines (the benchmark's family), smooth
states that vanish on the boundary, random directions, pointwise observations.  The kinds:

* ``blocks``    a linearization point through the C ABI: pointwise data, then the four
                blocks A, C, W_um, W_mm and the three vectors in one fused assembly, into
                buffers the program keeps (an outer Newton loop, a service);
* ``linpoint``  the same through ``PDEVariationalProblem``: two points in turn, as the
                iterates of a Newton loop, with the gradient at each;
* ``vectors``   residual, dR/dm and dR/du at a point without blocks (a line search, a
                gradient-based method);
* ``forward``   the forward problem at two trial parameters, each with its own operator
                set-up (a line search; a sampler): multigrid- or Jacobi-preconditioned,
                FP64 or mixed precision, matrix-free or assembled;
* ``hessian``   one action of the reduced Hessian at a solved point (two incremental
                solves), the inner step of Newton-CG and of low-rank eigensolvers;
* ``apply``     products with the assembled blocks and their transposes (``apply_ij``);
* ``prior``     the BiLaplacian prior's precision and its inverse applied to a vector.
"""

import math

import numpy as np
import torch

STATE, PARAMETER, ADJOINT = 0, 1, 2
RTOL = 1e-12                     # the solves' relative tolerance (the package's default)
NOISE = 1e-4                     # noise variance of the observations
GAMMA, DELTA = 0.1, 0.5          # the prior's coefficients
BLOCKS = ("A", "C", "Wum", "Wmm")


# ------------------------------------------------------------------------------ cases
def _case(kind, n, L=(1.0, 1.0, 1.0), sigma=0.1, pre="mg", prec="fp64", mf=True):
    c = {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "Lx": L[0], "Ly": L[1], "Lz": L[2],
         "sigma": sigma}
    if kind in ("forward", "hessian"):
        c.update(pre=pre, prec=prec, mf=bool(mf))
    return c


def listed():
    """The ranges' corners: the smallest calls, ordinary and ragged ones, the largest."""
    def named(name, c):
        return dict(c, name=name)

    return [
        # one request of a service on a tiny mesh: launches and latency
        named("blocks-tiny", _case("blocks", (8, 8, 8))),
        # a mesh cut to an anisotropic domain: no axis a multiple of anything
        named("blocks-ragged", _case("blocks", (37, 50, 23), (1.0, 1.4, 0.5), 0.5)),
        # the benchmark's linearization point
        named("blocks-64", _case("blocks", (64, 64, 64))),
        # Newton iterates through the problem class, gradient included
        named("linpoint-40", _case("linpoint", (40, 40, 40), sigma=0.5)),
        # gradients and residuals along a line search
        named("vectors-64", _case("vectors", (64, 64, 64), sigma=0.5)),
        # small forward solves (a service's ordinary request)
        named("forward-mg-12", _case("forward", (12, 12, 12), sigma=0.5)),
        # the package's default options: assembled Jacobian, Jacobi-preconditioned CG
        named("forward-default", _case("forward", (27, 18, 33), (1.0, 0.7, 1.2), 0.5,
                                       pre="jacobi", mf=False)),
        # the benchmark's forward solves at two trial points
        named("forward-mg-64", _case("forward", (64, 64, 64))),
        # the benchmark's Hessian action
        named("hessian-mg-64", _case("hessian", (64, 64, 64))),
        # the Hessian action with the single-precision V-cycle, on an ordinary mesh
        named("hessian-mixed-48", _case("hessian", (48, 32, 40), (1.0, 0.7, 0.8), 0.5,
                                        prec="mixed")),
        # block products of a caller with its own outer solver
        named("apply-ragged", _case("apply", (45, 52, 39), (0.9, 1.0, 0.8), 0.5)),
        # the prior inside a Newton-CG iteration
        named("prior-24", _case("prior", (24, 24, 24))),
    ]


# elements of a drawn case at most, by kind: no drawn case costs more than the largest
# listed one
_MOST = {"blocks": 64 ** 3, "linpoint": 48 ** 3, "vectors": 64 ** 3, "forward": 48 ** 3,
         "hessian": 48 ** 3, "apply": 48 ** 3, "prior": 16000}


def _axis(rng, lo, hi, even):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, v - v % 4) if even else v


def draw(rng):
    kind = rng.choice(("blocks", "blocks", "linpoint", "vectors", "forward", "forward",
                       "hessian", "apply", "prior"))
    pre = rng.choice(("mg", "mg", "jacobi"))
    prec = rng.choice(("fp64", "fp64", "mixed"))
    # multigrid meshes are mostly ones that coarsen; the rest is any size, odd ones too
    even = kind in ("forward", "hessian") and pre == "mg" and rng.random() < 0.7
    most = _MOST[kind]
    if kind in ("forward", "hessian") and pre == "jacobi":
        most = 12000
    lo = 4 if even else 3
    while True:
        n = [_axis(rng, lo, 80, even) for _ in range(3)]
        # half of the draws near a cube, as most meshes are
        if rng.random() < 0.5:
            n = [max(lo, v - v % 4 if even else v) for v in
                 (n[0], int(n[0] * rng.uniform(0.7, 1.4)), int(n[0] * rng.uniform(0.7, 1.4)))]
        if 64 <= n[0] * n[1] * n[2] <= most and max(n) <= 6 * min(n):
            break
    h = [rng.uniform(0.8, 1.25) for _ in range(3)]
    size = max(v * s for v, s in zip(n, h))
    L = [round(v * s / size, 3) for v, s in zip(n, h)]
    return _case(kind, n, L, rng.choice((0.1, 0.3, 0.5)), pre, prec,
                 mf=prec == "mixed" or pre == "mg" or rng.random() < 0.5)


def _n(case):
    return case["nx"], case["ny"], case["nz"]


def _L(case):
    return case["Lx"], case["Ly"], case["Lz"]


def _sizes(case):
    n = _n(case)
    ne = n[0] * n[1] * n[2]
    nd = (2 * n[0] + 1) * (2 * n[1] + 1) * (2 * n[2] + 1)
    nnz = math.prod(8 * v + 1 for v in n)
    return ne, nd, nnz


# ----------------------------------------------------------------------------- inputs
def _dev():
    return torch.device("cuda")


def _coords(case):
    """(ndof, 3) node coordinates, x fastest."""
    ax = [torch.arange(2 * n + 1, dtype=torch.float64, device=_dev()) * (L / (2 * n))
          for n, L in zip(_n(case), _L(case))]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], -1)


def _field(X, rng, sigma, nterms=32):
    """sum_j a_j cos(2 pi w_j . x + phi_j): the log-conductivity family of the benchmark."""
    a = rng.normal(0.0, sigma, nterms)
    w = rng.integers(-4, 5, size=(nterms, 3)).astype(np.float64)
    phi = rng.uniform(0.0, 2.0 * np.pi, nterms)
    out = torch.zeros(X.shape[0], dtype=torch.float64, device=X.device)
    for j in range(nterms):
        arg = (X[:, 0] * w[j, 0] + X[:, 1] * w[j, 1] + X[:, 2] * w[j, 2]) * (2.0 * np.pi)
        out += float(a[j]) * torch.cos(arg + float(phi[j]))
    return out


def _bump(X, case):
    """A smooth state: zero on the boundary."""
    out = torch.ones(X.shape[0], dtype=torch.float64, device=X.device)
    for d, L in enumerate(_L(case)):
        t = X[:, d] / L
        out = out * (4.0 * t * (1.0 - t))
    return out


def _inputs(case, seed):
    """The case's fields and points, from the seed alone."""
    rng = np.random.default_rng([int(seed), 17])
    X = _coords(case)
    m = _field(X, rng, case["sigma"])
    kind = case["kind"]
    got = {"m": m}
    if kind in ("blocks", "linpoint", "vectors", "apply"):
        b = _bump(X, case)
        got["u"] = 0.1 * b * (1.0 + 0.2 * _field(X, rng, 0.3))
        got["p"] = 0.5 * b * _field(X, rng, 0.4)
    if kind == "linpoint":
        got["u2"] = got["u"] * (1.0 + 0.1 * _field(X, rng, 0.2))
        got["p2"] = got["p"] + 0.05 * _bump(X, case) * _field(X, rng, 0.3)
    if kind in ("linpoint", "forward"):
        got["m2"] = m + 0.5 * _field(X, rng, 0.2 * case["sigma"])
    if kind in ("hessian", "apply", "prior"):
        got["v"] = torch.as_tensor(rng.standard_normal(X.shape[0]), device=_dev())
    if kind == "hessian":
        nobs = max(16, _sizes(case)[0] // 64)
        t = 0.05 + 0.9 * rng.random((nobs, 3))
        got["points"] = t * np.asarray(_L(case))
        got["data"] = 0.05 * np.prod(4.0 * t * (1.0 - t), axis=1) * (1 + 0.1 * rng.standard_normal(nobs))
    return got


def prepare(case, seed):
    import hippymfem_b200 as hm

    s = {"case": case}
    inp = _inputs(case, seed)
    mesh = s["mesh"] = hm.BoxMesh(_n(case), _L(case))
    V = s["V"] = hm.Q2Space(mesh)
    bc = s["bc"] = hm.DirichletBC(V)
    kind = case["kind"]

    def problem(**kw):
        return hm.PDEVariationalProblem([V, V, V], f=1.0, bc=bc, solver_tolerance=RTOL, **kw)

    if kind == "blocks":
        pat = s["pattern"] = hm.LatticePattern(mesh)
        s["vals"] = [pat.new_values() for _ in BLOCKS]
        s["vecs"] = [V.vector() for _ in range(3)]
        s["quad"] = torch.empty(mesh.quad_bytes() // 8 + 1, dtype=torch.float64, device=_dev())
        s["status"] = torch.zeros(1, dtype=torch.int32, device=_dev())
        s["x"] = [inp["u"], inp["m"], inp["p"]]
    elif kind == "linpoint":
        s["prob"] = problem()
        s["points"] = [[inp["u"], inp["m"], inp["p"]], [inp["u2"], inp["m2"], inp["p2"]]]
        s["grads"] = [V.vector(), V.vector()]
        s["prob"].pattern
    elif kind == "vectors":
        s["vecs"] = [V.vector() for _ in range(3)]
        need = hm._lib.lib.hm_lattice_vectors_workspace_bytes(mesh.handle, 3)
        s["work"] = torch.empty(need // 8 + 1, dtype=torch.float64, device=_dev())
        s["status"] = torch.zeros(1, dtype=torch.int32, device=_dev())
        s["x"] = [inp["u"], inp["m"], inp["p"]]
    elif kind == "forward":
        s["prob"] = problem(matrix_free_solves=case["mf"], solver_precision=case["prec"],
                            preconditioner=case["pre"])
        if not case["mf"]:
            s["prob"].pattern
        s["trials"] = [inp["m"], inp["m2"]]
        s["u"] = [V.vector(), V.vector()]
    elif kind == "hessian":
        prob = problem(matrix_free_solves=case["mf"], solver_precision=case["prec"],
                       preconditioner=case["pre"])
        misfit = hm.PointwiseStateObservation(V, inp["points"], data=inp["data"],
                                              noise_variance=NOISE)
        model = hm.Model(prob, None, misfit)
        u, p = V.vector(), V.vector()
        x = [u, inp["m"], p]
        model.solveFwd(u, x)
        model.solveAdj(p, x)
        model.setPointForHessianEvaluations(x)
        s["H"] = hm.ReducedHessian(model)
        s["v"], s["y"] = inp["v"], V.vector()
    elif kind == "apply":
        s["prob"] = problem()
        s["prob"].setLinearizationPoint([inp["u"], inp["m"], inp["p"]])
        s["v"] = inp["v"]
        s["out"] = [V.vector() for _ in _PRODUCTS]
    elif kind == "prior":
        s["prior"] = hm.BiLaplacianPrior(V, GAMMA, DELTA)
        s["v"] = inp["v"]
        s["out"] = [V.vector(), V.vector()]
    else:
        raise ValueError("no kind %r" % (kind,))
    return s


_PRODUCTS = ((ADJOINT, STATE), (ADJOINT, PARAMETER), (STATE, PARAMETER),
             (PARAMETER, PARAMETER), (PARAMETER, ADJOINT), (PARAMETER, STATE))


def run(s):
    kind = s["case"]["kind"]
    if kind in ("blocks", "vectors"):
        from hippymfem_b200._lib import HM_FP64, check, lib, ptr, stream_ptr

        mesh, (u, m, p) = s["mesh"], s["x"]
        st, pa, ad = (ptr(v) for v in s["vecs"])
        if kind == "vectors":
            check(lib.hm_lattice_vectors(mesh.handle, ptr(u), ptr(m), ptr(p), None, 1.0,
                                         ptr(s["bc"].marker), st, pa, ad, 0, ptr(s["work"]),
                                         ptr(s["status"]), stream_ptr()), "hm_lattice_vectors")
            return {"vecs": list(s["vecs"]), "status": s["status"]}
        check(lib.hm_lattice_quadrature(mesh.handle, ptr(u), ptr(m), ptr(p), HM_FP64,
                                        ptr(s["quad"]), ptr(s["status"]), stream_ptr()),
              "hm_lattice_quadrature")
        check(lib.hm_lattice_assemble(mesh.handle, ptr(s["quad"]), HM_FP64,
                                      ptr(s["pattern"].indptr), ptr(s["bc"].marker), 1.0,
                                      *[ptr(v) for v in s["vals"]], st, pa, ad, 0,
                                      stream_ptr()), "hm_lattice_assemble")
        return {"vals": list(s["vals"]), "vecs": list(s["vecs"]), "status": s["status"]}
    if kind == "linpoint":
        prob = s["prob"]
        for x, g in zip(s["points"], s["grads"]):
            prob.setLinearizationPoint(x)
            prob.evalGradientParameter(x, g)
        return {"vals": [b.values for b in (prob.A, prob.C, prob.Wum, prob.Wmm)],
                "grads": list(s["grads"])}
    if kind == "forward":
        for m, u in zip(s["trials"], s["u"]):
            s["prob"].solveFwd(u, [u, m, None])
        return list(s["u"])
    if kind == "hessian":
        return s["H"].mult(s["v"], s["y"])
    if kind == "apply":
        for (i, j), out in zip(_PRODUCTS, s["out"]):
            s["prob"].apply_ij(i, j, s["v"], out)
        return list(s["out"])
    s["prior"].R.mult(s["v"], s["out"][0])
    s["prior"].Rsolver.solve(s["out"][1], s["v"])
    return list(s["out"])


# ------------------------------------------------------------------------------- work
def work(case):
    """Bytes and FP64 operations one pass cannot do without.  A solve's are its operator's
    data and one read or write of x, r, p and q each iteration, for a nominal count."""
    ne, nd, nnz = _sizes(case)
    kind = case["kind"]
    point = ne * 27 * 2.0 * 90          # fields and pointwise data at the 27 points
    rows = ne * 27 * 2.0 * 60           # element vectors
    block = ne * 5500.0                 # an average block's sum-factorised contractions
    apply_ = ne * 2.0 * 1300            # one application of the Jacobian, sum-factorised
    if kind == "blocks":
        return {"bytes": 8.0 * (4 * nnz + 6 * nd) + nd + 4.0 * nd, "flops": point + 4 * block}
    if kind == "linpoint":
        return {"bytes": 2 * (8.0 * (4 * nnz + 4 * nd) + 5.0 * nd), "flops": 2 * (point + 4 * block)}
    if kind == "vectors":
        return {"bytes": 8.0 * 6 * nd, "flops": point + 3 * rows}
    its = 12 if case.get("pre") == "mg" else 8 * max(_n(case))
    step = 8.0 * (27 * ne + 7 * nd) if case.get("mf") else 8.0 * (nnz + 7 * nd)
    ops = apply_ if case.get("mf") else 2.0 * nnz
    if kind == "forward":
        return {"bytes": 2 * its * step, "flops": 2 * (its * ops + point)}
    if kind == "hessian":
        return {"bytes": 2 * its * step + 8.0 * 14 * nd, "flops": 2 * its * ops + 3 * (point + 3 * rows)}
    if kind == "apply":
        return {"bytes": 6 * 8.0 * (nnz + 2 * nd), "flops": 6 * 2.0 * nnz}
    return {"bytes": 60 * 8.0 * (nnz + 7 * nd), "flops": 60 * 2.0 * nnz}


# ------------------------------------------------------------------------------ exact
class _Q2:
    """The Q2 lattice in plain torch, FP64: element tables, gathers, element products."""

    def __init__(self, case):
        d = _dev()
        self.n, self.L = _n(case), _L(case)
        self.N = [2 * v + 1 for v in self.n]
        self.h = [L / v for L, v in zip(self.L, self.n)]
        nx, ny, nz = self.n
        s = math.sqrt(0.15)
        x = np.array([0.5 - s, 0.5, 0.5 + s])
        w = np.array([5.0, 8.0, 5.0]) / 18.0
        B = np.stack([2 * (x - 0.5) * (x - 1), -4 * x * (x - 1), 2 * x * (x - 0.5)], -1)
        D = np.stack([4 * x - 3, 4 - 8 * x, 4 * x - 1], -1)

        def tab(a, b, c):   # point q = q1 + 3 q2 + 9 q3, node a = a1 + 3 a2 + 9 a3
            return torch.as_tensor(np.einsum("xa,yb,zc->zyxcba", a, b, c).reshape(27, 27), device=d)

        self.B = tab(B, B, B)
        self.G = [tab(D, B, B) / self.h[0], tab(B, D, B) / self.h[1], tab(B, B, D) / self.h[2]]
        self.w = torch.as_tensor(np.einsum("x,y,z->zyx", w, w, w).reshape(27) * math.prod(self.h), device=d)
        e = torch.arange(nx * ny * nz, device=d)
        ex, ey, ez = e % nx, (e // nx) % ny, e // (nx * ny)
        a = torch.arange(27, device=d)
        self.ijk = [2 * ex[:, None] + a % 3, 2 * ey[:, None] + (a // 3) % 3, 2 * ez[:, None] + a // 9]
        self.edof = self.ijk[0] + self.N[0] * (self.ijk[1] + self.N[1] * self.ijk[2])
        self.nd = math.prod(self.N)
        i = torch.arange(self.nd, device=d)
        c = [i % self.N[0], (i // self.N[0]) % self.N[1], i // (self.N[0] * self.N[1])]
        self.ess = torch.zeros(self.nd, dtype=torch.bool, device=d)
        for v, N in zip(c, self.N):
            self.ess |= (v == 0) | (v == N - 1)

    def scatter(self, ye):
        return torch.zeros(self.nd, dtype=torch.float64, device=ye.device).index_add_(
            0, self.edof.reshape(-1), ye.reshape(-1))

    def fields(self, u, m, p):
        """D, grad u, grad p at the points."""
        D = self.w * torch.exp(m[self.edof] @ self.B.T)
        U, P = u[self.edof], p[self.edof]
        return D, [U @ g.T for g in self.G], [P @ g.T for g in self.G]

    def vectors(self, D, gu, gp, f):
        """dR/du, dR/dm, dR/dp."""
        st = sum((D * g) @ t for g, t in zip(gp, self.G))
        ad = sum((D * g) @ t for g, t in zip(gu, self.G)) - f * (self.w @ self.B)
        W = D * sum(a * b for a, b in zip(gu, gp))
        return self.scatter(st), self.scatter(W @ self.B), self.scatter(ad)

    def jac(self, D, x):
        """A x without elimination."""
        X = x[self.edof]
        return self.scatter(sum((D * (X @ g.T)) @ g for g in self.G))

    def product(self, i, j, D, gu, gp, v):
        """The (i, j) block with its elimination applied to v."""
        clean = v.masked_fill(self.ess, 0.0)
        if {i, j} == {STATE, ADJOINT}:
            return torch.where(self.ess, v, self.jac(D, clean))
        g = {ADJOINT: gu, STATE: gp}
        if (i, j) == (PARAMETER, PARAMETER):
            W = D * sum(a * b for a, b in zip(gu, gp))
            return self.scatter((W * (v[self.edof] @ self.B.T)) @ self.B)
        if j == PARAMETER:          # rows of the essential nodes are zero
            S = D * (v[self.edof] @ self.B.T)
            y = self.scatter(sum((S * a) @ t for a, t in zip(g[i], self.G)))
            return y.masked_fill(self.ess, 0.0)
        X = clean[self.edof]        # the transpose: those entries of v do not count
        return self.scatter((D * sum(a * (X @ t.T) for a, t in zip(g[j], self.G))) @ self.B)

    def element_block(self, name, D, gu, gp, sel):
        D, gu, gp = D[sel], [a[sel] for a in gu], [a[sel] for a in gp]
        if name == "A":
            return sum((D[:, :, None] * t).transpose(1, 2) @ t for t in self.G)
        if name == "Wmm":
            W = D * sum(a * b for a, b in zip(gu, gp))
            return (W[:, :, None] * self.B).transpose(1, 2) @ self.B
        g = gu if name == "C" else gp
        return sum((D * a)[:, :, None] * t for a, t in zip(g, self.G)).transpose(1, 2) @ self.B

    def slots(self, sel):
        """CSR position (diagonal first, then ascending columns) of each element entry."""
        lo, cnt, pre, tot = [], [], [], []
        for N in self.N:
            i = torch.arange(N, device=self.ess.device)
            even = i % 2 == 0
            a = torch.where(even, (i - 2).clamp(min=0), i - 1)
            b = torch.where(even, (i + 2).clamp(max=N - 1), i + 1)
            k = b - a + 1
            lo.append(a), cnt.append(k), pre.append(torch.cumsum(k, 0) - k), tot.append(int(k.sum()))
        r = [c[sel][:, :, None] for c in self.ijk]      # row node
        c = [c[sel][:, None, :] for c in self.ijk]      # column node
        n = [k[v] for k, v in zip(cnt, r)]
        start = pre[2][r[2]] * tot[0] * tot[1] + n[2] * (pre[1][r[1]] * tot[0] + n[1] * pre[0][r[0]])

        def rank(x):
            o = [v - a[rr] for v, a, rr in zip(x, lo, r)]
            return (o[2] * n[1] + o[1]) * n[0] + o[0]

        k, kd = rank(c), rank(r)
        return start + torch.where(k == kd, 0, torch.where(k < kd, k + 1, k)), math.prod(tot)

    def blocks(self, u, m, p):
        """The CSR values of A, C, W_um, W_mm."""
        D, gu, gp = self.fields(u, m, p)
        ne = D.shape[0]
        out = None
        for e0 in range(0, ne, 1 << 15):
            sel = slice(e0, min(ne, e0 + (1 << 15)))
            slot, nnz = self.slots(sel)
            if out is None:
                out = [torch.zeros(nnz, dtype=torch.float64, device=D.device) for _ in BLOCKS]
            ed = self.edof[sel]
            re, ce = self.ess[ed][:, :, None], self.ess[ed][:, None, :]
            for v, name in zip(out, BLOCKS):
                K = self.element_block(name, D, gu, gp, sel)
                if name == "A":
                    K = K.masked_fill(re | ce, 0.0)
                elif name != "Wmm":
                    K = K.masked_fill(re.expand_as(K), 0.0)
                v.index_add_(0, slot.reshape(-1), K.reshape(-1))
            diag = (ed[:, :, None] == ed[:, None, :]) & re
            out[0][slot[diag]] = 1.0
        return out, (D, gu, gp)

    def solve(self, D, b):
        """A^{-1} b with b zeroed on the essential nodes: CG, then twice again on the
        residual of the sum."""
        b = b.masked_fill(self.ess, 0.0)
        dg = self.scatter(sum(D @ (t * t) for t in self.G)).masked_fill_(self.ess, 1.0)
        x = torch.zeros_like(b)
        for rtol in (1e-12, 1e-3, 1e-3):
            r = b - self.jac(D, x).masked_fill_(self.ess, 0.0)
            d, z = torch.zeros_like(r), r / dg
            p, rz, stop = z.clone(), torch.dot(r, z), float(r.norm()) * rtol
            for it in range(6000):
                q = self.jac(D, p).masked_fill_(self.ess, 0.0)
                alpha = rz / torch.dot(p, q)
                d += alpha * p
                r -= alpha * q
                if it % 16 == 15 and not float(r.norm()) > stop:
                    break
                z = r / dg
                rz, old = torch.dot(r, z), rz
                p = z + (rz / old) * p
            x = x + torch.where(torch.isfinite(d), d, torch.zeros_like(d))
        return x

    def observation(self, points):
        """Node numbers and basis values (nobs, 27) of the points."""
        s = torch.as_tensor(np.asarray(points) / np.asarray(self.h), device=self.ess.device)
        idx, val = [], []
        for d in range(3):
            e = s[:, d].floor().clamp(0, self.n[d] - 1)
            t = s[:, d] - e
            idx.append(2 * e.long()[:, None] + torch.arange(3, device=s.device))
            val.append(torch.stack([2 * (t - 0.5) * (t - 1), -4 * t * (t - 1), 2 * t * (t - 0.5)], -1))
        nodes = (idx[0][:, None, None, :] + self.N[0] * (idx[1][:, None, :, None]
                                                         + self.N[1] * idx[2][:, :, None, None]))
        vals = val[2][:, :, None, None] * val[1][:, None, :, None] * val[0][:, None, None, :]
        return nodes.reshape(-1, 27), vals.reshape(-1, 27)


def _exact_hessian(q, inp):
    nodes, vals = q.observation(inp["points"])

    def obs(u):
        return (u[nodes] * vals).sum(1)

    def obs_t(y):
        return torch.zeros(q.nd, dtype=torch.float64, device=y.device).index_add_(
            0, nodes.reshape(-1), (vals * y[:, None]).reshape(-1)) / NOISE

    m, v = inp["m"], inp["v"]
    zero = torch.zeros_like(m)
    D, _, _ = q.fields(zero, m, zero)
    u = q.solve(D, q.scatter((q.w @ q.B).expand(D.shape[0], 27)))
    p = q.solve(D, -obs_t(obs(u) - torch.as_tensor(inp["data"], device=u.device)))
    D, gu, gp = q.fields(u, m, p)
    uhat = q.solve(D, q.product(ADJOINT, PARAMETER, D, gu, gp, v))
    phat = q.solve(D, obs_t(obs(uhat)) - q.product(STATE, PARAMETER, D, gu, gp, v))
    return (q.product(PARAMETER, PARAMETER, D, gu, gp, v) + q.product(PARAMETER, ADJOINT, D, gu, gp, phat)
            - q.product(PARAMETER, STATE, D, gu, gp, uhat))


def _exact_prior(case, v):
    """R v and R^{-1} v by the 1D generalized eigenvectors of (K, M) on each axis."""
    lam, vec, mass = [], [], []
    for n, L in zip(_n(case), _L(case)):
        h = L / n
        Ke = np.array([[7, -8, 1], [-8, 16, -8], [1, -8, 7]]) / (3 * h)
        Me = np.array([[4, 2, -1], [2, 16, 2], [-1, 2, 4]]) * (h / 30)
        K, M = np.zeros((2 * n + 1,) * 2), np.zeros((2 * n + 1,) * 2)
        for e in range(n):
            K[2 * e:2 * e + 3, 2 * e:2 * e + 3] += Ke
            M[2 * e:2 * e + 3, 2 * e:2 * e + 3] += Me
        C = np.linalg.cholesky(M)
        W = np.linalg.solve(C, np.linalg.solve(C, K).T)
        l, Q = np.linalg.eigh(0.5 * (W + W.T))
        lam.append(torch.as_tensor(l, device=_dev()))
        vec.append(torch.as_tensor(np.linalg.solve(C.T, Q), device=_dev()))   # M-orthonormal
        mass.append(torch.as_tensor(M, device=_dev()))

    def along(mats, x):
        x = torch.einsum("ax,zyx->zya", mats[0], x)
        x = torch.einsum("by,zya->zba", mats[1], x)
        return torch.einsum("cz,zba->cba", mats[2], x)

    s = lam[2][:, None, None] + lam[1][None, :, None] + lam[0][None, None, :]
    a = GAMMA * s + DELTA
    X = v.reshape([2 * n + 1 for n in _n(case)][::-1])
    c = along([e.T for e in vec], X)                       # V^T x
    inv = along(vec, c / (a * a))                          # (A M^-1 A)^-1 = V a^-2 V^T
    c = along([(m @ e).T for m, e in zip(mass, vec)], X)   # V^-1 x
    fwd = along([m @ e for m, e in zip(mass, vec)], c * a * a)
    return [fwd.reshape(-1), inv.reshape(-1)]


def exact(case, seed):
    """What ``run`` returns, in plain FP64 torch."""
    kind = case["kind"]
    inp = _inputs(case, seed)
    if kind == "prior":
        return _exact_prior(case, inp["v"])
    q = _Q2(case)
    if kind == "blocks":
        vals, (D, gu, gp) = q.blocks(inp["u"], inp["m"], inp["p"])
        return {"vals": vals, "vecs": list(q.vectors(D, gu, gp, 1.0)), "status": None}
    if kind == "linpoint":
        _, g1, _ = q.vectors(*q.fields(inp["u"], inp["m"], inp["p"]), 1.0)
        vals, (D, gu, gp) = q.blocks(inp["u2"], inp["m2"], inp["p2"])
        return {"vals": vals, "grads": [g1, q.vectors(D, gu, gp, 1.0)[1]]}
    if kind == "vectors":
        return {"vecs": list(q.vectors(*q.fields(inp["u"], inp["m"], inp["p"]), 1.0)), "status": None}
    if kind == "forward":
        one = torch.ones(1, dtype=torch.float64, device=_dev())
        out = []
        for m in (inp["m"], inp["m2"]):
            D = q.w * torch.exp(m[q.edof] @ q.B.T)
            out.append(q.solve(D, q.scatter((one * q.w @ q.B).expand(D.shape[0], 27))))
        return out
    if kind == "hessian":
        return _exact_hessian(q, inp)
    D, gu, gp = q.fields(inp["u"], inp["m"], inp["p"])
    return [q.product(i, j, D, gu, gp, inp["v"]) for i, j in _PRODUCTS]
