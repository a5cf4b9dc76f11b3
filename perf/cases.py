"""Measured workloads of the library: what a user's program has it do, through the Python binding of the C ABI.

A case is a dict of plain values.  `kind` says which call it makes:

  product   Operator.matvec / matvec_pair in FP64 (A p, A^H p, or both in one pass)
  solve     Operator.solve (FP64 BiCG, or FP32 sweeps inside FP64 refinement)
  waves     Operator.solve_multi for incident plane waves (lockstep, refined)
  batch     Batch.solve for ellipsoids of different sizes
  build     level set in host memory -> operator -> tube arrays on the host
  slice     Operator.evaluate_slice of a density
  gradient  Operator.misfit_gradient (boundary data, wave number, weights)
  combo     Operator.solve in the Combo formulation (refined)

The surfaces are the repository's: the sphere, the torus (R = 0.6, r = 0.25), ellipsoids and the bumpy sphere in
[-1, 1]^3 with a tube of three grid steps, and the [-2, 2]^3 Neumann sphere of the reference's defaults.  A seed turns
and mirrors the surface on its grid and sets the sources, waves and densities.

Single products in FP32 are not cases of their own: the solves are made of them.  Every solve asks for a residual far
below what FP32 products give, so its result carries FP64 accuracy whatever the order of the sums inside.
"""
import math

import numpy as np
import torch

import helmholtz_3d_torrone_gb300 as hz
from helmholtz_3d_torrone_gb300 import geometry as G

PI = math.pi
UNIT = dict(lo=-1.0, hi=1.0, factor=3.0, dirichlet=1)
WIDE = dict(lo=-2.0, hi=2.0, factor=2.0, dirichlet=0)


def listed():
    return [
        # the smallest call: one FP64 product of a coarse sphere, where latency and idle SMs count
        dict(UNIT, name="product_sphere24", kind="product", shape="sphere", N=24, k=5.0, mode="A"),
        # one BiCG iteration's two products on the 64^3 sphere (n = 19.6k), Neumann form
        dict(UNIT, name="pair_sphere64", kind="product", shape="sphere", N=64, k=5.0, mode="pair", dirichlet=0),
        # the largest: an FP64 residual of the adjoint system on the 128^3 torus (n = 145k)
        dict(UNIT, name="adjoint_torus128", kind="product", shape="torus", N=128, k=20.0, mode="AH"),
        # the 64^3 sphere with a point source, solved from start to end by refined GMRES
        dict(UNIT, name="solve_sphere64", kind="solve", shape="sphere", N=64, k=5.0, method="gmres", refined=True,
             tol=1e-12, restart=120),
        # an oscillatory solve on a torus, refined GMRES (n = 36k)
        dict(UNIT, name="solve_torus64", kind="solve", shape="torus", N=64, k=15.0, method="gmres", refined=True,
             tol=1e-11, restart=120),
        # refined BiCG on an ellipsoid of odd grid size (n = 24k)
        dict(UNIT, name="solve_ellipsoid67", kind="solve", shape="ellipsoid", N=67, k=12.0, method="bicg",
             refined=True, tol=1e-11, restart=40),
        # the reference driver's own default: [-2, 2]^3, Neumann, plain FP64 BiCG, a coarse grid
        dict(WIDE, name="bicg_neumann32", kind="solve", shape="sphere", N=32, k=2.0, method="bicg", refined=False,
             tol=1e-11, restart=40),
        # scattering of 16 plane waves by a torus in lockstep
        dict(UNIT, name="waves16_torus56", kind="waves", shape="torus", N=56, k=10.0, nrhs=16, tol=1e-11, restart=100),
        # an uneven batch of small ellipsoids solved together
        dict(UNIT, name="batch8_ellipsoids", kind="batch", shape="ellipsoid", N=32, k=5.0, nops=8, step=4, tol=1e-11),
        # from a distance grid to the tube arrays: what every new surface costs
        dict(UNIT, name="build_torus128", kind="build", shape="torus", N=128, k=20.0),
        # the field on a plane for a picture
        dict(UNIT, name="slice96_sphere48", kind="slice", shape="sphere", N=48, k=5.0, n2=96),
        # the gradients of a misfit at 64 receivers with respect to boundary data, wave number and weights
        dict(UNIT, name="gradient_bumpy45", kind="gradient", shape="bumpy", N=45, k=8.0, nrec=64, tol=1e-12),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["product", "product", "solve", "solve", "waves", "batch", "build", "slice", "gradient",
                       "combo"])
    k = round(rng.uniform(0.6, 20.0), 3)
    if kind == "product":
        shape = rng.choice(["sphere", "torus", "ellipsoid"])
        N = logint(48, 120) if shape == "torus" else logint(24, 128)
        return dict(UNIT, kind=kind, shape=shape, N=N, k=k, mode=rng.choice(["A", "AH", "pair"]),
                    dirichlet=rng.randint(0, 1))
    if kind == "solve":
        shape = rng.choice(["sphere", "torus", "ellipsoid"])
        refined = rng.random() < 0.75
        N = logint(48, 72) if shape == "torus" else logint(28, 72)
        if not refined:
            shape, N = "sphere", logint(24, 40)
        return dict(UNIT, kind=kind, shape=shape, N=N, k=min(k, N / 6.0), method=rng.choice(["gmres", "bicg"]),
                    refined=refined, tol=1e-11, restart=120)
    if kind == "waves":
        return dict(UNIT, kind=kind, shape="torus", N=logint(48, 60), k=round(rng.uniform(2.0, 10.0), 3),
                    nrhs=rng.randint(2, 24), tol=1e-11, restart=100)
    if kind == "batch":
        return dict(UNIT, kind=kind, shape="ellipsoid", N=logint(32, 40), k=round(rng.uniform(2.0, 6.0), 3),
                    nops=rng.randint(3, 9), step=rng.randint(1, 4), tol=1e-11)
    if kind == "build":
        return dict(UNIT, kind=kind, shape=rng.choice(["torus", "sphere"]), N=logint(48, 160), k=k)
    if kind == "slice":
        return dict(UNIT, kind=kind, shape="sphere", N=logint(28, 72), k=k, n2=logint(24, 112))
    if kind == "gradient":
        return dict(UNIT, kind=kind, shape="bumpy", N=logint(36, 48), k=round(rng.uniform(2.0, 8.0), 3),
                    nrec=logint(9, 150), tol=1e-12)
    return dict(WIDE, kind=kind, shape="sphere", N=logint(24, 44), k=round(rng.uniform(1.0, 4.0), 3), tol=1e-11,
                restart=60)


# ---------------------------------------------------------------- surfaces and inputs
def _params(case, N=None):
    return hz.params(N or case["N"], case["k"], int_l=case["lo"], int_u=case["hi"], factor=case["factor"],
                     dirichlet=case["dirichlet"])


def _turn(seed):
    """One of the 48 turns and reflections of the cube: (axis order, signs) for arrays and points in (y, x, z)."""
    rng = np.random.default_rng(seed)
    return tuple(int(a) for a in rng.permutation(3)), tuple(int(q) for q in rng.integers(0, 2, 3))


def _turned(d, seed):
    order, sign = _turn(seed)
    return np.ascontiguousarray(np.flip(np.transpose(d, order), [a for a in range(3) if sign[a]]))


def _grid(shape, N, lo, hi, axes=None):
    """The level set as a user's program has it: (N+1)^3 doubles in host memory, off the grid's symmetry planes."""
    h = (hi - lo) / N
    t = lo + np.arange(N + 1) * h
    Y, X, Z = t[:, None, None] - 0.11 * h, t[None, :, None] - 0.17 * h, t[None, None, :] - 0.05 * h
    if shape == "torus":
        d = 0.25 - np.sqrt((np.sqrt(X ** 2 + Y ** 2) - 0.6) ** 2 + Z ** 2)
    elif shape == "sphere":
        d = 0.25 * (hi - lo) - np.sqrt(X ** 2 + Y ** 2 + Z ** 2)
    elif shape == "ellipsoid":
        d = G.ellipsoid(N, axes=axes or (0.7, 0.5, 0.45), int_l=lo, int_u=hi, iters=25)
    else:
        d = hz.reinitialize(G.bumpy_sphere_levelset(N, int_l=lo, int_u=hi), N, h, 60)
    return np.broadcast_to(d, (N + 1,) * 3)


def _distance(case, seed):
    return _turned(_grid(case["shape"], case["N"], case["lo"], case["hi"]), seed)


def _source(case, seed):
    """A point inside the surface."""
    e = (np.random.default_rng(seed + 1).random(3) - 0.5) * 0.1
    if case["shape"] != "torus":
        return e
    order, sign = _turn(seed)
    c = np.array([0.0, 0.6, 0.0])[list(order)] * np.where(sign, -1.0, 1.0)  # (y, x, z)
    return e + c[[1, 0, 2]]


def _directions(m, seed):
    u = np.random.default_rng(seed + 2).standard_normal((m, 3))
    return u / np.linalg.norm(u, axis=1, keepdims=True)


def _density(xs, k, seed, m):
    """m densities on the tube: a few plane waves each, as boundary data and Krylov vectors are."""
    rng = np.random.default_rng(seed + 3)
    out = np.zeros((m, len(xs)), dtype=np.complex128)
    for r in range(m):
        for u in _directions(4, seed + 17 * r):
            out[r] += (rng.standard_normal() + 1j * rng.standard_normal()) * np.exp(1j * k * (xs @ u))
    return out


def _receivers(m, seed):
    return 0.95 * _directions(m, seed + 5)


def _batch(case):
    """(N, semi-axes, k) of the operators of a batch."""
    rng = np.random.default_rng(case["nops"])
    return [(case["N"] + case["step"] * i, tuple(rng.uniform(0.5, 0.7, 3)), case["k"]) for i in range(case["nops"])]


def _operator(case, d):
    op = hz.Operator(_params(case))
    op.set_distance(d)
    op.build()
    return op


def _combo_opts(case, p):
    eps = math.sqrt((case["hi"] - case["lo"]) / case["N"])
    return hz.dense_opts(hz.DENSE_COMBO, p, delta0=0.1 * eps, epsilon=eps, wavenum=case["k"], eta=-1.0)


def _options(case):
    meth = {"gmres": hz.GMRES, "bicg": hz.BICG}[case.get("method", "gmres")]
    prec = hz.PREC_F32_REFINED if case.get("refined", True) else hz.PREC_F64
    return hz.solve_opts(method=meth, precision=prec, tol=case["tol"], inner_tol=1e-6, restart=case.get("restart", 100))


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "batch":
        st["ops"] = []
        for N, axes, k in _batch(case):
            op = hz.Operator(_params(case, N))
            op.set_distance(_turned(_grid("ellipsoid", N, case["lo"], case["hi"], axes), seed + N))
            op.build()
            st["ops"].append(op)
        st["batch"] = hz.Batch(st["ops"])
        st["b"] = [op.rhs_point_source(_source(case, seed), hz.RHS_POINT_DIRICHLET) for op in st["ops"]]
        st["opts"] = hz.solve_opts(method=hz.BICGSTAB, precision=hz.PREC_F32_REFINED, tol=case["tol"])
        return st
    d = _distance(case, seed)
    if kind == "build":
        st["d"] = d
        return st
    if kind == "combo":
        op = hz.Operator(_params(case))
        op.set_combo(_combo_opts(case, op.p))
        op.set_distance(d)
        op.build()
        st["op"], st["opts"] = op, _options(case)
        st["b"] = op.rhs_point_source(_source(case, seed), hz.RHS_MONOPOLE_NEUMANN)
        return st
    op = st["op"] = _operator(case, d)
    if kind == "product":
        st["v"] = _density(op.tube()["xs"], case["k"], seed, 2)
    elif kind == "solve":
        kd = hz.RHS_POINT_DIRICHLET if case["dirichlet"] else hz.RHS_POINT_NEUMANN
        st["b"], st["opts"] = op.rhs_point_source(_source(case, seed), kd), _options(case)
        op.autotune()
    elif kind == "waves":
        st["b"], st["opts"] = op.rhs_plane_waves(_directions(case["nrhs"], seed)), _options(case)
    elif kind == "slice":
        st["v"] = _density(op.tube()["xs"], case["k"], seed, 1)[0]
    else:
        st["b"] = op.rhs_point_source(_source(case, seed), hz.RHS_POINT_DIRICHLET)
        st["rx"] = _receivers(case["nrec"], seed)
        st["target"], st["opts"] = _target(st["rx"], case["k"]), _options(case)
    return st


def _target(rx, k):
    """The field that the receivers should see: a point source's at the origin."""
    r = np.linalg.norm(rx, axis=1)
    return np.exp(1j * k * r) / (4 * PI * r)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "product":
        v, w = st["v"]
        if case["mode"] == "pair":
            return list(st["op"].matvec_pair(v, w, precision=hz.PREC_F64))
        return st["op"].matvec(v, precision=hz.PREC_F64, adjoint=case["mode"] == "AH")
    if kind in ("solve", "combo"):
        return st["op"].solve(st["b"], st["opts"])[0]
    if kind == "waves":
        return st["op"].solve_multi(st["b"], st["opts"])[0]
    if kind == "batch":
        return st["batch"].solve(st["b"], st["opts"])[0]
    if kind == "build":
        with _operator(case, st["d"]) as op:
            return op.tube()
    if kind == "slice":
        return st["op"].evaluate_slice(st["v"], axis=2, c=0.0, n2=case["n2"])
    J, g, dk, dw, _ = st["op"].misfit_gradient(st["b"], st["rx"], st["target"], opts=st["opts"])
    return dict(J=J, g=g, dk=dk, dw=dw)


# ---------------------------------------------------------------- work of one pass
PAIR = 40  # the reference's entry and its complex multiply-add (large3Dexample2.c:4471-4550)


def _points(case, N=None, axes=None):
    N = N or case["N"]
    h = (case["hi"] - case["lo"]) / N
    if case["kind"] == "combo":
        return 4 * PI * 1.0 * 2 * 0.9 * math.sqrt(h) / h ** 3  # both sides of the sphere of radius 1
    a, b, c = axes or (0.7, 0.5, 0.45)
    p = 1.6075  # Knud Thomsen's surface formula
    area = {"torus": 4 * PI * PI * 0.6 * 0.25, "sphere": 4 * PI * (0.25 * (case["hi"] - case["lo"])) ** 2,
            "ellipsoid": 4 * PI * (((a * b) ** p + (a * c) ** p + (b * c) ** p) / 3) ** (1 / p),
            "bumpy": 4 * PI * 0.25}[case["shape"]]
    return area * 2 * case["factor"] * h / h ** 3


def _products(case):
    """Products that a Krylov method cannot do without: about two a digit, more with the wave number."""
    return (2 + case["k"] / 4) * -math.log10(case["tol"]) / 2


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = [_points(case, N, axes) for N, axes, _ in _batch(case)]
        return {"bytes": sum(32 * m + 64 * m for m in n), "flops": sum(PAIR * m * m for m in n) * 2 * _products(case)}
    n = _points(case)
    if kind == "product":
        m = 2 if case["mode"] == "pair" else 1
        return {"bytes": (64 + 32 * m) * n, "flops": PAIR * n * n * m}
    if kind == "build":
        nodes = (case["N"] + 1) ** 3
        return {"bytes": 48 * nodes + 96 * n, "flops": 750 * nodes}
    if kind == "slice":
        return {"bytes": 80 * n + 16 * case["n2"] ** 2, "flops": PAIR * n * case["n2"] ** 2}
    per = {"solve": 2 if case.get("method") == "bicg" else 1, "combo": 3, "waves": 0.7 + 0.3 * case.get("nrhs", 1),
           "gradient": 2}[kind]
    cols = case.get("nrhs", 1)
    return {"bytes": (64 + 32 * cols) * n, "flops": PAIR * n * n * per * _products(case)}


# ---------------------------------------------------------------- the same in plain torch, 64 bits
def _weno(f, h):
    """One-sided fifth-order WENO derivatives of seven shifted grids (weno.c:259-345)."""
    eps = 1e-12
    ih = 1.0 / h
    aa, bb, cc, dd, ee, ff = [(f[i + 1] - f[i]) * ih for i in range(6)]
    df = (-bb + 7.0 * (cc + dd) - ee) / 12.0
    aa, bb, cc, dd, ee = bb - aa, cc - bb, dd - cc, ee - dd, ff - ee

    def side(p, q, r, s):  # p next to the node, s outermost
        i0 = 13.0 * (s - r) * (s - r) + 3.0 * (s - 3.0 * r) * (s - 3.0 * r)
        i1 = 13.0 * (r - q) * (r - q) + 3.0 * (r + q) * (r + q)
        i2 = 13.0 * (q - p) * (q - p) + 3.0 * (3.0 * q - p) * (3.0 * q - p)
        a0 = 1.0 / ((eps + i0) * (eps + i0))
        a1 = 6.0 / ((eps + i1) * (eps + i1))
        a2 = 3.0 / ((eps + i2) * (eps + i2))
        w1 = 1.0 / (a0 + a1 + a2)
        return a0 * w1, a2 * w1

    w0, w2 = side(bb, cc, dd, ee)
    pos = df + w0 * (ee - 2.0 * dd + cc) / 3.0 + (w2 - 0.5) * (dd - 2.0 * cc + bb) / 6.0
    w0, w2 = side(dd, cc, bb, aa)
    neg = df - w0 * (aa - 2.0 * bb + cc) / 3.0 - (w2 - 0.5) * (bb - 2.0 * cc + dd) / 6.0
    return pos, neg


def _gradient(d, N, h):
    """Upwind gradient (distance_application3D.c:56-140): axes x = 1, y = 0, z = 2, mirrored at the faces."""
    out = []
    i = torch.arange(N + 1, device=d.device)
    for ax in (1, 0, 2):
        f = []
        for m in range(-3, 4):
            q = (i + m).abs()
            f.append(d.index_select(ax, torch.where(q > N, 2 * N - q, q)))
        p, n = _weno(f, h)
        z = torch.zeros_like(p)
        pp, pm, np_, nm = torch.maximum(z, p), torch.minimum(z, p), torch.maximum(z, n), torch.minimum(z, n)
        out.append(torch.where(d > 0, torch.where(pm.abs() > np_.abs(), pm, np_),
                               torch.where(pp.abs() > nm.abs(), pp, nm)))
    return out


def _curvatures(d, N, h):
    """Mean and Gaussian curvature (distance_application3D.c:35-53) with limited differences."""
    ix = [torch.arange(N + 1, device=d.device).view([-1 if a == b else 1 for b in range(3)]) for a in range(3)]

    def less(a, b):
        return torch.where(a.abs() < b.abs(), a, b)

    def second(ax, xorder):
        def at(m):
            return torch.roll(d, -m, ax)
        l0 = d
        fwd = (2.0 * l0 - 5.0 * at(1) + 4.0 * at(2) - at(3)) / (h * h)
        mid = (at(1) - 2.0 * l0 + at(-1)) / (h * h)
        bwd = (2.0 * l0 - 5.0 * at(-1) + 4.0 * at(-2) - at(-3)) / (h * h)
        dpp, dp, dn, dnn = at(2) - at(1), at(1) - l0, l0 - at(-1), at(-1) - at(-2)
        a, b = dp * dnn <= 0.0, dpp * dn <= 0.0
        both = less(less(fwd, mid), bwd) if xorder else less(less(fwd, bwd), mid)
        r = torch.where(a & b, both, torch.where(a, less(fwd, mid), torch.where(b, less(bwd, mid), mid)))
        c = ix[ax]
        r = torch.where(c < 3, less(fwd, mid), torch.where(c > N - 3, less(bwd, mid), r))
        r = torch.where(c == 0, 2.0 * (at(1) - l0) / (h * h), r)
        return torch.where(c == N, 2.0 * (at(-1) - l0) / (h * h), r)

    def cross(ua, va):
        def at(u, v):
            return torch.roll(d, (-u, -v), (ua, va))
        coef = (1.0, -4.0, 3.0)
        corner = at(1, 1) - at(-1, 1) - at(1, -1) + at(-1, -1)
        fin = torch.full_like(d, 1000000.0)
        for si in (-1, 0, 1):
            for sj in (-1, 0, 1):
                if si == 0 and sj == 0:
                    v = corner
                else:
                    v = torch.zeros_like(d)
                    if si == 0:
                        for c in (2, 1, 0):
                            v = v + (-1.0 * sj * coef[2 - c]) * (at(1, sj * c) - at(-1, sj * c))
                    elif sj == 0:
                        for c in (2, 1, 0):
                            v = v + (-1.0 * si * coef[2 - c]) * (at(si * c, 1) - at(si * c, -1))
                    else:
                        for ci in (2, 1, 0):
                            for cj in (2, 1, 0):
                                v = v + (coef[2 - ci] * coef[2 - cj] * (si * sj)) * at(si * ci, sj * cj)
                fin = less(v, fin)
        ca, cb = ix[ua], ix[va]
        edge = (ca < 2) | (ca > N - 2) | (cb < 2) | (cb > N - 2)
        r = torch.where(edge, corner, fin) / (4.0 * h * h)
        return torch.where((ca == 0) | (ca == N) | (cb == 0) | (cb == N), torch.zeros_like(r), r)

    dxx, dyy, dzz = second(1, True), second(0, False), second(2, False)
    dxy, dxz, dyz = cross(0, 1), cross(1, 2), cross(0, 2)
    return -0.5 * (dxx + dyy + dzz), (dxx * dyy + dyy * dzz + dxx * dzz) - (dxy * dxy + dyz * dyz + dxz * dxz)


def _trilinear(g, i, j, k, lx, ly, lz, h):
    """Interpolation in the cell (i, j, k) = (y, x, z) (interpolate3D.c:49-53)."""
    v = [g[i + a, j + b, k + c] for b in (0, 1) for a in (0, 1) for c in (0, 1)]  # x, then y, then z
    hx, hy, hz_ = h - lx, h - ly, h - lz
    return (v[0] * hx * hy * hz_ + v[1] * hx * hy * lz + v[2] * hx * ly * hz_ + v[3] * hx * ly * lz +
            v[4] * lx * hy * hz_ + v[5] * lx * hy * lz + v[6] * lx * ly * hz_ + v[7] * lx * ly * lz) / (h * h * h)


def _surface(d, N, lo, hi, k, factor, combo=None):
    """The tube and its arrays (large3Dexample2.c:548-597, 4340-4452) as a dict of torch tensors."""
    d = torch.from_numpy(d).cuda()
    h = (hi - lo) / N
    g = _gradient(d, N, h)
    mc, gc = _curvatures(d, N, h)
    eps, tau = factor * h, 2.0 * h
    if combo:
        node = ((d.abs() <= combo[1]) & (d.abs() >= combo[0])).nonzero()
    else:
        node = (d.abs() <= eps).nonzero()
    i, j, l = node.unbind(1)
    dd = d[i, j, l]
    x = [lo + h * q.double() - dd * gg[i, j, l] for q, gg in zip((j, i, l), g)]
    jac = 1 + 2.0 * dd * mc[i, j, l] + dd * dd * gc[i, j, l]
    cj, ci, cl = [((q - lo) / h).long() for q in x]
    lx, ly, lz = [q - lo - c.double() * h for q, c in zip(x, (cj, ci, cl))]
    n = [_trilinear(gg, ci, cj, cl, lx, ly, lz, h) for gg in g]
    for _ in range(2):
        r = torch.sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2])
        n = [q / r for q in n]
    cm, cg = [_trilinear(q, ci, cj, cl, lx, ly, lz, h) for q in (mc, gc)]
    reg = -(cm / (4.0 * PI * tau) - 5.0 * tau * (2.0 * cm) * (4.0 * cm * cm - cg) / (512.0 * PI)
            - 25.0 * tau * (2.0 * cm) * cg / (1536.0 * PI) + k * k * tau * 2.0 * cm / (48.0 * PI))
    t = dict(idx=(i * (N + 1) + j) * (N + 1) + l, xs=torch.stack(x, 1), nrm=torch.stack(n, 1), jac=jac, reg=reg)
    if combo:  # SineWeight (functions.c:835-866)
        s = (dd / combo[1]).abs()
        w = torch.exp(0.5 / ((s - 0.1) * (s - 1.0))) * (-759.2781934172483 * s + 446.2604260472818)
        w = torch.where((s <= combo[0] / combo[1]) | (s >= 1.0), torch.zeros_like(w), w) / (2.0 * combo[1])
        t["w"], t["dist"] = h * h * h * jac * w, dd.abs()
        return t, tau
    t["delta"] = (1.0 / (2.0 * eps)) * (1.0 + torch.cos(PI * dd / eps))
    t["w"] = h * h * h * t["delta"] * jac
    t["dreg"] = -(2.0 * k * tau * 2.0 * cm / (48.0 * PI))
    return t, tau


def _layers(x, nx, t, k):
    """rho, e^{ik rho} and (x - y).n for the rows x against every tube point y; n of the rows if nx is given."""
    dif = [x[:, a, None] - t["xs"][None, :, a] for a in range(3)]
    rho = torch.sqrt(dif[0] * dif[0] + dif[1] * dif[1] + dif[2] * dif[2])
    if nx is None:
        inn = sum(dif[a] * t["nrm"][None, :, a] for a in range(3))
    else:
        inn = sum(dif[a] * nx[:, a, None] for a in range(3))
    del dif
    return rho, torch.polar(torch.ones_like(rho), k * rho), inn


def _rows(t, k, tau, dirichlet, a, b, dk=False):
    """Rows a:b of the matrix without its diagonal term (large3Dexample2.c:4463-4564), or of its k-derivative."""
    rho, e, inn = _layers(t["xs"][a:b], None if dirichlet else t["nrm"][a:b], t, k)
    near = rho <= tau
    rho = torch.where(near, torch.ones_like(rho), rho)
    if dk:
        m = e * (inn * (-k / (4 * PI * rho)))
        reg = t["dreg"]
    else:
        m = e * torch.complex(-1.0 / rho, torch.full_like(rho, k)) * (inn / (4 * PI * rho * rho))
        reg = t["reg"]
    reg = (reg[None, :] if dirichlet else reg[a:b, None]).expand_as(rho)
    return torch.where(near, reg.to(m.dtype), m) * t["w"][None, :]


def _combo_rows(t, k, tau, a, b, eta=-1.0):
    """Rows of the Combo matrix (HelmholtzKernel.c:399-607)."""
    x, nx = t["xs"][a:b], t["nrm"][a:b]
    rho, e, inn = _layers(x, nx, t, k)
    near = rho <= tau
    rho = torch.where(near, torch.ones_like(rho), rho)
    part = e * torch.complex(-1.0 / rho, torch.full_like(rho, k)) * (-inn / (4 * PI * rho * rho))
    part = torch.where(near, t["reg"][a:b, None].expand_as(rho).to(part.dtype), part)
    y = [x[:, c, None] + t["dist"][None, :] * nx[:, c, None] - t["xs"][None, :, c] for c in range(3)]
    r = torch.sqrt(y[0] * y[0] + y[1] * y[1] + y[2] * y[2])
    g = torch.polar(1.0 / r, k * r)
    ip1 = nx @ t["nrm"].T
    ip2 = sum(y[c] * nx[:, c, None] for c in range(3)) / r
    ip3 = sum(y[c] * t["nrm"][None, :, c] for c in range(3)) / r
    hyp = g * (torch.complex(-1.0 / r, torch.full_like(r, k)) * (ip1 / r)
               + torch.complex(3.0 / (r * r) - k * k, -3.0 * k / r) * (ip2 * ip3))
    m = (-1j * eta * part + hyp / (4 * PI)) * t["w"][None, :]
    return m


def _chunk(n):
    return max(1, (48 << 20) // max(n, 1))


def _matrix(rows, n, diag):
    m = torch.empty(n, n, dtype=torch.complex128, device="cuda")
    for a in range(0, n, _chunk(n)):
        b = min(n, a + _chunk(n))
        m[a:b] = rows(a, b)
    m.diagonal().add_(diag)
    return m


def _gmres(A, b, tol=1e-14, most=400):
    """Unrestarted GMRES on a stored matrix, twice with the true residual."""
    x = torch.zeros_like(b)
    for _ in range(2):
        r = b - A @ x
        beta = torch.linalg.vector_norm(r)
        if float(beta) <= 1e-15 * float(torch.linalg.vector_norm(b)):
            break
        V, H = [r / beta], np.zeros((most + 1, most), dtype=np.complex128)
        for j in range(most):
            w = A @ V[j]
            Q = torch.stack(V, 1)
            for _ in range(2):
                c = Q.mH @ w
                w = w - Q @ c
                H[: j + 1, j] += c.cpu().numpy()
            nw = torch.linalg.vector_norm(w)
            H[j + 1, j] = float(nw)
            V.append(w / nw)
            g = np.zeros(j + 2, dtype=np.complex128)
            g[0] = float(beta)
            y, *_ = np.linalg.lstsq(H[: j + 2, : j + 1], g, rcond=None)
            if np.linalg.norm(g - H[: j + 2, : j + 1] @ y) <= tol * float(beta):
                break
        x = x + torch.stack(V[: len(y)], 1) @ torch.from_numpy(y).cuda()
    return x


def _point_source(t, src, k, dirichlet):
    """The field of a point source on the surface, or its derivative along the outward normal."""
    dif = t["xs"] - torch.from_numpy(src).cuda()
    r = torch.sqrt((dif * dif).sum(1))
    if dirichlet:
        return torch.polar(1.0 / (4 * PI * r), k * r)
    dn = -(dif * t["nrm"]).sum(1) / r
    return torch.polar(dn / (4 * PI * r * r), k * r) * torch.complex(-torch.ones_like(r), k * r)


def exact(case, seed):
    kind, k, dirichlet = case["kind"], case["k"], case["dirichlet"]
    if kind == "batch":
        out = []
        for N, axes, kk in _batch(case):
            d = _turned(_grid("ellipsoid", N, case["lo"], case["hi"], axes), seed + N)
            t, tau = _surface(d, N, case["lo"], case["hi"], kk, case["factor"])
            A = _matrix(lambda a, b: _rows(t, kk, tau, dirichlet, a, b), len(t["w"]), 0.5)
            out.append(_gmres(A, _point_source(t, _source(case, seed), kk, 1)))
        return out
    d = _distance(case, seed)
    combo = None
    if kind == "combo":
        eps = math.sqrt((case["hi"] - case["lo"]) / case["N"])
        combo = (0.1 * eps, eps)
    t, tau = _surface(d, case["N"], case["lo"], case["hi"], k, case["factor"], combo)
    n = len(t["w"])
    if kind == "build":
        return {q: t[q] for q in ("idx", "xs", "nrm", "delta", "jac", "reg", "w")}
    if kind == "product":
        v, w = torch.from_numpy(_density(t["xs"].cpu().numpy(), k, seed, 2)).cuda()
        q, qt = 0.5 * v, 0.5 * (w if case["mode"] == "pair" else v)
        for a in range(0, n, _chunk(n)):
            b = min(n, a + _chunk(n))
            m = _rows(t, k, tau, dirichlet, a, b)
            if case["mode"] != "AH":
                q[a:b] += m @ v
            if case["mode"] != "A":
                qt += m.mH @ (w if case["mode"] == "pair" else v)[a:b]
        return [q, qt] if case["mode"] == "pair" else (qt if case["mode"] == "AH" else q)
    if kind == "slice":
        v = torch.from_numpy(_density(t["xs"].cpu().numpy(), k, seed, 1)[0]).cuda()
        n2, lo, hi, N = case["n2"], case["lo"], case["hi"], case["N"]
        h, step = (hi - lo) / N, (hi - lo) / (n2 - 1)
        u = lo + torch.arange(n2, device="cuda", dtype=torch.float64) * step
        x = torch.stack([u[:, None].expand(n2, n2), u[None, :].expand(n2, n2), torch.zeros(n2, n2).cuda().double()], 2)
        x = x.reshape(-1, 3)
        out = torch.empty(n2 * n2, dtype=torch.complex128, device="cuda")
        for a in range(0, n2 * n2, _chunk(n)):
            b = min(n2 * n2, a + _chunk(n))
            rho, e, inn = _layers(x[a:b], None, t, k)
            m = e * torch.complex(-1.0 / rho, torch.full_like(rho, k)) * (inn / (4 * PI * rho * rho))
            out[a:b] = torch.where(rho > tau, m, torch.zeros_like(m)) @ (v * t["w"])
        # the field is left out inside the body: where the interpolated level set is positive
        c = torch.floor((x - lo) / h).long()
        ok = ((c >= 0) & (c < N)).all(1)
        c = c.clamp(0, N - 1)
        f = (x - lo) / h - c.double()
        g = torch.from_numpy(d).cuda()
        acc = sum((f[:, 1] if a else 1 - f[:, 1]) * (f[:, 0] if b else 1 - f[:, 0]) * (f[:, 2] if e else 1 - f[:, 2])
                  * g[c[:, 1] + a, c[:, 0] + b, c[:, 2] + e] for a in (0, 1) for b in (0, 1) for e in (0, 1))
        return torch.where(ok & (acc > 0), torch.zeros_like(out), out).reshape(n2, n2)
    if kind == "combo":
        A = _matrix(lambda a, b: _combo_rows(t, k, tau, a, b), n, -0.5j)
        src = torch.from_numpy(_source(case, seed)).cuda()
        r = torch.sqrt(((t["xs"] - src) ** 2).sum(1))
        s, c = torch.sin(k * r), torch.cos(k * r)
        return _gmres(A, torch.complex(s / r + c / (k * r * r), s / (k * r * r) - c / r))
    A = _matrix(lambda a, b: _rows(t, k, tau, dirichlet, a, b), n, 0.5)
    if kind == "waves":
        dirs = torch.from_numpy(_directions(case["nrhs"], seed)).cuda()
        return torch.stack([_gmres(A, torch.polar(torch.ones(n, device="cuda", dtype=torch.float64),
                                                  k * (t["xs"] @ u))) for u in dirs])
    x = _gmres(A, _point_source(t, _source(case, seed), k, dirichlet))
    if kind == "solve":
        return x
    rx = _receivers(case["nrec"], seed)
    rho, e, inn = _layers(torch.from_numpy(rx).cuda(), None, t, k)
    E = e * torch.complex(-1.0 / rho, torch.full_like(rho, k)) * (inn / (4 * PI * rho * rho)) * t["w"]
    dE = e * (inn * (-k / (4 * PI * rho))) * t["w"]
    r = E @ x - torch.from_numpy(_target(rx, k)).cuda()
    lam = _gmres(A.mH.contiguous(), E.mH @ r)
    dA = torch.cat([_rows(t, k, tau, dirichlet, a, min(n, a + _chunk(n)), dk=True) @ x
                    for a in range(0, n, _chunk(n))])
    dk = 2 * torch.vdot(r, dE @ x).real - 2 * torch.vdot(lam, dA).real
    dw = torch.where(t["w"] != 0, (lam.conj() * x).real / t["w"], torch.zeros_like(t["w"]))
    return dict(J=float((r.abs() ** 2).sum()), g=2 * lam, dk=float(dk), dw=dw)
