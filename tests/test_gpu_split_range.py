"""The rule that sends an FP64 product to the split sweep (sweep_split.cu) or
to the sweep in FP64 instructions, on both sides of each of its bounds, entry by
entry: a density on one point gives a column of the oracle's matrix."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def two_spheres(N):
    """Two spheres; a tile of 256 points in blocked order holds points of both."""
    t = -1 + np.arange(N + 1) * (2.0 / N)
    Y, X, Z = t[:, None, None], t[None, :, None], t[None, None, :]
    f = [0.2 - np.sqrt((X - c) ** 2 + (Y - 0.01) ** 2 + (Z - 0.02) ** 2) for c in (-0.6, 0.6)]
    return np.maximum(*f)


def column_errors(hz, oracle, p, d, count, rng, mode=0):
    """Errors of columns of A and A^H over their entries' size, with max(rho,
    tau) and max |x|: sources with the closest far neighbours and `count`
    others.  An entry's size has |x_t - x_s| for the projection
    (w (k + 1/rho) / (4 pi rho))."""
    import oracle as O
    po = O.make_params(p.N, p.wave, int_l=p.int_l, int_u=p.int_u, factor=p.factor, tau_factor=p.tau_factor,
                       dirichlet=p.dirichlet, interior=p.interior)
    tp = oracle.pipeline(po, d)
    are, aim = oracle.dense(po, tp)
    xs, w, reg = np.asarray(tp["xs"]).reshape(-1, 3), np.asarray(tp["w"]), np.asarray(tp["reg"])
    tau = p.tau_factor * (p.int_u - p.int_l) / p.N
    with hz.Operator(p) as op:
        op.set_distance(d)
        op.set_f64_mode(mode)
        n = op.build()
        assert n == len(w)
        near = np.full(n, np.inf)
        for i in range(0, n, 512):
            r = np.linalg.norm(xs[i:i + 512, None] - xs[None], axis=2)
            near[i:i + 512] = np.where(r > tau, r, np.inf).min(axis=1)
        pick = np.concatenate([np.argsort(near)[:count], rng.integers(0, n, count)])
        for adjoint in (False, True):
            for s in pick:
                v = np.zeros(n, dtype=complex)
                v[s] = 1 - 0.5j
                q = op.matvec(v, adjoint=adjoint)
                A = (are[s] - 1j * aim[s]) if adjoint else are[:, s] + 1j * aim[:, s]
                rho = np.linalg.norm(xs - xs[s], axis=1)
                far = rho > tau
                size = np.abs(np.where(p.dirichlet ^ adjoint, reg[s], reg))
                size[far] = (p.wave + 1 / rho[far]) / (4 * np.pi * rho[far])
                size *= w if adjoint else w[s]
                err = np.abs(q - A * v[s]) / abs(v[s])
                err[s] = max(0.0, err[s] - 2.0 ** -52)  # beside the diagonal's 1/2
                yield err[size > 0] / size[size > 0], np.maximum(rho, tau)[size > 0], np.abs(xs).max()


def columns(hz, oracle, p, d, count, rng):
    """Largest error of an entry over its bound: r^2 off by 2^-43, three halves
    of it in the entry, the rest of the split arithmetic 2^-44; coordinates times
    k 2^-53 of |x| each, seven times that over rho."""
    worst, n = 0.0, 0
    for err, rho, x in column_errors(hz, oracle, p, d, count, rng):
        worst, n = max(worst, float(np.max(err / (2.0 ** -42 + 2.0 ** -50 * x / rho)))), len(err)
    return worst, n


@pytest.mark.parametrize("tau_factor", [2.0, 1.0, 0.999, 0.25, 0.02, 1e-3, 1e-6])
@pytest.mark.parametrize("k,dirichlet", [(5.0, 1), (0.5, 0)])
def test_near_field_radius(hz, oracle, tau_factor, k, dirichlet):
    """Pairs down to tau, where the fixed-point r^2 of a tile keeps few bits of
    itself."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    p = hz.params(24, k, int_l=-1.0, int_u=1.0, factor=3.0, tau_factor=tau_factor, dirichlet=dirichlet)
    worst, n = columns(hz, oracle, p, G.sphere(24, radius=0.5, center=(0.011, 0.017, 0.005)), 12,
                       np.random.default_rng(1))
    assert n >= 2048 and worst <= 1.0


@pytest.mark.parametrize("tau_factor", [2.0, 1.0])
def test_wide_tiles(hz, oracle, tau_factor):
    """Tiles of 20 grid steps, whose r^2 has an absolute error of 2^-52 of their
    squared size."""
    p = hz.params(48, 9.0, int_l=-1.0, int_u=1.0, factor=3.0, tau_factor=tau_factor, dirichlet=1)
    worst, n = columns(hz, oracle, p, two_spheres(48), 40, np.random.default_rng(2))
    assert n >= 2048 and worst <= 1.0


@pytest.mark.parametrize("half,k,dirichlet", [
    (1e-9, 1 / 64, 1), (3e-10, 1 / 64, 0), (1e-10, 1 / 64, 1),            # k tau far below 2^-28
    (1.0, 2.0 ** -28 * 6.0 * 0.999, 1), (1.0, 2.0 ** -28 * 6.0 * 1.001, 0),  # tau = 1/6: on both sides of it
    (1e-7, 5e7, 1), (1e7, 5e-7, 0), (1e20, 5e-20, 1), (1e-15, 5e15, 0),   # other units of length
    (100.0, 0.01, 1)])
def test_units_of_length(hz, oracle, half, k, dirichlet):
    """k times the box decides, not k."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    d = G.sphere(24, radius=0.5, center=(0.011, 0.017, 0.005)) * half
    p = hz.params(24, k, int_l=-half, int_u=half, factor=3.0, dirichlet=dirichlet)
    worst, n = columns(hz, oracle, p, d, 8, np.random.default_rng(3))
    assert n >= 2048 and worst <= 1.0
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        V = np.exp(1j * np.outer([1, 2, 3], np.arange(n) / n))
        one = np.array([op.matvec(v) for v in V])
        assert np.max(np.abs(op.matvec_multi(V, precision=hz.PREC_F64) - one)) <= 2.0 ** -42 * 4
        pq, pt = op.matvec_pair(V[0], V[1])
        assert np.max(np.abs(pq - one[0])) <= 2.0 ** -42 * 4
        assert np.max(np.abs(pt - op.matvec(V[1], adjoint=True))) <= 2.0 ** -42 * 4


@pytest.mark.parametrize("k,dirichlet", [(5.0, 1), (4.0, 0)])
def test_entries_in_both_arithmetics(hz, oracle, k, dirichlet):
    """Split arithmetic: entries off by 2^-46.5 of themselves, root mean square
    (and by no more than the other tests' bound); FP64 instructions by less than
    a quarter of that."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    p = hz.params(24, k, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=dirichlet)
    d = G.sphere(24, radius=0.5, center=(0.011, 0.017, 0.005))

    def rms(mode):
        e = [e for e, _, _ in column_errors(hz, oracle, p, d, 20, np.random.default_rng(5), mode=mode)]
        return float(np.sqrt(np.mean(np.concatenate(e) ** 2)))

    split, plain = rms(hz.F64_SPLIT), rms(hz.F64_PLAIN)
    assert split <= 2.0 ** -46 and plain <= split / 4


def test_switching_the_arithmetic(hz):
    """hz_set_f64_mode before and after the build, in products, columns, solves
    (whose graphs hold the sweep's launches), gradients and batches."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    p = hz.params(24, 5.0, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=1)
    d = G.sphere(24, radius=0.5, center=(0.011, 0.017, 0.005))
    rx = G.random_sphere_points(5, 0.9, seed=6)
    with hz.Operator(p) as op, hz.Operator(p) as first:
        first.set_f64_mode(hz.F64_PLAIN)
        for o in (op, first):
            o.set_distance(d)
            n = o.build()
        v = np.exp(1j * np.arange(n) / n)

        def outputs(o):
            q, qt = o.matvec_pair(v, v)
            x, info = o.solve(v, method=hz.BICG, precision=hz.PREC_F64, tol=1e-9)
            g = o.misfit_gradient(v, rx, np.ones(5, dtype=complex), method=hz.GMRES, precision=hz.PREC_F64, tol=1e-9)
            with hz.Batch([o]) as b:
                bq = b.matvec([v], precision=hz.PREC_F64)[0]
            return [o.matvec(v), o.matvec(v, adjoint=True), q, qt, o.matvec_multi([v, 2 * v], precision=hz.PREC_F64),
                    x, g[1], np.array([g[0], g[2]]), bq]

        split, plain = outputs(op), outputs(first)
        for a, b in zip(split, plain):
            assert not np.array_equal(a, b) and np.max(np.abs(a - b)) <= 1e-7 * np.max(np.abs(b))
        for mode, want in ((hz.F64_PLAIN, plain), (hz.F64_SPLIT, split)):
            op.set_f64_mode(mode)
            for a, b in zip(outputs(op), want):
                assert np.array_equal(a, b)
            op.build()
            for a, b in zip(outputs(op), want):
                assert np.array_equal(a, b)
        with pytest.raises(hz.HzError) as e:
            op.set_f64_mode(2)
        assert e.value.code == hz.HZ_ERR_ARG


@pytest.mark.parametrize("N,kh", [(24, 0.41), (24, 0.43), (24, 0.5), (24, 0.79), (34, 0.49), (34, 0.7), (44, 0.79)])
def test_smooth_densities_lose_nothing(hz, N, kh):
    """Products of plane-wave densities, A and A^H of both problems, against rows
    in long double: what runs by default is off by no more than the FP64
    instructions (5 % for the sample of rows)."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    LD, k = np.longdouble, kh * N / 2
    err = np.zeros(2)
    for dirichlet in (1, 0):
        rng = np.random.default_rng(N)
        with hz.Operator(hz.params(N, k, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=dirichlet)) as op:
            op.set_distance(G.sphere(N, radius=0.5, center=(0.011, 0.017, 0.005)))
            n = op.build()
            t = op.tube()
            x, nrm, w, reg = t["xs"].reshape(-1, 3), t["nrm"].reshape(-1, 3).astype(LD), t["w"], t["reg"].astype(LD)
            V = []
            for _ in range(4):
                u = rng.standard_normal((4, 3))
                a = rng.standard_normal(4) + 1j * rng.standard_normal(4)
                V.append(np.exp(1j * k * (x @ (u / np.linalg.norm(u, axis=1)[:, None]).T)) @ a)
            rows = rng.choice(n, 32, replace=False)
            for adjoint in (False, True):
                src = bool(dirichlet) != adjoint  # whose normal the entry has
                want = np.empty((len(V), len(rows)), dtype=np.clongdouble)
                for i, r in enumerate(rows):
                    D = x[r].astype(LD) - x.astype(LD)
                    rho = np.sqrt((D * D).sum(axis=1))
                    far = np.sqrt(((x[r] - x) ** 2).sum(axis=1)) > op.p.tau_factor * 2.0 / N
                    rho[~far] = 1
                    c, s = np.cos(LD(k) * rho), np.sin(LD(k) * rho)
                    f = (D * (nrm if src else nrm[r])).sum(axis=1) / (4 * np.arctan(LD(1)) * 4 * rho * rho)
                    e = (-(c / rho + LD(k) * s) + 1j * (LD(k) * c - s / rho)) * f
                    e = np.where(far, -e.conj() if adjoint else e, (reg if src else reg[r]) + 0j)
                    e = e * (w[r] if adjoint else w).astype(LD)
                    want[:, i] = [(e * v).sum() + v[r] / 2 for v in V]
                for m, mode in enumerate((hz.F64_SPLIT, hz.F64_PLAIN)):
                    op.set_f64_mode(mode)
                    got = np.array([op.matvec(v, adjoint=adjoint)[rows] for v in V])
                    err[m] += float((np.abs(got - want) ** 2).sum() / (np.abs(want) ** 2).sum())
    assert err[0] <= 1.05 ** 2 * err[1]


def rms_errors(hz, op, adjoint, V, rows):
    """Root mean square error of the default product and of the one in FP64
    instructions, against rows in long double."""
    LD, p = np.longdouble, op.p
    t = op.tube()
    x, nrm, w, reg = t["xs"].reshape(-1, 3), t["nrm"].reshape(-1, 3).astype(LD), t["w"], t["reg"].astype(LD)
    src, k = bool(p.dirichlet) != adjoint, LD(p.wave)
    want = np.empty((len(V), len(rows)), dtype=np.clongdouble)
    for i, r in enumerate(rows):
        D = x[r].astype(LD) - x.astype(LD)
        rho = np.sqrt((D * D).sum(axis=1))
        far = np.sqrt(((x[r] - x) ** 2).sum(axis=1)) > p.tau_factor * (p.int_u - p.int_l) / p.N
        rho[~far] = 1
        c, s = np.cos(k * rho), np.sin(k * rho)
        f = (D * (nrm if src else nrm[r])).sum(axis=1) / (4 * np.arctan(LD(1)) * 4 * rho * rho)
        e = (-(c / rho + k * s) + 1j * (k * c - s / rho)) * f
        e = np.where(far, -e.conj() if adjoint else e, (reg if src else reg[r]) + 0j)
        e = e * (w[r] if adjoint else w).astype(LD)
        want[:, i] = [(e * v).sum() + v[r] / 2 for v in V]
    out = []
    for mode in (hz.F64_SPLIT, hz.F64_PLAIN):
        op.set_f64_mode(mode)
        got = np.array([op.matvec(v, adjoint=adjoint)[rows] for v in V])
        out.append(float(np.sqrt(np.mean(np.abs(got - want) ** 2))))
    return out


@pytest.mark.parametrize("N,kh", [(22, 0.055), (22, 0.36), (24, 0.05), (24, 0.11), (24, 0.23), (26, 0.1), (26, 0.17),
                                  (30, 0.04), (30, 0.07), (30, 0.1), (36, 0.033), (36, 0.05)])
@pytest.mark.parametrize("dirichlet", [0, 1])
def test_long_waves_lose_nothing(hz, N, kh, dirichlet):
    """Plane waves of few points and of wavelengths up to 100 grid steps, A and
    A^H by themselves.  256 real samples a side give the root mean square to 4.4 %
    for normal errors; 1.25 is four times the ratio's 6.2 %."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    k, rng = kh * N / 2, np.random.default_rng(N)
    with hz.Operator(hz.params(N, k, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=dirichlet)) as op:
        op.set_distance(G.sphere(N, radius=0.5, center=(0.011, 0.017, 0.005)))
        n = op.build()
        x, V = op.tube()["xs"].reshape(-1, 3), []
        for _ in range(4):
            u = rng.standard_normal((4, 3))
            a = rng.standard_normal(4) + 1j * rng.standard_normal(4)
            V.append(np.exp(1j * k * (x @ (u / np.linalg.norm(u, axis=1)[:, None]).T)) @ a)
        rows = rng.choice(n, 32, replace=False)
        for adjoint in (False, True):
            split, plain = rms_errors(hz, op, adjoint, V, rows)
            assert split <= 1.25 * plain


@pytest.mark.parametrize("shape,N,k,dirichlet,interior,half", [
    ("sphere", 24, 5.0, 1, 0, 1.0), ("sphere", 27, 4.8, 0, 1, 1.0), ("sphere", 31, 3.0, 0, 0, 2.0),
    ("torus", 36, 7.0, 1, 0, 1.0), ("torus", 36, 2.0, 0, 1, 1.0), ("ellipsoid", 33, 6.0, 1, 1, 1.0)])
def test_split_forms_against_plain(hz, shape, N, k, dirichlet, interior, half):
    """Every form of the split products inside its range (the arithmetics differ,
    so it ran), against FP64 instructions: A, A^H, the fused pass, blocks of 4, 8
    and 16 columns with their remainders, dA/dk.  Entries within 2^-44 a side, a
    row's sum |A_ts p_s| below 4 max |p| (8 on the torus)."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    d = (G.sphere(N, radius=0.5 * half, center=(0.011, 0.017, 0.005), int_l=-half, int_u=half) if shape == "sphere" else
         G.torus(N) if shape == "torus" else G.ellipsoid(N, axes=(0.7, 0.6, 0.55)))
    p = hz.params(N, k, int_l=-half, int_u=half, factor=2.0 if shape == "torus" else 3.0, dirichlet=dirichlet,
                  interior=interior)
    rng = np.random.default_rng(N)
    rx = half * G.random_sphere_points(5, 0.9, seed=6)
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        V = np.exp(2j * np.pi * rng.random((21, n)))
        b = np.exp(1j * np.arange(n) / n)
        out = []
        for mode in (hz.F64_SPLIT, hz.F64_PLAIN):
            op.set_f64_mode(mode)
            q = [op.matvec(V[0]), op.matvec(V[1], adjoint=True), *op.matvec_pair(V[0], V[1])]
            for m in (1, 3, 4, 5, 8, 9, 16, 21):
                q += list(op.matvec_multi(V[:m], precision=hz.PREC_F64))
            g = op.misfit_gradient(b, rx, np.ones(5, dtype=complex), method=hz.GMRES, precision=hz.PREC_F64, tol=1e-12)
            out.append((q, g[2]))
        for a, w in zip(out[0][0], out[1][0]):
            assert not np.array_equal(a, w)
            assert np.max(np.abs(a - w)) <= 2.0 ** -43 * (8 if shape == "torus" else 4)
        assert abs(out[0][1] - out[1][1]) <= 1e-8 * abs(out[1][1])
