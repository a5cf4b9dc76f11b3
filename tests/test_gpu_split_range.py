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


def columns(hz, oracle, p, d, count, rng, scale=1.0):
    """(largest error of a column's entries over their bound, n): sources with
    the closest far neighbours and `count` others.  The bound's scale is the
    entry with |x_t - x_s| for the projection (w (k + 1/rho) / (4 pi rho))."""
    import oracle as O
    po = O.make_params(p.N, p.wave, int_l=p.int_l, int_u=p.int_u, factor=p.factor, tau_factor=p.tau_factor,
                       dirichlet=p.dirichlet, interior=p.interior)
    tp = oracle.pipeline(po, d)
    are, aim = oracle.dense(po, tp)
    xs, w, reg = np.asarray(tp["xs"]).reshape(-1, 3), np.asarray(tp["w"]), np.asarray(tp["reg"])
    tau = p.tau_factor * (p.int_u - p.int_l) / p.N
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        assert n == len(w)
        near = np.full(n, np.inf)
        for i in range(0, n, 512):
            r = np.linalg.norm(xs[i:i + 512, None] - xs[None], axis=2)
            near[i:i + 512] = np.where(r > tau, r, np.inf).min(axis=1)
        pick = np.concatenate([np.argsort(near)[:count], rng.integers(0, n, count)])
        worst = 0.0
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
                # r^2 off by 2^-43, three halves of it in the entry, the rest of
                # the split arithmetic 2^-44; coordinates times k 2^-53 of |x|
                # each, seven times that over rho
                tol = 2.0 ** -42 + 2.0 ** -50 * np.abs(xs).max() / np.maximum(rho, tau)
                err = np.abs(q - A * v[s]) / abs(v[s])
                err[s] -= 2.0 ** -52
                worst = max(worst, float(np.max(err / np.where(size > 0, tol * size, np.inf))))
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
