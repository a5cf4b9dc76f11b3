"""The FP64 products in split FP32 arithmetic (sweep_split.cu) against the
oracle's matrix, at the edges of the range they serve: tubes just below and
above 2,048 points (the FP64 sweep below), a ragged last tile, tiles that
straddle the surface (the torus), the smallest and largest k h, Neumann and
Dirichlet, interior and exterior, the [-2, 2]^3 box.

Over a row the entries of the split sweep are off by less than 2^-44 of
sum |A_ts p_s|, their sum adds at most as much again, and the oracle's own
sequential sum less than 2^-44 at these sizes: the rows are compared with
2^-42 of that sum.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 2.0 ** -42
CASES = [  # shape, N, k, dirichlet, interior, half width of the box
    ("sphere", 19, 5.0, 1, 0, 1.0),
    ("sphere", 21, 5.0, 1, 0, 1.0),
    ("sphere", 21, 8.4, 0, 0, 1.0),
    ("sphere", 24, 0.02, 1, 0, 1.0),
    ("sphere", 24, 0.5, 0, 1, 1.0),
    ("sphere", 31, 3.0, 0, 0, 2.0),
    ("torus", 36, 14.0, 1, 0, 1.0),
    ("torus", 36, 2.0, 0, 1, 1.0),
    ("ellipsoid", 33, 12.0, 1, 1, 1.0),
]


@pytest.mark.parametrize("case", CASES)
def test_products_against_the_oracle_matrix(hz, oracle, case):
    import oracle as O
    from helmholtz_3d_torrone_gb300 import geometry as G
    shape, N, k, dirichlet, interior, half = case
    factor = 2.0 if shape == "torus" else 3.0
    if shape == "sphere":
        d = G.sphere(N, radius=0.5 * half, center=(0.011, 0.017, 0.005), int_l=-half, int_u=half)
    elif shape == "torus":
        d = G.torus(N)
    else:
        d = G.ellipsoid(N, axes=(0.7, 0.6, 0.55))
    p = hz.params(N, k, int_l=-half, int_u=half, factor=factor, dirichlet=dirichlet, interior=interior)
    po = O.make_params(N, k, int_l=-half, int_u=half, factor=factor, dirichlet=dirichlet, interior=interior)
    tp = oracle.pipeline(po, d)
    are, aim = oracle.dense(po, tp)
    A = are + 1j * aim
    rng = np.random.default_rng(N)
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        v = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        u = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        q, qt = op.matvec(v), op.matvec(u, adjoint=True)
        assert np.all(np.abs(q - A @ v) <= BOUND * (np.abs(A) @ np.abs(v)))
        assert np.all(np.abs(qt - A.conj().T @ u) <= BOUND * (np.abs(A).T @ np.abs(u)))
        pq, pt = op.matvec_pair(v, u)
        assert np.all(np.abs(pq - q) <= BOUND * (np.abs(A) @ np.abs(v)))
        assert np.all(np.abs(pt - qt) <= BOUND * (np.abs(A).T @ np.abs(u)))
        # densities of any size: powers of two scale the product exactly
        for e in (-600, 600):
            assert np.array_equal(op.matvec(np.ldexp(v.real, e) + 1j * np.ldexp(v.imag, e)),
                                  np.ldexp(q.real, e) + 1j * np.ldexp(q.imag, e))
        assert not np.any(op.matvec(np.zeros(n, dtype=complex)))


def test_nonfinite_density_and_short_waits(hz):
    """What the FP64 sweep reports the split sweep reports: a NaN or Inf
    density, and data waits that give up."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    p = hz.params(24, 5.0, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=1)
    with hz.Operator(p) as op:
        op.set_distance(G.sphere(24, radius=0.5, center=(0.011, 0.017, 0.005)))
        n = op.build()
        v = np.ones(n, dtype=complex)
        want = op.matvec(v)
        for bad in (np.nan, np.inf):
            w = v.copy()
            w[3] = bad
            with pytest.raises(hz.HzError) as e:
                op.matvec(w)
            assert e.value.code == hz.HZ_ERR_NONFINITE
        try:
            hz.set_wait_limit(0)
            with pytest.raises(hz.HzError) as e:
                op.matvec(v)
            assert e.value.code == hz.HZ_ERR_DEVICE_WAIT
        finally:
            hz.set_wait_limit(-1)
        assert np.array_equal(op.matvec(v), want)


@pytest.mark.parametrize("nrhs", [1, 4, 5, 8, 9, 16, 19])
def test_columns_equal_single_products(hz, nrhs):
    """Blocks of 4, 8 and 16 columns, their remainders and a zero column: the
    same entries as the single product, summed in another order."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    for dirichlet in (0, 1):
        p = hz.params(24, 6.0, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=dirichlet)
        with hz.Operator(p) as op:
            op.set_distance(G.sphere(24, radius=0.5, center=(0.011, 0.017, 0.005)))
            n = op.build()
            rng = np.random.default_rng(nrhs)
            V = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
            V *= 10.0 ** rng.integers(-20, 20, nrhs)[:, None]
            V[nrhs // 2] = 0.0
            Q = op.matvec_multi(V, precision=hz.PREC_F64)
            for v, q in zip(V, Q):
                # a row's sum |A_ts p_s| is below 4 max |p| on this sphere
                assert np.max(np.abs(q - op.matvec(v))) <= BOUND * 4 * np.max(np.abs(v))


def test_wave_number_gradient(hz):
    """dJ/dk where dA/dk runs in split arithmetic, against central differences
    (their truncation and the solver's tolerance: 1e-5)."""
    from helmholtz_3d_torrone_gb300 import geometry as G
    k, N = 6.0, 24
    rng = np.random.default_rng(5)
    rx = G.random_sphere_points(7, 0.9, seed=6)
    target = rng.standard_normal(7) + 1j * rng.standard_normal(7)

    def misfit(kk, dirichlet):
        p = hz.params(N, kk, int_l=-1.0, int_u=1.0, factor=3.0, dirichlet=dirichlet)
        with hz.Operator(p) as op:
            op.set_distance(G.sphere(N, radius=0.5, center=(0.011, 0.017, 0.005)))
            n = op.build()
            assert n >= 2048
            b = np.exp(1j * np.arange(n) / n)
            J, _, dk, _, _ = op.misfit_gradient(b, rx, target, method=hz.BICG, precision=hz.PREC_F64, tol=1e-13)
            return J, dk

    for dirichlet in (0, 1):
        h = 1e-5
        fd = (misfit(k + h, dirichlet)[0] - misfit(k - h, dirichlet)[0]) / (2 * h)
        assert abs(misfit(k, dirichlet)[1] - fd) <= 1e-5 * abs(fd)
