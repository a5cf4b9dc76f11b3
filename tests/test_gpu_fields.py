"""Fields of layer densities at receivers (evaluate.cu) against the oracle, over
the branches of the FP64 pair: phase table, plain arithmetic, skipped pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOUND = 2.0 ** -42


@pytest.mark.parametrize("case", [("sphere", 16, 6.0, 1, 0), ("sphere", 31, 0.05, 0, 1), ("sphere", 16, 1e-14, 1, 0),
                                  ("torus", 36, 14.0, 0, 0), ("ellipsoid", 33, 12.0, 1, 1)])
@pytest.mark.parametrize("m", [1, 304, 1217, 1500])
def test_fields_against_the_oracle(hz, oracle, case, m):
    """Receivers on tube points (skipped pairs), within tau of them, around the
    tube, far off and beyond k rho = 4000; k too small for the phase table; one
    receiver a block, four, and a ragged last four; both layers.  A pair's
    phase k rho is off by a few ulps on either side and its factor by less than
    2^-48; the sums add less than 2^-44."""
    import oracle as O
    from helmholtz_3d_torrone_gb300 import geometry as G
    shape, N, k, dirichlet, interior = case
    factor = 2.0 if shape == "torus" else 3.0
    d = (G.sphere(N, radius=0.5, center=(0.011, 0.017, 0.005)) if shape == "sphere" else
         G.torus(N) if shape == "torus" else G.ellipsoid(N, axes=(0.7, 0.6, 0.55)))
    p = hz.params(N, k, int_l=-1.0, int_u=1.0, factor=factor, dirichlet=dirichlet, interior=interior)
    po = O.make_params(N, k, int_l=-1.0, int_u=1.0, factor=factor, dirichlet=dirichlet, interior=interior)
    tp = oracle.pipeline(po, d)
    rng = np.random.default_rng(m)
    xs, w = np.asarray(tp["xs"]).reshape(-1, 3), np.asarray(tp["w"])
    pick = xs[rng.integers(0, len(xs), m)]
    rx = np.where((np.arange(m) % 5 == 0)[:, None], pick, rng.uniform(-1, 1, (m, 3)))
    rx[1::5] = pick[1::5] + 1e-3 * rng.standard_normal(pick[1::5].shape)
    rx[2::5] *= min(50.0 / k, 1e6)
    rx[3::25] *= min(9000.0 / k, 1e8)
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        sigma = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        for layer in (hz.SINGLE_LAYER, hz.DOUBLE_LAYER):
            u = op.evaluate(rx, sigma, layer)
            want = oracle.evaluate(po, tp, sigma, rx, layer == hz.DOUBLE_LAYER)
            tau = 1e-9 + po.tau_factor * 2.0 / N
            for i in range(m):
                rho = np.linalg.norm(xs - rx[i], axis=1)
                size = np.abs(w * sigma)[rho > 0.1 * tau] / rho[rho > 0.1 * tau] / (4 * np.pi)
                if layer == hz.DOUBLE_LAYER:
                    size = size * (k + 1 / rho[rho > 0.1 * tau])
                assert abs(u[i] - want[i]) <= (BOUND + 2.0 ** -49 * k * rho.max()) * size.sum()
            assert np.array_equal(op.evaluate(rx[:1], np.ldexp(sigma.real, 40) + 1j * np.ldexp(sigma.imag, 40), layer),
                                  np.ldexp(op.evaluate(rx[:1], sigma, layer).real, 40) +
                                  1j * np.ldexp(op.evaluate(rx[:1], sigma, layer).imag, 40))
            bad = sigma.copy()
            bad[5] = np.inf
            with np.errstate(invalid="ignore"):
                assert not np.all(np.isfinite(op.evaluate(rx, bad, layer)))


@pytest.mark.parametrize("dirichlet", [0, 1])
def test_fields_far_from_the_origin(hz, oracle, dirichlet):
    """A box at 10^6: the coordinates' own rounding (10^-10) is all that is
    lost, and receivers within 3e-9 of tau of a point fall on the side of tau
    that their stored coordinates say."""
    import oracle as O
    from helmholtz_3d_torrone_gb300 import geometry as G
    N, k, lo = 24, 6.3, 1e6
    d = G.sphere(N, radius=0.5, center=(lo + 1.011, lo + 1.017, lo + 1.005), int_l=lo, int_u=lo + 2)
    p = hz.params(N, k, int_l=lo, int_u=lo + 2, factor=3.0, dirichlet=dirichlet)
    po = O.make_params(N, k, int_l=lo, int_u=lo + 2, factor=3.0, dirichlet=dirichlet)
    tp = oracle.pipeline(po, d)
    rng = np.random.default_rng(7)
    xs, w = np.asarray(tp["xs"]).reshape(-1, 3), np.asarray(tp["w"])
    m = 400
    u = rng.standard_normal((m, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    tau = po.tau_factor * 2.0 / N
    rx = xs[rng.integers(0, len(xs), m)] + tau * (1 + 3e-9 * rng.uniform(-1, 1, (m, 1))) * u
    rx[::4] = lo + 1 + 0.3 * u[::4]
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        assert np.array_equal(op.tube()["xs"].reshape(-1, 3), xs)
        sigma = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        for layer in (hz.SINGLE_LAYER, hz.DOUBLE_LAYER):
            got = op.evaluate(rx, sigma, layer)
            want = oracle.evaluate(po, tp, sigma, rx, layer == hz.DOUBLE_LAYER)
            for i in range(m):
                rho = np.linalg.norm(xs - rx[i], axis=1)
                far = rho > 0.1 * tau
                size = np.abs(w * sigma)[far] / rho[far] / (4 * np.pi)
                if layer == hz.DOUBLE_LAYER:
                    size = size * (k + 1 / rho[far])
                assert abs(got[i] - want[i]) <= (BOUND + 2.0 ** -49 * k * rho.max()) * size.sum()


@pytest.mark.parametrize("half,k", [(1e102, 1e-104), (1e101, 1e-101), (1e-9, 5e9), (1e9, 5e-9)])
@pytest.mark.parametrize("dirichlet", [0, 1])
def test_fields_in_other_units_of_length(hz, oracle, half, k, dirichlet):
    """Boxes whose k^3 leaves the FP64 range, and ones whose k^3 does not (boxes
    below 1e-18 are out of reach: the interpolation adds 1e-19 to a coordinate)."""
    import oracle as O
    from helmholtz_3d_torrone_gb300 import geometry as G
    N = 16
    d = G.sphere(N, radius=0.5, center=(0.011, 0.017, 0.005)) * half
    p = hz.params(N, k, int_l=-half, int_u=half, factor=3.0, dirichlet=dirichlet)
    po = O.make_params(N, k, int_l=-half, int_u=half, factor=3.0, dirichlet=dirichlet)
    tp = oracle.pipeline(po, d)
    rng = np.random.default_rng(8)
    xs, w = np.asarray(tp["xs"]).reshape(-1, 3), np.asarray(tp["w"])
    rx = half * rng.uniform(-1, 1, (40, 3))
    with hz.Operator(p) as op:
        op.set_distance(d)
        n = op.build()
        sigma = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        for layer in (hz.SINGLE_LAYER, hz.DOUBLE_LAYER):
            got = op.evaluate(rx, sigma, layer)
            want = oracle.evaluate(po, tp, sigma, rx, layer == hz.DOUBLE_LAYER)
            for i in range(len(rx)):
                rho = np.sqrt((((xs - rx[i]) / half) ** 2).sum(axis=1)) * half
                far = rho > 0.1 * po.tau_factor * 2 * half / N
                size = np.abs(w * sigma)[far] / rho[far] / (4 * np.pi)
                if layer == hz.DOUBLE_LAYER:
                    size = size * (k + 1 / rho[far])
                assert abs(got[i] - want[i]) <= (BOUND + 2.0 ** -49 * k * rho.max()) * size.sum()
