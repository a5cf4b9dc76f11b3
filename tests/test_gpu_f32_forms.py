"""The forms of the FP32 products (sweep_f32.cu, sweep_multi.cu) against the
FP64 product: coordinates times k or not, tiles whose phase is taken about the
tile or reduced per pair, tubes on both sides of the unit sizes (24 and 80 tiles).

An FP32 entry is off by a few 2^-24 from its offsets (2^-24 of the tile's
radius over rho, rho >= tau: up to 8), its phase (2^-24 k rho) and the SFU's sine
and cosine (4e-7): below 2e-6 + 1.2e-7 k rho.  Rows are compared with that times a
bound on sum |A_ts p_s|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operator(hz, shape, N, k, dirichlet, half=1.0, interior=0):
    from helmholtz_3d_torrone_gb300 import geometry as G
    d = (G.torus(N) if shape == "torus" else G.sphere(N, radius=0.5, center=(0.011, 0.017, 0.005))) * half
    op = hz.Operator(hz.params(N, k, int_l=-half, int_u=half, factor=3.0, dirichlet=dirichlet, interior=interior))
    op.set_distance(d)
    return op, op.build()


def row_sums(op, rows):
    """sum_s |A_ts| and sum_s |A_st| of rows t from above, from the tube: the
    entries with |x_t - x_s| for the projection, and the regularised ones."""
    t = op.tube()
    xs, w, reg = t["xs"].reshape(-1, 3), t["w"], np.abs(t["reg"])
    tau, k = op.p.tau_factor * (op.p.int_u - op.p.int_l) / op.p.N, abs(op.p.wave)
    rho = np.linalg.norm(xs[rows, None] - xs[None], axis=2)
    far = rho > tau
    rho[~far] = 1.0
    e = np.where(far, (k + 1 / rho) / (4 * np.pi * rho), np.maximum(reg[rows, None], reg[None]))
    return e @ w + 0.5, w[rows] * e.sum(axis=1) + 0.5, 2e-6 + 1.2e-7 * k * np.linalg.norm(np.ptp(xs, axis=0))


@pytest.mark.parametrize("shape,N,k,half", [
    ("sphere", 24, 0.0, 1.0), ("sphere", 24, -3.0, 1.0), ("sphere", 24, 1e-6, 1.0),      # unscaled
    ("sphere", 24, 2.0 ** -14 * 0.999, 1.0), ("sphere", 24, 2.0 ** -14, 1.0),            # on both sides of it
    ("sphere", 24, 2.0 ** -13, 1e-15), ("sphere", 24, 2.0 ** -13, 2.0 ** -27 * 6 * 0.999),
    ("sphere", 24, 2.0 ** -13, 2.0 ** -27 * 6 * 1.001),                                  # k tau = 2^-40
    ("sphere", 24, 1.0, 1.0), ("sphere", 24, 30.0, 1.0),                                 # centred; reduced per pair
    ("sphere", 33, 5.0, 1.0), ("sphere", 37, 5.0, 1.0), ("torus", 47, 7.0, 1.0), ("torus", 50, 60.0, 1.0)])
@pytest.mark.parametrize("dirichlet,interior", [(1, 0), (0, 1)])
def test_fp32_products(hz, shape, N, k, half, dirichlet, interior):
    rng = np.random.default_rng(N)
    op, n = operator(hz, shape, N, k, dirichlet, half, interior)
    V = np.exp(2j * np.pi * rng.random((5, n)))
    if k < 0:  # the FP64 product serves k >= 0: A(-k) v = conj(A(k) conj(v))
        ref, _ = operator(hz, shape, N, -k, dirichlet, half, interior)
        with ref:
            Q = np.array([ref.matvec(v.conj()).conj() for v in V])
            qt = ref.matvec(V[1].conj(), adjoint=True).conj()
    else:
        Q, qt = np.array([op.matvec(v) for v in V]), op.matvec(V[1], adjoint=True)
    rows = rng.choice(n, 200, replace=False)
    with op:
        sums, sumh, tol = row_sums(op, rows)

        def close(a, b, s):
            return np.max(np.abs(a - b)[rows] / s) <= tol

        for cfg in range(8):
            op.set_sweep_config(cfg)
            assert close(op.matvec(V[0], precision=hz.PREC_F32), Q[0], sums)
            assert close(op.matvec(V[1], precision=hz.PREC_F32, adjoint=True), qt, sumh)
            a, b = op.matvec_pair(V[0], V[1], precision=hz.PREC_F32)
            assert close(a, Q[0], sums) and close(b, qt, sumh)
        for q, want in zip(op.matvec_multi(V, precision=hz.PREC_F32), Q):
            assert close(q, want, sums)
        with hz.Batch([op]) as batch:
            for v in range(4):
                batch.set_variant(v)
                assert close(batch.matvec([V[0]])[0], Q[0], sums)


def test_phase_modes_give_one_product(hz):
    """hz_set_phase_mode takes both settings, and both run the same sweep."""
    op, n = operator(hz, "sphere", 24, 9.0, 1)
    v = np.exp(1j * np.arange(n))
    with op:
        out = []
        for mode in (hz.PHASE_DIRECT, hz.PHASE_SPLIT):
            op.set_phase_mode(mode)
            out.append([op.matvec(v, precision=hz.PREC_F32), *op.matvec_pair(v, v, precision=hz.PREC_F32)])
        for a, b in zip(*out):
            assert np.array_equal(a, b)
        for mode in (-1, 2):
            with pytest.raises(hz.HzError) as e:
                op.set_phase_mode(mode)
            assert e.value.code == hz.HZ_ERR_ARG
