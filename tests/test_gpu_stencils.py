"""The gradient and curvature grids (stencils.cu) bit for bit against the
oracle where the shared and rewritten arithmetic could round another way:
noise (every branch of the stencils), flat and linear parts (zeros and signed
zeros), values far from 1 (the plain divisions), steps that are and are not
powers of two, grids of one segment, ragged segments and only boundary nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def fields(N, H, seed):
    rng = np.random.default_rng(seed)
    t = (np.arange(N + 1) - 0.37 * N) * H
    Y, X, Z = t[:, None, None], t[None, :, None], t[None, None, :]
    smooth = np.sqrt(X ** 2 + Y ** 2 + 0.5 * Z ** 2 + 0.01) - 0.4
    noise = rng.standard_normal((N + 1,) * 3)
    flat = np.where(X > 0.1, 0.0, np.broadcast_to(0.25 * Y + Z, noise.shape))
    mixed = smooth + 1e-9 * noise * rng.integers(0, 2, noise.shape)
    yield from (smooth, noise, flat, -flat, mixed, np.round(4 * noise) / 4, 10.0 ** rng.integers(-12, 5) * noise)
    for e in (-1000, -520, -300, -60, 60, 250):
        yield np.ldexp(noise, e)


@pytest.mark.parametrize("N", [8, 15, 16, 31, 47])
@pytest.mark.parametrize("step", ["box", "odd", "tiny", "large"])
def test_grids_bitexact_vs_oracle(hz, oracle, N, step):
    H = {"box": 2.0 / N, "odd": 0.0123456789 + 1.0 / N, "tiny": 2.0 ** -400, "large": 3.1e90}[step]
    for d in fields(N, 2.0 / N, N):
        d = np.ascontiguousarray(np.broadcast_to(d, (N + 1,) * 3))
        got = list(hz.assign_gradient(d, N, H)) + list(hz.assign_curvatures(d, N, H))
        with np.errstate(all="ignore"):
            want = list(oracle.gradient(N, H, d)) + list(oracle.curvatures(N, H, d))
        for g, w in zip(got, want):
            g, w = np.asarray(g).ravel(), np.asarray(w).ravel()
            ok = (g.view(np.uint64) == w.view(np.uint64)) | (np.isnan(g) & np.isnan(w))
            assert np.all(ok)
        if step == "box":
            for g, w in zip(hz.assign_gradient(d, N, H, weno_order=3), oracle.gradient(N, H, d, order=3)):
                assert np.array_equal(np.asarray(g).ravel().view(np.uint64), np.asarray(w).ravel().view(np.uint64))


@pytest.mark.parametrize("N", [8, 31])
@pytest.mark.parametrize("step", ["box", "tiny"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_nonfinite_nodes(hz, oracle, N, step, value):
    """NaN and infinities at a few nodes, corners and neighbours among them: the
    same nodes become NaN or infinite as in the oracle, the others keep their bits."""
    H = {"box": 2.0 / N, "tiny": 2.0 ** -400}[step]
    rng = np.random.default_rng(N)
    for d in list(fields(N, 2.0 / N, N))[:3]:
        d = np.array(np.broadcast_to(d, (N + 1,) * 3))
        at = rng.integers(0, N + 1, (4, 3))
        at[0] = 0
        at[1] = (N, N, N // 2)
        at[3] = np.minimum(at[2] + (0, 1, 2), N)
        d[tuple(at.T)] = value * np.array([1, 1, 1, -1])
        got = list(hz.assign_gradient(d, N, H)) + list(hz.assign_curvatures(d, N, H))
        with np.errstate(all="ignore"):
            want = list(oracle.gradient(N, H, d)) + list(oracle.curvatures(N, H, d))
        for g, w in zip(got, want):
            g, w = np.asarray(g).ravel(), np.asarray(w).ravel()
            assert np.all((g.view(np.uint64) == w.view(np.uint64)) | (np.isnan(g) & np.isnan(w)))
