"""Slice sums of the FP32 contexts keep the digits of responsibilities far below
their row's largest: a pixel whose photons come only from such patterns gets
its value from them, however dark (sharp posteriors and sparse counts leave
most pixels so).  Against 64 bits of the context's own P and phi.  Each term
carries the FP32 rounding of P / phi (2^-22), a sum of n of them n 2^-24 at
most, and the result is rounded once more: (n + 8) 2^-24, n <= N.  Sizes at
the edges of the pixel and pattern blocks, one and two count planes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lik,side,N,R,npa,top", [
    ("poisson", 18, 60, 300, 324, 1), ("poisson", 18, 257, 129, 257, 200),
    ("poisson", 70, 31, 140, 4097, 1), ("poisson", 70, 300, 65, 4096, 16383),
    ("gauss", 18, 255, 200, 15, 127), ("gauss", 18, 16, 128, 17, 300), ("poisson", 18, 1, 40, 1, 3),
    ("poisson", 18, 1100, 33, 200, 1), ("poisson", 18, 5000, 20, 100, 2),
    ("poisson", 230, 9, 24, 52_000, 1),  # a slice longer than shared memory
])
def test_dark_pixels_keep_their_digits(lik, side, N, R, npa, top):
    import emc_b200 as E
    rng = np.random.default_rng(N + R)
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    qa, wa = E.generate_rotations(3)
    pick = rng.permutation(len(wa))[:R]
    mask = np.zeros(side * side, np.int32)
    act = np.sort(rng.permutation(side * side)[:npa])
    mask[act] = 1
    model = np.exp(rng.normal(0, 1.5, side ** 3)).astype(np.float32)
    counts = (rng.random((N, side * side)) < min(0.3, 40 / npa + 0.01)).astype(np.float32)
    counts *= rng.integers(1, 4, counts.shape)
    counts[rng.random(counts.shape) < 0.002] = top
    counts[:, act[0]] = np.arange(N) % 2 * top
    scale = np.exp(rng.normal(0, 0.5, N)).astype(np.float32)
    with E.Context(side, N, R, likelihood=lik, sigma=0.05) as ctx:
        ctx.set_geometry(x, y, z, mask)
        ctx.set_rotations(qa[pick].copy(), wa[pick].copy())
        ctx.set_patterns(counts)
        ctx.set_model(model)
        ctx.set_scaling(scale)
        for whole in (False, True):
            ctx.set_model(model)
            ctx.set_scaling(scale)
            if whole:
                ctx.iterate()
            else:
                ctx.expand()
                ctx.maximize()
                ctx.compress()
            P, phi = ctx.get_buffer(E.BUF_RESP), ctx.get_scaling().astype(np.float64)
            U = ctx.get_buffer(E.BUF_SLICES).astype(np.float64)
            T = P.astype(np.float64).sum(1)
            live = T > 1e-10
            K = counts[:, act].astype(np.float64)
            ref = (P[live] / phi) @ K / T[live, None]
            # what FP32 holds of the largest value's small terms: P / phi down to
            # its smallest normal number
            tiny = K.sum(0) * 1.2e-38 / T[live, None]
            tol = (min(N, 4096) + 8) * 2.0 ** -24 * ref + tiny
            assert (np.abs(U[live] - ref) <= tol).all(), (np.abs(U[live] - ref) / (ref + tiny)).max()
            if N > 50 and top == 1:  # sharp posteriors and few photons a pixel
                X = P[live] / phi
                dark = (ref * T[live, None] < 2.0 ** -24 * X.max(1)[:, None]) & (ref > 0)
                assert dark.any()
