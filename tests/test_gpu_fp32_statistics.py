"""The FP32 contexts' statistics sweep.

With a sharp posterior (one rotation holds all of it) the new scaling is one
quotient, num / den, formed in FP64 and rounded once: it equals the FP32
rounding of that quotient.  Poisson: den is the sum of the slice's FP32 values,
exact in FP64 in any order here, since the model's voxels are multiples of 2^-20
below 16, and longer than an FP32 mantissa.  Broad posteriors: sum P log P, the scaling
and the log-likelihood against 64 bits of the context's own log-likelihoods."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE = 18


def _setup(N, R, lik, counts, model, scale):
    import emc_b200 as E
    x, y, z = E.detector_coordinates(SIDE, 1e-10, 1.0 / SIDE, 1.0)
    qa, wa = E.generate_rotations(3)
    pick = np.random.default_rng(9).permutation(len(wa))[:R]
    ctx = E.Context(SIDE, N, R, likelihood=lik)
    ctx.set_geometry(x, y, z, np.ones(SIDE * SIDE, np.int32))
    ctx.set_rotations(qa[pick].copy(), wa[pick].copy())
    ctx.set_patterns(counts)
    ctx.set_model(model)
    ctx.set_scaling(scale)
    return ctx


@pytest.mark.parametrize("N,R", [(1, 33), (70, 64), (257, 300)])
def test_poisson_scaling_of_sharp_posteriors_is_rounded_once(N, R):
    import emc_b200 as E
    from oracle import oracle as O
    rng = np.random.default_rng(N)
    model = (rng.integers(1, 1 << 24, SIDE ** 3) * 2.0 ** -20).astype(np.float32)
    x, y, z = E.detector_coordinates(SIDE, 1e-10, 1.0 / SIDE, 1.0)
    qa, _ = E.generate_rotations(3)
    pick = np.random.default_rng(9).permutation(len(qa))[:R]
    cfg = O.make_config(SIDE, N, R, likelihood=O.LL_POISSON)
    S = O.expand(cfg, model, qa[pick], x, y, z)  # [R][side^2], the voxels themselves
    true = rng.integers(0, R, N)
    counts = np.rint(S[true] * 15).astype(np.float32)
    with _setup(N, R, "poisson", counts, model, np.full(N, 15, np.float32)) as ctx:
        ctx.expand()
        ctx.maximize()
        P, phi = ctx.get_buffer(E.BUF_RESP), ctx.get_scaling()
    best = P.argmax(0)
    sharp = P.astype(np.float64).sum(0) - P.max(0) < 1e-12
    assert sharp.mean() > 0.9
    num, den = counts.astype(np.float64).sum(1), S.astype(np.float64).sum(1)[best]
    np.testing.assert_array_equal(phi[sharp], (num / den).astype(np.float32)[sharp])


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
@pytest.mark.parametrize("N,R", [(31, 63), (64, 257), (300, 640)])
def test_statistics_of_broad_posteriors(lik, N, R):
    """phi against num / sum_r P X of the context's own P (FP32, each 2^-24 of
    its exponent's rounding off: |LL - lse| stays below 20) and 64-bit X."""
    import emc_b200 as E
    from oracle import oracle as O
    rng = np.random.default_rng(N)
    model = (0.5 + rng.random(SIDE ** 3)).astype(np.float32)
    counts = rng.poisson(0.05, (N, SIDE * SIDE)).astype(np.float32)
    counts[:, 3] += 1
    scale = (0.05 * (0.5 + rng.random(N))).astype(np.float32)
    x, y, z = E.detector_coordinates(SIDE, 1e-10, 1.0 / SIDE, 1.0)
    qa, _ = E.generate_rotations(3)
    pick = np.random.default_rng(9).permutation(len(qa))[:R]
    cfg = O.make_config(SIDE, N, R, likelihood=O.LL_POISSON if lik == "poisson" else O.LL_GAUSS)
    S = O.expand(cfg, model, qa[pick], x, y, z).astype(np.float64)
    K = counts.astype(np.float64)
    with _setup(N, R, lik, counts, model, scale) as ctx:
        st = ctx.iterate()
        P, phi = ctx.get_buffer(E.BUF_RESP).astype(np.float64), ctx.get_scaling()
    LL = O.loglik(cfg, S.astype(np.float32), counts, np.ones(SIDE * SIDE, np.int32), scale)
    if lik == "poisson":
        num, X = K.sum(1), np.broadcast_to(S.sum(1)[:, None], P.shape)
    else:
        num, X = (K * K).sum(1), S @ K.T
    # weights 2^-24 (|d| <= 20, then expf's own 2 ulp) each way
    tol = 2 * (20 + 4) * 2.0 ** -24
    np.testing.assert_allclose(phi, num / (P * X).sum(0), rtol=tol)
    lse = np.log(np.exp(LL - LL.max(0)).sum(0)) + LL.max(0)
    Q = np.exp(LL - lse)
    ref = (Q * (LL - lse)).sum()
    np.testing.assert_allclose(st["sum_plogp"], ref, rtol=tol, atol=tol * N)
    np.testing.assert_allclose(st["total_loglik"], lse.sum(), rtol=1e-6, atol=1e-5 * N)


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
@pytest.mark.parametrize("N,R,top", [(15, 127, 128), (16, 128, 127), (257, 129, 300), (129, 640, 16383)])
def test_scaling_at_tile_edges_and_with_two_count_planes(lik, N, R, top):
    """num / sum_r P X with the context's own P, whatever their sharpness: the
    gaussian cross term comes out of the byte contraction's log-likelihood."""
    import emc_b200 as E
    from oracle import oracle as O
    rng = np.random.default_rng(N + R)
    model = (0.5 + rng.random(SIDE ** 3)).astype(np.float32)
    counts = rng.poisson(0.3, (N, SIDE * SIDE)).astype(np.float32)
    counts[np.arange(N), rng.integers(SIDE * SIDE, size=N)] = top
    scale = ((0.5 + rng.random(N)) * counts.sum(1) / SIDE ** 2).astype(np.float32)
    x, y, z = E.detector_coordinates(SIDE, 1e-10, 1.0 / SIDE, 1.0)
    qa, _ = E.generate_rotations(3)
    pick = np.random.default_rng(9).permutation(len(qa))[:R]
    cfg = O.make_config(SIDE, N, R, likelihood=O.LL_POISSON if lik == "poisson" else O.LL_GAUSS)
    S = O.expand(cfg, model, qa[pick], x, y, z).astype(np.float64)
    K = counts.astype(np.float64)
    with _setup(N, R, lik, counts, model, scale) as ctx:
        ctx.expand()
        ctx.maximize()
        P, phi = ctx.get_buffer(E.BUF_RESP).astype(np.float64), ctx.get_scaling()
    if lik == "poisson":
        num, X = K.sum(1), np.broadcast_to(S.sum(1)[:, None], P.shape)
    else:
        num, X = (K * K).sum(1), S @ K.T
    # P's normalisation cancels in the sweep's own sums: divided out here too
    np.testing.assert_allclose(phi, num * P.sum(0) / (P * X).sum(0), rtol=2 * (20 + 4) * 2.0 ** -24)
