"""FP32 contexts on the CUDA cores (fractional counts): a pattern whose
log-likelihood has no finite value at any rotation (K / phi overflows when
squared in FP32) takes no part, as in the reference's softmax: its
responsibilities are 0, its scaling stays, and the others are as without it."""
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


def test_a_pattern_without_a_finite_likelihood_takes_no_part():
    import emc_b200 as E
    rng = np.random.default_rng(4)
    N, R = 40, 130
    model = (0.5 + rng.random(SIDE ** 3)).astype(np.float32)
    counts = rng.poisson(1.0, (N, SIDE * SIDE)).astype(np.float32) + np.float32(0.5)
    scale = np.ones(N, np.float32)
    with _setup(N - 1, R, "gauss", counts[1:], model, scale[1:]) as ctx:
        ctx.iterate()
        m_ref, s_ref = ctx.get_model(), ctx.get_scaling()
    scale[0] = 1e-25
    with _setup(N, R, "gauss", counts, model, scale) as ctx:
        st = ctx.iterate()
        P, m, s = ctx.get_buffer(E.BUF_RESP), ctx.get_model(), ctx.get_scaling()
    assert not P[:, 0].any()
    assert s[0] == scale[0]
    np.testing.assert_array_equal(s[1:], s_ref)
    assert np.isfinite(st["sum_plogp"])
    assert np.linalg.norm(m - m_ref) <= 1e-6 * np.linalg.norm(m_ref)
