"""The FP32 responsibility pass and the byte operand of P / phi over their block
shapes (8, 16 or 32 rows; one or two patterns a thread; four or eight rows of
digits; rows of a multiple of four or not), against FP64 on the responsibilities
that are read back.

  P        sums to 1 per pattern: FP32 rounding of each (2^-23 with the
           exponential's, 2^-20 in all)
  T        FP64 sums of P, rounded to FP32 (2^-23)
  U        FP32 rounding of P / phi (2^-22) and of the result, and the
           fixed-point step 2^-31 of the row maximum per photon
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,R", [(300, 4999), (301, 10001), (513, 18961), (600, 19000), (1030, 9)])
def test_block_shapes(N, R):
    import emc_b200 as E
    side = 16
    rng = np.random.default_rng(N)
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    q, w = E.generate_rotations(8)
    pick = np.sort(rng.permutation(len(w))[:R])
    mask = np.zeros(side * side, np.int32)
    mask[rng.permutation(side * side)[:61]] = 1
    counts = rng.poisson(2.0, (N, side * side)).astype(np.float32)
    counts[:, np.flatnonzero(mask)[0]] = 1
    K = counts[:, mask == 1].astype(np.float64)
    with E.Context(side, N, R) as ctx:
        ctx.set_geometry(x, y, z, mask)
        ctx.set_rotations(q[pick].copy(), w[pick].copy())
        ctx.set_patterns(counts)
        ctx.set_model((0.1 + 4 * rng.random(side ** 3)).astype(np.float32))
        ctx.set_scaling((0.3 + rng.random(N)).astype(np.float32))
        ctx.expand()
        ctx.maximize()
        P = ctx.get_buffer(E.BUF_RESP).astype(np.float64)
        phi = ctx.get_scaling().astype(np.float64)
        ctx.compress_insert()
        T, U = ctx.get_buffer(E.BUF_TOTALRESP), ctx.get_buffer(E.BUF_SLICES)
    np.testing.assert_allclose(P.sum(0), 1.0, rtol=2.0 ** -20)
    total = P.sum(1)
    np.testing.assert_allclose(T, total, rtol=2.0 ** -23)
    X = P / phi
    per = 1.0 / np.maximum(total, 1e-300)[:, None]
    ref = X @ K * per
    step = X.max(1)[:, None] * 2.0 ** -31 * K.sum(0) * per
    live = total > 1e-10
    assert (np.abs(U - ref) <= step + 2.0 ** -21 * ref + 1e-30)[live].all()
