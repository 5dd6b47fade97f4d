"""The expansion at the edges of its blocks (16 rotations or fewer, 256 pixels,
several chunks of a large detector per block), against the oracle: FP32 nearest
slices are exact, the others carry FP32 weights or logarithms (1e-6) or the 22
bits of the FP16 pair (1e-6 of the largest value).  The row sums show in the
poisson scaling, sum K / sum_r P_r sum W_r, whose P come from the engine."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,lik,interp", [("fp32", "gauss", "nearest"), ("fp32", "poisson", "trilinear"),
                                             ("fp32", "poisson", "nearest"),
                                             ("mixed", "poisson", "nearest"),
                                             ("mixed", "gauss", "trilinear")])
@pytest.mark.parametrize("side,R,npa", [(16, 1, 1), (17, 3, 255), (17, 17, 257), (19, 33, 361),
                                        (33, 130, 513), (131, 5, 17161)])
def test_slices_and_row_sums(prec, lik, interp, side, R, npa):
    import emc_b200 as E
    rng = np.random.default_rng(side * 100 + R)
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    q, w = E.generate_rotations(3)
    pick = rng.permutation(len(w))[:R]
    mask = np.zeros(side * side, np.int32)
    mask[rng.permutation(side * side)[:npa]] = 1
    counts = rng.poisson(1.0, (2, side * side)).astype(np.float32)
    model = (0.1 + rng.random(side ** 3)).astype(np.float32)
    cfg = O.make_config(side, 2, R, likelihood=O.LL_POISSON if lik == "poisson" else O.LL_GAUSS,
                        interp=O.TRILINEAR if interp == "trilinear" else O.NEAREST)
    with E.Context(side, 2, R, likelihood=lik, interp=interp, precision=prec) as ctx:
        ctx.set_geometry(x, y, z, mask)
        ctx.set_rotations(q[pick].copy(), w[pick].copy())
        ctx.set_patterns(counts)
        ctx.set_model(model)
        ctx.set_scaling(np.ones(2, np.float32))
        ctx.expand()
        S = ctx.get_buffer(E.BUF_SLICES)
        ctx.maximize()
        P, phi = ctx.get_buffer(E.BUF_RESP).astype(np.float64), ctx.get_scaling()
    act = np.flatnonzero(mask)
    ref = O.expand(cfg, model, q[pick], x, y, z)[:, act]
    out = np.log(np.maximum(ref, 1e-10)) if lik == "poisson" else ref
    if (prec, lik, interp) == ("fp32", "gauss", "nearest"):
        np.testing.assert_array_equal(S, out.astype(np.float32))
    else:
        assert np.abs(S - out).max() <= 2e-6 * max(1.0, np.abs(out).max())
    if lik == "poisson":
        want = counts[:, act].sum(1) / (P.T @ ref.sum(1))
        # trilinear weights are FP32 products; the sums themselves are FP64
        np.testing.assert_allclose(phi, want, rtol=2e-6)


@pytest.mark.parametrize("side", [2, 15, 16, 37])
def test_table_gives_the_voxels_themselves(side):
    """FP32 poisson reads (W, log W) from a table where there is room for it;
    without room, the model and the logarithm: the same bits."""
    import emc_b200 as E
    rng = np.random.default_rng(side)
    # any pixel positions, many of them on the rounding's halves and the edges
    n = side * side
    x, y, z = (rng.integers(-side, side + 1, n).astype(np.float32) * np.float32(0.5) for _ in range(3))
    q, w = E.generate_rotations(3)
    q = q[:200].copy()
    q[0] = [1, 0, 0, 0]  # the identity keeps the halves
    counts = np.ones((3, n), np.float32)
    model = rng.random(side ** 3).astype(np.float32)
    out = []
    for limit in (False, True):
        with E.Context(side, 3, len(q), likelihood="poisson") as ctx:
            ctx.set_geometry(x, y, z, np.ones(n, np.int32))
            ctx.set_rotations(q, w[:200].copy())
            ctx.set_patterns(counts)
            ctx.set_model(model)
            if limit:
                ctx.set_memory_limit(ctx.memory_used - 1)
            ctx.expand()
            out.append(ctx.get_buffer(E.BUF_SLICES))
    np.testing.assert_array_equal(out[0], out[1])
    cfg = O.make_config(side, 3, len(q), likelihood=O.LL_POISSON)
    ref = np.log(np.maximum(O.expand(cfg, model, q, x, y, z), 1e-10))
    np.testing.assert_allclose(out[0], ref, rtol=1e-6, atol=1e-6)
