"""The row-sum sweep of the mixed responsibility pass at the edges of its blocks
(1,024 patterns, four a thread; 8 to 32 rotations), for sharp posteriors, of
which most elements are left at a comparison, and broad ones.

T_r against the FP64 sum of the responsibilities that are read back (the same
FP32 exponentials): four additions in a thread, five over a warp, eight warps
and the blocks of patterns, each 2^-24 (below 2^-19 together), and N
responsibilities below 1e-30 that the sweep leaves out.  The entries that it
compacts show in the slice sums of the lists, against the dense contraction's
(22 bits of P / (T phi) and FP32 sums: 1e-5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
@pytest.mark.parametrize("contrast", [0.01, 3.0])
@pytest.mark.parametrize("N,R", [(1, 1), (3, 31), (127, 33), (1023, 7), (1025, 65), (1030, 700),
                                 (4098, 20)])
def test_row_sums_and_lists(lik, contrast, N, R):
    import emc_b200 as E
    side = 16
    rng = np.random.default_rng(N + R)
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    q, w = E.generate_rotations(3)
    pick = rng.permutation(len(w))[:R]
    counts = rng.poisson(1.0, (N, side * side)).astype(np.float32)
    counts[:, 0] = 1
    model = np.exp(contrast * rng.normal(0, 1, side ** 3)).astype(np.float32)
    out = []
    for lists in (False, True):
        with E.Context(side, N, R, likelihood=lik, precision="mixed") as ctx:
            ctx.set_geometry(x, y, z, np.ones(side * side, np.int32))
            ctx.set_rotations(q[pick].copy(), w[pick].copy())
            ctx.set_patterns(counts)
            ctx.set_model(model)
            ctx.set_scaling(np.ones(N, np.float32))
            ctx.set_sparse_compress(lists)
            ctx.expand()
            ctx.maximize()
            P = ctx.get_buffer(E.BUF_RESP).astype(np.float64)
            ctx.compress()
            T = ctx.get_buffer(E.BUF_TOTALRESP)
            np.testing.assert_allclose(T, P.sum(1), rtol=2.0 ** -19, atol=N * 1e-30)
            out.append(ctx.get_model())
    a, b = out
    assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a)
