"""FP32 contexts: the contractions on byte digits (kernels_i8.cu) at the edges
of their tiles, against the FP64 oracle and against the CUDA-core form.

Sizes around the tile (128 rotations, 256 rows of the other operand, 128-byte
K-steps) and the 16-byte row pitch; counts of one and two base-128 planes.

Tolerances, from the arithmetic:
  log-likelihood  a slice value carries its FP32 rounding (2^-23, logarithm
                  included) and the fixed-point step of its row (2^-31 of the
                  row maximum); each enters the sum once per photon
  responsibility  L1 per pattern <= 2 x the log-likelihood error + 2^-20
  slice sum       FP32 rounding of P / phi (2^-22) and of the result, and the
                  fixed-point step 2^-31 of the row maximum per photon
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _data(side, N, R, npa, top, seed):
    import emc_b200 as E
    rng = np.random.default_rng(seed)
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    q, w = E.generate_rotations(3)
    pick = rng.permutation(len(w))[:R]
    mask = np.zeros(side * side, np.int32)
    mask[rng.permutation(side * side)[:npa]] = 1
    counts = rng.poisson(1.0, (N, side * side)).astype(np.float32)
    counts[rng.random(counts.shape) < 0.02] = top
    counts[:, rng.integers(side * side)] = top
    if N > 2:
        counts[1] = 0  # a pattern without photons
    model = (rng.random(side ** 3) * np.exp(rng.normal(0, 1.5, side ** 3))).astype(np.float32)
    return dict(x=x, y=y, z=z, q=q[pick].copy(), w=w[pick].copy(), mask=mask, counts=counts,
                model0=model, scaling0=(0.5 + rng.random(N)).astype(np.float32), side=side)


def _context(d, lik, interp):
    import emc_b200 as E
    ctx = E.Context(d["side"], len(d["counts"]), len(d["w"]), likelihood=lik, interp=interp)
    ctx.set_geometry(d["x"], d["y"], d["z"], d["mask"])
    ctx.set_rotations(d["q"], d["w"])
    ctx.set_patterns(d["counts"])
    ctx.set_model(d["model0"])
    ctx.set_scaling(d["scaling0"])
    return ctx


@pytest.mark.parametrize("lik,interp", [("gauss", "nearest"), ("poisson", "trilinear")])
@pytest.mark.parametrize("N,R,npa,top", [
    (1, 1, 1, 3), (15, 127, 127, 127), (16, 128, 128, 100), (17, 129, 129, 128),
    (255, 257, 15, 127), (256, 130, 17, 200), (257, 300, 255, 2000), (129, 640, 257, 16383),
])
def test_stages_at_tile_edges(lik, interp, N, R, npa, top):
    import emc_b200 as E
    d = _data(18, N, R, npa, top, N * 1000 + R)
    act = np.flatnonzero(d["mask"])
    K = d["counts"][:, act].astype(np.float64)
    cfg = O.make_config(18, N, R, interp=O.TRILINEAR if interp == "trilinear" else O.NEAREST,
                        likelihood=O.LL_POISSON if lik == "poisson" else O.LL_GAUSS)
    with _context(d, lik, interp) as ctx:
        held = ctx.memory_used
        with _context(d, lik, interp) as plain:
            # a limit below what is held makes the byte operands go: the
            # CUDA-core contractions of the same calls
            plain.set_memory_limit(held - 1)
            assert plain.memory_used < held
            plain.expand()
            plain.maximize()
            P_plain, phi_plain = plain.get_buffer(E.BUF_RESP), plain.get_scaling()
        ctx.expand()
        S = ctx.get_buffer(E.BUF_SLICES).astype(np.float64)
        ctx.maximize()
        P = ctx.get_buffer(E.BUF_RESP)
        S_ref = O.expand(cfg, d["model0"], d["q"], d["x"], d["y"], d["z"])
        LL = O.loglik(cfg, S_ref, d["counts"], d["mask"], d["scaling0"])
        P_ref, _, _ = O.softmax(LL)
        per_count = np.abs(S).max() * (2.0 ** -31 + 2.0 ** -22)
        err = K.sum(1) * per_count
        if lik == "gauss":
            phi0 = d["scaling0"].astype(np.float64)
            err = (2 * err / phi0 + (S * S).sum(1).max() * 2.0 ** -22) / (2 * len(act) * 0.4 ** 2)
        else:
            err = err + d["scaling0"] * S_ref[:, act].sum(1).max() * 2.0 ** -22
        l1 = np.abs(P.astype(np.float64) - P_ref).sum(0)
        assert (l1 <= 2 * np.expm1(np.minimum(err, 1.0)) + 2.0 ** -20).all(), (l1 / err).max()
        # the CUDA-core form: its FP32 partial sums round each product's
        # neighbourhood too, 32 terms at a time
        plain_err = 2 * np.expm1(np.minimum(40 * err, 1.0)) + 2.0 ** -19
        assert (np.abs(P.astype(np.float64) - P_plain).sum(0) <= plain_err).all()
        np.testing.assert_allclose(ctx.get_scaling(), phi_plain, rtol=1e-5 + plain_err.max())
        # slice sums from the context's own P and phi
        T = P.astype(np.float64).sum(1)
        phi = ctx.get_scaling().astype(np.float64)
        ctx.compress_insert()
        U = ctx.get_buffer(E.BUF_SLICES)
        X = P / phi
        ref = X @ K / np.maximum(T, 1e-300)[:, None]
        step = X.max(1)[:, None] * 2.0 ** -31 * K.sum(0) / np.maximum(T, 1e-300)[:, None]
        live = T > 1e-10
        assert (np.abs(U - ref) <= step + 2.0 ** -21 * ref + 1e-30)[live].all()
        ctx.normalize()


def test_counts_that_are_not_integers_keep_the_cuda_core_form():
    """Fractional counts (and counts above two planes) cannot be bytes; an
    upload of small integers after them can."""
    import emc_b200 as E
    d = _data(16, 33, 140, 200, 50, 7)
    for scale in (0.5, 400.0):
        odd = dict(d, counts=d["counts"] * np.float32(scale))
        with _context(odd, "gauss", "nearest") as ctx, _context(d, "gauss", "nearest") as good:
            assert ctx.memory_used < good.memory_used
            ctx.iterate()
            cfg = O.make_config(16, 33, 140, likelihood=O.LL_GAUSS)
            m_ref, _, _, _ = O.iterate(cfg, odd["counts"], d["mask"], d["q"], d["w"], d["x"],
                                       d["y"], d["z"], d["model0"], d["scaling0"])
            m = ctx.get_model()
            assert np.linalg.norm(m - m_ref) <= 1e-5 * np.linalg.norm(m_ref)
            ctx.set_patterns(d["counts"])
            assert ctx.memory_used == good.memory_used
