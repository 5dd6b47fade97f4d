"""Trilinear insertion by pairs of voxels along x, at odd and even sides (rows
of voxels start at odd and even indices) and with pixels beyond the grid:
against the oracle's insertion of the engine's own responsibilities, from
lists (poisson) and from the dense contraction (gaussian).

A voxel sums about n = 8 R pixels / side^3 FP32 terms in any order, so its
relative error is below n 2^-24 (all terms positive); the dense slice sums add
the FP32 accumulation of N patterns in the contraction."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [15, 16, 17, 33])
@pytest.mark.parametrize("lik", ["poisson", "gauss"])
def test_insertion_matches_oracle(side, lik):
    import emc_b200 as E
    rng = np.random.default_rng(side)
    x, y, z = E.detector_coordinates(side, 1e-10, 2.0 / side, 1.0)
    q, w = E.generate_rotations(3)
    N, R, npix = 70, len(w), side * side
    # coordinates stretched past the grid: corners outside on both ends
    x, y = (np.ascontiguousarray(1.2 * t, np.float32) for t in (x, y))
    mask = (rng.random(npix) < 0.9).astype(np.int32)
    counts = rng.poisson(2.0, (N, npix)).astype(np.float32)
    model = (0.2 + rng.random(side ** 3)).astype(np.float32)
    cfg = O.make_config(side, N, R, interp=O.TRILINEAR,
                        likelihood=O.LL_POISSON if lik == "poisson" else O.LL_GAUSS)
    with E.Context(side, N, R, likelihood=lik, interp="trilinear", precision="mixed") as ctx:
        ctx.set_geometry(x, y, z, mask)
        ctx.set_rotations(q, w)
        ctx.set_patterns(counts)
        ctx.set_model(model)
        ctx.set_scaling(np.ones(N, np.float32))
        ctx.set_sparse_compress(lik == "poisson")
        ctx.expand()
        ctx.maximize()
        P, phi = ctx.get_buffer(E.BUF_RESP).astype(np.float64), ctx.get_scaling()
        ctx.compress()
        got, weight = ctx.get_model(), ctx.get_buffer(E.BUF_WEIGHT)
    acc, wacc, _ = O.compress(cfg, P, counts, mask, phi.astype(np.float64), q, w, x, y, z)
    ref = O.normalize_model(acc, wacc)
    n = max(8 * R * mask.sum() / side ** 3, 64)
    tol = n * 2.0 ** -24 + (N * 2.0 ** -22 if lik == "gauss" else 2.0 ** -20)
    assert np.abs(weight - wacc).max() <= (tol + 1e-6) * wacc.max()
    assert np.linalg.norm(got - ref) <= (tol + 1e-6) * np.linalg.norm(ref)
    assert ((weight > 0) == (wacc > 0))[wacc > 1e-20 * wacc.max()].all()
