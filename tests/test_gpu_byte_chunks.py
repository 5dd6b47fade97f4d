"""FP32 contexts whose digit planes do not fit 2 GB contract over chunks of
rotations: 36,540 rotations x 16,384 pixels are two, of 18,304 and 18,236.  The
memory that the byte operands take stays bounded.  Responsibilities and slice
sums against 64 bits of the context's own slices and responsibilities, by chunk
edge and overall.  Responsibilities: |LL - lse| < 32 where they count, rounded to
FP32 and through expf, 36 2^-24; slice sums: P / phi (2^-22), nine terms and the
result, (9 + 8) 2^-24 of a value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
def test_chunks_of_rotations(lik):
    import torch

    import emc_b200 as E
    rng = np.random.default_rng(8)
    side, N = 128, 9
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    q, w = E.generate_rotations(9)
    R = len(w)
    assert R == 36540
    # few photons: posteriors spread over the rotations of both chunks
    counts = (rng.random((N, side * side)) < 5e-4).astype(np.float32)
    counts[2, 7] = 200  # two count planes
    model = (0.5 + rng.random(side ** 3)).astype(np.float32)
    scale = np.maximum(counts.sum(1), 1) / np.float32(side * side)
    K = torch.from_numpy(counts).cuda().double()

    def buffer(ctx, which, cols):
        ptr, nbytes = ctx.device_buffer(which)
        ctx.synchronize()
        t = torch.as_tensor(E._CudaArray(ptr, nbytes // 4), device="cuda")
        return t.reshape(R, cols).double()

    with E.Context(side, N, R, likelihood=lik) as ctx:
        ctx.set_geometry(x, y, z, np.ones(side * side, np.int32))
        ctx.set_rotations(q, w)
        before = ctx.memory_used
        ctx.set_patterns(counts)
        # besides the staging of the images: digits of every rotation are 2.39e9
        assert ctx.memory_used - before < 2.2e9
        ctx.set_model(model)
        ctx.set_scaling(scale)
        ctx.expand()
        S = buffer(ctx, E.BUF_SLICES, side * side)
        phi = torch.from_numpy(scale).cuda().double()
        if lik == "poisson":
            LL = S @ K.T - S.exp().sum(1)[:, None] * phi
        else:
            inv = 1 / (2 * side * side * 0.4 ** 2)
            LL = (2 * (S @ K.T) / phi - (S * S).sum(1)[:, None] - (K * K).sum(1) / phi ** 2) * inv
        del S
        P_ref = torch.softmax(LL, 0)
        ctx.maximize()
        P = buffer(ctx, E.BUF_RESP, N)
        phi = torch.from_numpy(ctx.get_scaling()).cuda().double()
        ctx.compress_insert()
        U = buffer(ctx, E.BUF_SLICES, side * side)
        T = P.sum(1)
        U_ref = (P / phi) @ K / T.clamp_min(1e-300)[:, None]
        live = T > 1e-10
        assert live[:18304].any() and live[18304:].any()
        for rows in (slice(0, 128), slice(18176, 18304), slice(18304, 18432), slice(R - 128, R),
                     slice(0, R)):
            # poisson: sum W of the slices' rounded logarithms (2^-22 of phi sum W)
            tol = 36 * 2.0 ** -24 + (2.0 ** -22 * 10 if lik == "poisson" else 0)
            assert (P[rows] - P_ref[rows]).norm() <= tol * P_ref[rows].norm(), rows
            err = (U[rows] - U_ref[rows])[live[rows]].abs()
            assert (err <= 17 * 2.0 ** -24 * U_ref[rows][live[rows]] + 1e-30).all(), rows
        ctx.normalize()
        assert np.isfinite(ctx.get_model()).all()
