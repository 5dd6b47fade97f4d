"""FP32 contexts, stage by stage: scaling, responsibilities and slices that the
program changes between two stages count as they are then, on the byte
contractions as on the CUDA cores (which a memory limit below what is held
brings back).  The two forms differ by FP32 partial sums: 1e-5 of the norm.
The last case leaves every responsibility as it is and takes the scaling far
down, where fixed point relative to an outdated row maximum would overflow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE, N, R = 18, 90, 260


def _tensor(ctx, which):
    import torch

    import emc_b200 as E
    ptr, nbytes = ctx.device_buffer(which)
    return torch.as_tensor(E._CudaArray(ptr, nbytes // 4), device="cuda")


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
@pytest.mark.parametrize("factor", [0.97, 0.5, 1e-3, 40.0])
@pytest.mark.parametrize("change", ["scaling", "one_scaling", "responsibilities", "slices"])
def test_changes_between_stages(lik, factor, change):
    import torch

    import emc_b200 as E
    rng = np.random.default_rng(3)
    x, y, z = E.detector_coordinates(SIDE, 1e-10, 1.0 / SIDE, 1.0)
    qa, wa = E.generate_rotations(3)
    pick = rng.permutation(len(wa))[:R]
    mask = np.ones(SIDE * SIDE, np.int32)
    model = (0.1 + rng.random(SIDE ** 3)).astype(np.float32)
    counts = rng.poisson(1.0, (N, SIDE * SIDE)).astype(np.float32)
    out = []
    for plain in (False, True):
        with E.Context(SIDE, N, R, likelihood=lik) as ctx:
            ctx.set_geometry(x, y, z, mask)
            ctx.set_rotations(qa[pick].copy(), wa[pick].copy())
            ctx.set_patterns(counts)
            held = ctx.memory_used
            if plain:
                ctx.set_memory_limit(held - 1)
                assert ctx.memory_used < held
            ctx.set_model(model)
            ctx.set_scaling(np.ones(N, np.float32))
            ctx.expand()
            if change == "slices":
                ctx.synchronize()
                _tensor(ctx, E.BUF_SLICES).mul_(min(factor, 2.0))
                torch.cuda.synchronize()
            ctx.maximize()
            phi = ctx.get_scaling()
            if change == "scaling":
                ctx.set_scaling(phi * np.float32(factor))
            elif change == "one_scaling":
                phi[::7] *= np.float32(factor)
                ctx.set_scaling(phi)
            elif change == "responsibilities":
                _tensor(ctx, E.BUF_RESP).mul_(factor)
                torch.cuda.synchronize()
            ctx.compress_insert()
            U = ctx.get_buffer(E.BUF_SLICES)
            ctx.normalize()
            out.append((U, ctx.get_model(), ctx.get_scaling()))
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
