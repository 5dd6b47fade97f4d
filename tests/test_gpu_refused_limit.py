"""A memory limit that cannot be met is refused and changes nothing; one that
can be met by giving the faster operands of an FP32 context back is accepted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
def test_a_refused_limit_gives_nothing_back(lik):
    import emc_b200 as E
    rng = np.random.default_rng(3)
    side, N, R = 18, 90, 260
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    qa, wa = E.generate_rotations(3)
    with E.Context(side, N, R, likelihood=lik) as ctx:
        ctx.set_geometry(x, y, z, np.ones(side * side, np.int32))
        ctx.set_rotations(qa[:R].copy(), wa[:R].copy())
        counts = rng.poisson(1.0, (N, side * side)).astype(np.float32)
        ctx.set_patterns(counts)
        held = ctx.memory_used
        for limit in (1, held // 100):
            with pytest.raises(E.EmcError) as ei:
                ctx.set_memory_limit(limit)
            assert ei.value.status == 1
            assert ctx.memory_used == held
        ctx.set_memory_limit(held)  # holds as it is
        assert ctx.memory_used == held
        ctx.set_memory_limit(held - 1)
        less = ctx.memory_used
        assert less < held
        # without the limit the next upload has the operands back
        ctx.set_memory_limit(0)
        ctx.set_patterns(counts)
        assert less < ctx.memory_used <= held
