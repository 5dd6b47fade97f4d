"""Mixed contexts whose memory limit has room for the compacted entries but not
for lists as long as those could get (256 patterns x 3,240 rotations: 15.7 MB
and 13.1 MB) iterate all the same, from shorter lists or, in iterations that
keep more entries, from the dense operand: within 1e-5 of the iterations without
a limit (the dense operand keeps 22 bits of P / (T phi))."""
import numpy as np
import pytest

from parity import make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", ["iterate", "stages"])
@pytest.mark.parametrize("room", [17 << 20, 20 << 20, 27 << 20])
def test_no_room_for_lists(room, run):
    from emc_b200 import workloads as W
    d = W.make("small32")

    def iterate(ctx):
        if run == "iterate":
            ctx.iterate(stats=False)
        else:
            ctx.expand()
            ctx.maximize()
            ctx.compress()

    models = []
    for limited in (False, True):
        with make_ctx(d, "poisson", "nearest", "mixed") as ctx:
            held = ctx.memory_used
            if limited:
                ctx.set_memory_limit(held + room)
            for _ in range(5):
                iterate(ctx)
            ctx.synchronize()
            if limited:
                assert ctx.memory_used <= held + room
            models.append(ctx.get_model())
    a, b = models
    assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
