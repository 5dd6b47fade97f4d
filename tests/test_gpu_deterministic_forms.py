"""Deterministic contexts: which form a contraction takes follows from the data
and the tuning alone, neither from the memory that happens to be free nor from
what earlier iterations made room for, so a run continued in a fresh context is
bitwise the run that went on."""
import numpy as np
import pytest

from parity import make_ctx

pytestmark = pytest.mark.gpu


def _state(ctx):
    import emc_b200 as E
    return ctx.get_model(), ctx.get_buffer(E.BUF_WEIGHT), ctx.get_scaling()


@pytest.mark.parametrize("lik", ["gauss", "poisson"])
def test_fp32_does_not_depend_on_the_memory_left(lik):
    from emc_b200 import workloads as W
    d = W.make("small32")
    out = []
    for limited in (False, True):
        with make_ctx(d, lik) as ctx:
            ctx.set_deterministic(True)
            if limited:
                ctx.set_memory_limit(ctx.memory_used - 1)
                ctx.set_patterns(d["counts"])  # under the limit
            ctx.iterate()
            ctx.iterate()
            out.append(_state(ctx))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_a_resumed_mixed_run_takes_the_same_lists(tmp_path):
    """1,500 patterns of 60 photons: the second iteration keeps more entries
    than a fresh context has room for, and fewer than lists are worth."""
    from test_gpu_list_growth import _context
    path = str(tmp_path / "state")
    with _context() as ctx:
        ctx.set_deterministic(True)
        ctx.iterate()
        ctx.save_state(path, 1)
        ctx.iterate()
        after = ctx.memory_used
        ctx.load_state(path)
        ctx.iterate()  # the second iteration again, with room from the first time
        went_on = _state(ctx)
    with _context() as ctx:
        ctx.set_deterministic(True)
        ctx.load_state(path)
        ctx.iterate()
        assert ctx.memory_used == after  # room was made within the iteration
        for a, b in zip(went_on, _state(ctx)):
            np.testing.assert_array_equal(a, b)
