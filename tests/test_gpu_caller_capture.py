"""An iteration captured by the caller into a CUDA graph of its own, right
after uploads that may still be in flight and after iterations whose list count
may be, against ordinary iterations.  A replay works on what the context holds
then: after an upload of other patterns (other photon lists, counts of another
width) it gives what an ordinary iteration gives.  Replay and iteration differ
by the order of FP32 sums, and in the mixed contexts by the FP16 split of the
dense compress operand (22 bits of P / (T phi)): 1e-5 of the model's norm.  A
captured FP32 iteration contracts on the CUDA cores, so its replay is compared
with a context that a memory limit keeps on them (their FP32 sums of (S - K /
phi)^2 are further than that from the byte contractions where counts are in
the hundreds)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE, N, R = 20, 70, 300


def _counts(rng, mean, top=0):
    k = rng.poisson(mean, (N, SIDE * SIDE)).astype(np.float32)
    k[:, 5] = 1 + top
    return k


@pytest.mark.parametrize("before", [0, 3])
@pytest.mark.parametrize("prec,lik,lists", [("mixed", "poisson", True), ("mixed", "poisson", False),
                                            ("mixed", "gauss", True), ("fp32", "gauss", False),
                                            ("fp32", "poisson", False)])
def test_an_iteration_captured_by_the_caller(prec, lik, lists, before):
    import torch

    import emc_b200 as E
    rng = np.random.default_rng(11)
    x, y, z = E.detector_coordinates(SIDE, 1e-10, 1.0 / SIDE, 1.0)
    qa, wa = E.generate_rotations(3)
    pick = rng.permutation(len(wa))[:R]
    mask = np.ones(SIDE * SIDE, np.int32)
    mask[rng.permutation(SIDE * SIDE)[:150]] = 0
    mask[5] = 1
    model = (0.1 + rng.random(SIDE ** 3)).astype(np.float32)
    scale = (0.5 + rng.random(N)).astype(np.float32)
    uploads = [_counts(rng, 1.0), _counts(rng, 0.2), _counts(rng, 3.0, 400), _counts(rng, 1.5)]

    def context():
        ctx = E.Context(SIDE, N, R, likelihood=lik, precision=prec)
        ctx.set_geometry(x, y, z, mask)
        ctx.set_rotations(qa[pick].copy(), wa[pick].copy())
        ctx.set_patterns(uploads[0])
        if prec == "mixed":
            ctx.set_sparse_compress(lists)
        return ctx

    def start(ctx):
        ctx.set_model(model)
        ctx.set_scaling(scale)

    def check(a, b, what):
        for u, v in ((a.get_model(), b.get_model()), (a.get_scaling(), b.get_scaling())):
            assert np.isfinite(u).all()
            assert np.linalg.norm(u - v) <= 1e-5 * np.linalg.norm(v), what

    with context() as ctx, context() as ref, context() as same:
        if prec == "fp32":
            same.set_memory_limit(same.memory_used - 1)
        for c in (ctx, ref, same):
            start(c)
            for _ in range(before):
                c.iterate(stats=False)
            start(c)
        stream = torch.cuda.ExternalStream(ctx.stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            ctx.iterate(stats=False)
        for k, counts in enumerate(uploads):
            for c in (ctx, ref, same):
                if k:
                    c.set_patterns(counts)
                start(c)
            ctx.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            same.iterate()
            ctx.synchronize()
            check(ctx, same, ("replay", k))
            # ordinary iterations in between, whose lists may be built anew
            for c in (ctx, ref):
                start(c)
                for _ in range(4):
                    c.iterate(stats=False)
                c.synchronize()
            check(ctx, ref, ("iterations", k))
        del graph
