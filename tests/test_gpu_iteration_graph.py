"""Iterations replayed as a CUDA graph against the same iterations launched one
by one (profiling keeps them so).  Every iteration starts from the same model
and scaling, so the two differ only in the order of the insertion's FP32
atomics: at most n 2^-24 of a voxel's sum of n positive contributions, here
n < 1,000 (1e-4 with the weights' sum).  Each phase has five iterations, of
which the first ones are launched and the last ones replayed, and changes what
the captured launches read or how many there have to be."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,lik,interp", [("fp32", "gauss", "nearest"), ("fp32", "poisson", "trilinear"),
                                             ("mixed", "poisson", "nearest"),
                                             ("mixed", "gauss", "trilinear")])
def test_replayed_iterations_follow_every_change(prec, lik, interp):
    import emc_b200 as E
    rng = np.random.default_rng(5)
    side, N, R = 20, 70, 300
    x, y, z = E.detector_coordinates(side, 1e-10, 1.0 / side, 1.0)
    qa, wa = E.generate_rotations(3)
    model = (0.1 + rng.random(side ** 3)).astype(np.float32)
    scale = (0.5 + rng.random(N)).astype(np.float32)
    mask = np.ones(side * side, np.int32)
    mask[rng.permutation(side * side)[:150]] = 0
    mask[0] = 1

    def counts(mean):
        k = rng.poisson(mean, (N, side * side)).astype(np.float32)
        k[:, 0] = 1
        return k
    first, dense, sparse, odd = counts(1.0), counts(8.0), counts(0.05), counts(1.0) * np.float32(0.5)

    def rotations(seed):
        pick = np.random.default_rng(seed).permutation(len(wa))[:R]
        return qa[pick].copy(), wa[pick].copy()

    phases = [lambda c: None,
              lambda c: c.set_patterns(dense),
              lambda c: c.set_patterns(sparse),
              lambda c: c.set_rotations(*rotations(2)),
              lambda c: c.set_sparse_compress(not c.tuning()["compress_sparse"]),
              lambda c: c.set_tuning(3, 3)]
    if prec == "fp32":  # not bytes, then no room for bytes: the CUDA-core contractions
        phases.insert(3, lambda c: c.set_patterns(odd))
        phases += [lambda c: c.set_patterns(first),
                   lambda c: c.set_memory_limit(c.memory_used - 1)]
    results = []
    for eager in (True, False):
        with E.Context(side, N, R, likelihood=lik, interp=interp, precision=prec) as ctx:
            ctx.set_profiling(eager)
            ctx.set_geometry(x, y, z, mask)
            ctx.set_rotations(*rotations(1))
            ctx.set_patterns(first)
            out = []
            for change in phases:
                change(ctx)
                for _ in range(5):
                    ctx.set_model(model)
                    ctx.set_scaling(scale)
                    st = ctx.iterate()
                    out.append((ctx.get_model(), ctx.get_scaling(), ctx.get_buffer(E.BUF_TOTALRESP),
                                st["total_loglik"]))
            results.append(out)
    for i, (a, b) in enumerate(zip(*results)):
        np.testing.assert_allclose(b[0], a[0], rtol=1e-4, atol=1e-6 * a[0].max(), err_msg=str(i))
        np.testing.assert_allclose(b[1], a[1], rtol=1e-6, err_msg=str(i))
        np.testing.assert_allclose(b[2], a[2], rtol=1e-5, atol=1e-12, err_msg=str(i))
        np.testing.assert_allclose(b[3], a[3], rtol=1e-9, err_msg=str(i))
