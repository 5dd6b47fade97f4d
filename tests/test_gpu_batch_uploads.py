"""A captured batch after what its datasets' own calls may change: patterns
uploaded anew (longer and shorter photon lists), iterations of a member on its
own, another tuning.  Every replay is the separate iteration's result from the
same model and scaling, up to the order of the insertion's FP32 sums (at most n
2^-24 of a voxel's sum of n < 160 contributions: 1e-5); a second iteration would
carry that difference through the posteriors."""
import numpy as np
import pytest

from parity import make_ctx, rel

pytestmark = pytest.mark.gpu


def _datasets():
    from emc_b200 import workloads as W
    ws = [W.Workload("b16", 16, 2, 64, 400.0, 0.3, 1.5, 1, seed=1),
          W.Workload("b24", 24, 3, 200, 600.0, 0.3, 2.0, 1, seed=2)]
    return [W.make(w) for w in ws]


def test_a_captured_batch_follows_its_datasets():
    import emc_b200 as E
    ds = _datasets()
    rng = np.random.default_rng(1)
    counts = [[d["counts"],
               rng.permutation(d["counts"]),                                      # other photons
               np.minimum(d["counts"], 1) * (rng.random(d["counts"].shape) < .3),  # shorter lists
               d["counts"] + (rng.random(d["counts"].shape) < .5)]                 # longer ones
              for d in ds]
    ctxs = [make_ctx(d, "poisson", "nearest", "mixed") for d in ds]
    solo = [make_ctx(d, "poisson", "nearest", "mixed") for d in ds]
    try:
        with E.Batch(ctxs) as b:
            b.capture()
            for step in range(1, 6):
                who = step % 2
                for group in (ctxs, solo):
                    if step < 4:
                        for c, k in zip(group, counts):
                            c.set_patterns(np.ascontiguousarray(k[step], np.float32))
                    elif step == 4:
                        group[who].iterate()  # a member on its own in between
                    else:
                        group[who].set_tuning(3, 3)
                    for c, d in zip(group, ds):
                        c.set_model(d["model0"])
                        c.set_scaling(d["scaling0"])
                b.launch(1)
                b.synchronize()
                for c in solo:
                    c.iterate()
                for c, r in zip(ctxs, solo):
                    assert rel(c.get_model(), r.get_model()) < 1e-5, step
                    assert rel(c.get_scaling(), r.get_scaling()) < 1e-5, step
            # captured again right after an upload
            for c, s, k in zip(ctxs, solo, counts):
                c.set_patterns(k[0])
                s.set_patterns(k[0])
            b.capture()
            for group in (ctxs, solo):
                for c, d in zip(group, ds):
                    c.set_model(d["model0"])
                    c.set_scaling(d["scaling0"])
            b.launch(1)
            b.synchronize()
            for c, s in zip(ctxs, solo):
                s.iterate()
                assert rel(c.get_model(), s.get_model()) < 1e-5
    finally:
        for c in ctxs + solo:
            c.close()
