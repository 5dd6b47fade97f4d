"""A batch with more tiles than SMs or SM pairs, its datasets of unequal depth:
the tile list handed out by load, the datasets' own stages on streams of their
own, directly and replayed, against the datasets iterated one by one (FP32
atomics in another order: 1e-5, as in the other batch tests)."""
import numpy as np
import pytest

from parity import make_ctx, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lists", [True, False])
def test_unequal_datasets_with_more_tiles_than_sms(lists):
    import emc_b200 as E
    from emc_b200 import workloads as W
    sizes = [(32, 4, 700), (16, 4, 1100), (24, 3, 130), (16, 2, 1)]
    ds = [W.make(W.Workload(f"b{i}", s, lv, n, 400.0, 0.3, 2.0, 1, seed=10 + i))
          for i, (s, lv, n) in enumerate(sizes)]
    refs = []
    for d in ds:
        with make_ctx(d, "poisson", "nearest", "mixed") as c:
            c.set_sparse_compress(lists)
            for _ in range(4):
                c.iterate()
            refs.append((c.get_model(), c.get_scaling()))
    ctxs = [make_ctx(d, "poisson", "nearest", "mixed") for d in ds]
    try:
        for c in ctxs:
            c.set_sparse_compress(lists)
        with E.Batch(ctxs) as b:
            b.iterate()
            b.synchronize()
            b.capture()
            b.launch(3)
            b.synchronize()
            for c, (m, s) in zip(ctxs, refs):
                assert rel(c.get_model(), m) < 1e-5
                assert rel(c.get_scaling(), s) < 1e-5
    finally:
        for c in ctxs:
            c.close()
