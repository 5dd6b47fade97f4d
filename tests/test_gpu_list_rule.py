"""Mixed contexts compress from responsibility lists only while the lists are
short enough to be faster; broad posteriors take the dense contraction.  Both
give the same model: the dense operand keeps 22 bits of P / (T phi) and sums
in FP32 (measured within 1e-6 of the lists), so 1e-5 over three iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lik,N", [("gauss", 300), ("gauss", 129), ("poisson", 256)])
def test_list_rule_agrees_with_the_dense_contraction(lik, N):
    import emc_b200 as E
    from emc_b200 import workloads as W
    d = W.make("small32", n_patterns=N)
    models = []
    for lists in (True, False):
        with E.Context(32, N, len(d["w"]), likelihood=lik, precision="mixed") as ctx:
            ctx.set_geometry(d["x"], d["y"], d["z"], d["mask"])
            ctx.set_rotations(d["q"], d["w"])
            ctx.set_patterns(d["counts"])
            ctx.set_model(d["model0"])
            ctx.set_scaling(d["scaling0"])
            ctx.set_sparse_compress(lists)
            held = []
            for _ in range(3):
                ctx.iterate()
                held.append(ctx.memory_used)
            models.append(ctx.get_model())
            if lists and lik == "gauss":
                # entries of every pair would need 20 bytes each: never grown
                assert held[-1] == held[0]
    a, b = models
    assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
