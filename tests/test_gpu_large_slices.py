"""cuda_get_slices of a model whose voxel index passes 32 bits (side^3 = 2.2e9
at side 1,300, 8.8 GB): every slice value is the model's voxel.  The model is
each voxel's own index hashed to 24 bits, so a value names its voxel."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Sp3Matrix(C.Structure):
    _fields_ = [("x", C.c_uint), ("y", C.c_uint), ("z", C.c_uint), ("data", C.c_void_p)]


@pytest.mark.parametrize("side", [1291, 1300])
def test_slices_of_a_model_beyond_32_bit_indices(side):
    import torch

    import emc_b200 as E
    L = E.lib()
    free, _ = torch.cuda.mem_get_info()
    if free < 5 * 4 * side ** 3:
        pytest.skip("needs 45 GB of device memory")
    v = torch.arange(side ** 3, device="cuda", dtype=torch.int64)
    model = ((v * 2654435761) >> 8 & 0xffffff).float()
    del v
    n = side * side
    # random points of the box, from its first voxels to its last
    rng = np.random.default_rng(side)
    k = rng.integers(1, side, (3, n))
    k[:, :4] = [[side - 1, 1, side - 1, 1]] * 2 + [[side - 1, side - 1, 1, 1]]
    c = side / 2 + 0.5
    xyz = [torch.from_numpy((a - c).astype(np.float32)).cuda() for a in k]
    quat = torch.tensor([1.0, 0.0, 0.0, 0.0], device="cuda")
    out = torch.full((n,), -1.0, device="cuda")
    m = Sp3Matrix(side, side, side, None)
    torch.cuda.synchronize()
    L.cuda_get_slices(C.byref(m), *[C.c_void_p(t.data_ptr()) for t in (model, out, quat, *xyz)], 1)
    assert L.emc_legacy_last_status() == 0
    pos = [torch.from_numpy(a).cuda() for a in k]
    # coordinates and their sum with the centre are halves: exact in FP32
    idx = (pos[2] * side + pos[1]) * side + pos[0]
    assert torch.equal(out, model[idx])
