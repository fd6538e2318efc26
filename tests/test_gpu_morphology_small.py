"""Sphere morphology of small, flat and one-row volumes (run with -m gpu): against the oracle, results
identical, and the scratch of a plane within what (radius + 3) planes take."""
import numpy as np
import pytest
import torch

import oracle
from maxibone_b200 import _lib, device
from maxibone_b200 import morphology as mo

pytestmark = pytest.mark.gpu


# Fewer words than warps, so that a warp takes 1 to 16 of them; volumes of fewer planes than a block
# and its radius reach; rows and words past the volume's edge in every tile.
@pytest.mark.parametrize("shape,r", [((1, 1, 1), 0), ((16, 16, 16), 1), ((16, 16, 16), 8), ((5, 40, 70), 12),
                                     ((20, 50, 97), 3), ((1, 300, 260), 32), ((2, 33, 257), 31), ((3, 1, 5000), 9),
                                     ((70, 1, 33), 32), ((65, 2, 40), 5), ((40, 90, 130), 16), ((9, 64, 1000), 4)])
def test_small_volumes_match_oracle(shape, r):
    rng = np.random.default_rng(sum(shape) + r)
    m = (rng.random(shape) > 0.99).astype(np.uint8)
    m[tuple(rng.integers(0, n) for n in shape)] = 2
    for mask, dilate, fn in ((m, True, mo.dilate_3d_sphere), ((m == 0).astype(np.uint8) * 3, False, mo.erode_3d_sphere)):
        out = np.full(shape, 9, np.uint8)
        fn(mask, r, out)
        np.testing.assert_array_equal(out, oracle.morphology_sphere(mask, r, dilate))


@pytest.mark.parametrize("nz,r", [(1, 32), (3, 16), (12, 5)])
def test_scratch_of_few_planes(nz, r):
    shape = (nz, 4096, 8192)
    plane = shape[1] * shape[2] // 8
    mask = torch.zeros(shape, dtype=torch.uint8, device="cuda")
    mask[:, ::50, ::70] = 1
    out = torch.empty_like(mask)
    torch.cuda.synchronize()
    mo.dilate_3d_sphere(mask[:, :64, :64].contiguous(), r, out[:, :64, :64].contiguous())  # loads the kernels
    assert _lib.lib().maxi_release_cached_memory() == 0
    before = torch.cuda.mem_get_info()[0]
    mo.dilate_3d_sphere(mask, r, out)
    used = before - torch.cuda.mem_get_info()[0]
    assert used <= (r + 3) * nz * plane + (8 << 20)
    packed = device.bitpack(mask).view(nz, shape[1], shape[2] // 32)
    if r <= 15:  # the bit-packed form's x offsets reach 31 - r: the whole sphere up to 15
        result = torch.empty_like(packed)
        mo.dilate_3d_sphere_bitpacked(packed, r, result)
        assert torch.equal(device.bitunpack(result, mask.numel()).view(shape), out)
    _lib.lib().maxi_release_cached_memory()
