"""Sphere morphology where its tiles and blocks of planes end (run with -m gpu): against the
oracle, results identical."""
import numpy as np
import pytest
import torch

import oracle
from maxibone_b200 import morphology as mo

pytestmark = pytest.mark.gpu


# Rows around the 32-row tile; rows of 3, 8, 9, 16 and 17 words (tiles of 8 and 16 words, scratch
# rows of a multiple of 4); plane counts that leave a last block of one plane; the radii at
# both ends of the buckets that the kernel is compiled for (multiples of 4), 0 and the
# largest.  A few set (or cleared) voxels, so that a wrong neighbour shows.
@pytest.mark.parametrize("shape,r", [((33, 33, 96), 4), ((40, 31, 257), 5), ((49, 64, 288), 8), ((7, 65, 512), 9),
                                     ((97, 32, 544), 12), ((5, 63, 70), 13), ((50, 40, 300), 17), ((3, 96, 520), 24),
                                     ((64, 33, 33), 28), ((35, 34, 260), 29), ((2, 2, 600), 32), ((1, 1, 1), 3)])
def test_tile_edges_match_oracle(shape, r):
    rng = np.random.default_rng(r)
    m = (rng.random(shape) > 0.999).astype(np.uint8)
    m[tuple(rng.integers(0, n) for n in shape)] = 2  # nonzero, bit 0 clear
    for mask, dilate, fn in ((m, True, mo.dilate_3d_sphere), ((m == 0).astype(np.uint8) * 3, False, mo.erode_3d_sphere)):
        out = np.full(shape, 9, np.uint8)
        fn(mask, r, out)
        np.testing.assert_array_equal(out, oracle.morphology_sphere(mask, r, dilate))


# Few blocks and many: the same result whatever the planes per block come to (a slab of the
# volume, far enough from its cut faces, is the slab of the result).
@pytest.mark.parametrize("r", [3, 16, 20])
def test_slab_of_a_large_volume_equals_its_own_run(r):
    g = torch.Generator(device="cuda").manual_seed(r)
    m = (torch.rand((300, 260, 512), generator=g, device="cuda") > 0.9998).to(torch.uint8)
    whole, slab = torch.empty_like(m), torch.empty_like(m[100:180])
    mo.dilate_3d_sphere(m, r, whole)
    mo.dilate_3d_sphere(m[100:180].contiguous(), r, slab)
    assert torch.equal(slab[r:-r], whole[100 + r:180 - r])
    # unaligned uint8 rows take the other pack and unpack
    flat = torch.zeros(m.numel() + 1, dtype=torch.uint8, device="cuda")
    shifted = flat[1:].view(m.shape)
    shifted.copy_(m)
    out = torch.empty_like(m)
    mo.dilate_3d_sphere(shifted, r, out)
    assert torch.equal(out, whole)
