"""The field combination over every value of its divisors' range and at the edges of its row walk
(run with -m gpu): against the oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from maxibone_b200.fields import combine_fields

pytestmark = pytest.mark.gpu


# Every uint16 value up to the field's maximum, for small, odd, all-ones and even maxima; the
# two fields run against each other so that their difference takes many values.
@pytest.mark.parametrize("gmax,emax", [(65535, 65535), (65534, 3), (1, 40961), (32767, 32768), (49999, 257), (2, 2)])
def test_every_value_of_both_fields(gmax, emax):
    n = 65536
    g = (np.arange(n) % (gmax + 1)).astype(np.uint16)
    e = ((np.arange(n)[::-1] * 7919) % (emax + 1)).astype(np.uint16)
    g[-1], e[0] = gmax, emax
    g, e = g.reshape(1, 256, 256), e.reshape(1, 256, 256)
    np.testing.assert_array_equal(combine_fields(g, e), oracle.combine_fields(g, e))


# Rows shorter than, equal to and longer than the lanes of one row; rows without 16-byte
# alignment; planes with no voxel inside the cylinder or none outside it; equal fields
# (the difference is 0 everywhere, and so is the range).
@pytest.mark.parametrize("shape,same", [((3, 40, 8), False), ((2, 31, 256), False), ((2, 30, 264), False),
                                        ((1, 9, 1000), False), ((4, 17, 250), False), ((2, 1, 64), False),
                                        ((1, 2, 2), False), ((5, 1, 1), False), ((2, 33, 72), True)])
def test_row_walks_match_oracle(shape, same):
    rng = np.random.default_rng(sum(shape))
    g = rng.integers(1, 60000, shape, dtype=np.uint16)
    e = g.copy() if same else rng.integers(1, 65535, shape, dtype=np.uint16)
    want = oracle.combine_fields(g, e)
    np.testing.assert_array_equal(combine_fields(g, e), want)
    # a view that is not 16-byte aligned
    n = g.size
    flat = torch.zeros((3, n + 1), dtype=torch.int16, device="cuda")
    views = [flat[k, 1:].view(shape) for k in range(3)]
    views[0].copy_(torch.from_numpy(g.view(np.int16)))
    views[1].copy_(torch.from_numpy(e.view(np.int16)))
    combine_fields(views[0], views[1], views[2])
    np.testing.assert_array_equal(views[2].cpu().numpy().view(np.uint16), want)
