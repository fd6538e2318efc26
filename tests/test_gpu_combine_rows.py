"""The field combination of a few long rows (run with -m gpu): against the oracle, bit for bit, and as fast
as of many short ones."""
import numpy as np
import pytest
import torch

import oracle
from maxibone_b200.fields import combine_fields

pytestmark = pytest.mark.gpu


# Rows so long and few that several warps or blocks share each: whole and ragged ends, rows that start
# inside a 16-byte word, one row.
@pytest.mark.parametrize("shape", [(1, 1, 1 << 18), (1, 1, 100003), (1, 3, 40008), (2, 4, 16384), (1, 7, 20001)])
def test_long_rows_match_oracle(shape):
    rng = np.random.default_rng(sum(shape))
    g = rng.integers(1, 60000, shape, dtype=np.uint16)
    e = rng.integers(1, 65535, shape, dtype=np.uint16)
    np.testing.assert_array_equal(combine_fields(g, e), oracle.combine_fields(g, e))


def _device_us(shape):
    from torch.profiler import ProfilerActivity, profile

    g = torch.Generator(device="cuda").manual_seed(1)
    gauss, edt = (torch.randint(1, 60000, shape, generator=g, device="cuda", dtype=torch.int32).to(torch.int16)
                  for _ in range(2))
    out = torch.empty_like(gauss)
    combine_fields(gauss, edt, out)
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        combine_fields(gauss, edt, out)
        torch.cuda.synchronize()
    times = [e.device_time for e in p.events() if "combined_" in e.name]
    if len(times) != 2:
        pytest.skip("no kernel times from the profiler")
    return sum(times)


# A few long rows once ran on a warp each, 300 times longer than as many voxels in short rows.
def test_long_rows_fill_the_chip():
    assert _device_us((1, 4, 1 << 22)) <= 4.0 * _device_us((1, 4096, 4096))
