"""The axis histograms of few bins, few planes and long rows or columns (run with -m gpu): against
the oracle, counts identical, and not slower than with many bins."""
import numpy as np
import pytest
import torch

import oracle
from maxibone_b200.histograms import axis_histograms

pytestmark = pytest.mark.gpu


# Rings shared by several blocks (few bins, one plane); tall blocks, whose rows a ring meets above
# and below its centre only, with the centre inside, beside and beyond them; wide blocks with
# radii up to the largest whose square fits 31 bits and above.
@pytest.mark.parametrize("shape,offset,center,voxel_bins,n_r", [
    ((1, 900, 700), (0, 0, 0), (450, 350), 8, 571), ((1, 900, 700), (0, 100, 50), (450, 350), 64, 300),
    ((3, 700, 701), (0, 0, 0), (0, 700), 1, 1000), ((40, 300, 128), (0, 3, 9), (20, 60), 16, 290),
    ((2, 5000, 40), (0, 0, 0), (2500, 20), 64, 2501), ((2, 5000, 40), (0, 7, 3), (2500, 900), 64, 2700),
    ((2, 5000, 40), (0, 0, 0), (9000, 10), 512, 9001), ((30, 3, 3000), (0, 1, 0), (1, 1500), 512, 1501),
    ((1, 2, 70000), (0, 0, 0), (1, 0), 32, 70001), ((1, 2, 70000), (0, 0, 5), (0, 40000), 32, 40001),
    ((1, 2, 70000), (0, 0, 0), (0, 0), 32, 46276), ((1, 2, 70000), (0, 0, 0), (0, 0), 32, 46277),
    ((1, 70001, 3), (0, 0, 1), (70000, 1), 32, 70001),
])
def test_rings_match_oracle(shape, offset, center, voxel_bins, n_r):
    rng = np.random.default_rng(sum(shape) + voxel_bins)
    voxels = rng.integers(0, 45000, shape, dtype=np.uint16)
    want = oracle.axis_histograms(voxels, offset, shape, voxel_bins, n_r, center, (1.0, 32000.0))
    got = [np.full((n, voxel_bins), 3, np.uint64) for n in (shape[2], shape[1], shape[0], n_r)]
    axis_histograms(voxels, offset, *got, center, (1.0, 32000.0), 0)
    for g, w, name in zip(got, want, ("x", "y", "z", "r")):
        np.testing.assert_array_equal(g, w + np.uint64(3), err_msg=name)


def _time(shape, voxel_bins):
    nz, ny, nx = shape
    g = torch.Generator(device="cuda").manual_seed(1)
    voxels = (torch.rand(shape, generator=g, device="cuda") * 31000).to(torch.int16)
    n_r = int(np.hypot(ny // 2, nx // 2)) + 1
    bins = [torch.zeros((n, voxel_bins), dtype=torch.int64, device="cuda") for n in (nx, ny, nz, n_r)]
    times = []
    for _ in range(6):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        begin.record()
        axis_histograms(voxels, (0, 0, 0), *bins, (ny // 2, nx // 2), (1.0, 32000.0))
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    return min(times)


# With few bins the radial histogram once ran in a handful of blocks: 10 times the time of 512
# bins at these sizes.
@pytest.mark.parametrize("shape", [(1, 4096, 4096), (64, 1024, 1024)])
def test_few_bins_take_no_longer(shape):
    assert _time(shape, 64) <= 2.0 * _time(shape, 512)


# A block without a counted voxel ends after the first of the four histograms; one counted voxel, at
# the block's first and last place and beside an offset, brings the others.
@pytest.mark.parametrize("where", [None, (0, 0, 0), (11, 150, 299), (5, 3, 40)])
@pytest.mark.parametrize("voxel_bins", [16, 4096])
def test_blocks_with_hardly_a_counted_voxel(where, voxel_bins):
    shape, offset = (12, 151, 300), (0, 0, 0)
    voxels = np.zeros(shape, np.uint16)
    voxels[::3] = 65535
    if where == (5, 3, 40):
        offset = (0, 3, 40)
        voxels[:, :3] = voxels[:, :, :40] = 900
    if where:
        voxels[where] = 20000
    n_r = 169
    want = oracle.axis_histograms(voxels, offset, shape, voxel_bins, n_r, (75, 150), (1.0, 32000.0))
    assert (want[2].sum() > 0) == bool(where)
    got = [np.full((n, voxel_bins), 3, np.uint64) for n in (shape[2], shape[1], shape[0], n_r)]
    axis_histograms(voxels, offset, *got, (75, 150), (1.0, 32000.0), 0)
    for g, w, name in zip(got, want, ("x", "y", "z", "r")):
        np.testing.assert_array_equal(g, w + np.uint64(3), err_msg=name)
