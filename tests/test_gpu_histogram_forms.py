"""The histograms' shared-memory forms where their tiles, strips and rings end (run with
-m gpu): against the oracle, counts identical."""
import numpy as np
import pytest

import oracle
from maxibone_b200.histograms import axis_histograms, field_histogram

pytestmark = pytest.mark.gpu


def _voxels(shape, seed, hi):
    rng = np.random.default_rng(seed)
    v = rng.integers(0, hi, shape, dtype=np.uint16)
    v[rng.random(shape) < 0.2] = 0
    return v


# Volumes above the size at which the direct form gives way.  Rows with and without 16-byte
# alignment, a last strip of one voxel, offsets inside a vector; centres in the middle, at a
# corner and outside, radii cut off by n_r; bins of one word up to the most that the shared
# forms take and one more; ranges whose bins need the thresholds (76 bins over 1 .. 76, 2304
# over 1 .. 2304), since no fixed-point line gives them.
@pytest.mark.parametrize("gshape,nzb,offset,center,voxel_bins,vrange,n_r", [
    ((20, 96, 128), 20, (0, 0, 0), (48, 64), 512, (1.0, 32000.0), 81),
    ((20, 96, 128), 20, (0, 5, 13), (48, 64), 4096, (1.0, 32000.0), 50),
    ((19, 97, 129), 19, (0, 0, 0), (0, 0), 1000, (1, 40000), 200),
    ((40, 64, 89), 30, (7, 3, 8), (500, 10), 8192, (100.5, 30000.25), 600),
    ((3, 300, 344), 3, (0, 0, 16), (150, 172), 8193, (1, 65535), 300),
    ((17, 80, 104), 17, (0, 0, 0), (40, 52), 76, (1, 76), 70),
    ((17, 80, 104), 17, (0, 1, 1), (40, 52), 2304, (1, 2304), 70),
    ((2, 700, 100), 2, (0, 0, 0), (350, 3), 1, (5, 60000), 400),
])
def test_axis_forms_match_oracle(gshape, nzb, offset, center, voxel_bins, vrange, n_r):
    voxels = _voxels((nzb, gshape[1], gshape[2]), sum(gshape), 3000 if vrange[1] < 3000 else 45000)
    want = oracle.axis_histograms(voxels, offset, gshape, voxel_bins, n_r, center, vrange)
    got = [np.full((n, voxel_bins), 3, np.uint64) for n in (gshape[2], gshape[1], gshape[0], n_r)]
    axis_histograms(voxels, offset, *got, center, vrange, 0)
    for g, w, name in zip(got, want, ("x", "y", "z", "r")):
        np.testing.assert_array_equal(g, w + np.uint64(3), err_msg=name)


# field_histogram above the size from which its keys are partitioned: the pipeline's bins (158
# partitions, the last with fewer field bins); odd rows and offsets; one partition; the most
# partitions (one field bin each) and one more, which the direct form counts; ranges that need
# thresholds; rows of one voxel, more of them than one batch holds; all voxels in one cell, which
# many blocks then share; nothing to count.
@pytest.mark.parametrize("vshape,fshape,offset,bins_shape,vrange,frange,constant", [
    ((49, 360, 360), (25, 180, 180), (0, 0, 0), (2048, 4096), (1, 32000), (1, 65535), None),
    ((65, 257, 257), (65, 257, 257), (0, 5, 13), (37, 1000), (1, 40000), (1, 65535), None),
    ((2, 2100, 1000), (1, 700, 333), (0, 0, 8), (1, 1), (100, 60000), (1, 65535), None),
    ((7, 1030, 900), (7, 103, 90), (1, 1029, 1), (256, 53248), (1, 65535), (1, 65535), None),
    ((7, 1030, 900), (7, 103, 90), (0, 0, 0), (257, 53248), (1, 65535), (1, 65535), None),
    ((11, 640, 640), (6, 320, 320), (0, 3, 2), (2304, 76), (1, 76), (1, 2304), None),
    ((34, 1000003, 1), (9, 500002, 1), (0, 2, 0), (300, 512), (1, 32000), (1, 65535), None),
    ((56, 333, 344), (28, 167, 172), (0, 0, 0), (2048, 4096), (1, 32000), (1, 65535), 31000),
    ((56, 333, 344), (28, 167, 172), (0, 0, 0), (2048, 4096), (1, 32000), (1, 65535), 0),
])
def test_partitioned_field_histogram_matches_oracle(vshape, fshape, offset, bins_shape, vrange, frange, constant):
    if constant is None:
        voxels = _voxels(vshape, sum(vshape), 100 if vrange[1] < 100 else 45000)
        field = _voxels(fshape, sum(fshape), 3000 if frange[1] < 3000 else 65536)
    else:
        voxels, field = np.full(vshape, constant, np.uint16), np.full(fshape, 65535, np.uint16)
    want = oracle.field_histogram(voxels, field, offset, bins_shape, vrange, frange)
    got = np.full(bins_shape, 3, np.uint64)
    field_histogram(voxels, field, offset, got, vrange, frange, 0)
    np.testing.assert_array_equal(got, want + np.uint64(3))
