"""The FP32 x pass's tile form with padded taps, and the radii beside its range (run with -m gpu):
equal to the generic pass bit for bit."""
import numpy as np
import pytest

from test_gpu_stream_f32 import _kernel, _mask, _run
import torch

pytestmark = pytest.mark.gpu


# 2^24 voxels and more, aligned rows: one to three taps of padding a side, none, and one too many.
@pytest.mark.parametrize("radius", [0, 1, 3, 5, 7, 9, 13, 17, 20, 21, 23, 28, 29, 31, 33])
def test_padded_taps_equal_the_generic_pass(radius):
    shape = (64, 513, 516)
    mask = _mask(shape, radius)
    kernel = _kernel(radius, radius)
    got_u16, got = _run(mask, shape, kernel, 2)
    want_u16, want = _run(mask, shape, np.pad(kernel, 130 - radius), 2)
    assert torch.equal(got, want)
    assert torch.equal(got_u16, want_u16)


# Row lengths on both sides of the choice by how far they fill their last tile, with a remainder.
@pytest.mark.parametrize("nx,radius", [(1004, r) for r in (1, 3, 5, 7, 8, 9, 13, 17, 21, 24, 29, 32)] +
                         [(nx, r) for nx in (124, 132, 256, 380, 388, 640, 892, 900, 1100, 2180) for r in (8, 12, 31)])
def test_row_lengths_equal_the_generic_pass(nx, radius):
    shape = (3, -(-(1 << 24) // (3 * nx)), nx)
    mask = _mask(shape, radius)
    kernel = _kernel(radius, radius)
    got_u16, got = _run(mask, shape, kernel, 2)
    want_u16, want = _run(mask, shape, np.pad(kernel, 130 - radius), 2)
    assert torch.equal(got, want)
    assert torch.equal(got_u16, want_u16)
