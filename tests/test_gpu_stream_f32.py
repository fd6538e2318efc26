"""The FP32 passes against the generic pass, bit for bit (run with -m gpu).

Both sum every output over the taps in increasing order with one FMA each.  The generic
pass runs for radii above 128: the same kernel padded with zero taps to radius 130 goes
there, and a zero tap leaves the sum as it is (an FMA of 0 and a finite value), so the
results have to be equal in every bit.
"""
import ctypes

import numpy as np
import pytest
import torch

from maxibone_b200 import _lib, device

pytestmark = pytest.mark.gpu


def _kernel(radius, seed):
    k = np.random.default_rng(seed).uniform(0.1, 1.0, 2 * radius + 1)  # no symmetry: a reversed or shifted tap shows
    return (k / k.sum()).astype(np.float32)


def _run(mask, shape, kernel, reps, offset=0):
    n = int(np.prod(shape))
    out = torch.zeros(n + offset, dtype=torch.uint16, device="cuda")[offset:]
    field = torch.zeros(n + offset, dtype=torch.float32, device="cuda")[offset:]
    device.diffuse(mask, kernel, reps, output=out, field_out=field, shape=shape)
    return out.view(torch.int16), field


def _mask(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand(shape, generator=g, device="cuda") < 0.1).to(torch.uint8)


# Axes and rows around the 64-wide column tile, the 64- and 128-long chunks and the 16-place
# period of the window; taps around that period; axes shorter than the radius; rings that
# wrap (axes of several chunks in one segment); rows without any alignment.
SHAPES = [(1, 1, 1), (1, 1, 129), (63, 2, 64), (64, 65, 127), (65, 64, 128), (3, 130, 257), (200, 3, 66),
          (17, 70, 333), (300, 129, 36), (2, 1100, 65), (5, 7, 1027)]


@pytest.mark.parametrize("radius", [0, 1, 7, 8, 15, 16, 32, 33, 97, 128])
@pytest.mark.parametrize("shape", SHAPES)
def test_stream_passes_equal_the_generic_pass(shape, radius):
    kernel = _kernel(radius, radius)
    wide = np.pad(kernel, 130 - radius)
    mask = _mask(shape, sum(shape))
    got_u16, got = _run(mask, shape, kernel, 2)
    want_u16, want = _run(mask, shape, wide, 2)
    assert torch.equal(got, want)
    assert torch.equal(got_u16, want_u16)


# Volumes on both sides of the x pass's choice between its two forms: 2^24 voxels, rows of a
# multiple of 4, the radii with unrolled taps, outputs that allow vector access.
@pytest.mark.parametrize("shape,radius,offset", [((64, 512, 512), 16, 0), ((64, 512, 512), 16, 1),
                                                 ((64, 512, 516), 32, 0), ((64, 512, 516), 31, 0),
                                                 ((65, 517, 515), 4, 0), ((63, 512, 512), 24, 0)])
def test_x_pass_forms_equal_the_generic_pass(shape, radius, offset):
    kernel = _kernel(radius, 3)
    mask = _mask(shape, 5)
    packed = device.bitpack(mask)
    want_u16, want = _run(mask, shape, np.pad(kernel, 130 - radius), 2)
    for m in (mask, packed):
        got_u16, got = _run(m, shape, kernel, 2, offset)
        assert torch.equal(got, want)
        assert torch.equal(got_u16, want_u16)


# The allocation-free call hands a uint8 mask to the passes as it is.
@pytest.mark.parametrize("shape,radius,shift", [((20, 33, 70), 5, 0), ((33, 40, 128), 12, 0), ((33, 40, 128), 12, 3)])
def test_uint8_mask_in_the_passes(shape, radius, shift):
    kernel = _kernel(radius, 7)
    n = int(np.prod(shape))
    buf = torch.zeros(n + shift, dtype=torch.uint8, device="cuda")
    mask = buf[shift:].view(shape)
    mask.copy_(_mask(shape, 9) * 7)
    want_u16, want = _run(mask, shape, np.pad(kernel, 130 - radius), 3)
    out = torch.zeros(n, dtype=torch.uint16, device="cuda")
    field = torch.zeros(n, dtype=torch.float32, device="cuda")
    _lib.check(_lib.lib().maxi_diffusion_device_noalloc(
        mask.data_ptr(), 0, *shape, kernel.ctypes.data_as(ctypes.c_void_p), kernel.shape[0], 3, out.data_ptr(),
        field.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(field, want)
    assert torch.equal(out.view(torch.int16), want_u16)
