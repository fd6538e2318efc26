"""Calls of several host threads on streams of their own (run with -m gpu): each gives what it
gives alone, whatever size the other threads' calls have."""
import threading

import numpy as np
import pytest
import torch

from maxibone_b200 import device, morphology
from maxibone_b200.histograms import axis_histograms

pytestmark = pytest.mark.gpu

CALLS = 150


def _mask(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand(shape, generator=g, device="cuda") < 0.1).to(torch.uint8)


def _diffusion(radius, field):
    shape = (24, 72, 64)
    mask = _mask(shape, radius)
    kernel = np.full(2 * radius + 1, 1.0 / (2 * radius + 1), np.float32)
    workspace = torch.empty(device.workspace_bytes(shape, "f32"), dtype=torch.uint8, device="cuda")
    out = torch.empty(shape, dtype=torch.uint16, device="cuda")
    return lambda: device.diffuse(mask, kernel, 6, output=out, field=field, workspace=workspace), [out.view(torch.int16)]


def _morphology(radius):
    mask = _mask((20, 40, 128), radius)
    out = torch.empty_like(mask)
    return lambda: morphology.dilate_3d_sphere(mask, radius, out), [out]


def _axis(voxel_bins):
    g = torch.Generator(device="cuda").manual_seed(voxel_bins)
    shape = (16, 96, 128)
    voxels = (torch.rand(shape, generator=g, device="cuda") * 30000).to(torch.int16)
    bins = [torch.zeros((n, voxel_bins), dtype=torch.int64, device="cuda") for n in (128, 96, 16, 81)]

    def call():
        for b in bins:
            b.zero_()
        axis_histograms(voxels, (0, 0, 0), *bins, (48, 64), (1.0, 32000.0))
    return call, bins


# Pairs of calls that share a kernel but not the size of its shared memory.
@pytest.mark.parametrize("make,sizes", [
    (lambda r: _diffusion(r, "f32"), (5, 100, 128)), (lambda r: _diffusion(r, "bf16"), (16, 32, 65, 128)),
    (_morphology, (13, 16)), (_morphology, (29, 32)), (_axis, (64, 512, 4096)),
], ids=["f32", "bf16", "morphology16", "morphology32", "axis"])
def test_threads_with_different_sizes(make, sizes):
    work = []
    for size in sizes:
        call, outs = make(size)
        call()
        torch.cuda.synchronize()
        work.append((call, outs, [o.clone() for o in outs], torch.cuda.Stream()))
    torch.cuda.synchronize()
    errors = []

    def run(call, stream):
        try:
            with torch.cuda.stream(stream):
                for _ in range(CALLS):
                    call()
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(call, stream)) for call, _, _, stream in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for _, outs, want, _ in work:
        for o, w in zip(outs, want):
            assert torch.equal(o, w)
