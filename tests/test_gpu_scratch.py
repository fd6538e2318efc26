"""The memory that the field steps keep between calls (run with -m gpu): calls of two threads do
not wait for each other, and what is kept is bounded and given back."""
import ctypes
import threading
import time

import numpy as np
import pytest
import torch

from maxibone_b200 import _lib, diffusion, gauss_kernel
from maxibone_b200.fields import combine_fields
from maxibone_b200.histograms import axis_histograms, field_histogram

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _u16(shape, seed, hi=60000):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(1, hi, shape, generator=g, device="cuda", dtype=torch.int32).to(torch.int16)


def _histogram(nz):
    voxels, field = _u16((nz, 1024, 1024), 1, 32000), _u16((nz // 2, 512, 512), 2)
    bins = torch.zeros((256, 512), dtype=torch.int64, device="cuda")

    def call():
        bins.zero_()
        field_histogram(voxels, field, (0, 0, 0), bins, (1.0, 32000.0), (1.0, 65535.0))
        return bins
    return call


def _combination():
    gauss, edt = _u16((8, 64, 64), 3), _u16((8, 64, 64), 4)
    output = torch.empty_like(gauss)
    return lambda: combine_fields(gauss, edt, output)


def _release():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert _lib.lib().maxi_release_cached_memory() == 0
    return torch.cuda.mem_get_info()[0]


# One thread's call queues up behind half a second of other work on its stream; another thread's
# call on another stream, begun later, ends first.
@pytest.mark.parametrize("first,second", [(_combination, _combination), (_combination, lambda: _histogram(8)),
                                          (lambda: _histogram(8), _combination)],
                         ids=["combine-combine", "combine-histogram", "histogram-combine"])
def test_calls_of_two_threads_do_not_wait_for_each_other(first, second):
    calls = {"late": first(), "early": second()}
    for call in calls.values():
        call()
    streams = {name: torch.cuda.Stream() for name in calls}
    torch.cuda.synchronize()
    ended, begun = [], threading.Event()

    def run(name):
        with torch.cuda.stream(streams[name]):
            if name == "late":
                torch.cuda._sleep(1_000_000_000)
                begun.set()
            calls[name]()
        ended.append(name)

    late, early = (threading.Thread(target=run, args=(name,)) for name in ("late", "early"))
    late.start()
    begun.wait()
    time.sleep(0.05)
    early.start()
    late.join()
    early.join()
    assert ended == ["early", "late"]


def test_kept_memory_is_bounded_and_given_back():
    call = _histogram(256)  # 512 MB of keys
    call()
    before = _release()
    call()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= 640 * MB
    assert _release() >= before - 32 * MB


def test_histogram_without_room_for_its_keys():
    call = _histogram(128)  # 256 MB of keys
    want = call().clone()
    free = _release()
    filler = torch.empty(free - 160 * MB, dtype=torch.uint8, device="cuda")
    try:
        assert torch.equal(call(), want)
    finally:
        del filler
        _release()


# A volume that fits once the histogram's keys are given back runs in device memory.
def test_in_memory_diffusion_takes_the_kept_memory_back(capfd):
    shape = (128, 512, 512)  # 11.125 bytes a voxel: 356 MiB
    mask = np.zeros(shape, np.uint8)
    mask[::7, ::5, ::3] = 1
    out = np.empty(shape, np.uint16)
    kernel = gauss_kernel(1.0).astype(np.float32)
    call = _histogram(256)
    _release()
    call()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - 160 * MB, dtype=torch.uint8, device="cuda")
    try:
        _lib.check(_lib.lib().maxi_diffusion_in_memory(
            mask.ctypes.data, *shape, kernel.ctypes.data, len(kernel), 1, out.ctypes.data, 1))
        ctypes.CDLL(None).fflush(None)
        said = capfd.readouterr().out
        assert "complete" in said and "out-of-core" not in said
    finally:
        del filler
        _release()
    want = np.empty(shape, np.uint16)
    diffusion(mask, kernel, want, 1)
    np.testing.assert_array_equal(out, want)


# These calls wait for their stream, so one on a stream that is being captured is refused.  It leaves no
# memory of the capture's behind for the next call to use.
@pytest.mark.parametrize("make", [_combination, lambda: _histogram(8), lambda: _axis()],
                         ids=["combine", "histogram", "axis"])
def test_refused_under_capture(make):
    call = make()
    want = [t.clone() for t in _tensors(call())]
    _release()  # the refused call finds no kept buffer
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        try:
            with pytest.raises(_lib.MaxiError):
                call()
        finally:
            graph.capture_end()
    del graph
    torch.cuda.synchronize()
    for _ in range(2):
        for got, expected in zip(_tensors(call()), want):
            assert torch.equal(got, expected)


def _tensors(result):
    return result if isinstance(result, list) else [result]


def _axis():
    voxels = _u16((16, 128, 128), 5, 32000)
    bins = [torch.zeros((n, 512), dtype=torch.int64, device="cuda") for n in (128, 128, 16, 92)]

    def call():
        for b in bins:
            b.zero_()
        axis_histograms(voxels, (0, 0, 0), *bins, (64, 64), (1.0, 32000.0))
        return bins
    return call
