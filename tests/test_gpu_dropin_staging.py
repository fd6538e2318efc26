"""The drop-in call's staged copies at the edges of their chunks (run with -m gpu): pageable
arrays in and out give what the device call gives on the same mask."""
import threading

import numpy as np
import pytest
import torch

from maxibone_b200 import _lib, device, diffusion, gauss_kernel

pytestmark = pytest.mark.gpu


def _case(shape, seed):
    mask = (np.random.default_rng(seed).random(shape) < 0.1).astype(np.uint8)
    kernel = gauss_kernel(1.0).astype(np.float32)
    out = torch.empty(shape, dtype=torch.uint16, device="cuda")
    device.diffuse(torch.from_numpy(mask).cuda(), kernel, 1, output=out)
    return mask, kernel, out.view(torch.int16).cpu().numpy().view(np.uint16)


# Bytes in and out around the smallest staged copy (4 MiB), whole and partial 1 MiB chunks,
# fewer chunks than host threads and a number that is no multiple of them.
@pytest.mark.parametrize("shape", [(64, 256, 128), (64, 256, 256), (1, 1, (4 << 20) - 1), (1, 1, (4 << 20) + 1),
                                   (19, 701, 400), (40, 512, 640)])
def test_staged_copies_at_chunk_edges(shape):
    mask, kernel, want = _case(shape, sum(shape))
    for _ in range(2):  # the second call reuses the staging buffers
        got = np.full(shape, 7, np.uint16)
        diffusion(mask, kernel, got, 1)
        np.testing.assert_array_equal(got, want)
    assert _lib.lib().maxi_release_cached_memory() == 0
    got = np.empty(shape, np.uint16)
    diffusion(mask, kernel, got, 1)
    np.testing.assert_array_equal(got, want)


def test_concurrent_calls_share_the_staging_buffers():
    cases = [_case((20, 500, 600), s) for s in (1, 2, 3)]
    got = [[np.empty(c[0].shape, np.uint16) for _ in range(3)] for c in cases]

    def run(i):
        for g in got[i]:
            diffusion(cases[i][0], cases[i][1], g, 1)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c, gs in zip(cases, got):
        for g in gs:
            np.testing.assert_array_equal(g, c[2])
