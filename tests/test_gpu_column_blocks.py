"""The tensor-core z and y passes where their columns' blocks of 128 rows begin and end (run
with -m gpu), within the bounds of the CUDA-core form and of FP64."""
import numpy as np
import pytest

from maxibone_b200 import gauss_kernel
from maxibone_b200.synthetic import random_mask
from test_gpu_tensor_cores import TC_VS_CC, VS_F64, run

pytestmark = pytest.mark.gpu


# Columns of one to five tiles, ending on a block's edge, one row past it and where the last
# block lies past the volume's end; more columns than CTAs, so that the ring runs on from one
# column to the next; two and three blocks a tile (radius up to 64 and above).
@pytest.mark.parametrize("radius", [16, 64, 65, 128])
@pytest.mark.parametrize("shape", [(128, 129, 72), (385, 20, 64), (24, 513, 136), (97, 241, 264), (1, 64, 1032)])
def test_column_blocks(shape, radius):
    mask = random_mask(shape, 0.02, seed=sum(shape) + radius)
    kernel = gauss_kernel(radius / 4.0).astype(np.float32)
    _, want = run(mask, kernel, 2, "f64")
    for field in ("f16", "bf16"):
        u16, got = run(mask, kernel, 2, field, True, True)
        _, cc = run(mask, kernel, 2, field, False, True)
        assert np.abs(got - cc).max() <= TC_VS_CC[field]
        assert np.abs(got.astype(np.float64) - want).max() <= VS_F64[field]
        assert np.all(u16[mask > 0] == 65535)
