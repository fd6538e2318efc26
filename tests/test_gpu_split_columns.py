"""The tensor-core z and y passes with both coefficient halves (split_coefficients) on either side of
radius 64, above which their tiles have 64 columns (run with -m gpu): within the bounds of the
CUDA-core form and of FP64."""
import numpy as np
import pytest
import torch

from maxibone_b200 import _lib, device, gauss_kernel
from maxibone_b200.synthetic import random_mask
from test_gpu_tensor_cores import TC_VS_CC, VS_F64, run

pytestmark = pytest.mark.gpu


# The column lengths of test_gpu_column_blocks; the x extents end in a whole 64-column tile, 8 columns
# past one, and 8 past two of them.
@pytest.mark.parametrize("radius", [64, 65, 128])
@pytest.mark.parametrize("shape", [(128, 129, 72), (385, 20, 64), (24, 513, 136), (97, 241, 264), (1, 64, 1032)])
def test_split_column_blocks(shape, radius):
    mask = random_mask(shape, 0.02, seed=sum(shape) + radius)
    kernel = gauss_kernel(radius / 4.0).astype(np.float32)
    assert kernel.shape[0] == 2 * radius + 1
    _, want = run(mask, kernel, 2, "f64")
    m = torch.from_numpy(mask).cuda()
    for field in ("f16", "bf16"):
        got = torch.empty(shape, dtype=torch.float32, device="cuda")
        u16 = torch.empty(shape, dtype=torch.uint16, device="cuda")
        device.diffuse(m, kernel, 2, output=u16, field=field, field_out=got, split_coefficients=True)
        path = device.last_path()
        tensor = _lib.PATH_TENSOR_CORES_ZY | _lib.PATH_TENSOR_CORES_X
        assert path & tensor == tensor and not path & _lib.PATH_CUDA_CORES, hex(path)
        torch.cuda.synchronize()
        device.tensor_core_status()
        _, cc = run(mask, kernel, 2, field, False, True)
        got = got.cpu().numpy()
        assert np.abs(got - cc).max() <= TC_VS_CC[field]
        assert np.abs(got.astype(np.float64) - want).max() <= VS_F64[field]
        assert np.all(got[mask > 0] == 1.0)
        assert np.all(u16.cpu().numpy()[mask > 0] == 65535)
