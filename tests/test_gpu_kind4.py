"""Kind 4 on both of its kernels (direct sums for little work, block-Toeplitz GEMMs beyond) at sizes around the line
between them, against the float32 CUDA-core family, as in test_gpu_ragged.py."""
import pytest
import torch

from tests.test_gpu_parity import TOL_BF16
from tests.test_gpu_ragged import run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,D,B", [(1, 8, 1), (8, 8, 3), (9, 16, 70), (64, 768, 5), (96, 8, 300), (127, 768, 1), (128, 768, 2), (128, 768, 7), (128, 768, 12),
                                   (100, 512, 30), (129, 8, 1), (200, 1536, 1), (255, 24, 6), (256, 768, 4), (300, 400, 9), (383, 16, 4),
                                   (505, 8, 2), (512, 8, 5), (512, 256, 9), (250, 700, 6), (512, 700, 3), (512, 640, 16)])
@pytest.mark.parametrize("residual,u_dtype", [(True, torch.float16), (True, torch.bfloat16), (False, torch.bfloat16)])
def test_kind4(L, D, B, residual, u_dtype):
    e = run_both(4, L, D, B, residual, u_dtype, 93)
    assert e < TOL_BF16, e
