"""Flat complex FP64 products beyond 1024, whose K is split 8 ways (csrc/gemm_f64.cu), at the edges of that rule and of its ranges; tolerance
as in test_gpu_kernels.py."""
import numpy as np
import pytest

from test_gpu_kernels import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1025, 1030), (32, 1600, 257), (33, 1025, 100), (7, 2048, 512), (1601, 31, 700), (8, 2049, 300), (5, 1030, 3)])
@pytest.mark.parametrize("opA,opB,conjA,conjB", [(0, 0, 0, 0), (1, 0, 1, 0), (0, 1, 0, 1)])
def test_flat_complex(opA, opB, conjA, conjB, shape):
    M, N, K = shape
    out, ref = _run(M, N, K, opA, opB, cplx=True, conjA=bool(conjA), conjB=bool(conjB), beta=0.5)
    assert np.abs(out - ref).max() <= 1e-12 * max(1.0, np.abs(ref).max()) * np.sqrt(K)
