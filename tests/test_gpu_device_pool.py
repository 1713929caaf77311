"""Released device blocks are kept for the next object (csrc/ri_core.cu): results on recycled memory, on several
threads at once, and the bound on what is kept."""
import gc
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import mo  # noqa: E402

SIZES = [(24, 96), (40, 160), (41, 163), (64, 256)]


def rotate(n, naux, seed):
    rng = np.random.default_rng(seed)
    B = rng.standard_normal((naux, n, n))
    B = 0.5 * (B + B.transpose(0, 2, 1))
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    U = np.zeros((2 * n, 2 * n))
    U[:n, :n] = U[n:, n:] = q
    got = mo.RiNonRelSpinMoEri.from_tensor(B.reshape(naux, n * n), n).rotated(U).b()
    ref = (q.T @ B @ q).reshape(naux, n * n)
    # two products of n terms, each element and its reference rounded: 4 (n + 2) 2^-53 of |q|^T |B| |q|
    return np.all(np.abs(got - ref) <= 4 * (n + 2) * 2.0 ** -53 * (np.abs(q.T) @ np.abs(B) @ np.abs(q)).reshape(naux, n * n))


def test_results_on_recycled_blocks_and_threads():
    keep = mo.RiNonRelSpinMoEri.from_tensor(np.zeros((8, 64)), 8)  # blocks stay with the library while an object lives
    assert all(rotate(*SIZES[k % 4], k) for k in range(12))
    with ThreadPoolExecutor(4) as ex:
        assert all(ex.map(lambda k: rotate(*SIZES[(k // 3) % 4], k), range(48)))
    assert keep.b().shape == (8, 64) and not keep.b().any()


def test_what_is_kept_is_bounded():
    keep = mo.RiNonRelSpinMoEri.from_tensor(np.zeros((8, 64)), 8)
    gc.collect()
    free0, total = torch.cuda.mem_get_info()
    for k in range(8):  # blocks of 0.6 to 1.2 GB, no two alike
        n = 256 + 8 * k
        zero = torch.zeros(1200 + 50 * k, n * n, device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        e = mo.RiNonRelSpinMoEri.from_tensor(zero, n)
        del e, zero
        torch.cuda.empty_cache()
    gc.collect()
    assert torch.cuda.mem_get_info()[0] >= free0 - total // 64 - (64 << 20)
    del keep
