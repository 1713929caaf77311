"""When the digit planes of a store exist: from the first product that reads them on, and until an allocation of the library fails for
want of memory.  Results do not depend on it.  The tensors are larger than all that the library keeps of released blocks."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import mo, ri  # noqa: E402


def free():
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def tensor(n, naux, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    B = torch.randn((naux, n, n), dtype=torch.float64, device="cuda", generator=g)
    return (B + B.transpose(1, 2)).reshape(naux, n * n).contiguous()


def warm_up():
    """Kernels and library handles take device memory of their own on their first use."""
    store = ri.RiStore(tensor(160, 400, 9), nl=160)
    ri.jk_occupied(store, torch.eye(160, dtype=torch.float64, device="cuda")[:, :32].contiguous())
    store.close()


def test_planes_are_made_by_the_first_product_and_given_back():
    n, naux, nocc = 320, 4000, 24
    size = 8 * naux * n * n  # 3.3 GB
    warm_up()
    B = tensor(n, naux, 1)
    C = torch.linalg.qr(B[0].reshape(n, n))[0][:, :nocc].contiguous()
    store = ri.RiStore(B, nl=n)
    f1 = free()
    first = [t.clone() for t in ri.jk_occupied(store, C)]
    assert f1 - free() > size  # the planes, and a tenth of that in scratch
    again = ri.jk_occupied(store, C)
    assert all(torch.equal(a, b) for a, b in zip(first, again))
    moB = mo.buildRiNonRelSpinMoEri(store, n, C.new_zeros((n, n)).fill_diagonal_(1.0)).b()
    gc.collect()
    fill = torch.empty(free() - (1 << 30), dtype=torch.uint8, device="cuda")
    other = ri.RiStore(B, nl=n)  # 3.3 GB where 1 GB is free: the planes of the idle store make room
    assert torch.cuda.mem_get_info()[0] >= 0
    del fill
    torch.cuda.empty_cache()
    assert all(torch.equal(a, b) for a, b in zip(first, ri.jk_occupied(store, C)))
    assert torch.equal(first[1], ri.jk_occupied(other, C)[1])  # (J of a store without packed triangles adds in another order)
    assert np.array_equal(moB, mo.buildRiNonRelSpinMoEri(store, n, C.new_zeros((n, n)).fill_diagonal_(1.0)).b())
    store.close()
    other.close()


def test_a_captured_exchange_keeps_its_planes():
    """A captured build is replayed after the library ran out of memory once: its graph reads the planes it was captured with."""
    import ctypes

    from rerdmft_b200 import _lib as L

    n, naux, nocc = 256, 6000, 24
    B = tensor(n, naux, 2)
    C = torch.linalg.qr(B[0].reshape(n, n))[0][:, :nocc].contiguous()
    store = ri.RiStore(B, nl=n)
    J, K = torch.zeros((n, n), dtype=torch.float64, device="cuda"), torch.zeros((n, n), dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    opts = L.opts(L.RR_MEM_DEVICE, stream=st.cuda_stream, sync=0)

    def call():
        L.check(L.lib().rr_ri_jk_occupied(store.handle, C.data_ptr(), nocc, J.data_ptr(), K.data_ptr(), ctypes.byref(opts)))

    call()
    torch.cuda.synchronize()
    want = [J.clone(), K.clone()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st, capture_error_mode="thread_local"):
        call()
    J.zero_()
    K.zero_()
    fill = torch.empty(free() - (1 << 29), dtype=torch.uint8, device="cuda")
    with pytest.raises(Exception):
        ri.RiStore(B, nl=n)  # 3.1 GB where 0.5 GB is free and the planes are taken
    del fill
    torch.cuda.empty_cache()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(J, want[0]) and torch.equal(K, want[1])
    del graph
    store.close()
