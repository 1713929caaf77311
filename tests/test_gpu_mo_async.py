"""FP64 MO builds of several tensors from one RI handle, unfinished at the same time on streams of their own (the builds only read the
handle), beside a Fock build's exchange on a third stream: bit for bit the tensors that single builds give."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import _lib as L  # noqa: E402
from rerdmft_b200 import mo, ri, synth  # noqa: E402


@pytest.mark.parametrize("n,naux", [(160, 480), (131, 500)])
def test_builds_side_by_side(n, naux):
    rng = np.random.default_rng(n)
    store = ri.RiStore(synth.ri_tensor(n, naux, n, box=8.0), nl=n)
    Cs = [torch.as_tensor(np.linalg.qr(rng.standard_normal((n, n)))[0].copy(), device="cuda") for _ in range(3)]
    occ = Cs[2][:, :60].contiguous()
    alone = [mo.buildRiNonRelSpinMoEri(store, n, C) for C in Cs[:2]]
    want = [e.b().copy() for e in alone]
    Jw, Kw = (t.cpu().numpy() for t in ri.jk_occupied(store, occ))
    streams = [torch.cuda.Stream() for _ in range(3)]
    J, K = torch.empty((n, n), dtype=torch.float64, device="cuda"), torch.empty((n, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lib = L.lib()
    for _ in range(5):
        for e, C, st in zip(alone, reversed(Cs[:2]), streams):  # the other orbitals first: the results below are new ones
            L.check(lib.rr_mo_build_nonrel_into(store.handle, C.data_ptr(), e.handle,
                                                ctypes.byref(L.opts(L.RR_MEM_DEVICE, stream=st.cuda_stream, sync=0))))
        for e, C, st in zip(alone, Cs, streams):
            L.check(lib.rr_mo_build_nonrel_into(store.handle, C.data_ptr(), e.handle,
                                                ctypes.byref(L.opts(L.RR_MEM_DEVICE, stream=st.cuda_stream, sync=0))))
        L.check(lib.rr_ri_jk_occupied(store.handle, occ.data_ptr(), occ.shape[1], J.data_ptr(), K.data_ptr(),
                                      ctypes.byref(L.opts(L.RR_MEM_DEVICE, stream=streams[2].cuda_stream, sync=0))))
        torch.cuda.synchronize()
        assert all(np.array_equal(e.b(), w) for e, w in zip(alone, want))
        assert np.array_equal(J.cpu().numpy(), Jw) and np.array_equal(K.cpu().numpy(), Kw)
