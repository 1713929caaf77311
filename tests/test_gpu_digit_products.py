"""The FP64 exchange and MO transforms on the INT8 tensor cores (csrc/oz.cu, oz_exchange.cu) against extended
precision, at the edges of their tiles, K blocks and padded column groups, with resident digit planes and with
planes made range by range.

Tolerance.  K_ab = sum_k T_ak T_bk: either factor carries the rounding of T to FP64 (2^-53 of its value), the digit
cut and the dropped pairs are below that (2^-64 of the row bound, at most 2^6 above the row's largest value here), the
INT64 sums are exact, and up to 56 partial sums are added in FP64, so the error is below 2^-50 of
sqrt(K_aa K_bb) (Cauchy-Schwarz); doubled twice for the complex parts: 2^-48.  An MO element has the same two
roundings against |C|^T |B| |C|."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import _lib as L  # noqa: E402
from rerdmft_b200 import mo, ri, synth  # noqa: E402

REL = 2.0 ** -48
X = np.longdouble


def drop_planes(store):
    had = ctypes.c_int32()
    L.check(L.lib().rr_test_drop_digit_planes(store.handle, ctypes.byref(had)))
    return had.value


def exchange(B, cf, cu):
    """sum_P (B^P cf)(B^P cu)^dagger for the two half-transforms' operands in extended precision."""
    def half(c):
        re = np.tensordot(B.astype(X), c.real.astype(X), (1, 0))  # (P, a, i): contracts the first AO index
        im = np.tensordot(B.astype(X), c.imag.astype(X), (1, 0))
        return re.transpose(1, 0, 2).reshape(B.shape[1], -1), im.transpose(1, 0, 2).reshape(B.shape[1], -1)
    fr, fi = half(cf)
    ur, ui = half(cu)
    return fr @ ur.T + fi @ ui.T, fi @ ur.T - fr @ ui.T


# naux n^2 nocc >= 2e8: the digit path; n around the 64- and 128-wide tiles, nocc around the groups of 8, 16 and 64
# columns, naux nocc8 off the 32-byte K blocks
NONREL = [(127, 401, 31), (129, 371, 33), (128, 200, 64), (161, 131, 65), (193, 67, 81)]


@pytest.mark.parametrize("planes", ["resident", "ranges"])
@pytest.mark.parametrize("n,naux,nocc", NONREL)
def test_nonrel_exchange(n, naux, nocc, planes):
    rng = np.random.default_rng(n)
    B = synth.ri_tensor(n, naux, n, box=8.0)
    C = np.linalg.qr(rng.standard_normal((n, nocc)))[0]
    store = ri.RiStore(B, nl=n)
    if planes == "ranges":
        assert drop_planes(store) == 1
    _, K = ri.jk_occupied(store, C)
    ref, _ = exchange(B.reshape(naux, n, n), C, C)
    d = np.sqrt(np.diag(ref)).astype(float)
    assert np.all(np.abs(K - ref.astype(float)) <= REL * np.outer(d, d))
    assert np.array_equal(K, K.T)


def test_nonrel_exchange_of_a_general_tensor():
    """B^P not symmetric, columns of very different size and a zero one, large and small coefficients."""
    n, naux, nocc = 133, 359, 33
    rng = np.random.default_rng(5)
    B = rng.standard_normal((naux, n, n)) * np.exp(rng.uniform(-60, 60, n))[None, None, :]
    B[:, :, 7] = 0.0
    C = rng.standard_normal((n, nocc)) * np.exp(rng.uniform(-30, 30, nocc))[None, :]
    _, K = ri.jk_occupied(ri.RiStore(B.reshape(naux, -1), nl=n), C)
    ref, _ = exchange(B, C, C)
    d = np.sqrt(np.diag(ref)).astype(float)
    assert np.all(np.abs(K - ref.astype(float)) <= REL * np.outer(d, d))
    assert np.all(K[7] == 0.0)


def test_non_finite_values_come_through():
    n, naux, nocc = 128, 200, 64
    rng = np.random.default_rng(6)
    B = synth.ri_tensor(n, naux, 9, box=8.0)
    C = np.linalg.qr(rng.standard_normal((n, nocc)))[0]
    store = ri.RiStore(B, nl=n)
    Cb = C.copy()
    Cb[3, 5] = np.nan
    _, K = ri.jk_occupied(store, Cb)
    assert np.isnan(K).all()
    _, K = ri.jk_occupied(store, C)  # and the handle is fine afterwards
    assert np.isfinite(K).all()
    Bb = B.copy()
    Bb[4, 17] = np.inf
    _, K = ri.jk_occupied(ri.RiStore(Bb, nl=n), C)
    assert not np.isfinite(K[17]).any()


@pytest.mark.parametrize("planes", ["resident", "ranges"])
@pytest.mark.parametrize("nl,ns,naux,r", [(8, 17, 9, 1), (33, 65, 40, 5), (64, 129, 31, 8), (70, 96, 50, 17)])
def test_four_component_two_electron(nl, ns, naux, r, planes):
    rng = np.random.default_rng(nl)
    BL, BS = synth.ri_tensor(nl, naux, nl, box=5.0), 0.2 * synth.ri_tensor(ns, naux, ns, box=5.0)
    nu = 2 * nl + 2 * ns
    C = np.linalg.qr(rng.standard_normal((nu, r)) + 1j * rng.standard_normal((nu, r)))[0]
    src = ri.RiDirectEriSource(nl, ns, BL, BS)
    if planes == "ranges":
        assert drop_planes(src.store) == 1
    G = ri.riFockTwoElectronDirect(src, np.zeros((nu, nu), dtype=complex), C, np.ones(r))
    off = [0, nl, 2 * nl, 2 * nl + ns, nu]
    T = [BL.reshape(naux, nl, nl)] * 2 + [BS.reshape(naux, ns, ns)] * 2
    K = np.zeros((nu, nu), dtype=np.clongdouble)
    for f in range(4):
        for u in range(4):
            cf, cu = C[off[f]:off[f + 1]], C[off[u]:off[u + 1]]
            half = [np.tensordot(t.astype(X), c.astype(np.clongdouble), (1, 0)).transpose(1, 0, 2).reshape(t.shape[1], -1)
                    for t, c in ((T[f], cf), (T[u], cu))]
            K[off[f]:off[f + 1], off[u]:off[u + 1]] = half[0] @ half[1].conj().T
    d = np.sqrt(np.diag(K).real).astype(float)
    assert np.all(np.abs(G + K.astype(complex)) <= REL * np.outer(d, d))


@pytest.mark.parametrize("planes", ["resident", "ranges"])
@pytest.mark.parametrize("n,naux", [(120, 117), (127, 98), (129, 95), (136, 90)])
def test_mo_transform(n, naux, planes):
    """n a multiple of four takes the stores of four K bytes, the others the byte stores."""
    rng = np.random.default_rng(n)
    B = rng.standard_normal((naux, n, n))
    C = rng.standard_normal((n, n))
    store = ri.RiStore(B.reshape(naux, -1), nl=n)
    if planes == "ranges":
        assert drop_planes(store) == 1
    got = mo.buildRiNonRelSpinMoEri(store, n, C).b().reshape(naux, n, n)
    Bx, Cx = B.astype(X), C.astype(X)
    half = np.tensordot(Bx, Cx, (1, 0)).transpose(0, 2, 1)  # (P, j, a)
    ref = np.tensordot(half, Cx, (2, 0))
    bound = np.tensordot(np.tensordot(np.abs(B), np.abs(C), (1, 0)).transpose(0, 2, 1), np.abs(C), (2, 0))
    assert np.all(np.abs(got - ref.astype(float)) <= 2.0 ** -50 * bound)


@pytest.mark.parametrize("planes", ["resident", "ranges"])
@pytest.mark.parametrize("nl,ns,naux,nt", [(8, 16, 5, 3), (20, 44, 30, 40), (33, 70, 20, 65)])
def test_four_component_mo_transform(nl, ns, naux, nt, planes):
    rng = np.random.default_rng(nl)
    BL, BS = rng.standard_normal((naux, nl, nl)), rng.standard_normal((naux, ns, ns))
    nu = 2 * nl + 2 * ns
    C = rng.standard_normal((nu, nt)) + 1j * rng.standard_normal((nu, nt))
    src = ri.RiDirectEriSource(nl, ns, BL.reshape(naux, -1), BS.reshape(naux, -1))
    if planes == "ranges":
        assert drop_planes(src.store) == 1
    got = mo.buildRiMoEri(src, C).b().reshape(naux, nt, nt)
    off = [0, nl, 2 * nl, 2 * nl + ns, nu]
    ref = np.zeros((naux, nt, nt), dtype=np.clongdouble)
    bound = np.zeros((naux, nt, nt))
    for f, B in enumerate((BL, BL, BS, BS)):
        c = C[off[f]:off[f + 1]]
        cx = c.astype(np.clongdouble)
        ref += np.einsum("ai,paj->pij", cx.conj(), np.tensordot(B.astype(X), cx, (2, 0)))
        bound += np.einsum("ai,paj->pij", np.abs(c), np.tensordot(np.abs(B), np.abs(c), (2, 0)))
    assert np.all(np.abs(got - ref.astype(complex)) <= 2.0 ** -50 * np.sqrt(2.0) * bound)
