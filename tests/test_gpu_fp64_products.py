"""rr_ri_set_fp64_products: RR_FP64_DMMA handles form exchange and MO transforms as FP64 sums, whose errors are bounded element by element;
the digit products keep the normwise bound of the header, and come back with RR_FP64_DIGITS bit for bit.

Tolerances: a sum of k FP64 products in any order is off by at most k 2^-53 of the sum of their magnitudes; T = B C has n terms, K naux nocc,
and both factors of K carry T's error: (2 n + naux nocc + 4) 2^-53 of A^T A, A = |B| |C|.  B_mo: (2 n + 4) 2^-53 of |C|^T |B| |C|;
either plus n^2 products of terms that underflow, far below 1e-300."""
import ctypes

import numpy as np
import pytest

from test_gpu_digit_products import REL, X, exchange

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import _lib as L  # noqa: E402
from rerdmft_b200 import mo, ri, synth  # noqa: E402

U = 2.0 ** -53
TINY = 1e-300


def test_small_elements_of_an_extended_system():
    """Centres 50 bohr apart along a chain and localised orbitals: elements of K over 60 orders of magnitude."""
    n, naux, nocc = 144, 240, 48
    rng = np.random.default_rng(3)
    r, ra = np.sort(rng.uniform(0.0, 50.0, n)), rng.uniform(0.0, 50.0, naux)
    g = np.exp(-0.3 * (ra[:, None] - r[None, :]) ** 2)
    c = rng.standard_normal((naux, n, n))
    B = 0.5 * (c + c.transpose(0, 2, 1)) * g[:, :, None] * g[:, None, :]
    C = np.exp(-0.5 * (r[:, None] - r[None, ::3]) ** 2) * rng.standard_normal((n, nocc))
    store = ri.RiStore(B.reshape(naux, -1), nl=n)
    ref, _ = exchange(B, C, C)
    a = np.tensordot(np.abs(B), np.abs(C), (1, 0)).transpose(1, 0, 2).reshape(n, -1)
    by_element = (2 * n + naux * nocc + 4) * U * (a @ a.T) + TINY
    d = np.sqrt(np.diag(ref)).astype(float)
    digits = ri.jk_occupied(store, C)[1]
    assert np.all(np.abs(digits - ref.astype(float)) <= REL * np.outer(d, d))
    store.set_fp64_products("dmma")
    K = ri.jk_occupied(store, C)[1]
    assert np.all(np.abs(K - ref.astype(float)) <= by_element)
    Cm = np.exp(-0.5 * (r[:, None] - r[None, :]) ** 2) * rng.standard_normal((n, n))
    got = mo.buildRiNonRelSpinMoEri(store, n, Cm).b().reshape(naux, n, n)
    Cx = Cm.astype(X)
    mo_ref = np.tensordot(np.tensordot(B.astype(X), Cx, (1, 0)).transpose(0, 2, 1), Cx, (2, 0))
    mo_abs = np.tensordot(np.tensordot(np.abs(B), np.abs(Cm), (1, 0)).transpose(0, 2, 1), np.abs(Cm), (2, 0))
    assert np.all(np.abs(got - mo_ref.astype(float)) <= (2 * n + 4) * U * mo_abs + TINY)
    store.set_fp64_products("digits")
    assert np.array_equal(ri.jk_occupied(store, C)[1], digits)
    norm = np.sqrt((B ** 2).sum(1)).max(1)[:, None, None] * np.outer(*[np.sqrt((Cm ** 2).sum(0))] * 2)[None]
    got = mo.buildRiNonRelSpinMoEri(store, n, Cm).b().reshape(naux, n, n)
    assert np.all(np.abs(got - mo_ref.astype(float)) <= U * norm + (2 * n + 4) * U * mo_abs)


def test_relativistic_builds_follow_the_handle():
    s = synth.x2c_system(24, 96, 8, seed=5)
    src = ri.RiX2cEriSource(24, s["B"], s["X"], s["S"])
    digits = ri.x2cFockMatrix(s["h"], src, s["P0"])
    src.store.set_fp64_products("dmma")
    dmma = ri.x2cFockMatrix(s["h"], src, s["P0"])
    assert not np.array_equal(digits, dmma) and np.abs(digits - dmma).max() <= 1e-12 * max(1.0, np.abs(dmma).max())
    src.store.set_fp64_products("digits")
    assert np.array_equal(ri.x2cFockMatrix(s["h"], src, s["P0"]), digits)


def test_unknown_kind_is_refused():
    store = ri.RiStore(np.ones((3, 16)), nl=4)
    assert L.lib().rr_ri_set_fp64_products(store.handle, 2) == L.RR_ERR_ARG
    assert L.lib().rr_ri_set_fp64_products(ctypes.c_void_p(), 0) == L.RR_ERR_ARG
