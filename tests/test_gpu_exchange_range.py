"""The FP64 exchange on digit planes where the half-transformed rows lie far below the bound that sets their exponents: nearly
dependent functions with large cancelling coefficients, and functions far from every occupied orbital.  csrc/oz.cu, refit_kernel.

Tolerance: that of FP64 arithmetic in any order.  T_a = sum_q B_qa c_q is off by at most n 2^-53 A_a, A_a = sum_q |B_qa| |c_q|, so K_ab by
at most delta_a d_b + d_a delta_b + delta_a delta_b with delta_a = n 2^-53 |A_a| and d_a = sqrt(K_aa) (2-norms over the aux rows and orbitals,
Cauchy-Schwarz), and the sum of K_ab by 2^-48 d_a d_b (test_gpu_digit_products.py); twice that for the complex parts."""
import numpy as np
import pytest

from test_gpu_digit_products import X, drop_planes, exchange

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import ri, synth  # noqa: E402


def tensor(kind, n, naux, seed):
    """B (naux, n, n) and the map from ordinary coefficients to the ones that go with it."""
    B = synth.ri_tensor(n, naux, seed, box=8.0).reshape(naux, n, n)
    M = np.eye(n)
    if kind == "dependent":  # function 2 k + 1 is function 2 k plus 2^-20 of its own
        for k in range(n // 4):
            M[2 * k + 1, 2 * k + 1] = 2.0 ** -20
            M[2 * k + 1, 2 * k] = 1.0
        B = np.einsum("ab,pbc,dc->pad", M, B, M, optimize=True)
        return 0.5 * (B + B.transpose(0, 2, 1)), lambda c: np.linalg.solve(M.T, c)
    far = np.arange(n) >= {"far": n // 2, "three": n - 3}[kind]  # nothing occupied there, 2^-30 of overlap with the rest
    B = B * np.where(far[:, None] != far[None, :], 2.0 ** -30, 1.0)
    return B, lambda c: np.where(far[:, None], 0.0, c)


def norms(B, c):
    """2-norms over (P, j) of sum_q |B_qa| |c_q| for every a."""
    a = np.tensordot(np.abs(B), np.abs(c), (1, 0))
    return np.sqrt((a ** 2).sum(axis=(0, 2)))


def bound(delta, d):
    return np.outer(delta, d) + np.outer(d, delta) + np.outer(delta, delta) + 2.0 ** -48 * np.outer(d, d)


@pytest.mark.parametrize("planes", ["resident", "ranges"])
@pytest.mark.parametrize("kind,n,naux,nocc", [("dependent", 129, 201, 61), ("far", 128, 371, 33), ("three", 161, 131, 65)])
def test_nonrel_exchange(kind, n, naux, nocc, planes):
    B, to = tensor(kind, n, naux, n)
    C = to(np.linalg.qr(np.random.default_rng(n).standard_normal((n, nocc)))[0])
    store = ri.RiStore(B.reshape(naux, -1), nl=n)
    if planes == "ranges":
        assert drop_planes(store) == 1
    _, K = ri.jk_occupied(store, C)
    ref, _ = exchange(B, C, C)
    d = np.sqrt(np.diag(ref)).astype(float)
    assert np.all(np.abs(K - ref.astype(float)) <= bound(n * 2.0 ** -53 * norms(B, C), d))
    assert np.array_equal(K, K.T)


@pytest.mark.parametrize("planes", ["resident", "ranges"])
@pytest.mark.parametrize("kl,ks,nl,ns,naux,r", [("dependent", "far", 33, 65, 40, 5), ("three", "dependent", 64, 129, 31, 9)])
def test_four_component_two_electron(kl, ks, nl, ns, naux, r, planes):
    rng = np.random.default_rng(nl)
    BL, tl = tensor(kl, nl, naux, nl)
    BS, ts = tensor(ks, ns, naux, ns)
    nu = 2 * nl + 2 * ns
    C = np.linalg.qr(rng.standard_normal((nu, r)) + 1j * rng.standard_normal((nu, r)))[0]
    off = [0, nl, 2 * nl, 2 * nl + ns, nu]
    T, to = [BL, BL, BS, BS], [tl, tl, ts, ts]
    C = np.concatenate([to[f](C[off[f]:off[f + 1]]) for f in range(4)])
    src = ri.RiDirectEriSource(nl, ns, BL.reshape(naux, -1), BS.reshape(naux, -1))
    if planes == "ranges":
        assert drop_planes(src.store) == 1
    G = ri.riFockTwoElectronDirect(src, np.zeros((nu, nu), dtype=complex), C, np.ones(r))
    half = [np.tensordot(T[f].astype(X), C[off[f]:off[f + 1]].astype(np.clongdouble), (1, 0)).transpose(1, 0, 2).reshape(T[f].shape[1], -1)
            for f in range(4)]
    K = np.concatenate([np.concatenate([half[f] @ half[u].conj().T for u in range(4)], axis=1) for f in range(4)])
    d = np.sqrt(np.diag(K).real).astype(float)
    delta = np.concatenate([T[f].shape[1] * 2.0 ** -53 * norms(T[f], C[off[f]:off[f + 1]]) for f in range(4)])
    assert np.all(np.abs(G + K.astype(complex)) <= 2.0 * bound(delta, d))
