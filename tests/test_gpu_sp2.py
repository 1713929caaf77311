"""The one-launch SP2 purification and the small Ritz problem (csrc/sp2.cu) against numpy's eigensolver, around the tiles of
16, chunks of K and grid sizes.

Projector tolerance: a step rounds each element of X X at most (n + 2) times and its update twice, a perturbation d of
X turns its invariant subspaces by at most d / gap (gap relative to the spectral interval), about 40 steps, the
eigensolver's own error below that: 4 * 40 (n + 4) 2^-53 / gap.  Ritz values: reduction, tridiagonalisation and
bisection are backward stable, 1e-10 of the interval leaves a factor 1e3 for 32 x 32 problems with cond(M) up to 100."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import _lib as L  # noqa: E402


def hermitian(n, nocc, cplx, seed, gap=0.25):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0.0)
    q = np.linalg.qr(a)[0]
    e = np.sort(rng.uniform(0.0, 1.0 - gap, n))
    e[nocc:] += gap
    F = (q * e) @ q.conj().T
    return np.ascontiguousarray(0.5 * (F + F.conj().T)), q[:, :nocc] @ q[:, :nocc].conj().T


def sp2(F, nocc, lo, hi, sure=1, steps=120):
    Fd = torch.as_tensor(F, device="cuda")
    X = torch.empty_like(Fd)
    torch.cuda.synchronize()
    out = ctypes.c_double(-1.0)
    L.check(L.lib().rr_test_sp2(Fd.data_ptr(), F.shape[0], float(nocc), int(np.iscomplexobj(F)), lo, hi, sure, steps, X.data_ptr(),
                                ctypes.byref(out)))
    return X.cpu().numpy(), out.value


@pytest.mark.parametrize("n,nocc,cplx", [(1, 1, False), (2, 1, False), (15, 4, False), (16, 15, False), (17, 8, False), (33, 5, False),
                                         (161, 40, False), (263, 60, False), (400, 40, False), (512, 100, False), (1, 1, True), (15, 3, True),
                                         (17, 9, True), (33, 32, True), (197, 30, True), (400, 80, True)])
def test_projector(n, nocc, cplx):
    F, ref = hermitian(n, nocc, cplx, 7 * n + nocc)
    X, outcome = sp2(F, nocc, -0.1, 1.1)
    assert outcome == 0.0
    assert np.abs(X - ref).max() <= 160 * (n + 4) * 2.0 ** -53 / (0.25 / 1.2)
    assert np.array_equal(X, X.conj().T)


def test_outcomes():
    F, _ = hermitian(40, 10, False, 5)
    assert sp2(F, 10, 0.2, 0.8, sure=0)[1] == 1.0  # eigenvalues outside the interval
    assert sp2(F, 10, -0.1, 1.1, steps=3)[1] == 1.0


@pytest.mark.parametrize("cplx", [False, True])
def test_ritz(cplx):
    rng = np.random.default_rng(11)
    def draw():
        return rng.standard_normal((32, 32)) + (1j * rng.standard_normal((32, 32)) if cplx else 0.0)
    for k in range(6):
        q = np.linalg.qr(draw())[0]
        M = (q * np.geomspace(0.1, 10.0, 32)) @ q.conj().T
        M = 0.5 * (M + M.conj().T)
        T = draw()
        T = 0.5 * (T + T.conj().T) if k else np.diag(np.arange(32.0)).astype(T.dtype)  # (a reducible matrix too)
        w = np.linalg.eigvals(np.linalg.solve(M, T)).real
        lo, hi, m = w.min(), w.max(), 0.1 * (w.max() - w.min())
        Td, Md = torch.as_tensor(np.ascontiguousarray(T), device="cuda"), torch.as_tensor(np.ascontiguousarray(M), device="cuda")
        torch.cuda.synchronize()
        b = np.array([-1e6, hi + 0.5 * m])  # the upper end stays where it is narrower
        L.check(L.lib().rr_test_ritz(Td.data_ptr(), Md.data_ptr(), int(cplx), b.ctypes.data))
        assert abs(b[0] - (lo - m)) <= 1e-10 * (hi - lo) and b[1] == hi + 0.5 * m
    M[0, 0] = -1.0
    Md = torch.as_tensor(np.ascontiguousarray(M), device="cuda")
    torch.cuda.synchronize()
    b = np.array([-3.0, 4.0])
    L.check(L.lib().rr_test_ritz(Td.data_ptr(), Md.data_ptr(), int(cplx), b.ctypes.data))
    assert b.tolist() == [-3.0, 4.0]  # not positive definite: unchanged
