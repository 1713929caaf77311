"""The one-launch Cholesky factor-and-apply of the occupied recovery (csrc/chol_apply.cu): r around its panels of 8
(real) and 4 (complex) columns and up to what shared memory holds, row counts around one row per SM, Gram matrices
on both sides of the near-identity rule.

Checked: the invariants that the recovery uses, X X^H = Y M^-1 Y^H and X X^H = Y M Y^H (they hold for the triangular
and the symmetric factor alike).  Tolerance: factor, substitution and products are backward stable with constants of at
most (r + 2) roundings each, complex arithmetic and the reference's own solve together a factor 8; a perturbation of M of
that size moves M^-1 by cond(M) times it: 8 (r + 2) 2^-53 cond(M) |M^-+1| |y_i| |y_j|."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import _lib as L  # noqa: E402


def apply(M, Y, times_l):
    r, n, cplx = M.shape[0], Y.shape[0], np.iscomplexobj(M)
    Md, Yd = torch.as_tensor(M, device="cuda"), torch.as_tensor(Y, device="cuda")
    out = torch.zeros_like(Yd)
    torch.cuda.synchronize()
    ran, status = ctypes.c_int32(), ctypes.c_int32()
    L.check(L.lib().rr_test_chol_apply(Md.data_ptr(), r, Yd.data_ptr(), n, int(cplx), int(times_l), out.data_ptr(),
                                       ctypes.byref(ran), ctypes.byref(status)))
    return out.cpu().numpy(), ran.value, status.value


def operands(r, n, cplx, spread, rng):
    """M = 1 + Hermitian with inf-norm `spread` (near the identity), or eigenvalues from 0.3 to 3 (spread None)."""
    draw = (lambda *s: rng.standard_normal(s) + 1j * rng.standard_normal(s)) if cplx else (lambda *s: rng.standard_normal(s))
    if spread is None:
        q = np.linalg.qr(draw(r, r))[0]
        M = (q * np.geomspace(0.3, 3.0, r)) @ q.conj().T
    else:
        E = draw(r, r)
        E = E + E.conj().T
        M = np.eye(r) + E * (spread / (r * max(np.abs(E.real).max(), np.abs(E.imag).max())))
    M = 0.5 * (M + M.conj().T)
    return np.ascontiguousarray(M), np.ascontiguousarray(draw(n, r))


@pytest.mark.parametrize("spread", [None, 1e-9, 3.9e-6, 4.1e-6])
@pytest.mark.parametrize("times_l", [False, True])
@pytest.mark.parametrize("cplx,r,n", [(False, 1, 1), (False, 7, 148), (False, 8, 149), (False, 9, 24), (False, 31, 297), (False, 120, 400),
                                      (False, 161, 160), (True, 1, 2), (True, 3, 148), (True, 4, 149), (True, 5, 40), (True, 33, 297),
                                      (True, 80, 400), (True, 113, 144)])
def test_chol_apply(cplx, r, n, times_l, spread):
    rng = np.random.default_rng(1000 * r + n)
    M, Y = operands(r, n, cplx, spread, rng)
    X, ran, status = apply(M, Y, times_l)
    assert ran == 1 and status == 0
    ref = Y @ M @ Y.conj().T if times_l else Y @ np.linalg.solve(M, Y.conj().T)
    w = np.linalg.eigvalsh(M)
    y = np.linalg.norm(Y, axis=1)
    tol = 8 * (r + 2) * 2.0 ** -53 * (w[-1] / w[0]) * (w[-1] if times_l else 1 / w[0])
    assert np.all(np.abs(X @ X.conj().T - ref) <= tol * np.outer(y, y))


@pytest.mark.parametrize("cplx", [False, True])
def test_non_positive_pivot_and_nan_are_reported(cplx):
    M = np.diag([1.0, 2.0, -1.0, 4.0, 1.0, 1.0, 1.0, 1.0, 1.0]).astype(complex if cplx else float)
    Y = np.ones((5, 9), dtype=M.dtype)
    assert apply(M, Y, False)[1:] == (1, 1)
    M[2, 2] = np.nan
    assert apply(M, Y, True)[1:] == (1, 1)


def test_too_large_for_shared_memory_is_refused():
    M, Y = operands(200, 8, False, None, np.random.default_rng(1))
    X, ran, _ = apply(M, Y, False)
    assert ran == 0 and not X.any()
