"""The one-launch occupied recovery (csrc/recover_small.cu) through the Fock builds, at the sizes where it begins and ends
(79 real and 56 complex rows fit), with fewer orthonormal functions than AOs, more occupied ones than its shared memory takes,
none at all, and densities whose occupations are away from 0 and 1 (sign iterations, weighted factor).
Tolerance: the Fock builds' 1e-10 against the oracle."""
import numpy as np
import pytest

from oracle import ri_oracle as ro
from rerdmft_b200 import ri, synth

pytestmark = pytest.mark.gpu


def density(s, nocc, occ, seed):
    """sum_i occ_i c_i c_i^T over orthonormal orbitals (C^T S C = 1)."""
    rng = np.random.default_rng(seed)
    q = np.linalg.qr(rng.standard_normal((s["X"].shape[1], s["X"].shape[1])))[0][:, :nocc]
    c = s["X"] @ q
    return (c * (2.0 * np.asarray(occ))) @ c.T


@pytest.mark.parametrize("n,naux,nocc,drop", [(1, 3, 1, 0), (5, 11, 2, 0), (24, 60, 5, 3), (33, 70, 31, 0), (64, 90, 20, 1), (79, 100, 14, 0),
                                              (79, 60, 60, 0), (80, 100, 14, 0), (30, 40, 0, 0)])
def test_nonrel(n, naux, nocc, drop):
    s = synth.nonrel_system(n, naux, max(nocc, 1), seed=n)
    s["X"] = np.ascontiguousarray(s["X"][:, :n - drop])
    D = density(s, nocc, np.ones(nocc), n)
    F = ri.nonRelFockMatrix(s["h"], ri.RiNonRelEriSource(n, s["B"], s["X"], s["S"]), D)
    assert np.abs(F - ro.nonrel_fock(s["h"], s["B"], D, s["S"], s["X"])).max() <= 1e-10


def test_nonrel_occupations_between():
    s = synth.nonrel_system(40, 80, 9, seed=3)
    D = density(s, 12, np.r_[np.ones(6), 0.93, 0.8, 0.71, 0.3, 0.1, 1e-3], 4)
    F = ri.nonRelFockMatrix(s["h"], ri.RiNonRelEriSource(40, s["B"], s["X"], s["S"]), D)
    assert np.abs(F - ro.nonrel_fock(s["h"], s["B"], D, s["S"], s["X"])).max() <= 1e-10


@pytest.mark.parametrize("nl,naux,ne", [(1, 4, 2), (12, 48, 4), (20, 40, 36), (28, 60, 8), (29, 60, 8)])
@pytest.mark.parametrize("scale", [1.0, 0.85])
def test_x2c(nl, naux, ne, scale):
    x = synth.x2c_system(nl, naux, ne, seed=nl)
    P = scale * x["P0"]
    F = ri.x2cFockMatrix(x["h"], ri.RiX2cEriSource(nl, x["B"], x["X"], x["S"]), P)
    assert np.abs(F - ro.x2c_fock(x["h"], x["B"], P, x["S"], x["X"])).max() <= 1e-10
