"""Whole SCF loops at the smallest sizes (the purification's workspace does not shrink with n) against the oracle's loops: energies
per iteration to 1e-8 Ha, same iteration count, as in test_gpu_scf.py."""
import numpy as np
import pytest

from oracle import ri_oracle as o
from rerdmft_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import ri, scf  # noqa: E402
from rerdmft_b200._lib import RrError  # noqa: E402


def check(r, ro):
    assert r["converged"] == ro["converged"] and r["iterations"] == ro["iterations"]
    assert np.abs(r["history"] - ro["history"]).max() <= 1e-8


@pytest.mark.parametrize("n,nocc", [(2, 1), (3, 2), (8, 3), (9, 4)])
def test_nonrel(n, nocc):
    s = synth.nonrel_system(n, 4 * n + 2, nocc, seed=n)
    src = ri.RiNonRelEriSource(n, s["B"], s["X"], s["S"])
    check(scf.runNonRelativisticHartreeFock(src, s["h"], s["X"], s["D0"], int(s["n_electrons"])), o.nonrel_scf(s))


@pytest.mark.parametrize("nl,ne", [(2, 2), (3, 4), (4, 4)])
def test_x2c(nl, ne):
    s = synth.x2c_system(nl, 4 * nl + 2, ne, seed=nl)
    src = ri.RiX2cEriSource(nl, s["B"], s["X"], s["S"])
    check(scf.runX2CHartreeFockScf(s["h"], src, s["X"], s["P0"], int(s["n_electrons"])), o.x2c_scf(s))


@pytest.mark.parametrize("nl,ns,ne", [(1, 2, 2), (2, 4, 2)])
def test_dhf(nl, ns, ne):
    s = synth.rkb_system(nl, ns, 6 * nl, ne, seed=nl)
    src = ri.RiDirectEriSource(nl, ns, s["B_LL"], s["B_SS"], s["v_total"], s["s_full"], s["x_full"])
    check(scf.runDiracHartreeFockScf(s["h"], src, s["x_full"], s["P0"], int(s["n_electrons"])), o.dhf_scf(s))


def test_one_level_is_refused():
    """All eigenvalues equal: the spectral interval is empty, and the purification ends with its error (60 and 120 steps)."""
    s = synth.nonrel_system(1, 6, 1, seed=1)
    src = ri.RiNonRelEriSource(1, s["B"], s["X"], s["S"])
    with pytest.raises(RrError, match="purification did not converge"):
        scf.runNonRelativisticHartreeFock(src, s["h"], s["X"], s["D0"], 2)
    s = synth.x2c_system(1, 6, 2, seed=1)
    src = ri.RiX2cEriSource(1, s["B"], s["X"], s["S"])
    with pytest.raises(RrError, match="purification did not converge"):
        scf.runX2CHartreeFockScf(s["h"], src, s["X"], s["P0"], 2)
