"""Every class kernel of the integral engine (csrc/eri_class_*.cu: pairs up to (dd| and (fs|, aux s .. f) and the warp
kernel's nearest classes against the oracle, with shells that share a centre, shells apart, and tight shells so
far apart that their primitive pairs underflow.  Tolerance as for the other integral tests: 1e-12 of the largest."""
import numpy as np
import pytest

from oracle import integrals_oracle as io
from rerdmft_b200 import basis as bs
from rerdmft_b200 import integrals as gi

pytestmark = pytest.mark.gpu


def shell(rng, l, nprim, center, tight=1.0):
    ex = [float(x) * tight for x in sorted(rng.uniform(0.15, 6.0, nprim), reverse=True)]
    co = [float(x) for x in rng.uniform(0.2, 1.0, nprim)]
    return [bs.BasisFunction("X", *map(float, center), l, c, list(ex), list(co)) for c in bs.cartesian_components(l)]


@pytest.mark.parametrize("la,lb", [(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (2, 2), (3, 0), (3, 1)])
def test_class(la, lb):
    rng = np.random.default_rng(10 * la + lb)
    cen = rng.uniform(-1.5, 1.5, (3, 3))
    far = cen[0] + 9.0
    orb = shell(rng, la, 2, cen[0]) + shell(rng, lb, 3, cen[1]) + shell(rng, lb, 1, cen[0]) + shell(rng, la, 2, far, 40.0)
    aux = [f for l in range(4) for f in shell(rng, l, 1 + l % 2, cen[l % 3])] + shell(rng, 1, 1, far)
    bs.normalize_cartesian_basis(orb)
    bs.normalize_cartesian_basis(aux)
    ref = io.three_center_raw(orb, aux)
    raw = gi.threeCenterIntegralsRaw(orb, aux)
    assert np.abs(raw - ref).max() <= 1e-12 * np.abs(ref).max()
    M, mref = gi.auxMetric(aux), io.aux_metric(aux)
    assert np.abs(M - mref).max() <= 1e-12 * np.abs(mref).max()
