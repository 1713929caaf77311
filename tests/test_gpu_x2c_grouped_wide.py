"""Lockstep X2C-HF batches with an instance beyond the one-launch purification (more than 400 functions): the others' results are bit for
bit those they have alone, and the wide one agrees with the single-instance loop."""
import numpy as np
import pytest

from rerdmft_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rerdmft_b200 import ri, scf  # noqa: E402


@pytest.mark.parametrize("wide", [0, 2])  # first and last of the list
def test_results_do_not_depend_on_a_wide_neighbour(wide):
    shapes = [(20, 80, 4), (33, 132, 14)]
    shapes.insert(wide, (203, 220, 6))
    systems = [synth.x2c_system(nl, naux, ne, seed=400 + k + 10 * wide) for k, (nl, naux, ne) in enumerate(shapes)]
    probs = [dict(eri=ri.RiX2cEriSource(s["nl"], s["B"], s["X"], s["S"]), h_x2c=s["h"], x_large=s["X"], initial_density=s["P0"],
                  n_electrons=s["n_electrons"]) for s in systems]
    batch = scf.runX2CHartreeFockScfBatch(probs, mode="grouped")
    for k, p in enumerate(probs):
        alone = scf.runX2CHartreeFockScfBatch([p], mode="grouped")[0]
        assert alone["converged"] and alone["iterations"] == batch[k]["iterations"]
        assert np.array_equal(alone["history"], batch[k]["history"])
        assert np.array_equal(alone["P"], batch[k]["P"])
    s = systems[wide]
    single = scf.runX2CHartreeFockScf(s["h"], probs[wide]["eri"], s["X"], s["P0"], s["n_electrons"])
    assert abs(batch[wide]["energy"] - single["energy"]) <= 1e-9
    assert np.abs(batch[wide]["P"] - single["P"]).max() <= 1e-7
    for p in probs:
        p["eri"].store.close()
