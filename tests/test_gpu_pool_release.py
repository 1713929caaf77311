"""Kept device blocks go back to the driver with the last object, also after a lockstep scan, whose workspaces stay for the process.  In a
process of its own: objects of other tests would count."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CODE = """
import gc
import torch
from rerdmft_b200 import ri, scf, synth

def scan():
    ss = [synth.x2c_system(nl, 4 * nl, 4, seed=nl) for nl in (10, 14)]
    probs = [dict(eri=ri.RiX2cEriSource(s["nl"], s["B"], s["X"], s["S"]), h_x2c=s["h"], x_large=s["X"], initial_density=s["P0"],
                  n_electrons=s["n_electrons"]) for s in ss]
    assert all(r["converged"] for r in scf.runX2CHartreeFockScfBatch(probs, mode="grouped"))
    for p in probs:
        p["eri"].store.close()

def store():
    return ri.RiStore(torch.ones(400, 300 * 300, dtype=torch.float64, device="cuda"), nl=300)  # 288 MB and more

store().close()  # the first use of a kernel loads it, which takes device memory of its own
scan()
gc.collect()
torch.cuda.empty_cache()
torch.cuda.synchronize()
free0 = torch.cuda.mem_get_info()[0]
kept = store()
assert torch.cuda.mem_get_info()[0] < free0 - 280e6
kept.close()
torch.cuda.empty_cache()
print("lost", free0 - torch.cuda.mem_get_info()[0])
assert free0 - torch.cuda.mem_get_info()[0] <= 32 << 20
"""


def test_blocks_go_back_after_a_scan():
    r = subprocess.run([sys.executable, "-c", CODE], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
