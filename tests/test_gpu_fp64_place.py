"""FP64 full-list forces of a system are the same bits whatever else its batch holds:
alone, behind systems whose particle counts and list lengths differ, and stepped
with them; lists of a dilute gas, of a dense fluid, and longer than one round (96)."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch
from test_gpu_fused_rebin import gas

pytestmark = pytest.mark.gpu

ALL = ("rx", "ry", "rz", "vx", "vy", "vz", "fx", "fy", "fz", "pe")


def systems():
    out = [workloads.lj_fcc_system(5, 0.8442, 1.2, 1), gas(9, 331, 2), workloads.lj_fcc_system(6, 0.95, 1.0, 3),
           workloads.lj_fcc_system(5, 0.7, 1.4, 4), workloads.lj_fcc_system(7, 1.15, 0.8, 5)]
    for k, w in enumerate(out):  # odd counts: every system begins elsewhere in a group of eight
        keep = len(w["r"]) - (1, 2, 5, 3, 0)[k]
        for q in ("r", "v", "id"):
            w[q] = w[q][:keep]
        w["n_atoms"] = keep
    return out


def batch_of(ws):
    b = new_batch([w["n_atoms"] for w in ws], [ncells(w["geom"]) for w in ws], list_per_atom=250.0)
    ss = [b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"]) for w in ws]
    b.init_particles(-1, xnb.PREC_FP64)
    return b, ss


@pytest.mark.parametrize("steps", [0, 60])
def test_same_bits_alone_and_in_a_batch(steps):
    ws = systems()
    b, ss = batch_of(ws)
    if steps:
        b.step(steps, xnb.PREC_FP64, xnb.STEP_ENERGY)
    b.check_errors()
    for w, s in zip(ws, ss):
        alone, (q,) = batch_of([w])
        if steps:
            alone.step(steps, xnb.PREC_FP64, xnb.STEP_ENERGY)
        assert_bitwise_equal(b.download(s), alone.download(q), fields=ALL)
        alone.close()
    b.close()
