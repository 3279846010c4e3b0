"""backup_r's encoding inside the rebin's last pass, as a pass of its own and in the
fused rebin: FP64_EXACT runs with several rebuilds equal the oracle bit for bit,
with the same rebuilds, where the cells are full, sparse, and too many particles
for the first form."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch, oracle_from
from test_gpu_fused_rebin import gas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system,steps", [
    (lambda: workloads.lj_fcc_system(9, 0.8442, 2.0, 3), 60),    # ~19 per cell
    (lambda: workloads.lj_fcc_system(12, 0.34, 2.0, 3), 60),     # ~8 per cell, at the line
    (lambda: gas(12, 400, 3), 30),                               # most cells empty
    (lambda: workloads.lj_fcc_system(24, 0.8442, 2.0, 3), 25),   # 55,296 atoms
], ids=["full", "line", "sparse", "large"])
@pytest.mark.parametrize("flags", [xnb.STEP_HOST_SYNC, 0], ids=["sync", "fused"])
def test_exact_run_equals_the_oracle(system, steps, flags):
    w = system()
    b = new_batch([w["n_atoms"]], [ncells(w["geom"])])
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
    b.init_particles(s, xnb.PREC_FP64_EXACT)
    o = oracle_from(w)
    o.init()
    rebuilt = sum(int(o.step()) for _ in range(steps))
    b.step(steps, xnb.PREC_FP64_EXACT, flags)
    b.check_errors()
    assert b.info(s).rebuilds == rebuilt >= 2
    assert_bitwise_equal(b.download(s), o.particles())
    b.close()
