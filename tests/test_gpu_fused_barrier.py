"""A grid barrier of the fused rebin that runs out of time (XNB_STEP_BARRIER_CHECK: the
first one of a rebuild waits 20 ms for a block that does not exist) is reported for
the systems that were to be rebuilt, leaves the others alone, and is over with its
launch: systems added afterwards step as in a fresh batch."""
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch

pytestmark = pytest.mark.gpu


def test_batch_goes_on_after_a_barrier_ran_out():
    hot, still = workloads.lj_fcc_system(7, 0.8442, 1.44, 8), workloads.lj_fcc_system(6, 0.8442, 1.0, 9)
    still["v"] = 0.0 * still["v"]  # a lattice at rest: its trigger never fires
    b = new_batch([w["n_atoms"] for w in (hot, still)], [ncells(w["geom"]) for w in (hot, still)])
    s, q = (b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"]) for w in (hot, still))
    b.init_particles(-1, xnb.PREC_MIXED)
    b.step(40, xnb.PREC_MIXED, xnb.STEP_BARRIER_CHECK)
    assert b.info(s).error_bits == xnb.ERRBIT_BARRIER and b.info(q).error_bits == 0
    assert b.info(q).rebuilds == 0
    with pytest.raises(xnb.XnbError) as e:
        b.check_errors()
    assert e.value.code == -5
    b.step(10, xnb.PREC_MIXED, 0)  # not rebuilt again, not waited for
    b.step(1, xnb.PREC_MIXED, xnb.STEP_HOST_SYNC)
    b.remove_system(s)
    s = b.add_system(xnb.lj_params(hot["geom"]), hot["r"], hot["v"], hot["id"])
    b.init_particles(s, xnb.PREC_MIXED)
    b.step(60, xnb.PREC_MIXED, 0)
    b.check_errors()
    for w, mine, steps in ((hot, s, 60), (still, q, 111)):
        ref = new_batch([w["n_atoms"]], [ncells(w["geom"])])
        r = ref.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
        ref.init_particles(r, xnb.PREC_MIXED)
        ref.step(steps, xnb.PREC_MIXED, xnb.STEP_HOST_SYNC)
        assert b.info(mine).rebuilds == ref.info(r).rebuilds
        assert_bitwise_equal(b.download(mine), ref.download(r))
        ref.close()
    b.close()
