"""Mixed forces of sparse batches at the line between the two-stage form and one
thread per particle: the same bits as the staged form's sequential sums on either
side of it, whatever number of threads per particle is set."""
import pytest

from exanbody_gb300 import xnb
from helpers import assert_bitwise_equal, ncells, new_batch
from test_gpu_fused_rebin import gas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20000, 28800, 28801, 33000])  # 24-entry slots: two stages up to 28,800
@pytest.mark.parametrize("lanes", [1, 4])
def test_forces_equal_the_sequential_sums(n, lanes):
    w = gas(46, n, n)
    b = new_batch([n], [ncells(w["geom"])])
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
    b.set_force_lanes(lanes)
    b.init_particles(s, xnb.PREC_MIXED)
    assert b.info(s).list_cap == 24 * n
    b.step(5, xnb.PREC_MIXED, 0)  # with the kick
    for energy in (True, False):
        out = []
        for form in (xnb.FORCE_THREAD, xnb.FORCE_STAGED):
            b.set_force_form(form)
            b.lennard_jones_force(s, xnb.PREC_MIXED, energy)
            out.append(b.download(s))
        b.set_force_form(xnb.FORCE_THREAD)
        assert_bitwise_equal(out[0], out[1], fields=("fx", "fy", "fz", "pe") if energy else ("fx", "fy", "fz"))
    b.check_errors()
    b.close()
