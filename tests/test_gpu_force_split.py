"""The two-stage mixed force kernel (batches of up to 50,000 particles) against
the sequential walk of the staged form: the same bits at the edges of its rows
and blocks -- particle counts off the block's group, lists longer than one
chunk of shared memory, lists of none and one pair, images on every side."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,keep,rcut,mass", [
    (7, None, 2.5, 1.0),    # 1,372 atoms: 4 past the last full group
    (6, 857, 2.5, 2.0),     # odd count, forces divided by the mass
    (6, 1, 2.5, 1.0),       # one atom, no pair
    (6, 2, 2.5, 1.0),       # two atoms, at most one pair
    (11, None, 4.2, 1.0),   # ~325 list entries: four chunks of 96
])
def test_split_equals_the_sequential_walk(n, keep, rcut, mass):
    w = workloads.lj_fcc_system(n, 0.8442, 1.2, 40 + n, rcut=rcut)
    r, v, ids = (w[k][:keep] for k in ("r", "v", "id"))
    r = r + np.random.default_rng(n).normal(0.0, 0.05, r.shape)
    b = new_batch([len(r)], [ncells(w["geom"])])
    if rcut > 4.0:
        b = xnb.Batch(len(r), ncells(w["geom"]), 600 * len(r))
    s = b.add_system(xnb.lj_params(w["geom"], rcut=rcut, mass=mass, divide_by_mass=mass != 1.0), r, v, ids)
    b.init_particles(s, xnb.PREC_MIXED)
    for energy in (True, False):
        out = []
        for form in (xnb.FORCE_THREAD, xnb.FORCE_STAGED):
            b.set_force_form(form)
            b.lennard_jones_force(s, xnb.PREC_MIXED, energy)
            out.append(b.download(s))
        b.set_force_form(xnb.FORCE_THREAD)
        assert_bitwise_equal(out[0], out[1], fields=("fx", "fy", "fz", "pe"))
    if rcut > 4.0:
        assert b.info(s).max_nbr > 256
    b.check_errors()
    b.close()
