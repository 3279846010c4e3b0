"""The one-thread mixed walk of larger batches (from 500,000 particles on) against
the sequential FP64 sums of the staged form: the same bits with images on every
side, coordinates that are zero (no FP32 mirror to step from), sums outside the
exact integer range (close contacts), odd list lengths, a partly filled block,
and systems that keep the marking walk (origin off zero, long cutoff)."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,noise,keep,rcut,mass,shift", [
    (50, 0.05, None, 2.5, 1.0, 0.0),    # a thermal fluid of 500,000 atoms, the fewest that take the walk
    (51, 0.0, None, 2.5, 1.0, 0.0),     # the lattice itself: a face of atoms at coordinate 0 on each axis
    (51, 0.2, 500001, 2.5, 2.0, 0.0),   # overlapping atoms, an odd count
    (50, 0.05, 499999, 2.5, 1.0, 0.0),  # one below: the marking walk
    (50, 0.05, None, 2.5, 1.0, -17.0),  # origin off zero: the marking walk
    (50, 0.05, None, 3.2, 1.0, 0.0),    # a long cutoff: the marking walk
])
def test_walk_equals_the_sequential_sums(n, noise, keep, rcut, mass, shift):
    w = workloads.lj_fcc_system(n, 0.8442, 1.2, 31, rcut=rcut)
    r, v, ids = (w[k][:keep] for k in ("r", "v", "id"))
    r = r + np.random.default_rng(5).normal(0.0, 1.0, r.shape) * noise if noise else r - r.min(axis=0)
    geom = dict(w["geom"])
    geom["origin"] = tuple(o + shift for o in geom["origin"])
    geom["extent"] = tuple(o + shift for o in geom["extent"])
    b = new_batch([len(r)], [ncells(geom)]) if rcut < 3.0 else xnb.Batch(len(r), ncells(geom), 320 * len(r))
    s = b.add_system(xnb.lj_params(geom, rcut=rcut, mass=mass, divide_by_mass=mass != 1.0), r + shift, v, ids)
    b.init_particles(s, xnb.PREC_MIXED)
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
