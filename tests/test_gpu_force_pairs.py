"""The FP64 and FP64_EXACT force kernels (a warp per eight particles) against the
oracle at the edges of their groups and rounds: particle counts off the groups of
8 and 32, no pair and one pair, lists longer than one round of 96 entries, runs
that pass several particles with a few pairs each, other units, masses."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, force_error, forces, ncells
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rho,keep,rcut,eps,sigma,mass", [
    (6, 0.8442, 857, 2.5, 1.0, 1.0, 1.0),    # odd count
    (6, 0.8442, 33, 2.5, 0.7, 1.05, 2.5),    # one particle past a block, divided by the mass
    (6, 0.8442, 1, 2.5, 1.0, 1.0, 1.0),      # no pair
    (6, 0.8442, 2, 2.5, 1.0, 1.0, 1.0),      # two particles
    (9, 0.10, None, 2.5, 1.0, 1.0, 1.0),     # ~6 pairs each: runs cross several particles
    (11, 0.8442, None, 3.9, 1.3, 0.98, 1.0),  # ~260 list entries: three rounds
])
def test_forces_and_energies(n, rho, keep, rcut, eps, sigma, mass):
    w = workloads.lj_fcc_system(n, rho, 1.0, 60 + n, rcut=rcut)
    g = w["geom"]
    r = (w["r"] + np.random.default_rng(n).normal(0.0, 0.07, w["r"].shape)) % np.array(g["extent"])
    r, v, ids = r[:keep], w["v"][:keep], w["id"][:keep]
    div = mass != 1.0
    o = OracleSystem(g["origin"], g["extent"], g["dims"], g["cell_size"], rcut, 0.3, eps, sigma, 0.005, mass=mass,
                     divide_by_mass=div, kind="omp")
    o.load_flat(r, v, ids)
    o.init()
    ref = o.particles()
    b = xnb.Batch(len(r), ncells(g), 700 * len(r) + 4096)
    s = b.add_system(xnb.lj_params(g, epsilon=eps, sigma=sigma, rcut=rcut, mass=mass, divide_by_mass=div), r, v, ids)
    b.init_particles(s, xnb.PREC_FP64_EXACT)
    assert_bitwise_equal(b.download(s), ref, fields=("fx", "fy", "fz", "pe"))
    if rcut > 3.0:
        assert b.info(s).max_nbr > 2 * 96
    for energy in (True, False):
        b.lennard_jones_force(s, xnb.PREC_FP64_EXACT, energy)
        assert_bitwise_equal(b.download(s), ref, fields=("fx", "fy", "fz") + (("pe",) if energy else ()))
        for prec in (xnb.PREC_FP64, xnb.PREC_FP64 | xnb.PREC_NEWTON):
            b.lennard_jones_force(s, prec, energy)
            got = b.download(s)
            if len(r) > 1 and np.abs(forces(ref)).max() > 0:
                assert force_error(forces(got), forces(ref))[0] <= 1e-12
            else:
                assert np.array_equal(forces(got), forces(ref))
            if energy:
                assert np.allclose(got["pe"], ref["pe"], rtol=1e-12, atol=1e-12 * max(1e-300, np.abs(ref["pe"]).max()))
    b.close()
