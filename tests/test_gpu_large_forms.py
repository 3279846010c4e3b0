"""Forms of the mixed step that only larger batches take: the threads-per-particle
split (above 50,000 particles), the single-visit walk with the second-half kick and
the position steps that each push writes (from 500,000 on), and the separate rebin
kernels without host synchronisation (above 100,000)."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, force_error, forces, ncells, new_batch, oracle_from

pytestmark = pytest.mark.gpu


def batch_of(ws, precision):
    b = new_batch([w["n_atoms"] for w in ws], [ncells(w["geom"]) for w in ws])
    ss = [b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"]) for w in ws]
    b.init_particles(-1, precision)
    return b, ss


@pytest.mark.parametrize("lanes", [2, 4])
def test_lanes_split_the_lists(lanes):
    w = workloads.lj_fcc_system(24, 0.8442, 1.44, 21)  # 55,296 atoms
    b, (s,) = batch_of([w], xnb.PREC_MIXED)
    b.step(25, xnb.PREC_MIXED, 0)
    out = []
    for n, prec in ((1, xnb.PREC_FP64_EXACT), (1, xnb.PREC_MIXED), (lanes, xnb.PREC_MIXED), (lanes, xnb.PREC_MIXED)):
        b.set_force_lanes(n)
        b.lennard_jones_force(s, prec, True)
        out.append(b.download(s))
    exact, one, many, again = out
    for P in (one, many):
        assert force_error(forces(P), forces(exact))[0] <= 1e-5
        assert abs(P["pe"].sum() - exact["pe"].sum()) <= 1e-5 * abs(exact["pe"].sum())
    # another order of the same FP64 sums: equal to rounding, and not the same kernel
    e, _ = force_error(forces(many), forces(one))
    assert 0.0 < e <= 1e-10
    assert_bitwise_equal(many, again, fields=("fx", "fy", "fz", "pe"))
    b.close()


@pytest.mark.parametrize("n,shift", [(50, 0.0), (51, 1e-3)])  # 500,000 and 530,604 atoms
def test_walk_steps_equal_the_staged_form(n, shift):
    w = workloads.lj_fcc_system(n, 0.8442, 1.44, 5)
    w["r"] = w["r"] + shift
    out = []
    for form in (xnb.FORCE_THREAD, xnb.FORCE_STAGED):
        b, (s,) = batch_of([w], xnb.PREC_MIXED)
        b.set_force_form(form)
        states = []
        for steps in (1, 2, 20):  # from a fresh rebin, from pushed positions alone, over rebuilds
            b.step(steps, xnb.PREC_MIXED, xnb.STEP_ENERGY)
            states.append(b.download(s))
        b.check_errors()
        out.append((states, b.info(s).rebuilds))
        b.close()
    assert out[0][1] == out[1][1] >= 1
    for t, g in zip(*(states for states, _ in out)):
        assert_bitwise_equal(t, g, fields=("rx", "ry", "rz", "vx", "vy", "vz", "fx", "fy", "fz", "pe"))


def test_asynchronous_rebin_of_a_large_batch():
    """30^3 cells (108,000 atoms): exact against the oracle, mixed against host-synchronised steps; and a
    system of 87,808 atoms beside another one (separate kernels) against itself alone (the fused rebin)."""
    w = workloads.lj_fcc_system(30, 0.8442, 1.44, 7)
    b, (s,) = batch_of([w], xnb.PREC_FP64_EXACT)
    o = oracle_from(w)
    o.init()
    rebuilt = sum(int(o.step()) for _ in range(25))
    b.step(25, xnb.PREC_FP64_EXACT, 0)
    b.check_errors()
    assert b.info(s).rebuilds == rebuilt >= 2
    assert_bitwise_equal(b.download(s), o.particles())
    b.close()
    out = []
    for flags in (0, xnb.STEP_HOST_SYNC):
        b, (s,) = batch_of([w], xnb.PREC_MIXED)
        b.step(40, xnb.PREC_MIXED, flags)
        b.check_errors()
        out.append((b.download(s), b.info(s).rebuilds, b.pairs(s)))
        b.close()
    assert out[0][1] == out[1][1] >= 3
    assert_bitwise_equal(out[0][0], out[1][0])
    assert all(np.array_equal(x, y) for x, y in zip(out[0][2], out[1][2]))
    ws = [workloads.lj_fcc_system(28, 0.8442, 1.44, 8), workloads.lj_fcc_system(16, 0.95, 1.0, 9)]
    out = []
    for group in (ws, ws[:1]):
        b, ss = batch_of(group, xnb.PREC_MIXED)
        b.step(40, xnb.PREC_MIXED, 0)
        b.check_errors()
        out.append((b.download(ss[0]), b.pairs(ss[0])))
        b.close()
    assert_bitwise_equal(out[0][0], out[1][0])
    assert all(np.array_equal(x, y) for x, y in zip(out[0][1], out[1][1]))
