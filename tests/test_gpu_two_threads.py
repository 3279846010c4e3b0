"""Two host threads, each with its own batch and stream, step at once. The
batches differ in what their launches ask of shared memory (a dense and a dilute
fluid, a large and a small stage of the lists built with the rebin, SNAP
potentials of different order), and a launch's limit is the kernel's, not the
thread's: every launch has to go through, and results are those of one thread."""
import threading

import numpy as np
import pytest

from exanbody_gb300 import snap, workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch, ni_deck_params

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def at_once(*calls):
    failed = []

    def guarded(f):
        try:
            f()
        except Exception as e:  # reported by the test's own thread
            failed.append(e)

    ts = [threading.Thread(target=guarded, args=(f,)) for f in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed, failed


def batch(rho, cap, stream):
    w = workloads.lj_fcc_system(8, rho, 1.2, 5)
    b = new_batch([w["n_atoms"]], [ncells(w["geom"])])
    b.stream = stream
    b.set_tuning(cap, 64)
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
    b.init_particles(s, xnb.PREC_MIXED)
    return b, s


# list slots of about 140 and 40 entries; stages of 1,024 and 96 candidates
@pytest.mark.parametrize("settings", [((1.0, 640), (0.2, 640)), ((0.84, 1024), (0.84, 96))], ids=["lists", "stages"])
def test_steps(settings):
    streams = [torch.cuda.Stream() for _ in settings]
    pairs = [batch(rho, cap, st.cuda_stream) for (rho, cap), st in zip(settings, streams)]
    at_once(*[lambda b=b: [b.step(200, xnb.PREC_MIXED, 0) for _ in range(3)] for b, _ in pairs])
    for (rho, cap), (b, s) in zip(settings, pairs):
        b.check_errors()
        one, q = batch(rho, cap, streams[0].cuda_stream)
        one.step(600, xnb.PREC_MIXED, 0)
        one.check_errors()
        assert_bitwise_equal(b.download(s), one.download(q))
        one.close()
        b.close()


def test_snap_forces():
    files = __file__.rsplit("/", 1)[0] + "/golden/snap/%s_Zuo_JPCA2020.snap"
    r = snap.lattice("FCC", 16, 3.48, 0.05, 2)
    made = []
    for element in ("Ni", "Mo"):  # twojmax 8 and 6
        st = torch.cuda.Stream()
        b = xnb.Batch(len(r), 64, 400 * len(r), stream=st.cuda_stream)
        s = b.add_system(ni_deck_params(), r, 0.0 * r, np.arange(len(r), dtype=np.uint64))
        b.init_particles(s, xnb.PREC_FP64)
        pot = snap.Potential(snap.read_lammps(files % element + "param", files % element + "coeff"))
        pot.force(b, s)
        made.append((b, s, pot, b.download(s)))
    at_once(*[lambda b=b, s=s, p=p: [p.force(b, s) for _ in range(30)] for b, s, p, _ in made])
    for b, s, pot, one in made:
        many = b.download(s)
        for k in ("fx", "fy", "fz"):  # atomic sums: equal to rounding
            assert np.abs(many[k] - one[k]).max() <= 1e-10 * np.abs(one[k]).max()
        b.close()
