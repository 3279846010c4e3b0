"""Full-precision forces of short lists, which a warp filters for its eight particles
at once (up to 96 entries together): gases and clusters around each whole step of
32 entries and around 96, empty lists between full ones, systems of different
cutoff and box within one group of eight. FP64_EXACT equals the oracle bit for bit;
FP64 and the half lists agree with it within 1e-12 (|dF_i| / max(|F_i|, F_rms)),
a pair's roundings (2^-53 each, under 100 of them) and a sum of a few dozen terms."""
import numpy as np
import pytest

from exanbody_gb300 import xnb
from helpers import assert_bitwise_equal, forces, ncells, new_batch
from oracle.oracle import OracleSystem

pytestmark = pytest.mark.gpu


def clusters(dims, sizes, cs=3.4, seed=1):
    """Cluster k of sizes[k] atoms ~1.05 apart in cell 2k (every other cell empty): lists of sizes[k] - 1
    entries and, through nearby cells, of their neighbours' atoms."""
    rng = np.random.default_rng(seed)
    r = []
    for k, m in enumerate(sizes):
        c = 2 * k
        corner = np.array([c % dims[0], c // dims[0] % dims[1], c // (dims[0] * dims[1])]) * cs
        q = np.arange(m)
        r.append(corner + 0.6 + np.stack([q % 3, q // 3 % 3, q // 9], 1) * 1.05 + rng.uniform(-0.05, 0.05, (m, 3)))
    r = np.concatenate(r)
    geom = {"origin": (0.0,) * 3, "extent": tuple(d * cs for d in dims), "dims": dims, "cell_size": cs}
    return {"r": r, "v": np.zeros_like(r), "id": np.arange(len(r), dtype=np.uint64), "geom": geom}


CASES = {
    "pairs": [((8, 7, 6), [2, 1, 1, 2, 3, 1] * 28, 2.5)],
    "threes": [((8, 7, 6), [4, 5, 3, 0, 1, 6] * 28, 2.5)],       # ~32 entries per eight
    "mid": [((8, 7, 6), [9, 8, 1, 0, 7, 10] * 28, 2.5)],         # ~64
    "edge": [((8, 7, 6), [12, 13, 14, 1, 11] * 33, 2.5)],        # ~96, on either side of it
    "systems": [((5, 4, 3), [3, 1, 5, 2], 2.5), ((4, 4, 4), [1, 1], 2.9), ((3, 4, 5), [7, 2, 1], 2.2),
                ((2, 3, 3), [1, 2], 3.0), ((4, 3, 5), [6, 1, 1, 2], 2.7)],
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_short_lists(case):
    ws = [(clusters(d, m, seed=k + 1), rc) for k, (d, m, rc) in enumerate(CASES[case])]
    b = new_batch([len(w["r"]) for w, _ in ws], [ncells(w["geom"]) for w, _ in ws], list_per_atom=200.0)
    ss = [b.add_system(xnb.lj_params(w["geom"], rcut=rc), w["r"], w["v"], w["id"]) for w, rc in ws]
    b.init_particles(-1, xnb.PREC_FP64_EXACT)
    exact = [b.download(s) for s in ss]
    for (w, rc), s, G in zip(ws, ss, exact):
        g = w["geom"]
        o = OracleSystem(g["origin"], g["extent"], g["dims"], g["cell_size"], rc, 0.3, 1.0, 1.0, 0.005, kind="omp")
        o.load_flat(w["r"], w["v"], w["id"])
        o.init()
        assert_bitwise_equal(G, o.particles(), fields=("rx", "ry", "rz", "fx", "fy", "fz", "pe"))
    for prec in (xnb.PREC_FP64, xnb.PREC_FP64 | xnb.PREC_NEWTON):
        b.lennard_jones_force(-1, prec, True)
        for s, G in zip(ss, exact):
            F = b.download(s)
            mag = np.linalg.norm(forces(G), axis=1)  # zero throughout where nothing lies within the cutoff
            off = np.linalg.norm(forces(F) - forces(G), axis=1)
            assert (off <= 1e-12 * np.maximum(mag, np.sqrt((mag**2).mean()))).all(), prec
            assert np.abs(F["pe"] - G["pe"]).max() <= 1e-12 * max(np.abs(G["pe"]).max(), 1e-300)
    b.close()
