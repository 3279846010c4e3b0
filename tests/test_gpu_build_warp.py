"""The warp-per-cell neighbour build at its edges, lists equal to the oracle's
entry for entry: cells of 0 to ~60 random particles (last groups of one to four
particles, more than 32 per cell, runs longer than one step), boxes of two and
three cells per axis (every run wraps around), stages that overflow to the
block-per-cell build, and slots with room for less than one chunk."""
import numpy as np
import pytest

from exanbody_gb300 import xnb
from helpers import ncells, new_batch, oracle_from

pytestmark = pytest.mark.gpu


def uniform(dims, n, seed):
    """n particles at random sites of a fine grid with jitter: none closer than 0.1."""
    rng = np.random.default_rng(seed)
    cs = 2.95
    L = [d * cs for d in dims]
    g = [int(x / 0.3) for x in L]
    sites = rng.choice(g[0] * g[1] * g[2], n, replace=False)
    ijk = np.stack([sites % g[0], (sites // g[0]) % g[1], sites // (g[0] * g[1])], 1)
    r = (ijk + 0.5 + rng.uniform(-0.3, 0.3, (n, 3))) * (np.array(L) / np.array(g))
    geom = {"origin": (0.0,) * 3, "extent": tuple(L), "dims": tuple(dims), "cell_size": cs}
    return {"r": r, "v": np.zeros((n, 3)), "id": np.arange(n, dtype=np.uint64), "geom": geom, "n_atoms": n}


@pytest.mark.parametrize("dims,n,cap,factor", [
    ((4, 5, 6), 400, 640, 1.3),     # ~3 per cell
    ((5, 4, 4), 2500, 640, 1.3),    # ~31 per cell, some above 32
    ((5, 4, 4), 4000, 1024, 1.3),   # ~50 per cell
    ((2, 3, 2), 350, 640, 1.3),     # ~29 per cell, every neighbour cell through an image
    ((6, 6, 6), 4000, 192, 1.3),    # the stage holds part of the neighbourhoods only
    ((16, 16, 17), 30000, 640, 1.0),  # more cells than the warps shared by 2 or 4
    ((6, 6, 6), 4000, 640, 1.0),    # slots sized to the largest count + 16: the last chunks run guarded
])
def test_lists_equal_the_oracle(dims, n, cap, factor):
    w = uniform(dims, n, n + cap)
    b = new_batch([n], [ncells(w["geom"])], list_per_atom=600.0)
    b.set_tuning(cap, 64)
    b.set_subcell_pruning(False)
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"], list_factor=factor)
    b.init_particles(s, xnb.PREC_FP64_EXACT)
    o = oracle_from(w)
    o.init()
    ga, gb, gc = b.pairs(s)
    oa, ob, oc = o.pairs()
    assert np.array_equal(gc, oc) and np.array_equal(ga, oa) and np.array_equal(gb, ob)
    for prec in (xnb.PREC_FP64, xnb.PREC_FP64 | xnb.PREC_NEWTON):  # the lower halves
        b.lennard_jones_force(s, prec, False)
        f = b.download(s)
        if prec == xnb.PREC_FP64:
            full = f
    for k in ("fx", "fy", "fz"):
        scale = np.abs(full[k]).max()
        assert np.allclose(f[k], full[k], rtol=1e-9, atol=1e-12 * scale)
    b.close()
