"""The warp-per-cell neighbour build of sparse cells, whose candidates are listed one
by one (up to 256 in the 27 cells, when the stage leaves room for the listing), lists
equal to the oracle's entry for entry: a handful of particles in mostly empty cells,
candidate counts around each whole step of 32 and around the largest, stages that
hold the listing, only part of the candidates or neither, boxes whose every
neighbour cell is an image."""
import numpy as np
import pytest

from exanbody_gb300 import xnb
from helpers import ncells, new_batch, oracle_from
from test_gpu_build_warp import uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n,cap", [
    ((9, 8, 7), 1, 640),       # one particle, its own only candidate
    ((9, 8, 7), 40, 640),      # most cells empty
    ((7, 6, 6), 252, 640),     # ~27 candidates: one step, sometimes two
    ((7, 6, 6), 1200, 640),    # ~128: the loads of four steps, sometimes of a second four
    ((7, 6, 6), 2390, 640),    # ~256: listed one by one, or as runs
    ((7, 6, 6), 2390, 320),    # the smallest stage that holds the largest listing
    ((7, 6, 6), 2390, 288),    # one that does not: listed up to 224
    ((7, 6, 6), 600, 64),      # none: runs, and cells that go on to the block-per-cell build
    ((2, 2, 2), 40, 640),      # ~135 through every image
    ((2, 3, 2), 113, 640),     # ~254 through every image
    ((20, 19, 18), 7000, 640),  # ~1 per cell, a warp per cell
])
def test_lists_equal_the_oracle(dims, n, cap):
    w = uniform(dims, n, n + cap)
    b = new_batch([n], [ncells(w["geom"])], list_per_atom=600.0)
    b.set_tuning(cap, 64)
    b.set_subcell_pruning(False)
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
    b.init_particles(s, xnb.PREC_FP64_EXACT)
    o = oracle_from(w)
    o.init()
    ga, gb, gc = b.pairs(s)
    oa, ob, oc = o.pairs()
    assert np.array_equal(gc, oc) and np.array_equal(ga, oa) and np.array_equal(gb, ob)
    b.close()



def test_lists_built_in_the_rebins_launch():
    """The same build inside the fused rebin (at most 1,024 cells), against the separate kernels."""
    w = uniform((9, 8, 7), 1, 11)
    g = w["geom"]
    rng = np.random.default_rng(4)
    cell = rng.choice(9 * 8 * 7, 400, replace=False)
    ijk = np.stack([cell % 9, (cell // 9) % 8, cell // 72], 1)
    r, v = (ijk + rng.uniform(0.2, 0.8, (400, 3))) * g["cell_size"], rng.normal(0.0, 1.5, (400, 3))
    out = []
    for flags in (0, xnb.STEP_HOST_SYNC):
        b = new_batch([400], [ncells(g)])
        s = b.add_system(xnb.lj_params(g), r, v, np.arange(400, dtype=np.uint64))
        b.init_particles(s, xnb.PREC_MIXED)
        b.step(60, xnb.PREC_MIXED, flags)
        b.check_errors()
        out.append((b.info(s).rebuilds, b.pairs(s)))
        b.close()
    assert out[0][0] == out[1][0] > 0
    assert all(np.array_equal(x, y) for x, y in zip(out[0][1], out[1][1]))
