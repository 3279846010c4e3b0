"""The fused rebin (asynchronous steps of batches up to 100,000 particles and
16,384 cells) against the separate kernels of the host-synchronised schedule,
bit for bit: far more cells than one scan pass holds, mostly empty; dense cells
with a sub-grid; many systems of one batch rebuilding at different steps."""
import numpy as np
import pytest

from exanbody_gb300 import workloads, xnb
from helpers import assert_bitwise_equal, ncells, new_batch

pytestmark = pytest.mark.gpu


def gas(dims, n, seed):
    """n atoms of a hot gas on distinct sites, ~0.1 per cell of 2.9 sigma."""
    rng = np.random.default_rng(seed)
    cs = 2.9
    sites = rng.choice(dims**3, n, replace=False)
    ijk = np.stack([sites % dims, (sites // dims) % dims, sites // dims**2], 1)
    r = (ijk + 0.5 + rng.uniform(-0.3, 0.3, (n, 3))) * cs
    geom = {"origin": (0.0,) * 3, "extent": (dims * cs,) * 3, "dims": (dims,) * 3, "cell_size": cs}
    return {"r": r, "v": rng.normal(0.0, 3.0, (n, 3)), "id": np.arange(n, dtype=np.uint64), "geom": geom,
            "n_atoms": n}


def many():
    return [workloads.lj_fcc_system(2 + k % 4 + 2, 0.75 + 0.01 * k, 0.7 + 0.05 * k, k) for k in range(20)]


@pytest.mark.parametrize("systems,cap", [
    (lambda: [gas(25, 1500, 3)], 640),                              # 15,625 cells: eight scan passes
    (lambda: [workloads.lj_fcc_system(12, cell_factor=2.0)], 640),  # ~190 atoms per cell, sub-grid side 3
    (many, 640),                                                    # lists built by the same launch
    (many, 192),                                                    # and part of them block per cell
], ids=["gas", "dense", "many", "many_wide"])
@pytest.mark.parametrize("precision", [xnb.PREC_FP64_EXACT, xnb.PREC_MIXED])
def test_fused_rebin_equals_the_separate_kernels(systems, cap, precision):
    out = []
    for flags in (0, xnb.STEP_HOST_SYNC):
        ws = systems()
        b = new_batch([w["n_atoms"] for w in ws], [ncells(w["geom"]) for w in ws], max_systems=len(ws))
        b.set_tuning(cap, 64)
        ss = [b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"]) for w in ws]
        b.init_particles(-1, precision)
        b.step(40, precision, flags)
        b.check_errors()
        out.append([(b.download(s), b.info(s).rebuilds, b.pairs(s)) for s in ss])
        b.close()
    for (f, rf, pf), (h, rh, ph) in zip(*out):
        assert rf == rh > 0
        assert_bitwise_equal(f, h)
        assert all(np.array_equal(x, y) for x, y in zip(pf, ph))
