"""The mixed SNAP kernel where its shared-memory plan changes: every number of
CTAs per SM (twojmax 1 to 9), rounds that hold all neighbours and neighbourhoods
of several rounds, against the FP64 kernel. The files' coefficients keep the mixed
path's 1e-5; drawn ones of one size cancel more in the forces: FP32 rounding
(6e-8) through nine levels and ~10^3 summed terms (x 30), with forces a thirtieth
of their terms, stays below 1e-4."""
import numpy as np
import pytest

from exanbody_gb300 import snap, xnb
from helpers import ncells, new_batch
from test_gpu_snap import block
from test_snap_oracle import potential

pytestmark = pytest.mark.gpu


def drawn(cfg, twojmax):
    count = sum(1 for j1 in range(twojmax + 1) for j2 in range(j1 + 1)
                for j in range(j1 - j2, min(twojmax, j1 + j2) + 1, 2) if j >= j1)
    c = np.random.default_rng(twojmax).normal(0.0, 0.01, count + 1)
    return dict(cfg, twojmax=twojmax, ncoeffall=count + 1, elements=[dict(cfg["elements"][0], coeffs=list(c))])


@pytest.mark.parametrize("el,n,a,dims,twojmax", [
    ("Mo", 8, 2.60, 3, None),   # ~46 neighbours: two rounds of 32
    ("Ni", 8, 3.15, 4, None),   # 42 neighbours: two rounds of 21
    ("Mo", 8, 3.15, 4, 1), ("Mo", 8, 3.15, 4, 3), ("Mo", 8, 3.15, 4, 5), ("Mo", 8, 3.15, 4, 7),
    ("Mo", 8, 3.15, 4, 9),      # rounds of 15 of the 26 neighbours
])
def test_mixed_matches_fp64(el, n, a, dims, twojmax):
    cfg = potential(el)
    tol = 1e-5
    if twojmax is not None:
        cfg, tol = drawn(cfg, twojmax), 1e-4
    r, L = block(el, n, a, 9, sigma=0.12)
    ids = np.arange(1, len(r) + 1, dtype=np.uint64)
    geom = {"origin": (0.0, 0.0, 0.0), "extent": (L, L, L), "dims": (dims,) * 3, "cell_size": L / dims}
    b = new_batch([len(r)], [ncells(geom)])
    s = b.add_system(xnb.lj_params(geom, rcut=cfg["rcutfac"], rcut_inc=1.0), r, np.zeros_like(r), ids)
    b.init_particles(s, xnb.PREC_FP64)
    pot = snap.Potential(cfg)
    out = []
    for mixed in (False, True):
        pot.force(b, s, energy=True, mixed=mixed)
        D = b.download(s)
        out.append((np.stack([D[k] for k in ("fx", "fy", "fz")], 1), D["pe"]))
    mag = np.linalg.norm(out[0][0], axis=1)
    rel = np.linalg.norm(out[1][0] - out[0][0], axis=1) / np.maximum(mag, np.sqrt((mag ** 2).mean()))
    assert rel.max() <= tol
    assert np.max(np.abs(out[1][1] - out[0][1])) <= tol * np.max(np.abs(out[0][1]))
    b.close()
