"""A captured step graph is current only while the batch's systems select the
kernels it holds: a system with its origin off zero gives its place to one of as
many particles and cells whose box exceeds 1024 sigma, whose residuals are not
packed (another mixed force kernel)."""
import ctypes

import numpy as np
import pytest

from exanbody_gb300 import xnb
from helpers import assert_bitwise_equal

pytestmark = pytest.mark.gpu

N, CELL = 480, 2.9


def system(dims, origin):
    """N atoms, one in every third cell."""
    rng = np.random.default_rng(7)
    cell = 3 * np.arange(N)
    ijk = np.stack([cell % dims[0], (cell // dims[0]) % dims[1], cell // (dims[0] * dims[1])], 1)
    r = (ijk + rng.uniform(0.3, 0.7, (N, 3))) * CELL + np.asarray(origin)
    geom = {"origin": origin, "extent": tuple(o + d * CELL for o, d in zip(origin, dims)), "dims": dims,
            "cell_size": CELL}
    return {"r": r, "v": rng.normal(0.0, 1.0, (N, 3)), "id": np.arange(N, dtype=np.uint64), "geom": geom}


def place(b, w):
    s = b.add_system(xnb.lj_params(w["geom"]), w["r"], w["v"], w["id"])
    b.init_particles(s, xnb.PREC_MIXED)
    return s


def test_graph_of_packed_residuals_refuses_a_long_box():
    import torch

    first, second = system((10, 12, 12), (-17.0, 0.0, 0.0)), system((360, 2, 2), (0.0, 0.0, 0.0))
    stream = torch.cuda.Stream()
    b = xnb.Batch(N, 1440, 200 * N)
    b.stream = ctypes.c_void_p(stream.cuda_stream)
    s = place(b, first)
    g = b.graph(5, xnb.PREC_MIXED, 0)
    assert g.current()
    b.remove_system(s)
    s = place(b, second)
    assert not g.current()
    with pytest.raises(xnb.XnbError):
        g.launch()
    g.close()
    # captured again, its steps are those of the same system in a batch of its own
    g = b.graph(5, xnb.PREC_MIXED, 0)
    g.launch()
    b.check_errors()
    alone = xnb.Batch(N, 1440, 200 * N)
    q = place(alone, second)
    alone.step(5, xnb.PREC_MIXED, xnb.STEP_HOST_SYNC)
    assert_bitwise_equal(b.download(s), alone.download(q))
    g.close()
    b.close()
    alone.close()
