"""The positions' steps (16 bytes per particle, written by every push) belong to the
batches whose forces read them: those with room for 500,000 particles."""
import pytest

from exanbody_gb300 import xnb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def bytes_of(particles):
    free = torch.cuda.mem_get_info()[0]
    b = xnb.Batch(particles, 1000, 1000)
    used = free - torch.cuda.mem_get_info()[0]
    b.close()
    return used


def test_allocated_for_large_batches_only():
    bytes_of(1000)  # the library's own first allocations
    small, large = bytes_of(499999), bytes_of(500000)
    assert large - small >= 500000 * 16  # one particle more, and the array
