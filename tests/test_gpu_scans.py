"""The prefix sums over super k-mer records (64-item rows of a warp, 4096-item
blocks, sums of blocks) at their edges, against the CPU oracle's states and
counts.  Whole numbers: equality."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 255, 257, 4095, 4096, 4097, 8191, 8193, 20_001])
def test_record_prefix_edges(n):
    """n records of one k-mer each: n super k-mers."""
    rows = np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(n).integers(0, 4, (n, 31))]
    seq, off = o.concat_records([r.tobytes() for r in rows])
    g, _ = assert_parity(seq, off, 31, num_bins=4)
    assert g.stats()["n_superkmers"] == n
    g.close()
