"""The ends of super k-mer records (whether a base precedes the first k-mer and
one follows the last), which the minimizer scan writes into them."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity
from tests.inputs import random_records
from tests.test_gpu_sharded import exchange_emulated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 21, 63])
@pytest.mark.parametrize("gap", [1, 40])
def test_ends_at_tile_edges(k, gap):
    """Placeholders on every position around a tile's edges (the scan's tiles
    start at multiples of 2048 k-mer positions; a record's neighbours there are
    looked up, inside a tile they follow from the neighbouring segment)."""
    base = np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(k + gap).integers(0, 4, 6 * 2048)]
    recs = []
    for d in list(range(-3, 4)) + [k - 2, k - 1, k, k + 1]:
        s = base.copy()
        for t in range(1, 6):
            s[t * 2048 + d: t * 2048 + d + gap] = ord("N")
        recs.append(s.tobytes() + b"ACGT" * 512)
    for r in recs:  # alone, so that its positions are the tile positions
        seq, off = o.concat_records([r])
        g, _ = assert_parity(seq, off, k, num_bins=8)
        g.close()


def test_exchanged_records_have_bare_positions():
    """Records on the wire are position << 24 | (n - 1) << 12 | bin."""
    k = 31
    recs = random_records(71, k, n_records=40, max_len=5000)
    seq, off = o.concat_records(recs)
    ctxs, _, routed = exchange_emulated(seq, off, k, 2)
    for g in ctxs:
        g.close()
    for rec, _ in routed:
        r = np.asarray(rec).view(np.uint64)
        pos, n = r >> np.uint64(24), ((r >> np.uint64(12)) & np.uint64(0xFFF)) + np.uint64(1)
        assert np.all(pos + n + np.uint64(k - 1) <= np.uint64(len(seq) + len(recs)))
