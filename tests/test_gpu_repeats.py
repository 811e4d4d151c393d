"""Group dedup and sequence that repeats, against the CPU oracle.  Whole
numbers: equality.

Runs of 8 Mi k-mers or more look at how much they repeat first: lists that
would overflow get a split of one bit more, or go without groups at the widest
split.  A group that overflows all the same (tandem arrays) is split by
warps."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _random(n, seed):
    return ACGT[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


# 9.4 and 12.2 M k-mers a bin, 2^16 sub-buckets of ~143 and ~187: groups of 32, lists of 184 a sub-bucket;
# ~3 M a bin, 2^14 sub-buckets of ~181: groups of 16, lists of 176
@pytest.mark.parametrize("n_bases,copies,bins,bits,overflow", [
    (9_400_000, 1, 1, 16, False), (9_400_000, 2, 1, 16, False), (12_200_000, 1, 1, 16, False),
    (12_200_000, 2, 1, 16, False), (12_200_000, 12, 1, 16, False),
    (8_900_000, 1, 3, 14, False), (8_900_000, 2, 3, 15, False), (8_900_000, 20, 3, 15, False),
    (8_300_000, 2, 3, 14, True)])  # too small for a look
def test_lists_of_repeated_sequence(n_bases, copies, bins, bits, overflow):
    unit = _random(n_bases // copies, n_bases + copies)
    seq, off = o.concat_records([unit] * copies)
    g, _ = assert_parity(seq, off, 31, num_bins=bins)
    st = g.stats()
    assert st["sort_msd_bits"] == bits and (st["dedup_overflow"] > 0) == overflow
    g.close()


@pytest.mark.parametrize("unit", [1, 2, 31, 37, 1_000])
def test_tandem_arrays(unit):
    s = _random(unit, unit)
    seq, off = o.concat_records([(s * (600_000 // unit + 1))[:600_001], _random(50_000, 1)])
    g, _ = assert_parity(seq, off, 31, num_bins=4)
    assert g.stats()["dedup_overflow"] > 0
    g.close()
