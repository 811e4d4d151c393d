"""Group dedup and sequence that repeats, against the CPU oracle.  Whole
numbers: equality.

Tandem arrays: a group holds thousands of copies of a key, overflows, and is
split by warps."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _random(n, seed):
    return ACGT[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


@pytest.mark.parametrize("unit", [1, 2, 31, 37, 1_000])
def test_tandem_arrays(unit):
    s = _random(unit, unit)
    seq, off = o.concat_records([(s * (600_000 // unit + 1))[:600_001], _random(50_000, 1)])
    g, _ = assert_parity(seq, off, 31, num_bins=4)
    assert g.stats()["dedup_overflow"] > 0
    g.close()
