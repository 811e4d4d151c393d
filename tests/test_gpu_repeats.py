"""Group dedup and sequence that repeats, against the CPU oracle.  Whole
numbers: equality.

Runs of 8 Mi k-mers or more look at how much they repeat first: lists that
would overflow get a split of one bit more, or go without groups at the widest
split.  A group that overflows all the same (tandem arrays) is split by
warps."""
import numpy as np
import pytest

import cf1_rs_b200 as cg
from oracle import oracle as o
from tests.gpu_util import assert_parity, sort_by_key

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


def test_a_shard_looks_at_its_own_bins():
    """Shards 0 and 1 of 2 keep every second of six bins: each looks at one that
    is its own."""
    n = 17_800_000
    unit = _random(n // 2, n)
    seq, off = o.concat_records([unit] * 2)
    ref = o.run(31, seq, off, nthreads=8, method=0)
    keys, states = [], []
    for shard in range(2):
        with cg.Cf1Gpu(k=31, num_bins=6, shard_index=shard, shard_count=2) as g:
            g.add_records(seq, off)
            g.run()
            st = g.stats()
            assert st["sort_msd_bits"] == 15 and st["dedup_overflow"] == 0
            k, s = g.dump_states()
            keys.append(k)
            states.append(s)
    k, s = sort_by_key(np.concatenate(keys), np.concatenate(states))
    assert np.array_equal(k, ref.keys) and np.array_equal(s, ref.states)
