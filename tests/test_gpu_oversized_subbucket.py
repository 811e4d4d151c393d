"""A sub-bucket no dedup kernel holds: more distinct k-mers than the block
kernel's hash set and piece take, all with one split prefix and the same low
ten key bits.  The run falls back to the LSD sort.  A context that ran before
holds the placed counts of that run's slices; the fallback must not read
them.  Whole numbers: equality."""
import numpy as np
import pytest

from cf1_rs_b200 import Cf1Gpu
from oracle import oracle as o
from tests.gpu_util import sort_by_key

K = 31
SPREAD = 0xD6E8FEB86659FD93  # the split's multiplier (KEY_SPREAD_MUL)
NO_MSD = 2**64 - 1
CODE = {b: i for i, b in enumerate(b"ACGT")}


def _one_subbucket(n, seed):
    """n records of one k-mer each, A...CATGA: canonical as they are (the
    reverse complement starts with T), low ten bits CATGA's, and the top five
    bits of the spread key 9 -- one of the 32 sub-buckets such a bin has."""
    rng = np.random.default_rng(seed)
    recs = {}
    while len(recs) < n:
        mid = rng.integers(0, 4, (100_000, K - 6))
        key = np.zeros(len(mid), np.uint64)
        for j in range(K - 6):
            key = (key << np.uint64(2)) | mid[:, j].astype(np.uint64)
        for b in b"CATGA":
            key = (key << np.uint64(2)) | np.uint64(CODE[b])
        hit = np.nonzero((key * np.uint64(SPREAD)) >> np.uint64(59) == 9)[0]
        for i in hit[: n - len(recs)]:
            recs[int(key[i])] = b"A" + bytes(b"ACGT"[c] for c in mid[i]) + b"CATGA"
    return list(recs.values())


def _check(g, seq, off):
    ref = o.run(K, seq, off, nthreads=4, method=0)
    g.reset_input()
    g.add_records(seq, off)
    g.run()
    keys, st = sort_by_key(*g.dump_states())
    assert np.array_equal(keys, ref.keys) and np.array_equal(st, ref.states)
    g.verify_bijection()


def test_crafted_records_share_split_and_low_bits():
    recs = _one_subbucket(4300, 1)
    seq, off = o.concat_records(recs)
    ref = o.run(K, seq, off, nthreads=4, method=0)
    assert len(ref.keys) == 4300 and len(set(int(k) & 1023 for k in ref.keys)) == 1
    assert len(set((int(k) * SPREAD % 2**64) >> 59 for k in ref.keys)) == 1


@pytest.mark.gpu
def test_oversized_subbucket_after_another_run():
    rng = np.random.default_rng(2)
    plain = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 150_000)].tobytes()
    g = Cf1Gpu(k=K, num_bins=1, mode="bbhash")
    try:
        _check(g, *o.concat_records([plain]))
        assert g.stats()["sort_msd_bits"] != NO_MSD
        for n in (4300, 5800):
            _check(g, *o.concat_records(_one_subbucket(n, n)))
            assert g.stats()["sort_msd_bits"] == NO_MSD  # the LSD sort took the run
        _check(g, *o.concat_records([plain[:6_000]]))
        assert g.stats()["sort_msd_bits"] != NO_MSD
    finally:
        g.close()
