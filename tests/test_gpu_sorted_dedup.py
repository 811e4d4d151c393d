"""Phase-3 dedup of the sorted form (learned index, 128-bit keys) at the edges
of its rank kernel, against the CPU oracle: no split, runs at its capacity
(4096 64-bit or 2048 128-bit keys), many copies of a key, and more than 48
different keys on one position (left to the block kernel).  Whole numbers:
equality, and in the learned form every bin's keys must ascend."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _random(n, seed):
    return ACGT[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


def _check(recs, k, **kw):
    seq, off = o.concat_records(recs)
    g, _ = assert_parity(seq, off, k, mode="learned", **kw)
    keys, _ = g.dump_states()
    if keys.ndim == 1:
        steps = keys[1:] > keys[:-1]
    else:
        steps = (keys[1:, 1] > keys[:-1, 1]) | ((keys[1:, 1] == keys[:-1, 1]) & (keys[1:, 0] > keys[:-1, 0]))
    starts = np.cumsum(g.bin_distinct_counts()).astype(np.int64)[:-1] - 1
    inside = np.ones(len(steps), bool)
    inside[starts[(starts >= 0) & (starts < len(steps))]] = False
    assert steps[inside].all()
    g.close()


@pytest.mark.parametrize("k", [7, 31, 33, 63])
@pytest.mark.parametrize("n_keys", [1, 2, 512, 513, 1024, 1025, 2048, 2049, 4096, 4097, 40_000, 300_000])
def test_run_sizes(k, n_keys):
    _check([_random(n_keys + k - 1, n_keys + k)], k, num_bins=1)


@pytest.mark.parametrize("k", [31, 63])
def test_copies_and_close_keys(k):
    rng = np.random.default_rng(k)
    base = _random(20_000, 1)
    rc = base.translate(bytes.maketrans(b"ACGT", b"TGCA"))[::-1]
    many = [base, rc, base[:7_000]] + [base[3_000:5_000]] * 60 + [b"A" * 3_000, b"AG" * 1_500]
    _check(many, k, num_bins=1)
    _check(many, k, num_bins=7, batched=True)
    # records that begin alike: hundreds of keys within one position
    head = b"AACCAGATTACAAACC"
    close = [head + ACGT[rng.integers(0, 4, k - len(head))].tobytes() for _ in range(700)]
    _check(close + [base], k, num_bins=1)
    _check(close + [base], k, num_bins=1, state_update="sideset")


@pytest.mark.parametrize("mode,k", [("learned", 31), ("learned", 63), ("bbhash", 63)])
@pytest.mark.parametrize("copies", [3, 40, 700])
def test_tandem_array(mode, k, copies):
    """A 171-base unit repeated, every copy with one substitution: positions
    with up to hundreds of copies of their first key, and other keys beside."""
    rng = np.random.default_rng(copies + k)
    unit = rng.integers(0, 4, 171)
    rows = np.tile(unit, (copies, 1))
    rows[np.arange(copies), rng.integers(0, 171, copies)] = rng.integers(0, 4, copies)
    seq, off = o.concat_records([np.frombuffer(b"ACGT", np.uint8)[rows.ravel()].tobytes(),
                                 np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 20_000)].tobytes()])
    g, _ = assert_parity(seq, off, k, mode=mode, num_bins=2)
    g.close()
