"""Phase-3 dedup of the BBHash form at the sizes where its kernels change
over, against the CPU oracle.  All values are whole numbers: equality."""
import numpy as np
import pytest

import cf1_rs_b200 as cg
from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu


def _random(n, seed):
    return np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


def _narrow_split(tmp_path, n_bases):
    """A tuner line that sets the split one bit below the default."""
    size_class = (n_bases + 1).bit_length() - 1  # floor(log2) of the input with its record separator
    cache = tmp_path / "tuner.txt"
    cache.write_text(f"cf1tune 1 wide=0 sorted=0 batched=0 size={size_class} sk_tile=2048 msd_delta=-1 "
                     "p1_ms=1.000 p3_ms=1.000\n")
    return str(cache)


@pytest.mark.parametrize("update", ["sideset", "cas"])
def test_block_kernel_without_payload_bytes(tmp_path, update):
    """States formed in phase 4: the dedup carries no bytes, and sub-buckets
    of ~383 distinct keys go to the block kernel, whose level-0 ranks still
    need their part of its shared memory."""
    n = 24_540
    seq, off = o.concat_records([_random(n, n)])
    g, _ = assert_parity(seq, off, 31, num_bins=1, state_update=update, tuner_cache=_narrow_split(tmp_path, n))
    assert g.stats()["dedup_overflow"] > 0
    g.close()


@pytest.mark.parametrize("k", [31, 15])
@pytest.mark.parametrize("n_bases", [31, 222, 224, 6_170, 6_180, 120_000, 200_000, 3_200_001])
def test_group_dedup_split_widths(k, n_bases):
    """One bin of random sequence: no split and one sub-bucket (up to 192
    k-mers), a group that is the whole bin (up to 32 sub-buckets), one more
    sub-bucket bit, splits of 5 bits (keys and bytes) and 6 bits (packed
    words) above the groups, and a two-pass split."""
    seq, off = o.concat_records([_random(n_bases, n_bases + k)])
    assert_parity(seq, off, k, num_bins=1)[0].close()


@pytest.mark.parametrize("update", ["phase3", "sideset"])
@pytest.mark.parametrize("n_random", [100, 150_000, 400_000])
def test_groups_left_to_the_block_kernel(n_random, update):
    """Tandem arrays and homopolymers put thousands of copies of a k-mer in a
    group: it passes the group dedup's capacity and goes to the block kernel,
    beside groups that do not."""
    s = _random(n_random, n_random)
    recs = [s, b"A" * 20_000, b"AC" * 9_000, b"ACGTTGC" * 3_000, s[: n_random // 3] * 2, _random(40, 1) * 400]
    seq, off = o.concat_records(recs)
    g, _ = assert_parity(seq, off, 31, num_bins=3, state_update=update)
    assert g.stats()["dedup_overflow"] > 0
    g.close()


def test_repeated_keys_within_a_group():
    """Every k-mer twice to forty times, in both strands: most level-0 bits
    are set more than once by copies of one key."""
    base = _random(30_000, 3)
    rc = base.translate(bytes.maketrans(b"ACGT", b"TGCA"))[::-1]
    recs = [base, rc, base[:9_000]] + [base[2_000:4_500]] * 38
    seq, off = o.concat_records(recs)
    for bins in (1, 16, 500):
        assert_parity(seq, off, 31, num_bins=bins)[0].close()


@pytest.mark.parametrize("n_bases,copies", [(3_145_700, 1), (3_145_800, 1), (15_870, 3), (15_600, 3), (1_060_000, 3)])
def test_group_size_change_over(n_bases, copies):
    """Both sides of the split width where groups go from 16 to 32 sub-buckets
    (192 * 2^14 k-mers in a bin), and groups of 16 and 32 whose occurrences,
    three of every key, pass or just fit the list."""
    seq, off = o.concat_records([_random(n_bases, n_bases)] * copies)
    g, _ = assert_parity(seq, off, 31, num_bins=1)
    g.close()
