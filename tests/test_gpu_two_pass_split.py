"""Splits of more than 11 bits, which take two passes, in the forms whose
second pass differs, against the CPU oracle: packed words (split on their own
top bits), keys without bytes, and 128-bit keys split by their hash.  One bin
of random sequence.  Whole numbers: equality."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu


def _random(n, seed):
    return np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


@pytest.mark.parametrize("update", ["phase3", "sideset"])
def test_subbuckets_left_to_the_block_kernel(tmp_path, update):
    """One bit below the default 13: passes of 6 + 6 bits and ~383 distinct
    keys a sub-bucket, about half of which pass the warp dedup's 384."""
    n = 1_570_000
    seq, off = o.concat_records([_random(n, n)])
    size_class = (n + 1).bit_length() - 1  # floor(log2) of the input with its record separator
    cache = tmp_path / "tuner.txt"
    cache.write_text(f"cf1tune 1 wide=0 sorted=0 batched=0 size={size_class} sk_tile=2048 msd_delta=-1 "
                     "p1_ms=1.000 p3_ms=1.000\n")
    g, _ = assert_parity(seq, off, 31, num_bins=1, state_update=update, tuner_cache=str(cache))
    st = g.stats()
    assert st["tuner_state"] == 1 and st["sort_msd_bits"] == 12 and st["dedup_overflow"] > 0
    g.close()


def test_bin_past_the_widest_split():
    """More than 225 * 2^16 k-mers in a bin: the warp dedup at the widest
    split, passes of 8 + 8 bits."""
    n = 14_800_000
    seq, off = o.concat_records([_random(n, n)])
    g, _ = assert_parity(seq, off, 31, num_bins=1)
    assert g.stats()["sort_msd_bits"] == 16
    g.close()


def test_128_bit_keys_by_hash():
    """3.4 M k-mers of 63 bases: 12 bits of the hash, 6 + 6."""
    n = 3_400_000
    seq, off = o.concat_records([_random(n, n)])
    g, _ = assert_parity(seq, off, 63, num_bins=1)
    assert g.stats()["sort_msd_bits"] == 12
    g.close()
