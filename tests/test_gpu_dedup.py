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
