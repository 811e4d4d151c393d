"""Runs of the rank dedup (cf1_msdsort.cu) at the sizes where their plan, the
copy and the placement change over, against the CPU oracle.  One bin: splits
of up to 10 bits are one stretch of the plan, wider ones several; from 2^22
sub-buckets on a warp takes 32 of them.  Whole numbers: equality."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _random(n, seed):
    return ACGT[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


NO_MSD = 2**64 - 1


# sub-buckets aim at 1024 keys (sorted, 64 bits), 512 (128 bits), 1536 (128 bits by hash)
@pytest.mark.parametrize("arrays", [False, True])
@pytest.mark.parametrize("k,mode,n_bases,bits", [
    (31, "learned", 1_000_000, 10), (31, "learned", 2_000_000, 11), (31, "learned", 5_000_000, 13),
    (63, "learned", 500_000, 10), (63, "learned", 1_000_000, 11), (63, "bbhash", 1_500_000, 10),
    (63, "bbhash", 3_000_000, 11)])
def test_stretches(k, mode, n_bases, bits, arrays):
    """With arrays, 29,000 copies of a k-mer beside the runs: 64-bit ones go to
    the block kernel, 128-bit ones (more than it holds) send the run to the LSD
    sort."""
    recs = [_random(n_bases - 30_000, n_bases)]
    recs += [b"T" * 12 + b"A" * 29_000, b"TTTTTTTG" * 100] if arrays else [_random(29_900, 1)]
    seq, off = o.concat_records(recs)
    g, _ = assert_parity(seq, off, k, mode=mode, num_bins=1)
    assert g.stats()["sort_msd_bits"] == (NO_MSD if arrays and k == 63 else bits)
    g.close()


def _least_mer(seed):
    """A 15-mer of very small order value (mix_order)."""
    cand = np.random.default_rng(seed).integers(0, 1 << 30, 400_000).astype(np.uint64)
    rc, y = np.zeros_like(cand), cand.copy()
    for _ in range(15):
        rc = (rc << np.uint64(2)) | (np.uint64(3) - (y & np.uint64(3)))
        y >>= np.uint64(2)
    c = np.minimum(cand, rc)
    x = c.copy()
    for sh, mul in ((16, 0x7FEB352D), (15, 0x846CA68B), (16, 1)):
        x ^= x >> np.uint64(sh)
        x = (x * np.uint64(mul)) & np.uint64(0xFFFFFFFF)
    best = int(c[np.argmin(x)])
    return np.frombuffer(bytes(b"ACGT"[(best >> (2 * (14 - i))) & 3] for i in range(15)), np.uint8)


@pytest.mark.parametrize("k,mode,n", [(31, "learned", 1_150_000), (63, "learned", 600_000), (63, "bbhash", 1_700_000)])
def test_four_million_sub_buckets(k, mode, n):
    """One of 4096 bins holds the k-mers with a 15-mer of small order value in
    their middle (random bases before it, so the sorted split spreads them);
    all bins are split as wide as it needs, and most sub-buckets are empty."""
    recs = ACGT[np.random.default_rng(k).integers(0, 4, (n, k))]
    recs[:, (k - 15) // 2 : (k + 15) // 2] = _least_mer(5)
    seq = np.concatenate([recs.reshape(-1), np.frombuffer(_random(300_000, 3), np.uint8)])
    off = np.append(np.arange(n + 1, dtype=np.uint64) * np.uint64(k), np.uint64(len(seq)))
    g, _ = assert_parity(seq, off, k, mode=mode, num_bins=4096)
    bits = g.stats()["sort_msd_bits"]
    assert bits <= 16 and 4096 << bits >= 1 << 22
    g.close()
