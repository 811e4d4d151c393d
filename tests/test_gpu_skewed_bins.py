"""BBHash's last levels when one bin holds nearly all keys: below 65536 keys
its CTA walks them in the one launch, above that the large levels get
launches of their own, the whole device on each.  Whole numbers: equality
with the oracle."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


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
    return bytes(b"ACGT"[(best >> (2 * (14 - i))) & 3] for i in range(15))


def _skewed(n, gap, seed):
    """The 15-mer every 15 + gap bases: it is the minimizer of every window
    that holds it whole, so those windows share a bin."""
    fill = ACGT[np.random.default_rng(seed).integers(0, 4, (n // (15 + gap), gap))]
    mer = _least_mer(5)
    return b"".join(mer + f.tobytes() for f in fill)


# k = 63: BBHash starts with all keys of the bin, nearly all of the input;
# k = 31: with the ~1% that levels 0 and 1 leave of 17 in 30
@pytest.mark.parametrize("k,gap,share,sizes", [(63, 30, 0.95, (60_000, 71_000)),
                                               (31, 15, 0.55, (11_250_000, 12_200_000))])
def test_largest_bin_decides(k, gap, share, sizes):
    launches = []
    for n in sizes:
        seq, off = o.concat_records([_skewed(n, gap, n)])
        g, _ = assert_parity(seq, off, k, num_bins=512)
        assert int(g.bin_distinct_counts().max()) > share * n
        launches.append(g.stats()["n_kernel_launches"])
        g.close()
    assert launches[1] >= launches[0] + 4
