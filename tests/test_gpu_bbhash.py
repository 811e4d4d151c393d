"""BBHash levels built in one launch (bb_tail_kernel): a bijection and the
oracle's states from one key up to its threshold of 16384 keys a bin, past it
(large levels in launches of their own first), and with one bin whose blocks
exceed shared memory.  Whole numbers: equality."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _random(n, seed):
    return ACGT[np.random.default_rng(seed).integers(0, 4, n)].tobytes()


@pytest.mark.parametrize("n_keys", [1, 2, 7, 8, 9, 1_000, 16_384, 16_385, 70_000])
def test_tail_levels_from_level_0(n_keys):
    seq, off = o.concat_records([_random(n_keys + 62, n_keys)])
    g, ref = assert_parity(seq, off, 63, num_bins=1)
    s = g.stats()
    assert s["n_distinct"] == n_keys and s["bbhash_levels"] >= 1
    keys, _ = g.dump_states()
    img = g.export_mphf()
    import cf1_rs_b200 as cg

    assert np.array_equal(np.sort(cg.host_query(img, keys)), np.arange(n_keys, dtype=np.uint64))
    g.close()


def test_one_bin_above_shared_memory():
    """A 15-mer of very small order value every few bases makes it the
    minimizer of every window: one bin holds all ~120k keys, while the 16 bins'
    average is below the threshold; its level-0 block of 15000 words is
    marked in global memory."""
    rng = np.random.default_rng(5)
    cand = rng.integers(0, 1 << 30, 400_000).astype(np.uint64)

    def rc(x):
        y = np.zeros_like(x)
        for _ in range(15):
            y = (y << np.uint64(2)) | (np.uint64(3) - (x & np.uint64(3)))
            x = x >> np.uint64(2)
        return y

    c = np.minimum(cand, rc(cand))
    x = c & np.uint64(0xFFFFFFFF)
    for sh, mul in ((16, 0x7FEB352D), (15, 0x846CA68B), (16, None)):
        x ^= x >> np.uint64(sh)
        if mul:
            x = (x * np.uint64(mul)) & np.uint64(0xFFFFFFFF)
    best = int(c[np.argmin(x)])
    mer = bytes(b"ACGT"[(best >> (2 * (14 - i))) & 3] for i in range(15))
    fill = ACGT[rng.integers(0, 4, (120_000 // 45, 30))]
    seq, off = o.concat_records([b"".join(mer + f.tobytes() for f in fill)])
    g, _ = assert_parity(seq, off, 63, num_bins=16)
    assert int(g.bin_distinct_counts().max()) > 100_000
    g.close()
