"""Keys that BBHash level 0 crowds together: thousands of distinct k-mers
whose spread keys share their top five bits, alone in their bin.  Level 0
places few of them, so the levels after it need as much room again as level
0 had.  Whole numbers: equality with the oracle."""
import numpy as np
import pytest

from oracle import oracle as o
from tests.gpu_util import assert_parity

pytestmark = pytest.mark.gpu

K = 31
SPREAD = 0xD6E8FEB86659FD93  # BBHash level 0's multiplier (KEY_SPREAD_MUL)


def crowded(n, seed):
    """n records of one k-mer A...A each (canonical as they are: the reverse
    complement starts with T), the spread key's top five bits 9."""
    rng = np.random.default_rng(seed)
    recs = []
    while len(recs) < n:
        mer = rng.integers(0, 4, (100_000, K))
        mer[:, 0] = mer[:, -1] = 0
        key = np.zeros(len(mer), np.uint64)
        for j in range(K):
            key = (key << np.uint64(2)) | mer[:, j].astype(np.uint64)
        hit = np.nonzero((key * np.uint64(SPREAD)) >> np.uint64(59) == 9)[0]
        recs += [bytes(b"ACGT"[c] for c in mer[i]) for i in hit[: n - len(recs)]]
    return recs


@pytest.mark.parametrize("n,sort_mode", [(4_300, "lsd"), (2_500, "msd"), (40_000, "lsd")])
def test_levels_after_a_crowded_one(n, sort_mode):
    rng = np.random.default_rng(n)
    plain = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 3_000)].tobytes()
    for recs, bins in ((crowded(n, n), 1), (crowded(n, n + 1) + [plain], 64)):
        seq, off = o.concat_records(recs)
        assert_parity(seq, off, K, num_bins=bins, sort_mode=sort_mode)[0].close()


def test_streamed_and_again_with_ordinary_keys():
    """The run repeated inside a streamed call, and the context's next runs."""
    import cf1_rs_b200 as cg

    seq, off = o.concat_records(crowded(2_500, 7))
    rng = np.random.default_rng(8)
    seq2, off2 = o.concat_records([np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, 30_000)].tobytes()])
    with cg.Cf1Gpu(k=K, num_bins=1) as g:
        for s, f in ((seq, off), (seq2, off2), (seq, off)):
            ref = o.run(K, s, f, nthreads=4, method=0)
            words = g.run_streamed(s, f)
            keys, st = g.dump_states()
            order = np.argsort(keys)
            assert np.array_equal(keys[order], ref.keys) and np.array_equal(st[order], ref.states)
            assert np.array_equal(words, g.states())
            g.verify_bijection()
