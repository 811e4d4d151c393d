"""The exported MPHF image holds the entries the levels have, each once: no
room between the blocks of the last levels, which are built in one launch with
a region a bin.  Whole numbers: equality."""
import numpy as np
import pytest

import cf1_rs_b200 as cg

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


@pytest.mark.parametrize("k,bins,n", [(31, 128, 30_011), (63, 128, 30_011), (31, 4096, 200_000), (63, 1, 300_000),
                                      (31, 1, 8), (63, 3, 70)])
@pytest.mark.parametrize("mode", ["bbhash", "learned"])
def test_no_room_between_blocks(k, bins, n, mode):
    seq = ACGT[np.random.default_rng(n + k).integers(0, 4, n + k)]
    # (learned, error bound 1: most bins fall back to BBHash)
    with cg.Cf1Gpu(k=k, num_bins=bins, mode=mode, learned_max_err=1 if mode == "learned" else 0) as g:
        g.add_records(seq, np.array([0, len(seq)], np.uint64))
        g.run()
        img = g.export_mphf()
        levels, nbins = int(img.view(np.uint32)[6]), int(img.view(np.uint32)[5])
        meta_off, ar_words = int(img[9]), int(img[11])
        meta = img[meta_off // 8 : meta_off // 8 + 2 * levels * nbins].reshape(-1, 2)
        off, words = meta[:, 0].astype(np.int64), (meta[:, 1] & np.uint64(0xFFFFFFFF)).astype(np.int64)
        off, words = off[words > 0], words[words > 0]
        order = np.argsort(off)
        assert words.sum() == ar_words
        assert np.array_equal(off[order], np.concatenate([[0], np.cumsum(words[order])[:-1]])[: len(words)])
        keys, _ = g.dump_states()
        slots = cg.host_query(img, keys)
        assert np.array_equal(np.sort(slots), np.arange(len(keys), dtype=np.uint64))
        assert np.array_equal(slots, g.query(keys))
