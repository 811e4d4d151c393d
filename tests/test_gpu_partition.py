"""The device partition (bucket -> bin table) against the oracle's restatement
of the reference's greedy walk (src/minimizer.rs:116-144), on histograms that
lag (buckets above the target), reach the bin cap early, or hold fewer records
than bins.  cf1gpu_xshard_route takes any histogram and tags every record with
its bin, so the records of ~558k super k-mers read the table back bucket by
bucket.  All values are whole numbers: equality."""
import numpy as np
import pytest

import cf1_rs_b200 as cg
from oracle import oracle as o

pytestmark = pytest.mark.gpu

NB = 65536


def _hist(kind: str) -> np.ndarray:
    rng = np.random.default_rng(7)
    h = np.zeros(NB, np.uint32)
    if kind == "even":
        h[:] = 9
    elif kind == "random":
        h = rng.integers(0, 20, NB).astype(np.uint32)
    elif kind == "first":  # one bucket far above the target, then a long lag
        h = rng.integers(0, 3, NB).astype(np.uint32)
        h[0] = 500_000
    elif kind == "last":
        h[NB - 1] = 123_457
    elif kind == "spikes":  # heavy buckets in every part of the walk, lags that overlap
        h = rng.integers(0, 12, NB).astype(np.uint32)
        h[rng.integers(0, NB, 300)] = rng.integers(1000, 200_000, 300)
    elif kind == "few":  # fewer records than most bin counts: target 0 or 1
        h[rng.integers(0, NB, 100)] = 1
    elif kind == "wide":  # a total above 2^32
        h = rng.integers(0, 300_000, NB).astype(np.uint32)
        h[5000:5040] = 4_000_000_000
    return h


@pytest.mark.parametrize("bins", [1, 7, 128, 4096])
def test_partition_matches_the_greedy_walk(bins):
    x = cg.SynthInput(1)
    k, tile = 31, 2048
    seq = np.concatenate([np.asarray(x.seq), np.frombuffer(b"N", np.uint8)])
    pos, _, bucket = o.superkmers(seq, k, tile)
    bucket_at = np.zeros(len(seq), np.int64)
    bucket_at[pos.astype(np.int64)] = bucket
    g = cg.Cf1Gpu(k=k, num_bins=bins, sk_tile=tile)
    g.add_records(x.seq, x.offsets)
    try:
        for kind in ("even", "random", "first", "last", "spikes", "few", "wide", "zero"):
            h = _hist(kind)
            lut, _ = o.partition(h, bins)
            _, n = g.xshard_scan()
            rec, _ = g.xshard_route(h, n)
            b = bucket_at[(rec >> np.uint64(24)).astype(np.int64)]
            assert np.unique(b).size > NB - 200  # nearly every bucket is read back
            assert np.array_equal((rec & np.uint64(0xFFF)).astype(np.uint16), lut[b]), kind
    finally:
        g.close()
