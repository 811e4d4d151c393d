"""Contexts of their own in host threads of their own, on inputs whose runs
launch the same kernels with other amounts of shared memory (other split
widths, bin counts and update modes): every run succeeds, with the states of
the same run alone.  Whole numbers: equality."""
import threading

import numpy as np
import pytest

from cf1_rs_b200 import Cf1Gpu
from oracle import oracle as o

pytestmark = pytest.mark.gpu

ACGT = np.frombuffer(b"ACGT", np.uint8)


def _one_context(seq, off, opts, runs, start, failures):
    try:
        g = Cf1Gpu(k=31, **opts)
        try:
            g.add_records(seq, off)
            g.run()
            want = g.states()
            start.wait()
            for i in range(runs):
                g.run_resident()
                if not np.array_equal(g.states(), want):
                    failures.append(f"{opts}: other states in run {i}")
                    return
        finally:
            g.close()
    except Exception as e:  # noqa: BLE001 -- reported by the test
        failures.append(f"{opts}: {e}")
        start.abort()


@pytest.mark.parametrize("opts", [
    # packed passes of 10, 6, 7 and 8 bits of one bin
    [(2_900_000, dict(num_bins=1)), (150_000, dict(num_bins=1)), (250_000, dict(num_bins=1)), (500_000, dict(num_bins=1))],
    # 4096, 512, 16 and 1 bins
    [(400_000, dict(num_bins=b)) for b in (4096, 512, 16, 1)],
    # the sorted form with and without side sets, whose long runs go to the block kernel
    [(300_000, dict(num_bins=4, mode="learned", state_update=u)) for u in ("phase3", "sideset", "cas")],
], ids=["widths", "bins", "updates"])
def test_contexts_in_threads(opts):
    failures, start = [], threading.Barrier(len(opts))
    threads = []
    for i, (n, kw) in enumerate(opts):
        s = ACGT[np.random.default_rng(i).integers(0, 4, n)].tobytes()
        seq, off = o.concat_records([s, b"ACGTTGC" * 3000] if "mode" in kw else [s])
        threads.append(threading.Thread(target=_one_context, args=(seq, off, kw, 150, start, failures)))
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
