"""cf1gpu_distinct_kmers_noalloc at the edges of its kernels' tiles (256
positions of the extraction, 2048 keys of the sort) against numpy.  All values
are whole numbers: equality."""
import numpy as np
import pytest

import cf1_rs_b200 as cg

pytestmark = pytest.mark.gpu


def _reference(seq: np.ndarray, k: int) -> np.ndarray:
    n = len(seq) - k + 1
    if n <= 0:
        return np.zeros(0, np.uint64)
    code = np.full(256, 4, np.uint64)
    for i, b in enumerate(b"ACGT"):
        code[b] = code[b | 32] = i
    c = code[seq]
    fw = np.zeros(n, np.uint64)
    rc = np.zeros(n, np.uint64)
    bad = np.zeros(n, bool)
    for j in range(k):
        b = c[j: j + n]
        bad |= b == 4
        fw = (fw << np.uint64(2)) | (b & np.uint64(3))
        rc |= (np.uint64(3) - (b & np.uint64(3))) << np.uint64(2 * j)
    return np.unique(np.minimum(fw, rc)[~bad])


@pytest.mark.parametrize("k", [1, 15, 31])
def test_noalloc_tile_edges(k):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(k)
    for n in (k - 1, k, k + 1, 255, 256, 257, 256 + k - 1, 2048, 2048 + k - 1, 2048 + k, 4097, 100_000,
              cg.NOALLOC_MAX_BASES):
        seq = np.frombuffer(b"ACGTacgt", np.uint8)[rng.integers(0, 8, n)].copy()
        if n > 600:
            seq[rng.integers(0, n, n // 300)] = ord("N")
            seq[n // 2: n // 2 + n // 8] = seq[: n // 8]
        d = torch.from_numpy(seq).cuda() if n else torch.zeros(1, dtype=torch.uint8, device="cuda")
        out = torch.zeros(max(1, n), dtype=torch.int64, device="cuda")
        cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
        st = cg.distinct_kmers_noalloc(d.data_ptr(), n, k, out.data_ptr(), out.numel(), cnt.data_ptr())
        assert st == cg.OK
        torch.cuda.synchronize()
        got = out[: int(cnt.item())].cpu().numpy().view(np.uint64)
        assert np.array_equal(got, _reference(seq, k)), n
