"""Representative workloads of the k-mer state path, for timing it.

Each case is one call sequence a program makes through the public entry points
of ``cf1_rs_b200`` on seeded synthetic input (the five workloads of
``csrc/cf1_synth.cpp``, scaled):

  streamed : ``Cf1Gpu.run_streamed`` -- records in page-locked host memory in,
             state words in page-locked host memory out (the one-call form)
  staged   : ``reset_input`` + ``add_records`` + ``run`` + ``states`` from
             ordinary host arrays (the package's quick-start sequence)
  resident : ``run_resident`` + ``states`` on input uploaded beforehand (a
             program that runs several settings over one input)
  query    : ``query`` -- a batch of canonical k-mers against a built index
  noalloc  : ``distinct_kmers_noalloc`` on one device-resident record

All outputs are whole numbers (state words, slots, keys) and compared for
equality, so ``exact`` has nothing to give.
"""
import numpy as np
import torch

import cf1_rs_b200 as cg

FULL_BP = {1: 5e6, 2: 130e6, 3: 200e6, 4: 1e9, 5: 3.1e9}  # bases of a workload at scale 1 (2: about)


def _run(name, how, workload, bp, k=31, bins=128, mode="bbhash", batched=False, short=False):
    return {"name": name, "how": how, "workload": workload, "bp": int(bp), "k": k, "bins": bins, "mode": mode,
            "batched": batched, "short": short}


def listed():
    return [
        # a plasmid or a virus: the smallest call, where launches and waits count
        _run("plasmid_30kb", "streamed", 1, 30_011),
        # one bacterial genome through the quick-start calls
        _run("bacterium_5mb", "staged", 1, 5_000_000),
        # a transcriptome: many short records, exons shared by isoforms, short records tracked
        _run("transcripts_40mb", "streamed", 2, 40_000_003, short=True),
        # a small eukaryote at a shorter k and fewer bins
        _run("genome_20mb_k21", "streamed", 3, 20_000_017, k=21, bins=64),
        # a mid-size repetitive genome, both MPHF forms
        _run("genome_200mb", "resident", 3, 200_000_000),
        _run("genome_200mb_learned", "resident", 3, 200_000_000, mode="learned", batched=True),
        # 128-bit k-mers, both MPHF forms
        _run("genome_100mb_k63", "resident", 4, 100_000_007, k=63),
        _run("genome_150mb_k63_learned", "streamed", 4, 150_000_001, k=63, mode="learned", batched=True),
        # human-like repeat content at 256 bins: device time, and end to end
        _run("human_like_1gb", "resident", 5, 1_000_000_000, bins=256),
        _run("human_like_1gb_streamed", "streamed", 5, 1_000_000_000, bins=256),
        # phase 5 asking for the slots of a batch of k-mers
        {"name": "query_8m", "how": "query", "workload": 3, "bp": 50_000_000, "k": 31, "bins": 128, "mode": "bbhash",
         "queries": 8_000_000},
        # a caller that cannot allocate: one record at the entry point's limit
        {"name": "noalloc_1m", "how": "noalloc", "bp": cg.NOALLOC_MAX_BASES, "k": 31},
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm, odd."""
    return int(lo * (hi / lo) ** rng.random()) | 1


def draw(rng):
    p = rng.random()
    if p < 0.1:
        return {"how": "noalloc", "bp": min(_spread(rng, 1000, cg.NOALLOC_MAX_BASES), cg.NOALLOC_MAX_BASES),
                "k": rng.choice([15, 21, 27, 31])}
    if p < 0.2:
        return {"how": "query", "workload": rng.choice([1, 3, 5]), "bp": _spread(rng, 1e6, 1e8), "k": rng.choice([21, 31]),
                "bins": rng.choice([64, 128, 256]), "mode": rng.choice(["bbhash", "learned"]),
                "queries": _spread(rng, 1e4, 8e6)}
    wide = rng.random() < 0.25
    learned = rng.random() < 0.35
    workload = rng.choice([1, 2, 3, 4, 5])
    top = 150e6 if wide else 300e6 if learned else 1e9
    if workload in (1, 2):
        top = min(top, 100e6)
    if workload == 5 and wide:  # tandem arrays of 128-bit k-mers
        top = 40e6
    c = _run("", rng.choice(["streamed", "staged", "resident"]), workload, _spread(rng, 30e3, top),
             k=rng.choice([33, 45, 55, 63] if wide else [15, 21, 25, 27, 31, 31, 31]), bins=rng.choice([32, 64, 128, 256, 512]),
             mode="learned" if learned else "bbhash", batched=rng.random() < 0.5, short=rng.random() < 0.3)
    if c["k"] == 15:  # 2^29 canonical 15-mers: larger inputs would be almost all repeats
        c["bp"] = min(c["bp"], 100_000_001)
    del c["name"]
    return c


def _synth(case, seed):
    return cg.SynthInput(case["workload"], scale=case["bp"] / FULL_BP[case["workload"]], seed=1 + seed)


def _pinned(a):
    t = torch.empty(max(1, a.nbytes), dtype=torch.uint8, pin_memory=True)
    v = t.numpy()[: a.nbytes].view(a.dtype)
    v[:] = a
    return v, t


def _words(case):
    """Zeroed state words with room for any seed's input (its length varies a
    little with the seed); words past the last one stay zero."""
    return np.zeros(int(case["bp"] * 1.25) // 12 + 4096, np.uint64)


def _context(case):
    return cg.Cf1Gpu(k=case["k"], num_bins=case["bins"], mode=case["mode"], batched=case.get("batched", False),
                     track_short_seqs=case.get("short", False))


def _codes(seq):
    """2-bit codes of ASCII bases (others read as A) on the GPU."""
    table = np.zeros(256, np.uint8)
    for i, b in enumerate(b"ACGT"):
        table[b] = table[b | 32] = i
    return torch.from_numpy(table[seq]).cuda()


def _canonical_at(codes, pos, k):
    fw = torch.zeros_like(pos)
    rc = torch.zeros_like(pos)
    for j in range(k):
        b = codes[pos + j].to(torch.int64)
        fw = (fw << 2) | b
        rc = rc | ((3 - b) << (2 * j))
    return torch.minimum(fw, rc)


def _prepare_query(case, seed):
    x = _synth(case, seed)
    g = _context(case)
    g.add_records(x.seq, x.offsets)
    g.run()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, k = case["queries"], case["k"]
    pos = torch.randint(0, len(x.seq) - k, (n,), generator=gen, device="cuda")
    keys = _canonical_at(_codes(np.asarray(x.seq)), pos, k)
    # one in eight is looked up with other low bits: most of those are absent
    other = torch.randint(0, 8, (n,), generator=gen, device="cuda") == 0
    keys = torch.where(other, keys ^ torch.randint(1, 1 << 20, (n,), generator=gen, device="cuda"), keys)
    return {"how": "query", "ctx": g, "keys": keys.cpu().numpy().view(np.uint64)}


def _prepare_noalloc(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["bp"]
    seq = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[
        torch.randint(0, 4, (n,), generator=gen, device="cuda")]
    if n >= 1000:  # a repeat and a placeholder run, as in a contig
        seq[n // 2: n // 2 + n // 8] = seq[: n // 8]
        seq[n // 3: n // 3 + 100] = ord("N")
    out = torch.zeros(n, dtype=torch.int64, device="cuda")
    return {"how": "noalloc", "seq": seq, "k": case["k"], "out": out,
            "n": torch.zeros(1, dtype=torch.int64, device="cuda")}


def prepare(case, seed):
    if case["how"] == "query":
        return _prepare_query(case, seed)
    if case["how"] == "noalloc":
        return _prepare_noalloc(case, seed)
    x = _synth(case, seed)
    g = _context(case)
    s = {"how": case["how"], "ctx": g, "off": np.array(x.offsets, np.uint64)}
    if case["how"] == "staged":
        s["seq"] = np.array(x.seq)
        s["words"] = _words(case)
    elif case["how"] == "streamed":
        s["seq"], s["keep_seq"] = _pinned(np.asarray(x.seq))
        s["words"], s["keep_words"] = _pinned(_words(case))
    else:
        seq, keep = _pinned(np.asarray(x.seq))
        g.add_records(seq, s["off"])
        g.upload()
        s["words"], s["keep_words"] = _pinned(_words(case))
    return s


def run(s):
    how = s["how"]
    if how == "noalloc":
        st = cg.distinct_kmers_noalloc(s["seq"].data_ptr(), s["seq"].numel(), s["k"], s["out"].data_ptr(),
                                       s["out"].numel(), s["n"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st != cg.OK:
            raise RuntimeError(f"distinct_kmers_noalloc: status {st}")
        return {"n": s["n"], "keys": s["out"]}
    g = s["ctx"]
    if how == "query":
        return g.query(s["keys"]).view(np.int64)
    if how == "streamed":
        g.run_streamed(s["seq"], s["off"], s["words"])
    elif how == "staged":
        g.reset_input()
        g.add_records(s["seq"], s["off"])
        g.run()
        g.states(s["words"][: (g.total_kmers() + 11) // 12])
    else:
        g.run_resident()
        g.states(s["words"][: (g.total_kmers() + 11) // 12])
    return {"n": g.total_kmers(), "words": s["words"].view(np.int64)}


def work(case):
    if case["how"] == "noalloc":
        return {"bytes": case["bp"] * 9, "flops": 0}
    if case["how"] == "query":
        return {"bytes": case["queries"] * 16, "flops": 0}
    # the bases read once, five bits of state per distinct k-mer written once
    return {"bytes": case["bp"] * (1 + 8 / 12), "flops": 0}


def exact(case, seed):
    return None
