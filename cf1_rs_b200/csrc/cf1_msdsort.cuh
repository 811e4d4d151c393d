// Phase 3a in MSD form (cf1_msdsort.cu): per-bin multisplit on the top bits,
// shared-memory sort + unique of each sub-bucket.
#pragma once
#include "cf1_internal.cuh"

namespace cf1 {

// What a run of msd_sort_unique reads back, in page-locked memory of the
// caller's.
struct MsdRead {
  uint64_t n_distinct, runs;
  uint32_t overflow;  // units (unsorted) or runs (sorted) left to the block kernel
  uint32_t oversize;  // a sub-bucket fits nowhere
  uint32_t l0_err;    // Level0Out::err
};

struct MsdScratch {
  DevBuf tile_off, hist, scan_tmp, sb_off, sb_off1, cnt, out_off, flag, clist, ccount, coff, runs, ov, ovc;
  // groups the group dedup left: their sub-buckets' offsets, counts and list
  DevBuf sub_off, sub_cnt, jlist;
  uint32_t last_overflow = 0;  // sub-buckets the last unsorted run left to the block kernel
  // The last run's units, 2^unit_bits per bin: what sb_off, cnt and out_off
  // have one entry for.  A unit is a sub-bucket, or a group of sub-buckets
  // (unsorted form, group dedup).
  int unit_bits = 0;
  // Group dedup: the kept keys are the occurrences with a bit in keep, still
  // words of a first pass of kept_packed bits (0: plain keys).
  bool kept_bits = false;
  int kept_packed = 0;
  DevBuf keep;
  cudaEvent_t ev[2] = {nullptr, nullptr};  // around the last dedup kernel launch
  float ms_dedup = 0;                      // its device time
  ~MsdScratch() {
    for (auto e : ev)
      if (e) cudaEventDestroy(e);
  }
};

// Top bits to split on so that the largest bin's sub-buckets hold about a
// third of the shared-memory capacity.
template <class KeyT>
int msd_prefix_bits(uint64_t max_bin_keys, bool sorted);

// keys: n keys segmented by bin (seg_off[0..nbins]); alt: n scratch keys.
// Writes the distinct keys of every bin to dist and their offsets to
// dist_off[0..nbins]: sorted within each bin, or (sorted = false) in
// sub-bucket order with any order inside a sub-bucket.  Returns false
// (nothing written) when a sub-bucket is larger than the shared-memory
// capacity; keys are then clobbered and the caller re-expands and takes the
// LSD path.
// Level 0 of the BBHash form, built by the unsorted (64-bit) dedup: with the
// sub-buckets split on the top P bits of key * KEY_SPREAD_MUL -- level 0's own
// hash -- and every bin's level-0 block a multiple of 2^P words, sub-bucket
// j of bin b owns words [j, j + 1) * (block / 2^P) of it alone, so its CTA
// marks, clears and writes them with no atomics in global memory and lists
// the keys it does not place.
// BBHash levels 0 and 1 built by the unsorted dedup: each sub-bucket j (bin
// b, slice sub) marks its keys in its slice of level 0 (sw0 words), and the
// keys level 0 leaves in its slice of level 1 (sw1 words; level 1 is sliced,
// see BBView); the keys level 1 leaves are listed for level 2.
struct Level0Out {
  ulonglong2 *AR = nullptr;                // level-0 entries (each slice writes all of its); nullptr: off
  const uint64_t *woff = nullptr;          // [nbins + 1] level-0 block offsets (sw0 << P words per bin)
  ulonglong2 *AR1 = nullptr;               // level-1 entries (each slice writes all of its)
  const uint64_t *woff1 = nullptr;         // [nbins + 1] level-1 block offsets (sw1 << P words per bin)
  uint64_t *surv = nullptr;                // keys level 1 leaves: bin b's from surv_off[b]
  const uint64_t *surv_off = nullptr;      // [nbins + 1]; bin b's room is surv_off[b+1] - surv_off[b]
  unsigned long long *surv_cnt = nullptr;  // [nbins], zeroed
  uint32_t *err = nullptr;                 // set when a slice or a bin's room is too small
  // Each slice's entries are written as {placed bits, placed bits of the
  // slice before the word}; placed[j] / placed1[j] = the keys level 0 / 1
  // places in sub-bucket j, from which the build turns the entries' ranks
  // into level-wide ones.
  uint32_t *placed = nullptr;   // [nsub]
  uint32_t *placed1 = nullptr;  // [nsub]
  // Joined side sets (payload bytes beside the keys): a key level 0 places
  // gets local rank r inside its slice (the set bits before its bit), and
  // its byte goes to l0pay[sub-bucket start + r]; a key level 1 places, rank
  // r1 in its level-1 slice, to l0pay[sub-bucket start + placed[j] + r1]; a
  // key level 1 leaves takes its byte along to surv_pay.
  bool with_pay = false;
  uint8_t *l0pay = nullptr;    // filled by msd_sort_unique: the payload buffer the kept bytes are not in
  uint8_t *surv_pay = nullptr; // beside surv
  // The same per unit: uplaced[q] / uplaced1[q] keys (the arrays above when a
  // unit is a sub-bucket).  A group's bytes lie at its start: level 0's of
  // all its sub-buckets in order, then level 1's.
  uint32_t *uplaced = nullptr, *uplaced1 = nullptr;  // [units]
};

// How much the keys of the unsorted 64-bit form repeat, from a few bins, added
// to got (device, zeroed; it stays so for inputs not worth a look): keys looked
// at, bits they set, keys that share theirs.  And from those, on the host,
// whether an eighth of the keys (offsets seg_off) and more lie in bins where the
// group dedup's lists overflow on a split of P bits: their mean and 1.5 standard
// deviations do, the keys' copies coming together.
constexpr uint32_t REPEATS = 3;
void msd_look_for_repeats(const uint64_t *keys, uint64_t n, const uint64_t *seg_off, uint32_t nbins, uint64_t *got,
                          MsdScratch &sc, cudaStream_t s);
bool msd_lists_overflow(const uint64_t *seg_off, uint32_t nbins, int P, const uint64_t *got);

// max_bin: the keys of the largest bin.
// With dist = nullptr the distinct keys stay where the dedup left them, at
// the start of each unit's range of *kept (keys or alt), and
// msd_compact writes dist later; dist_off is written either way.
// With pkeys/palt (one side-set code per key, beside keys and alt), each
// distinct key leaves with the OR of its copies' side-set bytes at the same place
// of *kept_pay (pkeys or palt, beside *kept); the group dedup leaves no bytes
// there (*kept_pay = nullptr: they went to l0's outputs).  groups = false:
// the unsorted 64-bit form goes without the group dedup.
template <class KeyT>
bool msd_sort_unique(KeyT *keys, KeyT *alt, uint64_t n, uint64_t max_bin, const uint64_t *seg_off, uint32_t nbins,
                     int key_bits, int P, KeyT *dist, uint64_t *dist_off, MsdScratch &sc, MsdRead &rd,
                     cudaStream_t s, bool sorted = true, const Level0Out *l0 = nullptr, KeyT **kept = nullptr, uint8_t *pkeys = nullptr,
                     uint8_t *palt = nullptr, uint8_t **kept_pay = nullptr, uint8_t **l0pay_buf = nullptr, bool groups = true);

// The deferred copy: distinct keys of the last msd_sort_unique (nunit
// units, left in `kept`) to dist, bins in order.
template <class KeyT>
void msd_compact(const KeyT *kept, uint64_t nunit, KeyT *dist, MsdScratch &sc, cudaStream_t s);

}  // namespace cf1
