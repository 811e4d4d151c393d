// Phase 3a, MSD form: distinct canonical k-mers per bin, sorted or not.
//
//   1. one or two multisplit passes on the top P bits of the keys (sorted) or
//      of key * KEY_SPREAD_MUL (distinct only, up to 5 bits less), segmented
//      by bin (P chosen so a sub-bucket fits shared memory);
//   2. one CTA per run of sub-buckets keeps one copy of each key: by rank in
//      the run's key range (sorted, sr_dedup_kernel) or by the keys' BBHash
//      bits (distinct only, gd_dedup_kernel); what neither holds goes to one
//      CTA per sub-bucket with a shared-memory hash set, which in the sorted
//      form then counting-sorts on the next 10 bits, insertion-sorts the small
//      buckets (bitonic sort of the whole sub-bucket if any bucket is large);
//      distinct keys stay at the start;
//   3. a scan of the per-sub-bucket counts and a copy into the dense distinct
//      array; a bin's first sub-bucket gives its slot offset.
// A sub-bucket above CAP keys (long homopolymers, huge tandem arrays) makes
// the caller fall back to the LSD path (cf1_phase3_sort.cu) for the run.
#include <cmath>
#include <cstddef>

#include "cf1_device_util.cuh"
#include "cf1_internal.cuh"
#include "cf1_mphf.cuh"
#include "cf1_msdsort.cuh"

namespace cf1 {

namespace {

constexpr int MS_BLOCK = 512;
constexpr int MS_BITS = 11;  // most bits of a pass
// Keys a thread of a multisplit pass holds: 128 bytes of them.
template <class KeyT>
constexpr int ms_items() { return KOps<KeyT>::WORDS == 1 ? 16 : 8; }
template <class KeyT>
constexpr uint32_t ms_tile() { return MS_BLOCK * ms_items<KeyT>(); }
constexpr uint32_t MS_RUN = 8;  // tiles a CTA of the counting kernel takes
constexpr int CS_BLOCK = 512;  // 16 warps: shared memory allows 2 CTAs per SM
constexpr int CS_BITS = 10;
constexpr uint32_t CS_BUCKETS = 1u << CS_BITS;
// Insertion sort up to this many keys per bucket.  Repeats put hundreds of
// copies of one k-mer in a bucket; insertion sort passes over equal keys at
// once, so large buckets of few distinct values stay cheap.
constexpr uint32_t CS_SMALL = 512;
constexpr uint32_t CS_DEDUP_MIN = 64;  // 64-bit sub-buckets above this size are deduplicated first

// Keys a sub-bucket's shared-memory sort holds.  The unsorted (deduplicate
// only) path keeps 64-bit sub-buckets at half that size, so its shared memory
// fits four CTAs per SM instead of two.
constexpr uint32_t cs_cap_for(bool wide, bool sorted) { return wide ? 4096u : (sorted ? 8192u : 4096u); }
template <class KeyT, bool SORTED = true>
constexpr uint32_t cs_cap() { return cs_cap_for(KOps<KeyT>::WORDS == 2, SORTED); }

// Digit of a key in a multisplit pass: bits [shift, shift + width) of the key
// or, when only the distinct keys and not their order are needed (hashed),
// of H * MS_HASH_MUL, H the key's BBHash hash (the key itself for 64-bit
// keys).  The product's top bits spread any key set evenly, where the key's
// own top bits -- the first bases of a canonical k-mer -- are skewed
// several-fold, and they are BBHash level 0's: keys that end up side by side
// have their level-0 bits side by side.
constexpr uint64_t MS_HASH_MUL = KEY_SPREAD_MUL;
template <class KeyT>
CF1_D uint32_t ms_digit(const KeyT &k, int shift, uint32_t mask, bool hashed);
template <>
CF1_D uint32_t ms_digit<uint64_t>(const uint64_t &k, int shift, uint32_t mask, bool hashed) {
  return (uint32_t)((hashed ? k * MS_HASH_MUL : k) >> shift) & mask;
}
template <>
CF1_D uint32_t ms_digit<Key2>(const Key2 &k, int shift, uint32_t mask, bool hashed) {
  if (hashed) return (uint32_t)((bb_key_hash(k) * MS_HASH_MUL) >> shift) & mask;
  return KOps<Key2>::digit(k, shift, mask);
}


// ---------------------------------------------------------------- multisplit pass
// One pass splits every segment on a digit of up to 11 bits:
//   ms_hist_kernel    counts the segments' digits (a CTA takes MS_RUN tiles,
//                     in shared memory, and adds its counts to the totals);
//   a scan of the totals, which gives the sub-segments' offsets;
//   ms_scatter_kernel moves the tiles.
// Up to 11 bits in one pass because a pass is bound by its traffic: a tile of
// 8192 keys still gives 1024 digits runs of 64 bytes, whose partial sectors L2
// merges.  (1 Gbp, 10 bits: passes of 6 and 4 bits 4.63 + 3.95 ms and their
// counts 1.18 + 1.15, one pass 5.71 and 1.13; 100 Mbp of 128-bit keys, 9 bits:
// 2.72 and 0.51, now 1.40 and 0.25.)

// Segment and stretch [start, end) of run t: tiles of `tile` keys, MS_RUN at a
// time (tile_off counts tiles; a run never crosses a segment's edge).
template <class KeyT>
__global__ void __launch_bounds__(MS_BLOCK) ms_hist_kernel(const KeyT *keys, const uint64_t *seg_off,
                                                           const uint32_t *run_off, uint32_t nseg, int shift, int bits,
                                                           bool hashed, uint32_t *tot) {
  extern __shared__ uint32_t ms_h[];  // [1 << bits]
  const uint32_t t = blockIdx.x, dig = 1u << bits;
  if (t >= run_off[nseg]) return;
  for (uint32_t d = threadIdx.x; d < dig; d += MS_BLOCK) ms_h[d] = 0;
  __syncthreads();
  const TileSpan sp = tile_span(seg_off, run_off, nseg, t, ms_tile<KeyT>() * MS_RUN);
#pragma unroll 4
  for (uint64_t i = sp.start + threadIdx.x; i < sp.end; i += MS_BLOCK)
    atomicAdd(&ms_h[ms_digit(keys[i], shift, dig - 1, hashed)], 1u);
  __syncthreads();
  uint32_t *g = tot + ((uint64_t)sp.seg << bits);
  for (uint32_t d = threadIdx.x; d < dig; d += MS_BLOCK)
    if (ms_h[d]) atomicAdd(&g[d], ms_h[d]);
}

// Multisplit of one tile: every key takes its place among the tile's keys of
// its digit from a shared-memory counter (the order inside a digit does not
// matter: every sub-bucket is sorted or deduplicated whole afterwards), a scan
// of the counters gives tile-local starts, one atomic a digit reserves the
// tile's run in the digit's sub-segment, the tile is staged in shared memory in
// digit order, and the runs are written out with consecutive threads on
// consecutive addresses.  All of a thread's loads are issued before the first
// is used, and the keys stay in registers for the staging step.
// With pin/pout, each key's payload (its side-set code) moves with it;
// with PACK (pin, no pout; hashed 64-bit keys, pack = the pass's bits) the
// code goes into the key's packed output word (see pay_code).
template <class KeyT, bool PACK>
__global__ void __launch_bounds__(MS_BLOCK, 2) ms_scatter_kernel(const KeyT *in, KeyT *out, const uint64_t *seg_off,
                                                                 const uint32_t *tile_off, uint32_t nseg, int shift,
                                                                 int bits, bool hashed, const uint64_t *sub_off,
                                                                 uint32_t *cursor, const uint8_t *pin, uint8_t *pout,
                                                                 int pack) {
  constexpr int ITEMS = ms_items<KeyT>();
  constexpr uint32_t TILE = ms_tile<KeyT>();
  constexpr uint32_t PER = (1u << MS_BITS) / MS_BLOCK;  // digits a thread scans, at most
  extern __shared__ __align__(16) unsigned char ms_smem[];
  const uint32_t dig = 1u << bits;
  KeyT *stage = reinterpret_cast<KeyT *>(ms_smem);             // [TILE]
  uint64_t *base = reinterpret_cast<uint64_t *>(stage + TILE);  // [dig] out index of a digit's key, less its stage index
  uint32_t *cnt = reinterpret_cast<uint32_t *>(base + dig);     // [dig] counts, then tile-local starts
  uint8_t *pstage = reinterpret_cast<uint8_t *>(cnt + dig);     // [TILE] when pin
  __shared__ uint32_t sm[MS_BLOCK / 32];
  const uint32_t t = blockIdx.x;
  if (t >= tile_off[nseg]) return;
  const TileSpan sp = tile_span(seg_off, tile_off, nseg, t, TILE);
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const uint32_t n = (uint32_t)(sp.end - sp.start), i0 = warp * (ITEMS * 32) + lane;
  KeyT key[ITEMS];
  uint32_t pb[ITEMS / 4];  // payload bytes, four to a register
#pragma unroll
  for (int q = 0; q < ITEMS / 4; q++) pb[q] = 0;
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    const uint32_t li = i0 + r * 32;
    key[r] = li < n ? in[sp.start + li] : KeyT{};
    if (pin && li < n) pb[r >> 2] |= (uint32_t)pin[sp.start + li] << (8 * (r & 3));
  }
  for (uint32_t d = tid; d < dig; d += MS_BLOCK) cnt[d] = 0;
  __syncthreads();
  uint32_t pk[ITEMS];  // rank << MS_BITS | digit
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    if (i0 + r * 32 < n) {
      const uint32_t d = ms_digit(key[r], shift, dig - 1, hashed);
      pk[r] = (atomicAdd(&cnt[d], 1u) << MS_BITS) | d;
    }
  }
  __syncthreads();
  {
    const uint32_t per = dig > MS_BLOCK ? dig / MS_BLOCK : 1u, d0 = tid * per;
    uint32_t c[PER], own = 0;
#pragma unroll
    for (uint32_t i = 0; i < PER; i++) {
      c[i] = i < per && d0 + i < dig ? cnt[d0 + i] : 0u;
      own += c[i];
    }
    uint32_t tot, run = block_exclusive_scan<MS_BLOCK>(own, sm, tot);
    const uint64_t g = ((uint64_t)sp.seg << bits) + d0;
#pragma unroll
    for (uint32_t i = 0; i < PER; i++) {
      if (i < per && d0 + i < dig) {
        cnt[d0 + i] = run;
        if (c[i]) base[d0 + i] = sub_off[g + i] + atomicAdd(&cursor[g + i], c[i]) - run;
        run += c[i];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    if (i0 + r * 32 < n) {
      const uint32_t at = cnt[pk[r] & ((1u << MS_BITS) - 1)] + (pk[r] >> MS_BITS);
      stage[at] = key[r];
      if (pin) pstage[at] = (uint8_t)(pb[r >> 2] >> (8 * (r & 3)));
    }
  }
  __syncthreads();
#pragma unroll 4
  for (uint32_t i = tid; i < n; i += MS_BLOCK) {
    const KeyT k = stage[i];
    const uint64_t o = base[ms_digit(k, shift, dig - 1, hashed)] + i;
    if constexpr (PACK) {  // hashed 64-bit keys with payloads: the packed word (see pay_code)
      out[o] = ((k * MS_HASH_MUL) << pack) | pstage[i];
    } else {
      out[o] = k;
      if (pout) pout[o] = pstage[i];
    }
  }
}

// ---------------------------------------------------------------- chunk sort
template <class KeyT>
CF1_D void cs_swap_if(KeyT &a, KeyT &b, bool up) {
  if ((b < a) == up) {
    KeyT t = a;
    a = b;
    b = t;
  }
}

// Replaces T[a, a+n) by its distinct keys (any order) through an
// open-addressing set in shared memory; returns their count, or ~0u when
// they do not fit in three quarters of the set.  Every probe sequence is
// bounded by the set size.  Warps step through the keys together, so the
// insert count and the give-up test are per warp; the set is emptied into T
// a warp-sized group of slots at a time.  With TP (payload bytes parallel to
// T), the payloads of a key's copies are ORed into its slot's byte of SPw
// (cap bytes of shared memory) and written beside the key: the per-side join
// of the vertex's occurrences.  A pass that gives up leaves T and TP as they
// were.
CF1_D uint32_t cs_hash_dedup(uint64_t *T, uint64_t a, uint64_t n, uint64_t *S, uint32_t cap, uint32_t *s_cnt,
                             uint32_t *sm, uint8_t *TP = nullptr, uint32_t *SPw = nullptr) {
  (void)sm;
  const unsigned tid = threadIdx.x, lane = lane_id();
  const uint64_t EMPTY = ~0ull;  // above every key (keys use at most 62 bits)
  uint32_t tsize = 64, tbits = 6;  // a power of two >= 1.5 n, at most cap
  while (tsize < cap && (uint64_t)tsize < n + n / 2) {
    tsize <<= 1;
    tbits++;
  }
  for (uint32_t i = tid; i < tsize; i += CS_BLOCK) S[i] = EMPTY;
  if (TP)
    for (uint32_t i = tid; i < tsize / 4; i += CS_BLOCK) SPw[i] = 0;
  if (tid == 0) *s_cnt = 0;
  __syncthreads();
  const uint32_t limit = tsize / 4 * 3;
  for (uint64_t base = tid - lane; base < n; base += CS_BLOCK) {
    uint32_t seen = 0;
    if (lane == 0) seen = *reinterpret_cast<volatile uint32_t *>(s_cnt);
    if (__shfl_sync(FULL, seen, 0) > limit) break;
    const uint64_t i = base + lane;
    bool added = false;
    if (i < n) {
      const uint64_t key = T[a + i];
      const uint32_t pay = TP ? TP[a + i] : 0u;  // loaded beside the key, not after the probe
      uint32_t h = (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> (64 - tbits));  // multiplicative hashing
      for (uint32_t probe = 0; probe < tsize; probe++) {
        unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long *>(S + h), EMPTY, key);
        if (old == EMPTY || old == key) {
          added = old == EMPTY;
          if (TP) atomicOr(&SPw[h >> 2], pay << (8 * (h & 3)));
          break;
        }
        h = (h + 1) & (tsize - 1);
      }
    }
    const unsigned b = __ballot_sync(FULL, added);
    if (lane == 0 && b) atomicAdd(s_cnt, (uint32_t)__popc(b));
  }
  __syncthreads();
  const uint32_t d = *s_cnt;
  __syncthreads();
  if (d > limit) return ~0u;
  if (tid == 0) *s_cnt = 0;
  __syncthreads();
  for (uint32_t base = tid - lane; base < tsize; base += CS_BLOCK) {
    const uint64_t v = S[base + lane];
    const bool f = v != EMPTY;
    const unsigned b = __ballot_sync(FULL, f);
    uint32_t o = 0;
    if (lane == 0 && b) o = atomicAdd(s_cnt, (uint32_t)__popc(b));
    o = __shfl_sync(FULL, o, 0);
    if (f) {
      const uint64_t at = a + o + __popc(b & lanemask_lt());
      T[at] = v;
      if (TP) TP[at] = (uint8_t)(SPw[(base + lane) >> 2] >> (8 * ((base + lane) & 3)));
    }
  }
  __syncthreads();
  return d;
}

// Bucket of a key for the shared-memory counting sort: the bits
// [s1, s1+b1) minus off1, followed by the bits [s2, s2+b2).  A plain
// sub-bucket uses the next bits below its prefix (b2 = 0); a chunk of pieces
// of a split sub-bucket uses the piece index relative to the chunk's first
// piece, then further bits.
struct CsDigit {
  int s1, b1, s2, b2;
  uint32_t off1;
  template <class KeyT>
  CF1_D uint32_t operator()(const KeyT &k) const {
    uint32_t d1 = b1 ? KOps<KeyT>::digit(k, s1, (1u << b1) - 1) - off1 : 0u;
    uint32_t d2 = b2 ? KOps<KeyT>::digit(k, s2, (1u << b2) - 1) : 0u;
    return (d1 << b2) | d2;
  }
};

struct CsShared {
  uint32_t *hist, *cur, *sm;
  int *big;
  uint8_t *SP = nullptr;  // payload bytes beside S (CAP), when the keys carry payloads
};

template <class KeyT>
CF1_D void cs_swap_if(KeyT &a, KeyT &b, uint8_t *pa, uint8_t *pb, bool up) {
  if ((b < a) == up) {
    KeyT t = a;
    a = b;
    b = t;
    if (pa) {
      uint8_t u = *pa;
      *pa = *pb;
      *pb = u;
    }
  }
}

// Sorted distinct keys of src[0, m) (m <= CAP, keys all in [0, 1024) buckets
// of dig) into out[0, tot); returns tot.  src is fully read into shared
// memory before out is written, so they may overlap.  With srcP/outP (and
// sh.SP), each key's payload byte moves with it and the payloads of a key's
// copies are ORed.  All threads call it.
template <class KeyT>
CF1_D uint32_t cs_sort_unique_range(const KeyT *src, uint32_t m, const CsDigit &dig, KeyT *S, const CsShared &sh,
                                    KeyT *out, bool distinct, const uint8_t *srcP = nullptr,
                                    uint8_t *outP = nullptr) {
  uint8_t *SP = srcP ? sh.SP : nullptr;
  constexpr uint32_t CAP = cs_cap<KeyT>();
  const unsigned tid = threadIdx.x;
  for (uint32_t i = tid; i < CS_BUCKETS; i += CS_BLOCK) sh.hist[i] = 0;
  if (tid == 0) *sh.big = 0;
  __syncthreads();
  for (uint32_t i = tid; i < m; i += CS_BLOCK) atomicAdd(&sh.hist[dig(src[i])], 1u);
  __syncthreads();
  {
    constexpr int PER = CS_BUCKETS / CS_BLOCK;
    uint32_t v[PER], s = 0;
#pragma unroll
    for (int q = 0; q < PER; q++) {
      v[q] = sh.hist[tid * PER + q];
      s += v[q];
    }
    uint32_t tot;
    uint32_t pre = block_exclusive_scan<CS_BLOCK>(s, sh.sm, tot);
#pragma unroll
    for (int q = 0; q < PER; q++) {
      sh.hist[tid * PER + q] = pre;
      sh.cur[tid * PER + q] = pre;
      pre += v[q];
    }
  }
  __syncthreads();
  for (uint32_t i = tid; i < m; i += CS_BLOCK) {
    KeyT key = src[i];
    const uint32_t at = atomicAdd(&sh.cur[dig(key)], 1u);
    S[at] = key;
    if (SP) SP[at] = srcP[i];
  }
  __syncthreads();
  // insertion sort per bucket (bucket b spans [hist[b], cur[b]))
  for (uint32_t b = tid; b < CS_BUCKETS; b += CS_BLOCK) {
    uint32_t lo = sh.hist[b], hi = sh.cur[b];
    if (hi - lo > CS_SMALL) {
      *sh.big = 1;
      continue;
    }
    for (uint32_t i = lo + 1; i < hi; i++) {
      KeyT x = S[i];
      const uint8_t xp = SP ? SP[i] : 0;
      uint32_t q = i;
      while (q > lo && x < S[q - 1]) {
        S[q] = S[q - 1];
        if (SP) SP[q] = SP[q - 1];
        q--;
      }
      S[q] = x;
      if (SP) SP[q] = xp;
    }
  }
  __syncthreads();
  if (*sh.big) {  // bitonic sort of the whole range, padded to a power of two
    uint32_t P2 = 1;
    while (P2 < m) P2 <<= 1;
    for (uint32_t i = m + tid; i < P2; i += CS_BLOCK) {
      S[i] = KOps<KeyT>::max_key();
      if (SP) SP[i] = 0;
    }
    __syncthreads();
    for (uint32_t size = 2; size <= P2; size <<= 1) {
      for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
        for (uint32_t i = tid; i < P2 / 2; i += CS_BLOCK) {
          uint32_t lo = 2 * i - (i & (stride - 1));
          cs_swap_if(S[lo], S[lo + stride], SP ? SP + lo : nullptr, SP ? SP + lo + stride : nullptr,
                     (lo & size) == 0);
        }
        __syncthreads();
      }
    }
  }
  (void)CAP;
  if (distinct) {  // already one copy per key: plain copy out
    for (uint32_t i = tid; i < m; i += CS_BLOCK) {
      out[i] = S[i];
      if (SP) outP[i] = SP[i];
    }
    __syncthreads();
    return m;
  }
  // adjacent-unique; a run's first key takes the OR of the run's payloads
  return block_select<CS_BLOCK>(
      m, [&](uint32_t i) { return i == 0 || S[i] != S[i - 1]; },
      [&](uint32_t i, uint32_t r) {
        out[r] = S[i];
        if (SP) {
          uint32_t p = SP[i];
          for (uint32_t j = i + 1; j < m && S[j] == S[i]; j++) p |= SP[j];
          outP[r] = (uint8_t)p;
        }
      },
      sh.sm);
}

// Level-0 and level-1 slices of sub-bucket j (bin j >> P, slice j mod 2^P)
// over its n distinct keys (see Level0Out); set/col: L0_SW_MAX words of
// shared memory each (level 0's sw words, then level 1's sw1); lb: lb_cap
// u16 of shared memory for the keys' bits in the slices (a slice has at most
// L0_SW_MAX * 64 < 2^16 - 2 bits).  All threads call it.
constexpr uint32_t L0_SW_MAX = 768;
static_assert(L0_SW_MAX * sizeof(uint32_t) <= cs_cap_for(false, false), "l0_slice's pw fits the payload area");
// With kpay (the keys' joined payload bytes) and o.with_pay, the payloads go
// out as Level0Out describes; pw: L0_SW_MAX u32 of shared memory.
CF1_D void l0_slice(const uint64_t *keys, uint32_t n, uint64_t j, int P, const Level0Out &o,
                    unsigned long long *set, unsigned long long *col, uint16_t *lb, uint32_t lb_cap, uint32_t *sm,
                    unsigned long long *s_base, const uint8_t *kpay, uint64_t a, uint32_t *pw) {
  constexpr uint16_t BAD = 0xFFFF, AT0 = 0xFFFE;  // lb[i]: no bit / placed at level 0 / else its level-1 bit
  const bool pay = o.with_pay && kpay;
  const unsigned tid = threadIdx.x;
  const uint32_t bin = (uint32_t)(j >> P), sub = (uint32_t)(j & ((1ull << P) - 1));
  const uint64_t W = o.woff[bin + 1] - o.woff[bin];
  const uint32_t sw = (uint32_t)(W >> P);
  const uint32_t sw1 = (uint32_t)((o.woff1[bin + 1] - o.woff1[bin]) >> P);
  const uint64_t first1 = o.woff1[bin] + (uint64_t)sub * sw1;
  if (n == 0) {  // every slice writes all its entries (the array is not cleared first)
    for (uint32_t w = tid; w < sw; w += CS_BLOCK)
      o.AR[o.woff[bin] + (uint64_t)sub * sw + w] = make_ulonglong2(0ull, 0ull);
    for (uint32_t w = tid; w < sw1; w += CS_BLOCK) o.AR1[first1 + w] = make_ulonglong2(0ull, 0ull);
    if (tid == 0) o.placed[j] = o.placed1[j] = 0;
    return;
  }
  // level 1 uses the words of set, col and pw after level 0's
  if (sw > L0_SW_MAX || sw + sw1 > L0_SW_MAX || sw1 > CS_BLOCK || sw == 0 || n > lb_cap) {
    if (tid == 0) {
      atomicOr(o.err, 1u);
      o.placed[j] = o.placed1[j] = 0;
    }
    return;
  }
  const uint64_t first = o.woff[bin] + (uint64_t)sub * sw;  // the slice's first entry
  const uint64_t lo_bit = (uint64_t)sub * sw * 64;
  for (uint32_t w = tid; w < sw; w += CS_BLOCK) set[w] = col[w] = 0;
  __syncthreads();
  for (uint32_t i = tid; i < n; i += CS_BLOCK) {
    const uint64_t b = bb_pos(keys[i], 0, (uint32_t)W) - lo_bit;
    if (b >= (uint64_t)sw * 64) {  // not this slice's key: cannot happen with the shared hash
      atomicOr(o.err, 1u);
      lb[i] = BAD;
      continue;
    }
    lb[i] = (uint16_t)b;
    const unsigned long long bit = 1ull << (b & 63);
    if (atomicOr(&set[b >> 6], bit) & bit) atomicOr(&col[b >> 6], bit);
  }
  __syncthreads();
  // the placed bits of the slice before each word (words 2t and 2t+1 per
  // thread: sw <= L0_SW_MAX <= 2 CS_BLOCK), written beside the word
  uint32_t placed0 = 0;
  {
    const uint32_t w0 = 2 * tid, w1 = w0 + 1;
    const uint32_t c0 = w0 < sw ? (uint32_t)popc64(set[w0] & ~col[w0]) : 0u;
    const uint32_t c1 = w1 < sw ? (uint32_t)popc64(set[w1] & ~col[w1]) : 0u;
    const uint32_t pre_w = block_exclusive_scan<CS_BLOCK>(c0 + c1, sm, placed0);
    if (w0 < sw) {
      pw[w0] = pre_w;
      o.AR[first + w0] = make_ulonglong2(set[w0] & ~col[w0], (unsigned long long)pre_w);
    }
    if (w1 < sw) {
      pw[w1] = pre_w + c0;
      o.AR[first + w1] = make_ulonglong2(set[w1] & ~col[w1], (unsigned long long)(pre_w + c0));
    }
  }
  if (pay) {
    // a placed key's rank in the slice: the placed bits before its bit
    __syncthreads();
    for (uint32_t i = tid; i < n; i += CS_BLOCK) {
      const uint32_t b = lb[i];
      if (b == BAD) continue;
      const uint64_t fin = set[b >> 6] & ~col[b >> 6];
      const uint64_t bit = 1ull << (b & 63);
      if (fin & bit) o.l0pay[a + pw[b >> 6] + (uint32_t)popc64(fin & (bit - 1))] = kpay[i];
    }
  }
  // level 1 (sliced, sw1 words): the keys whose level-0 bit collided
  unsigned long long *set1 = set + sw, *col1 = col + sw;
  uint32_t *pw1 = pw + sw;
  for (uint32_t w = tid; w < sw1; w += CS_BLOCK) set1[w] = col1[w] = 0;
  __syncthreads();
  for (uint32_t i = tid; i < n; i += CS_BLOCK) {
    const uint32_t b = lb[i];
    if (b == BAD) continue;
    if (!((col[b >> 6] >> (b & 63)) & 1)) {
      lb[i] = AT0;
      continue;
    }
    const uint32_t p1 = bb_slice_pos(keys[i], 1, sw1);
    const unsigned long long bit = 1ull << (p1 & 63);
    if (atomicOr(&set1[p1 >> 6], bit) & bit) atomicOr(&col1[p1 >> 6], bit);
    lb[i] = (uint16_t)p1;
  }
  __syncthreads();
  const unsigned long long g1 = tid < sw1 ? set1[tid] & ~col1[tid] : 0ull;  // sw1 <= CS_BLOCK
  uint32_t placed1;
  const uint32_t pre1 = block_exclusive_scan<CS_BLOCK>((uint32_t)popc64(g1), sm, placed1);
  if (tid < sw1) {
    pw1[tid] = pre1;
    o.AR1[first1 + tid] = make_ulonglong2(g1, (unsigned long long)pre1);
  }
  if (tid == 0) {
    o.placed[j] = placed0;
    o.placed1[j] = placed1;
  }
  __syncthreads();
  // level-1 ranks, and the keys level 1 leaves go on to level 2
  uint32_t c = 0;
  for (uint32_t i = tid; i < n; i += CS_BLOCK) {
    const uint32_t p1 = lb[i];
    if (p1 == BAD || p1 == AT0) continue;
    const uint64_t fin = set1[p1 >> 6] & ~col1[p1 >> 6], bit = 1ull << (p1 & 63);
    if (!(fin & bit)) c++;
    else if (pay) o.l0pay[a + placed0 + pw1[p1 >> 6] + (uint32_t)popc64(fin & (bit - 1))] = kpay[i];
  }
  uint32_t tot;
  uint32_t pre = block_exclusive_scan<CS_BLOCK>(c, sm, tot);
  if (tid == 0) {
    unsigned long long base = ~0ull;
    if (tot) {
      base = atomicAdd(&o.surv_cnt[bin], (unsigned long long)tot);
      if (base + tot > o.surv_off[bin + 1] - o.surv_off[bin]) {
        atomicOr(o.err, 1u);
        base = ~0ull;
      }
    }
    *s_base = base;
  }
  __syncthreads();
  if (*s_base != ~0ull) {
    uint64_t out = o.surv_off[bin] + *s_base + pre;
    for (uint32_t i = tid; i < n; i += CS_BLOCK) {
      const uint32_t p1 = lb[i];
      if (p1 == BAD || p1 == AT0) continue;
      if (!(((set1[p1 >> 6] & ~col1[p1 >> 6]) >> (p1 & 63)) & 1)) {
        if (pay) o.surv_pay[out] = kpay[i];
        o.surv[out++] = keys[i];
      }
    }
  }
  __syncthreads();
}

// Sorted distinct keys of one sub-bucket T[a, a+n), written back at a
// (SORTED = false: distinct keys in any order -- 64-bit keys then skip the
// sort whenever the shared-memory set holds the sub-bucket).
// Sub-buckets above CAP keys: 64-bit keys are first reduced to one copy each
// through a shared-memory set; if still above CAP, the sub-bucket is split on
// its next `bits` bits into U[a, a+n) (the free ping-pong buffer), runs of
// consecutive pieces up to CAP keys are sorted one after another, and their
// distinct keys are appended at T[a].  Only a single piece above CAP keys
// makes the kernel report the sub-bucket as oversized.
// With TP/UP (payload bytes parallel to T and U), every distinct key leaves
// with the OR of its copies' payloads beside it in TP.
// Runs (sorted form): with runs, CTA c takes the consecutive sub-buckets
// [j0, j1) of one bin that the plan packed together, sorts the run as one
// range -- its bucket is the sub-bucket's place in the run, then the next key
// bits -- and credits all its distinct keys to sub-bucket j0.
template <class KeyT, bool SORTED>
__global__ void __launch_bounds__(CS_BLOCK, SORTED ? 2 : 4) cs_sort_unique_kernel(KeyT *T, KeyT *U, const uint64_t *sb_off,
                                                                  uint64_t nsub, int shift, int bits, uint32_t *cnt,
                                                                  uint32_t *oversize, int P, Level0Out l0,
                                                                  uint8_t *TP, uint8_t *UP, const uint2 *runs,
                                                                  const uint32_t *jlist, const uint32_t *klist,
                                                                  bool codes) {
  constexpr uint32_t CAP = cs_cap<KeyT, SORTED>();
  constexpr bool L0 = !SORTED && KOps<KeyT>::WORDS == 1;
  __shared__ unsigned long long s_l0base;
  extern __shared__ __align__(16) unsigned char cs_smem[];
  KeyT *S = reinterpret_cast<KeyT *>(cs_smem);                    // [CAP]
  uint32_t *hist = reinterpret_cast<uint32_t *>(S + CAP);         // [CS_BUCKETS]
  uint32_t *cur = hist + CS_BUCKETS;                              // [CS_BUCKETS]
  uint32_t *pstart = cur + CS_BUCKETS;                            // [CS_BUCKETS + 1]
  uint16_t *cb = reinterpret_cast<uint16_t *>(pstart + CS_BUCKETS + 1);  // [CS_BUCKETS + 1]
  uint32_t *SPw = reinterpret_cast<uint32_t *>(cb + CS_BUCKETS + 2);     // [CAP / 4] payloads, when TP
  __shared__ uint32_t sm[CS_BLOCK / 32];
  __shared__ int s_big, s_nchunks, s_bad;
  __shared__ uint32_t s_cnt;
  const uint32_t run = klist ? klist[blockIdx.x] : blockIdx.x;  // klist: the runs the rank dedup left
  uint64_t j = run, jend = j + 1;
  if (jlist) {  // the sub-buckets the warp dedup left
    j = jlist[blockIdx.x];
    jend = j + 1;
  } else if (runs) {
    j = runs[run].x;
    jend = runs[run].y;
  }
  if (j >= nsub) return;
  const uint64_t a = sb_off[j], n = sb_off[jend] - a;
  const unsigned tid = threadIdx.x;
  if (codes && TP) {  // payloads as they travel: the bytes they stand for
    for (uint64_t i = a + tid; i < a + n; i += CS_BLOCK) TP[i] = (uint8_t)pay_byte(TP[i]);
    __syncthreads();
  }
  // the sub-bucket's distinct keys end at T[a, a + result); ~0u: oversized
  auto body = [&]() -> uint32_t {
    if (n == 0) return 0;
    CsShared sh{hist, cur, sm, &s_big, TP ? reinterpret_cast<uint8_t *>(SPw) : nullptr};
    CsDigit plain{shift, bits, 0, 0, 0u};
    if (SORTED && jend - j > 1) {  // a packed run: bucket = place of the sub-bucket in the run, then the next bits
      const uint32_t span = (uint32_t)(jend - j);
      if (span > CS_BUCKETS) return ~0u;  // the plan never makes one; refused (LSD path) rather than mis-bucketed
      int g = 0;
      while ((1u << g) < span) g++;
      const int rest = shift + bits;  // the sub-bucket prefix sits at bits [rest, rest + P)
      const int b2 = 10 - g < rest ? 10 - g : rest;
      plain = CsDigit{rest, P, rest - b2, b2, (uint32_t)(j & ((1ull << P) - 1))};
    }
    uint32_t m = (uint32_t)n;
    bool distinct = false;
    // 64-bit keys: one copy of each key first.  Repeats put hundreds of
    // copies of a k-mer in one bucket, where sorting copies would dominate.
    if ((!SORTED || n > CS_DEDUP_MIN) && KOps<KeyT>::WORDS == 1) {
      uint32_t d = cs_hash_dedup(reinterpret_cast<uint64_t *>(T), a, n, reinterpret_cast<uint64_t *>(S), CAP, &s_cnt, sm,
                                 TP, SPw);
      if (d != ~0u) {
        m = d;
        distinct = true;
        if (!SORTED) return d;  // distinct keys are all that is needed
      }
    }
    if (m <= CAP)
      return cs_sort_unique_range<KeyT>(T + a, m, plain, S, sh, T + a, distinct, TP ? TP + a : nullptr,
                                        TP ? TP + a : nullptr);
    // local split on the next `bits` bits into U[a, a+n)
    const uint32_t npieces = 1u << bits, pmask = npieces - 1;
    for (uint32_t i = tid; i <= CS_BUCKETS; i += CS_BLOCK) pstart[i] = 0;
    __syncthreads();
    for (uint64_t i = tid; i < n; i += CS_BLOCK) atomicAdd(&pstart[KOps<KeyT>::digit(T[a + i], shift, pmask)], 1u);
    __syncthreads();
    if (tid == 0) {
      uint32_t run = 0;
      for (uint32_t p = 0; p < npieces; p++) {
        uint32_t v = pstart[p];
        pstart[p] = run;
        run += v;
      }
      pstart[npieces] = run;
      // greedy runs of consecutive pieces up to CAP keys
      int nc = 0, bad = 0;
      uint32_t acc = 0;
      cb[0] = 0;
      for (uint32_t p = 0; p < npieces; p++) {
        uint32_t sz = pstart[p + 1] - pstart[p];
        if (sz > CAP) {  // a piece of its own, deduplicated before sorting (64-bit keys)
          if (KOps<KeyT>::WORDS != 1) bad = 1;
          if (acc > 0) cb[++nc] = (uint16_t)p;
          cb[++nc] = (uint16_t)(p + 1);
          acc = 0;
          continue;
        }
        if (acc + sz > CAP && acc > 0) {
          cb[++nc] = (uint16_t)p;
          acc = 0;
        }
        acc += sz;
      }
      if (acc == 0) nc--;  // the loop already closed the last run
      cb[++nc] = (uint16_t)npieces;
      s_nchunks = nc;
      s_bad = bad;
    }
    __syncthreads();
    if (s_bad) return ~0u;
    for (uint32_t p = tid; p < npieces; p += CS_BLOCK) cur[p] = pstart[p];
    __syncthreads();
    for (uint64_t i = tid; i < n; i += CS_BLOCK) {
      KeyT key = T[a + i];
      const uint32_t at = atomicAdd(&cur[KOps<KeyT>::digit(key, shift, pmask)], 1u);
      U[a + at] = key;
      if (TP) UP[a + at] = TP[a + i];
    }
    __syncthreads();
    uint32_t outc = 0;
    for (int c = 0; c < s_nchunks; c++) {
      uint32_t p0 = cb[c], p1 = cb[c + 1];
      uint32_t span = p1 - p0;
      int g = 0;
      while ((1u << g) < span) g++;
      int b2 = 10 - g;
      if (b2 > shift) b2 = shift;
      CsDigit dig{shift, bits, shift - b2, b2, p0};
      uint32_t len = pstart[p1] - pstart[p0];
      bool dd = false;
      if (len > CS_DEDUP_MIN && KOps<KeyT>::WORDS == 1) {
        uint32_t d = cs_hash_dedup(reinterpret_cast<uint64_t *>(U), a + pstart[p0], len,
                                   reinterpret_cast<uint64_t *>(S), CAP, &s_cnt, sm, TP ? UP : nullptr, SPw);
        if (d != ~0u) {  // (a failed pass leaves U untouched)
          len = d;
          dd = true;
        }
        if (len > CAP) return ~0u;
      }
      outc += cs_sort_unique_range<KeyT>(U + a + pstart[p0], len, dig, S, sh, T + a + outc, dd,
                                         TP ? UP + a + pstart[p0] : nullptr, TP ? TP + a + outc : nullptr);
    }
    return outc;
  };
  const uint32_t res = body();
  if (tid == 0) {
    cnt[j] = res == ~0u ? 0 : res;
    if (res == ~0u) atomicOr(oversize, 1u);
  }
  for (uint64_t q = j + 1 + tid; q < jend; q += CS_BLOCK) cnt[q] = 0;
  if constexpr (L0) {
    if (l0.AR && res == ~0u) {  // no slice: its placed counts are read all the same (gd_gather_kernel)
      if (tid == 0) l0.placed[j] = l0.placed1[j] = 0;
    } else if (l0.AR) {
      __syncthreads();
      unsigned long long *h64 = reinterpret_cast<unsigned long long *>(hist);
      l0_slice(reinterpret_cast<const uint64_t *>(T) + a, res, j, P, l0, h64, h64 + L0_SW_MAX,
               reinterpret_cast<uint16_t *>(S), CAP * sizeof(KeyT) / 2, sm, &s_l0base, TP ? TP + a : nullptr, a,
               SPw);
    }
  }
}

// ---------------------------------------------------------------- rank dedup
// The sorted form's dedup, and that of 128-bit keys in the BBHash form
// (HASHED): one CTA per run of consecutive sub-buckets of a bin (the plan's
// runs), at most SrCfg::CAP keys, held in registers.  A key's position is
// its distance from the run's start in the key range (HASHED: in the range of
// the level-0 hash), scaled by a shift to NP = 8 CAP bits, so positions ascend
// with the keys (with the hash):
//   1. every occurrence marks its position (set; col when it was set
//      already).  A position marked once is one key, whose rank is the popcount
//      of set before it, plus
//   2. what the shared positions before it hold beyond one key: their
//      occurrences are gathered, position by position (numbered by a popcount
//      of col, counted by atomics), and one thread per position sorts its few
//      keys and joins the copies' payload bytes.  In a run with more than
//      SR_MANY occurrences on a position, the copies of every position's
//      first key join it before that, all at once: one thread walking tandem
//      arrays' hundreds of copies took 3.1 Gbp with them 180 ms, now 133;
//   3. keys and bytes are staged in shared memory by rank and written out.
// ~85% of the keys of unrepeated sequence have a position of their own.  A run
// that does not fit (a sub-bucket above CAP keys, more than SR_MAXD different
// keys on one position) is untouched and listed for cs_sort_unique_kernel,
// whose hash set, 1024-bucket counting sort and insertion sorts this replaces
// for the others: 200 Mbp 6.89 -> 2.86 ms, at k = 63 100 Mbp 3.51 -> 2.13 ms.
// Its bound is its barriers and instruction issue, as the group dedup's below.
constexpr int SR_BLOCK = 512;
constexpr uint32_t SR_MAXD = 48;
constexpr uint32_t SR_MANY = 32;  // (8 sent repeats of ordinary genomes there too: 200 Mbp 3.21 ms, 3.17 now)
template <class KeyT>
struct SrCfg {
  static constexpr int U = KOps<KeyT>::WORDS == 1 ? 8 : 4;  // keys per thread
  static constexpr uint32_t CAP = SR_BLOCK * U;
  static constexpr int LOGNP = KOps<KeyT>::WORDS == 1 ? 15 : 14;
  static constexpr uint32_t NP = 1u << LOGNP, NWORD = NP / 32;
  static constexpr int WPT = NWORD / SR_BLOCK;  // words of the bitmaps a thread scans
  static constexpr int CPT = CAP / 2 / SR_BLOCK;  // shared positions a thread scans
};
template <class KeyT>
struct SrSmem {
  using C = SrCfg<KeyT>;
  KeyT seg[C::CAP], stage[C::CAP];
  uint32_t set[C::NWORD], col[C::NWORD];
  uint32_t cnt[C::CAP / 2];                     // occurrences, then distinct keys, of a shared position
  uint16_t start[C::CAP / 2], ex[C::CAP / 2 + 2];  // its place in seg; keys beyond one a position before it
  uint16_t spre[C::NWORD], cpre[C::NWORD];      // set / col bits before a word
  uint8_t segp[C::CAP], stagep[C::CAP];
  uint32_t sm[SR_BLOCK / 32];
};

static_assert(offsetof(SrSmem<uint64_t>, stagep) % 4 == 0 && offsetof(SrSmem<Key2>, stagep) % 4 == 0, "joined in words");

template <class KeyT, bool HASHED>
__global__ void __launch_bounds__(SR_BLOCK, 2) sr_dedup_kernel(KeyT *T, uint8_t *TP, const uint64_t *sb_off,
                                                              uint64_t nsub, int P, int rest, uint32_t *cnt,
                                                              const uint2 *runs, uint32_t *ov, uint32_t *ov_cnt) {
  using C = SrCfg<KeyT>;
  extern __shared__ __align__(16) unsigned char sr_smem[];
  SrSmem<KeyT> &m = *reinterpret_cast<SrSmem<KeyT> *>(sr_smem);
  const unsigned tid = threadIdx.x;
  uint64_t j = blockIdx.x, jend = j + 1;
  if (runs) {
    j = runs[blockIdx.x].x;
    jend = runs[blockIdx.x].y;
  }
  if (j >= nsub) return;
  const uint64_t a = sb_off[j], n64 = sb_off[jend] - a;
  if (n64 > C::CAP) {
    if (tid == 0) ov[atomicAdd(ov_cnt, 1u)] = blockIdx.x;
    return;
  }
  for (uint64_t q = j + tid; q < jend; q += SR_BLOCK) cnt[q] = 0;
  if (n64 == 0) return;
  const uint32_t n = (uint32_t)n64, sub0 = (uint32_t)(j & ((1ull << P) - 1)), span = (uint32_t)(jend - j);
  int sh = rest - C::LOGNP;  // the run's range, span << rest, in at most NP positions
  while ((1u << (sh + C::LOGNP - rest)) < span) sh++;
  if (sh < 0) sh = 0;
  const uint32_t pos0 = sub0 << (rest - sh);
  auto pos_of = [&](const KeyT &k) -> uint32_t {
    if constexpr (HASHED) return ((uint32_t)((bb_key_hash(k) * MS_HASH_MUL) >> 32) >> sh) - pos0;
    else return KOps<KeyT>::digit(k, sh, 0xFFFFFFFFu) - pos0;
  };
  KeyT key[C::U];
  uint32_t pos[C::U];
  uint32_t pb[C::U / 4];
#pragma unroll
  for (int i = 0; i < C::U / 4; i++) pb[i] = 0;
#pragma unroll
  for (int u = 0; u < C::U; u++) {
    const uint32_t i = u * SR_BLOCK + tid;
    if (i < n) {
      key[u] = T[a + i];
      if (TP) pb[u >> 2] |= pay_byte(TP[a + i]) << (8 * (u & 3));
    }
  }
#pragma unroll
  for (int u = 0; u < C::U; u++) pos[u] = u * SR_BLOCK + tid < n ? pos_of(key[u]) : 0u;
  for (uint32_t w = tid; w < C::NWORD; w += SR_BLOCK) m.set[w] = m.col[w] = 0;
  __syncthreads();
  // 1. mark
#pragma unroll
  for (int u = 0; u < C::U; u++) {
    if (u * SR_BLOCK + tid < n) {
      const uint32_t p = pos[u], bm = 1u << (p & 31);
      if (atomicOr(&m.set[p >> 5], bm) & bm) atomicOr(&m.col[p >> 5], bm);
    }
  }
  __syncthreads();
  uint32_t nset, ncol;
  {
    uint32_t v = 0, x[C::WPT];
#pragma unroll
    for (int i = 0; i < C::WPT; i++) {
      const uint32_t w = tid * C::WPT + i;
      x[i] = (uint32_t)__popc(m.set[w]) | ((uint32_t)__popc(m.col[w]) << 16);
      v += x[i];
    }
    uint32_t tot, pre = block_exclusive_scan<SR_BLOCK>(v, m.sm, tot);
#pragma unroll
    for (int i = 0; i < C::WPT; i++) {
      const uint32_t w = tid * C::WPT + i;
      m.spre[w] = (uint16_t)pre;
      m.cpre[w] = (uint16_t)(pre >> 16);
      pre += x[i];
    }
    nset = tot & 0xFFFFu;
    ncol = tot >> 16;
  }
  uint32_t shared = 0, extra = 0;    // this thread's keys on shared positions; keys beyond one a position
  uint32_t copies = 0;               // copies of the first key that reached their position
  bool join = false;
  if (ncol) {  // uniform
    // 2. the shared positions' occurrences, counted, placed and sorted
    uint32_t *joined = reinterpret_cast<uint32_t *>(m.stagep);  // a position's first key's copies' payloads
    for (uint32_t c = tid; c < ncol; c += SR_BLOCK) m.cnt[c] = 0;
    __syncthreads();
    bool many = false;
    uint32_t slot[C::U];  // position | place among the position's occurrences << 16
#pragma unroll
    for (int u = 0; u < C::U; u++) {
      slot[u] = 0;
      if (u * SR_BLOCK + tid < n) {
        const uint32_t p = pos[u], bm = 1u << (p & 31), cw = m.col[p >> 5];
        if (cw & bm) {
          const uint32_t c = m.cpre[p >> 5] + (uint32_t)__popc(cw & (bm - 1));
          shared |= 1u << u;
          const uint32_t at = atomicAdd(&m.cnt[c], 1u);
          slot[u] = c | (at << 16);
          many |= at >= SR_MANY;
        }
      }
    }
    join = __syncthreads_or((int)many) != 0;
    if (join) {
      // copies of a position's first key join it here, all at once; what is
      // sorted below are the other keys
      for (uint32_t w = tid; 4 * w < ncol; w += SR_BLOCK) joined[w] = 0;
#pragma unroll
      for (int u = 0; u < C::U; u++)
        if (((shared >> u) & 1) && slot[u] < 0x10000u) m.stage[slot[u]] = key[u];
      __syncthreads();
#pragma unroll
      for (int u = 0; u < C::U; u++) {
        if (((shared >> u) & 1) && slot[u] >= 0x10000u) {
          const uint32_t c = slot[u] & 0xFFFFu;
          if (m.stage[c] == key[u]) {
            copies |= 1u << u;
            if (TP) atomicOr(&joined[c >> 2], ((pb[u >> 2] >> (8 * (u & 3))) & 0xFFu) << (8 * (c & 3)));
          } else {
            slot[u] = c | (((atomicAdd(&m.cnt[c], 0x10000u) >> 16) + 1) << 16);
          }
        }
      }
      __syncthreads();
      for (uint32_t c = tid; c < ncol; c += SR_BLOCK) m.cnt[c] = (m.cnt[c] >> 16) + 1;
      __syncthreads();
    }
    {
      uint32_t v = 0, x[C::CPT], tot;
#pragma unroll
      for (int i = 0; i < C::CPT; i++) {
        const uint32_t c = tid * C::CPT + i;
        x[i] = c < ncol ? m.cnt[c] : 0u;
        v += x[i];
      }
      uint32_t pre = block_exclusive_scan<SR_BLOCK>(v, m.sm, tot);
#pragma unroll
      for (int i = 0; i < C::CPT; i++) {
        const uint32_t c = tid * C::CPT + i;
        if (c < ncol) m.start[c] = (uint16_t)pre;
        pre += x[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < C::U; u++) {
      if (((shared & ~copies) >> u) & 1) {
        const uint32_t c = slot[u] & 0xFFFFu, at = m.start[c] + (slot[u] >> 16);
        uint32_t p = pb[u >> 2] >> (8 * (u & 3));
        if (join && slot[u] < 0x10000u) p |= joined[c >> 2] >> (8 * (c & 3));
        m.seg[at] = key[u];
        m.segp[at] = (uint8_t)p;
      }
    }
    __syncthreads();
    bool over = false;
    for (uint32_t c = tid; c < ncol && !over; c += SR_BLOCK) {
      // the position's distinct keys, ascending, at the front of its segment
      KeyT *S = m.seg + m.start[c];
      uint8_t *SP = m.segp + m.start[c];
      const uint32_t len = m.cnt[c];
      uint32_t d = 1;
      for (uint32_t i = 1; i < len; i++) {
        const KeyT x = S[i];
        const uint8_t xp = SP[i];
        uint32_t q = d;
        while (q > 0 && x < S[q - 1]) q--;
        if (q > 0 && S[q - 1] == x) {
          SP[q - 1] |= xp;
          continue;
        }
        if (d >= SR_MAXD) {
          over = true;
          break;
        }
        for (uint32_t r = d; r > q; r--) {
          S[r] = S[r - 1];
          SP[r] = SP[r - 1];
        }
        S[q] = x;
        SP[q] = xp;
        d++;
      }
      m.cnt[c] = d;
    }
    if (__syncthreads_or((int)over)) {  // nothing of the run was written but zero counts
      if (tid == 0) ov[atomicAdd(ov_cnt, 1u)] = blockIdx.x;
      return;
    }
    uint32_t v = 0, x[C::CPT];
#pragma unroll
    for (int i = 0; i < C::CPT; i++) {
      const uint32_t c = tid * C::CPT + i;
      x[i] = c < ncol ? m.cnt[c] - 1 : 0u;
      v += x[i];
    }
    uint32_t pre = block_exclusive_scan<SR_BLOCK>(v, m.sm, extra);
#pragma unroll
    for (int i = 0; i < C::CPT; i++) {
      const uint32_t c = tid * C::CPT + i;
      if (c <= ncol) m.ex[c] = (uint16_t)pre;
      pre += x[i];
    }
    if (tid == 0) m.ex[ncol] = (uint16_t)extra;  // (ncol may be CAP / 2: no thread's)
    __syncthreads();
  } else {
    if (tid == 0) m.ex[0] = 0;
    __syncthreads();
  }
  // 3. by rank
  auto rank_of = [&](uint32_t p) -> uint32_t {
    const uint32_t w = p >> 5, lm = (1u << (p & 31)) - 1;
    return m.spre[w] + (uint32_t)__popc(m.set[w] & lm) + m.ex[m.cpre[w] + (uint32_t)__popc(m.col[w] & lm)];
  };
#pragma unroll
  for (int u = 0; u < C::U; u++) {
    if (u * SR_BLOCK + tid < n && !((shared >> u) & 1)) {
      const uint32_t r = rank_of(pos[u]);
      m.stage[r] = key[u];
      m.stagep[r] = (uint8_t)(pb[u >> 2] >> (8 * (u & 3)));
    }
  }
  for (uint32_t c = tid; c < ncol; c += SR_BLOCK) {
    const uint32_t s0 = m.start[c], d = m.cnt[c], r = rank_of(pos_of(m.seg[s0]));
    for (uint32_t i = 0; i < d; i++) {
      m.stage[r + i] = m.seg[s0 + i];
      m.stagep[r + i] = m.segp[s0 + i];
    }
  }
  __syncthreads();
  const uint32_t tot = nset + extra;
  for (uint32_t i = tid; i < tot; i += SR_BLOCK) {
    T[a + i] = m.stage[i];
    if (TP) TP[a + i] = m.stagep[i];
  }
  if (tid == 0) cnt[j] = tot;
}

// ---------------------------------------------------------------- group dedup
// The unsorted (BBHash) form's dedup: one CTA per group of up to 16 or 32
// consecutive sub-buckets of a bin, whose level-0 slices (and level-1 slices)
// are consecutive words.  The group's keys sit in the CTA's registers (GD_U
// per thread) and are told apart by their BBHash bits instead of by a hash
// set:
//   1. every occurrence marks its level-0 bit (set; col when it was set
//      already).  A bit set once is one occurrence of one key: distinct, and
//      placed by level 0 -- ~88% of the occurrences of unrepeated sequence;
//   2. the occurrences on a bit set more than once go to a list, and compare
//      themselves with the first listed one of their bit (the bits numbered
//      by a popcount of col, no probing): all equal -- copies of one key,
//      placed, the first owning it and taking the OR of the copies' payload
//      bytes -- or not: the bit is cleared and its occurrences go to level 1;
//   3. those mark the group's level-1 slices the same way; the few that share
//      a level-1 bit (~1%) are compared pairwise, and what level 1 does not
//      place is listed for level 2.
// Ranks are popcounts of the placed bits, and the placed keys' bytes leave in
// rank order.  The keys stay where they are, packed: a bit per occurrence
// (keep) marks the first copy of every key, and gd_compact_kernel makes the
// dense array from them when one is asked for.  Nothing is written before the
// whole group is known to fit; a group that does not (more than MAXN
// occurrences, long slices, lists too long) is untouched and listed in ov.
//
// Groups because the split then needs four or five bits less (one pass up to
// 11 bits), and because the slices' scans and the barriers are shared by their
// sub-buckets: the same passes run by a warp on one sub-bucket of ~120 keys
// were slower than the warp's hash set below (1 Gbp: 40 against 18 ms).
// Instruction issue (65% of the slots) and its barriers bound it: ~220 warp
// instructions per 32 occurrences where the hash set took ~430.  Groups of 16,
// in CTAs half the size, four to an SM, wait less at the barriers (200 Mbp
// 2.00 against 1.88 ms, 40 Mb of transcripts 0.81 and 0.72, 1 Gbp 14.1 and
// 13.7) but need one more split bit, so they are taken while the split has at
// most GD_SPLIT bits all the same (its scatter of 1 Gbp: 5.6 ms on 10 bits,
// 7.2 on 11; of 200 Mbp 1.00 on 8 and 1.04 on 9), and not for a bin that one
// group of 32 holds unsplit.  The dedup of 200 Mbp went from 3.77 to 1.88 ms,
// of 1 Gbp (with tandem arrays) from 18.0 to 14.1 ms, of 5 Mbp from 632 to 74
// us (the warp kernel's runs of 64 sub-buckets left most warps idle); with
// three occurrences of every key (transcripts) the list is most of the group
// and it takes 0.72 against 0.59 ms, which the split's dropped pass (0.31 ms)
// makes up for.
constexpr int GD_U = 16;                 // keys per thread
constexpr int GD_BITS = 5;               // sub-buckets of a group (log2), at most
constexpr int MSD_MAX_BITS = 16;         // widest split
constexpr uint32_t GD_MAXSUB = 224;      // occurrences of a sub-bucket a group of 32 has room for, on average
constexpr int GD_SPLIT = 10;             // most split bits that groups of 16 sub-buckets are worth
constexpr int GD_MOVE = 512;             // threads of the kernels that move a listed group
constexpr uint32_t GD_SWMAX = 32;        // level-0 words of a slice: one a lane
constexpr uint32_t GD_PAIR = 4;          // threads that compare one occurrence of a shared level-1 bit
constexpr uint32_t GD_NONE = 0xFFFF, GD_OWN = 0x8000, GD_JOIN = 0x4000;
template <int BITS>
struct GdCfg {
  static constexpr int BLOCK = 16 << BITS;
  static constexpr uint32_t MAXN = BLOCK * GD_U;          // occurrences a group may hold
  static constexpr uint32_t WMAX = GD_SWMAX << BITS;      // level-0 words of a group
  static constexpr uint32_t W1MAX = (GD_SWMAX / 8) << BITS;  // level-1 words of a group
  static constexpr uint32_t MAXL = BITS == 5 ? 5888 : 2816;  // occurrences on a level-0 bit set more than once
  static constexpr uint32_t MAXC = BLOCK;                 // occurrences on a level-1 bit set more than once
};
template <int BITS>
struct GdSmem {
  using C = GdCfg<BITS>;
  // cleared at the start, 16 bytes at a time
  unsigned long long set[C::WMAX], col[C::WMAX];   // level 0: bits set (then: placed), bits set more than once
  unsigned long long set1[C::W1MAX], col1[C::W1MAX];
  uint32_t rp[C::MAXL / 8];                        // payload bytes beside rk
  uint32_t rk[C::MAXL / 2];                        // first listed occurrence of a bit; then the byte stage
  unsigned long long lk[C::MAXL];                  // the list (PK: packed words)
  unsigned long long cid[C::MAXC];                 // ids of the entries in cq
  uint32_t cpre[C::WMAX], fpre[C::WMAX];           // per half word (16 bits each): col / placed bits before it
  uint32_t fpre1[C::W1MAX];
  uint32_t tot[1 << BITS];                      // placed bits per slice
  uint32_t cp[C::MAXC];                            // payloads joined over a key's copies
  // an entry's bit number (GD_OWN | number when its key is level 0's and it is
  // the first), its level-1 bit when level 0 leaves it (GD_JOIN: its byte is
  // in lp), or GD_NONE: a copy
  uint16_t lx[C::MAXL];
  uint16_t cq[C::MAXC], cb[C::MAXC];               // entries on a level-1 bit set more than once, and that bit
  uint8_t lp[C::MAXL];                             // the list's payload bytes (PK: those joined at level 1)
  uint8_t lut[64];                                 // payload code -> byte
  uint32_t nlc, nc, kept, placed1;                 // nlc: list entries | bits set more than once << 16
};
template <int BITS>
constexpr bool gd_layout_ok() {
  using S = GdSmem<BITS>;
  using C = GdCfg<BITS>;
  return offsetof(S, set1) % 16 == 0 && offsetof(S, rk) % 16 == 0 &&
         offsetof(S, rp) == offsetof(S, col1) + sizeof(S::col1) &&  // cleared in one run
         (2 * sizeof(S::set1) + sizeof(S::rp)) % 16 == 0 &&
         sizeof(S) <= (BITS == 5 ? 113 : 56) * 1024 &&  // two CTAs per SM, or four
         C::MAXN + 4 <= sizeof(S::rk) &&                 // the byte stage
         C::W1MAX * 64 < GD_JOIN && C::MAXL / 2 < GD_JOIN;  // an entry's number, flags and level-1 bit in 16 bits
}
static_assert(gd_layout_ok<4>() && gd_layout_ok<5>());

// Popcount prefix of a thread's 64-bit word as its two half words' values
// (low half first) in one u32.
CF1_D uint32_t gd_halves(unsigned long long x, uint32_t pre) {
  return pre | ((pre + (uint32_t)__popc((uint32_t)x)) << 16);
}
// A warp's exclusive prefix of v, and the sum.
CF1_D uint32_t gd_warp_excl(uint32_t v, uint32_t &tot) {
  const uint32_t x = warp_inclusive_scan(v);
  tot = __shfl_sync(FULL, x, 31);
  return x - v;
}
// Shared-memory ORs under a predicate, as predicated instructions: written as
// `if`, each became a branch with its reconvergence in the unrolled loops.
CF1_D uint32_t gd_shared(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
CF1_D uint32_t gd_or_if(uint32_t pred, uint32_t addr, uint32_t v) {  // returns the old word, 0 without pred
  uint32_t old;
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %1, 0;\n mov.u32 %0, 0;\n @p atom.shared.or.b32 %0, [%2], %3;\n}"
      : "=r"(old)
      : "r"(pred), "r"(addr), "r"(v)
      : "memory");
  return old;
}
CF1_D void gd_red_or_if(uint32_t pred, uint32_t addr, uint32_t v) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p red.shared.or.b32 [%1], %2;\n}"
               :
               : "r"(pred), "r"(addr), "r"(v)
               : "memory");
}
// First word of a unit's keep bits: the units' occurrences one after another,
// every unit from a word of its own.
CF1_D uint64_t gd_keep_word(uint64_t a, uint64_t q) { return (a >> 5) + q; }

// PK: T holds packed words of a first pass of p1 bits (see pay_code); id(w)
// = h = key * MS_HASH_MUL without its top p1 bits stands for the key, which
// is h * KEY_SPREAD_INV.  Group q: bin q >> Pg, the keys whose hash's top Pg
// bits are q mod 2^Pg, in T[goff[q], goff[q + 1]); it is sub-buckets
// [q << g, (q + 1) << g), g = P - Pg.
template <bool PK, int BITS>
__global__ void __launch_bounds__(GdCfg<BITS>::BLOCK, BITS == 5 ? 2 : 4)
    gd_dedup_kernel(const uint64_t *T, const uint8_t *TP,
                                                              const uint64_t *goff, int Pg, int P, uint32_t *cnt,
                                                              uint32_t *keep, Level0Out l0, uint32_t *ov,
                                                              uint32_t *ov_cnt, int p1) {
  using C = GdCfg<BITS>;
  constexpr int GD_BLOCK = C::BLOCK;
  constexpr uint32_t GD_MAXN = C::MAXN, GD_MAXL = C::MAXL, GD_MAXC = C::MAXC;
  extern __shared__ __align__(16) unsigned char gd_smem[];
  GdSmem<BITS> &m = *reinterpret_cast<GdSmem<BITS> *>(gd_smem);
  constexpr uint32_t NW = GD_BLOCK / 32, SPW = (1u << BITS) / NW;  // warps; slices a warp takes
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const uint32_t q = blockIdx.x;
  const uint64_t a = goff[q], n64 = goff[q + 1] - a;
  const int g = P - Pg;
  const uint32_t subs = 1u << g, bin = q >> Pg, gi = q & ((1u << Pg) - 1);
  const bool pay = TP != nullptr, lv0 = l0.AR != nullptr, lpay = lv0 && l0.with_pay && pay;
  uint32_t sw, sw1;
  uint64_t first = 0, first1 = 0;
  if (lv0) {
    const uint64_t f0 = l0.woff[bin], f1 = l0.woff1[bin];
    const uint64_t w0 = (l0.woff[bin + 1] - f0) >> P;
    sw = w0 > GD_SWMAX ? GD_SWMAX + 1 : (uint32_t)w0;
    sw1 = (sw + 7) / 8;  // as level 1 is sized
    first = f0 + (uint64_t)(gi << g) * sw;
    first1 = f1 + (uint64_t)(gi << g) * sw1;
  } else {  // no levels wanted: the same bits, to tell the keys apart only
    sw = (uint32_t)min((n64 + 8 * subs - 1) / (8 * subs), (uint64_t)GD_SWMAX);
    sw1 = (sw + 7) / 8;
  }
  if (n64 > GD_MAXN || sw > GD_SWMAX) {
    if (tid == 0) ov[atomicAdd(ov_cnt, 1u)] = q;
    return;
  }
  const uint32_t n = (uint32_t)n64, gw = sw * subs, gw1 = sw1 * subs;
  const uint64_t *Tk = T + a + tid;
  unsigned long long key[GD_U];    // PK: the packed word
  uint32_t pb[PK ? 1 : GD_U / 4];  // payload codes, four to a register (PK: inside the word)
  const uint32_t act = tid < n ? (0xFFFFFFFFu >> (31 - (n - 1 - tid) / GD_BLOCK)) : 0u;  // this thread's keys
  if constexpr (!PK) {
#pragma unroll
    for (int i = 0; i < GD_U / 4; i++) pb[i] = 0;
  }
#pragma unroll
  for (int u = 0; u < GD_U; u++) {
    key[u] = 0;
    if (u * GD_BLOCK < n && ((act >> u) & 1)) {  // the first test is uniform, as in every loop over u
      key[u] = Tk[u * GD_BLOCK];
      if constexpr (!PK)
        if (pay) pb[u >> 2] |= (uint32_t)TP[a + tid + u * GD_BLOCK] << (8 * (u & 3));
    }
  }
  if (tid < 64) m.lut[tid] = (uint8_t)pay_byte(tid);
  if (tid == 0) m.nlc = m.nc = m.kept = 0;
  {
    const uint4 z = make_uint4(0, 0, 0, 0), o = make_uint4(~0u, ~0u, ~0u, ~0u);
    uint4 *s4 = reinterpret_cast<uint4 *>(m.set), *c4 = reinterpret_cast<uint4 *>(m.col);
    for (uint32_t w = tid; 2 * w < gw; w += GD_BLOCK) s4[w] = c4[w] = z;
    uint4 *z4 = reinterpret_cast<uint4 *>(m.set1), *r4 = reinterpret_cast<uint4 *>(m.rk);
    constexpr uint32_t NZ = (2 * sizeof(m.set1) + sizeof(m.rp)) / 16;
    for (uint32_t w = tid; w < NZ; w += GD_BLOCK) z4[w] = z;
    for (uint32_t w = tid; w < sizeof(m.rk) / 16; w += GD_BLOCK) r4[w] = o;
  }
  const uint64_t hi = PK ? (uint64_t)(gi >> (Pg - p1)) << (64 - p1) : 0;
  const uint32_t lowP = Pg ? ~((1u << Pg) - 1) : 0xFFFFFFFFu, scale = gw << 6;
  auto id = [&](unsigned long long w) -> unsigned long long { return PK ? w >> p1 : w; };
  auto key_of = [&](unsigned long long w) -> uint64_t { return PK ? (hi | (w >> p1)) * KEY_SPREAD_INV : w; };
  auto pay_of = [&](int u) -> uint32_t {
    if constexpr (PK) return (uint32_t)m.lut[(uint32_t)key[u] & 63u];
    else return (uint32_t)m.lut[(pb[u >> 2] >> (8 * (u & 3))) & 63u];
  };
  auto list_pay = [&](unsigned long long w, uint32_t i) -> uint32_t {
    return PK ? (uint32_t)m.lut[(uint32_t)w & 63u] : (uint32_t)m.lp[i];
  };
  // the key's level-0 bit in the group: its 32-bit hash scaled to the bin's
  // sw * 2^P words, minus the group's start, which is the hash without its
  // top Pg bits scaled to the group's words (exactly: the dropped bits' share
  // is a whole number of slices)
  auto bit_of = [&](unsigned long long w) -> uint32_t {
    const uint32_t x = PK ? (uint32_t)((w << (Pg - p1)) >> 32) & lowP : (uint32_t)((w * MS_HASH_MUL) >> 32) << Pg;
    return __umulhi(x, scale);
  };
  uint32_t *set32 = reinterpret_cast<uint32_t *>(m.set), *col32 = reinterpret_cast<uint32_t *>(m.col);
  uint32_t *set1w = reinterpret_cast<uint32_t *>(m.set1), *col1w = reinterpret_cast<uint32_t *>(m.col1);
  const uint16_t *cpre = reinterpret_cast<const uint16_t *>(m.cpre), *fpre = reinterpret_cast<const uint16_t *>(m.fpre),
                 *fpre1 = reinterpret_cast<const uint16_t *>(m.fpre1);
  __syncthreads();
  // 1. mark
  const uint32_t set_at = gd_shared(m.set), col_at = gd_shared(m.col);
  uint32_t hit = 0;
#pragma unroll
  for (int u = 0; u < GD_U; u++) {
    if (u * GD_BLOCK < n) {
      const uint32_t b = bit_of(key[u]), bm = 1u << (b & 31), w = (b >> 5) * 4;
      const uint32_t h = gd_or_if(act & (1u << u), set_at + w, bm) & bm;
      gd_red_or_if(h, col_at + w, bm);
      hit |= h;
    }
  }
  uint32_t cont = 0, k0 = 0;  // this thread's keys on a bit set more than once, and the first one's list entry
  uint32_t nl = 0;
  if (__syncthreads_or(hit != 0)) {
    // 2. the list, and the numbers of those bits (a warp a slice, one
    //    reservation each)
#pragma unroll
    for (int u = 0; u < GD_U; u++) {
      if (u * GD_BLOCK < n) {  // (lanes past the end test word 0; act drops them)
        const uint32_t b = bit_of(key[u]);
        cont |= ((col32[b >> 5] >> (b & 31)) & 1u) << u;
      }
    }
    cont &= act;
    // one reservation a warp: its list entries and its slices' bits
    unsigned long long x[SPW];
    uint32_t v = (uint32_t)__popc(cont), e[SPW];
#pragma unroll
    for (uint32_t r = 0; r < SPW; r++) {
      const uint32_t sl = warp + r * NW;
      x[r] = sl < subs && lane < sw ? m.col[sl * sw + lane] : 0ull;
      e[r] = (uint32_t)__popcll(x[r]);
    }
    static_assert(SPW == 2, "two slices a warp: one scan with the list, one of its own");
    uint32_t t0, t1;
    const uint32_t e0 = gd_warp_excl(v | (e[0] << 16), t0), e1 = gd_warp_excl(e[1], t1);
    uint32_t base = 0;
    if (lane == 0 && (t0 | t1)) base = atomicAdd(&m.nlc, t0 + (t1 << 16));
    base = __shfl_sync(FULL, base, 0);
    k0 = (base & 0xFFFFu) + (e0 & 0xFFFFu);
    if (k0 + v <= GD_MAXL) {
      uint32_t k = k0;
#pragma unroll
      for (int u = 0; u < GD_U; u++) {
        const bool c = (cont >> u) & 1;
        if (c) m.lk[k] = key[u];
        if constexpr (!PK)
          if (c) m.lp[k] = (uint8_t)pay_of(u);
        k += c;
      }
    }
    if (lane < sw) {
      const uint32_t c0 = base >> 16;
      if (warp < subs) m.cpre[warp * sw + lane] = gd_halves(x[0], c0 + (e0 >> 16));
      if (warp + NW < subs) m.cpre[(warp + NW) * sw + lane] = gd_halves(x[1], c0 + (t0 >> 16) + e1);
    }
    __syncthreads();
    nl = m.nlc & 0xFFFFu;
    if (nl > GD_MAXL) {  // uniform; nothing of the group was written
      if (tid == 0) ov[atomicAdd(ov_cnt, 1u)] = q;
      return;
    }
    for (uint32_t i = tid; i < nl; i += GD_BLOCK) {
      const unsigned long long w = m.lk[i];
      const uint32_t b = bit_of(w), bm = 1u << (b & 31);
      const uint32_t c = cpre[b >> 5] + (uint32_t)__popc(col32[b >> 5] & (bm - 1));  // below nl / 2
      m.lx[i] = (uint16_t)c;
      atomicMin(&m.rk[c], i);
      if (pay) atomicOr(&m.rp[c >> 2], list_pay(w, i) << (8 * (c & 3)));
    }
    __syncthreads();
    bool lbad = false;
    for (uint32_t i = tid; i < nl; i += GD_BLOCK) {
      const unsigned long long w = m.lk[i];
      const uint32_t f = m.rk[m.lx[i]];
      if (f != i && id(m.lk[f]) != id(w)) {
        const uint32_t b = bit_of(w);
        atomicAnd(&set32[b >> 5], ~(1u << (b & 31)));
        lbad = true;
      }
    }
    const bool anybad = __syncthreads_or((int)lbad) != 0;
    // 3. level 1
    bool hit1 = false;
    for (uint32_t i = tid; i < nl; i += GD_BLOCK) {
      const unsigned long long w = m.lk[i];
      const uint32_t b = bit_of(w);
      if (!anybad || ((set32[b >> 5] >> (b & 31)) & 1)) {
        const uint32_t c = m.lx[i];
        m.lx[i] = (uint16_t)(m.rk[c] == i ? GD_OWN | c : GD_NONE);
      } else {  // its bit there, from its own hash in its slice
        const uint32_t x = (uint32_t)((PK ? hi | (w >> p1) : w * MS_HASH_MUL) >> 32) << Pg;
        const uint32_t b1 = (g ? (x >> (32 - g)) * (sw1 << 6) : 0u) + bb_slice_pos(key_of(w), 1, sw1);
        const uint32_t bm1 = 1u << (b1 & 31);
        m.lx[i] = (uint16_t)b1;
        if (atomicOr(&set1w[b1 >> 5], bm1) & bm1) {
          hit1 = true;
          atomicOr(&col1w[b1 >> 5], bm1);
        }
      }
    }
    if (anybad && __syncthreads_or((int)hit1)) {
      // the few occurrences on a level-1 bit set more than once, pairwise
      for (uint32_t i = tid; i < nl; i += GD_BLOCK) {
        const uint32_t b1 = m.lx[i];
        if (b1 < GD_OWN && ((col1w[b1 >> 5] >> (b1 & 31)) & 1)) {
          const uint32_t o = atomicAdd(&m.nc, 1u);
          if (o < GD_MAXC) {
            const unsigned long long w = m.lk[i];
            m.cq[o] = (uint16_t)i;
            m.cb[o] = (uint16_t)b1;
            m.cid[o] = id(w);
            m.cp[o] = pay ? list_pay(w, i) : 0u;
          }
        }
      }
      __syncthreads();
      const uint32_t nc = m.nc;
      if (nc > GD_MAXC) {
        if (tid == 0) ov[atomicAdd(ov_cnt, 1u)] = q;
        return;
      }
      // (GD_PAIR threads an entry while there are enough)
      const uint32_t per = nc <= GD_BLOCK / GD_PAIR ? GD_PAIR : 1u, c = tid / per;
      unsigned long long v = 0;
      uint32_t b1 = GD_NONE, lead = GD_MAXC;  // the first copy of the entry's key
      bool bad = false;
      if (c < nc) {
        v = m.cid[c];
        b1 = m.cb[c];
        for (uint32_t j = tid % per; j < nc; j += per) {
          const bool on = m.cb[j] == b1, same = m.cid[j] == v;  // (equal keys have equal bits)
          bad |= on && !same;
          if (same) lead = min(lead, j);
        }
      }
      if (per > 1) {
#pragma unroll
        for (uint32_t o = 1; o < GD_PAIR; o <<= 1) {
          lead = min(lead, __shfl_xor_sync(FULL, lead, o));
          bad |= __shfl_xor_sync(FULL, (int)bad, o) != 0;
        }
      }
      if (c < nc && tid % per == 0) {
        if (bad) atomicAnd(&set1w[b1 >> 5], ~(1u << (b1 & 31)));
        if (lead != c) {
          atomicOr(&m.cp[lead], m.cp[c]);
          m.lx[m.cq[c]] = GD_NONE;
        } else {
          m.lx[m.cq[c]] = (uint16_t)(b1 | GD_JOIN);
        }
      }
      __syncthreads();
      // a key's first copy takes its copies' payloads
      if (tid < nc) m.lp[m.cq[tid]] = (uint8_t)m.cp[tid];
    }
  }
  // 4. the slices, with the placed bits of the slice before each word (a warp
  //    two slices, then the slices' bases)
  unsigned long long fin[SPW];
  uint32_t loc[SPW], st1 = 0;
  {
#pragma unroll
    for (uint32_t r = 0; r < SPW; r++) {
      const uint32_t sl = warp + r * NW;
      fin[r] = sl < subs && lane < sw ? m.set[sl * sw + lane] : 0ull;
    }
    uint32_t tot;
    const uint32_t e = gd_warp_excl((uint32_t)__popcll(fin[0]) | ((uint32_t)__popcll(fin[1]) << 16), tot);
    loc[0] = e & 0xFFFFu;
    loc[1] = e >> 16;
    if (lane == 0) {
      m.tot[warp] = tot & 0xFFFFu;
      m.tot[warp + NW] = tot >> 16;
    }
    if (lv0 && lane < sw) {
#pragma unroll
      for (uint32_t r = 0; r < SPW; r++) {
        const uint32_t sl = warp + r * NW;
        if (sl < subs) l0.AR[first + sl * sw + lane] = make_ulonglong2(fin[r], (unsigned long long)loc[r]);
      }
    }
    if (warp == NW - 1 && lane < subs)  // level 1: a slice a lane, its few words one after another
      for (uint32_t w = 0; w < sw1; w++) {
        const unsigned long long x = m.set1[lane * sw1 + w];
        if (lv0) l0.AR1[first1 + lane * sw1 + w] = make_ulonglong2(x, (unsigned long long)st1);
        m.fpre1[lane * sw1 + w] = gd_halves(x, st1);
        st1 += (uint32_t)__popcll(x);
      }
  }
  __syncthreads();
  const uint32_t st = lane < (1u << BITS) ? m.tot[lane] : 0u;
  uint32_t placed;
  const uint32_t sbase = gd_warp_excl(st, placed);
#pragma unroll
  for (uint32_t r = 0; r < SPW; r++) {
    const uint32_t sl = warp + r * NW, base = __shfl_sync(FULL, sbase, sl & 31);
    if (sl < subs && lane < sw) m.fpre[sl * sw + lane] = gd_halves(fin[r], base + loc[r]);
  }
  if (warp == NW - 1) {
    uint32_t p1s;
    const uint32_t sb1 = placed + gd_warp_excl(st1, p1s);  // level 1's bytes follow level 0's
    if (lane < subs) {
      for (uint32_t w = 0; w < sw1; w++) m.fpre1[lane * sw1 + w] += sb1 * 0x10001u;
      if (lv0) {
        const uint64_t j = ((uint64_t)q << g) + lane;
        l0.placed[j] = st;
        l0.placed1[j] = st1;
      }
    }
    if (lane == 0) {
      m.placed1 = p1s;
      if (lv0) {
        l0.uplaced[q] = placed;
        l0.uplaced1[q] = p1s;
      }
    }
  }
  __syncthreads();
  const uint32_t placed1 = m.placed1;
  // 5. the first copy of every key kept; each placed key's byte to its rank in
  //    the stage (rk's area: its last use was before the last barriers)
  //    from its alignment in l0pay on
  const uint32_t al = (uint32_t)(a & 3);
  uint8_t *stage = reinterpret_cast<uint8_t *>(m.rk) + al;
  uint32_t km = act;
  for (uint32_t t = cont; t; t &= t - 1)
    if (m.lx[k0++] == GD_NONE) km &= ~(t & (0u - t));
  const uint32_t own = lpay ? act & ~cont : 0u;
  uint32_t word = 0;  // lane u < GD_U: the warp's keep bits of row u
#pragma unroll
  for (int u = 0; u < GD_U; u++) {
    if (u * GD_BLOCK < n) {
      const unsigned bal = __ballot_sync(FULL, (km >> u) & 1);
      if (lane == u) word = bal;
      // (every lane's rank is in range; only keys with a bit of their own store)
      const uint32_t b = bit_of(key[u]), bm = 1u << (b & 31);
      const uint32_t r = fpre[b >> 5] + (uint32_t)__popc(set32[b >> 5] & (bm - 1));
      if ((own >> u) & 1) stage[r] = (uint8_t)pay_of(u);
    }
  }
  if (lane < GD_U && word) keep[gd_keep_word(a, q) + lane * NW + warp] = word;
  const uint32_t kept = __reduce_add_sync(FULL, (uint32_t)__popc(km));
  if (lane == 0 && kept) atomicAdd(&m.kept, kept);
  for (uint32_t i = tid; i < nl; i += GD_BLOCK) {
    const uint32_t x = m.lx[i];
    if (x == GD_NONE) continue;
    const unsigned long long w = m.lk[i];
    if (x & GD_OWN) {
      const uint32_t b = bit_of(w), bm = 1u << (b & 31);
      if (lpay)
        stage[fpre[b >> 5] + (uint32_t)__popc(set32[b >> 5] & (bm - 1))] =
            reinterpret_cast<const uint8_t *>(m.rp)[x & (GD_OWN - 1)];
    } else {
      const uint32_t b1 = x & (GD_JOIN - 1), bm1 = 1u << (b1 & 31), f = set1w[b1 >> 5];
      const uint8_t p = (x & GD_JOIN) ? m.lp[i] : (uint8_t)list_pay(w, i);
      if (f & bm1) {
        if (lpay) stage[fpre1[b1 >> 5] + (uint32_t)__popc(f & (bm1 - 1))] = p;
      } else if (lv0) {  // to the bin's level-2 list
        const unsigned long long o = atomicAdd(&l0.surv_cnt[bin], 1ull), s0 = l0.surv_off[bin];
        if (o < l0.surv_off[bin + 1] - s0) {
          l0.surv[s0 + o] = key_of(w);
          if (lpay) l0.surv_pay[s0 + o] = p;
        } else {
          atomicOr(l0.err, 1u);
        }
      }
    }
  }
  __syncthreads();
  if (tid == 0) cnt[q] = m.kept;
  if (lpay) {
    const uint32_t e = al + placed + placed1;  // bytes [al, e) of the words from a's
    uint8_t *out = l0.l0pay + (a - al);
    for (uint32_t w = tid; 4 * w < e; w += GD_BLOCK) {
      if (4 * w >= al && 4 * w + 4 <= e) reinterpret_cast<uint32_t *>(out)[w] = m.rk[w];
      else
        for (uint32_t i = max(4 * w, al); i < min(4 * w + 4, e); i++) out[i] = stage[i - al];
    }
  }
}

// Group bits of a split of P bits: groups of 16 while the split has at most
// GD_SPLIT bits then, else of 32; the whole bin where 32 hold it.
int gd_group_bits(int P) { return P <= GD_BITS ? P : P - 4 <= GD_SPLIT ? 4 : GD_BITS; }

// ---------------------------------------------------------------- repeats
// How much of the input repeats, for the group dedup's list: it has room for
// 72% (69%) of a group's occurrences, and copies of a key always share their
// bit, so groups near their capacity overflow it when most keys occur twice or
// more (reads at any coverage, assemblies of one species).  One to four bins,
// evenly spaced, the next one that is not empty: their keys in one 64th of the hash range mark a bitmap of 8
// bits an occurrence -- level 0's own density -- in global memory.  got: the
// keys marked, the bits set, the keys that share their bit.
constexpr uint32_t RP_CTAS = 512;  // of all bins
constexpr int RP_BITS = 6, RP_BLOCK = 512;
constexpr uint64_t RP_RANGE = 37;  // any of the 64
// Occurrences from which a look is taken: it costs 10-30 us, and below that a run
// with most of its groups left to the block kernel takes under a millisecond.
constexpr uint64_t RP_MIN = 8u << 20;
// Bins looked at: at most 1/16 of the keys, and two large ones tell as much as
// four (200 Mbp in 128 bins, 24 us for four of 1.6 M).
CF1_HD uint32_t rp_bins(uint64_t occ, uint32_t nbins) {
  return nbins < 32 ? 1 : nbins < 64 || occ / nbins > (1u << 19) ? 2 : 4;
}
CF1_HD uint64_t rp_words(uint64_t occ) { return (occ >> (RP_BITS + 2)) + 1; }  // u32 words of occ keys' bits
__global__ void __launch_bounds__(RP_BLOCK) rp_sample_kernel(const uint64_t *keys, const uint64_t *seg_off, uint32_t nbins,
                                                            uint32_t nb, uint32_t *set, uint32_t *col, unsigned long long *got) {
  const uint32_t per = RP_CTAS / nb, i = blockIdx.x / per, part = blockIdx.x % per;
  uint32_t bin = (uint32_t)((2ull * i + 1) * nbins / (2 * nb));
  // (a shard's bins are every shard_count-th one)
  for (const uint32_t stop = (uint32_t)((i + 1ull) * nbins / nb); bin + 1 < stop && seg_off[bin + 1] == seg_off[bin];) bin++;
  const uint64_t a = seg_off[bin], e = seg_off[bin + 1];
  const uint32_t words = (uint32_t)((e - a) >> (RP_BITS + 2));
  if (!words) return;
  __shared__ uint32_t sum[3];
  if (threadIdx.x < 3) sum[threadIdx.x] = 0;
  __syncthreads();
  uint32_t *s = set + (a >> (RP_BITS + 2)), *c = col + (a >> (RP_BITS + 2));
  uint32_t n = 0, bits = 0, shared = 0;
#pragma unroll 8
  for (uint64_t j = a + part * RP_BLOCK + threadIdx.x; j < e; j += per * RP_BLOCK) {
    const uint64_t h = keys[j] * MS_HASH_MUL;
    if (h >> (64 - RP_BITS) != RP_RANGE) continue;
    const uint32_t b = (uint32_t)(((h << RP_BITS >> 32) * (uint64_t)words) >> 27), bm = 1u << (b & 31);
    n++;
    if (!(atomicOr(&s[b >> 5], bm) & bm)) bits++;
    else shared += atomicOr(&c[b >> 5], bm) & bm ? 1 : 2;
  }
  n = warp_sum(n);
  bits = warp_sum(bits);
  shared = warp_sum(shared);
  if (lane_id() == 0 && n) {  // (an atomic a warp on three addresses of global memory would take most of the kernel)
    atomicAdd(&sum[0], n);
    atomicAdd(&sum[1], bits);
    atomicAdd(&sum[2], shared);
  }
  __syncthreads();
  if (threadIdx.x < 3 && sum[0]) atomicAdd(&got[threadIdx.x], (unsigned long long)sum[threadIdx.x]);
}

// Groups the dedup left: one CTA per listed group moves its keys (unpacked)
// and bytes from T / TP to the same range of U / UP, sub-bucket by
// sub-bucket, and writes the sub-buckets' offsets and list entries for the
// block kernel.
__global__ void __launch_bounds__(GD_MOVE) gd_split_kernel(const uint64_t *T, const uint8_t *TP, const uint64_t *goff,
                                                           const uint32_t *ov, int Pg, int P, int p1, uint64_t *U,
                                                           uint8_t *UP, uint64_t *sb_off, uint32_t *jlist) {
  __shared__ unsigned long long s_cnt[1 << GD_BITS], s_cur[1 << GD_BITS];
  const uint64_t q = ov[blockIdx.x], a = goff[q], e = goff[q + 1];
  const int g = P - Pg;
  const uint32_t subs = 1u << g, gi = (uint32_t)(q & ((1ull << Pg) - 1));
  const uint64_t hi = p1 ? (uint64_t)(gi >> (Pg - p1)) << (64 - p1) : 0;
  const unsigned tid = threadIdx.x;
  auto hash = [&](uint64_t x) -> uint64_t { return p1 ? hi | (x >> p1) : x * MS_HASH_MUL; };
  auto sub = [&](uint64_t h) -> uint32_t { return g ? (uint32_t)(h >> (64 - P)) & (subs - 1) : 0u; };
  // one atomic a sub-bucket of a warp's 32 keys: in tandem arrays most are
  // copies of one key (an atomic a key: 2 Mb of a 37-base unit 3.34 ms, 0.44
  // now, 5 Mb of one base 290 and 24)
  const unsigned lane = lane_id(), lt = lanemask_lt();
  if (tid < subs) s_cnt[tid] = 0;
  __syncthreads();
  for (uint64_t i0 = a + (tid - lane); i0 < e; i0 += GD_MOVE) {
    const uint32_t sb = i0 + lane < e ? sub(hash(T[i0 + lane])) : subs;
    const unsigned peers = __match_any_sync(FULL, sb);
    if (sb < subs && !(peers & lt)) atomicAdd(&s_cnt[sb], (unsigned long long)__popc(peers));
  }
  __syncthreads();
  if (tid == 0) {
    uint64_t run = a;
    for (uint32_t s = 0; s < subs; s++) {
      s_cur[s] = run;
      sb_off[(q << g) + s] = run;
      jlist[((uint64_t)blockIdx.x << g) + s] = (uint32_t)((q << g) + s);
      run += s_cnt[s];
    }
    sb_off[(q + 1) << g] = run;  // the next group's start: the same value if that group is listed too
  }
  __syncthreads();
  for (uint64_t i0 = a + (tid - lane); i0 < e; i0 += GD_MOVE) {
    const uint64_t i = i0 + lane, x = i < e ? T[i] : 0, h = hash(x);
    const uint32_t sb = i < e ? sub(h) : subs;
    const unsigned peers = __match_any_sync(FULL, sb);
    unsigned long long o = 0;
    if (sb < subs && !(peers & lt)) o = atomicAdd(&s_cur[sb], (unsigned long long)__popc(peers));
    o = __shfl_sync(FULL, o, __ffs(peers) - 1) + __popc(peers & lt);
    if (sb < subs) {
      U[o] = p1 ? h * KEY_SPREAD_INV : x;
      if (UP) UP[o] = (uint8_t)pay_byte(p1 ? (uint32_t)x : TP[i]);
    }
  }
}

// The listed groups' results back in the groups' form, one CTA each: the
// distinct keys the block kernel left at the sub-buckets' starts in U to the
// group's start in T (packed again when T is: p1), all of them kept, and the
// placed bytes it left in lp -- level 0's, then level 1's, sub-bucket by
// sub-bucket -- to l0pay.
__global__ void __launch_bounds__(GD_MOVE) gd_gather_kernel(const uint64_t *U, const uint8_t *lp, const uint64_t *goff,
                                                            const uint32_t *ov, int g, const uint64_t *sb_off,
                                                            const uint32_t *scnt, uint64_t *T, uint32_t *cnt,
                                                            uint32_t *keep, Level0Out l0, int p1) {
  const uint64_t q = ov[blockIdx.x], a0 = goff[q];
  uint64_t o = a0;
  for (uint64_t j = q << g; j < (q + 1) << g; j++) {
    const uint32_t c = scnt[j];
    const uint64_t a = sb_off[j];
    for (uint32_t i = threadIdx.x; i < c; i += GD_MOVE) T[o + i] = p1 ? (U[a + i] * MS_HASH_MUL) << p1 : U[a + i];
    o += c;
  }
  const uint64_t d = o - a0;
  if (threadIdx.x == 0) cnt[q] = (uint32_t)d;
  uint32_t *kw = keep + gd_keep_word(a0, q);
  for (uint64_t w = threadIdx.x; w * 32 < d; w += GD_MOVE)
    kw[w] = d - w * 32 >= 32 ? 0xFFFFFFFFu : (1u << (d - w * 32)) - 1;
  if (!l0.AR) return;
  o = a0;
  for (int l = 0; l < 2; l++) {
    const uint64_t start = o;
    for (uint64_t j = q << g; j < (q + 1) << g; j++) {
      const uint32_t c = l ? l0.placed1[j] : l0.placed[j];
      const uint64_t a = sb_off[j] + (l ? l0.placed[j] : 0u);
      if (lp)
        for (uint32_t i = threadIdx.x; i < c; i += GD_MOVE) l0.l0pay[o + i] = lp[a + i];
      o += c;
    }
    if (threadIdx.x == 0) (l ? l0.uplaced1 : l0.uplaced)[q] = (uint32_t)(o - start);
  }
}

// The dense array of the kept keys, one warp per group.
__global__ void __launch_bounds__(256) gd_compact_kernel(const uint64_t *T, const uint64_t *goff, const uint32_t *keep,
                                                        const uint64_t *out_off, uint64_t nunit, int Pg, int p1,
                                                        uint64_t *dist) {
  const uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= nunit) return;
  const uint64_t a = goff[q], n = goff[q + 1] - a, hi = p1 ? ((q & ((1ull << Pg) - 1)) >> (Pg - p1)) << (64 - p1) : 0;
  const uint32_t *kw = keep + gd_keep_word(a, q);
  const unsigned lane = lane_id(), lt = lanemask_lt();
  uint64_t o = out_off[q];
  for (uint64_t i = 0; i < n; i += 32) {
    const uint32_t k = kw[i >> 5];
    if ((k >> lane) & 1) {
      const uint64_t x = T[a + i + lane];
      dist[o + __popc(k & lt)] = p1 ? (hi | (x >> p1)) * KEY_SPREAD_INV : x;
    }
    o += __popc(k);
  }
}

// ---------------------------------------------------------------- warp dedup
// The unsorted (BBHash) form's dedup where sub-buckets are larger than the
// width rule's (bins of 14.7 M keys and more, whose split is capped at 16 bits,
// or a narrower split from the autotuner) and where sequence repeats at the
// widest split: one warp per sub-bucket and no block
// barriers: sub-buckets of a few hundred keys (the split of key *
// KEY_SPREAD_MUL spreads them evenly), a private 512-slot open-addressing set
// per warp in shared memory, and, with level 0 on, the sub-bucket's slice of
// BBHash level 0 marked, written and ranked by the same warp.  A warp takes
// runs of WD_RUN consecutive sub-buckets from a work counter (their offsets,
// keys and bins are then read in order, and uneven bins still balance).  A
// sub-bucket with more than WD_MAXD distinct keys (or a slice
// above WD_SWMAX words) is left untouched and listed in ov for the block
// kernel.
constexpr int WD_WARPS = 8;                 // warps per CTA
constexpr uint32_t WD_TW = 512;             // set slots per warp
constexpr uint32_t WD_MAXD = WD_TW / 4 * 3; // distinct keys a warp's set takes
constexpr uint32_t WD_SWMAX = 64;           // level-0 slice words a warp takes
constexpr uint32_t WD_SW1MAX = (WD_SWMAX + 7) / 8;  // level-1 slice words (an eighth of level 0's)
constexpr int WD_U = 4;                     // key loads in flight per lane
constexpr uint32_t WD_RUN = 64;             // sub-buckets a warp takes at a time
struct WdSmem {
  unsigned long long tab[WD_TW];
  unsigned long long set[WD_SWMAX], col[WD_SWMAX];     // level-0 slice: bits set, bits set twice
  unsigned long long set1[WD_SW1MAX], col1[WD_SW1MAX]; // level-1 slice
  uint8_t tpay[WD_TW];
  uint16_t ins[WD_MAXD];                    // the distinct keys' slots in insertion order
  uint8_t dp[WD_MAXD];                      // the distinct keys' joined payloads
  uint16_t pw[WD_SWMAX], pw1[WD_SW1MAX];    // placed bits before each word of the slices
};
static_assert(sizeof(WdSmem) % 8 == 0, "per-warp areas stay 8-byte aligned");

// PK: T holds packed words of a first pass of p1 bits (see pay_code); the
// set then holds each key's h = key * MS_HASH_MUL without its top p1 bits,
// level 0's bit comes from h directly, and the keys written back (T, the
// level-2 list) are h * KEY_SPREAD_INV.  TP is only written.
template <bool PK>
__global__ void __launch_bounds__(WD_WARPS * 32, 4) wd_dedup_kernel(uint64_t *T, uint8_t *TP, const uint64_t *sb_off,
                                                                   uint64_t nsub, int P, uint32_t *cnt, Level0Out l0,
                                                                   uint32_t *ov, uint32_t *ov_cnt, uint32_t *queue,
                                                                   int p1) {
  extern __shared__ __align__(16) unsigned char wd_smem[];
  WdSmem &m = reinterpret_cast<WdSmem *>(wd_smem)[threadIdx.x >> 5];
  const unsigned lane = lane_id(), lt = lanemask_lt();
  const unsigned long long EMPTY = ~0ull;  // above every key (keys use at most 62 bits)
  const bool pay = TP != nullptr, lv0 = l0.AR != nullptr, lpay = lv0 && l0.with_pay && pay;
  for (uint32_t i = lane; i < WD_TW; i += 32) {
    m.tab[i] = EMPTY;
    m.tpay[i] = 0;
  }
  __syncwarp();
  const uint64_t nruns = (nsub + WD_RUN - 1) / WD_RUN;
  for (;;) {
    uint32_t run = 0;
    if (lane == 0) run = atomicAdd(queue, 1u);
    run = __shfl_sync(FULL, run, 0);
    if (run >= nruns) break;
    const uint64_t j0 = (uint64_t)run * WD_RUN, j1 = j0 + WD_RUN < nsub ? j0 + WD_RUN : nsub;
    for (uint64_t j = j0; j < j1; j++) {
      const uint64_t a = sb_off[j], n = sb_off[j + 1] - a;
      const uint32_t bin = (uint32_t)(j >> P), sub = (uint32_t)(j & ((1ull << P) - 1));
      uint64_t W = 0, first = 0;
      uint32_t sw = 0;
      if (lv0) {
        W = l0.woff[bin + 1] - l0.woff[bin];
        sw = (uint32_t)(W >> P);
        first = l0.woff[bin] + (uint64_t)sub * sw;
      }
      bool over = lv0 && sw > WD_SWMAX;
      // PK: the h bits the sub-bucket's first-pass digit gives; a set entry
      // id stands for the key whose h is hi | id
      const uint64_t hi = PK ? (uint64_t)(sub >> (P - p1)) << (64 - p1) : 0;
      auto key_of = [&](unsigned long long id) -> uint64_t { return PK ? (hi | id) * KEY_SPREAD_INV : id; };
      auto l0_bit = [&](unsigned long long id) -> uint64_t {
        return PK ? (((uint64_t)(uint32_t)((hi | id) >> 32) * (uint32_t)W) >> 26) : bb_pos(id, 0, (uint32_t)W);
      };
      // 1. one copy of each key, its copies' payloads ORed (WD_U keys per lane
      //    loaded before the first is inserted).  Double hashing: the probe
      //    step is odd (so a probe sequence visits every slot) and comes from
      //    other bits of the same product, which keeps the runs a warp waits
      //    for (the longest of its 32 lanes) short at the set's load.  The
      //    first probes of a lane's WD_U keys are issued back to back; only
      //    the keys whose first slot held another key then walk on, one key
      //    index at a time.  (A key can find the set full only after more
      //    than WD_MAXD keys were claimed, so the sub-bucket goes to the block
      //    kernel anyway.)
      uint32_t d = 0;
      for (uint64_t base = 0; base < n && !over; base += 32 * WD_U) {
        unsigned long long key[WD_U];
        uint32_t p[WD_U], h[WD_U], stp[WD_U];
        bool claimed[WD_U], pend[WD_U];
  #pragma unroll
        for (int u = 0; u < WD_U; u++) {
          const uint64_t i = base + u * 32 + lane;
          if constexpr (PK) {
            const uint64_t w = i < n ? T[a + i] : 0;
            key[u] = i < n ? w >> p1 : EMPTY;
            p[u] = i < n ? pay_byte((uint32_t)w) : 0u;
          } else {
            key[u] = i < n ? T[a + i] : EMPTY;
            p[u] = (pay && i < n) ? pay_byte(TP[a + i]) : 0u;
          }
        }
  #pragma unroll
        for (int u = 0; u < WD_U; u++) {
          claimed[u] = pend[u] = false;
          h[u] = stp[u] = 0;
          if (key[u] != EMPTY) {
            const unsigned long long hk = key[u] * 0x9E3779B97F4A7C15ull;
            h[u] = (uint32_t)(hk >> 55);                                // top 9 bits: WD_TW = 512
            stp[u] = ((uint32_t)(hk >> 40) | 1u) & (WD_TW - 1);
            const unsigned long long old = atomicCAS(&m.tab[h[u]], EMPTY, key[u]);
            if (old == EMPTY || old == key[u]) {
              claimed[u] = old == EMPTY;
              if (pay) atomicOr(reinterpret_cast<uint32_t *>(m.tpay) + (h[u] >> 2), p[u] << (8 * (h[u] & 3)));
            } else {
              pend[u] = true;
              h[u] = (h[u] + stp[u]) & (WD_TW - 1);
            }
          }
        }
  #pragma unroll
        for (int u = 0; u < WD_U; u++) {
          if (over) break;  // the set stays below full: at most WD_MAXD + 32 * WD_U keys in it
          if (__any_sync(FULL, pend[u]) && pend[u]) {
            for (uint32_t probe = 1; probe < WD_TW; probe++) {
              const unsigned long long old = atomicCAS(&m.tab[h[u]], EMPTY, key[u]);
              if (old == EMPTY || old == key[u]) {
                claimed[u] = old == EMPTY;
                if (pay) atomicOr(reinterpret_cast<uint32_t *>(m.tpay) + (h[u] >> 2), p[u] << (8 * (h[u] & 3)));
                break;
              }
              h[u] = (h[u] + stp[u]) & (WD_TW - 1);
            }
          }
          const unsigned b = __ballot_sync(FULL, claimed[u]);
          const uint32_t r = d + __popc(b & lt);
          if (claimed[u] && r < WD_MAXD) m.ins[r] = (uint16_t)h[u];
          d += __popc(b);
          over = d > WD_MAXD;
        }
      }
      __syncwarp();
      if (over) {  // left to the block kernel: clear the whole set, list j
        for (uint32_t i = lane; i < WD_TW; i += 32) {
          m.tab[i] = EMPTY;
          m.tpay[i] = 0;
        }
        if (lane == 0) ov[atomicAdd(ov_cnt, 1u)] = (uint32_t)j;
        __syncwarp();
        continue;
      }
      const uint64_t lo_bit = (uint64_t)sub * sw * 64;
      if (lv0) {
        for (uint32_t w = lane; w < sw; w += 32) m.set[w] = m.col[w] = 0;
        __syncwarp();
      }
      // 2. the distinct keys (and bytes) to T[a, a + d); with level 0, each
      //    key's bit marked and its byte kept in dp, the key itself left in
      //    the set (ins[r] stays its slot) until step 5 empties it; a key's
      //    level-0 and level-1 bits are recomputed from it where needed
      bool bad = false;
      for (uint32_t r = lane; r < d; r += 32) {
        const uint32_t h = m.ins[r];
        const unsigned long long key = m.tab[h];
        const uint8_t pr = m.tpay[h];
        T[a + r] = key_of(key);
        if (pay) TP[a + r] = pr;
        m.tpay[h] = 0;
        if (lv0) {
          const uint64_t bpos = l0_bit(key) - lo_bit;
          if (bpos < (uint64_t)sw * 64) {
            const unsigned long long bit = 1ull << (bpos & 63);
            if (atomicOr(&m.set[bpos >> 6], bit) & bit) atomicOr(&m.col[bpos >> 6], bit);
          } else {
            bad = true;  // not this slice's key: cannot happen with the shared hash
          }
          m.dp[r] = pr;
        } else {
          m.tab[h] = EMPTY;
        }
      }
      if (lane == 0) cnt[j] = d;
      if (!lv0) {
        __syncwarp();
        continue;
      }
      if (__any_sync(FULL, bad) && lane == 0) atomicOr(l0.err, 1u);
      __syncwarp();
      // 3. the slice written; placed bits per word and their exclusive prefix
      //    (sw <= 64: two words a lane)
      const unsigned long long f0 = lane < sw ? m.set[lane] & ~m.col[lane] : 0ull;
      const unsigned long long f1 = lane + 32 < sw ? m.set[lane + 32] & ~m.col[lane + 32] : 0ull;
      const uint32_t c0 = (uint32_t)__popcll(f0), c1 = (uint32_t)__popcll(f1);
      const uint32_t i0 = warp_inclusive_scan(c0), i1 = warp_inclusive_scan(c1);
      const uint32_t t0 = __shfl_sync(FULL, i0, 31), placed = t0 + __shfl_sync(FULL, i1, 31);
      if (lane < sw) {
        m.pw[lane] = (uint16_t)(i0 - c0);
        l0.AR[first + lane] = make_ulonglong2(f0, (unsigned long long)(i0 - c0));
      }
      if (lane + 32 < sw) {
        m.pw[lane + 32] = (uint16_t)(t0 + i1 - c1);
        l0.AR[first + lane + 32] = make_ulonglong2(f1, (unsigned long long)(t0 + i1 - c1));
      }
      // 4. each key level 0 places: its byte to its rank, its slot emptied;
      //    each key it leaves marks its bit in the sub-bucket's level-1 slice
      //    (sw1 words, its bit from level 1's hash) and is moved to the front
      //    of ins / dp (nsv of them; a key's new index is never above its old
      //    one, and the warp reads a group before it writes it)
      const uint32_t sw1 = (uint32_t)((l0.woff1[bin + 1] - l0.woff1[bin]) >> P);
      const uint64_t first1 = l0.woff1[bin] + (uint64_t)sub * sw1;
      const bool l1ok = sw1 <= WD_SW1MAX;  // always: level 1 is sized from level 0
      if (lane < sw1 && l1ok) m.set1[lane] = m.col1[lane] = 0;
      __syncwarp();
      uint32_t nsv = 0;
      for (uint32_t r0 = 0; r0 < d; r0 += 32) {
        const uint32_t r = r0 + lane;
        bool lv = false;  // left by level 0
        uint32_t h = 0;
        uint8_t pr = 0;
        if (r < d) {
          h = m.ins[r];
          pr = m.dp[r];
          const unsigned long long key = m.tab[h];
          const uint64_t bpos = l0_bit(key) - lo_bit;
          if (bpos < (uint64_t)sw * 64) {
            const unsigned long long fin = m.set[bpos >> 6] & ~m.col[bpos >> 6], bit = 1ull << (bpos & 63);
            if (fin & bit) {
              if (lpay) l0.l0pay[a + m.pw[bpos >> 6] + (uint32_t)__popcll(fin & (bit - 1))] = pr;
              m.tab[h] = EMPTY;
            } else if (l1ok) {
              lv = true;
              const uint32_t q1 = bb_slice_pos(key_of(key), 1, sw1);
              const unsigned long long bit1 = 1ull << (q1 & 63);
              if (atomicOr(&m.set1[q1 >> 6], bit1) & bit1) atomicOr(&m.col1[q1 >> 6], bit1);
            } else {
              m.tab[h] = EMPTY;
            }
          } else {
            m.tab[h] = EMPTY;
          }
        }
        const unsigned lb = __ballot_sync(FULL, lv);
        __syncwarp();  // every lane's reads of this group before any lane's writes
        if (lv) {
          const uint32_t k = nsv + __popc(lb & lt);
          m.ins[k] = (uint16_t)h;
          m.dp[k] = pr;
        }
        nsv += __popc(lb);
        __syncwarp();
      }
      const unsigned long long g1 = (lane < sw1 && l1ok) ? m.set1[lane] & ~m.col1[lane] : 0ull;
      const uint32_t e1 = (uint32_t)__popcll(g1), k1 = warp_inclusive_scan(e1);
      const uint32_t placed1 = __shfl_sync(FULL, k1, 31);
      if (lane < sw1 && l1ok) {
        m.pw1[lane] = (uint16_t)(k1 - e1);
        l0.AR1[first1 + lane] = make_ulonglong2(g1, (unsigned long long)(k1 - e1));
      }
      if (lane == 0) {
        l0.placed[j] = placed;
        l0.placed1[j] = placed1;
      }
      // survivors of level 1: one reservation in the bin's list
      unsigned long long sbase = 0;
      const uint32_t nsurv = nsv - placed1;
      if (lane == 0 && (nsurv || !l1ok)) {
        if (l1ok) sbase = atomicAdd(&l0.surv_cnt[bin], (unsigned long long)nsurv);
        if (!l1ok || sbase + nsurv > l0.surv_off[bin + 1] - l0.surv_off[bin]) {
          atomicOr(l0.err, 1u);
          sbase = ~0ull;
        }
      }
      sbase = __shfl_sync(FULL, sbase, 0);
      __syncwarp();
      // 5. each key level 0 left: its byte to its level-1 rank or the key to
      //    level 2; the rest of the set emptied
      uint64_t so = l0.surv_off[bin] + sbase;
      for (uint32_t k0 = 0; k0 < nsv; k0 += 32) {
        const uint32_t k = k0 + lane;
        bool surv = false;
        unsigned long long key = 0;
        if (k < nsv) {
          const uint32_t h = m.ins[k];
          key = key_of(m.tab[h]);
          m.tab[h] = EMPTY;
          const uint32_t q1 = bb_slice_pos(key, 1, sw1);
          const unsigned long long fin1 = m.set1[q1 >> 6] & ~m.col1[q1 >> 6], bit1 = 1ull << (q1 & 63);
          if (fin1 & bit1) {
            if (lpay) l0.l0pay[a + placed + m.pw1[q1 >> 6] + (uint32_t)__popcll(fin1 & (bit1 - 1))] = m.dp[k];
          } else {
            surv = true;
          }
        }
        const unsigned sb = __ballot_sync(FULL, surv);
        if (surv && sbase != ~0ull) {
          const uint64_t at = so + __popc(sb & lt);
          l0.surv[at] = key;
          if (lpay) l0.surv_pay[at] = m.dp[k];
        }
        so += __popc(sb);
      }
      __syncwarp();
    }
  }
}

// Packed sub-buckets the warp dedup left to the block kernel, back to keys
// and payload bytes (one warp per listed sub-bucket).
__global__ void wd_unpack_kernel(uint64_t *T, uint8_t *TP, const uint64_t *sb_off, const uint32_t *ov,
                                 const uint32_t *ov_cnt, int P, int p1) {
  const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= *ov_cnt) return;
  const uint64_t j = ov[w], a = sb_off[j], n = sb_off[j + 1] - a;
  const uint32_t sub = (uint32_t)(j & ((1ull << P) - 1));
  const uint64_t hi = (uint64_t)(sub >> (P - p1)) << (64 - p1);
  for (uint64_t i = lane_id(); i < n; i += 32) {
    const uint64_t x = T[a + i];
    TP[a + i] = (uint8_t)pay_byte((uint32_t)x);
    T[a + i] = (hi | (x >> p1)) * KEY_SPREAD_INV;
  }
}

// Run plan of the sorted form: runs of consecutive sub-buckets packed
// greedily up to cap keys, a sub-bucket above cap keys being a run of its own.
// Stretches of up to 1024 sub-buckets (2^CP_BITS) of a bin are planned apart,
// which also keeps a run to the CS_BUCKETS sub-buckets its counting sort tells
// apart (sparse ranges of the key space -- canonical k-mers starting with
// TTT... -- hold thousands of near-empty ones at wide splits).  The runs of
// stretch q go to clist[q << bits ...] as first | end << 16, sub-buckets
// within the stretch; ccount[q] = how many.
// One warp per stretch walks its runs one after another: the end of a run is
// the last sub-bucket whose offset is within cap of the run's start, found by
// a 32-way search of the offsets (in shared memory, relative to the stretch's
// start).  Whole bins a warp left the device idle where bins are few: 200 Mbp
// in one bin, 2^16 sub-buckets, 17 ms.
constexpr int CP_BITS = 10;
static_assert(1u << CP_BITS <= CS_BUCKETS);
constexpr int CP_BLOCK = 256;
__global__ void __launch_bounds__(CP_BLOCK) cs_plan_kernel(const uint64_t *sb_off, int bits, uint32_t cap, uint32_t *clist,
                                                          uint32_t *ccount) {
  __shared__ uint64_t s_off[(1u << CP_BITS) + 1];
  const uint32_t b = blockIdx.x, per = 1u << bits;
  const uint64_t *o = sb_off + ((uint64_t)b << bits);
  for (uint32_t q = threadIdx.x; q <= per; q += CP_BLOCK) s_off[q] = o[q];
  __syncthreads();
  if (threadIdx.x >= 32) return;
  auto at = [&](uint32_t q) -> uint64_t { return s_off[q]; };
  const unsigned lane = lane_id();
  uint32_t *out = clist + ((uint64_t)b << bits);
  uint32_t nc = 0, start = 0;
  while (start < per) {
    // the largest end in (start, lim] with at(end) <= at(start) + cap; start + 1 at least
    const uint64_t top = at(start) + cap;
    uint32_t lo = start + 1, lim = per;  // at(lo) <= top or lo = start + 1
    while (lo < lim) {
      const uint32_t step = (lim - lo + 31) / 32;
      const uint32_t q = lo + (lane + 1) * step;
      const bool in = q <= lim && at(q) <= top;
      const unsigned m = __ballot_sync(FULL, in);  // a prefix of the lanes: the offsets do not decrease
      const uint32_t c = __popc(m), next = lo + c * step;
      lim = min(lim, lo + (c + 1) * step - 1);
      lo = next;
    }
    if (lane == 0) out[nc] = start | lo << 16;
    nc++;
    start = lo;
  }
  if (lane == 0) ccount[b] = nc;
}

// The stretches' runs one after another, as sub-buckets [x, y): one warp per
// stretch.
__global__ void __launch_bounds__(CP_BLOCK) cs_runs_kernel(const uint32_t *clist, const uint64_t *coff, uint32_t nstretch,
                                                          int bits, uint2 *runs) {
  const uint32_t b = (blockIdx.x * CP_BLOCK + threadIdx.x) >> 5;
  if (b >= nstretch) return;
  const uint64_t o = coff[b];
  const uint32_t n = (uint32_t)(coff[b + 1] - o), j0 = b << bits;  // (MAX_BINS << MSD_MAX_BITS sub-buckets fit)
  for (uint32_t r = lane_id(); r < n; r += 32) {
    const uint32_t x = clist[j0 + r];
    runs[o + r] = make_uint2(j0 + (x & 0xFFFFu), j0 + (x >> 16));
  }
}
static_assert((uint64_t)MAX_BINS << MSD_MAX_BITS <= 1ull << 28);

// One warp per sub-bucket or 32 (see warp_units): copy their distinct keys to
// the dense array.
template <class KeyT, bool MANY>
__global__ void cs_compact_kernel(const KeyT *T, const uint64_t *sb_off, const uint32_t *cnt, const uint64_t *out_off,
                                  uint64_t nsub, KeyT *dist) {
  warp_units<MANY>(cnt, 0, nsub, [&](uint64_t j, uint32_t c) {
    const uint64_t a = sb_off[j], o = out_off[j];
    for (uint32_t i = lane_id(); i < c; i += 32) dist[o + i] = T[a + i];
  });
}

__global__ void cs_bin_off_kernel(const uint64_t *out_off, uint32_t nbins, uint64_t per_bin, uint64_t *dist_off) {
  uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b <= nbins) dist_off[b] = out_off[(uint64_t)b * per_bin];
}

// Splits the segments of `in` into `out` on `bits` bits; sub_off[0 .. nseg <<
// bits] gets the sub-segments' offsets.
template <class KeyT>
void ms_pass(int bits, const KeyT *in, KeyT *out, uint64_t n, const uint64_t *seg_off, uint32_t nseg, int shift,
             bool hashed, uint64_t *sub_off, MsdScratch &sc, cudaStream_t s, const uint8_t *pin, uint8_t *pout,
             int pack = 0) {
  constexpr uint32_t TILE = ms_tile<KeyT>();
  if (bits < 1 || bits > MS_BITS) throw Error(-1, "MSD pass width must be 1..11 bits");
  const uint64_t nsub = (uint64_t)nseg << bits;
  uint32_t *tile_off = sc.tile_off.get<uint32_t>(2 * (nseg + 1)), *run_off = tile_off + nseg + 1;
  segment_tiles(seg_off, nseg, TILE, tile_off, s);
  segment_tiles(seg_off, nseg, TILE * MS_RUN, run_off, s);
  uint32_t *tot = sc.hist.get<uint32_t>(2 * nsub), *cursor = tot + nsub;
  CF1_CUDA(cudaMemsetAsync(tot, 0, 2 * nsub * sizeof(uint32_t), s));
  const size_t hsm = sizeof(uint32_t) << bits;
  ms_hist_kernel<KeyT><<<(unsigned)(ceil_div(n, TILE * MS_RUN) + nseg), MS_BLOCK, hsm, s>>>(in, seg_off, run_off, nseg,
                                                                                         shift, bits, hashed, tot);
  CF1_LAUNCH_CHECK();
  exclusive_scan_u32(tot, sub_off, nsub, sc.scan_tmp, s);
  const size_t smem = TILE * sizeof(KeyT) + ((sizeof(uint64_t) + sizeof(uint32_t)) << bits) + (pin ? TILE : 0);
  auto kern = ms_scatter_kernel<KeyT, false>;
  if constexpr (KOps<KeyT>::WORDS == 1)
    if (pack) kern = ms_scatter_kernel<KeyT, true>;
  // (the largest pass's, not this one's: the attribute is the function's on
  // the device, and another context may launch it at any width meanwhile)
  constexpr size_t MOST = TILE * sizeof(KeyT) + ((sizeof(uint64_t) + sizeof(uint32_t)) << MS_BITS) + TILE;
  CF1_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MOST));
  kern<<<(unsigned)(ceil_div(n, TILE) + nseg), MS_BLOCK, smem, s>>>(in, out, seg_off, tile_off, nseg, shift, bits, hashed,
                                                                   sub_off, cursor, pin, pout, pack);
  CF1_LAUNCH_CHECK();
}

}  // namespace

template <class KeyT>
void msd_compact(const KeyT *kept, uint64_t nsub, KeyT *dist, MsdScratch &sc, cudaStream_t s) {
  if (!nsub) return;
  if constexpr (KOps<KeyT>::WORDS == 1) {
    if (sc.kept_bits) {
      gd_compact_kernel<<<(unsigned)ceil_div(nsub * 32, 256), 256, 0, s>>>(
          kept, sc.sb_off.as<const uint64_t>(), sc.keep.as<const uint32_t>(), sc.out_off.as<const uint64_t>(), nsub,
          sc.unit_bits, sc.kept_packed, dist);
      CF1_LAUNCH_CHECK();
      return;
    }
  }
  const bool many = many_units(nsub);
  auto kern = many ? cs_compact_kernel<KeyT, true> : cs_compact_kernel<KeyT, false>;
  kern<<<(unsigned)ceil_div(nsub, many ? 256 : 8), 256, 0, s>>>(
      kept, sc.sb_off.as<const uint64_t>(), sc.cnt.as<const uint32_t>(), sc.out_off.as<const uint64_t>(), nsub, dist);
  CF1_LAUNCH_CHECK();
}

template <class KeyT>
int msd_prefix_bits(uint64_t max_bin_keys, bool sorted) {
  // Split on the key's own top bits (sorted), sub-buckets of the average bin
  // size run several times over it (the first bases of canonical k-mers are
  // skewed ~5x), so the aim is a quarter of what the rank dedup holds: the
  // sub-buckets it cannot hold go to the block kernel, which takes three
  // times as long per key (128-bit keys aimed at 2048, its whole capacity,
  // left it two fifths of them: 100 Mbp at k = 63 3.24 ms in the two kernels,
  // 2.13 ms now).
  // The unsorted 64-bit form (16 or 32 sub-buckets to a group)
  // aims at 192 for the largest bin.
  // 128-bit keys split by their hash are spread evenly: three quarters.
  const uint64_t target = sorted ? SrCfg<KeyT>::CAP / 4
                                 : KOps<KeyT>::WORDS == 1 ? WD_MAXD / 2 : SrCfg<KeyT>::CAP * 3 / 4;
  int p = 0;
  while (p < MSD_MAX_BITS && (max_bin_keys >> p) > target) p++;
  return p;
}

void msd_look_for_repeats(const uint64_t *keys, uint64_t n, const uint64_t *seg_off, uint32_t nbins, uint64_t *got,
                          MsdScratch &sc, cudaStream_t s) {
  // (bins past the widest split, on average, go without the group dedup anyway)
  if (n < RP_MIN || n / nbins > ((uint64_t)(GD_MAXSUB + 1) << MSD_MAX_BITS)) return;
  const uint64_t words = rp_words(n);
  uint32_t *set = sc.hist.get<uint32_t>(2 * words);  // free until the split
  CF1_CUDA(cudaMemsetAsync(set, 0, 2 * words * sizeof(uint32_t), s));
  rp_sample_kernel<<<RP_CTAS, RP_BLOCK, 0, s>>>(keys, seg_off, nbins, rp_bins(n, nbins), set, set + words,
                                               reinterpret_cast<unsigned long long *>(got));
  CF1_LAUNCH_CHECK();
}

bool msd_lists_overflow(const uint64_t *seg_off, uint32_t nbins, int P, const uint64_t *got) {
  if (!got[0]) return false;
  const int g = gd_group_bits(P);
  const double keys = (double)got[0], copies = keys / (double)got[1];
  uint64_t over = 0;
  for (uint32_t b = 0; b < nbins; b++) {
    const uint64_t occ = seg_off[b + 1] - seg_off[b];
    const double list = (double)got[2] / keys * std::ldexp((double)occ, g - P);
    if (list + 1.5 * std::sqrt(list * copies) > (g <= 4 ? GdCfg<4>::MAXL : GdCfg<5>::MAXL)) over += occ;
  }
  return over > (seg_off[nbins] - seg_off[0]) / 8;
}

template <class KeyT>
bool msd_sort_unique(KeyT *keys, KeyT *alt, uint64_t n, uint64_t max_bin, const uint64_t *seg_off, uint32_t nbins,
                     int key_bits, int P, KeyT *dist, uint64_t *dist_off, MsdScratch &sc, MsdRead &rd,
                     cudaStream_t s, bool sorted, const Level0Out *l0, KeyT **kept, uint8_t *pkeys, uint8_t *palt, uint8_t **kept_pay,
                     uint8_t **l0pay_buf, bool groups) {
  uint8_t *PT = pkeys;  // payloads beside T (nullptr: keys carry none)
  // passes on the top P bits: P1 then P2 (P2 may be 0) -- of the key, or of
  // its hash when only distinct keys are wanted (64-bit keys)
  const bool hashed = !sorted;
  constexpr bool W1 = KOps<KeyT>::WORDS == 1;
  if (hashed) key_bits = 64;
  else P = P < key_bits ? P : key_bits;  // short keys (k <= 7) have no more prefix bits than that
  // packed passes (see pay_code): the hashed split of keys with payloads
  // whose dedup builds BBHash level 0, with a first pass of >= 6 bits
  // Groups of 16 or 32 sub-buckets for the group dedup (see there), split on
  // the bits above theirs only, as long as the width rule's aim holds for the
  // largest bin: sub-buckets of at most WD_MAXD / 2 keys are three quarters of
  // what a group holds.
  // (At the widest split, bins of 12.6 to 14.7 M keys, up to 224: 32 of them
  // are 7168 of a group's 8192.  3.1 Gbp in 256 bins: 127 ms a run with the
  // warp sets, 106 with groups.)
  const bool grp = W1 && hashed && groups && (max_bin >> P) <= (P == MSD_MAX_BITS ? GD_MAXSUB : WD_MAXD / 2);
  const int g = grp ? gd_group_bits(P) : 0;
  const int PS = P - g;  // bits split on: a unit is a group, or a sub-bucket
  sc.unit_bits = PS;
  sc.kept_bits = false;
  const bool pk = W1 && hashed && pkeys && palt && l0 && l0->AR && l0->with_pay && PS >= (int)PACK_MIN_BITS;
  int P1 = PS > MS_BITS ? (PS + 1) / 2 : PS;
  if (pk && P1 < (int)PACK_MIN_BITS) P1 = PACK_MIN_BITS;
  const int P2 = PS - P1;
  KeyT *T = keys;
  const uint64_t nsub = (uint64_t)nbins << P, nunit = (uint64_t)nbins << PS;
  uint64_t *sb_off = sc.sb_off.get<uint64_t>(nunit + 1);  // the units' offsets
  if (PS == 0) {
    CF1_CUDA(cudaMemcpyAsync(sb_off, seg_off, (nbins + 1) * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s));
  } else if (n) {
    // sub-segments of pass 1: (bin, first digit), the segments of pass 2
    uint64_t *sb1 = P2 ? sc.sb_off1.get<uint64_t>(((uint64_t)nbins << P1) + 1) : sb_off;
    ms_pass<KeyT>(P1, keys, alt, n, seg_off, nbins, key_bits - P1, hashed, sb1, sc, s, pkeys, pk ? nullptr : palt,
                  pk ? P1 : 0);
    if (P2) {
      const uint32_t nseg2 = (uint32_t)((uint64_t)nbins << P1);
      if (pk)  // packed words: their own top bits are the next digit, the bytes travel inside
        ms_pass<KeyT>(P2, alt, keys, n, sb1, nseg2, 64 - P2, false, sb_off, sc, s, nullptr, nullptr);
      else
        ms_pass<KeyT>(P2, alt, keys, n, sb1, nseg2, key_bits - P1 - P2, hashed, sb_off, sc, s, palt, pkeys);
      T = keys;
      PT = pkeys;
    } else {
      T = alt;
      PT = palt;
    }
  } else {
    CF1_CUDA(cudaMemsetAsync(sb_off, 0, (nunit + 1) * sizeof(uint64_t), s));
  }
  uint32_t *cnt = sc.cnt.get<uint32_t>(nunit + 1);
  uint32_t *over = sc.flag.get<uint32_t>(1);
  CF1_CUDA(cudaMemsetAsync(over, 0, 4, s));
  int rest = key_bits - P;
  int bits = rest < CS_BITS ? rest : CS_BITS;
  int shift = rest - bits;
  if (bits <= 0) {
    bits = 1;  // every key of a sub-bucket is equal: one bucket
    shift = 0;
  }
  if (hashed) {  // the key's own bits: any bits split a sub-bucket into pieces
    bits = CS_BITS;
    shift = 0;
  }
  // S, hist, cur, pstart (u32) and the chunk bounds (u16)
  const uint32_t cap = cs_cap_for(KOps<KeyT>::WORDS == 2, sorted);
  const size_t smem_keys = cap * sizeof(KeyT) + (3 * CS_BUCKETS + 1) * sizeof(uint32_t) + (CS_BUCKETS + 2) * sizeof(uint16_t);
  const size_t smem = smem_keys + (pkeys || !sorted ? cap : 0);  // payloads; without them the unsorted form's l0_slice scratch
  auto kern = sorted ? cs_sort_unique_kernel<KeyT, true> : cs_sort_unique_kernel<KeyT, false>;
  // (with the payloads in any case, as ms_pass sets its own)
  CF1_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem_keys + cap)));
  KeyT *U = T == keys ? alt : keys;
  uint8_t *PU = pkeys ? (PT == pkeys ? palt : pkeys) : nullptr;
  if (l0pay_buf) *l0pay_buf = PU;
  uint32_t *ovc = sc.ovc.get<uint32_t>(2);  // overflow count, work counter
  CF1_CUDA(cudaMemsetAsync(ovc, 0, 2 * sizeof(uint32_t), s));
  // the units' counts scanned and all results read back with one wait; once
  // more when the block kernel had to take what the dedup left
  uint64_t *out_off = sc.out_off.get<uint64_t>(nunit + 1);
  auto finish = [&] {
    exclusive_scan_u32(cnt, out_off, nunit, sc.scan_tmp, s);
    cs_bin_off_kernel<<<(unsigned)ceil_div(nbins + 1, 256), 256, 0, s>>>(out_off, nbins, 1ull << PS, dist_off);
    CF1_LAUNCH_CHECK();
    CF1_CUDA(cudaMemcpyAsync(&rd.n_distinct, dist_off + nbins, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    CF1_CUDA(cudaMemcpyAsync(&rd.overflow, ovc, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CF1_CUDA(cudaMemcpyAsync(&rd.oversize, over, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    if (l0 && l0->AR) CF1_CUDA(cudaMemcpyAsync(&rd.l0_err, l0->err, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CF1_CUDA(cudaStreamSynchronize(s));
  };
  if (nsub) {
    Level0Out lo;
    if (l0 && hashed) lo = *l0;
    lo.with_pay = lo.with_pay && PT != nullptr;
    lo.l0pay = PU;
    for (auto &e : sc.ev)
      if (!e) CF1_CUDA(cudaEventCreate(&e));
    // sorted form (and 128-bit keys): consecutive small sub-buckets of a bin are packed into
    // one CTA's run (the top bits of canonical k-mers are skewed, so most
    // sub-buckets are far below the capacity the largest ones need)
    uint2 *runs = nullptr;
    uint64_t grid = nsub;
    if ((sorted || !W1) && P > 0) {
      const int sbits = P < CP_BITS ? P : CP_BITS;
      const uint32_t nstretch = (uint32_t)(nsub >> sbits);
      uint32_t *cl = sc.clist.get<uint32_t>(nsub);
      uint32_t *cc = sc.ccount.get<uint32_t>(nstretch + 1);
      uint64_t *co = sc.coff.get<uint64_t>(nstretch + 1);
      // runs the rank dedup holds; also at most 2/3 of the block kernel's
      // capacity, whose shared-memory set (a power of two >= 1.5 n slots,
      // filled to 3/4 at most) then always holds one
      static_assert(SrCfg<uint64_t>::CAP <= cs_cap_for(false, true) * 2 / 3 && SrCfg<Key2>::CAP <= cs_cap_for(true, true) * 2 / 3);
      cs_plan_kernel<<<nstretch, CP_BLOCK, 0, s>>>(sb_off, sbits, SrCfg<KeyT>::CAP, cl, cc);
      CF1_LAUNCH_CHECK();
      exclusive_scan_u32(cc, co, nstretch, sc.scan_tmp, s);
      CF1_CUDA(cudaMemcpyAsync(&rd.runs, co + nstretch, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
      CF1_CUDA(cudaStreamSynchronize(s));
      grid = rd.runs;
      runs = sc.runs.get<uint2>(grid);
      cs_runs_kernel<<<(unsigned)ceil_div((uint64_t)nstretch * 32, CP_BLOCK), CP_BLOCK, 0, s>>>(cl, co, nstretch, sbits, runs);
      CF1_LAUNCH_CHECK();
    }
    CF1_CUDA(cudaEventRecord(sc.ev[0], s));
    if (grp) {
      // one CTA per group; the groups it cannot hold go to the block kernel
      // sub-bucket by sub-bucket, through the free buffers
      uint32_t *ov = sc.ov.get<uint32_t>(nunit + 1);
      const bool small = g <= 4;
      auto gkern = small ? (pk ? gd_dedup_kernel<true, 4> : gd_dedup_kernel<false, 4>)
                         : (pk ? gd_dedup_kernel<true, 5> : gd_dedup_kernel<false, 5>);
      const size_t gsm = small ? sizeof(GdSmem<4>) : sizeof(GdSmem<5>);
      const int gblock = small ? GdCfg<4>::BLOCK : GdCfg<5>::BLOCK;
      CF1_CUDA(cudaFuncSetAttribute(gkern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gsm));
      uint64_t *T64 = reinterpret_cast<uint64_t *>(T), *U64 = reinterpret_cast<uint64_t *>(U);
      // a bit per occurrence: the first copy of its key (words of groups
      // that keep nothing there stay 0)
      const uint64_t nkeep = n / 32 + nunit + 1;
      uint32_t *keep = sc.keep.get<uint32_t>(nkeep);
      CF1_CUDA(cudaMemsetAsync(keep, 0, nkeep * sizeof(uint32_t), s));
      const int p1 = pk ? P1 : 0;
      gkern<<<(unsigned)nunit, gblock, gsm, s>>>(T64, PT, sb_off, PS, P, cnt, keep, lo, ov, ovc, p1);
      CF1_LAUNCH_CHECK();
      CF1_CUDA(cudaEventRecord(sc.ev[1], s));
      finish();
      const uint32_t h_ov = rd.overflow;
      const unsigned nov = h_ov << g;  // sub-buckets
      sc.last_overflow = nov;
      sc.kept_packed = p1;
      sc.kept_bits = true;
      if (h_ov) {
        uint64_t *sub_off = sc.sub_off.get<uint64_t>(nsub + 1);
        uint32_t *scnt = sc.sub_cnt.get<uint32_t>(nsub + 1), *jl = sc.jlist.get<uint32_t>(nov);
        Level0Out lb = lo;
        // the placed bytes go to PT, whose bytes of these groups have moved to
        // PU: a sub-bucket's are the block kernel's scratch until its slice
        lb.l0pay = PT;
        gd_split_kernel<<<h_ov, GD_MOVE, 0, s>>>(T64, PT, sb_off, ov, PS, P, p1, U64, PU, sub_off, jl);
        CF1_LAUNCH_CHECK();
        kern<<<nov, CS_BLOCK, smem, s>>>(U, T, sub_off, nsub, shift, rest > 0 ? bits : 0, scnt, over, P, lb, PU, PT,
                                         nullptr, jl, nullptr, false);
        CF1_LAUNCH_CHECK();
        gd_gather_kernel<<<h_ov, GD_MOVE, 0, s>>>(U64, lo.with_pay ? lb.l0pay : nullptr, sb_off, ov, g, sub_off, scnt,
                                                   T64, cnt, keep, lo, p1);
        CF1_LAUNCH_CHECK();
        CF1_CUDA(cudaEventRecord(sc.ev[1], s));
        finish();
      }
    } else if (W1 && hashed) {
      // the unsorted form: one warp per sub-bucket; the few it cannot hold
      // (more than WD_MAXD distinct keys) go to the block kernel after it
      uint32_t *ov = sc.ov.get<uint32_t>(nsub + 1);
      const size_t wsm = WD_WARPS * sizeof(WdSmem);
      auto wkern = pk ? wd_dedup_kernel<true> : wd_dedup_kernel<false>;
      CF1_CUDA(cudaFuncSetAttribute(wkern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wsm));
      const unsigned wgrid = persistent_grid(wkern, WD_WARPS * 32, wsm, -1, ceil_div(nsub, WD_WARPS));
      wkern<<<wgrid, WD_WARPS * 32, wsm, s>>>(reinterpret_cast<uint64_t *>(T), PT, sb_off, nsub, P, cnt, lo, ov, ovc,
                                              ovc + 1, pk ? P1 : 0);
      CF1_LAUNCH_CHECK();
      CF1_CUDA(cudaEventRecord(sc.ev[1], s));
      finish();
      const uint32_t h_ov = rd.overflow;
      sc.last_overflow = h_ov;
      if (h_ov && pk) {  // the block kernel takes keys and bytes
        wd_unpack_kernel<<<(unsigned)ceil_div((uint64_t)h_ov * 32, 256), 256, 0, s>>>(
            reinterpret_cast<uint64_t *>(T), PT, sb_off, ov, ovc, P, P1);
        CF1_LAUNCH_CHECK();
      }
      if (h_ov) {
        kern<<<h_ov, CS_BLOCK, smem, s>>>(T, U, sb_off, nsub, shift, rest > 0 ? bits : 0, cnt, over, P, lo, PT, PU,
                                          nullptr, ov, nullptr, !pk);
        CF1_LAUNCH_CHECK();
        CF1_CUDA(cudaEventRecord(sc.ev[1], s));
        finish();
      }
    } else {
      // a CTA per run; the runs it cannot hold go to the block kernel
      uint32_t *ov = sc.ov.get<uint32_t>(grid + 1);
      const size_t ssm = sizeof(SrSmem<KeyT>);
      auto skern = hashed && !W1 ? sr_dedup_kernel<KeyT, !W1> : sr_dedup_kernel<KeyT, false>;
      CF1_CUDA(cudaFuncSetAttribute(skern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm));
      skern<<<(unsigned)grid, SR_BLOCK, ssm, s>>>(T, PT, sb_off, nsub, P, hashed ? 32 - P : rest > 0 ? rest : 0, cnt, runs,
                                                 ov, ovc);
      CF1_LAUNCH_CHECK();
      CF1_CUDA(cudaEventRecord(sc.ev[1], s));
      finish();
      const uint32_t h_ov = rd.overflow;
      if (h_ov) {
        kern<<<h_ov, CS_BLOCK, smem, s>>>(T, U, sb_off, nsub, shift, rest > 0 ? bits : 0, cnt, over, P, lo, PT, PU, runs,
                                          nullptr, ov, true);
        CF1_LAUNCH_CHECK();
        CF1_CUDA(cudaEventRecord(sc.ev[1], s));
        finish();
      }
    }
  } else {
    finish();
  }
  sc.ms_dedup = 0;
  if (nsub) CF1_CUDA(cudaEventElapsedTime(&sc.ms_dedup, sc.ev[0], sc.ev[1]));
  if (rd.oversize) return false;
  if (kept) *kept = T;
  if (kept_pay) *kept_pay = grp ? nullptr : PT;
  if (dist) msd_compact<KeyT>(T, nunit, dist, sc, s);
  return true;
}

#define CF1_INST(KT)                                                                                              \
  template int msd_prefix_bits<KT>(uint64_t, bool);                                                                     \
  template bool msd_sort_unique<KT>(KT *, KT *, uint64_t, uint64_t, const uint64_t *, uint32_t, int, int, KT *,   \
                                    uint64_t *, MsdScratch &, MsdRead &, cudaStream_t, bool, const Level0Out *, KT **, uint8_t *, \
                                    uint8_t *, uint8_t **, uint8_t **, bool);                                 \
  template void msd_compact<KT>(const KT *, uint64_t, KT *, MsdScratch &, cudaStream_t);
CF1_INST(uint64_t)
CF1_INST(Key2)
#undef CF1_INST

}  // namespace cf1
