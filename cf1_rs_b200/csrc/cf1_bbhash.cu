// Per-bin GPU BBHash construction (the "plain" MPHF of this library).
//
// The reference builds one ph::fmph::Function over all distinct keys
// (src/mphf.rs:144-190; BBHash-style levels with relative_level_size 200).
// Here every bin gets its own levels so that phase 4, which walks the bins in
// order, touches one bin's bit arrays at a time.  Per level, over the keys not
// yet placed:
//   mark   : set the key's bit with atomicOr; a key that finds its bit set
//            marks the collision array instead;
//   clean  : bits that collided are cleared; a popcount prefix gives ranks;
//   filter : keys whose bit survived are placed, the rest go to the next level.
// The last levels, which have few keys, run in one launch (bb_tail_kernel).
// A bin's local slot of a key placed at level l is the number of keys of the
// bin placed at earlier levels plus the key's rank inside its level block.
// All levels live in one array of {bit word, level rank} entries, addressed
// through the per-(level, bin) BBMeta table.
#include <algorithm>
#include <cstring>

#include "../../include/cf1gpu.h"
#include "cf1_bbhash.cuh"
#include "cf1_device_util.cuh"
#include "cf1_mphf.cuh"

namespace cf1 {

namespace {

constexpr int BB_BLOCK = 256;
constexpr uint32_t BB_TILE = 4096;

// Keys of bin b at level 0: all its distinct keys when selected.
__global__ void bb_init_counts_kernel(const uint64_t *seg_off, const uint32_t *sel, uint32_t nbins, uint64_t *cnt) {
  uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nbins) cnt[b] = (sel == nullptr || sel[b]) ? seg_off[b + 1] - seg_off[b] : 0;
}

// Bits per key of a level: 8 at every level (ph::fmph uses gamma 2,
// src/mphf.rs:155-160).  A wide level places ~88% of its keys instead of
// ~61%, so a query -- and a warp of queries, which waits for its deepest
// lane -- walks fewer levels, and the build runs fewer.  At 2.7e9 keys the
// first level costs ~6.1 GB of HBM and the rest ~0.8 GB.  Measured at 3.1
// Gbp: 4 bits at level 0 ran phases 1-4 3% slower, 16 bits 1% slower (its
// first level's passes outweigh the shorter probes); 8 bits after level 0
// instead of 2 took the classification kernel from 50.9 to 46.3 ms and the
// build from 21.8 to 18.1 ms (16 levels down to 10).
constexpr uint32_t BB_GAMMA0 = 8, BB_GAMMA = 8;

// Words of each bin's block at this level (gamma bits per key, at least one
// word for a non-empty bin), the level's totals {keys, words} and the keys of
// its largest bin.
__global__ void bb_sizes_kernel(const uint64_t *cnt, uint32_t nbins, uint32_t gamma, uint64_t *wcnt,
                                unsigned long long *tot) {
  uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  uint64_t n = 0, words = 0;
  if (b < nbins) {
    n = cnt[b];
    words = n ? (gamma * n + 63) / 64 : 0;
    wcnt[b] = words;
  }
  const uint32_t largest = __reduce_max_sync(FULL, (uint32_t)n);  // (bins hold < 2^32 keys)
  n = warp_sum(n);
  words = warp_sum(words);
  if (lane_id() == 0 && (n | words)) {
    atomicMax(&tot[2], (unsigned long long)largest);
    atomicAdd(&tot[0], (unsigned long long)n);
    atomicAdd(&tot[1], (unsigned long long)words);
  }
}

// Marks every key's bit in this level's block of its bin.  The entry's rank
// half (y) collects the bits that more than one key set; AR points at this
// level's first entry and woff are the level-relative block offsets.  Keys
// of bin b are rem[start[b], start[b] + cnt[b]).
//
// When a tile's keys fall in a narrow stretch of the block -- at level 0 the
// unsorted phase-3 output is ordered by the same hash's top bits -- the tile
// marks a shared-memory copy of that stretch and merges it with one atomicOr
// per word (and one more per word with a collision) instead of one per key.
// Each key is hashed once (its position waits in a register for the stretch
// to be known): 100 M 128-bit keys in hash order, levels 0 and 1, 1.27 ->
// 0.78 ms; in key order the same keys took 2.84 ms, an atomic each.
constexpr uint32_t BB_WIN = 2048;  // words of the shared-memory stretch
constexpr int BB_ITEMS = BB_TILE / BB_BLOCK;
template <class KeyT>
__global__ void __launch_bounds__(BB_BLOCK) bb_mark_kernel(const KeyT *rem, const uint64_t *start, const uint64_t *cnt,
                                                           const uint32_t *tile_off, uint32_t nbins,
                                                           const uint64_t *woff, uint32_t level, ulonglong2 *AR) {
  __shared__ unsigned long long s_set[BB_WIN], s_col[BB_WIN];
  __shared__ uint32_t s_lo, s_hi;
  const uint32_t t = blockIdx.x;
  if (t >= tile_off[nbins]) return;
  TileSpan sp = tile_span_gapped(start, cnt, tile_off, nbins, t, BB_TILE);
  const uint64_t w0 = woff[sp.seg];
  const uint32_t nw = (uint32_t)(woff[sp.seg + 1] - w0);
  if (threadIdx.x == 0) {
    s_lo = ~0u;
    s_hi = 0;
  }
  __syncthreads();
  uint32_t word[BB_ITEMS];  // word of the block
  uint32_t bits[(BB_ITEMS + 3) / 4];  // the bit in it, four to a register
  uint32_t lo = ~0u, hi = 0;
#pragma unroll
  for (int i = 0; i < (BB_ITEMS + 3) / 4; i++) bits[i] = 0;
#pragma unroll
  for (int j = 0; j < BB_ITEMS; j++) {
    const uint64_t i = sp.start + (uint64_t)j * BB_BLOCK + threadIdx.x;
    word[j] = ~0u;
    if (i < sp.end) {
      const uint64_t pos = bb_pos(bb_key_hash(rem[i]), level, nw);
      word[j] = (uint32_t)(pos >> 6);
      bits[j >> 2] |= (uint32_t)(pos & 63) << (8 * (j & 3));
      lo = min(lo, word[j]);
      hi = max(hi, word[j]);
    }
  }
  lo = __reduce_min_sync(FULL, lo);
  hi = __reduce_max_sync(FULL, hi);
  if (lane_id() == 0) {
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
  }
  __syncthreads();
  const uint32_t wlo = s_lo, span = s_hi >= s_lo ? s_hi - s_lo + 1 : 0;
  const bool local = span > 0 && span <= BB_WIN;
  if (local) {
    for (uint32_t j = threadIdx.x; j < span; j += BB_BLOCK) s_set[j] = s_col[j] = 0;
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < BB_ITEMS; j++) {
    if (word[j] == ~0u) continue;
    const uint32_t b = (bits[j >> 2] >> (8 * (j & 3))) & 63, half = b >> 5, bit = 1u << (b & 31);
    if (local) {
      const uint32_t x = 2 * (word[j] - wlo) + half;
      if (atomicOr(reinterpret_cast<uint32_t *>(s_set) + x, bit) & bit)
        atomicOr(reinterpret_cast<uint32_t *>(s_col) + x, bit);
    } else {
      uint32_t *e = reinterpret_cast<uint32_t *>(AR + w0 + word[j]) + half;
      if (atomicOr(e, bit) & bit) atomicOr(e + 2, bit);
    }
  }
  if (!local) return;
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < span; j += BB_BLOCK) {
    const unsigned long long set = s_set[j];
    if (!set) continue;
    ulonglong2 *e = AR + w0 + wlo + j;
    const unsigned long long col = s_col[j] | (atomicOr(&e->x, set) & set);
    if (col) atomicOr(&e->y, col);
  }
}

// Clears the bits set by more than one key; popcount per word for the ranks.
__global__ void bb_clean_kernel(ulonglong2 *AR, uint32_t *pc, uint64_t nw) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nw) {
    ulonglong2 e = AR[i];
    uint64_t a = e.x & ~e.y;
    AR[i].x = a;
    pc[i] = (uint32_t)__popcll(a);
  }
}

__global__ void bb_rank_kernel(ulonglong2 *AR, const uint64_t *R, uint64_t nw) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nw) AR[i].y = R[i];
}

__global__ void bb_meta_kernel(const uint64_t *woff, const uint64_t *R, uint64_t level_base, uint64_t *base,
                               BBMeta *meta, uint32_t nbins) {
  uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nbins) return;
  uint64_t w0 = woff[b], w1 = woff[b + 1];
  BBMeta m;
  m.word_off = level_base + w0;
  m.nwords = (uint32_t)(w1 - w0);
  m.rank_adj = (uint32_t)(base[b] - R[w0]);
  meta[b] = m;
  base[b] += R[w1] - R[w0];
}

// Levels 0 and 1 as the phase-3 dedup left them (sliced, see BBView): each
// entry holds {placed bits, placed bits of its slice before it}.  One CTA per
// bin scans the bin's slices' placed counts (slices [b << P, (b + 1) << P))
// into srank -- the placed keys of the bin's slices before the slice -- and
// writes the bin's metadata, whose rank adjustment is the keys its earlier
// levels placed.
constexpr int BF_BLOCK = 1024;
__global__ void __launch_bounds__(BF_BLOCK) bb_sliced_kernel(const uint64_t *woff0, const uint64_t *woff1, int P,
                                                             uint64_t words0, const uint32_t *placed0,
                                                             const uint32_t *placed1, uint32_t *srank0,
                                                             uint32_t *srank1, uint64_t *base, BBMeta *meta,
                                                             uint32_t nbins) {
  __shared__ uint32_t sm[BF_BLOCK / 32];
  const uint32_t b = blockIdx.x, tid = threadIdx.x, ns = 1u << P;
  uint32_t before = 0;  // keys the bin's earlier levels placed (bins hold < 2^32 keys)
  for (int l = 0; l < 2; l++) {
    const uint32_t *placed = (l ? placed1 : placed0) + ((uint64_t)b << P);
    uint32_t *srank = (l ? srank1 : srank0) + ((uint64_t)b << P);
    const uint64_t *woff = l ? woff1 : woff0;
    uint32_t carry = 0;
    for (uint32_t j0 = 0; j0 < ns; j0 += 4 * BF_BLOCK) {  // four consecutive slices a thread
      const uint32_t j = j0 + 4 * tid;
      uint32_t v[4], c = 0;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        v[i] = j + i < ns ? placed[j + i] : 0u;
        c += v[i];
      }
      uint32_t tot;
      uint32_t pre = carry + block_exclusive_scan<BF_BLOCK>(c, sm, tot);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (j + i < ns) srank[j + i] = pre;
        pre += v[i];
      }
      carry += tot;
    }
    if (tid == 0) {
      BBMeta m;
      m.word_off = (l ? words0 : 0) + woff[b];
      m.nwords = (uint32_t)(woff[b + 1] - woff[b]);
      m.rank_adj = before;
      meta[(uint64_t)l * nbins + b] = m;
    }
    before += carry;
  }
  if (tid == 0) base[b] = before;
}

// The last levels, one CTA per bin, all of them in one launch: per level the
// bin's keys mark its block, the collided bits are cleared and ranked (ranks
// count from the block's start, the rank adjustment is the keys earlier levels
// placed) and the keys left go on.  Level l's keys are rem0 (l = l0), then r0
// / r1 in turn, at start[b].  Bin b's blocks lie in entries [off[b],
// off[b + 1]) from ar_base, one level after another; what is left of them is
// cleared.  Blocks up to BF_WORDS words are marked in shared memory.
//
// Launched once the keys left are few (BF_KEYS a bin on average: a level of
// that many keys takes the CTA ~15 us, and one launch of its own ~55 us with
// the wait for its size) and no bin has more than four times that, which its
// CTA would walk alone while the device idles (20 M 63-mers in one of 2048
// bins: 61 ms, the MPHF phase 0.7 ms with their large levels launched apart).
// A run's MPHF phase, nine launches and a wait per level before: 30 kb 240 ->
// 49 us, 200 Mbp 586 -> 87 us.
constexpr uint32_t BF_WORDS = 4096;
constexpr uint64_t BF_KEYS = 16384, BF_LARGEST = 4 * BF_KEYS;
// Entries reserved for n keys: the levels' blocks sum up to ~1.14 times the
// first one's words and a word a level.  Keys that a level's hash crowds
// together -- thousands of one sub-bucket, which share level 0's top bits --
// pass most of them on and need more: DEV_BB_ROOM, and the run is repeated
// with a launch a level (one_launch off), each sized by its keys.
CF1_HD uint64_t bf_room(uint64_t n) {
  const uint64_t w = (8 * n + 63) / 64;
  return n ? w + w / 4 + BB_MAX_LEVELS : 0;
}
__global__ void bb_room_kernel(const uint64_t *cnt, uint32_t nbins, uint64_t *room) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nbins) room[b] = bf_room(cnt[b]);
}
template <class KeyT>
__global__ void __launch_bounds__(BF_BLOCK) bb_tail_kernel(const KeyT *rem0, KeyT *r0, KeyT *r1, const uint64_t *start,
                                                           const uint64_t *cnt, uint32_t nbins, uint32_t l0,
                                                           ulonglong2 *AR, const uint64_t *off, uint64_t ar_base,
                                                           uint64_t ar_cap, const uint64_t *base, BBMeta *meta,
                                                           unsigned long long *got, uint32_t *err) {
  extern __shared__ __align__(16) unsigned long long bf_bits[];  // set, col
  __shared__ uint32_t sm[BF_BLOCK / 32];
  const uint32_t b = blockIdx.x, tid = threadIdx.x;
  const uint64_t region = ar_base + off[b], room = off[b + 1] - off[b], s0 = start[b];
  uint64_t n = cnt[b], used = 0;
  if (!n) return;
  if (region + room > ar_cap) {
    if (tid == 0) atomicOr(err, (uint32_t)DEV_OVERFLOW);
    return;
  }
  uint32_t before = (uint32_t)base[b], l = l0;
  const KeyT *rem = rem0 + s0;
  unsigned long long *set = bf_bits, *col = bf_bits + BF_WORDS;
  for (; n; l++) {
    const uint64_t nw = (8 * n + 63) / 64;
    if (l >= BB_MAX_LEVELS || used + nw > room) {
      if (tid == 0) atomicOr(err, (uint32_t)(l >= BB_MAX_LEVELS ? DEV_BIJECTION : DEV_BB_ROOM));
      return;
    }
    ulonglong2 *E = AR + region + used;
    const bool local = nw <= BF_WORDS;
    for (uint64_t w = tid; w < nw; w += BF_BLOCK) {
      if (local) set[w] = col[w] = 0;
      else E[w] = make_ulonglong2(0ull, 0ull);
    }
    __syncthreads();
    for (uint64_t i = tid; i < n; i += BF_BLOCK) {
      const uint64_t pos = bb_pos(bb_key_hash(rem[i]), l, (uint32_t)nw);
      const uint32_t w = (uint32_t)(pos >> 5), bit = 1u << (pos & 31);  // by half words
      uint32_t *x = local ? reinterpret_cast<uint32_t *>(set) + w
                          : reinterpret_cast<uint32_t *>(E + (w >> 1)) + (w & 1);
      uint32_t *y = local ? reinterpret_cast<uint32_t *>(col) + w
                          : reinterpret_cast<uint32_t *>(E + (w >> 1)) + 2 + (w & 1);
      if (atomicOr(x, bit) & bit) atomicOr(y, bit);
    }
    __syncthreads();
    uint32_t placed = 0;
    for (uint64_t w0 = 0; w0 < nw; w0 += BF_BLOCK) {
      const uint64_t w = w0 + tid;
      unsigned long long f = 0;
      if (w < nw) {
        if (local) f = set[w] & ~col[w];
        else {
          const ulonglong2 e = E[w];
          f = e.x & ~e.y;
        }
      }
      uint32_t tot;
      const uint32_t pre = block_exclusive_scan<BF_BLOCK>((uint32_t)__popcll(f), sm, tot);
      if (w < nw) {
        E[w] = make_ulonglong2(f, (unsigned long long)(placed + pre));
        if (local) set[w] = f;
      }
      placed += tot;
    }
    if (tid == 0) {
      BBMeta m;
      m.word_off = region + used;
      m.nwords = (uint32_t)nw;
      m.rank_adj = before;
      meta[(uint64_t)l * nbins + b] = m;
    }
    __syncthreads();
    KeyT *out = ((l & 1) ? r1 : r0) + s0;
    uint64_t left = 0;
    for (uint64_t i0 = 0; i0 < n; i0 += BF_BLOCK) {
      const uint64_t i = i0 + tid;
      KeyT key{};
      bool keep = false;
      if (i < n) {
        key = rem[i];
        const uint64_t pos = bb_pos(bb_key_hash(key), l, (uint32_t)nw);
        keep = !(((local ? set[pos >> 6] : E[pos >> 6].x) >> (pos & 63)) & 1);
      }
      uint32_t tot;
      const uint32_t pre = block_exclusive_scan<BF_BLOCK>(keep ? 1u : 0u, sm, tot);
      if (keep) out[left + pre] = key;
      left += tot;
    }
    __syncthreads();
    used += nw;
    before += placed;
    n = left;
    rem = out;
  }
  for (uint64_t w = used + tid; w < room; w += BF_BLOCK) AR[region + w] = make_ulonglong2(0ull, 0ull);
  if (tid == 0) {  // the deepest level, and the entries in use
    atomicMax(&got[0], (unsigned long long)l);
    atomicAdd(&got[1], (unsigned long long)used);
  }
}

// Keys whose bit did not survive go to the next level: each tile appends its
// survivors to out[start[b] + ...] behind one atomic on the bin's next count
// (the order of the keys inside a bin does not matter to BBHash).
template <class KeyT>
__global__ void __launch_bounds__(BB_BLOCK) bb_filter_kernel(const KeyT *rem, const uint64_t *start, const uint64_t *cnt,
                                                             const uint32_t *tile_off, uint32_t nbins,
                                                             const uint64_t *woff, uint32_t level, const ulonglong2 *AR,
                                                             unsigned long long *cnt_next, KeyT *out) {
  __shared__ uint32_t sm[BB_BLOCK / 32];
  __shared__ unsigned long long s_base;
  const uint32_t t = blockIdx.x;
  if (t >= tile_off[nbins]) return;
  TileSpan sp = tile_span_gapped(start, cnt, tile_off, nbins, t, BB_TILE);
  const uint64_t w0 = woff[sp.seg];
  const uint32_t nw = (uint32_t)(woff[sp.seg + 1] - w0);
  // consecutive threads on consecutive keys (sixteen consecutive ones a thread
  // touched a line per lane: 1.13 against 0.59 ms for those keys)
  uint32_t flags = 0;
#pragma unroll 4
  for (int j = 0; j < BB_ITEMS; j++) {
    const uint64_t i = sp.start + (uint64_t)j * BB_BLOCK + threadIdx.x;
    if (i < sp.end) {
      const uint64_t pos = bb_pos(bb_key_hash(rem[i]), level, nw);
      flags |= (uint32_t)(((AR[w0 + (pos >> 6)].x >> (pos & 63)) & 1) ^ 1) << j;
    }
  }
  uint32_t tot;
  uint32_t pre = block_exclusive_scan<BB_BLOCK>((uint32_t)__popc(flags), sm, tot);
  if (threadIdx.x == 0) s_base = tot ? atomicAdd(&cnt_next[sp.seg], (unsigned long long)tot) : 0;
  __syncthreads();
  uint64_t o = start[sp.seg] + s_base + pre;
#pragma unroll
  for (int j = 0; j < BB_ITEMS; j++)
    if ((flags >> j) & 1) out[o++] = rem[sp.start + (uint64_t)j * BB_BLOCK + threadIdx.x];
}

}  // namespace

template <class KeyT>
void BBHashBuild<KeyT>::clear() {
  tail_words_ = nullptr;
  total_words = used_words = dense_words = 0;
  levels = 0;
  bytes = 0;
  l1_slice_bits = -1;
  srank_words = 0;
}

template <class KeyT>
void BBHashBuild<KeyT>::reserve_entries(uint64_t words, uint64_t keep, cudaStream_t s) {
  const size_t need = words * sizeof(ulonglong2);
  if (ar_.p && need <= ar_.cap) return;
  size_t cap = std::max<size_t>(need + need / 4, 4096);
  void *np = nullptr;
  CF1_CUDA(cudaMalloc(&np, cap));
  if (keep && ar_.p) {
    CF1_CUDA(cudaMemcpyAsync(np, ar_.p, keep * sizeof(ulonglong2), cudaMemcpyDeviceToDevice, s));
    CF1_CUDA(cudaStreamSynchronize(s));
  }
  ar_.release();
  ar_.p = np;
  ar_.cap = cap;
}

template <class KeyT>
void BBHashBuild<KeyT>::begin(uint32_t nb, cudaStream_t s) {
  clear();
  nbins = nb;
  uint64_t *base = base_.get<uint64_t>(nbins);
  CF1_CUDA(cudaMemsetAsync(base, 0, nbins * sizeof(uint64_t), s));
  BBMeta *meta = meta_.get<BBMeta>((size_t)BB_MAX_LEVELS * nbins);
  CF1_CUDA(cudaMemsetAsync(meta, 0, (size_t)BB_MAX_LEVELS * nbins * sizeof(BBMeta), s));
  cnt_[0].get<uint64_t>(nbins);
  cnt_[1].get<uint64_t>(nbins);
  wcnt_.get<uint64_t>(nbins + 1);
  woff_.get<uint64_t>(nbins + 1);
  tile_off_.get<uint32_t>(nbins + 1);
  tot_.get<uint64_t>(3);
}

// Ranks and metadata of a level whose cleaned bits are in place: AR =
// entries [total_words, total_words + nw), woff = the bins' level-relative
// block offsets.
template <class KeyT>
void BBHashBuild<KeyT>::finish_level(uint32_t l, const uint64_t *woff, uint64_t nw, cudaStream_t s) {
  ulonglong2 *Al = ar_.as<ulonglong2>() + total_words;
  uint64_t *Rl = rtmp_.get<uint64_t>(nw + 1);
  uint32_t *pc = pc_.get<uint32_t>(nw);
  bb_clean_kernel<<<(unsigned)ceil_div(nw, 256), 256, 0, s>>>(Al, pc, nw);
  CF1_LAUNCH_CHECK();
  exclusive_scan_u32(pc, Rl, nw, scan_tmp_, s);
  bb_rank_kernel<<<(unsigned)ceil_div(nw, 256), 256, 0, s>>>(Al, Rl, nw);
  CF1_LAUNCH_CHECK();
  bb_meta_kernel<<<(unsigned)ceil_div(nbins, 256), 256, 0, s>>>(woff, Rl, total_words, base_.as<uint64_t>(),
                                                                meta_.as<BBMeta>() + (size_t)l * nbins, nbins);
  CF1_LAUNCH_CHECK();
}

// Levels l, l+1, ... until no key is left.  Level l's keys: bin b's are
// rem[start[b], start[b] + cnt_[l & 1][b]); each level writes the keys it
// does not place to r0 / r1 in turn at the same offsets.
template <class KeyT>
void BBHashBuild<KeyT>::run_levels(uint32_t l, const KeyT *rem, const uint64_t *start, KeyT *r0, KeyT *r1,
                                   uint64_t expect, uint64_t largest, uint32_t *err, cudaStream_t s) {
  KeyT *r[2] = {r0, r1};
  auto tail = [&] {  // all levels from l in one launch
    uint64_t *room = wcnt_.as<uint64_t>(), *off = woff_.as<uint64_t>(), *cur = cnt_[l & 1].as<uint64_t>();
    bb_room_kernel<<<(unsigned)ceil_div(nbins, 256), 256, 0, s>>>(cur, nbins, room);
    CF1_LAUNCH_CHECK();
    exclusive_scan_u64(room, off, nbins, scan_tmp_, s);
    unsigned long long *got = lv_.get<unsigned long long>(2);
    CF1_CUDA(cudaMemcpyAsync(got, tail_from_, sizeof(tail_from_), cudaMemcpyHostToDevice, s));
    const size_t smem = 2 * BF_WORDS * sizeof(unsigned long long);
    CF1_CUDA(cudaFuncSetAttribute(bb_tail_kernel<KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    bb_tail_kernel<KeyT><<<nbins, BF_BLOCK, smem, s>>>(rem, r0, r1, start, cur, nbins, l, ar_.as<ulonglong2>(), off,
                                                       total_words, ar_.cap / sizeof(ulonglong2), base_.as<uint64_t>(),
                                                       meta_.as<BBMeta>(), got, err);
    CF1_LAUNCH_CHECK();
    tail_words_ = off + nbins;
    levels = BB_MAX_LEVELS;  // until collect(): a walk ends at the first level a bin does not have
    dense_words = total_words;
  };
  tail_from_[0] = l;
  if (one_launch && expect <= BF_KEYS * nbins && largest <= BF_LARGEST) return tail();
  uint64_t *wcnt = wcnt_.as<uint64_t>(), *woff = woff_.as<uint64_t>();
  uint32_t *tile_off = tile_off_.as<uint32_t>();
  unsigned long long *tot = reinterpret_cast<unsigned long long *>(tot_.as<uint64_t>());
  for (;; l++) {
    uint64_t *cur = cnt_[l & 1].as<uint64_t>(), *nxt_cnt = cnt_[(l + 1) & 1].as<uint64_t>();
    CF1_CUDA(cudaMemsetAsync(tot, 0, 3 * sizeof(unsigned long long), s));
    bb_sizes_kernel<<<(unsigned)ceil_div(nbins, 256), 256, 0, s>>>(cur, nbins, l ? BB_GAMMA : BB_GAMMA0, wcnt, tot);
    CF1_LAUNCH_CHECK();
    uint64_t ht[3] = {0, 0, 0};
    CF1_CUDA(cudaMemcpyAsync(ht, tot, sizeof(ht), cudaMemcpyDeviceToHost, s));
    CF1_CUDA(cudaStreamSynchronize(s));
    const uint64_t remaining = ht[0], nw = ht[1];
    if (remaining == 0) break;
    if (one_launch && remaining <= BF_KEYS * nbins && ht[2] <= BF_LARGEST) {
      reserve_entries(total_words + bf_room(remaining) + nbins * (bf_room(1) + 1), total_words, s);
      tail_from_[0] = l;
      return tail();
    }
    if (l >= BB_MAX_LEVELS) throw Error(CF1GPU_ERR_BIJECTION, "BBHash: keys left after the last level");
    exclusive_scan_u64(wcnt, woff, nbins, scan_tmp_, s);
    reserve_entries(total_words + nw, total_words, s);
    ulonglong2 *Al = ar_.as<ulonglong2>() + total_words;
    CF1_CUDA(cudaMemsetAsync(Al, 0, nw * sizeof(ulonglong2), s));
    uint32_t ub = (uint32_t)(ceil_div(remaining, BB_TILE) + nbins);
    segment_tiles_counts(cur, nbins, BB_TILE, tile_off, s);
    bb_mark_kernel<KeyT><<<ub, BB_BLOCK, 0, s>>>(rem, start, cur, tile_off, nbins, woff, l, Al);
    CF1_LAUNCH_CHECK();
    finish_level(l, woff, nw, s);
    KeyT *out = r[l & 1];
    CF1_CUDA(cudaMemsetAsync(nxt_cnt, 0, nbins * sizeof(uint64_t), s));
    bb_filter_kernel<KeyT><<<ub, BB_BLOCK, 0, s>>>(rem, start, cur, tile_off, nbins, woff, l, Al,
                                                   reinterpret_cast<unsigned long long *>(nxt_cnt), out);
    CF1_LAUNCH_CHECK();
    total_words += nw;
    rem = out;
  }
  levels = l;
  used_words = dense_words = total_words;
  set_bytes();
}

template <class KeyT>
void BBHashBuild<KeyT>::set_bytes() {
  bytes = used_words * sizeof(ulonglong2) + (size_t)levels * nbins * sizeof(BBMeta) + 2 * srank_words * sizeof(uint32_t);
}

template <class KeyT>
void BBHashBuild<KeyT>::collect_begin(uint64_t *got, cudaStream_t s) {
  if (!tail_words_) return;
  CF1_CUDA(cudaMemcpyAsync(&got[0], tail_words_, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaMemcpyAsync(&got[1], lv_.p, 2 * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
}

template <class KeyT>
void BBHashBuild<KeyT>::collect_end(const uint64_t *got) {
  if (!tail_words_) return;
  tail_words_ = nullptr;
  total_words += got[0];
  used_words = dense_words + got[2];
  levels = std::max<uint32_t>((uint32_t)got[1], l1_slice_bits >= 0 ? 2 : 0);
  set_bytes();
}

template <class KeyT>
void BBHashBuild<KeyT>::build(const KeyT *keys, const uint64_t *seg_off, uint32_t nb, const uint32_t *sel,
                              uint32_t *err, cudaStream_t s, KeyT *ws0, KeyT *ws1, uint64_t ws_cap) {
  begin(nb, s);
  std::vector<uint64_t> hoff(nbins + 1);
  CF1_CUDA(cudaMemcpyAsync(hoff.data(), seg_off, (nbins + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaStreamSynchronize(s));
  uint64_t largest = 0;
  for (uint32_t b = 0; b < nbins; b++) largest = std::max(largest, hoff[b + 1] - hoff[b]);
  if (largest >= (1ull << 32))  // local slots are 32-bit
    throw Error(CF1GPU_ERR_INVALID_ARG, "BBHash: a bin holds 2^32 or more distinct keys; use more bins");
  const uint64_t n_all = hoff[nbins];
  // Keys of bin b at every level sit at [seg_off[b], seg_off[b] + cnt[b]) of
  // the level's key array: the distinct keys at level 0, then the two
  // workspaces in turn (the caller's, when big enough).
  KeyT *r0 = (ws0 && ws_cap >= n_all + 1) ? ws0 : rem_[0].get<KeyT>(n_all + 1);
  KeyT *r1 = (ws1 && ws_cap >= n_all + 1) ? ws1 : rem_[1].get<KeyT>(n_all + 1);
  bb_init_counts_kernel<<<(unsigned)ceil_div(nbins, 256), 256, 0, s>>>(seg_off, sel, nbins, cnt_[0].as<uint64_t>());
  CF1_LAUNCH_CHECK();
  // room for the usual level sizes (gamma0 bits per key, then ~12% and
  // fewer keys per level) so that the entry array rarely grows in mid-build
  reserve_entries((BB_GAMMA0 * n_all / 64 + nbins) * 3 / 2 + 64 * nbins + 64, 0, s);
  run_levels(0, keys, seg_off, r0, r1, n_all, largest, err, s);
}

template <class KeyT>
ulonglong2 *BBHashBuild<KeyT>::prepare_levels01(uint32_t nb, uint64_t words0, uint64_t words1, cudaStream_t s) {
  // with the later levels' room: at most a quarter of the occurrences reach
  // level 2 (the dedup's list holds no more), bf_room(that) in all
  const uint64_t words = words0 + words1;
  reserve_entries(words + words / 3 + (uint64_t)nb * 2 * BB_MAX_LEVELS + 64 * 1024, 0, s);
  return ar_.as<ulonglong2>();
}

template <class KeyT>
void BBHashBuild<KeyT>::build_from_levels01(uint32_t nb, int P, const uint64_t *woff0, uint64_t words0,
                                            const uint32_t *placed0, const uint64_t *woff1, uint64_t words1,
                                            const uint32_t *placed1, const KeyT *surv, const uint64_t *surv_off,
                                            const uint64_t *surv_cnt, uint64_t surv_total, uint64_t n_occ,
                                            uint64_t max_bin, uint32_t *err, cudaStream_t s, KeyT *ws0, KeyT *ws1, uint64_t ws_cap) {
  begin(nb, s);
  const uint64_t nsl = ((uint64_t)nbins << P) + 1;
  bb_sliced_kernel<<<nbins, BF_BLOCK, 0, s>>>(woff0, woff1, P, words0, placed0, placed1, srank_[0].get<uint32_t>(nsl),
                                              srank_[1].get<uint32_t>(nsl), base_.as<uint64_t>(), meta_.as<BBMeta>(),
                                              nbins);
  CF1_LAUNCH_CHECK();
  total_words = words0 + words1;
  l1_slice_bits = P;
  srank_words = (uint64_t)nbins << P;
  CF1_CUDA(cudaMemcpyAsync(cnt_[0].as<uint64_t>(), surv_cnt, nbins * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s));
  KeyT *r0 = (ws0 && ws_cap >= surv_total + 1) ? ws0 : rem_[0].get<KeyT>(surv_total + 1);
  KeyT *r1 = (ws1 && ws_cap >= surv_total + 1) ? ws1 : rem_[1].get<KeyT>(surv_total + 1);
  // level l reads cnt_[l & 1] and writes r[l & 1]; level 1 leaves ~1% of the keys
  run_levels(2, surv, surv_off, r0, r1, n_occ / 100, max_bin / 100, err, s);
  levels = std::max<uint32_t>(levels, 2);
  set_bytes();
}

template <class KeyT>
BBView BBHashBuild<KeyT>::view() const {
  BBView v;
  v.AR = ar_.as<const ulonglong2>();
  v.meta = meta_.as<const BBMeta>();
  v.levels = levels;
  v.nbins = nbins;
  v.l1_slice_bits = l1_slice_bits;
  v.pad = 0;
  v.srank[0] = l1_slice_bits >= 0 ? srank_[0].as<const uint32_t>() : nullptr;
  v.srank[1] = l1_slice_bits >= 0 ? srank_[1].as<const uint32_t>() : nullptr;
  return v;
}

template struct BBHashBuild<uint64_t>;
template struct BBHashBuild<Key2>;

}  // namespace cf1
