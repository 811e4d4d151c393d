// cf1gpu_distinct_kmers_noalloc: phase 3a (canonical k-mer extraction, LSD
// radix sort, adjacent-unique) for one record, with every byte of scratch in
// a fixed file-scope device array instead of memory allocated per call.
//
// Who needs this: code that must not allocate device memory while it runs --
// a host application that owns the whole device memory pool and hands the
// library only its input and output buffers, or a caller inside a section
// where cudaMalloc would synchronise the device or is forbidden.  Such a
// caller passes device pointers for the record and the outputs; the library
// uses only the array below.
//
// The array is sized for NA_MAX_BASES bases (1 Mi) and every GPU that loads
// this part of the library keeps it (17 MiB) until the process exits.
// All calls share it and it keeps the last call's contents, so each call
// first clears the counters it relies on.  Two calls whose work overlaps on
// the GPU (different streams, or different host threads on one device) race
// on the array and corrupt each other's results: serialise them.
//
// Host code never uses the array's name as an address (on the host it is only
// a stand-in symbol): the first call on each device, with that device
// current, looks up the device address with cudaGetSymbolAddress and caches
// it.  Make that first call before any stream capture on the device.
#include <mutex>

#include "../../include/cf1gpu.h"
#include "cf1_device_util.cuh"
#include "cf1_internal.cuh"

namespace cf1 {

namespace {

constexpr uint64_t NA_MAX_BASES = 1ull << 20;
constexpr int NA_BLOCK = 256;
constexpr int NA_ITEMS = 8;
constexpr uint32_t NA_TILE = NA_BLOCK * NA_ITEMS;            // 2048 keys
constexpr uint32_t NA_MAX_TILES = NA_MAX_BASES / NA_TILE;     // 512
constexpr uint32_t NA_DIGITS = 256;
constexpr int NA_NW = NA_BLOCK / 32;
// The histogram and scatter kernels index per-digit arrays by thread.
static_assert(NA_BLOCK == (int)NA_DIGITS, "one thread per radix digit");

// Scratch layout (byte offsets).
constexpr size_t NA_KEYS = 0;                                          // u64 [NA_MAX_BASES]
constexpr size_t NA_ALT = NA_KEYS + NA_MAX_BASES * 8;                  // u64 [NA_MAX_BASES]
constexpr uint32_t NA_HENTRIES = NA_DIGITS * NA_MAX_TILES;
constexpr size_t NA_HIST = NA_ALT + NA_MAX_BASES * 8;                  // u32 [NA_HENTRIES]
constexpr size_t NA_HSCAN = NA_HIST + NA_HENTRIES * 4;                 // u32 [NA_HENTRIES]
constexpr size_t NA_TCNT = NA_HSCAN + NA_HENTRIES * 4;                 // u32 [NA_MAX_TILES]
constexpr size_t NA_DTOT = NA_TCNT + NA_MAX_TILES * 4;                 // u32 [NA_DIGITS]
constexpr size_t NA_COUNT = NA_DTOT + NA_DIGITS * 4;                   // u32 number of keys (256-aligned)
constexpr size_t NA_SCRATCH_BYTES = NA_COUNT + 256;                    // 17.0 MiB in all

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_SCRATCH_BYTES];

struct Scratch {
  uint64_t *keys, *alt;
  uint32_t *hist, *hscan, *tcnt, *dtot, *count;
};

Scratch carve(unsigned char *base) {
  Scratch s;
  s.keys = reinterpret_cast<uint64_t *>(base + NA_KEYS);
  s.alt = reinterpret_cast<uint64_t *>(base + NA_ALT);
  s.hist = reinterpret_cast<uint32_t *>(base + NA_HIST);
  s.hscan = reinterpret_cast<uint32_t *>(base + NA_HSCAN);
  s.tcnt = reinterpret_cast<uint32_t *>(base + NA_TCNT);
  s.dtot = reinterpret_cast<uint32_t *>(base + NA_DTOT);
  s.count = reinterpret_cast<uint32_t *>(base + NA_COUNT);
  return s;
}

// The bits of x at the even positions of a u64 (a k-mer's low or high code
// bits, one base after another).
CF1_D uint64_t na_spread(uint32_t x) {
  uint64_t v = x;
  v = (v | (v << 16)) & 0x0000FFFF0000FFFFull;
  v = (v | (v << 8)) & 0x00FF00FF00FF00FFull;
  v = (v | (v << 4)) & 0x0F0F0F0F0F0F0F0Full;
  v = (v | (v << 2)) & 0x3333333333333333ull;
  return (v | (v << 1)) & 0x5555555555555555ull;
}

// Canonical k-mer of every placeholder-free window [p, p+k) (src/mphf.rs:
// 334-343 decode + canonicalise); order does not matter, the sort follows.
// A CTA reads its 256 bases and the 32 after them once and keeps them as
// three bit planes (code bits, placeholders), a warp vote per word; a window
// is a funnel shift of each plane, and the reverse complement is the
// complemented planes in the other bit order.  (One byte load per base of
// every window and an atomic a warp took 31 us for 1 Mi bases, this 14.)
__global__ void __launch_bounds__(NA_BLOCK) na_extract_kernel(const uint8_t *seq, uint64_t len, int k, uint64_t *keys,
                                                              uint32_t *count) {
  constexpr int NWORDS = NA_BLOCK / 32 + 1;
  __shared__ uint32_t lo[NWORDS], hi[NWORDS], nm[NWORDS];
  const uint64_t p0 = (uint64_t)blockIdx.x * NA_BLOCK;
  const unsigned tid = threadIdx.x, lane = lane_id();
  auto plane = [&](uint64_t p, uint32_t w) {
    const uint32_t u = p < len ? seq[p] & 0xDF : 'N';
    const bool ok = (u == 'A') | (u == 'C') | (u == 'G') | (u == 'T');
    uint32_t b = (u >> 1) & 3;
    b ^= b >> 1;
    const uint32_t l = __ballot_sync(FULL, b & 1), h = __ballot_sync(FULL, b >> 1), n = __ballot_sync(FULL, !ok);
    if (lane == 0) {
      lo[w] = l;
      hi[w] = h;
      nm[w] = n;
    }
  };
  plane(p0 + tid, tid >> 5);
  if (tid < 32) plane(p0 + NA_BLOCK + tid, NWORDS - 1);
  __syncthreads();
  const uint32_t w = tid >> 5, mask = (1u << k) - 1;  // k <= 31
  const uint32_t l = __funnelshift_r(lo[w], lo[w + 1], lane) & mask, h = __funnelshift_r(hi[w], hi[w + 1], lane) & mask;
  const bool ok = (__funnelshift_r(nm[w], nm[w + 1], lane) & mask) == 0;  // (bases past the end are placeholders)
  const uint64_t fw = na_spread(__brev(l) >> (32 - k)) | (na_spread(__brev(h) >> (32 - k)) << 1);
  const uint64_t rc = na_spread(~l & mask) | (na_spread(~h & mask) << 1);
  __shared__ uint32_t sm[NA_NW], s_base;  // one reservation a CTA
  uint32_t tot;
  const uint32_t pre = block_exclusive_scan<NA_BLOCK>(ok ? 1u : 0u, sm, tot);
  if (tid == 0) s_base = tot ? atomicAdd(count, tot) : 0u;
  __syncthreads();
  if (ok) keys[s_base + pre] = fw < rc ? fw : rc;
}

// Per tile digit counts, digit-major (digit d of tile t at d * ntiles + t).
// Launched over all ntiles tiles of the call's largest possible key count:
// tiles past the actual count write zeros, so every entry the scan reads was
// written by this call and nothing a previous call left reaches it.
__global__ void __launch_bounds__(NA_BLOCK) na_hist_kernel(const uint64_t *keys, const uint32_t *count, int shift,
                                                           uint32_t ntiles, uint32_t *H) {
  __shared__ uint32_t h[NA_DIGITS];
  const uint32_t t = blockIdx.x, n = *count;
  h[threadIdx.x] = 0;
  __syncthreads();
  uint64_t start = (uint64_t)t * NA_TILE, end = start + NA_TILE < n ? start + NA_TILE : n;
  for (uint64_t i = start + threadIdx.x; i < end; i += NA_BLOCK) atomicAdd(&h[(keys[i] >> shift) & 0xFF], 1u);
  __syncthreads();
  H[threadIdx.x * ntiles + t] = h[threadIdx.x];
}

// One CTA per digit: exclusive scan of its counts over the tiles (ntiles <=
// NA_MAX_TILES), and their sum.  The scatter adds the sums of the smaller
// digits itself.  (One CTA scanning all digits x tiles in 1024-entry rounds
// took 100 us a pass for 1 Mi bases, of the call's 920.)
__global__ void __launch_bounds__(NA_BLOCK) na_scan_kernel(const uint32_t *H, uint32_t ntiles, uint32_t *Hs,
                                                           uint32_t *dtot) {
  static_assert(NA_MAX_TILES <= 2 * NA_BLOCK, "two tiles a thread");
  __shared__ uint32_t sm[NA_NW];
  const uint32_t d = blockIdx.x, t = 2 * threadIdx.x;
  const uint32_t v0 = t < ntiles ? H[d * ntiles + t] : 0, v1 = t + 1 < ntiles ? H[d * ntiles + t + 1] : 0;
  uint32_t tot;
  const uint32_t pre = block_exclusive_scan<NA_BLOCK>(v0 + v1, sm, tot);
  if (t < ntiles) Hs[d * ntiles + t] = pre;
  if (t + 1 < ntiles) Hs[d * ntiles + t + 1] = pre + v0;
  if (threadIdx.x == 0) dtot[d] = tot;
}

// Stable scatter of one tile.  A warp takes 256 consecutive keys, 32 at a
// time, and ranks them by its own digit counters (match_any inside a round,
// the counters between rounds); a prefix over the warps gives tile-local
// places, the tile is staged in digit order and every digit's run is written
// by consecutive threads.
__global__ void __launch_bounds__(NA_BLOCK) na_scatter_kernel(const uint64_t *in, uint64_t *out, const uint32_t *count,
                                                              int shift, uint32_t ntiles, const uint32_t *Hs,
                                                              const uint32_t *dtot) {
  __shared__ uint64_t stage[NA_TILE];
  __shared__ uint32_t whist[NA_NW][NA_DIGITS];
  __shared__ uint32_t s_base[NA_DIGITS], sm[NA_NW];
  const uint32_t t = blockIdx.x, n = *count;
  const unsigned tid = threadIdx.x, warp = tid >> 5, lane = lane_id(), lt = lanemask_lt();
  const uint64_t start = (uint64_t)t * NA_TILE;
  if (start >= n) return;
  const uint32_t len = (uint32_t)(n - start < NA_TILE ? n - start : NA_TILE);
  uint64_t key[NA_ITEMS];
#pragma unroll
  for (int r = 0; r < NA_ITEMS; r++) {
    const uint32_t i = warp * (NA_ITEMS * 32) + r * 32 + lane;
    key[r] = i < len ? in[start + i] : 0;
  }
  for (uint32_t i = tid; i < NA_NW * NA_DIGITS; i += NA_BLOCK) (&whist[0][0])[i] = 0;
  uint32_t tot;
  const uint32_t gbase = block_exclusive_scan<NA_BLOCK>(dtot[tid], sm, tot) + Hs[tid * ntiles + t];
  uint32_t rank[NA_ITEMS];
#pragma unroll
  for (int r = 0; r < NA_ITEMS; r++) {
    const uint32_t i = warp * (NA_ITEMS * 32) + r * 32 + lane;
    const uint32_t d = i < len ? (uint32_t)(key[r] >> shift) & 0xFF : 0xFFFFFFFFu;
    const unsigned peers = __match_any_sync(FULL, d);
    const uint32_t c = d < NA_DIGITS ? whist[warp][d] : 0;
    rank[r] = c + __popc(peers & lt);
    __syncwarp();
    if (d < NA_DIGITS && (peers & lt) == 0) whist[warp][d] = c + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < NA_NW; w++) {
    const uint32_t v = whist[w][tid];
    whist[w][tid] = run;
    run += v;
  }
  const uint32_t first = block_exclusive_scan<NA_BLOCK>(run, sm, tot);  // the digit's tile-local start
  s_base[tid] = gbase - first;
#pragma unroll
  for (int w = 0; w < NA_NW; w++) whist[w][tid] += first;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < NA_ITEMS; r++) {
    const uint32_t i = warp * (NA_ITEMS * 32) + r * 32 + lane;
    if (i < len) stage[whist[warp][(uint32_t)(key[r] >> shift) & 0xFF] + rank[r]] = key[r];
  }
  __syncthreads();
  for (uint32_t i = tid; i < len; i += NA_BLOCK) {
    const uint64_t k = stage[i];
    out[s_base[(uint32_t)(k >> shift) & 0xFF] + i] = k;
  }
}

__global__ void __launch_bounds__(NA_BLOCK) na_unique_count_kernel(const uint64_t *keys, const uint32_t *count,
                                                                   uint32_t *tcnt) {
  __shared__ uint32_t sm[NA_NW];
  const uint32_t t = blockIdx.x, n = *count;
  uint64_t start = (uint64_t)t * NA_TILE, end = start + NA_TILE < n ? start + NA_TILE : n;
  uint32_t c = 0;
  for (uint64_t i = start + threadIdx.x; i < end; i += NA_BLOCK) c += (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
  uint32_t tot = block_sum<NA_BLOCK>(c, sm);
  if (threadIdx.x == 0) tcnt[t] = tot;
}

__global__ void __launch_bounds__(NA_BLOCK) na_unique_write_kernel(const uint64_t *keys, const uint32_t *count,
                                                                   const uint32_t *tcnt, uint32_t ntiles,
                                                                   uint64_t *out, uint64_t *n_out) {
  __shared__ uint32_t sm[NA_NW];
  const uint32_t t = blockIdx.x, n = *count;
  // the distinct keys of the tiles before this one
  uint32_t before = 0, all = 0;
  for (uint32_t i = threadIdx.x; i < ntiles; i += NA_BLOCK) {
    const uint32_t v = tcnt[i];
    all += v;
    before += i < t ? v : 0u;
  }
  before = block_sum<NA_BLOCK>(before, sm);
  uint64_t i0 = (uint64_t)t * NA_TILE + (uint64_t)threadIdx.x * NA_ITEMS;
  uint32_t flags = 0, c = 0;
#pragma unroll
  for (int j = 0; j < NA_ITEMS; j++) {
    uint64_t i = i0 + j;
    bool f = i < n && (i == 0 || keys[i] != keys[i - 1]);
    flags |= (uint32_t)f << j;
    c += f;
  }
  uint32_t tot;
  uint32_t pre = block_exclusive_scan<NA_BLOCK>(c, sm, tot);
  uint64_t o = before + pre;
#pragma unroll
  for (int j = 0; j < NA_ITEMS; j++)
    if ((flags >> j) & 1) out[o++] = keys[i0 + j];
  if (t == 0) {
    all = block_sum<NA_BLOCK>(all, sm);
    if (threadIdx.x == 0) *n_out = all;
  }
}

std::mutex g_addr_mu;
void *g_addr[64] = {};

}  // namespace

}  // namespace cf1

extern "C" int cf1gpu_distinct_kmers_noalloc(int device, uint32_t k, const uint8_t *d_seq, size_t len,
                                             uint64_t *d_keys_out, size_t out_cap, uint64_t *d_n_out, void *stream) {
  using namespace cf1;
  if (len > NA_MAX_BASES) return CF1GPU_ERR_TOO_LARGE;
  if (k < 1 || k > 31 || k % 2 == 0) return CF1GPU_ERR_INVALID_ARG;
  uint64_t max_keys = len >= k ? len - k + 1 : 0;
  if ((len && !d_seq) || !d_keys_out || !d_n_out || out_cap < max_keys) return CF1GPU_ERR_INVALID_ARG;
  if (device < 0 || device >= 64) return CF1GPU_ERR_INVALID_ARG;
  (void)cudaGetLastError();  // an earlier call's error is not this call's
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (s) {  // the work goes to `device`: a stream of another device is refused
    int sdev = -1;
    if (cudaStreamGetDevice(s, &sdev) != cudaSuccess) return CF1GPU_ERR_INVALID_ARG;
    if (sdev != device) return CF1GPU_ERR_INVALID_ARG;
  }
  int prev = -1;
  if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
  if (cudaSetDevice(device) != cudaSuccess) return CF1GPU_ERR_CUDA;
  void *base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_addr_mu);
    if (!g_addr[device]) {
      // once per device, with the device current: the array's device address
      if (cudaGetSymbolAddress(&g_addr[device], g_noalloc_scratch) != cudaSuccess) {
        g_addr[device] = nullptr;
        if (prev >= 0) cudaSetDevice(prev);
        return CF1GPU_ERR_CUDA;
      }
    }
    base = g_addr[device];
  }
  Scratch sc = carve(static_cast<unsigned char *>(base));
  uint32_t ntiles = (uint32_t)((max_keys + NA_TILE - 1) / NA_TILE);
  cudaError_t e = cudaMemsetAsync(sc.count, 0, sizeof(uint32_t), s);
  if (e == cudaSuccess && max_keys) {
    na_extract_kernel<<<(unsigned)((max_keys + 255) / 256), 256, 0, s>>>(d_seq, len, (int)k, sc.keys, sc.count);
    uint64_t *src = sc.keys, *dst = sc.alt;
    for (int shift = 0; shift < 2 * (int)k; shift += 8) {
      na_hist_kernel<<<ntiles, NA_BLOCK, 0, s>>>(src, sc.count, shift, ntiles, sc.hist);
      na_scan_kernel<<<NA_DIGITS, NA_BLOCK, 0, s>>>(sc.hist, ntiles, sc.hscan, sc.dtot);
      na_scatter_kernel<<<ntiles, NA_BLOCK, 0, s>>>(src, dst, sc.count, shift, ntiles, sc.hscan, sc.dtot);
      uint64_t *t = src;
      src = dst;
      dst = t;
    }
    na_unique_count_kernel<<<ntiles, NA_BLOCK, 0, s>>>(src, sc.count, sc.tcnt);
    na_unique_write_kernel<<<ntiles, NA_BLOCK, 0, s>>>(src, sc.count, sc.tcnt, ntiles, d_keys_out, d_n_out);
    e = cudaGetLastError();
  } else if (e == cudaSuccess) {
    e = cudaMemsetAsync(d_n_out, 0, sizeof(uint64_t), s);
  }
  if (prev >= 0) cudaSetDevice(prev);
  return e == cudaSuccess ? CF1GPU_OK : CF1GPU_ERR_CUDA;
}
