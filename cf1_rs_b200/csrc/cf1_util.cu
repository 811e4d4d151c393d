// Prefix sums and segment tiling.
#include "cf1_device_util.cuh"
#include "cf1_internal.cuh"

namespace cf1 {

std::atomic<uint64_t> g_launches{0};

namespace {

// Exclusive sums of up to 2^64 in two passes over the input: every CTA's sum,
// then (with the sums' own exclusive sums) the values.  A warp takes 256
// consecutive items as four rows of 64, two to a lane, so that loads and
// stores are 16 bytes a lane side by side; eight consecutive items a thread
// stored 8 bytes every 64.  Memory bound.  The k-mer counts of 22 M records
// (200 Mbp), read from the records instead of from a copy of their lengths:
// 0.21 ms before, 0.13 now; 111 M of 1 Gbp 0.97 and 0.60.
constexpr int SCAN_BLOCK = 512;
constexpr int SCAN_ROWS = 4;
constexpr uint64_t SCAN_WARP = 64 * SCAN_ROWS;  // items a warp takes
constexpr uint64_t SCAN_CHUNK = SCAN_BLOCK / 32 * SCAN_WARP;

template <class T>
struct ScanValues {  // plain counts
  const T *p;
  CF1_D uint64_t one(uint64_t i) const { return (uint64_t)p[i]; }
  CF1_D bool pairs() const { return ((uintptr_t)p & (2 * sizeof(T) - 1)) == 0; }
  CF1_D void two(uint64_t i, uint64_t &x, uint64_t &y) const {
    if constexpr (sizeof(T) == 4) {
      const uint2 v = *reinterpret_cast<const uint2 *>(p + i);
      x = v.x;
      y = v.y;
    } else {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p + i);
      x = v.x;
      y = v.y;
    }
  }
};
struct ScanRecords {  // the records' k-mer counts
  ScanValues<uint64_t> r;
  CF1_D uint64_t one(uint64_t i) const { return rec_n(r.one(i)); }
  CF1_D bool pairs() const { return r.pairs(); }
  CF1_D void two(uint64_t i, uint64_t &x, uint64_t &y) const {
    r.two(i, x, y);
    x = rec_n(x);
    y = rec_n(y);
  }
};

// Items i and i + 1 (i even), zero past the end.
template <class In>
CF1_D void scan_pair(const In &in, uint64_t i, uint64_t n, uint64_t &x, uint64_t &y) {
  if (i + 1 < n && in.pairs()) {
    in.two(i, x, y);
  } else {
    x = i < n ? in.one(i) : 0;
    y = i + 1 < n ? in.one(i + 1) : 0;
  }
}

template <class In>
__global__ void __launch_bounds__(SCAN_BLOCK) scan_reduce_kernel(In in, uint64_t n, uint64_t *sums) {
  __shared__ uint64_t sm[SCAN_BLOCK / 32];
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_CHUNK + (threadIdx.x >> 5) * SCAN_WARP + 2 * lane_id();
  uint64_t x[SCAN_ROWS], y[SCAN_ROWS], acc = 0;
#pragma unroll
  for (int r = 0; r < SCAN_ROWS; r++) scan_pair(in, base + r * 64, n, x[r], y[r]);
#pragma unroll
  for (int r = 0; r < SCAN_ROWS; r++) acc += x[r] + y[r];
  const uint64_t tot = block_sum<SCAN_BLOCK>(acc, sm);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

template <class In>
__global__ void __launch_bounds__(SCAN_BLOCK) scan_down_kernel(In in, uint64_t n, const uint64_t *block_off,
                                                               uint64_t *out) {
  __shared__ uint64_t sm[SCAN_BLOCK / 32];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  const uint64_t base = (uint64_t)blockIdx.x * SCAN_CHUNK + warp * SCAN_WARP + 2 * lane;
  uint64_t x[SCAN_ROWS], y[SCAN_ROWS], pre[SCAN_ROWS], run = 0;
#pragma unroll
  for (int r = 0; r < SCAN_ROWS; r++) scan_pair(in, base + r * 64, n, x[r], y[r]);
#pragma unroll
  for (int r = 0; r < SCAN_ROWS; r++) {  // exclusive sums inside the warp
    const uint64_t own = x[r] + y[r], v = warp_inclusive_scan(own);
    pre[r] = run + v - own;
    run += __shfl_sync(FULL, v, 31);
  }
  if (lane == 0) sm[warp] = run;
  __syncthreads();
  uint64_t off = block_off ? block_off[blockIdx.x] : 0;
  for (unsigned w = 0; w < warp; w++) off += sm[w];
  const bool pairs = ((uintptr_t)out & 15) == 0;
#pragma unroll
  for (int r = 0; r < SCAN_ROWS; r++) {
    const uint64_t i = base + r * 64, a = off + pre[r];
    if (i + 1 < n && pairs) {
      *reinterpret_cast<ulonglong2 *>(out + i) = make_ulonglong2(a, a + x[r]);
    } else {
      if (i < n) out[i] = a;
      if (i + 1 < n) out[i + 1] = a + x[r];
    }
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == SCAN_BLOCK - 1) out[n] = off + run;
}

__global__ void zero_total_kernel(uint64_t *out) { out[0] = 0; }

template <class In>
void scan_impl(const In &in, uint64_t *out, uint64_t n, DevBuf &scratch, size_t scratch_off, cudaStream_t s) {
  if (n == 0) {
    zero_total_kernel<<<1, 1, 0, s>>>(out);
    CF1_LAUNCH_CHECK();
    return;
  }
  uint64_t nb = ceil_div(n, SCAN_CHUNK);
  if (nb == 1) {
    scan_down_kernel<In><<<1, SCAN_BLOCK, 0, s>>>(in, n, nullptr, out);
    CF1_LAUNCH_CHECK();
    return;
  }
  // scratch layout at scratch_off: sums[nb], sums_scan[nb+1], deeper levels after.
  uint64_t *sums = reinterpret_cast<uint64_t *>(static_cast<char *>(scratch.p) + scratch_off);
  uint64_t *sums_scan = sums + nb;
  scan_reduce_kernel<In><<<(unsigned)nb, SCAN_BLOCK, 0, s>>>(in, n, sums);
  CF1_LAUNCH_CHECK();
  scan_impl(ScanValues<uint64_t>{sums}, sums_scan, nb, scratch, scratch_off + (2 * nb + 1) * sizeof(uint64_t), s);
  scan_down_kernel<In><<<(unsigned)nb, SCAN_BLOCK, 0, s>>>(in, n, sums_scan, out);
  CF1_LAUNCH_CHECK();
}

size_t scan_scratch_bytes(uint64_t n) {
  size_t bytes = 64;
  while (n > SCAN_CHUNK) {
    uint64_t nb = ceil_div(n, SCAN_CHUNK);
    bytes += (2 * nb + 1) * sizeof(uint64_t);
    n = nb;
  }
  return bytes;
}

// seg_off: offsets (segment b has seg_off[b+1] - seg_off[b] items) or, when
// counts is set, the item counts themselves.
__global__ void segment_tiles_kernel(const uint64_t *seg_off, uint32_t nseg, uint32_t tile, bool counts,
                                     uint32_t *tile_off) {
  constexpr int B = 1024;
  __shared__ uint32_t sm[B / 32];
  uint32_t carry = 0;
  for (uint32_t base = 0; base < nseg; base += B) {
    uint32_t b = base + threadIdx.x;
    uint32_t c = 0;
    if (b < nseg) c = (uint32_t)(((counts ? seg_off[b] : seg_off[b + 1] - seg_off[b]) + tile - 1) / tile);
    uint32_t tot;
    uint32_t pre = block_exclusive_scan<B>(c, sm, tot);
    if (b < nseg) tile_off[b] = carry + pre;
    carry += tot;
  }
  if (threadIdx.x == 0) tile_off[nseg] = carry;
}

}  // namespace

void exclusive_scan_u32(const uint32_t *in, uint64_t *out, uint64_t n, DevBuf &scratch, cudaStream_t s) {
  scratch.reserve(scan_scratch_bytes(n));
  scan_impl(ScanValues<uint32_t>{in}, out, n, scratch, 0, s);
}
void exclusive_scan_u64(const uint64_t *in, uint64_t *out, uint64_t n, DevBuf &scratch, cudaStream_t s) {
  scratch.reserve(scan_scratch_bytes(n));
  scan_impl(ScanValues<uint64_t>{in}, out, n, scratch, 0, s);
}

void record_kmer_prefix(const uint64_t *records, uint64_t n_rec, uint64_t *kpre, DevBuf &scratch, cudaStream_t s) {
  scratch.reserve(scan_scratch_bytes(n_rec));
  scan_impl(ScanRecords{{records}}, kpre, n_rec, scratch, 0, s);
}

void segment_tiles(const uint64_t *seg_off, uint32_t nseg, uint32_t tile, uint32_t *tile_off, cudaStream_t s) {
  segment_tiles_kernel<<<1, 1024, 0, s>>>(seg_off, nseg, tile, false, tile_off);
  CF1_LAUNCH_CHECK();
}

void segment_tiles_counts(const uint64_t *cnt, uint32_t nseg, uint32_t tile, uint32_t *tile_off, cudaStream_t s) {
  segment_tiles_kernel<<<1, 1024, 0, s>>>(cnt, nseg, tile, true, tile_off);
  CF1_LAUNCH_CHECK();
}

}  // namespace cf1
