// Per-bin learned index over the bins' sorted distinct keys.
//
// Two stages per bin (a recursive-model index):
//   root  : an MLP 1 -> LI_HIDDEN (ReLU) -> 1 trained on the GPU to map the
//           key's scaled top bits x to its rank fraction (the bin's empirical
//           CDF); leaf = floor(root(x) * n_leaves);
//   leaves: per leaf a line through its first and last key's (key, rank);
//           err = max |prediction - rank| over the keys the root sends there.
// A query evaluates the root, the leaf's line, and searches the sorted keys
// in [pred - err, pred + err].  A verification pass queries every key; a bin with a
// key outside its window, or with err above the threshold, is served by
// BBHash instead.
//
// The hidden units are clipped ReLUs, clamp(w1 x + b1, 0, 1): a sum of
// bounded non-decreasing ramps can follow any non-decreasing CDF, concave
// ones included (canonical k-mers are denser at small values).  Training
// projects the weights of both layers onto [0, inf) after every step.  With
// non-negative weights every rounded fma and the clamp are non-decreasing,
// so root(x) -- and the leaf index -- is non-decreasing in the key: the keys
// routed to a leaf are one contiguous run of ranks, and a leaf's error bound
// only measures how far the run bends from its line.  Before training the root is the identity (y = x), which
// is the same index without the network: the comparison of the two is
// reported in the stats.
#include <cmath>
#include <cstring>

#include "cf1_device_util.cuh"
#include "cf1_learned.cuh"
#include "cf1_mphf.cuh"

namespace cf1 {

namespace {

constexpr int LT_BLOCK = 256;
constexpr int LT_NW = LT_BLOCK / 32;
constexpr uint32_t LT_TILE = 16384;  // keys per CTA: the tile's set-up (segment, root, piece) is a chain of loads
constexpr uint32_t LT_MAX_SAMPLES = 4096;
constexpr int H = LI_HIDDEN;

// Adds one sample's MSE term (weight `scale`) and its gradient to g: the
// diagnostic entry for any first layer (cf1gpu_learned_grad).  No run calls it;
// the trainer forms its gradient from the ramps' sums (LiRamps below).
// Parameter layout: w1[0,H) b1[H,2H) w2[2H,3H) b2[3H]; hidden units are
// clipped ReLUs clamp(w1 x + b1, 0, 1) (li_act).  Queries evaluate the same
// function on its piecewise-linear form (LIRoot, li_root_eval).
CF1_HD void mlp_accumulate(const float *P, float x, float t, float scale, float *g, float &loss) {
  float z[H];
  float y = P[3 * H];
#pragma unroll
  for (int j = 0; j < H; j++) {
    z[j] = f_fma(P[j], x, P[H + j]);
    y = f_fma(P[2 * H + j], li_act(z[j]), y);
  }
  float e = y - t;
  loss += e * e * scale;
  float dy = 2.f * e * scale;
  g[3 * H] += dy;
#pragma unroll
  for (int j = 0; j < H; j++) {
    g[2 * H + j] += dy * li_act(z[j]);
    float dz = (z[j] > 0.f && z[j] < 1.f) ? dy * P[2 * H + j] : 0.f;
    g[j] += dz * x;
    g[H + j] += dz;
  }
}

// Trained parameters q (2H+1): knot logits theta[H], output weights w2[H],
// output bias b2.  The first layer is derived from the knots: widths
// d = softmax(theta), knots t_j = sum_{i<j} d_i, w1_j = 1/d_j,
// b1_j = -t_j/d_j, so unit j ramps over [t_j, t_j + d_j] and the ramps tile
// [0, 1] without gaps (a gap would be a flat stretch of the root, sending
// every key in it to one leaf).
constexpr int LI_NQ = 2 * H + 1;

// Because the ramps tile [0, 1], a sample x on ramp j has every earlier unit
// saturated and every later one at 0: its output is base_j + w2_j act(z_j)
// with base_j = b2 + sum_{i<j} w2_i, and with dy = dLoss/dy its gradient is
// dy for b2 and the w2 before j, dy act(z_j) for w2_j, dy w2_j (x, 1) for
// (w1_j, b1_j) inside the ramp.  So a step needs four sums per ramp instead
// of 16 units per sample:
//   A_j = sum dy, B_j = sum dy act(z_j), C_j = sum dz, D_j = sum dz x.
struct LiRamps {
  float knot[H], w1[H], b1[H], w2[H], base[H];
};

// Exclusive prefix (from lane 0) and suffix (from lane H - 1) sums, the sum
// and the maximum over lanes 0 .. H-1 of a warp (H = 16; the upper half warp
// repeats the lower).
CF1_D float li_prefix(float v, unsigned j) {
  float x = v;
#pragma unroll
  for (int o = 1; o < H; o <<= 1) {
    const float y = __shfl_up_sync(FULL, x, o, H);
    if (j >= (unsigned)o) x += y;
  }
  const float e = __shfl_up_sync(FULL, x, 1, H);
  return j ? e : 0.f;
}
CF1_D float li_suffix(float v, unsigned j) {
  float x = v;
#pragma unroll
  for (int o = 1; o < H; o <<= 1) {
    const float y = __shfl_down_sync(FULL, x, o, H);
    if (j + o < (unsigned)H) x += y;
  }
  const float e = __shfl_down_sync(FULL, x, 1, H);
  return j + 1 < (unsigned)H ? e : 0.f;
}
CF1_D float li_sum(float v) {
#pragma unroll
  for (int o = H / 2; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o, H);
  return v;
}
CF1_D float li_max(float v) {
#pragma unroll
  for (int o = H / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(FULL, v, o, H));
  return v;
}

// One warp, lane j (mod H) for unit j: the ramps of (theta_j, w2_j, b2) to s;
// returns the width d_j and knot t_j.
CF1_D void li_ramps(float theta, float w2, float b2, LiRamps &s, float &d, float &t) {
  const unsigned j = lane_id() % H;
  d = expf(theta - li_max(theta));
  d = d / li_sum(d);
  t = li_prefix(d, j);
  const float before = li_prefix(w2, j);
  const float w1 = 1.f / d;
  if (lane_id() < H) {
    s.knot[j] = t;
    s.w1[j] = w1;
    s.b1[j] = -t * w1;
    s.w2[j] = w2;
    s.base[j] = b2 + before;
  }
}

// The ramp of x: the last knot at or below it (binary search; knot[0] = 0).
CF1_D uint32_t li_ramp_of(const LiRamps &s, float x) {
  uint32_t j = 0;
#pragma unroll
  for (uint32_t o = H / 2; o > 0; o >>= 1) j += x >= s.knot[j + o] ? o : 0u;
  return j;
}
CF1_D float li_ramp_eval(const LiRamps &s, float x, uint32_t j, float &z) {
  z = f_fma(s.w1[j], x, s.b1[j]);
  return f_fma(s.w2[j], li_act(z), s.base[j]);
}

constexpr int LS_BLOCK = 512;  // training block
constexpr int LS_NW = LS_BLOCK / 32;
struct LiSums {
  float4 w[LS_NW][H];  // per warp and ramp: A, B, C, D
};

// Sums over a warp of four values a lane:
// four butterflies in six shuffles (two steps halve the values a lane keeps,
// three finish its quarter); lane 8 i holds value i.
CF1_D float li_reduce4(float a, float b, float c, float d) {
  const unsigned lane = lane_id();
  const bool hi = lane & 16, hi2 = lane & 8;
  float s0 = hi ? a : c, s1 = hi ? b : d;  // sent to the other half
  float k0 = hi ? c : a, k1 = hi ? d : b;  // kept
  k0 += __shfl_xor_sync(FULL, s0, 16);
  k1 += __shfl_xor_sync(FULL, s1, 16);
  float k = hi2 ? k1 : k0;
  k += __shfl_xor_sync(FULL, hi2 ? k0 : k1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) k += __shfl_xor_sync(FULL, k, o);
  return k;
}

// The block's samples x[0, n), targets t: every warp's sums per ramp.  All
// threads call it; the caller synchronises around it.  A warp takes 128
// consecutive samples at a time, four a lane (their searches and evaluations
// overlap), and reduces once per ramp among them: sorted samples (training)
// share a ramp or two, any others just take more rounds.
constexpr int LS_ROWS = 4;
CF1_D void li_accumulate(const LiRamps &s, const float *x, const float *t, uint32_t n, float scale, LiSums &sums) {
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  float *acc = reinterpret_cast<float *>(sums.w[warp]);
  acc[lane] = 0.f;
  acc[lane + 32] = 0.f;
  __syncwarp();
  for (uint32_t i0 = warp * (32 * LS_ROWS); i0 < n; i0 += LS_BLOCK * LS_ROWS) {
    float xi[LS_ROWS], dy[LS_ROWS], z[LS_ROWS];
    uint32_t j[LS_ROWS];
#pragma unroll
    for (int r = 0; r < LS_ROWS; r++) {
      const uint32_t i = i0 + r * 32 + lane;
      xi[r] = i < n ? x[i] : 0.f;
      dy[r] = i < n ? t[i] : 0.f;
      j[r] = li_ramp_of(s, xi[r]);
    }
    uint32_t todo = (uint32_t)H;  // the smallest ramp not reduced yet
#pragma unroll
    for (int r = 0; r < LS_ROWS; r++) {
      const float y = li_ramp_eval(s, xi[r], j[r], z[r]);
      dy[r] = 2.f * (y - dy[r]) * scale;
      if (i0 + r * 32 + lane >= n) j[r] = (uint32_t)H;
      todo = min(todo, j[r]);
    }
    todo = __reduce_min_sync(FULL, todo);
    while (todo < (uint32_t)H) {
      float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
      const float w2 = s.w2[todo];
      uint32_t next = (uint32_t)H;
#pragma unroll
      for (int r = 0; r < LS_ROWS; r++) {
        if (j[r] == todo) {
          const float dz = (z[r] > 0.f && z[r] < 1.f) ? dy[r] * w2 : 0.f;
          a += dy[r];
          b += dy[r] * li_act(z[r]);
          c += dz;
          d += dz * xi[r];
        } else if (j[r] > todo) {
          next = min(next, j[r]);
        }
      }
      const float v = li_reduce4(a, b, c, d);
      if ((lane & 7) == 0) acc[4 * todo + (lane >> 3)] += v;
      todo = __reduce_min_sync(FULL, next);
    }
  }
}

// One warp, lane j (mod H): the gradient with respect to (theta_j, w2_j) and
// b2 from the block's sums, by the chain rule through w1 = 1/d, b1 = -t/d, the
// knot sums and the softmax.
CF1_D void li_grad(const LiSums &sums, float d, float t, float &g_theta, float &g_w2, float &g_b2) {
  const unsigned j = lane_id() % H;
  float a = 0.f, b = 0.f, c = 0.f, e = 0.f;
#pragma unroll
  for (int w = 0; w < LS_NW; w++) {
    const float4 v = sums.w[w][j];
    a += v.x;
    b += v.y;
    c += v.z;
    e += v.w;
  }
  g_w2 = b + li_suffix(a, j);
  g_b2 = li_sum(a);
  const float w1 = 1.f / d;
  float gd = (c * t - e) * (w1 * w1);
  gd -= li_suffix(c * w1, j);  // t_j = sum_{i<j} d_i: d_i collects dL/dt_j of every j > i
  g_theta = d * (gd - li_sum(d * gd));
}

// Mean squared error of the block's samples, to every thread.
CF1_D float li_loss(const LiRamps &s, const float *x, const float *t, uint32_t n, float scale, float *sm) {
  float loss = 0.f;
  for (uint32_t i = threadIdx.x; i < n; i += LS_BLOCK) {
    float z;
    const float e = li_ramp_eval(s, x[i], li_ramp_of(s, x[i]), z) - t[i];
    loss += e * e * scale;
  }
  return block_sum<LS_BLOCK>(loss, sm);
}

// Adam step size per group: logits O(1), output weights O(1/H).
struct LiAdam {
  float m = 0.f, v = 0.f;
  // One update with gradient g; 1 / (1 - beta^step) come as c1, c2.
  CF1_D float step(float q, float g, float lr, float c1, float c2) {
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    m = beta1 * m + (1.f - beta1) * g;
    v = beta2 * v + (1.f - beta2) * g * g;
    const float mh = m * c1, vh = v * c2;
    return q - lr * mh / (sqrtf(vh) + eps);
  }
};

// Block reduction of the NPARAM gradient sums and the loss into red/sl.
CF1_D void reduce_grads(float *g, float loss, float (*red)[LI_NPARAM + 1]) {
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
  for (int p = 0; p < LI_NPARAM; p++) {
    float v = warp_sum(g[p]);
    if (lane == 0) red[warp][p] = v;
  }
  float l = warp_sum(loss);
  if (lane == 0) red[warp][LI_NPARAM] = l;
}

// One CTA per bin: full-batch Adam over the bin's CDF samples.  A step is the
// sums (all warps), a barrier, the update by one warp with a lane per unit,
// and a barrier; its latency, not throughput, is what a run of few bins waits
// for.  With 16 units per sample, the 49 gradient sums reduced one by one and
// the update on one thread a step took 9.5 us (128 bins of 200 Mbp, 300
// steps: 2.87 ms), this way 2.3 us (0.70 ms).
template <class KeyT>
__global__ void __launch_bounds__(LS_BLOCK) li_train_kernel(const KeyT *keys, const uint64_t *dist_off, LIRoot *roots,
                                                           int k, int steps, float lr, uint32_t max_samples,
                                                           float *loss_out) {
  __shared__ float sx[LT_MAX_SAMPLES], st[LT_MAX_SAMPLES];
  __shared__ LiRamps ramps;
  __shared__ LiSums sums;
  __shared__ float sm[LS_NW];
  const uint32_t b = blockIdx.x;
  const unsigned tid = threadIdx.x, j = lane_id() % H;
  const uint64_t base = dist_off[b], n = dist_off[b + 1] - base;
  LIRoot &R = roots[b];
  uint64_t hmin = 0, hmax = 0;
  float inv = 0.f;
  if (n) {
    hmin = KOps<KeyT>::high64(keys[base], k);
    hmax = KOps<KeyT>::high64(keys[base + n - 1], k);
    inv = hmax > hmin ? __fdiv_rn(1.f, u64_to_f(hmax - hmin)) : 0.f;
  }
  uint32_t S = (uint32_t)(n < max_samples ? n : max_samples);
  for (uint32_t i = tid; i < S; i += LS_BLOCK) {
    uint64_t r = (uint64_t)i * n / S;
    uint64_t h = KOps<KeyT>::high64(keys[base + r], k);
    sx[i] = f_mul(u64_to_f(h - hmin), inv);
    st[i] = (float)((double)r / (double)n);
  }
  // identity root: equal knot logits (unit j ramps over [j/H, (j+1)/H]),
  // output weights 1/H, so root(x) = x -- the index without a trained network
  float theta = 0.f, w2 = 1.f / (float)H, b2 = 0.f, d = 0.f, t = 0.f;  // lane j of warp 0: unit j's
  LiAdam at, aw, ab;
  if (tid < 32) li_ramps(theta, w2, b2, ramps, d, t);
  __syncthreads();
  const float scale = S ? 1.f / (float)S : 0.f;
  float b1t = 1.f, b2t = 1.f;
  for (int step = 0; step < steps && S > 0; step++) {
    li_accumulate(ramps, sx, st, S, scale, sums);
    __syncthreads();
    if (tid < 32) {
      float g_theta, g_w2, g_b2;
      li_grad(sums, d, t, g_theta, g_w2, g_b2);
      b1t *= 0.9f;
      b2t *= 0.999f;
      const float c1 = 1.f / (1.f - b1t), c2 = 1.f / (1.f - b2t);
      theta = at.step(theta, g_theta, lr, c1, c2);
      // projection onto w2 >= 0 (w1 = 1/d > 0 already): non-decreasing root
      w2 = fmaxf(aw.step(w2, g_w2, lr / (float)H, c1, c2), 0.f);
      b2 = ab.step(b2, g_b2, lr / (float)H, c1, c2);
      li_ramps(theta, w2, b2, ramps, d, t);
    }
    __syncthreads();
  }
  // The network on its piecewise-linear form: on [t_j, t_j + d_j) the value is
  // base_j + (w2_j / d_j) (x - t_j).  Then the output fold: an affine map with
  // a positive slope sends the bin's smallest key to 0 and its largest to
  // just below 1, so the leaves cover the keys.
  __shared__ LIRoot s_root;
  if (tid < 32) {
    if (tid < H) {
      s_root.knot[j] = t;
      s_root.base[j] = ramps.base[j];
      s_root.slope[j] = w2 / d;
    }
    if (tid == 0) {
      s_root.hmin = hmin;
      s_root.inv_range = inv;
    }
    __syncwarp();
    const float y0 = li_root_eval(s_root, li_x(s_root, hmin)), y1 = li_root_eval(s_root, li_x(s_root, hmax));
    __syncwarp();
    if (n && y1 > y0) {
      const float a = 0.99999905f / (y1 - y0);
      if (tid < H) {
        s_root.base[j] = a * (s_root.base[j] - y0);
        s_root.slope[j] *= a;
      }
      w2 *= a;
      b2 = a * b2 - a * y0;
      li_ramps(theta, w2, b2, ramps, d, t);
    }
  }
  __syncthreads();
  const float loss = li_loss(ramps, sx, st, S, scale, sm);  // with the trained parameters
  if (tid == 0) loss_out[b] = loss;
  if (tid < H) {
    R.knot[tid] = s_root.knot[tid];
    R.base[tid] = s_root.base[tid];
    R.slope[tid] = s_root.slope[tid];
  }
  if (tid == 0) {
    R.hmin = hmin;
    R.inv_range = inv;
  }
}

// The root of a tile's bin in shared memory, and the piece of it the whole
// tile lies on, when it does (piece < H).  The tile's keys ascend and li_x
// does not decrease with the key, so when its first and last key are on one
// piece, all are: most tiles then skip the 15 comparisons per key, and none
// reads the root from global memory (200 Mbp, the three passes over the keys:
// 4.07 -> 2.33 ms with this, larger tiles and the err pass's shared maxima).  (The judge does not assume the order: a tile with keys out of
// order is reported bad whatever their pieces.)
struct LiTile {
  LIRoot r;
  uint32_t piece;
};
CF1_D uint32_t li_piece(const LIRoot &r, float x) {
  uint32_t j = 0;
#pragma unroll
  for (int i = 1; i < H; i++) j += x >= r.knot[i] ? 1u : 0u;
  return j;
}
template <class KeyT>
CF1_D void li_tile(const LIRoot &R, const KeyT *keys, uint64_t start, uint64_t end, int k, LiTile &t) {
  constexpr uint32_t NWD = sizeof(LIRoot) / 4;
  static_assert(sizeof(LIRoot) % 4 == 0 && NWD <= LT_BLOCK, "a word a thread");
  if (threadIdx.x < NWD)
    reinterpret_cast<uint32_t *>(&t.r)[threadIdx.x] = reinterpret_cast<const uint32_t *>(&R)[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t a = li_piece(t.r, li_x(t.r, KOps<KeyT>::high64(keys[start], k)));
    const uint32_t b = li_piece(t.r, li_x(t.r, KOps<KeyT>::high64(keys[end - 1], k)));
    t.piece = a == b ? a : (uint32_t)H;
  }
  __syncthreads();
}
// Leaf of the key with high bits h: li_leaf_of(li_root_eval(li_x(h))), the
// piece given by the tile when it has one.
CF1_D uint32_t li_tile_leaf(const LiTile &t, uint64_t h) {
  const float x = li_x(t.r, h);
  const uint32_t j = t.piece < (uint32_t)H ? t.piece : li_piece(t.r, x);
  return li_leaf_of(t.r, f_fma(t.r.slope[j], f_sub(x, t.r.knot[j]), t.r.base[j]));
}

// Runs of equal leaves inside a warp (the lanes hold consecutive keys, and a
// monotone root sends consecutive keys to non-decreasing leaves, so a leaf is
// one run; the reductions below stay exact for any order): the lane of the
// run's first key, from the ballot of run heads.
CF1_D uint32_t run_head_lane(uint32_t leaf, unsigned lane, unsigned &heads) {
  const uint32_t prev = __shfl_up_sync(FULL, leaf, 1);
  heads = __ballot_sync(FULL, lane == 0 || leaf != prev);
  return 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
}
CF1_D bool run_tail(uint32_t leaf, unsigned lane) {
  const uint32_t next = __shfl_down_sync(FULL, leaf, 1);
  return lane == 31 || leaf != next;
}

// Per leaf: first and last local rank and key count, one atomic of each kind
// per run of a warp.
template <class KeyT>
__global__ void __launch_bounds__(LT_BLOCK) li_assign_kernel(const KeyT *keys, const uint64_t *dist_off,
                                                            const uint32_t *tile_off, uint32_t nbins,
                                                            const LIRoot *roots, int k, uint32_t *lfirst,
                                                            uint32_t *llast, uint32_t *ln) {
  const uint32_t t = blockIdx.x;
  if (t >= tile_off[nbins]) return;
  TileSpan sp = tile_span(dist_off, tile_off, nbins, t, LT_TILE);
  __shared__ LiTile s_tile;
  li_tile(roots[sp.seg], keys, sp.start, sp.end, k, s_tile);
  const LIRoot &R = s_tile.r;
  const uint64_t base = dist_off[sp.seg];
  const unsigned lane = lane_id();
  for (uint64_t i0 = sp.start; i0 < sp.end; i0 += LT_BLOCK) {
    uint64_t i = i0 + threadIdx.x;
    bool act = i < sp.end;
    uint32_t leaf = act ? li_tile_leaf(s_tile, KOps<KeyT>::high64(keys[i], k)) : 0xFFFFFFFFu;
    uint32_t rank = (uint32_t)(i - base);
    unsigned heads;
    const uint32_t hl = run_head_lane(leaf, lane, heads);
    const bool tail = run_tail(leaf, lane);
    if (act) {
      const uint64_t g = R.leaf_off + leaf;
      if (lane == hl) atomicMin(&lfirst[g], rank);
      if (tail) {
        atomicMax(&llast[g], rank);
        atomicAdd(&ln[g], lane - hl + 1);
      }
    }
  }
}

template <class KeyT>
__global__ void li_fit_kernel(const KeyT *keys, const uint64_t *dist_off, const uint64_t *leaf_off, uint32_t nbins,
                              uint64_t total_leaves, int k, const uint32_t *lfirst, const uint32_t *llast,
                              const uint32_t *ln, LILeaf *leaves) {
  uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total_leaves) return;
  LILeaf L;
  L.n = ln[g];
  if (L.n == 0) {
    L.hfirst = 0;
    L.first_rank = 0;
    L.err = 0;
    L.slope = 0.f;
    leaves[g] = L;
    return;
  }
  uint32_t b = upper_segment(leaf_off, nbins, g);
  uint64_t base = dist_off[b];
  uint32_t f = lfirst[g], l = llast[g];
  uint64_t hf = KOps<KeyT>::high64(keys[base + f], k), hl = KOps<KeyT>::high64(keys[base + l], k);
  L.hfirst = hf;
  L.first_rank = f;
  L.err = 0;
  L.slope = (l > f && hl > hf) ? __fdiv_rn((float)(l - f), u64_to_f(hl - hf)) : 0.f;
  leaves[g] = L;
}

// Per leaf: the largest |prediction - rank| over its keys.  A tile's leaves
// are consecutive (about 512 of them): their maxima are collected in shared
// memory (leaves outside the window, if any, go to global memory directly).
constexpr uint32_t LE_WIN = 1024;
template <class KeyT>
__global__ void __launch_bounds__(LT_BLOCK, 6) li_err_kernel(const KeyT *keys, const uint64_t *dist_off,
                                                         const uint32_t *tile_off, uint32_t nbins,
                                                         const LIRoot *roots, int k, LILeaf *leaves) {
  __shared__ LiTile s_tile;
  __shared__ uint32_t s_err[LE_WIN];
  const uint32_t t = blockIdx.x;
  if (t >= tile_off[nbins]) return;
  TileSpan sp = tile_span(dist_off, tile_off, nbins, t, LT_TILE);
  for (uint32_t i = threadIdx.x; i < LE_WIN; i += LT_BLOCK) s_err[i] = 0;
  li_tile(roots[sp.seg], keys, sp.start, sp.end, k, s_tile);
  const uint32_t leaf0 = li_tile_leaf(s_tile, KOps<KeyT>::high64(keys[sp.start], k));
  LILeaf *bl = leaves + s_tile.r.leaf_off;
  uint32_t rank = (uint32_t)(sp.start - dist_off[sp.seg]) + threadIdx.x;
#pragma unroll 4
  for (uint64_t i = sp.start + threadIdx.x; i < sp.end; i += LT_BLOCK, rank += LT_BLOCK) {
    const uint64_t h = KOps<KeyT>::high64(keys[i], k);
    const uint32_t leaf = li_tile_leaf(s_tile, h);
    int64_t d = li_predict(bl[leaf], h) - (int64_t)rank;
    d = d < 0 ? -d : d;
    const uint32_t e = d > 0xFFFFFFF0ll ? 0xFFFFFFF0u : (uint32_t)d;
    if (leaf - leaf0 < LE_WIN) atomicMax(&s_err[leaf - leaf0], e);
    else atomicMax(&bl[leaf].err, e);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < LE_WIN; i += LT_BLOCK)
    if (s_err[i]) atomicMax(&bl[leaf0 + i].err, s_err[i]);
}

// One CTA per bin: the bin's largest leaf error decides learned vs BBHash.
__global__ void __launch_bounds__(LT_BLOCK) li_decide_kernel(const uint64_t *dist_off, LIRoot *roots,
                                                            const LILeaf *leaves, uint32_t max_err, uint32_t *sel,
                                                            unsigned long long *errsum) {
  __shared__ uint32_t s_max;
  __shared__ unsigned long long s_sum;
  const uint32_t b = blockIdx.x;
  LIRoot &R = roots[b];
  if (threadIdx.x == 0) {
    s_max = 0;
    s_sum = 0;
  }
  __syncthreads();
  uint32_t m = 0;
  unsigned long long sum = 0;
  for (uint32_t j = threadIdx.x; j < R.n_leaves; j += LT_BLOCK) {
    const LILeaf &L = leaves[R.leaf_off + j];
    if (L.n) {
      m = L.err > m ? L.err : m;
      sum += (unsigned long long)L.err * L.n;
    }
  }
  atomicMax(&s_max, m);
  atomicAdd(&s_sum, sum);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t n = dist_off[b + 1] - dist_off[b];
    R.max_err = s_max;
    R.use_learned = (n > 0 && s_max <= max_err) ? 1u : 0u;
    sel[b] = (n > 0 && !R.use_learned) ? 1u : 0u;
    errsum[b] = s_sum;
  }
}

// Verification, the bijection judge: every key of a learned bin must come
// back as its own rank.  A query for keys[i] is the lower bound of the key in
// its window (li_local_slot); in a bin whose keys strictly increase that is i
// exactly when the window holds i.  So the pass checks each key's window and
// the order of each adjacent pair -- together a proof that the learned index
// maps the bin's keys one to one onto [0, n) -- in one streaming read of the
// keys, with no search.
template <class KeyT>
__global__ void __launch_bounds__(LT_BLOCK, 6) li_verify_kernel(const KeyT *keys, const uint64_t *dist_off,
                                                           const uint32_t *tile_off, uint32_t nbins, LIView v,
                                                           uint32_t *miss) {
  const uint32_t t = blockIdx.x;
  if (t >= tile_off[nbins]) return;
  TileSpan sp = tile_span(dist_off, tile_off, nbins, t, LT_TILE);
  if (!v.roots[sp.seg].use_learned) return;
  const uint64_t base = dist_off[sp.seg];
  __shared__ LiTile s_tile;
  li_tile(v.roots[sp.seg], keys, sp.start, sp.end, v.k, s_tile);
  // the window [p - err, p + err] clamped to the bin's ranks holds the rank r
  // exactly when |p - r| <= err
  const LILeaf *leaves = v.leaves + s_tile.r.leaf_off;
  bool bad = false;
#pragma unroll 4
  for (uint64_t i = sp.start + threadIdx.x; i < sp.end; i += LT_BLOCK) {
    const KeyT key = keys[i];
    const uint64_t h = KOps<KeyT>::high64(key, v.k);
    const LILeaf lf = leaves[li_tile_leaf(s_tile, h)];
    int64_t d = li_predict(lf, h) - (int64_t)(i - base);
    d = d < 0 ? -d : d;
    bad |= lf.n == 0 || d > (int64_t)lf.err || (i > base && !(keys[i - 1] < key));
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) miss[sp.seg] = 1;
}

__global__ void li_fixup_kernel(LIRoot *roots, const uint32_t *miss, uint32_t *sel, uint32_t nbins) {
  uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < nbins && miss[b]) {
    roots[b].use_learned = 0;
    sel[b] = 1;
  }
}

__global__ void __launch_bounds__(LT_BLOCK) li_grad_kernel(const float *params, const float *x, const float *t,
                                                          uint32_t n, float *grad, float *loss_out) {
  __shared__ float P[LI_NPARAM];
  __shared__ float red[LT_NW][LI_NPARAM + 1];
  if (threadIdx.x < LI_NPARAM) P[threadIdx.x] = params[threadIdx.x];
  __syncthreads();
  float g[LI_NPARAM];
#pragma unroll
  for (int p = 0; p < LI_NPARAM; p++) g[p] = 0.f;
  float loss = 0.f;
  const float scale = n ? 1.f / (float)n : 0.f;
  for (uint32_t i = threadIdx.x; i < n; i += LT_BLOCK) mlp_accumulate(P, x[i], t[i], scale, g, loss);
  reduce_grads(g, loss, red);
  __syncthreads();
  if (threadIdx.x <= LI_NPARAM) {
    float s = 0.f;
    for (int w = 0; w < LT_NW; w++) s += red[w][threadIdx.x];
    if (threadIdx.x < LI_NPARAM) grad[threadIdx.x] = s;
    else *loss_out = s;
  }
}

// One training step's gradient with respect to the trained parameters q:
// the same li_ramps, li_accumulate and li_grad calls li_train_kernel makes
// before its Adam update, over n given samples.
__global__ void __launch_bounds__(LS_BLOCK) li_grad_q_kernel(const float *q, const float *x, const float *t,
                                                            uint32_t n, float *gq_out, float *loss_out) {
  __shared__ LiRamps ramps;
  __shared__ LiSums sums;
  __shared__ float sm[LS_NW];
  const unsigned tid = threadIdx.x, j = tid % H;
  float d = 0.f, tk = 0.f;
  if (tid < 32) li_ramps(q[j], q[H + j], q[2 * H], ramps, d, tk);
  __syncthreads();
  const float scale = n ? 1.f / (float)n : 0.f;
  li_accumulate(ramps, x, t, n, scale, sums);
  __syncthreads();
  if (tid < 32) {
    float g_theta, g_w2, g_b2;
    li_grad(sums, d, tk, g_theta, g_w2, g_b2);
    if (tid < H) {
      gq_out[tid] = g_theta;
      gq_out[H + tid] = g_w2;
    }
    if (tid == 0) gq_out[2 * H] = g_b2;
  }
  const float loss = li_loss(ramps, x, t, n, scale, sm);
  if (tid == 0) *loss_out = loss;
}

}  // namespace

template <class KeyT>
void LearnedBuild<KeyT>::build(const KeyT *keys, const uint64_t *dist_off, uint32_t nb, int k, const LearnedOpts &o,
                               cudaStream_t s) {
  nbins = nb;
  stats = LearnedStats();
  std::vector<uint64_t> hoff(nbins + 1);
  CF1_CUDA(cudaMemcpyAsync(hoff.data(), dist_off, (nbins + 1) * sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaStreamSynchronize(s));
  std::vector<LIRoot> hroots(nbins);
  std::vector<uint64_t> hleaf(nbins + 1);
  uint64_t total_leaves = 0;
  uint32_t leaf_size = o.leaf_size ? o.leaf_size : 32;
  for (uint32_t b = 0; b < nbins; b++) {
    uint64_t n = hoff[b + 1] - hoff[b];
    uint64_t nl = n ? (n + leaf_size - 1) / leaf_size : 1;
    std::memset(&hroots[b], 0, sizeof(LIRoot));
    for (int p = 0; p < H; p++) {  // identity root until training writes its own
      hroots[b].knot[p] = (float)p / (float)H;
      hroots[b].base[p] = (float)p / (float)H;
      hroots[b].slope[p] = 1.f;
    }
    hroots[b].n_leaves = (uint32_t)nl;
    hroots[b].leaf_off = total_leaves;
    hroots[b].use_learned = n > 0;
    hleaf[b] = total_leaves;
    total_leaves += nl;
  }
  hleaf[nbins] = total_leaves;
  uint64_t n_total = hoff[nbins];
  LIRoot *roots = roots_.get<LIRoot>(nbins);
  uint64_t *leaf_off = leaf_off_.get<uint64_t>(nbins + 1);
  CF1_CUDA(cudaMemcpyAsync(roots, hroots.data(), nbins * sizeof(LIRoot), cudaMemcpyHostToDevice, s));
  CF1_CUDA(cudaMemcpyAsync(leaf_off, hleaf.data(), (nbins + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
  float *loss = loss_.get<float>(nbins);
  CF1_CUDA(cudaMemsetAsync(loss, 0, nbins * sizeof(float), s));
  uint32_t samples = o.max_samples > LT_MAX_SAMPLES ? LT_MAX_SAMPLES : (o.max_samples ? o.max_samples : 1);
  if (nbins) {
    li_train_kernel<KeyT><<<nbins, LS_BLOCK, 0, s>>>(keys, dist_off, roots, k, o.train_steps < 0 ? 0 : o.train_steps,
                                                     o.lr, samples, loss);
    CF1_LAUNCH_CHECK();
  }
  uint32_t *lfirst = lfirst_.get<uint32_t>(total_leaves);
  uint32_t *llast = llast_.get<uint32_t>(total_leaves);
  uint32_t *ln = ln_.get<uint32_t>(total_leaves);
  LILeaf *leaves = leaves_.get<LILeaf>(total_leaves);
  CF1_CUDA(cudaMemsetAsync(lfirst, 0xFF, total_leaves * 4, s));
  CF1_CUDA(cudaMemsetAsync(llast, 0, total_leaves * 4, s));
  CF1_CUDA(cudaMemsetAsync(ln, 0, total_leaves * 4, s));
  uint32_t *tile_off = tile_off_.get<uint32_t>(nbins + 1);
  segment_tiles(dist_off, nbins, LT_TILE, tile_off, s);
  uint32_t ub = (uint32_t)(ceil_div(n_total, LT_TILE) + nbins);
  li_assign_kernel<KeyT><<<ub, LT_BLOCK, 0, s>>>(keys, dist_off, tile_off, nbins, roots, k, lfirst, llast, ln);
  CF1_LAUNCH_CHECK();
  li_fit_kernel<KeyT><<<(unsigned)ceil_div(total_leaves, 256), 256, 0, s>>>(keys, dist_off, leaf_off, nbins, total_leaves,
                                                                            k, lfirst, llast, ln, leaves);
  CF1_LAUNCH_CHECK();
  li_err_kernel<KeyT><<<ub, LT_BLOCK, 0, s>>>(keys, dist_off, tile_off, nbins, roots, k, leaves);
  CF1_LAUNCH_CHECK();
  uint32_t *sel = sel_.get<uint32_t>(nbins);
  unsigned long long *errsum = errsum_.get<unsigned long long>(nbins);
  li_decide_kernel<<<nbins, LT_BLOCK, 0, s>>>(dist_off, roots, leaves, o.max_err, sel, errsum);
  CF1_LAUNCH_CHECK();
  uint32_t *miss = lfirst;  // reuse: one flag per bin
  CF1_CUDA(cudaMemsetAsync(miss, 0, nbins * 4, s));
  li_verify_kernel<KeyT><<<ub, LT_BLOCK, 0, s>>>(keys, dist_off, tile_off, nbins, view(k), miss);
  CF1_LAUNCH_CHECK();
  li_fixup_kernel<<<(unsigned)ceil_div(nbins, 256), 256, 0, s>>>(roots, miss, sel, nbins);
  CF1_LAUNCH_CHECK();
  // stats
  std::vector<LIRoot> r2(nbins);
  std::vector<unsigned long long> es(nbins);
  std::vector<float> hl(nbins);
  std::vector<uint32_t> hmiss(nbins);
  CF1_CUDA(cudaMemcpyAsync(hmiss.data(), miss, nbins * 4, cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaMemcpyAsync(r2.data(), roots, nbins * sizeof(LIRoot), cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaMemcpyAsync(es.data(), errsum, nbins * 8, cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaMemcpyAsync(hl.data(), loss, nbins * 4, cudaMemcpyDeviceToHost, s));
  CF1_CUDA(cudaStreamSynchronize(s));
  double esum = 0, wsum = 0, keys_learned = 0, lsum = 0;
  uint64_t nonempty = 0;
  for (uint32_t b = 0; b < nbins; b++) {
    uint64_t n = hoff[b + 1] - hoff[b];
    if (!n) continue;
    nonempty++;
    lsum += hl[b];
    stats.max_err_all = r2[b].max_err > stats.max_err_all ? r2[b].max_err : stats.max_err_all;
    stats.verify_miss_bins += hmiss[b] ? 1 : 0;
    if (r2[b].use_learned) {
      stats.learned_bins++;
      stats.max_err = r2[b].max_err > stats.max_err ? r2[b].max_err : stats.max_err;
      esum += (double)es[b];
      wsum += 2.0 * (double)es[b] + (double)n;
      keys_learned += (double)n;
    } else {
      stats.fallback_bins++;
    }
  }
  stats.leaves = total_leaves;
  stats.mean_err = keys_learned ? esum / keys_learned : 0;
  stats.mean_window = keys_learned ? wsum / keys_learned : 0;
  stats.train_loss = nonempty ? lsum / nonempty : 0;
  stats.bytes = nbins * sizeof(LIRoot) + total_leaves * sizeof(LILeaf);
}

template <class KeyT>
LIView LearnedBuild<KeyT>::view(int k) const {
  LIView v;
  v.roots = roots_.as<const LIRoot>();
  v.leaves = leaves_.as<const LILeaf>();
  v.k = k;
  return v;
}

template struct LearnedBuild<uint64_t>;
template struct LearnedBuild<Key2>;

void learned_grad_host(const float *params, const float *x, const float *t, size_t n, float *grad, float *loss) {
  DevBuf dp, dx, dt, dg;
  float *p = dp.get<float>(LI_NPARAM + 1);
  float *xx = dx.get<float>(n + 1);
  float *tt = dt.get<float>(n + 1);
  float *g = dg.get<float>(LI_NPARAM + 1);
  CF1_CUDA(cudaMemcpy(p, params, LI_NPARAM * 4, cudaMemcpyHostToDevice));
  if (n) {
    CF1_CUDA(cudaMemcpy(xx, x, n * 4, cudaMemcpyHostToDevice));
    CF1_CUDA(cudaMemcpy(tt, t, n * 4, cudaMemcpyHostToDevice));
  }
  li_grad_kernel<<<1, LT_BLOCK>>>(p, xx, tt, (uint32_t)n, g, g + LI_NPARAM);
  CF1_LAUNCH_CHECK();
  float out[LI_NPARAM + 1];
  CF1_CUDA(cudaMemcpy(out, g, (LI_NPARAM + 1) * 4, cudaMemcpyDeviceToHost));
  std::memcpy(grad, out, LI_NPARAM * 4);
  *loss = out[LI_NPARAM];
}

void learned_grad_q_host(const float *q, const float *x, const float *t, size_t n, float *grad_q, float *loss) {
  DevBuf dq, dx, dt, dg;
  float *qq = dq.get<float>(LI_NQ + 1);
  float *xx = dx.get<float>(n + 1);
  float *tt = dt.get<float>(n + 1);
  float *g = dg.get<float>(LI_NQ + 1);
  CF1_CUDA(cudaMemcpy(qq, q, LI_NQ * 4, cudaMemcpyHostToDevice));
  if (n) {
    CF1_CUDA(cudaMemcpy(xx, x, n * 4, cudaMemcpyHostToDevice));
    CF1_CUDA(cudaMemcpy(tt, t, n * 4, cudaMemcpyHostToDevice));
  }
  li_grad_q_kernel<<<1, LS_BLOCK>>>(qq, xx, tt, (uint32_t)n, g, g + LI_NQ);
  CF1_LAUNCH_CHECK();
  float out[LI_NQ + 1];
  CF1_CUDA(cudaMemcpy(out, g, (LI_NQ + 1) * 4, cudaMemcpyDeviceToHost));
  std::memcpy(grad_q, out, LI_NQ * 4);
  *loss = out[LI_NQ];
}

}  // namespace cf1
