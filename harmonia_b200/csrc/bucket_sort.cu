// Partition passes of the bucket sort (bucket_sort.cuh).
#include "bucket_sort.cuh"

#include <algorithm>

namespace hm {
namespace bsort {

namespace {

// ---- range and counts ----

constexpr int kRangeThreads = 256;
constexpr int kRangePer = 8;
constexpr int kRangeStep = 64;  // every 64th key

// Lowest and highest of a strided sample of the keys (always the first and
// the last); the last CTA to finish makes the map.  Keys beyond the sample's
// range go to the end buckets: about kRangeStep on either side, far inside a
// bucket's margin.
__global__ void __launch_bounds__(kRangeThreads) range_kernel(const int64_t *__restrict__ keys, int64_t n,
                                                              uint32_t nb, Ctl *ctl) {
  pdl_enter();
  __shared__ unsigned long long lo_w[kRangeThreads / 32], hi_w[kRangeThreads / 32];
  const int64_t slots = (int64_t)gridDim.x * kRangeThreads * kRangePer;
  int64_t k[kRangePer];
#pragma unroll
  for (int j = 0; j < kRangePer; j++) {
    const int64_t x = ((int64_t)blockIdx.x * kRangePer + j) * kRangeThreads + threadIdx.x;
    k[j] = __ldg(keys + min(x == slots - 1 ? n - 1 : x * kRangeStep, n - 1));
  }
  unsigned long long inv_lo = 0, hi = 0;
#pragma unroll
  for (int j = 0; j < kRangePer; j++) {
    const unsigned long long u = (unsigned long long)k[j] ^ kSign;
    inv_lo = max(inv_lo, ~u);
    hi = max(hi, u);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    inv_lo = max(inv_lo, __shfl_xor_sync(0xffffffffu, inv_lo, o));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  if ((threadIdx.x & 31) == 0) {
    lo_w[threadIdx.x >> 5] = inv_lo;
    hi_w[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < kRangeThreads / 32; w++) {
    inv_lo = max(inv_lo, lo_w[w]);
    hi = max(hi, hi_w[w]);
  }
  atomicMax(&ctl->inv_lo, inv_lo);
  atomicMax(&ctl->hi, hi);
  __threadfence();
  if (atomicAdd(&ctl->done, 1u) != gridDim.x - 1) return;
  __threadfence();
  const unsigned long long lo_all = ~atomicMax(&ctl->inv_lo, 0ull), hi_all = atomicMax(&ctl->hi, 0ull);
  Map m;
  make_map((int64_t)(lo_all ^ kSign), (int64_t)(hi_all ^ kSign), nb, &m);
  ctl->map = m;
}

constexpr int kCountThreads = 1024;
constexpr int kCountPer = 8;

// Pairs per bucket.  A counter that reaches kCap in one CTA sets skew (the
// batch is then not sorted here, and what a 16-bit counter carries into its
// neighbour no longer matters).
__global__ void __launch_bounds__(kCountThreads) count_kernel(const int64_t *__restrict__ keys, int64_t n,
                                                              uint32_t nb, Ctl *ctl, uint32_t *__restrict__ count) {
  pdl_enter();
  extern __shared__ __align__(16) uint32_t packed[];  // two 16-bit counters a word
  const Map map = ctl->map;
  for (uint32_t i = threadIdx.x; i < (nb + 1) / 2; i += kCountThreads) packed[i] = 0;
  __syncthreads();
  bool skew = false;
  const int64_t step = (int64_t)gridDim.x * kCountThreads * kCountPer;
  for (int64_t base = (int64_t)blockIdx.x * kCountThreads * kCountPer; base < n; base += step) {
    int64_t k[kCountPer];
#pragma unroll
    for (int j = 0; j < kCountPer; j++) {
      const int64_t i = base + j * kCountThreads + threadIdx.x;
      k[j] = i < n ? __ldg(keys + i) : 0;
    }
#pragma unroll
    for (int j = 0; j < kCountPer; j++) {
      if (base + j * kCountThreads + threadIdx.x < n) {
        const uint32_t b = map(k[j]);
        const uint32_t sh = (b & 1) * 16;
        skew |= ((atomicAdd(&packed[b >> 1], 1u << sh) >> sh) & 0xffffu) >= kCap;
      }
    }
  }
  if (__syncthreads_or(skew)) {
    if (threadIdx.x == 0) atomicOr(&ctl->skew, 1u);
    return;
  }
  for (uint32_t i = threadIdx.x; i < nb; i += kCountThreads) {
    const uint32_t c = (packed[i >> 1] >> ((i & 1) * 16)) & 0xffffu;
    if (c) atomicAdd(count + i, c);
  }
}

constexpr int kStartThreads = 1024;

// Exclusive scan of the counts: CTA c owns buckets [1024 c, 1024 c + 1024) and
// adds up the counts before them itself (at most 64 loads a thread from L2).
// Sets skew if a bucket is over kCap.
__global__ void __launch_bounds__(kStartThreads) starts_kernel(const uint32_t *__restrict__ count, uint32_t nb, int l2,
                                                               uint32_t n, uint32_t *__restrict__ start,
                                                               uint32_t *__restrict__ cur1,
                                                               uint32_t *__restrict__ cur2, Ctl *ctl) {
  pdl_enter();
  __shared__ uint32_t wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t first = blockIdx.x * kStartThreads;
  uint32_t before = 0;
  for (uint32_t i = tid; i < first; i += kStartThreads) before += count[i];
  const uint32_t mine = first + tid < nb ? count[first + tid] : 0;
  // the sums of the counts before this CTA's, spread over its threads, enter
  // the scan through the first warp
#pragma unroll
  for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __shared__ uint32_t bsum[32];
  if (lane == 31) wsum[warp] = incl;
  if (lane == 0) bsum[warp] = before;
  __syncthreads();
  uint32_t at = incl - mine;
  for (int w = 0; w < 32; w++) at += bsum[w];
  for (int w = 0; w < warp; w++) at += wsum[w];
  const uint32_t b = first + tid;
  if (b < nb) {
    start[b] = at;
    cur2[b] = at;
    if ((b & ((1u << l2) - 1)) == 0) cur1[b >> l2] = at;
    if (b == nb - 1) start[nb] = n;
  }
  if (__syncthreads_or(mine > (uint32_t)kCap) && tid == 0) atomicOr(&ctl->skew, 1u);
}

// ---- partition pass ----

// 256 threads of 8 pairs, six CTAs an SM: two 2^24-pair passes of 16-B pairs
// take 105 and 120 us; 512 x 8 with three CTAs 106 and 127, with two 118 and
// 140; 1024 x 4 with two 119 and 142; 256 x 16 with three 120 and 128 (82 us
// each at the measured copy rate).  The barriers between the steps of a tile
// cost less in small CTAs.
constexpr int kScThreads = 256;
constexpr int kScPer = 8;
constexpr int kScTile = kScThreads * kScPer;  // pairs of a tile
static_assert(kScThreads == 256, "a thread per digit");

template <typename V>
constexpr int scatter_smem() {
  return kScTile * (8 + (int)sizeof(V));
}

// One tile per CTA: digit counts by shared-memory atomics (whose old value is
// the pair's rank in its digit run), one cursor atomic per digit reserves the
// tile's run, the pairs are staged grouped by digit and written out so that
// consecutive threads store consecutive slots.  SECOND: tiles are cut inside
// the first pass's buckets (found from their starts), digit = the low l2 bits.
// GEN: payload = position.
template <typename V, bool GEN, bool SECOND>
__global__ void __launch_bounds__(kScThreads, 6) scatter_kernel(const int64_t *__restrict__ keys,
                                                                const V *__restrict__ vals, int64_t n,
                                                                const Ctl *__restrict__ ctl,
                                                                const uint32_t *__restrict__ start, int l1, int l2,
                                                                uint32_t *__restrict__ cur, int64_t *__restrict__ k_out,
                                                                V *__restrict__ v_out) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char dyn[];
  int64_t *skey = reinterpret_cast<int64_t *>(dyn);
  V *sval = reinterpret_cast<V *>(dyn + 8 * kScTile);
  __shared__ uint32_t cnt[256], tstart[256], adj[256];
  __shared__ uint32_t wsum[8];
  __shared__ uint32_t t_first, t_end, t_bucket;
  if (ctl->skew) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Map map = ctl->map;
  int64_t i0, i1;
  uint32_t bucket = 0;
  cnt[tid] = 0;
  if constexpr (SECOND) {
    // tiles of first-pass bucket tid: scan, and the bucket this CTA's tile is in
    uint32_t s = 0, e = 0, tiles = 0, incl = 0;
    if (tid < 1 << l1) {
      s = start[(uint32_t)tid << l2];
      e = start[(uint32_t)(tid + 1) << l2];
      tiles = (e - s + kScTile - 1) / kScTile;
    }
    incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    if (tid == 0) t_end = 0;
    __syncthreads();
    for (int w = 0; w < warp; w++) incl += wsum[w];
    if (blockIdx.x < incl && blockIdx.x >= incl - tiles) {
      t_first = s + (blockIdx.x - (incl - tiles)) * kScTile;
      t_end = min(e, t_first + kScTile);
      t_bucket = tid;
    }
    __syncthreads();
    if (t_end == 0) return;  // past the last tile
    i0 = t_first;
    i1 = t_end;
    bucket = t_bucket << l2;
  } else {
    i0 = (int64_t)blockIdx.x * kScTile;
    i1 = min(n, i0 + kScTile);
    __syncthreads();
  }
  const uint32_t sh = SECOND ? 0 : l2, mask = SECOND ? (1u << l2) - 1 : ~0u;
  int64_t k[kScPer];
#pragma unroll
  for (int j = 0; j < kScPer; j++) {
    const int64_t i = i0 + j * kScThreads + tid;
    k[j] = i < i1 ? __ldg(keys + i) : 0;
  }
  // the payloads go straight to their staged places once those are known
  constexpr int kLine = 128 / (int)sizeof(V);
  if (!GEN && i0 + tid * kLine < i1) prefetch_l2(vals + i0 + tid * kLine);
  uint32_t dr[kScPer];  // digit << 16 | rank in the tile's digit run
#pragma unroll
  for (int j = 0; j < kScPer; j++) {
    if (i0 + j * kScThreads + tid < i1) {
      const uint32_t d = (map(k[j]) >> sh) & mask;
      dr[j] = d << 16 | atomicAdd(&cnt[d], 1u);
    }
  }
  __syncthreads();
  uint32_t mine = 0, incl = 0, at = 0;
  mine = cnt[tid];
  if (mine) at = atomicAdd(cur + bucket + tid, mine);
  incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t before = incl - mine;
  for (int w = 0; w < warp; w++) before += wsum[w];
  tstart[tid] = before;
  adj[tid] = at - before;  // slot s of digit d goes to adj[d] + s (modulo 2^32)
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kScPer; j++) {
    if (i0 + j * kScThreads + tid < i1) {
      const uint32_t sl = tstart[dr[j] >> 16] + (dr[j] & 0xffffu);
      if constexpr (GEN) {
        sval[sl] = (V)(i0 + j * kScThreads + tid);
      } else {
        cp_async_element(sval + sl, vals + i0 + j * kScThreads + tid);
      }
      skey[sl] = k[j];
    }
  }
  if constexpr (!GEN) cp_async_wait();
  __syncthreads();
  const int m = (int)(i1 - i0);
#pragma unroll
  for (int j = 0; j < kScPer; j++) {
    const int sl = j * kScThreads + tid;
    if (sl < m) {
      const int64_t key = skey[sl];
      const uint32_t o = adj[(map(key) >> sh) & mask] + (uint32_t)sl;
      k_out[o] = key;
      v_out[o] = sval[sl];
    }
  }
}

}  // namespace

namespace {

size_t place(int64_t n, char *base, Work *w) {
  const Shape sh = shape_for(n);
  const int64_t nb = (int64_t)1 << sh.bits;
  size_t off = 0;
  auto take = [&](int64_t bytes) {
    char *p = base ? base + off : nullptr;
    off += (size_t)align_up(bytes, 256);
    return p;
  };
  Work x;
  x.ctl = reinterpret_cast<Ctl *>(take(sizeof(Ctl)));
  x.count = reinterpret_cast<uint32_t *>(take(4 * nb));
  x.start = reinterpret_cast<uint32_t *>(take(4 * (nb + 1)));
  x.cur1 = reinterpret_cast<uint32_t *>(take(4 * 256));
  x.cur2 = reinterpret_cast<uint32_t *>(take(4 * nb));
  if (w) *w = x;
  return off;
}

}  // namespace

size_t work_bytes(int64_t n) { return place(n, nullptr, nullptr); }

Work layout(int64_t n, void *base) {
  Work w;
  place(n, static_cast<char *>(base), &w);
  return w;
}

template <typename V>
int partition_pairs(const int64_t *keys, const V *vals, int64_t n, int64_t *k1, V *v1, int64_t *k2, V *v2,
                    const Work &w, int sms, cudaStream_t s) {
  const Shape sh = shape_for(n);
  const uint32_t nb = 1u << sh.bits;
  // the control block and the counts lie side by side
  cudaMemsetAsync(w.ctl, 0, (char *)(w.count + nb) - (char *)w.ctl, s);
  if (sh.bits == 0) return 0;
  constexpr int64_t kRangeKeys = (int64_t)kRangeThreads * kRangePer * kRangeStep;
  launch_pdl(range_kernel, (unsigned)((n + kRangeKeys - 1) / kRangeKeys), kRangeThreads, 0, s, keys, n, nb, w.ctl);
  const size_t csm = ((size_t)nb * 2 + 15) & ~(size_t)15;
  const int per_sm = csm > 100 * 1024 ? 1 : 2;
  opt_in_smem((const void *)count_kernel, 2 << kMaxBits);
  const int64_t count_ctas = (n + kCountThreads * kCountPer - 1) / (kCountThreads * kCountPer);
  launch_pdl(count_kernel, (unsigned)std::min<int64_t>(count_ctas, (int64_t)sms * per_sm), kCountThreads, csm, s, keys,
             n, nb, w.ctl, w.count);
  launch_pdl(starts_kernel, (nb + kStartThreads - 1) / kStartThreads, kStartThreads, 0, s, w.count, nb, sh.l2,
             (uint32_t)n, w.start, w.cur1, w.cur2, w.ctl);
  const unsigned tiles = (unsigned)((n + kScTile - 1) / kScTile);
  constexpr int sm = scatter_smem<V>();
  if (vals) {
    opt_in_smem((const void *)scatter_kernel<V, false, false>, sm);
    launch_pdl(scatter_kernel<V, false, false>, tiles, kScThreads, sm, s, keys, vals, n, w.ctl, w.start, sh.l1, sh.l2,
               w.cur1, k1, v1);
  } else {
    opt_in_smem((const void *)scatter_kernel<V, true, false>, sm);
    launch_pdl(scatter_kernel<V, true, false>, tiles, kScThreads, sm, s, keys, vals, n, w.ctl, w.start, sh.l1, sh.l2,
               w.cur1, k1, v1);
  }
  note_launch(4);
  if (sh.l2 == 0) return 1;
  opt_in_smem((const void *)scatter_kernel<V, false, true>, sm);
  launch_pdl(scatter_kernel<V, false, true>, tiles + (1u << sh.l1), kScThreads, sm, s, k1, v1, n, w.ctl, w.start,
             sh.l1, sh.l2, w.cur2, k2, v2);
  note_launch();
  return 2;
}

template int partition_pairs<int64_t>(const int64_t *, const int64_t *, int64_t, int64_t *, int64_t *, int64_t *,
                                      int64_t *, const Work &, int, cudaStream_t);
template int partition_pairs<int32_t>(const int64_t *, const int32_t *, int64_t, int64_t *, int32_t *, int64_t *,
                                      int32_t *, const Work &, int, cudaStream_t);

}  // namespace bsort
}  // namespace hm
