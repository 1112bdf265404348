// Query pre-sort (the reference's PSA, "partially sorted aggregation"):
// group a batch of queries by the top `bits` bits of their key, relative to
// the tree's key range, cut the buckets into work items for the join, and
// afterwards move per-query results from the grouped order back to the caller's order.
//
// The reference runs cub::DeviceRadixSort::SortPairs on bits [48,64) of
// (key, pos) before every search launch
// (open-harmonia/src/full-multi-prefix-sort-8thread.cu:305-309,
// open-harmonia/regular_bpt/prefix-sort.cu:288-293) and scatters results back
// through the permutation on the host.  Here:
//   * the bucket is taken relative to [key_min, key_max] of the tree so every
//     bucket holds loaded keys (fixed bits [48,64) leave half of them empty for
//     non-negative keys);
//   * one kernel counts all 2^bits buckets at once (16-bit counters in shared
//     memory) and one scans them, which gives the bucket starts and the cursors
//     of every pass;
//   * order inside a bucket does not matter, so a tile of a pass reserves its
//     run of every digit with one atomic on the digit's cursor: no per-tile
//     counts, no scan of them, nothing between the passes;
//   * up to 8 bits take one pass; more take two, most significant first: the
//     second pass partitions every first-pass bucket on its own, in tiles that
//     never straddle a bucket;
//   * each pass stages a tile in shared memory grouped by digit (12 B per query:
//     key, digit and position) and writes it out so consecutive threads store
//     consecutive slots;
//   * the payload is either a position (int32: in the input, or after the first
//     pass) or the query's offset inside its tile (uint16).  With offsets, the
//     pass also records where each digit run of a tile went, and its inverse
//     reads the tile's runs (each contiguous), places every result at its offset
//     in shared memory and writes the tile out in order, so no pass writes single
//     8-byte values at random addresses.
#include "async_copy.cuh"
#include "hm_internal.cuh"

#include <algorithm>

namespace hm {

namespace {

// A pass with an inverse works on tiles of kTile queries (offsets fit 16 bits;
// the inverse wants long runs: 78 us at 2^24 queries with 8192-query tiles, 124
// with 4096, 141 with 2048, against a pass of 89, 86 and 103 us), the second
// pass of a placed partition, which has none, on kSmallTile (4096 queries in
// 512 threads 106 us, 2048 in 256 threads 113).
constexpr int kTileThreads = 512, kTilePer = 16, kTileCtas = 2;
constexpr int kTile = kTileThreads * kTilePer;
constexpr int kSmallThreads = 512, kSmallPer = 8, kSmallCtas = 3;
constexpr int kSmallTile = kSmallThreads * kSmallPer;
static_assert(kTile < 65536 && kTileThreads >= 256 && kSmallThreads >= 256, "16-bit offsets; a thread per digit");

// Bucket of a key: top `bits` bits of (k - lo) over the tree's key range.  The
// join finds a bucket's leaves from the same boundaries, so a key above the
// range stays in the bucket of its offset while there is one: a replayed plan's
// range is that of its capture, and the tree may hold larger keys by then.
struct Bucket {
  int64_t lo;
  int shift;
  int maxd;
  __device__ __forceinline__ int operator()(int64_t k) const {
    if (k <= lo) return 0;
    const uint64_t d = ((uint64_t)k - (uint64_t)lo) >> shift;
    return d > (uint64_t)maxd ? maxd : (int)d;
  }
};

// A tile: elements [begin, begin + len) of the pass's input.
struct Tile {
  uint32_t begin, len;
};

// For a batch set, the first pass cuts each batch into its own tiles (a tile
// never straddles two batches).  Each tile carries its batch's pointers shifted
// by the batch's start: element i of the set is qbase[i] (queries), obase[i]
// (results).
struct TileIO {
  const int64_t *qbase;
  int64_t *obase;
};

// One CTA: the batch set's first-pass tiles; tiles past the last are empty.
__global__ void __launch_bounds__(1024) batch_tiles_kernel(BatchView bv, int max_tiles, Tile *__restrict__ tiles,
                                                           TileIO *__restrict__ tio) {
  pdl_enter();
  __shared__ int32_t pre[1024];
  const int tid = threadIdx.x, nb = bv.nb;
  const int per = (nb + 1023) / 1024;
  int32_t mine = 0;
  for (int x = 0; x < per; x++) {
    const int b = tid * per + x;
    if (b < nb) mine += (int32_t)((bv.qpre[b + 1] - bv.qpre[b] + kTile - 1) / kTile);
  }
  pre[tid] = mine;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {  // inclusive scan
    const int32_t v = tid >= o ? pre[tid - o] : 0;
    __syncthreads();
    pre[tid] += v;
    __syncthreads();
  }
  int32_t at = pre[tid] - mine;
  for (int x = 0; x < per; x++) {
    const int b = tid * per + x;
    if (b >= nb) break;
    const int64_t s = bv.qpre[b], e = bv.qpre[b + 1];
    const hm_batch bt = bv.batches[b];
    for (int64_t c0 = s; c0 < e; c0 += kTile, at++) {
      tiles[at] = Tile{(uint32_t)c0, (uint32_t)min((int64_t)kTile, e - c0)};
      tio[at] = TileIO{bt.q - s, bt.out - s};  // only indexed inside the batch
    }
  }
  for (int i = pre[1023] + tid; i < max_tiles; i += 1024) tiles[i] = Tile{0, 0};
}

constexpr int kCountThreads = 1024;
constexpr int kCountPer = 8;

// Queries per bucket, two 16-bit counters a word: a counter that reaches 2^15
// moves that much to the global count.  The barrier every second step bounds
// what a counter can receive before that happens (2^14), so none overflows.
template <bool BATCHED>
__global__ void __launch_bounds__(kCountThreads) psa_count_kernel(const int64_t *__restrict__ q,
                                                                  const Tile *__restrict__ tiles,
                                                                  const TileIO *__restrict__ tio, int max_tiles,
                                                                  int64_t n, uint32_t nb, Bucket bk,
                                                                  uint32_t *__restrict__ count) {
  pdl_enter();
  extern __shared__ __align__(16) uint32_t packed[];
  for (uint32_t i = threadIdx.x; i < (nb + 1) / 2; i += kCountThreads) packed[i] = 0;
  __syncthreads();
  constexpr int kStep = kCountThreads * kCountPer;
  static_assert(2 * kStep <= 1 << 14, "adds between barriers");
  int steps = 0;
  auto run = [&](const int64_t *src, int64_t i0, int64_t i1) {
    for (int64_t base = i0; base < i1; base += kStep) {  // uniform across the CTA
      int64_t k[kCountPer];
#pragma unroll
      for (int j = 0; j < kCountPer; j++) {
        const int64_t i = base + j * kCountThreads + threadIdx.x;
        k[j] = i < i1 ? __ldg(src + i) : 0;
      }
#pragma unroll
      for (int j = 0; j < kCountPer; j++) {
        if (base + j * kCountThreads + threadIdx.x < i1) {
          const uint32_t b = bk(k[j]), sh = (b & 1) * 16;
          if (((atomicAdd(&packed[b >> 1], 1u << sh) >> sh) & 0xffffu) == 0x7fffu) {
            atomicSub(&packed[b >> 1], 0x8000u << sh);
            atomicAdd(count + b, 0x8000u);
          }
        }
      }
      if ((++steps & 1) == 0) __syncthreads();
    }
  };
  if constexpr (BATCHED) {
    for (int t = blockIdx.x; t < max_tiles; t += gridDim.x) {
      const Tile c = tiles[t];
      if (c.len == 0) break;
      run(tio[t].qbase, c.begin, (int64_t)c.begin + c.len);
    }
  } else {
    for (int64_t base = (int64_t)blockIdx.x * kStep; base < n; base += (int64_t)gridDim.x * kStep)
      run(q, base, min(n, base + kStep));
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nb; i += kCountThreads) {
    const uint32_t c = (packed[i >> 1] >> ((i & 1) * 16)) & 0xffffu;
    if (c) atomicAdd(count + i, c);
  }
}

constexpr int kStartThreads = 1024;

// Bucket starts (nb + 1), the passes' cursors and the join's work items: CTA c
// owns buckets [1024 c, 1024 c + 1024) and adds up the counts and the items of
// those before them itself (at most 64 loads a thread from L2); its items are
// written a thread each, for a hot bucket has hundreds.  Launch latency and the
// reload of the counts bound it: 13.6 us for 2^14 buckets, against 5.9 and
// 10..17 us of two kernels.
__global__ void __launch_bounds__(kStartThreads) psa_starts_kernel(const uint32_t *__restrict__ count, uint32_t nb,
                                                                   int l2, uint32_t n, uint32_t *__restrict__ start,
                                                                   uint32_t *__restrict__ cur1,
                                                                   uint32_t *__restrict__ cur2, JoinItems ji) {
  pdl_enter();
  __shared__ uint32_t wsum[32], bsum[32], iwsum[32], ibsum[32];
  __shared__ uint32_t upto[kStartThreads], from[kStartThreads], len[kStartThreads];  // items up to, start, count
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t first = blockIdx.x * kStartThreads, im = ji.item_max;
  auto items_of = [&](uint32_t c) { return im ? (c + im - 1) / im : 0; };
  uint32_t before = 0, ibefore = 0;
#pragma unroll 4
  for (uint32_t i = tid; i < first; i += kStartThreads) {
    const uint32_t c = count[i];
    before += c;
    ibefore += items_of(c);
  }
  const uint32_t mine = first + tid < nb ? count[first + tid] : 0, imine = items_of(mine);
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    before += __shfl_xor_sync(0xffffffffu, before, o);
    ibefore += __shfl_xor_sync(0xffffffffu, ibefore, o);
  }
  uint32_t incl = mine, iincl = imine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o), z = __shfl_up_sync(0xffffffffu, iincl, o);
    if (lane >= o) {
      incl += y;
      iincl += z;
    }
  }
  if (lane == 31) {
    wsum[warp] = incl;
    iwsum[warp] = iincl;
  }
  if (lane == 0) {
    bsum[warp] = before;
    ibsum[warp] = ibefore;
  }
  __syncthreads();
  uint32_t at = incl - mine, iat = 0;
  for (int w = 0; w < 32; w++) {
    at += bsum[w];
    iat += ibsum[w];
  }
  for (int w = 0; w < warp; w++) {
    at += wsum[w];
    iincl += iwsum[w];
  }
  const uint32_t b = first + tid;
  if (b < nb) {
    start[b] = at;
    cur2[b] = at;
    if ((b & ((1u << l2) - 1)) == 0) cur1[b >> l2] = at;
    if (b == nb - 1) start[nb] = n;
  }
  if (im == 0) return;
  upto[tid] = iincl;
  from[tid] = at;
  len[tid] = mine;
  __syncthreads();
  const uint32_t total = upto[kStartThreads - 1];
  if (tid == 0 && first + kStartThreads >= nb) *ji.n_items = (int64_t)iat + total;
  for (uint32_t x = tid; x < total; x += kStartThreads) {
    uint32_t lo = 0;  // the bucket of item x: the first with upto > x
#pragma unroll
    for (uint32_t step = kStartThreads / 2; step > 0; step >>= 1)
      if (upto[lo + step - 1] <= x) lo += step;
    const uint32_t done = (x - (lo ? upto[lo - 1] : 0)) * im;
    const int32_t l0 = ji.leafb[first + lo], nl = ji.leafb[first + lo + 1] - l0 + 1;
    Item it;
    it.qa = (int32_t)(from[lo] + done);
    it.l0 = l0;
    it.b = (int32_t)(first + lo);
    it.len_nl = min(im, len[lo] - done) << 16 | (uint32_t)min(nl, 65535);  // a capped count is never staged
    ji.items[iat + x] = it;
  }
}

constexpr int stage_bytes(int tile) { return tile * 12; }

// One tile of a pass per CTA: rank every query inside its digit with
// shared-memory atomics, reserve the tile's runs (one cursor atomic per digit),
// scan the 256 tile counts, stage the tile grouped by digit as keys (8 B) plus
// an aux word (digit << 16 | position in the tile), then write it out so
// consecutive threads store consecutive slots of one digit run.
// SECOND: tiles are cut inside the first pass's buckets (from their starts);
// digit = the low l2 bits.  T: the payload, the offset inside the tile
// (uint16) or the position in the pass's input (int32).  runs / lens (may be
// null): where the tile's digit runs went, for the inverse; info: its tiles.
template <typename T, bool SECOND, bool BATCHED, int THREADS, int PER, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) psa_scatter_kernel(
    const int64_t *__restrict__ q, const Tile *__restrict__ tiles, const TileIO *__restrict__ tio, int64_t n,
    Bucket bk, const uint32_t *__restrict__ start, int l1, int l2, uint32_t *__restrict__ cur,
    int64_t *__restrict__ q_out, T *__restrict__ pay_out, uint32_t *__restrict__ runs, uint16_t *__restrict__ lens,
    Tile *__restrict__ info) {
  constexpr int TILE = THREADS * PER;
  pdl_enter();
  extern __shared__ __align__(16) unsigned char dyn[];
  int64_t *skey = reinterpret_cast<int64_t *>(dyn);
  uint32_t *saux = reinterpret_cast<uint32_t *>(dyn + 8 * TILE);
  __shared__ uint32_t cnt[256], tstart[256], adj[256];
  __shared__ uint32_t wsum[8];
  __shared__ uint32_t t_first, t_len, t_bucket;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t i0, len, bucket = 0;
  if (tid < 256) cnt[tid] = 0;
  if constexpr (SECOND) {
    // tiles of first-pass bucket tid, and the bucket this CTA's tile is in
    uint32_t s = 0, e = 0, nt = 0, incl = 0;
    if (tid < 256) {
      if (tid < 1 << l1) {
        s = start[(uint32_t)tid << l2];
        e = start[(uint32_t)(tid + 1) << l2];
        nt = (e - s + TILE - 1) / TILE;
      }
      incl = nt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) wsum[warp] = incl;
    }
    if (tid == 0) t_len = 0;
    __syncthreads();
    if (tid < 256) {
      for (int w = 0; w < warp; w++) incl += wsum[w];
      if (blockIdx.x < incl && blockIdx.x >= incl - nt) {
        t_first = s + (blockIdx.x - (incl - nt)) * TILE;
        t_len = min(e - t_first, (uint32_t)TILE);
        t_bucket = tid;
      }
    }
    __syncthreads();
    i0 = t_first;
    len = t_len;
    bucket = t_bucket << l2;
  } else if constexpr (BATCHED) {
    const Tile c = tiles[blockIdx.x];
    i0 = c.begin;
    len = c.len;
    __syncthreads();
  } else {
    i0 = blockIdx.x * (uint32_t)TILE;
    len = (uint32_t)min((int64_t)TILE, n - i0);
    __syncthreads();
  }
  if (info && !BATCHED && tid == 0) info[blockIdx.x] = Tile{len ? i0 : 0, len};
  if (len == 0) return;  // past the last tile
  const uint32_t sh = SECOND ? 0 : l2, mask = SECOND ? (1u << l2) - 1 : 0xffffu;
  const int64_t *src = (BATCHED ? tio[blockIdx.x].qbase : q) + i0;
  int64_t k[PER];
#pragma unroll
  for (int j = 0; j < PER; j++) k[j] = j * THREADS + tid < len ? __ldg(src + j * THREADS + tid) : 0;
  uint32_t dr[PER];  // digit << 16 | rank inside the tile's digit run
#pragma unroll
  for (int j = 0; j < PER; j++) {
    if (j * THREADS + tid < len) {
      const uint32_t d = ((uint32_t)bk(k[j]) >> sh) & mask;
      dr[j] = d << 16 | atomicAdd(&cnt[d], 1u);
    }
  }
  __syncthreads();
  uint32_t mine = 0, incl = 0, at = 0;
  if (tid < 256) {
    mine = cnt[tid];
    if (mine) at = atomicAdd(cur + bucket + tid, mine);
    incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
  }
  __syncthreads();
  if (tid < 256) {
    uint32_t before = incl - mine;
    for (int w = 0; w < warp; w++) before += wsum[w];
    tstart[tid] = before;
    adj[tid] = at - before;  // slot s of digit d goes to adj[d] + s (modulo 2^32)
    if (runs) {
      runs[blockIdx.x * 256u + tid] = at;
      lens[blockIdx.x * 256u + tid] = (uint16_t)mine;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < PER; j++) {
    if (j * THREADS + tid < len) {
      const uint32_t d = dr[j] >> 16, sl = tstart[d] + (dr[j] & 0xffffu);
      skey[sl] = k[j];
      saux[sl] = d << 16 | (uint32_t)(j * THREADS + tid);
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < PER; j++) {
    const uint32_t sl = j * THREADS + tid;
    if (sl < len) {
      const uint32_t a = saux[sl], o = adj[a >> 16] + sl, pos = a & 0xffffu;
      q_out[o] = skey[sl];
      pay_out[o] = (T)(sizeof(T) == 2 ? pos : i0 + pos);
    }
  }
}

// Inverse of one pass for 64-bit results, per tile.  The tile's elements sit in
// one contiguous run per digit; each carries its offset inside the tile.  The
// results are placed by offset in shared memory, then written to the tile's
// input range in order.  The runs are cut into units of kUnit elements (a
// skewed batch can put most of a tile in one run); warps take units
// round-robin, a lane per element so every load is one coalesced request,
// kRevBatch units at a time: the offsets are loaded first, then each result is
// copied from global memory straight to its slot with cp.async.  The tile is
// written out with 16-B stores when aligned.  Persistent CTAs take tiles
// blockIdx.x, blockIdx.x + gridDim.x, ...; the next tile's descriptor and run
// table are loaded into registers while the current one's copies are in flight.
constexpr int kRevThreads = 512, kRevCtas = 3;
constexpr int kRevWarps = kRevThreads / 32;
constexpr int kRevBatch = 2;  // units a warp reads at once
constexpr int kUnit = 64;     // elements of a unit (a multiple of 32)
constexpr int kUnitPer = kUnit / 32;

template <bool BATCHED>
__global__ void __launch_bounds__(kRevThreads, kRevCtas) psa_unpermute_kernel(
    const Tile *__restrict__ tiles, int max_tiles, const uint32_t *__restrict__ runs,
    const uint16_t *__restrict__ lens, const int64_t *__restrict__ res_in, const uint16_t *__restrict__ loc,
    int64_t *__restrict__ res_out, const TileIO *__restrict__ tio) {
  pdl_enter();
  extern __shared__ __align__(16) int64_t staged[];  // kTile results
  __shared__ uint32_t rs[256];
  __shared__ uint16_t rl[256];
  __shared__ int32_t up[257];
  __shared__ uint8_t unit_run[kTile / kUnit + 256];
  __shared__ int32_t wsum[8];
  int ci = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // this thread's run (digit tid) of the current tile, and the tile
  Tile c = ci < max_tiles ? tiles[ci] : Tile{0, 0};
  uint32_t ra = 0, rn = 0;
  int64_t *dst = BATCHED && c.len ? tio[ci].obase : res_out;
  if (tid < 256 && c.len) {
    ra = runs[ci * 256u + tid];
    rn = lens[ci * 256u + tid];
  }
  while (c.len) {
    const int len = (int)c.len;
    if (tid < 256) {  // runs and the exclusive scan of their units
      rs[tid] = ra;
      rl[tid] = (uint16_t)rn;
      const int32_t u = (int32_t)((rn + kUnit - 1) / kUnit);
      int32_t incl = u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) wsum[wid] = incl;
      up[tid + 1] = incl;
      if (tid == 0) up[0] = 0;
    }
    __syncthreads();
    if (tid < 256) {
      int32_t add = 0;
      for (int x = 0; x < wid; x++) add += wsum[x];
      const int32_t last = up[tid + 1] + add;
      up[tid + 1] = last;
      for (int u = last - (int32_t)((rn + kUnit - 1) / kUnit); u < last; u++) unit_run[u] = (uint8_t)tid;
    }
    __syncthreads();
    const int units = up[256];
    for (int u0 = wid; u0 < units; u0 += kRevWarps * kRevBatch) {
      uint16_t l[kRevBatch][kUnitPer];
      uint32_t a[kRevBatch];
      int cnt[kRevBatch];
#pragma unroll
      for (int x = 0; x < kRevBatch; x++) {
        const int u = u0 + x * kRevWarps;
        cnt[x] = 0;
        a[x] = 0;
        if (u < units) {
          const int d = unit_run[u];
          const int e0 = (u - up[d]) * kUnit;
          a[x] = rs[d] + e0;
          cnt[x] = min(kUnit, (int)rl[d] - e0);
#pragma unroll
          for (int h = 0; h < kUnitPer; h++)
            if (lane + 32 * h < cnt[x]) l[x][h] = __ldg(loc + a[x] + lane + 32 * h);
        }
      }
#pragma unroll
      for (int x = 0; x < kRevBatch; x++)
#pragma unroll
        for (int h = 0; h < kUnitPer; h++)
          if (lane + 32 * h < cnt[x]) cp_async_element(staged + l[x][h], res_in + a[x] + lane + 32 * h);
    }
    // the next tile's descriptor, run and output pointer, while the copies fly
    const int cn = ci + (int)gridDim.x;
    const Tile c_next = cn < max_tiles ? tiles[cn] : Tile{0, 0};
    uint32_t ra_n = 0, rn_n = 0;
    int64_t *dst_n = dst;
    if (c_next.len) {
      if (BATCHED) dst_n = tio[cn].obase;
      if (tid < 256) {
        ra_n = runs[cn * 256u + tid];
        rn_n = lens[cn * 256u + tid];
      }
    }
    cp_async_wait();
    __syncthreads();
    int64_t *o = dst + c.begin;
    if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) {
      const int pairs = len >> 1;
      const longlong2 *sv = reinterpret_cast<const longlong2 *>(staged);
      longlong2 *ov = reinterpret_cast<longlong2 *>(o);
      for (int x = tid; x < pairs; x += kRevThreads) ov[x] = sv[x];
      if ((len & 1) && tid == 0) o[len - 1] = staged[len - 1];
    } else {
      for (int x = tid; x < len; x += kRevThreads) o[x] = staged[x];
    }
    __syncthreads();  // staged, rs, rl, up and unit_run are refilled next
    ci = cn;
    c = c_next;
    ra = ra_n;
    rn = rn_n;
    dst = dst_n;
  }
}

Bucket make_bucket(const hm_tree *t, int bits) {
  Bucket d;
  d.lo = t->key_min;
  d.maxd = (1 << bits) - 1;
  uint64_t range = (uint64_t)t->key_max - (uint64_t)t->key_min;
  int len = 0;
  while (len < 64 && (range >> len) != 0) len++;
  d.shift = len > bits ? len - bits : 0;
  return d;
}

// Tiles of a pass over n queries in `parts` separate ranges, at most.
int64_t max_tiles(int64_t n, int parts, int tile) { return (n + tile - 1) / tile + (parts > 1 ? parts : 0); }

// What a pass leaves for its inverse.
struct Pass {
  Tile *tiles;
  uint32_t *runs;  // 256 per tile
  uint16_t *lens;
  int64_t mt;      // tiles, at most
};

struct Work {
  Pass p1, p2;
  uint32_t *count;  // 2^bits
  uint32_t *start;  // 2^bits + 1
  uint32_t *cur1, *cur2;
  int64_t *q_tmp;   // first-pass keys (two passes); the inverse's temporary
  void *pay1;       // first-pass payloads (two passes)
  uint16_t *loc;    // final offsets (offset mode)
  TileIO *tio;      // batch sets: the batches of each first-pass tile
};

size_t work_layout(int64_t n, int bits, bool offsets, Work *w, char *base, int batches = 1) {
  const bool two = bits > 8;
  const size_t pay = offsets ? 2 : 4, nb = (size_t)1 << bits;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += (size_t)align_up((int64_t)bytes, 256);
    return p;
  };
  auto pass = [&](Pass *p, int parts) {
    p->mt = max_tiles(n, parts, kTile);
    p->tiles = reinterpret_cast<Tile *>(take(sizeof(Tile) * p->mt));
    p->runs = reinterpret_cast<uint32_t *>(take(4 * 256 * p->mt));
    p->lens = reinterpret_cast<uint16_t *>(take(2 * 256 * p->mt));
  };
  Work x{};
  x.count = reinterpret_cast<uint32_t *>(take(4 * nb));
  x.start = reinterpret_cast<uint32_t *>(take(4 * (nb + 1)));
  x.cur1 = reinterpret_cast<uint32_t *>(take(4 * 256));
  x.cur2 = reinterpret_cast<uint32_t *>(take(4 * nb));
  if (offsets) {
    pass(&x.p1, batches);
    if (two) pass(&x.p2, 256);
  }
  x.q_tmp = two ? reinterpret_cast<int64_t *>(take(8 * n)) : nullptr;
  x.pay1 = two ? take(pay * n) : nullptr;
  x.loc = offsets ? reinterpret_cast<uint16_t *>(take(2 * n)) : nullptr;
  x.tio = batches > 1 || offsets ? reinterpret_cast<TileIO *>(take(sizeof(TileIO) * max_tiles(n, batches, kTile))) : nullptr;
  if (w) *w = x;
  return off;
}

// Counts, starts and (batch sets) the first pass's tiles.
void count_and_start(const Work &w, const Bucket &bk, const int64_t *q, int64_t n, int bits, int sms, cudaStream_t s,
                     const JoinItems *ji, const BatchView *bv) {
  const uint32_t nb = 1u << bits;
  cudaMemsetAsync(w.count, 0, 4 * (size_t)nb, s);
  const size_t smem = ((size_t)nb * 2 + 15) & ~(size_t)15;
  const int per_sm = smem > 100 * 1024 ? 1 : 2;
  const int64_t ctas = (n + kCountThreads * kCountPer - 1) / (kCountThreads * kCountPer);
  const unsigned grid = (unsigned)std::min<int64_t>(ctas, (int64_t)sms * per_sm);
  const Tile *tiles = w.p1.tiles;
  const TileIO *tio = w.tio;
  if (bv) {
    launch_pdl(batch_tiles_kernel, 1, 1024, 0, s, *bv, (int)w.p1.mt, w.p1.tiles, w.tio);
    opt_in_smem((const void *)psa_count_kernel<true>, 2 << 16);
    launch_pdl(psa_count_kernel<true>, grid, kCountThreads, smem, s, q, tiles, tio, (int)w.p1.mt, n, nb, bk, w.count);
  } else {
    opt_in_smem((const void *)psa_count_kernel<false>, 2 << 16);
    launch_pdl(psa_count_kernel<false>, grid, kCountThreads, smem, s, q, tiles, tio, 0, n, nb, bk, w.count);
  }
  const int l2 = bits > 8 ? bits - 8 : 0;
  launch_pdl(psa_starts_kernel, (nb + kStartThreads - 1) / kStartThreads, kStartThreads, 0, s,
             static_cast<const uint32_t *>(w.count), nb, l2, (uint32_t)n, w.start, w.cur1, w.cur2,
             ji ? *ji : JoinItems());
  note_launch(bv ? 3 : 2);
}

template <typename T, bool SECOND, bool BATCHED = false, int THREADS = kTileThreads, int PER = kTilePer,
          int CTAS = kTileCtas>
void one_pass(const Work &w, const Bucket &bk, const int64_t *q, int64_t n, int bits, uint32_t *cur, int64_t *q_out,
              T *pay_out, const Pass *inv, cudaStream_t s) {
  constexpr int TILE = THREADS * PER;
  const int l2 = bits > 8 ? bits - 8 : 0, l1 = bits - l2;
  const int64_t mt = BATCHED ? w.p1.mt : max_tiles(n, SECOND ? 256 : 1, TILE);
  auto k = psa_scatter_kernel<T, SECOND, BATCHED, THREADS, PER, CTAS>;
  opt_in_smem((const void *)k, stage_bytes(TILE));
  launch_pdl(k, (unsigned)mt, THREADS, stage_bytes(TILE), s, q, static_cast<const Tile *>(w.p1.tiles),
             static_cast<const TileIO *>(w.tio), n, bk, static_cast<const uint32_t *>(w.start), l1, l2, cur, q_out,
             pay_out, inv ? inv->runs : nullptr, inv ? inv->lens : nullptr, inv ? inv->tiles : nullptr);
  note_launch();
}

int device_sms() {
  static int sms[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!sms[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    sms[dev] = v;
  }
  return sms[dev];
}

template <bool BATCHED = false>
void unpermute_pass(const Pass &ps, const int64_t *res_in, const uint16_t *loc, int64_t *res_out, cudaStream_t s,
                    const TileIO *tio = nullptr) {
  auto k = psa_unpermute_kernel<BATCHED>;
  opt_in_smem((const void *)k, 8 * kTile);
  const unsigned grid = (unsigned)std::min<int64_t>(ps.mt, (int64_t)device_sms() * kRevCtas);
  launch_pdl(k, grid, kRevThreads, 8 * kTile, s, static_cast<const Tile *>(ps.tiles), (int)ps.mt,
             static_cast<const uint32_t *>(ps.runs), static_cast<const uint16_t *>(ps.lens), res_in, loc, res_out, tio);
  note_launch();
}

// The first pass in offset mode, or the only one (bits <= 8).
void first_pass(const Work &w, const Bucket &bk, const int64_t *q, int64_t n, int bits, int64_t *q_out, uint16_t *loc,
                cudaStream_t s, const BatchView *bv) {
  if (bv)
    one_pass<uint16_t, false, true>(w, bk, q, n, bits, w.cur1, q_out, loc, &w.p1, s);
  else
    one_pass<uint16_t, false>(w, bk, q, n, bits, w.cur1, q_out, loc, &w.p1, s);
}

}  // namespace

size_t partition_scratch_bytes(int64_t n, int bits, bool offsets, int batches) {
  return work_layout(n, bits, offsets, nullptr, nullptr, batches) + 256;
}

int partition_queries(const hm_tree *t, const int64_t *q, int64_t n, int bits, int64_t *q_out, int32_t *pos_out,
                      void *scratch, cudaStream_t s, const JoinItems *ji, const BatchView *bv) {
  if (n == 0) return HM_OK;
  if (bits < 1 || bits > 16 || n > INT32_MAX || n < 0) return HM_EINVAL;
  const bool offsets = pos_out == nullptr;
  if (!offsets && (bv || bits > 8)) return HM_EINVAL;  // input positions: one pass
  Work w;
  work_layout(n, bits, offsets, &w, static_cast<char *>(scratch), bv ? bv->nb : 1);
  const Bucket bk = make_bucket(t, bits);
  count_and_start(w, bk, q, n, bits, t->num_sms, s, ji, bv);
  if (!offsets) {
    one_pass<int32_t, false, false, kSmallThreads, kSmallPer, kSmallCtas>(w, bk, q, n, bits, w.cur1, q_out, pos_out,
                                                                          nullptr, s);
  } else if (bits <= 8) {
    first_pass(w, bk, q, n, bits, q_out, w.loc, s, bv);
  } else {
    first_pass(w, bk, q, n, bits, w.q_tmp, static_cast<uint16_t *>(w.pay1), s, bv);
    one_pass<uint16_t, true>(w, bk, w.q_tmp, n, bits, w.cur2, q_out, w.loc, &w.p2, s);
  }
  return cuda_err(cudaGetLastError());
}

int partition_queries_placed(const hm_tree *t, const int64_t *q, int64_t n, int bits, int64_t *q_out,
                             int32_t *place, void *scratch, cudaStream_t s, const JoinItems *ji,
                             const BatchView *bv) {
  if (n == 0) return HM_OK;
  if (bits <= 8 || bits > 16 || n > INT32_MAX || n < 0 || !place) return HM_EINVAL;
  Work w;
  work_layout(n, bits, true, &w, static_cast<char *>(scratch), bv ? bv->nb : 1);
  const Bucket bk = make_bucket(t, bits);
  count_and_start(w, bk, q, n, bits, t->num_sms, s, ji, bv);
  first_pass(w, bk, q, n, bits, w.q_tmp, static_cast<uint16_t *>(w.pay1), s, bv);
  one_pass<int32_t, true, false, kSmallThreads, kSmallPer, kSmallCtas>(w, bk, w.q_tmp, n, bits, w.cur2, q_out, place,
                                                                       nullptr, s);
  return cuda_err(cudaGetLastError());
}

int unpermute_first_pass(int64_t n, int bits, const int64_t *res1, int64_t *out, void *scratch, cudaStream_t s,
                         const BatchView *bv) {
  if (n == 0) return HM_OK;
  if (bits <= 8 || bits > 16 || n > INT32_MAX || n < 0) return HM_EINVAL;
  Work w;
  work_layout(n, bits, true, &w, static_cast<char *>(scratch), bv ? bv->nb : 1);
  const uint16_t *loc1 = static_cast<const uint16_t *>(w.pay1);
  if (bv)
    unpermute_pass<true>(w.p1, res1, loc1, nullptr, s, w.tio);
  else
    unpermute_pass(w.p1, res1, loc1, out, s);
  return cuda_err(cudaGetLastError());
}

int unpermute_results(int64_t n, int bits, int64_t *res_sorted, int64_t *out, void *scratch, cudaStream_t s,
                      const BatchView *bv) {
  if (n == 0) return HM_OK;
  if (bits < 1 || bits > 16 || n > INT32_MAX || n < 0) return HM_EINVAL;
  Work w;
  work_layout(n, bits, true, &w, static_cast<char *>(scratch), bv ? bv->nb : 1);
  const int64_t *res1 = res_sorted;  // results in first-pass order
  const uint16_t *loc1 = w.loc;
  if (bits > 8) {
    unpermute_pass(w.p2, res_sorted, w.loc, w.q_tmp, s);
    res1 = w.q_tmp;
    loc1 = static_cast<const uint16_t *>(w.pay1);
  }
  if (bv)
    unpermute_pass<true>(w.p1, res1, loc1, nullptr, s, w.tio);
  else
    unpermute_pass(w.p1, res1, loc1, out, s);
  return cuda_err(cudaGetLastError());
}

}  // namespace hm
