// Bucket join: point search for a pre-sorted batch that is large relative to
// the tree.
//
// After the query pre-sort (partition.cu) the queries of one bucket form a
// contiguous run and the bucket's keys lie in a contiguous range of leaves.
// Instead of one descent per query (search.cu), a CTA takes a run of one
// bucket, copies the bucket's leaf records (keys and values, 256 B per
// 16-key leaf) from HBM into shared memory in order, and answers every query of
// the run from there.  16-key leaves are staged by TMA and searched through
// 31-bit images of their first keys (join_tma_kernel); 64-key leaves, and
// batches of many queries per bucket, which first build a 64-slot directory of
// the bucket, by per-thread cp.async (join_kernel).  The leaf range of each
// bucket comes from one descent per bucket boundary (a separate kernel; kept per
// tree shape between calls).  Leaves are read once
// per run and sequentially, so the DRAM traffic of a batch with more queries than
// leaves falls from a random 160 B per query to the size of the touched leaf
// region.  A bucket whose leaves do not fit shared memory (very skewed keys)
// falls back to a scalar descent per query.  For batches up to 2^25 queries
// the results go straight to the queries' positions after the first pre-sort
// pass (recorded by the second), so only the first pass is undone.
//
// The per-query semantics are the reference's (child = number of separators
// <= key, open-harmonia/src/avx.cpp:2-54; equality in the leaf,
// open-harmonia/src/bpt.h:252-274): a key routed to leaf j lies between
// leaf j's first key and leaf j+1's first key, so the largest leaf of the
// range whose first key is <= q is the leaf the descent would reach.
#include "hm_internal.cuh"
#include "async_copy.cuh"
#include "warp_descent.cuh"

#include <cuda.h>  // CUtensorMap and its enums; the encoder is fetched through the runtime

#include <mutex>

#include <algorithm>

namespace hm {

namespace {

constexpr int kThreads = 256;
#ifndef HM_JOIN_PER_THREAD
#define HM_JOIN_PER_THREAD 1  // queries a thread answers per step (measured: 1 beats 2, 4 and 8)
#endif
constexpr int kPerThread = HM_JOIN_PER_THREAD;
constexpr int kRun = kThreads * kPerThread;  // queries a CTA answers per step
// Queries per work item of the cp.async join, at most: a bucket with more is
// cut into items (hot buckets of a skewed batch), each of which stages the
// bucket's leaves.  Small items keep the CTAs evenly loaded when a few keys
// draw many queries, large ones stage less: a sixteenth of an SM's share of the
// batch, between the two bounds (6 M Zipf queries on 64-key leaves: 218 us with
// items of 16384, 135 with 2560, 148 with 5120, 142 with 634).
constexpr int kItemMin = 1024, kItemMax = 16384;
static_assert(kItemMax < 65536, "an item's query count is kept in 16 bits");
#ifndef HM_JOIN_STAGES
#define HM_JOIN_STAGES 2  // shared-memory ring of the join kernel
#endif
#ifndef HM_JOIN_MINB
#define HM_JOIN_MINB 4  // resident join CTAs per SM the register budget allows
#endif
#ifndef HM_JOIN_SLACK
#define HM_JOIN_SLACK 4  // a stage holds mean + mean / HM_JOIN_SLACK + 8 leaves
#endif
constexpr int kStages = HM_JOIN_STAGES;
constexpr int kStageMax = (216 / kStages) * 1024;  // shared memory of one stage, at most

#ifndef HM_JOIN_MAX_BITS
#define HM_JOIN_MAX_BITS 16
#endif
static_assert(HM_JOIN_MAX_BITS <= 16, "a bucket number is kept in 16 bits");

// leafb[b], b in [0, nb] = leaf holding the smallest key of bucket b (bucket
// b's keys lie in leaves [leafb[b], leafb[b+1]]).  It depends only on the
// inner nodes, the key range and the bucket bits, so the launcher keeps it
// per tree shape and skips the descents while that holds.
// A chain of dependent loads per boundary bounds it: a warp takes 32
// neighbouring boundaries, which share most of their path, and ranks a node's
// keys over its lanes (2^14 boundaries over 2^21 leaves: 7 us; one thread
// each 15).
__global__ void bucket_bounds_kernel(DevTree t, int f, int64_t lo, int shift, int nb, int32_t *__restrict__ leafb) {
  pdl_enter();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if ((b & ~31) > nb) return;  // uniform in a warp
  const uint64_t off = (uint64_t)min(b, nb) << shift;
  // past the last boundary, and where it lies at or past Max_Key, no key is above it
  const bool past = b >= nb || off >= (uint64_t)kMaxKey - (uint64_t)lo;
  const int32_t leaf = descend_leaf_warp(t, f, past ? kMaxKey - 1 : (int64_t)((uint64_t)lo + off));
  if (b <= nb) leafb[b] = b == 0 ? 0 : past ? t.n_leaf - 1 : leaf;
}

// Words of one leaf in a stage: its keys at a stride of LC + 1 (leaf m's key s
// at m * (LC + 1) + s, so lanes reading different leaves fall in different
// banks), then, after all keys, its values densely (m * LC + s).
template <int LC>
__host__ __device__ constexpr int stage_leaf_bytes() {
  return (2 * LC + 1) * 8;
}

template <int LC>
struct Stage {
  int64_t *kp, *vp;
  __device__ Stage(int64_t *base, int ml) : kp(base), vp(base + ml * (LC + 1)) {}
  __device__ __forceinline__ int64_t first(int m) const { return kp[m * (LC + 1)]; }
  __device__ __forceinline__ int64_t key(int m, int c) const { return kp[m * (LC + 1) + c]; }
  __device__ __forceinline__ int64_t val(int m, int c) const { return vp[m * LC + c]; }
};

// Asynchronous copy of an item's leaf records into a stage (nothing when the
// leaves do not fit; such an item takes the scalar path).
template <int LC>
__device__ __forceinline__ void stage_leaves(const DevTree &t, const Item &it, Stage<LC> st, int ml) {
  constexpr int LI = LC >= 32 ? LC / 8 : 0;
  constexpr int ROW = LI + 2 * LC;
  constexpr int KS = LC + 1;
  if (it.nl() < 1 || it.nl() > ml) return;
  const longlong2 *src = reinterpret_cast<const longlong2 *>(t.leaf_rows + (int64_t)it.l0 * ROW);
  const int nvec = it.nl() * (ROW / 2);
  for (int v = threadIdx.x; v < nvec; v += kThreads) {
    const int m = v / (ROW / 2), w = 2 * (v - m * (ROW / 2));
    if (w < LI) continue;
    if (w < LI + LC) {
      cp_async_element(st.kp + m * KS + (w - LI), reinterpret_cast<const int64_t *>(src + v));
      cp_async_element(st.kp + m * KS + (w - LI) + 1, reinterpret_cast<const int64_t *>(src + v) + 1);
    } else {
      cp_async16(st.vp + m * LC + (w - LI - LC), src + v);
    }
  }
}

template <int LC, typename ST>
__device__ __forceinline__ int64_t lookup_staged(const ST &st, int nl, int span, int64_t q) {
  // leaf: the last of [1, nl) whose first key is <= q, else 0
  int m = 0;
  for (int step = span >> 1; step > 0; step >>= 1)
    if (m + step < nl && st.first(m + step) <= q) m += step;
  // slot: the last key <= q among the leaf's sorted keys (Max_Key pads the
  // tail), else slot 0
  int c = 0;
#pragma unroll
  for (int step = LC / 2; step > 0; step >>= 1)
    if (st.key(m, c + step) <= q) c += step;
  return st.key(m, c) == q ? st.val(m, c) : HM_NOT_FOUND;
}

// Directory of the staged leaves of one item (bucket b): slot j covers the
// keys [s_j, s_j+1) with s_j = bucket low + j << dshift, and dir[j] is the
// last leaf whose first key is <= s_j (0 if none), so a query of slot j lies
// in a leaf of [dir[j], dir[j+1]] (dir[D] = nl - 1).  Keys are compared in the
// biased unsigned order (k ^ sign bit), which is the signed order.
#ifndef HM_JOIN_DIR_BITS
#define HM_JOIN_DIR_BITS 6
#endif
constexpr int kDirBits = HM_JOIN_DIR_BITS;
constexpr int kDir = 1 << kDirBits;
#ifndef HM_JOIN_DIR_MIN
#define HM_JOIN_DIR_MIN 768  // mean queries per bucket from which the directory kernel runs
#endif

__host__ __device__ __forceinline__ uint64_t biased(int64_t k) { return (uint64_t)k ^ kSign; }

template <typename ST>
__device__ __forceinline__ void build_dir(const ST &st, int nl, int span, uint64_t lo_u, int dshift,
                                          int32_t *dir) {
  for (int j = threadIdx.x; j <= kDir; j += kThreads) {
    if (j == kDir) {
      dir[j] = nl - 1;
      continue;
    }
    uint64_t sj = lo_u + ((uint64_t)j << dshift);
    if (sj < lo_u) sj = ~0ull;  // past the top of the key space
    int m = 0;
    for (int step = span >> 1; step > 0; step >>= 1)
      if (m + step < nl && biased(st.first(m + step)) <= sj) m += step;
    dir[j] = m;
  }
}

template <int LC, typename ST>
__device__ __forceinline__ int64_t lookup_dir(const ST &st, int nl, const int32_t *dir, uint64_t lo_u, int dshift,
                                              int64_t q) {
  const uint64_t qu = biased(q);
  int m, hi;
  if (qu < lo_u) {  // below the bucket (bucket 0 only: not a loaded key)
    m = 0;
    hi = dir[0];
  } else {
    const uint64_t j = (qu - lo_u) >> dshift;
    const int jj = j < (uint64_t)kDir ? (int)j : kDir - 1;
    m = dir[jj];
    hi = dir[jj + 1];
  }
  while (m < hi && st.first(m + 1) <= q) m++;
  int c = 0;
#pragma unroll
  for (int step = LC / 2; step > 0; step >>= 1)
    if (st.key(m, c + step) <= q) c += step;
  (void)nl;
  return st.key(m, c) == q ? st.val(m, c) : HM_NOT_FOUND;
}

template <int LC>
__device__ __noinline__ int64_t lookup_scalar(const DevTree &t, int f, int64_t q) {
  constexpr int LI = LC >= 32 ? LC / 8 : 0;
  constexpr int ROW = LI + 2 * LC;
  const int32_t leaf = descend_leaf(t, f, q);
  const int64_t *kr = t.leaf_rows + (int64_t)leaf * ROW + LI;
  int64_t v = HM_NOT_FOUND;
#pragma unroll 4
  for (int s = 0; s < LC; s++)
    if (__ldg(kr + s) == q) v = __ldg(kr + LC + s);
  return v;
}

// Two of them at once, each level's loads of both under way together: a thread
// of the TMA join has two queries of an item of more than kJoinThreads, and one
// after the other they took twice as long (2^24 queries on 2^26 keys in groups
// of 4096, nearly all looked up this way: 2737 -> 2467 us).
template <int LC>
__device__ __noinline__ longlong2 lookup_scalar_pair(const DevTree &t, int f, int64_t qa, int64_t qb) {
  constexpr int LI = LC >= 32 ? LC / 8 : 0;
  constexpr int ROW = LI + 2 * LC;
  const int ix = f / 8, row = ix + f;
  int32_t na = 0, nb = 0;
  for (int l = 0; l < t.height; l++) {
    const int64_t *ra = t.inner + (int64_t)na * row, *rb = t.inner + (int64_t)nb * row;
    const int32_t fa = __ldg(t.prefix + na), fb = __ldg(t.prefix + nb);
    int ka = 0, kb = 0;
    for (int v = 0; v < ix / 2; v++) {
      const longlong2 a = __ldg(reinterpret_cast<const longlong2 *>(ra + 2 * v));
      const longlong2 b = __ldg(reinterpret_cast<const longlong2 *>(rb + 2 * v));
      ka += (a.x <= qa) + (a.y <= qa);
      kb += (b.x <= qb) + (b.y <= qb);
    }
    ka = 8 * min(ka, ix - 1);
    kb = 8 * min(kb, ix - 1);
    na = fa + ka;
    nb = fb + kb;
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const longlong2 a = __ldg(reinterpret_cast<const longlong2 *>(ra + ix + ka + 2 * v));
      const longlong2 b = __ldg(reinterpret_cast<const longlong2 *>(rb + ix + kb + 2 * v));
      na += (a.x <= qa) + (a.y <= qa);
      nb += (b.x <= qb) + (b.y <= qb);
    }
  }
  const int64_t *la = t.leaf_rows + (int64_t)(na - t.n_inner) * ROW + LI;
  const int64_t *lb = t.leaf_rows + (int64_t)(nb - t.n_inner) * ROW + LI;
  longlong2 r = make_longlong2(HM_NOT_FOUND, HM_NOT_FOUND);
#pragma unroll 4
  for (int s = 0; s < LC; s++) {
    if (__ldg(la + s) == qa) r.x = __ldg(la + LC + s);
    if (__ldg(lb + s) == qb) r.y = __ldg(lb + LC + s);
  }
  return r;
}

// Answers the queries of the current item kRun at a time (results to out in
// grouped order, or to out[place[i]]) while loading the next step's queries:
// this item's next run, else the first run of the next item.
template <int LC, bool DIR, bool PLACED, typename ST>
__device__ __forceinline__ void answer_item(const DevTree &t, int f, const ST &st, const Item &cur, const Item &next,
                                            bool staged, int span, uint64_t lo_u, int dshift, const int32_t *dir,
                                            const int64_t *__restrict__ qs, const int32_t *__restrict__ place,
                                            int64_t *__restrict__ out, int64_t (&q)[kPerThread],
                                            int32_t (&qo)[kPerThread]) {
  for (int r0 = 0; r0 < cur.len(); r0 += kRun) {
    // the next step's queries: this item's next run, else the next item's first
    const bool more = r0 + kRun < cur.len();
    const int32_t na = more ? cur.qa + r0 + kRun : next.qa;
    const int32_t nlen = more ? cur.len() - r0 - kRun : next.len();
    int64_t qn[kPerThread];
    int32_t on[kPerThread];
#pragma unroll
    for (int j = 0; j < kPerThread; j++) {
      const int r = j * kThreads + threadIdx.x;
      const bool in = r < nlen;
      qn[j] = in ? __ldg(qs + na + r) : 0;
      on[j] = PLACED ? (in ? __ldg(place + na + r) : 0) : na + r;
    }
#pragma unroll
    for (int j = 0; j < kPerThread; j++) {
      const int r = r0 + j * kThreads + threadIdx.x;
      if (r >= cur.len()) continue;
      int64_t v = HM_NOT_FOUND;
      if (q[j] != kMaxKey) {
        if (!staged)
          v = lookup_scalar<LC>(t, f, q[j]);
        else if (DIR)
          v = lookup_dir<LC>(st, cur.nl(), dir, lo_u, dshift, q[j]);
        else
          v = lookup_staged<LC>(st, cur.nl(), span, q[j]);
      }
      out[qo[j]] = v;  // grouped order: consecutive threads, consecutive slots
    }
#pragma unroll
    for (int j = 0; j < kPerThread; j++) {
      q[j] = qn[j];
      qo[j] = on[j];
    }
  }
}

// Persistent CTAs walk the items with a stride of the grid through a ring of
// kStages shared-memory stages: the leaves of the next kStages - 1 items are
// in flight (cp.async) while the current one is answered from shared memory,
// kRun queries per step.  Item descriptors are loaded kStages items ahead and
// the queries of the next step (of this item or the next) one step ahead.
// DIR: each staged item first builds its directory (batches with many queries
// per bucket); otherwise a query binary-searches the staged first keys.
// PLACED: grouped query i's result goes to out[place[i]] (its position before
// the last pre-sort pass, which the pass recorded), else to out[i].
template <int LC, bool DIR, bool PLACED>
__global__ void __launch_bounds__(kThreads, HM_JOIN_MINB) join_kernel(DevTree t, int f, const Item *__restrict__ items,
                                                        const int64_t *__restrict__ nitems,
                                                        const int64_t *__restrict__ qs,
                                                        const int32_t *__restrict__ place, int64_t *__restrict__ out,
                                                        int ml, uint64_t key_lo_u, int shift) {
  pdl_enter();
  static_assert(kStages >= 2, "a ring of at least two stages");
  extern __shared__ __align__(16) int64_t smem[];
  const int stage_words = ml * (2 * LC + 1);
  const int64_t n_items = *nitems;
  const int64_t g = gridDim.x;
  int64_t it = blockIdx.x;
  if (it >= n_items) return;
  const Item none{0, 0, 0, 0};
  __shared__ int32_t dir[DIR ? kDir + 1 : 1];
  const int dshift = shift > kDirBits ? shift - kDirBits : 0;
  Item d[kStages];  // items it, it + g, ..., it + (kStages - 1) g
#pragma unroll
  for (int x = 0; x < kStages; x++) d[x] = it + x * g < n_items ? items[it + x * g] : none;
#pragma unroll
  for (int x = 0; x < kStages - 1; x++) {
    stage_leaves<LC>(t, d[x], Stage<LC>(smem + x * stage_words, ml), ml);
    cp_async_commit();
  }
  int64_t q[kPerThread];
  int32_t qo[kPerThread];  // where each result goes
#pragma unroll
  for (int j = 0; j < kPerThread; j++) {
    const int r = j * kThreads + threadIdx.x;
    const bool in = r < d[0].len();
    q[j] = in ? __ldg(qs + d[0].qa + r) : 0;
    qo[j] = PLACED ? (in ? __ldg(place + d[0].qa + r) : 0) : d[0].qa + r;
  }
  int cur_stage = 0;
  for (; it < n_items; it += g) {
    const int fill = cur_stage == 0 ? kStages - 1 : cur_stage - 1;  // (cur + kStages - 1) % kStages
    stage_leaves<LC>(t, d[kStages - 1], Stage<LC>(smem + fill * stage_words, ml), ml);
    cp_async_commit();
    const Item dn = it + kStages * g < n_items ? items[it + kStages * g] : none;
    cp_async_wait_group<kStages - 1>();  // the current item's group is done
    __syncthreads();
    const Item cur = d[0];
    const Stage<LC> st(smem + cur_stage * stage_words, ml);
    const bool staged = cur.nl() >= 1 && cur.nl() <= ml;
    int span = 1;
    while (span < cur.nl()) span <<= 1;
    const uint64_t lo_u = key_lo_u + ((uint64_t)cur.b << shift);
    if (DIR && staged) {  // uniform across the CTA
      build_dir(st, cur.nl(), span, lo_u, dshift, dir);
      __syncthreads();
    }
    answer_item<LC, DIR, PLACED>(t, f, st, cur, d[1], staged, span, lo_u, dshift, dir, qs, place, out, q, qo);
    __syncthreads();  // this stage is refilled in the next iteration
#pragma unroll
    for (int x = 0; x < kStages - 1; x++) d[x] = d[x + 1];
    d[kStages - 1] = dn;
    cur_stage = cur_stage == kStages - 1 ? 0 : cur_stage + 1;
  }
  cp_async_wait_group<0>();
}

// The join for 16-key leaf records: a producer warp fills a ring of stages, the
// other warps look up.  An item's stage gets, all counted on its mbarrier, the
// leaf records by 2-D tiled TMA loads of 8 records at a time (one box for
// their keys, one for their values, 1 KiB each, 128-B swizzle: 16-B chunk j of
// row m lies at chunk j ^ (m mod 8); a box per producer lane), the item's first
// kJoinStep queries and their places by two bulk copies (from the 16-byte
// boundary below them), and its descriptor.  The last box may bring up to 7
// records past the item's range (the next bucket's leaves, or zeros past the
// last leaf), which are never searched.
//
// What an item costs is latency, so nothing of it is left to a load by the
// threads that wait for it, and the lookups are kept short: the leaf is found
// by a binary search over 31-bit images of the leaves' first keys (their offset
// from the bucket's lowest key, its top 31 bits; padded, so no step checks a
// bound), the slot by four probes of the leaf's keys whose swizzled address is
// one exclusive-or.  First keys with one image (dense groups of keys far apart)
// make the search end on a leaf past the key's, seen by its first key being
// above the key; whole first keys then decide, by a binary search too (2^24
// queries on 2^26 keys in groups of 256: 1838 us for the batch with a step back
// leaf by leaf, 1615 with the search, 1445 with the pairs of lookup_scalar_pair
// for the buckets that no stage holds).  Leaves and queries past the bucket take
// the last image, so that search settles them too: a replayed plan keeps the
// buckets of its capture, while write epochs may since have put larger keys into
// the last leaves.  An item has kJoinStep queries at most (a bucket of 256 and four
// standard deviations), so its lookups take one step.  A bucket of more, up to
// the 767 from which the directory is used, makes two or three items, each of
// which stages the bucket's leaves; such batches as a whole, against the
// former items of a whole bucket with one query a thread: 2^24 queries on 2^24
// keys 516 / 647 us, 2^25 on 2^26 keys 1058 / 1257.  An item takes one CTA
// barrier: past it every thread has left the item before, whose stage is then
// filled again.
// 2^24 queries on 2^26 keys (1.41 GB of records, queries, places and results):
// 237 us, 5.95 TB/s, 0.91 of the measured copy rate.  Before, with one thread
// issuing the loads between its lookups, 64-bit binary searches and one query
// a thread: 320 us; the producer warp took it to 288, two queries a thread and
// the fixed step count to 241 (one query a thread: 252), one step per item
// without a loop over steps to 237.
//
// Every wait is bounded: on a timeout the CTA records HM_ETIMEOUT in err, waits
// (bounded) for the loads it issued and returns.
constexpr int kJoinThreads = 160;            // that look up
constexpr int kJoinQueries = 2;              // of a thread at a time
constexpr int kJoinStep = kJoinThreads * kJoinQueries;
constexpr int kJoinCtas = 4;                 // resident on an SM
constexpr uint32_t kImageMax = 0x7fffffffu;  // of a key in the bucket
constexpr uint32_t kQueryBytes = (kJoinStep + 2) * 8, kPlaceBytes = (kJoinStep + 4) * 4;
constexpr uint32_t kItemBytes = (kQueryBytes + kPlaceBytes + 16 + 127) / 128 * 128;  // beside the records
static_assert(kQueryBytes % 16 == 0 && kPlaceBytes % 16 == 0, "bulk copies of whole 16-byte words");

__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ int64_t lds64(uint32_t a) {
  int64_t v;
  asm volatile("ld.shared.s64 %0, [%1];" : "=l"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ Item lds_item(uint32_t a) {
  Item i;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(i.qa), "=r"(i.l0), "=r"(i.b), "=r"(*reinterpret_cast<int *>(&i.len_nl))
               : "r"(a)
               : "memory");
  return i;
}
__device__ __forceinline__ void sts_item(uint32_t a, const Item &i) {
  asm volatile("st.shared.v4.s32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(i.qa), "r"(i.l0), "r"(i.b), "r"((int)i.len_nl)
               : "memory");
}

// Stages of the ring for a span of 2^steps leaves: three of up to 64 leaves or
// two of more, so that four CTAs share an SM.
__host__ __device__ constexpr int tma_stages(int steps) { return steps <= 6 ? 3 : 2; }

template <bool PLACED, int STEPS>
__global__ void __launch_bounds__(kJoinThreads + 32, kJoinCtas) join_tma_kernel(
    const __grid_constant__ CUtensorMap tmap, DevTree t, int f, const Item *__restrict__ items,
    const int64_t *__restrict__ nitems, const int64_t *__restrict__ qs, const int32_t *__restrict__ place,
    int64_t *__restrict__ out, int ml, uint64_t key_lo_u, int shift, unsigned *err) {
  constexpr int LC = 16, STAGES = tma_stages(STEPS);
  pdl_enter();
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ __align__(8) uint64_t bars[STAGES];
  const int n_items = (int)*nitems, g = (int)gridDim.x, tid = threadIdx.x, lane = tid & 31;
  int it = blockIdx.x;
  if (it >= n_items) return;
  const int rb = (ml + 7) & ~7;  // rows of a stage's key block (and value block)
  const uint32_t block = rb * 128;
  const uint32_t base = (smem_addr(dyn) + 1023u) & ~1023u;  // the swizzle's period; [stage][keys, values]
  const uint32_t rest = base + STAGES * 2 * block;      // [stage] queries, places, descriptor
  const uint32_t images = rest + STAGES * kItemBytes;   // [2][SPAN]
  constexpr int SPAN = 1 << STEPS;
  if (tid == 0) {
    for (int x = 0; x < STAGES; x++) mbar_init(&bars[x], 1);
    fence_mbar_init();
  }
  __syncthreads();
  const int ishift = max(0, shift - 31);
  const bool producer = tid >= kJoinThreads;
  // The producer warp: fills stage x with an item (past the last one only a
  // descriptor of no queries and the arrival).
  Item mine{0, 0, 0, 0};  // descriptor of this CTA's item number (fetched & ~31) + lane
  int fetched = 0;
  auto fill = [&](int x) {
    if ((fetched & 31) == 0) {
      const int64_t at = it + (int64_t)(fetched + lane) * g;
      mine = at < n_items ? items[at] : Item{0, 0, 0, 0};
    }
    Item itm;
    itm.qa = __shfl_sync(0xffffffffu, mine.qa, fetched & 31);
    itm.l0 = __shfl_sync(0xffffffffu, mine.l0, fetched & 31);
    itm.b = __shfl_sync(0xffffffffu, mine.b, fetched & 31);
    itm.len_nl = __shfl_sync(0xffffffffu, mine.len_nl, fetched & 31);
    fetched++;
    const int boxes = itm.nl() >= 1 && itm.nl() <= ml ? 2 * ((itm.nl() + 7) >> 3) : 0;
    const int len = itm.len();  // kJoinStep at most
    // whole 16-byte words around the queries and the places (both buffers end on 256 bytes)
    const uint32_t qb = len ? ((uint32_t)(len + (itm.qa & 1) + 1) & ~1u) * 8 : 0;
    const uint32_t pb = PLACED && len ? ((uint32_t)(len + (itm.qa & 3) + 3) & ~3u) * 4 : 0;
    const uint32_t r = rest + x * kItemBytes;
    fence_proxy_async_smem();  // the stage's earlier reads come before these writes
    if (lane == 0) {
      sts_item(r + kQueryBytes + kPlaceBytes, itm);
      mbar_expect_tx(&bars[x], (unsigned)boxes * 1024u + qb + pb);
      if (qb) bulk_g2s(r, qs + (itm.qa & ~1), qb, &bars[x]);
      if (pb) bulk_g2s(r + kQueryBytes, place + (itm.qa & ~3), pb, &bars[x]);
    }
    __syncwarp();
    for (int b = lane; b < boxes; b += 32)
      tma_load_2d(base + x * 2 * block + (b & 1) * block + (b >> 1) * 1024, &tmap, (b & 1) * 16, itm.l0 + 8 * (b >> 1),
                  &bars[x]);
  };
  if (producer)
    for (int x = 0; x < STAGES - 1; x++) fill(x);
  const int mine_n = (n_items - it + g - 1) / g;  // this CTA's items
  unsigned phase = 0;                             // bit x: parity of stage x's next phase
  for (int i = 0, st = 0; i < mine_n; i++, st = st == STAGES - 1 ? 0 : st + 1) {
    const bool ok = producer || mbar_wait_bounded(&bars[st], (phase >> st) & 1u, t.wait_polls);
    phase ^= 1u << st;
    const uint32_t kb = base + st * 2 * block, r = rest + st * kItemBytes, im = images + (i & 1) * SPAN * 4;
    Item cur{0, 0, 0, 0};
    int nl = 0;
    uint64_t lo_u = 0;
    bool staged = false;
    if (!producer && ok) {
      cur = lds_item(r + kQueryBytes + kPlaceBytes);
      nl = cur.nl();
      staged = nl >= 1 && nl <= ml;
      lo_u = key_lo_u + ((uint64_t)cur.b << shift);
      if (staged) {
        for (int m = tid; m < SPAN; m += kJoinThreads) {
          uint32_t v = ~0u;
          if (m < nl) {
            const uint64_t k = biased(lds64(kb + m * 128 + ((m & 7) << 4)));
            const uint64_t d = k <= lo_u ? 0 : (k - lo_u) >> ishift;
            v = (uint32_t)min(d, (uint64_t)kImageMax);
          }
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(im + m * 4), "r"(v) : "memory");
        }
      }
    }
    if (__syncthreads_or(!ok)) {  // a load that never landed: report, drain, stop
      if (tid == 0) {
        atomicOr(err, kErrTimeout);
        for (int x = 0; x < STAGES; x++)  // every stage has loads under way but the one before st
          if (x != (st == 0 ? STAGES - 1 : st - 1))
            mbar_wait_bounded(&bars[x], x == st ? ((phase >> x) & 1u) ^ 1u : (phase >> x) & 1u);
      }
      __syncthreads();
      return;
    }
    if (producer) {  // every thread has left the stage before
      fill(st == 0 ? STAGES - 1 : st - 1);
      continue;
    }
    const int len = cur.len();
    if (tid >= len) continue;
    int64_t q[kJoinQueries], v[kJoinQueries];
    int32_t qo[kJoinQueries];
#pragma unroll
    for (int j = 0; j < kJoinQueries; j++) {
      const int y = tid + j * kJoinThreads;
      q[j] = kMaxKey;
      qo[j] = -1;
      if (y < len) {
        qo[j] = cur.qa + y;
        q[j] = lds64(r + ((cur.qa & 1) + y) * 8);
        if constexpr (PLACED) qo[j] = (int32_t)lds32(r + kQueryBytes + ((cur.qa & 3) + y) * 4);
      }
    }
    if (staged) {
      uint32_t qi[kJoinQueries], m4[kJoinQueries];  // 4 * leaf: the last of [1, nl) whose image is <= the key's, else 0
#pragma unroll
      for (int j = 0; j < kJoinQueries; j++) {
        const uint64_t qu = biased(q[j]);
        const uint64_t d = qu <= lo_u ? 0 : (qu - lo_u) >> ishift;
        qi[j] = d > kImageMax ? kImageMax : (uint32_t)d;
        m4[j] = 0;
      }
#pragma unroll
      for (uint32_t step = 2 * SPAN; step >= 4; step >>= 1) {
#pragma unroll
        for (int j = 0; j < kJoinQueries; j++)
          if (lds32(im + m4[j] + step) <= qi[j]) m4[j] += step;
      }
      uint32_t row[kJoinQueries], x[kJoinQueries], c[kJoinQueries];  // c: 8 * slot
      int64_t key[kJoinQueries];
#pragma unroll
      for (int j = 0; j < kJoinQueries; j++) {
        row[j] = kb + (m4[j] << 5);
        x[j] = (m4[j] << 2) & 0x70u;
        c[j] = 0;
      }
      // the last key <= q of the leaf (Max_Key pads the tail), else slot 0
#pragma unroll
      for (uint32_t step = LC * 4; step >= 8; step >>= 1) {
#pragma unroll
        for (int j = 0; j < kJoinQueries; j++)
          if (lds64(row[j] + ((c[j] + step) ^ x[j])) <= q[j]) c[j] += step;
      }
#pragma unroll
      for (int j = 0; j < kJoinQueries; j++) key[j] = lds64(row[j] + (c[j] ^ x[j]));
#pragma unroll
      for (int j = 0; j < kJoinQueries; j++) {
        if (key[j] > q[j] && row[j] != kb) {
          // this leaf's image is the key's, but its first key lies above: the
          // last leaf before it whose first key does not, else the first
          const uint32_t end = m4[j] >> 2;
          uint32_t m = 0;
          for (uint32_t step = SPAN / 2; step > 0; step >>= 1)
            if (m + step < end && lds64(kb + (m + step) * 128 + (((m + step) & 7) << 4)) <= q[j]) m += step;
          row[j] = kb + m * 128;
          x[j] = (m & 7) << 4;
          c[j] = 0;
          for (uint32_t step = LC * 4; step >= 8; step >>= 1)
            if (lds64(row[j] + ((c[j] + step) ^ x[j])) <= q[j]) c[j] += step;
          key[j] = lds64(row[j] + (c[j] ^ x[j]));
        }
        v[j] = HM_NOT_FOUND;
        if (key[j] == q[j] && q[j] != kMaxKey) v[j] = lds64(row[j] + block + (c[j] ^ x[j]));
      }
    } else {
#pragma unroll
      for (int j = 0; j < kJoinQueries; j++) v[j] = HM_NOT_FOUND;
      if (len <= kJoinThreads) {
        if (q[0] != kMaxKey) v[0] = lookup_scalar<LC>(t, f, q[0]);
      } else {
        static_assert(kJoinQueries == 2, "a pair");
        const int64_t a = q[0] != kMaxKey ? q[0] : q[1], b = q[1] != kMaxKey ? q[1] : q[0];
        if (a != kMaxKey) {  // Max_Key is not looked up: the other key stands in for it
          const longlong2 r = lookup_scalar_pair<LC>(t, f, a, b);
          if (q[0] != kMaxKey) v[0] = r.x;
          if (q[1] != kMaxKey) v[1] = r.y;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kJoinQueries; j++)
      if (qo[j] >= 0) out[qo[j]] = v[j];
  }
  // the stages filled past the last item hold arrivals only
}

int64_t max_items(int64_t n, int nb, int item_max) { return n / item_max + nb + 1; }

int leaf_bytes(int lc) { return lc == 16 ? stage_leaf_bytes<16>() : stage_leaf_bytes<64>(); }

// Leaves one stage holds: room for the mean leaves per bucket, a quarter more
// and a margin, as an even count (keeps the value part 16-B aligned).  A
// bucket of more leaves takes the scalar path.
int stage_leaves_for(const hm_tree *t, int bits) {
  const int64_t mean = (t->n_leaf + ((int64_t)1 << bits) - 1) >> bits;
  int64_t ml = mean + mean / HM_JOIN_SLACK + 8;
  ml = std::min<int64_t>(ml, kStageMax / leaf_bytes(t->cfg.leaf_cap));
  return (int)(ml & ~int64_t(1));
}

}  // namespace

int join_bits(const hm_tree *t) {
  // HM_JOIN_MAX_BITS bits, or fewer while buckets still average at most 32 leaves
  // (64-key leaves: 16, with which more CTAs share an SM: 120 against 136 us for
  // 6 M Zipf queries; 8: 157)
  int b = 1;
  const int64_t most = t->cfg.leaf_cap == 16 ? 32 : 16;
  while (b < HM_JOIN_MAX_BITS && (t->n_leaf >> b) > most) b++;
  return b;
}

bool join_fits(const hm_tree *t) {
  if (t->cfg.leaf_cap != 16 && t->cfg.leaf_cap != 64) return false;
  const int bits = join_bits(t);
  const int64_t mean = (t->n_leaf + ((int64_t)1 << bits) - 1) >> bits;
  return mean + mean / HM_JOIN_SLACK + 8 <= stage_leaves_for(t, bits) + 1;
}

size_t join_scratch_bytes(int64_t n, int bits) {
  const int64_t nb = (int64_t)1 << bits;
  return (size_t)(align_up(4 * (nb + 1), 256) + 256 + align_up((int64_t)sizeof(Item) * max_items(n, (int)nb, std::min(kItemMin, kJoinStep)), 256)) +
         256;
}

namespace {

// Bucket geometry, as the partition computes it: bucket of k = (k - key_min) >> shift.
int bucket_shift(const hm_tree *t, int bits) {
  uint64_t range = (uint64_t)t->key_max - (uint64_t)t->key_min;
  int len = 0;
  while (len < 64 && (range >> len) != 0) len++;
  return len > bits ? len - bits : 0;
}

// The leaf of each bucket boundary (nb + 1 entries): kept per tree shape in
// the tree, else computed into leafb_scratch.
const int32_t *bucket_bounds(const hm_tree *t, int bits, int shift, int32_t *leafb_scratch, cudaStream_t s) {
  const int nb = 1 << bits;
  const unsigned gb = (unsigned)((nb + 1 + 255) / 256);
  int32_t *leafb = leafb_scratch;
  // kept per tree shape (not inside a graph capture, whose replays must
  // follow later changes of the tree)
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) {
    cudaGetLastError();
    cap = cudaStreamCaptureStatusActive;
  }
  bool want_leafb = true;
  bool fill_cache = false;
  // Held until the fill (if any) is enqueued and its event recorded: another
  // caller then finds the cache valid and waits on that event.  Once filled
  // the cache is only read, until a write to the tree changes its shape.
  std::unique_lock<std::mutex> cache_lock(t->mu, std::defer_lock);
  if (cap == cudaStreamCaptureStatusNone) {
    cache_lock.lock();
    const bool same = t->join_leafb_valid && t->join_leafb_gen == t->generation &&
                      t->join_leafb_shape == t->shape_version && t->join_leafb_lo == t->key_min &&
                      t->join_leafb_hi == t->key_max && t->join_leafb_nleaf == t->n_leaf && t->join_leafb_bits == bits;
    if (same) {
      leafb = t->join_leafb;
      want_leafb = false;
      cudaStreamWaitEvent(s, t->join_leafb_ready, 0);
    } else {
      t->join_leafb_valid = false;
      bool ok = true;
      if (t->join_leafb_cap < nb + 1) {
        if (t->join_leafb) cudaFree(t->join_leafb);
        t->join_leafb = nullptr;
        t->join_leafb_cap = 0;
        ok = cudaMalloc(&t->join_leafb, 4 * (size_t)(nb + 1)) == cudaSuccess;
        if (ok) t->join_leafb_cap = nb + 1;
      }
      if (ok && !t->join_leafb_ready)
        ok = cudaEventCreateWithFlags(&t->join_leafb_ready, cudaEventDisableTiming) == cudaSuccess;
      if (ok) {
        leafb = t->join_leafb;
        fill_cache = true;
      } else {
        cudaGetLastError();  // no cache: the boundaries are computed into scratch as in a capture
      }
    }
  }
  if (want_leafb) {
    launch_pdl(bucket_bounds_kernel, gb, 256, 0, s, t->view(), t->cfg.fanout, t->key_min, shift, nb, leafb);
    note_launch();
  }
  if (fill_cache && cudaEventRecord(t->join_leafb_ready, s) == cudaSuccess) {
    t->join_leafb_valid = true;
    t->join_leafb_gen = t->generation;
    t->join_leafb_shape = t->shape_version;
    t->join_leafb_lo = t->key_min;
    t->join_leafb_hi = t->key_max;
    t->join_leafb_nleaf = t->n_leaf;
    t->join_leafb_bits = bits;
  }
  return leafb;
}

using JoinKernel = void (*)(DevTree, int, const Item *, const int64_t *, const int64_t *, const int32_t *, int64_t *,
                            int, uint64_t, int);

template <bool PLACED>
JoinKernel pick_join(int lc, bool dir) {
  if (lc == 16) return dir ? join_kernel<16, true, PLACED> : join_kernel<16, false, PLACED>;
  if (lc == 64) return dir ? join_kernel<64, true, PLACED> : join_kernel<64, false, PLACED>;
  return nullptr;
}

#ifndef HM_JOIN_TMA
#define HM_JOIN_TMA 1  // 16-key leaves: stages filled by 2-D tiled TMA loads
#endif

using TmaJoinKernel = void (*)(const CUtensorMap, DevTree, int, const Item *, const int64_t *, const int64_t *,
                               const int32_t *, int64_t *, int, uint64_t, int, unsigned *);

// The TMA join does without a directory; batches that would use one (thousands
// of queries per bucket) take it only where measured (use_dir).
template <bool PLACED>
TmaJoinKernel pick_tma_join(int ml) {
  if (ml <= 32) return join_tma_kernel<PLACED, 5>;
  if (ml <= 64) return join_tma_kernel<PLACED, 6>;
  if (ml <= 128) return join_tma_kernel<PLACED, 7>;
  if (ml <= 256) return join_tma_kernel<PLACED, 8>;
  return join_tma_kernel<PLACED, 9>;
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up once per process (nullptr if
// the driver does not provide it: the join then stages with cp.async).
EncodeTiled encoder() {
  static EncodeTiled fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
    cudaGetLastError();
  });
  return fn;
}

// The leaf records of a 16-key tree as a 2-D tensor for TMA: n_leaf rows of
// 32 int64 (keys, then values; 256-B rows), boxes of 16 words x 8 rows
// (128-B inner extent, the 128-B swizzle's limit).
bool leaf_tensor_map(const hm_tree *t, CUtensorMap *m) {
  EncodeTiled enc = encoder();
  if (!enc || t->cfg.leaf_cap != 16 || t->leaf_index != 0 || t->n_leaf < 8) return false;  // a box's rows exist
  const cuuint64_t dim[2] = {32, (cuuint64_t)t->n_leaf};
  const cuuint64_t stride[1] = {32 * sizeof(int64_t)};
  const cuuint32_t box[2] = {16, 8};
  const cuuint32_t estride[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_INT64, 2, t->leaf_rows, dim, stride, box, estride,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Shared memory of the TMA join: alignment slack, per stage a key block and a
// value block of rb 128-B rows, the queries, places and descriptor, and the
// images of the first keys.
size_t tma_join_smem(int ml) {
  const size_t rb = (size_t)((ml + 7) & ~7);
  int steps = 5;
  while ((1 << steps) < ml) steps++;
  return 1024 + (size_t)tma_stages(steps) * (2 * rb * 128 + kItemBytes) + (2 << steps) * 4;
}

constexpr size_t kTmaSmem = 226 * 1024;  // of a CTA, at most

// Launch the join over the items (their count at nitems).
int run_tma_join(const hm_tree *t, TmaJoinKernel k, const CUtensorMap &tmap, int ml, int64_t n_items_max,
                 const Item *items, const int64_t *nitems, const int64_t *qs, const int32_t *place, int64_t *out,
                 int shift, cudaStream_t s) {
  const size_t smem = tma_join_smem(ml);
  const int per_sm = std::max(1, std::min(kJoinCtas, (int)((227 * 1024) / (smem + 1024))));
  const unsigned grid = (unsigned)std::min<int64_t>(n_items_max, (int64_t)t->num_sms * per_sm);
  int rc = opt_in_smem((const void *)k, (int)kTmaSmem);
  if (rc) return rc;
  // not a dependent launch: CTAs that start behind the pre-sort's find an SM's
  // shared memory carved out for those, and two of four fit (371 against 241 us)
  k<<<grid, kJoinThreads + 32, smem, s>>>(tmap, t->view(), t->cfg.fanout, items, nitems, qs, place, out, ml,
                                          biased(t->key_min), shift, t->d_err);
  note_launch();
  return HM_OK;
}

int run_join(const hm_tree *t, JoinKernel k, int ml, int64_t n_items_max, const Item *items, const int64_t *nitems,
             const int64_t *qs, const int32_t *place, int64_t *out, int shift, cudaStream_t s) {
  if (!k) return HM_EINVAL;
  const size_t smem = (size_t)kStages * ml * leaf_bytes(t->cfg.leaf_cap);
  const int per_sm = std::max(1, std::min(8, (int)((227 * 1024) / (smem + 1024))));
  const unsigned grid = (unsigned)std::min<int64_t>(n_items_max, (int64_t)t->num_sms * per_sm);
  int rc = opt_in_smem((const void *)k, kStages * kStageMax);
  if (rc) return rc;
  k<<<grid, kThreads, smem, s>>>(t->view(), t->cfg.fanout, items, nitems, qs, place, out, ml, biased(t->key_min),
                                 shift);  // as above
  note_launch();
  return HM_OK;
}

// measured: the directory pays from about three queries per thread and item
bool use_dir(int64_t n, int nb) { return HM_JOIN_DIR_BITS > 0 && n >= (int64_t)HM_JOIN_DIR_MIN * nb; }

// How the batch is joined: decided once, before its pre-sort.
struct JoinChoice {
  bool dir = false, tma = false;
  int ml = 0, item_max = 0;
  CUtensorMap tmap;
};

JoinChoice choose_join(const hm_tree *t, int bits, int64_t n) {
  JoinChoice c;
  c.dir = use_dir(n, 1 << bits);
  c.ml = stage_leaves_for(t, bits);
  c.tma = HM_JOIN_TMA && !c.dir && tma_join_smem(c.ml) <= kTmaSmem && leaf_tensor_map(t, &c.tmap);
  // the TMA join takes a step of queries per item: a fuller bucket's next step
  // is prefetched like any other item's
  const int64_t share = n / ((int64_t)t->num_sms * 16);
  c.item_max = c.tma ? kJoinStep : (int)std::min<int64_t>(kItemMax, std::max<int64_t>(kItemMin, share / kRun * kRun));
  return c;
}

JoinItems join_layout(int bits, void *scratch, int32_t **leafb_scratch) {
  char *p = static_cast<char *>(scratch);
  *leafb_scratch = reinterpret_cast<int32_t *>(p);
  p += align_up(4 * ((1 << bits) + 1), 256);
  JoinItems ji;
  ji.n_items = reinterpret_cast<int64_t *>(p);
  ji.items = reinterpret_cast<Item *>(p + 256);
  return ji;
}

}  // namespace

int prepare_join(const hm_tree *t, int bits, int64_t n, void *scratch, cudaStream_t s, JoinItems *ji) {
  int32_t *leafb_scratch = nullptr;
  *ji = join_layout(bits, scratch, &leafb_scratch);
  ji->leafb = bucket_bounds(t, bits, bucket_shift(t, bits), leafb_scratch, s);
  ji->item_max = (uint32_t)choose_join(t, bits, n).item_max;
  return cuda_err(cudaGetLastError());
}

int launch_join(const hm_tree *t, const int64_t *qs, int bits, int64_t n, int64_t *out, const JoinItems &ji,
                cudaStream_t s, const int32_t *place) {
  if (n <= 0) return HM_OK;
  const JoinChoice c = choose_join(t, bits, n);
  const int shift = bucket_shift(t, bits);
  const int64_t most = max_items(n, 1 << bits, c.item_max);
  int rc;
  if (c.tma) {
    rc = run_tma_join(t, place ? pick_tma_join<true>(c.ml) : pick_tma_join<false>(c.ml), c.tmap, c.ml, most, ji.items,
                      ji.n_items, qs, place, out, shift, s);
  } else {
    const JoinKernel k = place ? pick_join<true>(t->cfg.leaf_cap, c.dir) : pick_join<false>(t->cfg.leaf_cap, c.dir);
    rc = run_join(t, k, c.ml, most, ji.items, ji.n_items, qs, place, out, shift, s);
  }
  return rc ? rc : cuda_err(cudaGetLastError());
}

}  // namespace hm
