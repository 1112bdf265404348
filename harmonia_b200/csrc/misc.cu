// Device-wide exclusive scan, export of the tree contents, and the range scan
// with prefix-sum output compaction.
//
// Range reference: range_prefix_sort_1thread_search_1_thread_scan_kernel
// (open-harmonia/src/range.cu:101-227) descends with the start key and copies
// up to Range_Size = 8 records into fixed per-query slots (no compaction),
// with the end key forced to Max_Key (open-harmonia/src/range.cu:349-355).
// Here a query asks for the first len[i] records with key >= start[i], or
// (inclusive form) every record with start[i] <= key <= end[i]; a locate pass
// descends and computes each query's count, an exclusive scan
// turns counts into offsets, and a copy pass (a warp takes up to four queries)
// writes the records contiguously: leaves are ordered, so the records of a query are the
// key-ordered run that starts at (leaf, slot) and continues in leaf+1, ...
#include "ntg.cuh"

#include <algorithm>
#include <type_traits>

namespace hm {

namespace {

constexpr int kThreads = 256;

int scan_ctas(int64_t n) {
  int64_t c = (n + 4095) / 4096;
  if (c > 148 * 4) c = 148 * 4;
  if (c < 1) c = 1;
  return (int)c;
}

constexpr int kScanPer = 8;                    // elements per thread per scan step
constexpr int kScanStep = kThreads * kScanPer;  // elements per CTA per scan step

template <typename T>
__global__ void __launch_bounds__(kThreads) seg_sum_kernel(const T *__restrict__ in, int64_t n,
                                                           int64_t seg, int64_t *__restrict__ part,
                                                           const unsigned long long *go) {
  pdl_enter();
  if (go && *go == 0) return;
  __shared__ int64_t red[kThreads / 32];
  int64_t b0 = (int64_t)blockIdx.x * seg, b1 = min(n, b0 + seg);
  int64_t s = 0;
  for (int64_t base = b0; base < b1; base += kScanStep) {
    T v[kScanPer];
#pragma unroll
    for (int j = 0; j < kScanPer; j++) {  // all loads first
      const int64_t i = base + j * kThreads + threadIdx.x;
      v[j] = i < b1 ? in[i] : (T)0;
    }
#pragma unroll
    for (int j = 0; j < kScanPer; j++) s += (int64_t)v[j];
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t t = 0;
    for (int w = 0; w < kThreads / 32; w++) t += red[w];
    part[blockIdx.x] = t;
  }
}

// Exclusive scan of each segment, offset by the sum of the segments before it
// (each CTA adds up those of the at most 592 segment sums itself); the sum of
// all goes to *total (may be null).  go != null: nothing unless *go != 0.  A step
// stages kScanStep elements in shared memory (coalesced), each thread scans
// kScanPer consecutive ones (index i at i + i / 8: one pad word per 8 keeps
// the threads' runs in different banks), one block scan of the thread sums.
// A few CTAs per SM wait for each step's loads, so the next step's are issued
// before the scan (counts of 5.6 M leaves: 42 -> 33 us).
template <typename T>
__global__ void __launch_bounds__(kThreads) seg_scan_kernel(const T *__restrict__ in, int64_t n,
                                                            int64_t seg, const int64_t *__restrict__ part,
                                                            int64_t *__restrict__ out, int nctas,
                                                            int64_t *total, const unsigned long long *go) {
  pdl_enter();
  if (go && *go == 0) return;
  __shared__ int64_t buf[kScanStep + kScanStep / 8];
  __shared__ int64_t wsum[kThreads / 32];
  __shared__ int64_t carry;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int64_t b0 = (int64_t)blockIdx.x * seg, b1 = min(n, b0 + seg);
  {
    int64_t before = 0;
    for (int i = tid; i < (int)blockIdx.x; i += kThreads) before += part[i];
    for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) wsum[warp] = before;
    __syncthreads();
    if (tid == 0) {
      int64_t c = 0;
      for (int w = 0; w < kThreads / 32; w++) c += wsum[w];
      carry = c;
    }
    __syncthreads();
  }
  T nxt[kScanPer];  // the next step's elements are on their way while a step is scanned
  auto load = [&](int64_t base) {
#pragma unroll
    for (int j = 0; j < kScanPer; j++) {
      const int64_t i = base + j * kThreads + tid;
      nxt[j] = i < b1 ? in[i] : (T)0;
    }
  };
  load(b0);
  for (int64_t base = b0; base < b1; base += kScanStep) {
#pragma unroll
    for (int j = 0; j < kScanPer; j++) {
      const int e = j * kThreads + tid;
      buf[e + (e >> 3)] = (int64_t)nxt[j];
    }
    load(base + kScanStep);
    __syncthreads();
    int64_t x[kScanPer], local = 0;
#pragma unroll
    for (int j = 0; j < kScanPer; j++) {
      x[j] = buf[tid * (kScanPer + 1) + j];
      local += x[j];
    }
    int64_t incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int64_t run = carry + incl - local;
    for (int w = 0; w < warp; w++) run += wsum[w];
#pragma unroll
    for (int j = 0; j < kScanPer; j++) {
      buf[tid * (kScanPer + 1) + j] = run;
      run += x[j];
    }
    __syncthreads();
    if (tid == kThreads - 1) carry = run;
#pragma unroll
    for (int j = 0; j < kScanPer; j++) {
      const int e = j * kThreads + tid;
      const int64_t i = base + e;
      if (i < b1) out[i] = buf[e + (e >> 3)];
    }
    __syncthreads();
  }
  if (total && blockIdx.x == nctas - 1 && tid == 0) *total = carry;
}

__global__ void export_kernel(DevTree t, int lc, int li, int64_t *__restrict__ keys,
                              int64_t *__restrict__ vals) {
  const int64_t total = (int64_t)t.n_leaf * lc;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < total;
       x += (int64_t)gridDim.x * blockDim.x) {
    int64_t j = x / lc;
    int s = (int)(x - j * lc);
    if (s < t.leaf_cnt[j]) {
      int64_t o = t.leaf_base[j] + s;
      const int64_t *r = t.leaf_rows + j * (li + 2 * lc) + li;
      keys[o] = r[s];
      vals[o] = r[lc + s];
    }
  }
}

// Four lanes per key: descend, count the leaf's keys below the start key
// (global rank g through leaf_base).  Length form: count = min(len, keys from
// g to the end).  Inclusive form: the neighbouring group does the same with
// the end key and counts the keys <= it (the leaves before the end key's leaf
// hold only smaller keys, the ones after only larger, because separators fence
// the leaves), count = that rank - g, and nothing when end < start
// (BPlusTree::range_search, open-harmonia/src/bpt.cpp:695-769).  The end key
// Max_Key reaches the end of the key space.  1 M ranges on 2^26 keys: 171 us
// with one thread per range, 84 with four lanes, which read a node's words in
// one request.
template <int F, int LC, bool BETWEEN>
__global__ void __launch_bounds__(kThreads, 6) range_locate_kernel(
    DevTree t, const int64_t *__restrict__ start, const int32_t *__restrict__ len, const int64_t *__restrict__ end,
    int64_t n, int32_t *__restrict__ first_leaf, int32_t *__restrict__ first_slot, int64_t *__restrict__ count,
    unsigned *err) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int W = 4, G = kThreads / W, PER = BETWEEN ? G / 2 : G;  // ranges of a CTA step
  constexpr int LI = LC >= 32 ? LC / 8 : 0, LROW = LI + 2 * LC;
  if (!stage_top<F>(t, smem, err)) return;
  const int64_t *srows = reinterpret_cast<const int64_t *>(smem);
  const int32_t *spref = top_prefix<F>(t, smem);
  const uint64_t pol_inner = t.cache_hints == 1 ? policy_evict_last() : policy_evict_normal();
  const uint64_t pol_leaf = policy_evict_normal();
  const int sub = threadIdx.x % W, gid = threadIdx.x / W;
  const bool upper = BETWEEN && (gid & 1);
  for (int64_t base = (int64_t)blockIdx.x * PER; base < n; base += (int64_t)gridDim.x * PER) {
    const int64_t at = base + (BETWEEN ? gid / 2 : gid), i = min(at, n - 1);
    const int64_t key = __ldg((upper ? end : start) + i);
    const int64_t nav = key == kMaxKey ? kMaxKey - 1 : key;  // never rank the sentinel
    const int32_t leaf = descend_group<W, F>(t, srows, spref, nav, sub, pol_inner);
    // keys < start, or <= end (start: <= start - 1; nothing lies below the lowest key)
    const int64_t q = upper ? nav : nav - 1;
    const int64_t *row = t.leaf_rows + (int64_t)leaf * LROW;
    const int64_t lb = __ldg(t.leaf_base + leaf);
    int c;
    if constexpr (LI == 0) {
      c = count_le<W, LC, false>(row, q, sub, pol_leaf);
    } else {
      const int k = min(count_le<W, LI, false>(row, q, sub, pol_leaf), LI - 1);
      c = 8 * k + count_le<W, 8, false>(row + LI + 8 * k, q, sub, pol_leaf);
    }
    if (!upper && key == INT64_MIN) c = 0;  // start - 1 would wrap
    const int64_t g = lb + c;
    int64_t cnt;
    if constexpr (BETWEEN) {
      const int64_t ge_raw = __shfl_down_sync(0xffffffffu, key == kMaxKey ? t.n_keys : g, W);
      const int64_t e = __shfl_down_sync(0xffffffffu, key, W);
      cnt = e >= key && ge_raw > g ? ge_raw - g : 0;
    } else {
      const int64_t want = __ldg(len + i), rem = t.n_keys - g;
      cnt = want <= 0 ? 0 : want < rem ? want : rem;
    }
    if (key == kMaxKey || t.n_keys == 0) cnt = 0;
    if (sub == 0 && !upper && at < n) {
      first_leaf[i] = cnt > 0 ? leaf : 0;
      first_slot[i] = cnt > 0 ? c : 0;
      count[i] = cnt;
    }
  }
}

// The records of a query are the global ranks [g0, g0 + count) in key order
// (g0 = leaf_base[first leaf] + first slot).  A warp takes `per` neighbouring
// queries, their headers one per lane, in chunks of the records of at most
// kChunk / LC leaves.  The chunk's leaf_base entries say where each leaf's
// records go, so nothing is searched: a half-warp takes 16 slots of a leaf at a
// time and copies them asynchronously, a lane per slot, to their places in
// the warp's shared memory, where the output is put together; the next chunk's
// copies are in flight (its leaf_base entries before that) while this one is
// written out in 16-byte stores.  134 M records of 1 M queries on 2^26 keys:
// 840 us, 5.1 TB/s of records read and written (0.78 of the measured copy
// rate); 964 at best through registers, 1309 with a search for every record's
// leaf.  Chunks of 256 records: 855.  Taking the queries by key neighbourhood
// halves the reads from DRAM but not the time (875).  Nothing is written if
// the records do not fit in cap.
constexpr int kChunk = 128;       // records of a chunk, at most
constexpr int kBuf = kChunk + 4;  // words of one buffer (a word more for an odd start), whole 32-B sectors
constexpr int kCopyWarps = 8;

template <int LC>
__global__ void __launch_bounds__(kCopyWarps * 32) range_copy_kernel(
    DevTree t, const int32_t *__restrict__ first_leaf, const int32_t *__restrict__ first_slot,
    const int64_t *__restrict__ offsets, int64_t n, int per, int64_t cap,
    int64_t *__restrict__ okeys, int64_t *__restrict__ ovals) {
  pdl_enter();
  constexpr int LI = LC >= 32 ? LC / 8 : 0, ROW = LI + 2 * LC;
  constexpr int PIECES = LC / 16;     // 16-slot pieces of a leaf
  constexpr int LEAVES = kChunk / LC;  // leaves of a chunk
  extern __shared__ __align__(16) int64_t bufs[];
  if (offsets[n] > cap) return;
  const int lane = threadIdx.x & 31, half = lane >> 4, hl = lane & 15;
  int64_t *const buf = bufs + (threadIdx.x >> 5) * 4 * kBuf;  // [stage][keys, values]
  const int64_t i0 = (blockIdx.x * (int64_t)kCopyWarps + (threadIdx.x >> 5)) * per;
  const int m = (int)min((int64_t)per, n - i0);  // this warp's queries
  if (m <= 0) return;
  const int64_t mine = i0 + min(lane, m - 1);
  const int64_t h_off = offsets[mine];
  const int64_t h_rem = lane < m ? offsets[mine + 1] - h_off : 0;
  const int32_t h_leaf = first_leaf[mine], h_slot = first_slot[mine];
  auto base_of = [&](int32_t L) { return L < t.n_leaf ? __ldg(t.leaf_base + L) : t.n_keys; };
  const uint32_t some = __ballot_sync(0xffffffffu, h_rem > 0);  // queries with records
  if (some == 0) return;
  // the chunk to fetch next: query r, its leaves from L, whose first record is
  // the query's record x0; lb = their leaf_base entries, one per lane
  int r = __ffs(some) - 1;
  int32_t L = __shfl_sync(0xffffffffu, h_leaf, r);
  int64_t x0 = -__shfl_sync(0xffffffffu, h_slot, r);
  int64_t lb = base_of(L + min(lane, LEAVES));
  // Starts the copies of that chunk into stage st and moves on to the one
  // after it; *to = where its records go in the output, returns their number.
  auto fetch = [&](int st, int64_t *to) -> int {
    const int64_t off = __shfl_sync(0xffffffffu, h_off, r), rem = __shfl_sync(0xffffffffu, h_rem, r);
    const int32_t rb = (int32_t)(lb - __shfl_sync(0xffffffffu, lb, 0));  // the chunk's records before this leaf
    const int32_t wn = __shfl_sync(0xffffffffu, rb, LEAVES);
    const int32_t re = __shfl_down_sync(0xffffffffu, rb, 1);
    const int64_t left = rem - x0;  // records wanted from the chunk's first one on
    const int32_t lim = left < wn ? (int32_t)left : wn;
    const int32_t skip = x0 < 0 ? (int32_t)-x0 : 0;
    const int pieces = __popc(__ballot_sync(0xffffffffu, lane < LEAVES && rb < lim)) * PIECES;
    const int64_t *rows = t.leaf_rows + (int64_t)L * ROW + LI;
    *to = off + x0 + skip;
    // the next chunk and its leaf_base entries
    x0 += wn;
    L += LEAVES;
    if (x0 >= rem || wn <= 0) {
      const uint32_t rest = r == 31 ? 0 : some & (0xffffffffu << (r + 1));
      r = rest ? __ffs(rest) - 1 : 32;
      L = __shfl_sync(0xffffffffu, h_leaf, r & 31);
      x0 = -__shfl_sync(0xffffffffu, h_slot, r & 31);
    }
    if (r < 32) lb = base_of(L + min(lane, LEAVES));
    int64_t *kb = buf + st * 2 * kBuf + (((uintptr_t)(okeys + *to) >> 3) & 1) - skip;
    int64_t *vb = buf + st * 2 * kBuf + kBuf + (((uintptr_t)(ovals + *to) >> 3) & 1) - skip;
#pragma unroll 4
    for (int p0 = 0; p0 < pieces; p0 += 2) {
      const int p = p0 + half, j = min(p / PIECES, LEAVES - 1), s = (p % PIECES) * 16 + hl;
      const int32_t jb = __shfl_sync(0xffffffffu, rb, j), je = __shfl_sync(0xffffffffu, re, j);
      const int32_t x = jb + s;
      if (x < je && x >= skip && x < lim && p < pieces) {
        const int64_t *src = rows + j * ROW + s;
        cp_async_element(kb + x, src);
        cp_async_element(vb + x, src + LC);
      }
    }
    cp_async_commit();
    return max(lim - skip, 0);
  };
  // Writes c words at src (16-B aligned like dst - odd) to dst.
  auto write = [&](const int64_t *src, int64_t *dst, int c) {
    const int odd = ((uintptr_t)dst >> 3) & 1;
    dst -= odd;
    for (int e = 2 * lane; e < c + odd; e += 64) {
      const longlong2 w = *reinterpret_cast<const longlong2 *>(src + e);
      if (e >= odd && e + 1 < c + odd) {
        __stcs(reinterpret_cast<longlong2 *>(dst + e), w);
      } else {
        if (e >= odd) __stcs(dst + e, w.x);
        if (e + 1 < c + odd) __stcs(dst + e + 1, w.y);
      }
    }
  };
  int64_t to = 0;
  int c = fetch(0, &to), st = 0;
  for (;;) {
    const bool more = r < 32;
    int64_t to_n = 0;
    int c_n = 0;
    if (more) {
      c_n = fetch(st ^ 1, &to_n);
      cp_async_wait_group<1>();
    } else {
      cp_async_wait_group<0>();
    }
    __syncwarp();
    write(buf + st * 2 * kBuf, okeys + to, c);
    write(buf + st * 2 * kBuf + kBuf, ovals + to, c);
    __syncwarp();  // the stage is filled again next
    if (!more) break;
    st ^= 1;
    c = c_n;
    to = to_n;
  }
}

unsigned grid_for_items(int64_t items, unsigned cap) {
  int64_t b = (items + kThreads - 1) / kThreads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (unsigned)b;
}

}  // namespace

size_t scan_scratch_bytes(int64_t n) { return sizeof(int64_t) * (scan_ctas(n) + 8); }

template <typename T>
void exclusive_scan(const T *in, int64_t *out, int64_t n, void *scratch, cudaStream_t s) {
  const int nctas = scan_ctas(n);
  const int64_t seg = (n + nctas - 1) / nctas;
  int64_t *part = static_cast<int64_t *>(scratch);
  if (n == 0) {
    cudaMemsetAsync(out, 0, sizeof(int64_t), s);
    return;
  }
  const unsigned long long *go = nullptr;
  launch_pdl(seg_sum_kernel<T>, nctas, kThreads, 0, s, in, n, seg, part, go);
  launch_pdl(seg_scan_kernel<T>, nctas, kThreads, 0, s, in, n, seg, part, out, nctas, out + n, go);
  note_launch(2);
}


void exclusive_scan_i64(const int64_t *in, int64_t *out, int64_t n, void *scratch, cudaStream_t s) {
  exclusive_scan<int64_t>(in, out, n, scratch, s);
}

void exclusive_scan_i32(const int32_t *in, int64_t *out, int64_t n, void *scratch, cudaStream_t s) {
  exclusive_scan<int32_t>(in, out, n, scratch, s);
}

void rescan_leaf_base(const hm_tree *t, const unsigned long long *go, void *scratch, cudaStream_t s) {
  const int nctas = scan_ctas(t->n_leaf);
  const int64_t seg = (t->n_leaf + nctas - 1) / nctas;
  int64_t *part = static_cast<int64_t *>(scratch), *total = nullptr;
  launch_pdl(seg_sum_kernel<int32_t>, nctas, kThreads, 0, s, t->leaf_cnt, t->n_leaf, seg, part, go);
  launch_pdl(seg_scan_kernel<int32_t>, nctas, kThreads, 0, s, t->leaf_cnt, t->n_leaf, seg, part, t->leaf_base, nctas,
             total, go);
  note_launch(2);
}

void export_contents(const hm_tree *t, int64_t *d_keys, int64_t *d_vals, cudaStream_t s) {
  if (t->n_keys == 0) return;
  export_kernel<<<grid_for_items(t->n_leaf * t->cfg.leaf_cap, 148u * 32), kThreads, 0, s>>>(
      t->view(), t->cfg.leaf_cap, t->leaf_index, d_keys, d_vals);
  note_launch();
}

int range_locate(const hm_tree *t, const int64_t *start, const int32_t *len, const int64_t *end, int64_t n,
                 int32_t *first_leaf, int32_t *first_slot, int64_t *count, cudaStream_t s) {
  const bool wide = t->cfg.leaf_cap != 16, f128 = t->cfg.fanout != 64;
  auto pick = [&](auto between) {
    constexpr bool B = decltype(between)::value;
    return f128 ? (wide ? range_locate_kernel<128, 64, B> : range_locate_kernel<128, 16, B>)
                : (wide ? range_locate_kernel<64, 64, B> : range_locate_kernel<64, 16, B>);
  };
  auto k = end ? pick(std::true_type()) : pick(std::false_type());
  const size_t smem = search_smem_bytes(t);
  if (smem > 48 * 1024) {
    int rc = opt_in_smem((const void *)k, (int)smem);
    if (rc) return rc;
  }
  const int64_t per = end ? kThreads / 8 : kThreads / 4;
  const unsigned grid = (unsigned)std::min<int64_t>((n + per - 1) / per, (int64_t)t->num_sms * 6);
  DevTree v = t->view();
  v.wait_polls = kSpinLimit;  // hm_set_wait_limit is for the point searches
  k<<<grid, kThreads, smem, s>>>(v, start, len, end, n, first_leaf, first_slot, count, t->d_err);
  note_launch();
  return cuda_err(cudaGetLastError());
}

int range_copy_out(const hm_tree *t, const int32_t *first_leaf, const int32_t *first_slot,
                   const int64_t *offsets, int64_t n, int64_t cap, int64_t *okeys, int64_t *ovals, cudaStream_t s) {
  // a few queries a warp, so that enough warps have work
  const int per = (int)std::min<int64_t>(4, std::max<int64_t>(1, n / (t->num_sms * 48)));
  const unsigned blocks = (unsigned)((n + per * kCopyWarps - 1) / (per * kCopyWarps));
  auto k = t->cfg.leaf_cap == 16 ? range_copy_kernel<16> : range_copy_kernel<64>;
  constexpr int smem = kCopyWarps * 4 * kBuf * 8;
  int rc = opt_in_smem((const void *)k, smem);
  if (rc) return rc;
  launch_pdl(k, std::max(blocks, 1u), kCopyWarps * 32, smem, s, t->view(), first_leaf, first_slot, offsets, n,
             per, cap, okeys, ovals);
  note_launch();
  return cuda_err(cudaGetLastError());
}

}  // namespace hm
