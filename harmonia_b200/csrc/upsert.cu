// One epoch of batched upserts applied on the GPU.
//
// Reference: BPlusTree::insert_parallel_Newupdate_batch
// (open-harmonia/src/bpt-ppi-update-batch.cpp:86-200): 56 CPU threads
// descend per key, update an existing key under the leaf mutex
// (value = key-1, :47) or insert into the record list if it has room
// (:59-67), a leaf inner split otherwise (:71-76), a serial insert for the
// rest (:151-170) and a periodic re-BFS of the inner nodes
// (rebuild_without_leaf, open-harmonia/src/bpt-ppi-update.cpp:320-463).  The
// reference never refreshes the GPU copy.
//
// Here the epoch runs on the device tree itself, enqueued as one chain of
// kernels whose outcome the host reads once:
//   1. bucket sort of the batch by key (payload = input position, so the last
//      of equal keys is known; an LSD sort where its keys crowd a bucket);
//   2. every key descends; a hit overwrites the value in place (supplied
//      value, or key-1 under HM_UPSERT_REF_KEY_MINUS_1), a miss sets a bit;
//   3. the misses of one leaf are placed in its sorted row if it has room
//      (separators stay valid: a key routed to leaf j lies in
//      [separator_j, separator_j+1)), and leaf_base is rescanned;
//   4. if a leaf had no room, its subtree is rebalanced, or the tree is
//      rebuilt: the current contents and the left-over keys are merged (each
//      element's output slot = own rank + rank in the other run) and
//      bulk-loaded into a fresh arena with the same parameters.
#include "bucket_sort.cuh"
#include "warp_descent.cuh"

#include <algorithm>
#include <cstring>

namespace hm {


namespace {

constexpr int kThreads = 256;
constexpr int kApply = 128;      // threads of apply_kernel
constexpr int kRowThreads = 128;  // threads of leaf_rows_kernel

unsigned grid_for(int64_t items) {
  int64_t b = (items + kThreads - 1) / kThreads;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return (unsigned)b;
}

// ---- the batch in key order ----

// Last step of the batch's bucket sort: a CTA sorts one bucket in shared memory
// and writes its keys and their input positions, equal keys in input order.
// start == nullptr: the whole batch is one bucket.
__global__ void __launch_bounds__(bsort::kSortThreads, 5) epoch_sort_kernel(
    const int64_t *__restrict__ keys, const int32_t *__restrict__ pos, const uint32_t *__restrict__ start, uint32_t n,
    int64_t *__restrict__ sk, int32_t *__restrict__ spos, bsort::Ctl *ctl) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char dyn[];
  auto &sm = *reinterpret_cast<bsort::SortSmem<int32_t> *>(dyn);
  if (ctl->skew) return;
  const uint32_t s0 = start ? start[blockIdx.x] : 0;
  const int m = (int)((start ? start[blockIdx.x + 1] : n) - s0);
  if (m == 0) return;
  const bsort::Map map = ctl->map;
  auto emit = [&](int i, int64_t k, int32_t p, bool) {
    sk[s0 + i] = k;
    spos[s0 + i] = p;
    if (i == 0 || i == m - 1) {
      if (k == kMaxKey) atomicOr(&ctl->flags, 2u);  // sorts last
      if (s0 + i == 0) ctl->ends[0] = k;
      if (s0 + i == n - 1) ctl->ends[1] = k;
    }
  };
  if (start)
    bsort::sort_bucket<int32_t, false>(sm, map, keys + s0, pos + s0, m, emit);
  else
    bsort::sort_bucket<int32_t, true>(sm, map, keys, nullptr, m, emit);
}

// The same results from an LSD-sorted batch.
__global__ void lsd_finish_kernel(const uint64_t *__restrict__ uk, int64_t n, int64_t *__restrict__ sk,
                                  bsort::Ctl *ctl) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = (int64_t)(uk[i] ^ kSign);
    sk[i] = k;
    if (i == 0) ctl->ends[0] = k;
    if (i == n - 1) {
      ctl->ends[1] = k;
      if (k == kMaxKey) ctl->flags = 2u;
    }
  }
}

// Ctl::user of an epoch.
enum { kUserChanged = 0, kUserOverflow = 1, kUserEmpty = 2, kUserErr = 3 };  // keys added or removed; ...; error word

// A leaf's keys are one run of the sorted batch.  Nearly all runs end within a
// word of the mask, but a key that fills much of a batch makes a long one, of
// which few keys or none are marked.  A warp looks through such a run's marks
// kMarkStep words at a time, a latency of memory each, in a function of its own.
// 4096K keys, half of them one new key: 0.78 ms, 33.9 with a word at a time
// (0.66 without the new key).
constexpr int kMarkWords = 16, kMarkStep = 32 * kMarkWords;

// The nearest word with a set bit in a step of the mask: words w0 + d, w0 + 2 d,
// ... (d = 1 or -1) as far as they are in [0, words); -1 if none (all lanes).
__device__ __forceinline__ int64_t marked_word(const uint32_t *__restrict__ mask, int64_t w0, int d, int64_t words,
                                               uint32_t *bits) {
  const int lane = threadIdx.x & 31;
  uint32_t v[kMarkWords], any = 0;
#pragma unroll
  for (int x = 0; x < kMarkWords; x++) {
    const int64_t at = w0 + d * (x * 32 + lane + 1);
    v[x] = at >= 0 && at < words ? mask[at] : 0;
  }
#pragma unroll
  for (int x = 0; x < kMarkWords; x++) any |= v[x];
  if (!__any_sync(0xffffffffu, any != 0)) return -1;
  int64_t found = -1;
#pragma unroll
  for (int x = 0; x < kMarkWords; x++) {
    const uint32_t some = __ballot_sync(0xffffffffu, v[x] != 0);
    if (some && found < 0) {
      const int from = __ffs(some) - 1;
      *bits = __shfl_sync(0xffffffffu, v[x], from);
      found = w0 + d * (x * 32 + from + 1);
    }
  }
  return found;
}

// The rest of marked_before from word w on, and of next_marked.
__device__ __noinline__ bool marked_before_word(const uint32_t *__restrict__ mask, const int32_t *__restrict__ leaf_of,
                                                int64_t w, int64_t words, int32_t leaf) {
  for (; w > 0 && leaf_of[w * 32 - 1] == leaf; w -= kMarkStep) {
    uint32_t bits = 0;
    const int64_t at = marked_word(mask, w, -1, words, &bits);
    if (at >= 0) return leaf_of[at * 32 + 31 - __clz(bits)] == leaf;
  }
  return false;
}
__device__ __noinline__ int64_t marked_from_word(const uint32_t *__restrict__ mask, const int32_t *__restrict__ leaf_of,
                                                 int64_t w, int64_t words, int32_t leaf) {
  for (; w < words && leaf_of[w * 32] == leaf; w += kMarkStep) {
    uint32_t bits = 0;
    const int64_t at = marked_word(mask, w - 1, 1, words, &bits);
    if (at >= 0) {
      const int64_t i = at * 32 + __ffs(bits) - 1;
      return leaf_of[i] == leaf ? i : -1;
    }
  }
  return -1;
}

// Whether a set bit of mask before position i belongs to a key of the same
// leaf as position i's (all lanes, the same arguments).
__device__ __forceinline__ bool marked_before(const uint32_t *__restrict__ mask, const int32_t *__restrict__ leaf_of,
                                              int64_t i, int64_t n, int32_t leaf) {
  if (i == 0 || leaf_of[i - 1] != leaf) return false;
  const int64_t w = (i - 1) >> 5;
  const uint32_t m = mask[w] & (0xffffffffu >> (31 - ((i - 1) & 31)));
  if (m) return leaf_of[w * 32 + 31 - __clz(m)] == leaf;
  return marked_before_word(mask, leaf_of, w, (n + 31) / 32, leaf);
}

// First set bit of mask at or after i whose key lies in `leaf`; -1 if none
// (all lanes, the same arguments).
__device__ __forceinline__ int64_t next_marked(const uint32_t *__restrict__ mask, const int32_t *__restrict__ leaf_of,
                                               int64_t i, int64_t n, int32_t leaf) {
  if (i >= n || leaf_of[i] != leaf) return -1;
  const uint32_t m = mask[i >> 5] >> (i & 31);
  if (m) {
    i += __ffs(m) - 1;
    return leaf_of[i] == leaf ? i : -1;
  }
  return marked_from_word(mask, leaf_of, (i >> 5) + 1, (n + 31) / 32, leaf);
}

// Up to 32 marked keys of the sorted batch that a warp works on, and the last
// leaf's marked keys past them (one more than it can hold at most).
template <int LC>
struct WarpRows {
  int64_t key[32 + LC + 1], val[32 + LC + 1];  // by lane, then the last leaf's others (upsert)
  uint32_t members[32];                        // the lanes of the r-th leaf
  int32_t head[32];                            // the first of them
};

// The rows of the nh listed leaves, by groups of LC / 4 lanes that hold four
// slots each (eight 16-key leaves at a time).  Upsert: a leaf's new keys are
// placed among the sorted ones; a leaf without room for all of them is left as
// it is.  Delete: the emptied slots (Max_Key) are squeezed out in key order.
// Adds the keys stored or removed to *changed (per lane).  The leaf `last` has
// `extra` keys past the warp's 32.
template <int LC, bool DEL>
__device__ __forceinline__ void write_rows(WarpRows<LC> &wr, int nh, int32_t leaf, int32_t last, int extra,
                                           int64_t *leaf_rows, int32_t *leaf_cnt, bsort::Ctl *ctl, int *changed) {
  constexpr int LI = LC >= 32 ? LC / 8 : 0;
  constexpr int ROW = LI + 2 * LC;
  constexpr int G = LC / 4, NG = 32 / G;
  const int lane = threadIdx.x & 31, g = lane & (G - 1);
  for (int b = 0; b < nh; b += NG) {
    const int hi = b + lane / G;
    const bool act = hi < nh;
    uint32_t todo = act ? wr.members[hi] : 0;
    const int32_t lf = __shfl_sync(0xffffffffu, leaf, act ? wr.head[hi] : 0);
    int64_t *kr = leaf_rows + (int64_t)lf * ROW + LI, *vr = kr + LC;
    int64_t k[4], v[4];
    int to[4];  // where the slot's record goes
    {
      const longlong2 a = *reinterpret_cast<const longlong2 *>(kr + 4 * g);
      const longlong2 c = *reinterpret_cast<const longlong2 *>(kr + 4 * g + 2);
      const longlong2 d = *reinterpret_cast<const longlong2 *>(vr + 4 * g);
      const longlong2 e = *reinterpret_cast<const longlong2 *>(vr + 4 * g + 2);
      k[0] = a.x, k[1] = a.y, k[2] = c.x, k[3] = c.y;
      v[0] = d.x, v[1] = d.y, v[2] = e.x, v[3] = e.y;
    }
    const int cnt = leaf_cnt[lf];
    bool used[4];
#pragma unroll
    for (int x = 0; x < 4; x++) used[x] = 4 * g + x < cnt;
    if constexpr (DEL) {
      int mine = 0;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        used[x] &= k[x] != kMaxKey;
        mine += used[x];
      }
      int incl = mine;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o, G);
        if (g >= o) incl += y;
      }
      const int live = __shfl_sync(0xffffffffu, incl, G - 1, G);
      int at = incl - mine;
#pragma unroll
      for (int x = 0; x < 4; x++) to[x] = used[x] ? at++ : -1;
      __syncwarp();  // every lane has read its slots
      if (act) {
#pragma unroll
        for (int x = 0; x < 4; x++) {
          const int s = 4 * g + x;
          if (to[x] >= 0 && to[x] != s) {
            kr[to[x]] = k[x];
            vr[to[x]] = v[x];
          }
          if (s >= live && s < cnt) {
            kr[s] = kMaxKey;
            vr[s] = HM_NOT_FOUND;
          }
        }
        if (g == 0) {
          leaf_cnt[lf] = live;
          *changed += cnt - live;
          if (live == 0) ctl->user[kUserEmpty] = 1;
        }
      }
    } else {
      int64_t nk[4], nv[4];
      int ns[4], m = 0;
#pragma unroll
      for (int x = 0; x < 4; x++) {
        to[x] = 4 * g + x;
        ns[x] = -1;
      }
      int more = act && lf == last ? extra : 0, at = 32;
      bool over = false;
      while (__any_sync(0xffffffffu, todo != 0 || more > 0)) {
        int64_t q = 0, val = 0;
        bool have = todo != 0 || more > 0;
        if (have) {
          int j = at;
          if (todo != 0) {
            j = __ffs(todo) - 1;
            todo &= todo - 1;
          } else {
            at++;
            more--;
          }
          q = wr.key[j];
          val = wr.val[j];
        }
        if (have && cnt + m == LC) {  // no room
          over = true;
          have = false;
          todo = 0;
          more = 0;
        }
        int below = 0;
#pragma unroll
        for (int x = 0; x < 4; x++) below += have && used[x] && k[x] < q;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
        if (have) {
#pragma unroll
          for (int x = 0; x < 4; x++) {
            to[x] += used[x] && k[x] > q;
            if (4 * g + x == m) {  // the lane of slot m keeps the m-th new key
              nk[x] = q;
              nv[x] = val;
              ns[x] = below + m;
            }
          }
          m++;
        }
      }
      __syncwarp();  // every lane has read its slots
      if (act && !over) {
#pragma unroll
        for (int x = 0; x < 4; x++) {
          if (used[x] && to[x] != 4 * g + x) {
            kr[to[x]] = k[x];
            vr[to[x]] = v[x];
          }
          if (ns[x] >= 0) {
            kr[ns[x]] = nk[x];
            vr[ns[x]] = nv[x];
          }
        }
        if (g == 0) {
          leaf_cnt[lf] = cnt + m;
          *changed += m;
        }
      }
      if (over && g == 0) ctl->user[kUserOverflow] = 1;
    }
    if constexpr (LI > 0) {
      __syncwarp();
      if (act && g < LI) kr[g - LI] = 8 * (g + 1) < LC ? kr[8 * (g + 1)] : kMaxKey;
    }
  }
  __syncwarp();
}

// The batch against the leaves: a warp takes 32 neighbouring keys of the
// sorted batch, finds their leaves, and looks each key up in its leaf with
// four lanes (all 32 leaves' loads are issued before the first is used).
// Upsert: the last of equal keys counts; a stored key's value is overwritten
// (supplied value, or key - 1 under HM_UPSERT_REF_KEY_MINUS_1), a new key sets
// its bit in mask.  Delete: a stored key's slot becomes Max_Key and its bit is
// set.  leaf_of gets every key's leaf.  Nothing happens if a key of an upsert
// is Max_Key.
//
// Bound by DRAM on scattered sectors: a key's 128-B key row, the sector its
// value is written to and its value's sector.  Launched in full after the
// sort, not as a dependent launch: an SM keeps the shared-memory carve-out of
// the CTAs it runs, and CTAs that start behind the sort's would run the whole
// kernel with the little L1 the sort leaves (4096K keys on 2^26: 277 against
// 200 us).
template <int LC, bool DEL>
__global__ void __launch_bounds__(kApply, 10) apply_kernel(DevTree t, int f, int flags, const int64_t *__restrict__ sk,
                                                         const int32_t *__restrict__ spos,
                                                         const int64_t *__restrict__ vals, int64_t n,
                                                         int64_t *leaf_rows, int32_t *__restrict__ leaf_of,
                                                         uint32_t *__restrict__ mask, bsort::Ctl *ctl,
                                                         const unsigned *__restrict__ err) {
  constexpr int LI = LC >= 32 ? LC / 8 : 0;
  constexpr int ROW = LI + 2 * LC;
  const int lane = threadIdx.x & 31;
  const int64_t word = blockIdx.x * (int64_t)(kApply / 32) + (threadIdx.x >> 5), w0 = word * 32;
  if (w0 >= n) return;
  const int64_t i = min(w0 + lane, n - 1);
  const int64_t key = __ldg(sk + i);
  bool live = w0 + lane < n;
  int32_t pos = 0;
  int64_t val = 0;
  if constexpr (DEL) {
    live &= key != kMaxKey;  // never stored
  } else {
    live &= i == n - 1 || __ldg(sk + min(i + 1, n - 1)) != key;
    pos = __ldg(spos + i);
  }
  if (ctl->skew || (!DEL && (ctl->flags & 2u))) return;
  if (word == 0 && lane == 0) ctl->user[kUserErr] = *err;
  const int32_t leaf = descend_leaf_warp(t, f, DEL && key == kMaxKey ? kMaxKey - 1 : key);
  if (w0 + lane < n) leaf_of[i] = leaf;
  // four lanes per key, eight keys per step
  const int sub = lane & 3;
  longlong2 a[4], b[4];
  int base[4];
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int32_t lf = __shfl_sync(0xffffffffu, leaf, s * 8 + (lane >> 2));
    const int64_t *r = leaf_rows + (int64_t)lf * ROW;
    base[s] = 0;
    if constexpr (LI == 0) {
      a[s] = *reinterpret_cast<const longlong2 *>(r + 2 * sub);
      b[s] = *reinterpret_cast<const longlong2 *>(r + 8 + 2 * sub);
    } else {
      a[s] = *reinterpret_cast<const longlong2 *>(r + 2 * sub);  // the leaf's index words
    }
  }
  if constexpr (!DEL) val = flags & HM_UPSERT_REF_KEY_MINUS_1 ? key - 1 : __ldg(vals + pos);
  if constexpr (LI != 0) {
    static_assert(LI == 0 || LI == 8, "two index words a lane");
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const int64_t q = __shfl_sync(0xffffffffu, key, s * 8 + (lane >> 2));
      int k = (a[s].x <= q) + (a[s].y <= q);
      k += __shfl_xor_sync(0xffffffffu, k, 1);
      k += __shfl_xor_sync(0xffffffffu, k, 2);
      base[s] = 8 * min(k, LI - 1);
      const int32_t lf = __shfl_sync(0xffffffffu, leaf, s * 8 + (lane >> 2));
      a[s] = *reinterpret_cast<const longlong2 *>(leaf_rows + (int64_t)lf * ROW + LI + base[s] + 2 * sub);
      b[s] = make_longlong2(0, 0);
    }
  }
  const uint32_t lives = __ballot_sync(0xffffffffu, live);
  bool hit = false;
#pragma unroll
  for (int s = 0; s < 4; s++) {
    const int own = s * 8 + (lane >> 2);
    const int64_t q = __shfl_sync(0xffffffffu, key, own);
    const int32_t lf = __shfl_sync(0xffffffffu, leaf, own);
    const int64_t v = __shfl_sync(0xffffffffu, val, own);
    int slot = -1;
    if constexpr (LI == 0) {
      if (a[s].x == q) slot = 2 * sub;
      if (a[s].y == q) slot = 2 * sub + 1;
      if (b[s].x == q) slot = 8 + 2 * sub;
      if (b[s].y == q) slot = 8 + 2 * sub + 1;
    } else {
      if (a[s].x == q) slot = base[s] + 2 * sub;
      if (a[s].y == q) slot = base[s] + 2 * sub + 1;
    }
    if (!((lives >> own) & 1u)) slot = -1;
    if (slot >= 0) {
      int64_t *r = leaf_rows + (int64_t)lf * ROW + LI + slot;
      if constexpr (DEL)
        r[0] = kMaxKey;
      else
        r[LC] = v;
    }
    const uint32_t m = __ballot_sync(0xffffffffu, slot >= 0);
    if (lane >> 3 == s) hit = (m >> (4 * (lane & 7))) & 0xfu;
  }
  const uint32_t out = __ballot_sync(0xffffffffu, live && (DEL ? hit : !hit));
  if (lane == 0) mask[word] = out;
}

// Position of the k-th set bit of w (k < __popc(w)).
__device__ __forceinline__ int nth_bit(uint32_t w, int k) {
  int at = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    const int c = __popc((w >> at) & ((1u << step) - 1u));
    if (k >= c) {
      k -= c;
      at += step;
    }
  }
  return at;
}

// The rows of the leaves of the marked keys.  A warp takes wpw words of the
// mask (few in a small batch, for more warps) and their marked keys 32 at a
// time, one per lane, so that their loads are in flight together; a leaf is
// handled where its first marked key lies.  The bounds hold the registers at
// what the short runs need: with 80 instead of 72 the epoch pair of 4096K keys
// takes 544 instead of 536 us.
template <int LC, bool DEL>
__global__ void __launch_bounds__(kRowThreads, DEL ? 10 : 7) leaf_rows_kernel(const int64_t *__restrict__ sk,
                                                                const int32_t *__restrict__ spos,
                                                                const int64_t *__restrict__ vals, int64_t n, int wpw,
                                                                const int32_t *__restrict__ leaf_of,
                                                                const uint32_t *__restrict__ mask, int64_t *leaf_rows,
                                                                int32_t *leaf_cnt, bsort::Ctl *ctl) {
  pdl_enter();
  __shared__ WarpRows<LC> s_rows[kRowThreads / 32];
  if (ctl->skew || (!DEL && (ctl->flags & 2u))) return;
  const int lane = threadIdx.x & 31;
  WarpRows<LC> &wr = s_rows[threadIdx.x >> 5];
  const int64_t words = (n + 31) / 32;
  const int64_t base = (blockIdx.x * (int64_t)(kRowThreads / 32) + (threadIdx.x >> 5)) * wpw;
  const uint32_t mine = lane < wpw && base + lane < words ? mask[base + lane] : 0;
  const int cnt = __popc(mine);
  int incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  int changed = 0;
  int32_t last = -1;  // leaf of the last marked key of the round before
  for (int c0 = 0; c0 < total; c0 += 32) {
    const int r = min(c0 + lane, total - 1);
    const bool valid = c0 + lane < total;
    int wl = 0;  // the lane whose word holds marked key r
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, incl, wl + step - 1) <= r) wl += step;
    const uint32_t w = __shfl_sync(0xffffffffu, mine, wl);
    const int below = __shfl_sync(0xffffffffu, incl - cnt, wl);
    const int64_t i = (base + wl) * 32 + nth_bit(w, r - below);
    const int32_t leaf = leaf_of[i];
    if (!DEL) {
      wr.key[lane] = sk[i];
      wr.val[lane] = vals[spos[i]];
    }
    const int32_t up = __shfl_up_sync(0xffffffffu, leaf, 1);
    bool head = valid && leaf != (lane == 0 ? last : up);
    if (c0 == 0) {
      const bool before = marked_before(mask, leaf_of, __shfl_sync(0xffffffffu, i, 0), n, __shfl_sync(0xffffffffu, leaf, 0));
      if (lane == 0) head = !before;
    }
    const uint32_t heads = __ballot_sync(0xffffffffu, head);
    const uint32_t members = __match_any_sync(0xffffffffu, leaf) & __ballot_sync(0xffffffffu, valid);
    if (head) {
      const int h = __popc(heads & ((1u << lane) - 1u));
      wr.head[h] = lane;
      wr.members[h] = members;
    }
    last = __shfl_sync(0xffffffffu, leaf, 31);
    int extra = 0;
    if (!DEL) {
      for (int64_t at = __shfl_sync(0xffffffffu, i, 31) + 1; extra <= LC; at++) {
        at = next_marked(mask, leaf_of, at, n, last);
        if (at < 0) break;
        if (lane == 0) {
          wr.key[32 + extra] = sk[at];
          wr.val[32 + extra] = vals[spos[at]];
        }
        extra++;
      }
    }
    __syncwarp();
    write_rows<LC, DEL>(wr, __popc(heads), leaf, last, extra, leaf_rows, leaf_cnt, ctl, &changed);
  }
  changed = __reduce_add_sync(0xffffffffu, changed);
  if (lane == 0 && changed > 0) atomicAdd(&ctl->user[kUserChanged], (unsigned long long)changed);
}

// New keys that their leaf had no room for, as flags to scan.
__global__ void left_over_kernel(const int64_t *__restrict__ sk, const int32_t *__restrict__ leaf_of,
                                 const uint32_t *__restrict__ mask, int64_t n, int lc, int li,
                                 const int64_t *__restrict__ leaf_rows, int32_t *__restrict__ miss) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    bool left = (mask[i >> 5] >> (i & 31)) & 1u;
    if (left) {
      const int64_t q = sk[i];
      const int64_t *kr = leaf_rows + (int64_t)leaf_of[i] * (li + 2 * lc) + li;
      for (int s = 0; s < lc; s++) left &= kr[s] != q;
    }
    miss[i] = left;
  }
}

__global__ void compact_miss_kernel(const int64_t *__restrict__ sk, const int32_t *__restrict__ spos,
                                    const int64_t *__restrict__ vals, const int32_t *__restrict__ leaf_of,
                                    const int32_t *__restrict__ miss, const int64_t *__restrict__ at, int64_t n,
                                    int64_t *__restrict__ mk, int64_t *__restrict__ mv, int32_t *__restrict__ ml) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (miss[i]) {
      int64_t o = at[i];
      mk[o] = sk[i];
      mv[o] = vals[spos[i]];
      ml[o] = leaf_of[i];
    }
  }
}

// For each run of left-over keys on one leaf (they are in key order, so
// leaves are non-decreasing): its first key is marked and gets the run's
// length and leaf.
__global__ void miss_runs_kernel(const int32_t *__restrict__ ml, int64_t nm, int32_t *__restrict__ run_len,
                                 int32_t *__restrict__ run_leaf, int32_t *__restrict__ is_start) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nm;
       i += (int64_t)gridDim.x * blockDim.x) {
    bool st = (i == 0) || ml[i] != ml[i - 1];
    is_start[i] = st ? 1 : 0;
    if (st) {
      int64_t e = i + 1;
      while (e < nm && ml[e] == ml[i]) e++;
      run_len[i] = (int32_t)(e - i);
      run_leaf[i] = ml[i];
    }
  }
}

// ---- subtree rebalancing (an epoch whose new keys overflow a leaf) ----
//
// The subtree of a last-level inner node p is its children leaves [a, b].
// When a leaf overflows but p's subtree still has room for its keys and all
// the epoch's new keys routed into it, the subtree's keys are re-spread
// evenly over the same leaves and p's separators rewritten; nothing outside
// the subtree changes (p's own separator in its parent stays a valid fence,
// because every new key routed here is at least that separator).  Only when
// some subtree has no room is the whole tree rebuilt.

struct Subtree {
  int64_t lvl0, lvl1;  // last inner level: nodes [lvl0, lvl1); lvl1 == n_inner
  int64_t n_inner, n_leaf;
};

__device__ __forceinline__ int64_t first_miss_at_or_after(const int32_t *__restrict__ ml, int64_t nm, int64_t leaf) {
  int64_t lo = 0, hi = nm;  // first miss whose leaf >= leaf
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (ml[mid] < leaf) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void subtree_leaves(const int32_t *__restrict__ prefix, const Subtree &g, int64_t p,
                                               int64_t *a, int64_t *b) {
  const int64_t c0 = prefix[p];
  const int64_t c1 = p + 1 < g.lvl1 ? prefix[p + 1] : g.n_inner + g.n_leaf;
  *a = c0 - g.n_inner;
  *b = c1 - 1 - g.n_inner;
}

// One thread per run of misses: its leaf's parent (run_parent, as an index
// into the last level); an overflowing leaf marks its parent when the
// subtree has room, else flags bit2 (rebuild the tree).
__global__ void subtree_mark_kernel(const int32_t *__restrict__ prefix, const int32_t *__restrict__ leaf_cnt,
                                    const int64_t *__restrict__ leaf_base, int lc, Subtree g,
                                    const int32_t *__restrict__ is_start, const int32_t *__restrict__ run_len,
                                    const int32_t *__restrict__ run_leaf, const int32_t *__restrict__ ml,
                                    int64_t nm, int32_t *__restrict__ run_parent, int32_t *__restrict__ mark,
                                    unsigned *flags) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nm;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (!is_start[i]) continue;
    const int64_t leaf = run_leaf[i];
    int64_t lo = g.lvl0, hi = g.lvl1 - 1;  // last node p with prefix[p] <= the leaf's id
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) >> 1;
      if (prefix[mid] <= g.n_inner + leaf) lo = mid; else hi = mid - 1;
    }
    run_parent[i] = (int32_t)(lo - g.lvl0);
    if (leaf_cnt[leaf] + run_len[i] <= lc) continue;
    int64_t a, b;
    subtree_leaves(prefix, g, lo, &a, &b);
    const int64_t keys = leaf_base[b] + leaf_cnt[b] - leaf_base[a];
    const int64_t adds = first_miss_at_or_after(ml, nm, b + 1) - first_miss_at_or_after(ml, nm, a);
    if (keys + adds <= (b - a + 1) * (int64_t)lc) {
      mark[lo - g.lvl0] = 1;
    } else {
      atomicOr(flags, 4u);
    }
  }
}

// One CTA per last-level node; marked ones are rebalanced.  The existing
// records are gathered into shared memory first, then every element (old or
// new) is written to its place in the merged order, spread evenly over the
// subtree's leaves (leaf jj gets positions [part_start(jj), part_start(jj+1))).
__global__ void subtree_rebalance_kernel(int64_t *inner, const int32_t *__restrict__ prefix, int64_t *leaf_rows,
                                         int32_t *leaf_cnt, const int64_t *__restrict__ leaf_base, int f, int lc,
                                         int li, Subtree g, const int32_t *__restrict__ mark,
                                         const int64_t *__restrict__ mk, const int64_t *__restrict__ mv,
                                         const int32_t *__restrict__ ml, int64_t nm) {
  extern __shared__ __align__(16) longlong2 staged[];  // the subtree's existing records
  if (!mark[blockIdx.x]) return;
  const int64_t p = g.lvl0 + blockIdx.x;
  int64_t a, b;
  subtree_leaves(prefix, g, p, &a, &b);
  const int64_t nl = b - a + 1, row = li + 2 * lc;
  const int64_t base = leaf_base[a];
  const int64_t K = leaf_base[b] + leaf_cnt[b] - base;
  const int64_t m0 = first_miss_at_or_after(ml, nm, a), m1 = first_miss_at_or_after(ml, nm, b + 1);
  const int64_t M = m1 - m0, T = K + M;
  for (int64_t x = threadIdx.x; x < nl * lc; x += blockDim.x) {
    const int64_t j = a + x / lc, sl = x % lc;
    if (sl < leaf_cnt[j]) {
      const int64_t *r = leaf_rows + j * row + li;
      staged[leaf_base[j] - base + sl] = make_longlong2(r[sl], r[lc + sl]);
    }
  }
  __syncthreads();
  const int64_t q = T / nl, rem = T % nl;
  auto put = [&](int64_t pos, int64_t k, int64_t v) {
    const int64_t jj = pos < rem * (q + 1) ? pos / (q + 1) : rem + (pos - rem * (q + 1)) / q;
    const int64_t sl = pos - part_start(jj, T, nl);
    int64_t *r = leaf_rows + (a + jj) * row + li;
    r[sl] = k;
    r[lc + sl] = v;
  };
  for (int64_t e = threadIdx.x; e < K; e += blockDim.x) {  // old record: own index + new keys below it
    const int64_t k = staged[e].x;
    int64_t lo = m0, hi = m1;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (mk[mid] < k) lo = mid + 1; else hi = mid;
    }
    put(e + (lo - m0), k, staged[e].y);
  }
  for (int64_t i = threadIdx.x; i < M; i += blockDim.x) {  // new key: own index + old keys below it
    const int64_t k = mk[m0 + i];
    int64_t lo = 0, hi = K;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (staged[mid].x < k) lo = mid + 1; else hi = mid;
    }
    put(i + lo, k, mv[m0 + i]);
  }
  for (int64_t x = threadIdx.x; x < nl * lc; x += blockDim.x) {  // padding and counts
    const int64_t jj = x / lc, sl = x % lc;
    const int64_t len = part_start(jj + 1, T, nl) - part_start(jj, T, nl);
    if (sl >= len) {
      int64_t *r = leaf_rows + (a + jj) * row + li;
      r[sl] = kMaxKey;
      r[lc + sl] = HM_NOT_FOUND;
    }
    if (sl == 0) leaf_cnt[a + jj] = (int32_t)len;
  }
  __syncthreads();
  for (int64_t x = threadIdx.x; x < nl * li; x += blockDim.x) {  // 64-key leaves: index words
    const int64_t jj = x / li, w = x % li;
    int64_t *r = leaf_rows + (a + jj) * row;
    r[w] = 8 * (w + 1) < lc ? r[li + 8 * (w + 1)] : kMaxKey;
  }
  int64_t *pr = inner + p * (f / 8 + f);
  for (int sidx = threadIdx.x; sidx < f; sidx += blockDim.x)  // separators: first key of child s + 1
    pr[f / 8 + sidx] = sidx < nl - 1 ? leaf_rows[(a + sidx + 1) * row + li] : kMaxKey;
  __syncthreads();
  for (int w = threadIdx.x; w < f / 8; w += blockDim.x) pr[w] = 8 * (w + 1) < f ? pr[f / 8 + 8 * (w + 1)] : kMaxKey;
}

// Merge of two sorted, disjoint runs: out slot = own index + rank in the other run.
__global__ void merge_rank_kernel(const int64_t *__restrict__ a, const int64_t *__restrict__ av, int64_t na,
                                  const int64_t *__restrict__ b, int64_t nb, bool strict,
                                  uint64_t *__restrict__ ok, int64_t *__restrict__ ov) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < na;
       i += (int64_t)gridDim.x * blockDim.x) {
    int64_t k = a[i];
    int64_t lo = 0, hi = nb;  // first b >= k (strict) or > k
    while (lo < hi) {
      int64_t mid = (lo + hi) >> 1;
      bool before = strict ? (b[mid] < k) : (b[mid] <= k);
      if (before) lo = mid + 1; else hi = mid;
    }
    ok[i + lo] = (uint64_t)k ^ kSign;
    ov[i + lo] = av[i];
  }
}

size_t al(int64_t bytes) { return (size_t)align_up(bytes, 256); }

// Keys in one upsert or delete epoch, at most: the batch sort carries each
// key's input position as an int32 (such a batch would need about 200 GB of
// scratch anyway).
constexpr int64_t kMaxEpochKeys = 0x7fffffff;

// A batch in key order on its way through the tree (device memory of one
// scratch lease).
struct Epoch {
  int64_t n = 0;
  int64_t *ka = nullptr, *kb = nullptr;  // sort buffers; the sorted keys end in sk
  int32_t *pa = nullptr, *pb = nullptr;
  int64_t *sk = nullptr;
  int32_t *spos = nullptr;
  int32_t *leaf_of = nullptr;
  uint32_t *mask = nullptr;
  void *sort_scratch = nullptr, *scan_scratch = nullptr;
  bsort::Ctl *ctl = nullptr;
  ReadSlot slot;  // held before the tree changes: its size and key range follow from what is read

  static size_t sort_bytes(int64_t n) {
    return std::max(al((int64_t)radix_scratch_bytes(n)), bsort::fits(n) ? bsort::work_bytes(n) : 0) +
           al(sizeof(bsort::Ctl));
  }
  static size_t scan_bytes(const hm_tree *t, int64_t n) {
    return al((int64_t)scan_scratch_bytes(std::max<int64_t>(n, t->n_leaf) + 1));
  }
  static size_t bytes(const hm_tree *t, int64_t n) {
    return 2 * al(8 * n) + 3 * al(4 * n) + al(4 * (n / 32 + 1)) + sort_bytes(n) + scan_bytes(t, n);
  }
  char *place(const hm_tree *t, int64_t n_, char *p) {
    n = n_;
    auto take = [&](size_t b) { char *r = p; p += b; return r; };
    ka = reinterpret_cast<int64_t *>(take(al(8 * n)));
    kb = reinterpret_cast<int64_t *>(take(al(8 * n)));
    pa = reinterpret_cast<int32_t *>(take(al(4 * n)));
    pb = reinterpret_cast<int32_t *>(take(al(4 * n)));
    leaf_of = reinterpret_cast<int32_t *>(take(al(4 * n)));
    mask = reinterpret_cast<uint32_t *>(take(al(4 * (n / 32 + 1))));
    sort_scratch = take(sort_bytes(n));
    scan_scratch = take(scan_bytes(t, n));
    return p;
  }

  // Bucket sort of the batch; enqueues only.  The control block's skew says
  // whether the batch's keys crowd a bucket, nothing was sorted then.
  void bucket_sort(const hm_tree *t, const int64_t *keys, cudaStream_t s) {
    const bsort::Work w = bsort::layout(n, sort_scratch);
    ctl = w.ctl;
    const int passes = bsort::partition_pairs<int32_t>(keys, nullptr, n, ka, pa, kb, pb, w, t->num_sms, s);
    const int64_t *in_k = passes == 2 ? kb : passes == 1 ? ka : keys;
    const int32_t *in_p = passes == 2 ? pb : passes == 1 ? pa : nullptr;
    sk = passes == 1 ? kb : ka;
    spos = passes == 1 ? pb : pa;
    constexpr int sm = (int)sizeof(bsort::SortSmem<int32_t>);
    opt_in_smem((const void *)epoch_sort_kernel, sm);
    launch_pdl(epoch_sort_kernel, 1u << bsort::shape_for(n).bits, bsort::kSortThreads, sm, s, in_k, in_p,
               static_cast<const uint32_t *>(passes ? w.start : nullptr), (uint32_t)n, sk, spos, ctl);
    note_launch();
  }

  // LSD sort of the batch, for keys that the bucket sort does not take.
  void lsd_sort(const int64_t *keys, cudaStream_t s) {
    ctl = reinterpret_cast<bsort::Ctl *>(static_cast<char *>(sort_scratch) + al((int64_t)radix_scratch_bytes(n)));
    cudaMemsetAsync(ctl, 0, sizeof(bsort::Ctl), s);
    uint64_t *u = reinterpret_cast<uint64_t *>(ka), *ua = reinterpret_cast<uint64_t *>(kb);
    transform_keys_in(keys, u, n, s);
    const bool alt = radix_sort_positions(u, pa, ua, pb, n, 0, 64, sort_scratch, s);
    sk = alt ? ka : kb;
    spos = alt ? pb : pa;
    lsd_finish_kernel<<<grid_for(n), kThreads, 0, s>>>(alt ? ua : u, n, sk, ctl);
    note_launch();
  }

  // The sorted batch against the tree's leaves, and leaf_base after it.
  void apply(const hm_tree *t, const int64_t *vals, int flags, bool del, cudaStream_t s) {
    const unsigned key_grid = (unsigned)((n + kApply - 1) / kApply);
    const int64_t words = (n + 31) / 32;
    const int wpw = (int)std::min<int64_t>(32, std::max<int64_t>(1, words / (t->num_sms * 16)));
    const unsigned row_grid = (unsigned)((words + wpw * (kRowThreads / 32) - 1) / (wpw * (kRowThreads / 32)));
    const bool wide = t->cfg.leaf_cap != 16;
    const int64_t *csk = sk;
    const int32_t *cpos = spos, *cleaf = leaf_of;
    const uint32_t *cmask = mask;
    const unsigned *err = t->d_err;
    auto look = del ? (wide ? apply_kernel<64, true> : apply_kernel<16, true>)
                    : (wide ? apply_kernel<64, false> : apply_kernel<16, false>);
    look<<<key_grid, kApply, 0, s>>>(t->view(), t->cfg.fanout, flags, csk, cpos, vals, n, t->leaf_rows, leaf_of, mask,
                                     ctl, err);
    auto rows = del ? (wide ? leaf_rows_kernel<64, true> : leaf_rows_kernel<16, true>)
                    : (wide ? leaf_rows_kernel<64, false> : leaf_rows_kernel<16, false>);
    launch_pdl(rows, row_grid, kRowThreads, 0, s, csk, cpos, vals, n, wpw, cleaf, cmask, t->leaf_rows, t->leaf_cnt,
               ctl);
    note_launch(2);
    rescan_leaf_base(t, &ctl->user[kUserChanged], scan_scratch, s);
  }

  int run(const hm_tree *t, const int64_t *keys, const int64_t *vals, int flags, bool del, bsort::Ctl *h,
          cudaStream_t s) {
    if (!slot.ok()) return HM_ENOMEM;
    h->skew = 1;
    if (bsort::fits(n)) {
      bucket_sort(t, keys, s);
      apply(t, vals, flags, del, s);
      int rc = read(h, s);
      if (rc) return rc;
    }
    if (h->skew) {
      lsd_sort(keys, s);
      apply(t, vals, flags, del, s);
      return read(h, s);
    }
    return HM_OK;
  }

  int read(bsort::Ctl *h, cudaStream_t s) const {
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? cuda_err(e) : slot.read(h, ctl, sizeof(*h), s);
  }
};

}  // namespace

// Bulk-loads n1 sorted (sign-flipped) keys and their values into a fresh arena
// with the tree's parameters and swaps it in; the old arena is freed.
int rebuild_from_sorted(hm_tree *t, const uint64_t *ck, const int64_t *cv, int64_t n1, cudaStream_t s) {
  BuildTarget nt = t->target();  // new shape; the arena is swapped in at the end
  int rc = shape(n1, t->cfg, &nt.height, nt.lvl_start, &nt.n_inner, &nt.n_leaf);
  if (rc) return rc;
  size_t off_prefix = al(nt.n_inner * nt.inner_row * 8);
  size_t off_lrows = off_prefix + al(align_up(nt.n_inner, 4) * 4);
  size_t off_lcnt = off_lrows + al(nt.n_leaf * nt.leaf_row * 8);
  size_t off_lbase = off_lcnt + al(nt.n_leaf * 4);
  size_t total = off_lbase + al(nt.n_leaf * 8);
  int64_t tn = std::max<int64_t>(std::max<int64_t>(n1, nt.n_leaf), 1);
  char *tmp = nullptr;
  void *arena = nullptr;
  cudaError_t e = dev_alloc(&arena, total);
  if (e == cudaSuccess) e = dev_alloc(reinterpret_cast<void **>(&tmp), 2 * al(8 * tn));
  if (e != cudaSuccess) {
    dev_release(arena);
    dev_release(tmp);
    return cuda_err(e);
  }
  int64_t *tmp_a = reinterpret_cast<int64_t *>(tmp);
  int64_t *tmp_b = reinterpret_cast<int64_t *>(tmp + al(8 * tn));
  char *base = static_cast<char *>(arena);
  nt.inner = reinterpret_cast<int64_t *>(base);
  nt.prefix = reinterpret_cast<int32_t *>(base + off_prefix);
  nt.leaf_rows = reinterpret_cast<int64_t *>(base + off_lrows);
  nt.leaf_cnt = reinterpret_cast<int32_t *>(base + off_lcnt);
  nt.leaf_base = reinterpret_cast<int64_t *>(base + off_lbase);
  rc = build_from_sorted(nt, ck, cv, n1, tmp_a, tmp_b, s);
  e = cudaStreamSynchronize(s);
  dev_release(tmp);
  if (rc == HM_OK && e != cudaSuccess) rc = cuda_err(e);
  if (rc) {
    dev_release(arena);
    return rc;
  }
  cudaDeviceSynchronize();  // no call of any stream may still read the old arena
  dev_release(t->arena);
  t->arena = arena;
  t->arena_bytes = total;
  t->inner = nt.inner;
  t->prefix = nt.prefix;
  t->leaf_rows = nt.leaf_rows;
  t->leaf_cnt = nt.leaf_cnt;
  t->leaf_base = nt.leaf_base;
  t->height = nt.height;
  std::memcpy(t->lvl_start, nt.lvl_start, sizeof(t->lvl_start));
  t->n_inner = nt.n_inner;
  t->n_leaf = nt.n_leaf;
  t->n_keys = n1;
  t->generation++;
  return HM_OK;
}

int upsert_epoch(hm_tree *t, const int64_t *d_keys, const int64_t *d_vals, int64_t n, int flags, unsigned *err,
                 cudaStream_t s) {
  if (n <= 0) return HM_OK;
  if (n > kMaxEpochKeys) return HM_ETOOLARGE;
  const int lc = t->cfg.leaf_cap, li = t->leaf_index;
  // the batch's own memory, then what an epoch with overflowing leaves needs:
  // at, mk, mv (8 B), miss, ml, is_start, run_len, run_leaf, run_parent (4 B)
  // and the subtree marks, one per last-level node
  const size_t s8 = al(8 * (n + 1)), s4 = al(4 * (n + 1));
  ScratchLease lease(t, s);
  int rc = lease.acquire(Epoch::bytes(t, n) + 3 * s8 + 6 * s4 + al(4 * (t->n_inner + 1)));
  if (rc) return rc;
  Epoch ep;
  char *p = ep.place(t, n, static_cast<char *>(lease.ptr()));
  bsort::Ctl h{};
  rc = ep.run(t, d_keys, d_vals, flags, false, &h, s);
  if (rc) return rc;
  if (h.flags & 2u) return HM_EMAXKEY;
  *err = (unsigned)h.user[kUserErr];
  const bool was_empty = t->n_keys == 0;
  t->n_keys += (int64_t)h.user[kUserChanged];
  // a stored key lies between key_min and key_max already
  if (was_empty || h.ends[0] < t->key_min) t->key_min = h.ends[0];
  if (was_empty || h.ends[1] > t->key_max) t->key_max = h.ends[1];
  if (!h.user[kUserOverflow]) return HM_OK;

  // Some leaf has no room for its new keys: rebalance the subtrees (last-level
  // nodes) that have room; if one has none, rebuild the tree.
  auto take = [&](size_t b) { char *r = p; p += b; return r; };
  int64_t *at = reinterpret_cast<int64_t *>(take(s8));
  int64_t *mk = reinterpret_cast<int64_t *>(take(s8));
  int64_t *mv = reinterpret_cast<int64_t *>(take(s8));
  int32_t *miss = reinterpret_cast<int32_t *>(take(s4));
  int32_t *ml = reinterpret_cast<int32_t *>(take(s4));
  int32_t *is_start = reinterpret_cast<int32_t *>(take(s4));
  int32_t *run_len = reinterpret_cast<int32_t *>(take(s4));
  int32_t *run_leaf = reinterpret_cast<int32_t *>(take(s4));
  int32_t *run_parent = reinterpret_cast<int32_t *>(take(s4));
  int32_t *mark = reinterpret_cast<int32_t *>(p);
  left_over_kernel<<<grid_for(n), kThreads, 0, s>>>(ep.sk, ep.leaf_of, ep.mask, n, lc, li, t->leaf_rows, miss);
  exclusive_scan_i32(miss, at, n, ep.scan_scratch, s);
  compact_miss_kernel<<<grid_for(n), kThreads, 0, s>>>(ep.sk, ep.spos, d_vals, ep.leaf_of, miss, at, n, mk, mv, ml);
  note_launch(2);
  int64_t nm = 0;
  cudaError_t e = cudaMemcpyAsync(&nm, at + n, 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_err(e);
  const Subtree g{t->lvl_start[t->height - 1], t->n_inner, t->n_inner, t->n_leaf};
  const int64_t last_nodes = g.lvl1 - g.lvl0;
  miss_runs_kernel<<<grid_for(nm), kThreads, 0, s>>>(ml, nm, run_len, run_leaf, is_start);
  cudaMemsetAsync(mark, 0, 4 * last_nodes, s);
  subtree_mark_kernel<<<grid_for(nm), kThreads, 0, s>>>(t->prefix, t->leaf_cnt, t->leaf_base, lc, g, is_start, run_len,
                                                         run_leaf, ml, nm, run_parent, mark, &ep.ctl->flags);
  note_launch(2);
  rc = ep.read(&h, s);
  if (rc) return rc;
  if (!(h.flags & 4u)) {
    const size_t smem = (size_t)t->cfg.fanout * lc * sizeof(longlong2);
    rc = opt_in_smem((const void *)subtree_rebalance_kernel, 128 * 64 * (int)sizeof(longlong2));  // up to 128 KiB
    if (rc) return rc;
    subtree_rebalance_kernel<<<(unsigned)last_nodes, kThreads, smem, s>>>(
        t->inner, t->prefix, t->leaf_rows, t->leaf_cnt, t->leaf_base, t->cfg.fanout, lc, li, g, mark, mk, mv, ml, nm);
    note_launch();
    t->shape_version++;  // separators of the last inner level changed
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_err(e);
    rescan_leaf_base(t, nullptr, ep.scan_scratch, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_err(e);
    t->n_keys += nm;
    return HM_OK;
  }
  // Rebuild: contents (already carrying the rest of this epoch) merged with
  // the left-over keys, then a bulk load into a fresh arena.
  const int64_t n0 = t->n_keys, n1 = n0 + nm;
  const int64_t tn = std::max<int64_t>(n1, 1);
  char *tmp = nullptr;
  e = dev_alloc(reinterpret_cast<void **>(&tmp), 4 * al(8 * tn));
  if (e != cudaSuccess) return cuda_err(e);
  int64_t *ek = reinterpret_cast<int64_t *>(tmp);
  int64_t *ev = reinterpret_cast<int64_t *>(tmp + al(8 * tn));
  uint64_t *ck = reinterpret_cast<uint64_t *>(tmp + 2 * al(8 * tn));
  int64_t *cv = reinterpret_cast<int64_t *>(tmp + 3 * al(8 * tn));
  export_contents(t, ek, ev, s);
  merge_rank_kernel<<<grid_for(n0), kThreads, 0, s>>>(ek, ev, n0, mk, nm, true, ck, cv);
  merge_rank_kernel<<<grid_for(nm), kThreads, 0, s>>>(mk, mv, nm, ek, n0, true, ck, cv);
  note_launch(2);
  rc = rebuild_from_sorted(t, ck, cv, n1, s);
  release_after(tmp, s);
  return rc;
}

// One epoch of deletes (no counterpart in the reference, whose
// BPlusTree::remove is an empty stub, open-harmonia/src/bpt.cpp:771-773):
// sort the batch, mark each stored key's slot, squeeze the touched leaves in
// place and rescan leaf_base.  Separators stay valid (the remaining keys of
// leaf j still lie between its separators), so the inner levels are
// untouched.  A leaf left empty would break the invariant that every leaf's
// first key is a key of the leaf (the bucket join searches leaves by first
// key), so such an epoch ends in a rebuild of the remaining contents instead.
int delete_epoch(hm_tree *t, const int64_t *d_keys, int64_t n, int64_t *removed_out, unsigned *err, cudaStream_t s) {
  if (removed_out) *removed_out = 0;
  if (n <= 0) return HM_OK;
  if (n > kMaxEpochKeys) return HM_ETOOLARGE;
  ScratchLease lease(t, s);
  int rc = lease.acquire(Epoch::bytes(t, n));
  if (rc) return rc;
  Epoch ep;
  ep.place(t, n, static_cast<char *>(lease.ptr()));
  bsort::Ctl h{};
  rc = ep.run(t, d_keys, nullptr, 0, true, &h, s);
  if (rc) return rc;
  *err = (unsigned)h.user[kUserErr];
  const int64_t removed = (int64_t)h.user[kUserChanged];
  if (removed_out) *removed_out = removed;
  t->n_keys -= removed;
  if (!h.user[kUserEmpty]) return HM_OK;
  // a leaf emptied: rebuild from the remaining contents
  const int64_t n1 = t->n_keys, tn = std::max<int64_t>(n1, 1);
  char *tmp = nullptr;
  cudaError_t e = dev_alloc(reinterpret_cast<void **>(&tmp), 3 * al(8 * tn));
  if (e != cudaSuccess) return cuda_err(e);
  int64_t *ek = reinterpret_cast<int64_t *>(tmp);
  int64_t *ev = reinterpret_cast<int64_t *>(tmp + al(8 * tn));
  uint64_t *ck = reinterpret_cast<uint64_t *>(tmp + 2 * al(8 * tn));
  export_contents(t, ek, ev, s);
  if (n1 > 0) transform_keys_in(ek, ck, n1, s);
  rc = rebuild_from_sorted(t, ck, ev, n1, s);
  release_after(tmp, s);
  return rc;
}

}  // namespace hm
