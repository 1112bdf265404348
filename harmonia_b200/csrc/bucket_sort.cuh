// Bucket sort of (int64 key, payload) pairs: the sort of the bulk loader and
// of large write epochs.
//
// An LSD radix sort reads and writes every pair once per 8 key bits, eight
// times for 64-bit keys.  Here the pairs are partitioned by the leading bits
// of their position in the batch's key range, in one or two passes of at most
// 8 bits each, until a bucket averages at most 1536 pairs, and every bucket is
// then sorted by one CTA in shared memory: three reads and writes of the pairs
// instead of eight and their counts.
//
//   range_kernel    lowest and highest of a sample of the keys; keys outside
//                   go to the end buckets, so the map stays monotone
//   count_kernel    pairs per bucket (16-bit counters in shared memory)
//   starts_kernel   exclusive scan: bucket starts, and the cursors from which
//                   a tile reserves its place
//   scatter_kernel  one partition pass; a tile reserves its run of every digit
//                   with one atomic on the digit's cursor.  That leaves the
//                   order inside a bucket open, which the last step settles,
//                   so no pass needs per-tile counts, their scan or a look-back
//   (caller)        sorts each bucket with sort_bucket() and writes it where
//                   the caller wants it
//
// A batch whose keys crowd a bucket past kCap (strongly clustered keys, one
// key repeated thousands of times) sets Ctl::skew, on which the later kernels
// return without writing; the caller then takes the LSD sort.
#pragma once

#include "async_copy.cuh"
#include "hm_internal.cuh"

namespace hm {
namespace bsort {

constexpr int kCap = 2048;     // pairs a bucket may hold: what one CTA sorts
constexpr int kMean = 1536;    // pairs a bucket averages at most
constexpr int kMaxBits = 16;   // 2^16 16-bit counters are 128 KiB of shared memory
// With few buckets the map's whole factor leaves some of them empty (2 of 2.7:
// 3000 even keys put 2200 into one); with eight the others get an eighth more at
// most.  3000 even keys load in 44 us, 168 by way of the LSD sort.
constexpr int kMinBits = 3;
constexpr int64_t kMaxPairs = (int64_t)kMean << kMaxBits;

// Monotone map of keys to buckets: the offset from lo, shifted up to use all
// 64 bits, times a 32-bit factor (a plain shift would leave up to half of the
// buckets empty where the range is just above a power of two).
struct Map {
  int64_t lo, hi;
  int32_t shl;
  uint32_t mul;
  __device__ __forceinline__ uint32_t top(int64_t k) const {
    const uint64_t off = k <= lo ? 0 : (uint64_t)min(k, hi) - (uint64_t)lo;
    return (uint32_t)((off << shl) >> 32);
  }
  __device__ __forceinline__ uint32_t operator()(int64_t k) const { return __umulhi(top(k), mul); }
  // Where k lies inside its bucket, from 0 to 2^32 - 1.
  __device__ __forceinline__ uint32_t inside(int64_t k) const { return top(k) * mul; }
};

// Factor for nb buckets over a range (hi - lo): the top 32 bits h of the
// shifted offset are at most r, so h * (nb * 2^32 / (r + 1)) / 2^32 < nb.
__host__ __device__ inline void make_map(int64_t lo, int64_t hi, uint32_t nb, Map *m) {
  m->lo = lo;
  m->hi = hi;
  const uint64_t range = (uint64_t)hi - (uint64_t)lo;
  int shl = 0;
#ifdef __CUDA_ARCH__
  shl = range ? __clzll((long long)range) : 63;
#else
  shl = range ? __builtin_clzll(range) : 63;
#endif
  const uint64_t r = (range << shl) >> 32;
  m->shl = shl;
  m->mul = (uint32_t)(((uint64_t)nb << 32) / (r + 1));
}

// Control block in device memory; zero before the first kernel.
struct Ctl {
  unsigned long long inv_lo, hi;  // largest ~k and k of the sample (biased keys)
  unsigned done;                  // CTAs of range_kernel that finished
  unsigned skew;                  // a bucket over kCap: nothing is sorted
  unsigned flags;                 // bit 0: a key twice, bit 1: a key equals Max_Key
  unsigned pad;
  int64_t ends[2];                // lowest and highest key (written by the caller's last step)
  unsigned long long user[4];     // the caller's own results
  Map map;
};

struct Shape {
  int bits = 0, l1 = 0, l2 = 0;  // buckets 2^bits; passes of l1 and l2 bits (l2 == 0: one pass)
  int passes() const { return bits == 0 ? 0 : l2 == 0 ? 1 : 2; }
};

inline bool fits(int64_t n) { return n > 0 && n <= kMaxPairs; }

inline Shape shape_for(int64_t n) {
  Shape s;
  if (n <= kCap) return s;
  s.bits = kMinBits;
  while (s.bits < kMaxBits && (n >> s.bits) >= kMean) s.bits++;
  s.l2 = s.bits > 8 ? s.bits / 2 : 0;
  s.l1 = s.bits - s.l2;
  return s;
}

// Device work area: control block, counts, starts and cursors.
struct Work {
  Ctl *ctl;
  uint32_t *count;  // 2^bits
  uint32_t *start;  // 2^bits + 1
  uint32_t *cur1;   // 2^l1
  uint32_t *cur2;   // 2^bits
};

size_t work_bytes(int64_t n);
Work layout(int64_t n, void *base);

// Partitions n pairs (vals == nullptr: the payload is each key's position)
// into w's buckets: the pairs end in (k2, v2) after two passes, (k1, v1) after
// one, and are left in place (n <= kCap) after none.  Returns the number of
// passes.  Counts its own launches.
template <typename V>
int partition_pairs(const int64_t *keys, const V *vals, int64_t n, int64_t *k1, V *v1, int64_t *k2, V *v2,
                    const Work &w, int sms, cudaStream_t s);

#ifdef __CUDACC__

constexpr int kSortThreads = 256;
constexpr int kSortPer = kCap / kSortThreads;
constexpr int kBins = 2048;  // bins of the counting step inside a bucket
constexpr int kBinBits = 11;
constexpr int kCrowded = 8;  // a bin of more pairs than this: other bins, then the bitonic sort
constexpr int kPad = kCrowded;  // sentinels on either side of the grouped keys

template <typename V>
struct SortSmem {
  alignas(16) int64_t key[kCap + 2 * kPad];  // kPad sentinels, the keys grouped by bin, kPad sentinels
  alignas(16) V val[kCap];
  alignas(16) uint32_t bin[kBins];
  unsigned long long lo[kSortThreads / 32], hi[kSortThreads / 32];
  uint32_t wsum[kSortThreads / 32];
  uint32_t most;  // pairs in the fullest bin
};

// The m <= kCap pairs in shared memory by a bitonic network, equal keys by
// payload (all threads; k and v hold the pairs at their places).
template <typename V>
__device__ __noinline__ void bitonic_sort(int64_t *k, V *v, int m) {
  int p = 1;
  while (p < m) p <<= 1;
  // pairs past m count as larger than all and never move below it
  for (int size = 2; size <= p; size <<= 1) {
    for (int step = size >> 1; step > 0; step >>= 1) {
      for (int x = threadIdx.x; x < p / 2; x += kSortThreads) {
        const int i = 2 * x - (x & (step - 1));  // the pair (i, o) of this step, i < o
        // the first step of a size compares mirrored, so every step puts the smaller first
        const int o = step == size >> 1 ? (i & ~(size - 1)) + size - 1 - (i & (size - 1)) : i + step;
        if (o < m) {
          const int64_t ki = k[i], ko = k[o];
          const V vi = v[i], vo = v[o];
          if (ko < ki || (ko == ki && vo < vi)) {
            k[i] = ko;
            v[i] = vo;
            k[o] = ki;
            v[o] = vi;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Sorts the m <= kCap pairs at (keys, vals) of one bucket by key, equal keys
// by payload (all threads of a kSortThreads CTA), and calls
// emit(rank, key, payload, twin) for each, twin = another pair has its key;
// neighbouring threads emit neighbouring ranks, give or take a few.
//
// The kernel is bound by instructions and shared-memory accesses, not by HBM,
// so it does little per pair: the keys are counted into kBins bins by their
// place in the bucket (about half a pair a bin), grouped by bin, and a pair's
// rank is its grouped position corrected by comparing it with the few
// positions on either side that its bin can reach (one less than the fullest
// bin's pairs).  Keys that crowd those bins are binned over their own lowest
// to highest key instead, and, where that crowds too, sorted by a bitonic
// network.  GEN: payload = position.
template <typename V, bool GEN, typename Emit>
__device__ __forceinline__ void sort_bucket(SortSmem<V> &sm, const Map &map, const int64_t *__restrict__ keys,
                                            const V *__restrict__ vals, int m, Emit emit) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int64_t *const gk = sm.key + kPad;
  int64_t k[kSortPer];
#pragma unroll
  for (int j = 0; j < kSortPer; j++) {
    const int i = j * kSortThreads + tid;
    if (j * kSortThreads >= m) break;
    if (i < m) k[j] = __ldg(keys + i);
  }
  // the payloads go straight to their grouped places once those are known
  constexpr int kLine = 128 / (int)sizeof(V);
  if (!GEN && tid * kLine < m) prefetch_l2(vals + tid * kLine);
  if (tid < kPad) {
    sm.key[tid] = INT64_MIN;
    gk[m + tid] = INT64_MAX;
  }
  unsigned long long lo = 0;
  int shl = 0;
  uint32_t mul = 0;
  for (int attempt = 0;; attempt++) {
    uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int x = 0; x < kBins / 4 / kSortThreads; x++)
      reinterpret_cast<uint4 *>(sm.bin)[x * kSortThreads + tid] = zero;
    if (tid == 0) sm.most = 0;
    __syncthreads();
    uint32_t at[kSortPer], most = 0;
#pragma unroll
    for (int j = 0; j < kSortPer; j++) {
      if (j * kSortThreads >= m) break;
      if (j * kSortThreads + tid < m) {
        uint32_t b;
        if (attempt == 0) {
          b = map.inside(k[j]) >> (32 - kBinBits);
        } else {
          const unsigned long long off = ((unsigned long long)k[j] ^ kSign) - lo;
          b = min(__umulhi((uint32_t)((off << shl) >> 32), mul), (uint32_t)kBins - 1);
        }
        const uint32_t r = atomicAdd(&sm.bin[b], 1u);
        at[j] = b << 16 | r;
        most = max(most, r + 1);
      }
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0 && most > 0) atomicMax(&sm.most, most);
    __syncthreads();
    most = sm.most;
    if (most > kCrowded) {  // uniform across the CTA
      if (attempt == 0) {   // bins over the keys' own range
        unsigned long long hi = 0;
        lo = ~0ull;
#pragma unroll
        for (int j = 0; j < kSortPer; j++) {
          if (j * kSortThreads + tid < m) {
            const unsigned long long u = (unsigned long long)k[j] ^ kSign;
            lo = min(lo, u);
            hi = max(hi, u);
          }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
          hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (lane == 0) {
          sm.lo[warp] = lo;
          sm.hi[warp] = hi;
        }
        __syncthreads();
        for (int w = 0; w < kSortThreads / 32; w++) {
          lo = min(lo, sm.lo[w]);
          hi = max(hi, sm.hi[w]);
        }
        shl = hi > lo ? __clzll((long long)(hi - lo)) : 63;
        // kBins * 2^32 / (top word of the range + 1), a little low so that no bin is past the last
        const uint32_t top = (uint32_t)(((hi - lo) << shl) >> 32);
        mul = (uint32_t)__fdividef(8796093022208.0f * 0.999999f, (float)top + 1.0f);
        continue;
      }
#pragma unroll
      for (int j = 0; j < kSortPer; j++) {
        const int i = j * kSortThreads + tid;
        if (i < m) {
          gk[i] = k[j];
          if constexpr (GEN) {
            sm.val[i] = (V)i;
          } else {
            sm.val[i] = __ldg(vals + i);
          }
        }
      }
      __syncthreads();
      bitonic_sort(gk, sm.val, m);
      for (int i = tid; i < m; i += kSortThreads) {
        const int64_t key = gk[i];
        emit(i, key, sm.val[i], (i > 0 && gk[i - 1] == key) || (i + 1 < m && gk[i + 1] == key));
      }
      return;
    }
    // exclusive scan of the bins, kBins / kSortThreads consecutive ones a thread
    static_assert(kBins == 8 * kSortThreads, "two 16-B words of bins a thread");
    const uint4 c0 = *reinterpret_cast<const uint4 *>(&sm.bin[tid * 8]);
    const uint4 c1 = *reinterpret_cast<const uint4 *>(&sm.bin[tid * 8 + 4]);
    const uint32_t sum = c0.x + c0.y + c0.z + c0.w + c1.x + c1.y + c1.z + c1.w;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) sm.wsum[warp] = incl;
    __syncthreads();
    uint32_t run = incl - sum;
    for (int w = 0; w < warp; w++) run += sm.wsum[w];
    uint4 r0, r1;
    r0.x = run;
    r0.y = r0.x + c0.x;
    r0.z = r0.y + c0.y;
    r0.w = r0.z + c0.z;
    r1.x = r0.w + c0.w;
    r1.y = r1.x + c1.x;
    r1.z = r1.y + c1.y;
    r1.w = r1.z + c1.z;
    *reinterpret_cast<uint4 *>(&sm.bin[tid * 8]) = r0;
    *reinterpret_cast<uint4 *>(&sm.bin[tid * 8 + 4]) = r1;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortPer; j++) {
      if (j * kSortThreads >= m) break;
      if (j * kSortThreads + tid < m) {
        const uint32_t p = sm.bin[at[j] >> 16] + (at[j] & 0xffffu);
        const int i = j * kSortThreads + tid;
        if constexpr (GEN) {
          sm.val[p] = (V)i;
        } else {
          cp_async_element(sm.val + p, vals + i);
        }
        gk[p] = k[j];
      }
    }
    if constexpr (!GEN) cp_async_wait();
    __syncthreads();
    for (int p = tid; p < m; p += kSortThreads) {
      const int64_t key = gk[p];
      int r = p;
      bool twin = false;
      for (int d = 1; d < (int)most; d++) {
        const int64_t before = gk[p - d], after = gk[p + d];
        r += (after < key) - (before > key);
        twin |= before == key || after == key;
      }
      const V val = sm.val[p];
      if (twin) {  // or a sentinel's value
        twin = false;
        for (int d = 1; d < (int)most; d++) {
          if (p - d >= 0 && gk[p - d] == key) {
            twin = true;
            r -= sm.val[p - d] > val;
          }
          if (p + d < m && gk[p + d] == key) {
            twin = true;
            r += sm.val[p + d] < val;
          }
        }
      }
      emit(r, key, val, twin);
    }
    return;
  }
}

#endif  // __CUDACC__

}  // namespace bsort
}  // namespace hm
