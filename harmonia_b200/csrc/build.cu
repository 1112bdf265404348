// GPU bulk loader: sorted (key, value) pairs -> leaves, then inner levels
// bottom-up with the breadth-first prefix-sum child array.
//
// The reference builds its tree by serial inserts and re-lays it out on the
// CPU (BPlusTree::insert + BPlusTree::sort + prepareArray,
// open-harmonia/src/bpt.cpp:357-409, open-harmonia/src/traversal.cpp:35-195),
// about four minutes at 2^26 keys.  Here every level is one kernel over
// (node, word) pairs: each thread computes one output word directly from the
// level below.  The leaves come straight out of the bucket sort
// (bucket_sort.cuh) that brings the pairs into key order: 2^24 pairs load in
// 0.55 ms, against 2.70 with an eight-pass LSD sort in front of a leaf kernel
// (which a rebuild from sorted contents, and keys that crowd a bucket, still
// take).  Keys are spread evenly: with m items over p parts, part j starts at
// j*(m/p) + min(j, m%p) (part_start), at the leaf level and at every inner
// level.
#include "bucket_sort.cuh"

namespace hm {

namespace {

constexpr int kThreads = 256;

unsigned blocks_for(int64_t items) {
  int64_t b = (items + kThreads - 1) / kThreads;
  return (unsigned)(b < 1 ? 1 : b);
}

__global__ void transform_in_kernel(const int64_t *__restrict__ keys, uint64_t *__restrict__ u,
                                    int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    u[i] = (uint64_t)keys[i] ^ kSign;
}

// flags bit0: duplicate key, bit1: key == Max_Key.
__global__ void check_sorted_kernel(const uint64_t *__restrict__ u, int64_t n, unsigned *flags) {
  unsigned f = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t k = u[i];
    if (i > 0 && u[i - 1] == k) f |= 1u;
    if ((int64_t)(k ^ kSign) == kMaxKey) f |= 2u;
  }
  if (f) atomicOr(flags, f);
}

// One thread per (leaf, word) of the leaf rows: index words, keys, values.
__global__ void leaf_kernel(const uint64_t *__restrict__ u, const int64_t *__restrict__ vals,
                            int64_t n, int64_t n_leaf, int lc, int li,
                            int64_t *__restrict__ leaf_rows, int32_t *__restrict__ leaf_cnt,
                            int64_t *__restrict__ leaf_base, int64_t *__restrict__ submin) {
  const int row = li + 2 * lc;
  const int64_t total = n_leaf * (int64_t)row;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int64_t j = t / row;
    int w = (int)(t - j * row);
    int64_t s = part_start(j, n, n_leaf), e = part_start(j + 1, n, n_leaf);
    if (w >= li + lc) {  // value word
      int slot = w - li - lc;
      leaf_rows[t] = (s + slot < e) ? vals[s + slot] : (int64_t)HM_NOT_FOUND;
      continue;
    }
    int slot = w < li ? 8 * (w + 1) : w - li;  // index word w mirrors key slot 8(w+1)
    int64_t k = kMaxKey;
    if (slot < lc && s + slot < e) k = (int64_t)(u[s + slot] ^ kSign);
    leaf_rows[t] = k;
    if (w >= li) {
      if (slot == 0) {
        leaf_cnt[j] = (int32_t)(e - s);
        leaf_base[j] = s;
        submin[j] = (s < e) ? (int64_t)(u[s] ^ kSign) : kMaxKey;
      }
    }
  }
}

// Last step of the bulk loader's bucket sort: a CTA sorts one bucket in shared
// memory and writes its records straight to their leaf rows.  A record's rank
// in the whole load is the bucket's start plus its place in the bucket, which
// gives its leaf and slot; the thread with a leaf's first record writes the
// leaf's count, base and subtree minimum, the one with its last record the
// padding.  start == nullptr: all n pairs are one bucket.  Bound by issue
// slots (74 % of the cycles issue) and shared-memory accesses (71 % of the L1
// data pipe's peak): 212 us at 2^24 pairs, against 82 us for their bytes at the
// measured copy rate; the separate last sort passes, check and leaf kernel
// it stands for took 430.
__global__ void __launch_bounds__(bsort::kSortThreads, 5) leaf_sort_kernel(
    const int64_t *__restrict__ keys, const int64_t *__restrict__ vals, const uint32_t *__restrict__ start, uint32_t n,
    uint32_t n_leaf, int lc, int li, int64_t *__restrict__ leaf_rows, int32_t *__restrict__ leaf_cnt,
    int64_t *__restrict__ leaf_base, int64_t *__restrict__ submin, bsort::Ctl *ctl) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char dyn[];
  auto &sm = *reinterpret_cast<bsort::SortSmem<int64_t> *>(dyn);
  if (ctl->skew) return;
  const uint32_t s0 = start ? start[blockIdx.x] : 0;
  const int m = (int)((start ? start[blockIdx.x + 1] : n) - s0);
  if (m == 0) return;
  // the first rem leaves hold q + 1 records, the others q
  const uint32_t q = n / n_leaf, rem = n % n_leaf, big = rem * (q + 1);
  // leaf and slot of the bucket's first record; inside the bucket a 32-bit
  // reciprocal divides (exact below 2^16), unless its leaves are of both sizes
  const bool in_big = s0 < big, mixed = in_big && s0 + m > big;
  const uint32_t len0 = in_big ? q + 1 : q, x0 = in_big ? s0 : s0 - big;
  const uint32_t sl0 = x0 % len0, j0 = (in_big ? 0 : rem) + x0 / len0;
  const uint32_t inv = len0 > 1 ? 0xffffffffu / len0 + 1 : 0;
  const int row = li + 2 * lc;
  unsigned f = 0;
  const bsort::Map map = ctl->map;
  bsort::sort_bucket<int64_t, false>(sm, map, keys + s0, vals + s0, m, [&](int i, int64_t k, int64_t v, bool twin) {
    uint32_t j, len = len0;
    int sl;
    if (!mixed) {
      const uint32_t x = sl0 + i, dj = inv ? __umulhi(x, inv) : x;
      sl = (int)(x - dj * len);
      j = j0 + dj;
    } else {
      const uint32_t r = s0 + i, first = r < big ? 0 : big;
      len = r < big ? q + 1 : q;
      sl = (int)((r - first) % len);
      j = (r < big ? 0 : rem) + (r - first) / len;
    }
    int64_t *lr = leaf_rows + (int64_t)j * row + li;
    lr[sl] = k;
    lr[lc + sl] = v;
    if (sl == 0) {
      leaf_cnt[j] = (int32_t)len;
      leaf_base[j] = s0 + i;
      submin[j] = k;
    } else if (li > 0 && (sl & 7) == 0) {
      lr[sl / 8 - 1 - li] = k;  // index word w mirrors key slot 8(w+1)
    }
    if ((int)len < lc && sl == (int)len - 1) {
      for (int p = (int)len; p < lc; p++) {
        lr[p] = kMaxKey;
        lr[lc + p] = HM_NOT_FOUND;
      }
    }
    if (li > 0 && sl == (int)len - 1)
      for (int w = (int)(len - 1) / 8; w < li; w++) lr[w - li] = kMaxKey;
    if (twin) f |= 1u;
    if (i == 0 || i == m - 1) {
      if (k == kMaxKey) f |= 2u;  // sorts last
      if (s0 + i == 0) ctl->ends[0] = k;
      if (s0 + i == n - 1) ctl->ends[1] = k;
    }
  });
  if (f) atomicOr(&ctl->flags, f);
}

// One thread per (node, word) of one inner level.  m = nodes of the level
// below, whose subtree minima are in submin_below; child_base = BFS id of the
// level below's first node (n_inner for leaves).
__global__ void inner_kernel(int64_t nodes, int64_t m, int f, int64_t lvl_base,
                             int64_t child_base, const int64_t *__restrict__ submin_below,
                             int64_t *__restrict__ inner, int32_t *__restrict__ prefix,
                             int64_t *__restrict__ submin_here) {
  pdl_enter();
  const int ix = f / 8, row = ix + f;
  const int64_t total = nodes * (int64_t)row;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    int64_t i = t / row;
    int w = (int)(t - i * row);
    int64_t c0 = part_start(i, m, nodes), c1 = part_start(i + 1, m, nodes);
    int slot = w < ix ? 8 * (w + 1) : w - ix;
    // separator `slot` = minimum key of child slot+1
    int64_t c = c0 + 1 + slot;
    int64_t k = (slot < f && c < c1) ? submin_below[c] : kMaxKey;
    inner[(lvl_base + i) * row + w] = k;
    if (w == ix) {
      prefix[lvl_base + i] = (int32_t)(child_base + c0);
      submin_here[i] = submin_below[c0];
    }
  }
}

}  // namespace

int shape(int64_t n, const hm_config &c, int *height, int64_t *lvl_start, int64_t *n_inner,
          int64_t *n_leaf) {
  if (n < 0) return HM_EINVAL;
  int64_t nl = n == 0 ? 1 : (n + c.leaf_fill - 1) / c.leaf_fill;
  int64_t sizes[kMaxLevels];
  int h = 0;
  int64_t m = nl;
  do {
    if (h >= kMaxLevels) return HM_ETOOLARGE;
    int64_t nodes = (m + c.inner_fill - 1) / c.inner_fill;
    sizes[h++] = nodes;
    m = nodes;
  } while (m > 1);
  int64_t acc = 0;
  for (int l = 0; l < h; l++) {
    lvl_start[l] = acc;
    acc += sizes[h - 1 - l];
  }
  lvl_start[h] = acc;
  if (acc > INT32_MAX / 2 || nl > INT32_MAX / 2) return HM_ETOOLARGE;
  *height = h;
  *n_inner = acc;
  *n_leaf = nl;
  return HM_OK;
}

void transform_keys_in(const int64_t *keys, uint64_t *ukeys, int64_t n, cudaStream_t s) {
  if (n <= 0) return;
  transform_in_kernel<<<min(blocks_for(n), 148u * 16), kThreads, 0, s>>>(keys, ukeys, n);
  note_launch();
}

void check_sorted_keys(const uint64_t *ukeys, int64_t n, unsigned *d_flags, cudaStream_t s) {
  if (n <= 0) return;
  check_sorted_kernel<<<min(blocks_for(n), 148u * 16), kThreads, 0, s>>>(ukeys, n, d_flags);
  note_launch();
}

int build_inner(const BuildTarget &b, int64_t *submin, int64_t *tmp, cudaStream_t s);

int build_from_sorted(const BuildTarget &b, const uint64_t *ukeys, const int64_t *vals, int64_t n,
                      int64_t *tmp_a, int64_t *tmp_b, cudaStream_t s) {
  const BuildTarget *t = &b;
  const int lc = t->leaf_cap;
  int64_t leaf_words = t->n_leaf * (int64_t)t->leaf_row;
  leaf_kernel<<<min(blocks_for(leaf_words), 148u * 32), kThreads, 0, s>>>(
      ukeys, vals, n, t->n_leaf, lc, t->leaf_index, t->leaf_rows, t->leaf_cnt, t->leaf_base, tmp_a);
  note_launch();
  return build_inner(b, tmp_a, tmp_b, s);
}

// The inner levels bottom-up; submin holds each leaf's smallest key, tmp is
// as large.
int build_inner(const BuildTarget &b, int64_t *submin, int64_t *tmp, cudaStream_t s) {
  const BuildTarget *t = &b;
  const int f = t->fanout;
  int64_t *below = submin, *here = tmp;
  int64_t m = t->n_leaf;
  for (int l = t->height - 1; l >= 0; l--) {
    int64_t nodes = t->lvl_start[l + 1] - t->lvl_start[l];
    int64_t words = nodes * (int64_t)t->inner_row;
    launch_pdl(inner_kernel, min(blocks_for(words), 148u * 32), kThreads, 0, s, nodes, m, f, t->lvl_start[l],
               t->lvl_start[l + 1], below, t->inner, t->prefix, here);
    note_launch();
    std::swap(below, here);
    m = nodes;
  }
  return cuda_err(cudaGetLastError());
}

size_t build_work_bytes(int64_t n, int64_t n_leaf) {
  size_t bytes = (size_t)align_up((int64_t)bsort::work_bytes(n), 256);
  if (bsort::shape_for(n).passes() == 1) bytes += 2 * 8 * (size_t)align_up(n_leaf, 32);
  return bytes;
}

int build_from_pairs(const BuildTarget &b, const int64_t *keys, const int64_t *vals, int64_t n, int64_t *k1,
                     int64_t *v1, int64_t *k2, int64_t *v2, void *work, int sms, bsort::Ctl **ctl, cudaStream_t s) {
  const bsort::Work w = bsort::layout(n, work);
  *ctl = w.ctl;
  const int passes = bsort::partition_pairs<int64_t>(keys, vals, n, k1, v1, k2, v2, w, sms, s);
  const int64_t *pk = passes == 2 ? k2 : passes == 1 ? k1 : keys, *pv = passes == 2 ? v2 : passes == 1 ? v1 : vals;
  // The subtree minima go to the buffers that the partition left free; after one
  // pass those may be the inputs, which the LSD sort still needs on skew (the
  // inner levels are then built from nothing, and again after that sort), so the
  // work area holds them.  A test of skew in inner_kernel instead would add a
  // load to each level's chain (178 K pairs: 65.2 against 64.3 us).
  int64_t *ta = k1, *tb = v1;
  if (passes == 1) {
    ta = reinterpret_cast<int64_t *>(static_cast<char *>(work) + align_up((int64_t)bsort::work_bytes(n), 256));
    tb = ta + align_up(b.n_leaf, 32);
  }
  constexpr int sm = (int)sizeof(bsort::SortSmem<int64_t>);
  opt_in_smem((const void *)leaf_sort_kernel, sm);
  const unsigned grid = 1u << bsort::shape_for(n).bits;
  launch_pdl(leaf_sort_kernel, grid, bsort::kSortThreads, sm, s, pk, pv,
             static_cast<const uint32_t *>(passes ? w.start : nullptr), (uint32_t)n, (uint32_t)b.n_leaf, b.leaf_cap,
             b.leaf_index, b.leaf_rows, b.leaf_cnt, b.leaf_base, ta, w.ctl);
  note_launch();
  return build_inner(b, ta, tb, s);
}

}  // namespace hm
