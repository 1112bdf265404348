// Primitives of the narrowed-thread-group descent, shared by the point search
// (search.cu) and the range locate (misc.cu): loads with an L2 policy, the
// count of keys <= q by a group of W lanes, and the staging of the top levels
// in shared memory.
#pragma once

#include "async_copy.cuh"
#include "hm_internal.cuh"

namespace hm {

// L2 cache policies (createpolicy): inner rows are re-read by every query and
// should stay in L2; leaf rows are touched about once per batch.
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// 16-B read-only global load with an L2 cache policy.
__device__ __forceinline__ longlong2 ldg2(const int64_t *p, uint64_t pol) {
  longlong2 r;
  asm volatile("ld.global.nc.L2::cache_hint.v2.s64 {%0, %1}, [%2], %3;"
               : "=l"(r.x), "=l"(r.y)
               : "l"(p), "l"(pol));
  return r;
}
// 32-B read-only global load with an L2 cache policy; p 32-byte aligned.
struct Quad {
  int64_t x[4];
};
__device__ __forceinline__ Quad ldg4(const int64_t *p, uint64_t pol) {
  Quad r;
  asm volatile("ld.global.nc.L2::cache_hint.v4.b64 {%0, %1, %2, %3}, [%4], %5;"
               : "=l"(r.x[0]), "=l"(r.x[1]), "=l"(r.x[2]), "=l"(r.x[3])
               : "l"(p), "l"(pol));
  return r;
}
__device__ __forceinline__ int64_t ldg1(const int64_t *p, uint64_t pol) {
  int64_t r;
  asm volatile("ld.global.nc.L2::cache_hint.s64 %0, [%1], %2;" : "=l"(r) : "l"(p), "l"(pol));
  return r;
}
__device__ __forceinline__ int32_t ldg1(const int32_t *p, uint64_t pol) {
  int32_t r;
  asm volatile("ld.global.nc.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(r) : "l"(p), "l"(pol));
  return r;
}

template <bool SMEM>
__device__ __forceinline__ longlong2 load2(const int64_t *p, uint64_t pol) {
  if constexpr (SMEM) {
    return *reinterpret_cast<const longlong2 *>(p);
  } else {
    return ldg2(p, pol);
  }
}

// Sum over the W lanes of an aligned group.
template <int W>
__device__ __forceinline__ int group_sum(int v) {
#pragma unroll
  for (int o = W / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Number of keys <= q among LEN sorted keys at p, counted by the W lanes of a
// group (lane `sub` reads vectors sub, sub+W, ...).
template <int W, int LEN, bool SMEM>
__device__ __forceinline__ int count_le(const int64_t *p, int64_t q, int sub, uint64_t pol) {
  if constexpr (!SMEM && LEN % (4 * W) == 0) {  // rows are 32-byte aligned; half the requests of 16-B loads
    constexpr int N = LEN / (4 * W);
    Quad v[N];
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = ldg4(p + 4 * (sub + i * W), pol);
    int c = 0;
#pragma unroll
    for (int i = 0; i < N; i++) c += (v[i].x[0] <= q) + (v[i].x[1] <= q) + (v[i].x[2] <= q) + (v[i].x[3] <= q);
    return group_sum<W>(c);
  }
  constexpr int NV = LEN / 2;
  constexpr int VPL = (NV + W - 1) / W;
  longlong2 v[VPL];
#pragma unroll
  for (int i = 0; i < VPL; i++) {
    int vi = sub + i * W;
    if (NV % W == 0 || vi < NV)
      v[i] = load2<SMEM>(p + 2 * vi, pol);
    else
      v[i] = make_longlong2(kMaxKey, kMaxKey);
  }
  int c = 0;
#pragma unroll
  for (int i = 0; i < VPL; i++) c += (v[i].x <= q) + (v[i].y <= q);
  return group_sum<W>(c);
}

// Child position in an inner row: index stage then slice stage.
template <int W, int F, bool SMEM>
__device__ __forceinline__ int rank_inner(const int64_t *row, int64_t q, int sub, uint64_t pol) {
  int k = count_le<W, F / 8, SMEM>(row, q, sub, pol);
  k = min(k, F / 8 - 1);
  return 8 * k + count_le<W, 8, SMEM>(row + F / 8 + 8 * k, q, sub, pol);
}

// The top levels in a CTA's shared memory: smem_nodes rows, then their
// first-child ids, then the mbarrier of their copy.
template <int F>
__device__ __forceinline__ int32_t *top_prefix(const DevTree &t, unsigned char *smem) {
  return reinterpret_cast<int32_t *>(smem + (unsigned)t.smem_nodes * (F / 8 + F) * 8u);
}

// Bulk-copies them (all threads); false if the bounded wait gave up, which it
// records in *err.
template <int F>
__device__ __forceinline__ bool stage_top(const DevTree &t, unsigned char *smem, unsigned *err) {
  if (t.smem_nodes <= 0) return true;
  const unsigned rows_bytes = (unsigned)t.smem_nodes * (F / 8 + F) * 8u;
  const unsigned pref_bytes = ((unsigned)t.smem_nodes * 4u + 15u) & ~15u;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + rows_bytes + pref_bytes);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
    mbar_expect_tx(bar, rows_bytes + pref_bytes);
    bulk_g2s(smem_addr(smem), t.inner, rows_bytes, bar);
    bulk_g2s(smem_addr(smem + rows_bytes), t.prefix, pref_bytes, bar);
  }
  __syncthreads();
  if (mbar_wait_bounded(bar, 0, t.wait_polls)) return true;
  if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
  mbar_wait_bounded(bar);  // let the copy land (default bound) before the CTA exits
  return false;
}

// Leaf whose key range holds q (the same in all W lanes; q < Max_Key).
template <int W, int F>
__device__ __forceinline__ int32_t descend_group(const DevTree &t, const int64_t *srows, const int32_t *spref,
                                                 int64_t q, int sub, uint64_t pol) {
  constexpr int ROW = F / 8 + F;
  int32_t node = 0;
  for (int lvl = 0; lvl < t.height; lvl++) {
    if (lvl < t.smem_levels) {
      node = spref[node] + rank_inner<W, F, true>(srows + (int64_t)node * ROW, q, sub, pol);
    } else {
      const int32_t first = ldg1(t.prefix + node, pol);
      node = first + rank_inner<W, F, false>(t.inner + (int64_t)node * ROW, q, sub, pol);
    }
  }
  return node - t.n_inner;
}

}  // namespace hm
