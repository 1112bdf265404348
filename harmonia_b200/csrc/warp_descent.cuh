// Descent of a warp's 32 keys that are in key order, shared by the write epochs
// (upsert.cu) and the bucket boundaries of the join (join.cu).
#pragma once

#include "hm_internal.cuh"

namespace hm {

// Keys <= q in a node of 64 sorted keys of which lane l holds 2l and 2l + 1.
__device__ __forceinline__ int warp_rank(longlong2 p, int64_t q) {
  int pos = 0;  // lanes whose first key is <= q
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (__shfl_sync(0xffffffffu, p.x, pos + step - 1) <= q) pos += step;
  if (__shfl_sync(0xffffffffu, p.x, pos) <= q) pos++;  // pos <= 31 here
  const int64_t y = __shfl_sync(0xffffffffu, p.y, max(pos - 1, 0));
  return pos == 0 ? 0 : 2 * pos - 1 + (y <= q);
}

// Leaf of each of a warp's 32 keys, which are in key order.  While the lowest
// and the highest key go to the same child the warp descends as one, with one
// dependent load a level: a lane holds two of the node's keys, and ballots
// count those <= a key.  Where they part, every lane ranks its key among the
// keys the warp holds.  Below that two neighbouring nodes are still searched
// that way; only keys that spread further search alone (two loads a level).
__device__ __forceinline__ int32_t descend_leaf_warp(const DevTree &t, int f, int64_t q) {
  const int ix = f / 8, row = ix + f, lane = threadIdx.x & 31;
  const int64_t q0 = __shfl_sync(0xffffffffu, q, 0), q1 = __shfl_sync(0xffffffffu, q, 31);
  int32_t node = 0;  // the warp's, then the lane's
  int l = 0;
  for (; l < t.height; l++) {
    const int64_t *r = t.inner + (int64_t)node * row + ix;
    const int32_t first = __ldg(t.prefix + node);
    const longlong2 p = __ldg(reinterpret_cast<const longlong2 *>(r + 2 * lane));
    longlong2 p2 = make_longlong2(kMaxKey, kMaxKey);
    if (f > 64) p2 = __ldg(reinterpret_cast<const longlong2 *>(r + 64 + 2 * lane));
    int c0 = __popc(__ballot_sync(0xffffffffu, p.x <= q0)) + __popc(__ballot_sync(0xffffffffu, p.y <= q0));
    int c1 = __popc(__ballot_sync(0xffffffffu, p.x <= q1)) + __popc(__ballot_sync(0xffffffffu, p.y <= q1));
    if (f > 64) {
      c0 += __popc(__ballot_sync(0xffffffffu, p2.x <= q0)) + __popc(__ballot_sync(0xffffffffu, p2.y <= q0));
      c1 += __popc(__ballot_sync(0xffffffffu, p2.x <= q1)) + __popc(__ballot_sync(0xffffffffu, p2.y <= q1));
    }
    if (c0 == c1) {
      node = first + c0;
      continue;
    }
    node = first + warp_rank(p, q);
    if (f > 64) node += warp_rank(p2, q);
    l++;
    break;
  }
  for (; l < t.height; l++) {
    const int32_t n0 = __shfl_sync(0xffffffffu, node, 0), n1 = __shfl_sync(0xffffffffu, node, 31);
    if (n1 - n0 <= 1) {
      const int64_t *ra = t.inner + (int64_t)n0 * row + ix, *rb = t.inner + (int64_t)n1 * row + ix;
      const longlong2 pa = __ldg(reinterpret_cast<const longlong2 *>(ra + 2 * lane));
      const longlong2 pb = __ldg(reinterpret_cast<const longlong2 *>(rb + 2 * lane));
      const int32_t first = __ldg(t.prefix + node);
      const int ca = warp_rank(pa, q), cb = warp_rank(pb, q);
      int c = node == n0 ? ca : cb;
      if (f > 64) {
        const longlong2 pa2 = __ldg(reinterpret_cast<const longlong2 *>(ra + 64 + 2 * lane));
        const longlong2 pb2 = __ldg(reinterpret_cast<const longlong2 *>(rb + 64 + 2 * lane));
        const int ca2 = warp_rank(pa2, q), cb2 = warp_rank(pb2, q);
        c += node == n0 ? ca2 : cb2;
      }
      node = first + c;
      continue;
    }
    const int64_t *r = t.inner + (int64_t)node * row;
    const int32_t first = __ldg(t.prefix + node);
    int k = 0;
    for (int v = 0; v < ix / 2; v++) {
      const longlong2 p = __ldg(reinterpret_cast<const longlong2 *>(r + 2 * v));
      k += (p.x <= q) + (p.y <= q);
    }
    k = min(k, ix - 1);
    int c = 8 * k;
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const longlong2 p = __ldg(reinterpret_cast<const longlong2 *>(r + ix + 8 * k + 2 * v));
      c += (p.x <= q) + (p.y <= q);
    }
    node = first + c;
  }
  return node - t.n_inner;
}

}  // namespace hm
