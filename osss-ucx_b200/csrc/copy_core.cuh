/*
 * copy_core.cuh -- byte copies at any alignment, 16 bytes at a time.
 *
 * The copies of the collectives are bound by memory bandwidth as long as
 * they move whole aligned vectors; byte or word loops are bound by the
 * load/store unit (a warp's byte loop moves 32 bytes per instruction).  So
 * a copy whose source is shifted against its dest still writes aligned
 * 16-byte vectors, each cut out of the two aligned source vectors that hold
 * its bytes.  The second of the two is the first of the next lane's, so it
 * is read from L1; a vector is loaded only when it holds at least one byte
 * of the source, so no access leaves the arena (slices are 16-byte
 * aligned), and bytes of it that are not the source's are dropped.
 */
#pragma once
#include <stdint.h>

namespace b200 {
namespace {

/* 16 bytes from byte sh (0..15) of the 32 bytes lo, hi */
__device__ __forceinline__ uint4 cut16(uint4 lo, uint4 hi, unsigned sh) {
  const bool two = sh & 8, one = sh & 4;
  const unsigned a0 = two ? lo.z : lo.x, a1 = two ? lo.w : lo.y, a2 = two ? hi.x : lo.z,
                 a3 = two ? hi.y : lo.w, a4 = two ? hi.z : hi.x, a5 = two ? hi.w : hi.y;
  const unsigned c0 = one ? a1 : a0, c1 = one ? a2 : a1, c2 = one ? a3 : a2, c3 = one ? a4 : a3,
                 c4 = one ? a5 : a4;
  const unsigned b = (sh & 3) * 8;
  return make_uint4(__funnelshift_r(c0, c1, b), __funnelshift_r(c1, c2, b),
                    __funnelshift_r(c2, c3, b), __funnelshift_r(c3, c4, b));
}

/* the first n1 bytes (0..16) of a, the rest of b */
__device__ __forceinline__ uint4 join16(uint4 a, uint4 b, int n1) {
  auto word = [&](unsigned x, unsigned y, int n) {
    const unsigned m = n >= 4 ? 0xffffffffu : n <= 0 ? 0u : (1u << (8 * n)) - 1u;
    return (x & m) | (y & ~m);
  };
  return make_uint4(word(a.x, b.x, n1), word(a.y, b.y, n1 - 4), word(a.z, b.z, n1 - 8),
                    word(a.w, b.w, n1 - 12));
}

/* nv whole vectors to the 16-byte aligned d from s at any alignment, by
 * threads tid of nthr; U vectors in flight per thread.  Plain loads: the
 * serving loop's sources may have been written by an earlier request of the
 * same kernel. */
template <int U>
__device__ __forceinline__ void vectors_copy(char *d, const char *s, uint64_t nv, int tid,
                                             int nthr) {
  const unsigned sh = (unsigned)(uintptr_t)s & 15u;
  const uint4 *p = (const uint4 *)(s - sh);
  uint4 *q = (uint4 *)d;
  const uint64_t st = (uint64_t)nthr;
  uint64_t i = (uint64_t)tid;
  if (sh == 0) {
    for (; i + (2 * U - 1) * st < nv; i += 2 * U * st) {
      uint4 x[2 * U];
#pragma unroll
      for (int u = 0; u < 2 * U; u++) x[u] = p[i + u * st];
#pragma unroll
      for (int u = 0; u < 2 * U; u++) q[i + u * st] = x[u];
    }
    for (; i < nv; i += st) q[i] = p[i];
    return;
  }
  for (; i + (U - 1) * st < nv; i += U * st) {
    uint4 x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      x[u] = p[i + u * st];
      y[u] = p[i + u * st + 1];
    }
#pragma unroll
    for (int u = 0; u < U; u++) q[i + u * st] = cut16(x[u], y[u], sh);
  }
  for (; i < nv; i += st) q[i] = cut16(p[i], p[i + 1], sh);
}

}  // namespace
}  // namespace b200
