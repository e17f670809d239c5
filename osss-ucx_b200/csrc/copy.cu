/*
 * copy.cu -- the data-movement collectives: fcollect, collect, alltoall,
 * strided alltoall and broadcast.
 *
 * In the reference every byte crosses a process boundary as a UCX put
 * (fcollect: log2(P) Bruck rounds plus an in-place byte rotation,
 * src/shcoll/src/fcollect.c:370-403 and util/rotate.c:22-54; alltoall:
 * P-1 puts per PE, alltoall.c:75-110; strided alltoall: one put per
 * element, alltoalls.c:54-90).  The result of each is a fixed permutation
 * of bytes that does not depend on the algorithm, so here each collective
 * is one copy kernel that moves every byte once from its source slice to
 * its final place: no rounds, no intermediate copies, no rotation.
 *
 * fcollect, collect, broadcast and alltoall write each dest row as the
 * aligned 16-byte vectors it spans, whatever the offsets and block sizes:
 * a vector is cut out of the source blocks that meet in it (copy_core.cuh),
 * and only the two vectors at the row's ends are written in bytes.  The
 * strided form copies elements.
 */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "copy_core.cuh"
#include "internal.cuh"

namespace b200 {
namespace {

__device__ __forceinline__ uint4 ld16(const char *p) {
  uint4 u;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
      : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
      : "l"(p));
  return u;
}
/* a vector the next lane reads too */
__device__ __forceinline__ uint4 ld16l1(const char *p) {
  uint4 u;
  asm("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];"
      : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
      : "l"(p));
  return u;
}
__device__ __forceinline__ void st16(char *p, uint4 u) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(u.x), "r"(u.y), "r"(u.z),
               "r"(u.w)
               : "memory");
}

/* streaming store (evict-first in L2): for data this kernel does not read
 * again, such as fcollect's P copies of each source vector */
__device__ __forceinline__ void st16cs(char *p, uint4 u) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(u.x), "r"(u.y), "r"(u.z),
               "r"(u.w)
               : "memory");
}

/* The bytes [i0, i1) of a vector, 16 bytes at virtual address s of which the
 * first n1 bytes (and none below i0) come from there, the others from c on,
 * counted from the vector's byte 0 too.  All loads are issued together. */
__device__ __forceinline__ uint4 meet16(const char *s, const char *c, int i0, int n1, int i1) {
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 lo = zero, hi = zero, clo = zero, chi = zero;
  const int sh = (int)((uintptr_t)s & 15), csh = (int)((uintptr_t)c & 15);
  if (sh + i0 < 16) lo = ld16l1(s - sh);
  if (sh + n1 > 16) hi = ld16l1(s - sh + 16);
  if (n1 < i1) {
    if (csh + n1 < 16) clo = ld16l1(c - csh);
    if (csh + i1 > 16) chi = ld16l1(c - csh + 16);
  }
  return join16(cut16(lo, hi, sh), cut16(clo, chi, csh), n1);
}

/* What a dest row concatenates: P blocks, block k read at src0 + k*step. */
struct Even { /* of B bytes each */
  uint64_t B;
  __device__ __forceinline__ int find(uint64_t x, int, uint64_t *b) const {
    if ((x | B) >> 32 == 0) { /* half the instructions */
      const unsigned k = (unsigned)x / (unsigned)B;
      *b = (unsigned)x - k * (unsigned)B;
      return (int)k;
    }
    const uint64_t k = x / B;
    *b = x - k * B;
    return (int)k;
  }
  __device__ __forceinline__ uint64_t size(int) const { return B; }
};
struct Whole { /* one block, the row */
  uint64_t len;
  __device__ __forceinline__ int find(uint64_t x, int, uint64_t *b) const {
    *b = x;
    return 0;
  }
  __device__ __forceinline__ uint64_t size(int) const { return len; }
};
/* of uneven sizes: pre[k] = the row position of block k, pre[P] = the row's
 * length.  The table is the kernel's parameter (N entries at most), read
 * through the constant cache; N = 0: a table in device memory. */
template <int N>
struct Uneven {
  uint64_t pre[N];
};
template <>
struct Uneven<0> {
  const uint64_t *pre;
};
template <int N>
struct Table {
  const Uneven<N> &t;
  /* the last k with pre[k] <= x: x is below the row's length, so that
   * block is not empty */
  __device__ __forceinline__ int find(uint64_t x, int P, uint64_t *b) const {
    int lo = 0, hi = P;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (t.pre[mid] <= x)
        lo = mid;
      else
        hi = mid;
    }
    *b = x - t.pre[lo];
    return lo;
  }
  __device__ __forceinline__ uint64_t size(int k) const { return t.pre[k + 1] - t.pre[k]; }
};
__device__ __forceinline__ Even blocks(const Even &e) { return e; }
__device__ __forceinline__ Whole blocks(const Whole &w) { return w; }
template <int N>
__device__ __forceinline__ Table<N> blocks(const Uneven<N> &t) {
  return Table<N>{t};
}

/* The copy of a row of len bytes, nblk blocks, from src0 on to P members'
 * dests from dst0 on, mpc members a CTA, all but `skip`.  Padded to 32 bytes
 * past a multiple of 64: a launch takes the host least with so many bytes of
 * parameters (an empty kernel: 2.05 us at 32, 96, 160, 224, 288 or 1120 bytes, 2.4
 * within 8 of these, 2.7 elsewhere; fcollect of 8 x 128 bytes, a call from
 * Python: 3.9 us with 72 bytes, 3.2 with 96). */
template <class BLK>
struct Row {
  const char *src0;
  char *dst0;
  uint64_t step, len;
  int P, nblk, mpc, skip;
  BLK prm;
  char pad[(32 + 64 - (48 + sizeof(BLK)) % 64) % 64];
};
static_assert(sizeof(Row<Even>) % 64 == 32 && sizeof(Row<Uneven<136>>) % 64 == 32, "see above");

/* fcollect, collect and broadcast: every member's dest row is the same
 * `len` bytes, the blocks one after the other (fcollect.c:370-403,
 * collect.c:35-591).  One thread per 16-byte vector of the row: it puts the
 * vector together once and writes it into the members of its blockIdx.y
 * (all but `skip`).  Bound by the writes, P per vector read; streaming
 * stores, since this kernel does not read them again.  In a graph, 128
 * members x 32 KiB: 88.3 us with one pass per source member and six CTAs an
 * SM, 76.2 now (91.8 and 82.4 a call in a row); x 32764 bytes, then 4-byte
 * words: 278 -> 76.6; a collect of 64 members x 32 KiB on average, a call in a
 * row, 4-byte words and an uploaded table: 45.5 -> 24.5. */
template <class BLK>
__global__ void __launch_bounds__(256, 6) k_spread(const __grid_constant__ Row<BLK> r) {
  const auto blk = blocks(r.prm);
  const char *const src0 = r.src0;
  char *const dst0 = r.dst0;
  const uint64_t step = r.step, len = r.len;
  const int P = r.P, nblk = r.nblk, mpc = r.mpc, skip = r.skip;
  const int a = (int)((uintptr_t)dst0 & 15); /* the row begins at byte a of vector 0 */
  const int64_t x0 = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 16 - a;
  const int i0 = x0 < 0 ? a : 0;
  const int i1 = (int64_t)len - x0 < 16 ? (int)((int64_t)len - x0) : 16;
  const int j0 = blockIdx.y * mpc, j1 = j0 + mpc < P ? j0 + mpc : P;
  uint4 u = make_uint4(0, 0, 0, 0);
  uint64_t left = 0;
  const char *s = nullptr;
  int k = 0;
  if (i1 > i0) {
    uint64_t b;
    k = blk.find((uint64_t)(x0 + i0), nblk, &b);
    left = blk.size(k) - b;
    s = src0 + (uint64_t)k * step + b;
  }
  /* one way for the whole warp, so that its loads are issued together */
  const bool inside = __all_sync(~0u, i1 <= i0 || (left >= 16 && i1 - i0 == 16));
  if (i1 > i0) {
    if (inside) {
      const unsigned sh = (unsigned)(uintptr_t)s & 15u;
      u = ld16l1(s - sh);
      if (sh) u = cut16(u, ld16l1(s - sh + 16), sh);
    } else {
      const int n1 = left < (uint64_t)(i1 - i0) ? i0 + (int)left : i1;
      if (n1 == i1 || blk.size(k + 1) >= (uint64_t)(i1 - n1)) {
        u = meet16(s - i0, src0 + (uint64_t)(k + 1) * step - n1, i0, n1, i1);
      } else { /* small blocks, more than two of them: byte by byte */
        unsigned w[4] = {0, 0, 0, 0};
        for (int i = i0; i < i1; i++) {
          while (left == 0) { /* the next block with a byte */
            left = blk.size(++k);
            s = src0 + (uint64_t)k * step;
          }
          const unsigned c = (unsigned)(unsigned char)*s << (8 * (i & 3));
#pragma unroll
          for (int q = 0; q < 4; q++) w[q] |= i >> 2 == q ? c : 0;
          s++;
          left--;
        }
        u = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    if (i1 - i0 == 16) {
      char *d = dst0 + x0 + (uint64_t)j0 * step;
      for (int j = j0; j < j1; j++, d += step)
        if (j != skip) st16cs(d, u);
    }
  }
  /* the row's ends, in bytes: the members over the warp's lanes */
  unsigned ends = __ballot_sync(~0u, i1 > i0 && i1 - i0 < 16);
  while (ends) {
    const int from = __ffs(ends) - 1;
    ends &= ends - 1;
    const unsigned w[4] = {__shfl_sync(~0u, u.x, from), __shfl_sync(~0u, u.y, from),
                           __shfl_sync(~0u, u.z, from), __shfl_sync(~0u, u.w, from)};
    const int e0 = __shfl_sync(~0u, i0, from), e1 = __shfl_sync(~0u, i1, from);
    char *d = dst0 + __shfl_sync(~0u, x0, from);
    for (int j = j0 + (int)(threadIdx.x & 31); j < j1; j += 32)
      if (j != skip)
#pragma unroll
        for (int i = 0; i < 16; i++)
          if (i >= e0 && i < e1) d[(uint64_t)j * step + i] = (char)(w[i >> 2] >> (8 * (i & 3)));
  }
}

/* Short rows: one thread per byte of the row.  What bounds them is the launch
 * and one round of loads, and there is no vector to put together first (3 us
 * in a graph for 8 members x 4 bytes by k_spread, 1.5 this way). */
template <class BLK>
__global__ void __launch_bounds__(256) k_spread_bytes(const __grid_constant__ Row<BLK> r) {
  const auto blk = blocks(r.prm);
  const uint64_t x = (uint64_t)blockIdx.x * 256 + threadIdx.x;
  if (x >= r.len) return;
  uint64_t b;
  const int k = blk.find(x, r.nblk, &b);
  const char c = r.src0[(uint64_t)k * r.step + b];
  const int j0 = blockIdx.y * r.mpc, j1 = j0 + r.mpc < r.P ? j0 + r.mpc : r.P;
  char *d = r.dst0 + x + (uint64_t)j0 * r.step;
  for (int j = j0; j < j1; j++, d += r.step)
    if (j != r.skip) *d = c;
}

/* broadcast of aligned rows to few members: neighbouring vectors by a grid
 * that strides, each written to every member (but the root).  For broadcasts
 * that stay in L2, and to one member, where nothing pays for k_spread's
 * setting up of each vector. */
__global__ void __launch_bounds__(256) k_broadcast(const char *src, char *dst0, uint64_t step,
                                                   int P, int root, uint64_t n) {
  for (uint64_t v = (uint64_t)blockIdx.x * 256 + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * 256) {
    const uint4 u = ld16(src + v * 16);
    for (int j = 0; j < P; j++)
      if (j != root) st16(dst0 + (uint64_t)j * step + v * 16, u);
  }
}

/* fcollect staged through shared memory with the bulk-copy engine: a CTA
 * brings a tile of source k into shared memory with one cp.async.bulk load
 * (completion counted on an mbarrier), then issues one cp.async.bulk store
 * of the tile to each member's dest, so the P writes of every byte are
 * issued by the copy engine rather than by P store instructions per thread.
 * Two buffers: the load of the next tile overlaps the stores of this one.
 * Needs 16-byte aligned offsets, step and size (the vector path's rule).
 * Every wait is bounded; one that runs out sets the TIMEOUT status bit and
 * the CTA stops issuing. */
constexpr unsigned kFcBulkTile = 8192; /* bytes per tile */
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ bool mbar_wait(uint64_t *m, unsigned phase) {
  for (unsigned i = 0; i < (1u << 24); i++) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(m)), "r"(phase)
        : "memory");
    if (ok) return true;
    __nanosleep(32);
  }
  return false;
}
__device__ __forceinline__ void bulk_load(void *dst_smem, const char *src, unsigned bytes,
                                          uint64_t *m) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(m)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst_smem)),
      "l"(src), "r"(bytes), "r"(smem_addr(m))
      : "memory");
}

__global__ void __launch_bounds__(256) k_fcollect_bulk(const char *src0, char *dst0,
                                                       uint64_t step, int P, uint64_t nbytes,
                                                       int *status) {
  __shared__ __align__(128) char buf[2][kFcBulkTile];
  __shared__ __align__(8) uint64_t mbar[2];
  __shared__ int s_ok;
  const int k = blockIdx.y;
  const char *src = src0 + (uint64_t)k * step;
  const uint64_t ntiles = (nbytes + kFcBulkTile - 1) / kFcBulkTile;
  uint64_t t = blockIdx.x;
  if (t >= ntiles) return;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar[0])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbar[1])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_ok = 1;
  }
  __syncthreads();
  auto tile_bytes = [&](uint64_t tt) {
    const uint64_t off = tt * kFcBulkTile;
    return (unsigned)(nbytes - off < kFcBulkTile ? nbytes - off : kFcBulkTile);
  };
  if (threadIdx.x == 0) bulk_load(buf[0], src + t * kFcBulkTile, tile_bytes(t), &mbar[0]);
  unsigned phase[2] = {0, 0};
  bool issued = false;
  for (int b = 0; t < ntiles; t += gridDim.x, b ^= 1) {
    const uint64_t off = t * kFcBulkTile;
    const unsigned bytes = tile_bytes(t);
    /* every thread that stores waits for the tile itself */
    const bool ready = mbar_wait(&mbar[b], phase[b]);
    phase[b] ^= 1;
    if (!ready) {
      if (threadIdx.x == 0) atomicOr(status, (int)B200SHM_STATUS_TIMEOUT);
      s_ok = 0;
    }
    __syncthreads();
    if (!s_ok) break;
    for (int j = threadIdx.x; j < P; j += blockDim.x) {
      char *d = dst0 + (uint64_t)j * step + (uint64_t)k * nbytes + off;
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(d),
                   "r"(smem_addr(buf[b])), "r"(bytes)
                   : "memory");
      issued = true;
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    /* the stores of the previous tile (the other buffer) have read it */
    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0 && t + gridDim.x < ntiles)
      bulk_load(buf[b ^ 1], src + (t + gridDim.x) * kFcBulkTile, tile_bytes(t + gridDim.x),
                &mbar[b ^ 1]);
  }
  /* this thread's stores complete before the CTA ends */
  if (issued) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncthreads();
}

/* alltoall: member j's dest[k*B + b] = member k's src[j*B + b].
 * A CTA writes 256 * U vectors, its tile, of one dest row (blockIdx.y,
 * striding where a team has more rows than the grid's y extent). */

/* Where the bytes of a tile come from: the tile begins at position x0 of
 * the row, byte b0 of block k0.  It crosses at most one block end when B is
 * larger than it; otherwise `recip` = floor(2^32 / B) + 1 and
 * umulhi(position, recip) is the block exactly: positions stay at or below
 * B + TILE <= 2^15 and B <= 2^14, so the product's error, at most position
 * / 2^32, is below 1 / B. */
template <int TILE>
struct BlockWalk {
  int64_t x0, b0;
  uint64_t k0;
  int lim; /* the tile offset of block k0's end, at most TILE */
  uint64_t jump; /* from a block's end to the next block's first byte */
  unsigned B32, recip;
  __device__ __forceinline__ BlockWalk(int a, uint64_t step, uint64_t B, unsigned r) {
    x0 = (int64_t)blockIdx.x * TILE - a;
    k0 = x0 > 0 ? (uint64_t)x0 / B : 0;
    b0 = x0 - (int64_t)(k0 * B);
    lim = (int64_t)B - b0 < TILE ? (int)((int64_t)B - b0) : TILE;
    jump = step - B;
    B32 = (unsigned)B;
    recip = r;
  }
  /* the source of the byte at tile offset t, from that of offset 0 in k0;
   * *rem: bytes left in its block, or in the tile where that is less */
  __device__ __forceinline__ const char *at(const char *col, int t, int *rem) const {
    if (recip) {
      const unsigned bi = (unsigned)((int)b0 + t), q = __umulhi(bi, recip);
      *rem = (int)((q + 1) * B32 - bi);
      return col + t + q * jump;
    }
    const bool past = t >= lim;
    *rem = past ? TILE - t : lim - t;
    return col + t + (past ? jump : 0);
  }
};

/* Blocks of whole aligned vectors, neighbouring threads on neighbouring
 * dest vectors whatever the block size (one block pair a CTA left most
 * threads of small blocks idle).  128 members x 64 KiB: 333 -> 318 us (6.7
 * TB/s); x 4 KiB: 37.0 -> 22.3; x 1008 bytes: 8.35 -> 7.7. */
template <int U>
__global__ void __launch_bounds__(256, 4) k_alltoall(const char *src0, char *dst0, uint64_t step,
                                                     int P, uint64_t B, unsigned recip) {
  const BlockWalk<4096 * U> w(0, step, B, recip);
  const int64_t end = (int64_t)((uint64_t)P * B) - w.x0;
  for (uint64_t j = blockIdx.y; j < (uint64_t)P; j += gridDim.y) {
    char *row = dst0 + j * step + w.x0;
    const char *col = src0 + j * B + w.k0 * step + w.b0;
    uint4 x[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int t = ((int)threadIdx.x + u * 256) * 16;
      int rem;
      const char *s = w.at(col, t, &rem);
      if (t < end) x[u] = ld16(s);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int t = ((int)threadIdx.x + u * 256) * 16;
      if (t < end) st16(row + t, x[u]);
    }
  }
}

/* 16 bytes from byte 4 * Q + bits / 8 of lo, hi */
template <int Q>
__device__ __forceinline__ uint4 cut_at(uint4 lo, uint4 hi, unsigned bits) {
  const unsigned w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  return make_uint4(
      __funnelshift_r(w[Q], w[Q + 1], bits), __funnelshift_r(w[Q + 1], w[Q + 2], bits),
      __funnelshift_r(w[Q + 2], w[Q + 3], bits), __funnelshift_r(w[Q + 3], w[Q + 4], bits));
}
/* A lane's vectors of a warp whose bytes lie in one block: 512 apart at
 * the 16-byte aligned d, from s at the shift 4 * Q + bits / 8. */
template <int U, int Q>
__device__ __forceinline__ void cut_run(char *d, const char *s, unsigned bits) {
  uint4 lo[U], hi[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    lo[u] = ld16l1(s + u * 512);
    hi[u] = Q == 0 && bits == 0 ? lo[u] : ld16l1(s + u * 512 + 16);
  }
#pragma unroll
  for (int u = 0; u < U; u++) st16(d + u * 512, cut_at<Q>(lo[u], hi[u], bits));
}

/* Any offsets and blocks of 16 bytes or more: each aligned dest vector is
 * cut out of two neighbouring source vectors, the second of which is the
 * next lane's first and comes from L1.  A warp writes 32 * U vectors in a
 * row.  What bounds it off the memory is the instructions per vector: where
 * the warp's bytes lie in one block, the shift is the warp's, the word part
 * of it a branch and the rest one funnel shift a word; the warps in whose
 * bytes a block ends look for the block of each vector.  (The same search
 * for every vector took 163 instructions each and 457 us for 128 members x
 * 65532 bytes.)  Against one word of the blocks' common width a thread: 128
 * members x 65532 bytes 1800 -> 321 us (6.7 TB/s), x 9999 289 -> 59.5, x 1004
 * 23.6 -> 12.4. */
template <int U>
__global__ void __launch_bounds__(256, U > 2 ? 4 : 6)
    k_alltoall_shift(const char *src0, char *dst0, uint64_t step, int P, uint64_t B,
                     unsigned recip) {
  const int a = (int)((uintptr_t)dst0 & 15);
  const BlockWalk<4096 * U> w(a, step, B, recip);
  const int64_t end = (int64_t)((uint64_t)P * B) - w.x0;
  const int lane = (int)(threadIdx.x & 31), tw = (int)(threadIdx.x >> 5) * 512 * U;
  if (tw >= end) return;
  for (uint64_t j = blockIdx.y; j < (uint64_t)P; j += gridDim.y) {
    char *row = dst0 + j * step + w.x0;
    const char *col = src0 + j * B + w.k0 * step + w.b0;
    int rem;
    const char *s = w.at(col, tw, &rem);
    if (w.x0 + tw >= 0 && tw + 512 * U <= end && rem >= 512 * U) {
      const unsigned sh = (unsigned)(uintptr_t)s & 15u, bits = (sh & 3) * 8;
      char *d = row + tw + lane * 16;
      s += lane * 16 - (int)sh;
      switch (sh >> 2) {
      case 0: cut_run<U, 0>(d, s, bits); break;
      case 1: cut_run<U, 1>(d, s, bits); break;
      case 2: cut_run<U, 2>(d, s, bits); break;
      default: cut_run<U, 3>(d, s, bits);
      }
      continue;
    }
#pragma unroll 1
    for (int u = 0; u < U; u++) {
      const int t = tw + u * 512 + lane * 16;
      if (w.x0 + t >= 0 && t + 16 <= end) {
        s = w.at(col, t, &rem);
        st16(row + t, meet16(s, s + w.jump, 0, rem < 16 ? rem : 16, 16));
      } else if (t < end) {
        /* the row's ends, byte by byte: put together like the others they cost
         * the warps that cross blocks 5 to 17 %, and steps so small that their
         * latency shows go by words */
#pragma unroll 1
        for (int i = 0; i < 16; i++) {
          const int64_t y = w.x0 + t + i;
          if (y < 0 || t + i >= end) continue;
          const uint64_t k = (uint64_t)y / B;
          row[t + i] = src0[j * B + k * step + ((uint64_t)y - k * B)];
        }
      }
    }
  }
}

/* alltoall of small blocks and of few words: one thread per word of the
 * flattened [pair][word] space, in the sources' order. */
template <class W>
__global__ void __launch_bounds__(256) k_alltoall_flat(const char *src0, char *dst0,
                                                       uint64_t step, int P, uint64_t nw) {
  const uint64_t total = (uint64_t)P * (uint64_t)P * nw;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t pr = i / nw, w = i - pr * nw;
    const uint64_t k = pr / (uint64_t)P, j = pr - k * (uint64_t)P;
    ((W *)(dst0 + j * step))[k * nw + w] = ((const W *)(src0 + k * step))[j * nw + w];
  }
}

/* strided alltoall (alltoalls.c:39-50, 78-83): element t from member k to
 * member l: src_k[(l*n + t)*sst] -> dest_l[(k*n + t)*dst].
 * Pairs k*P + l over blockIdx.y, grid-stride as in k_alltoall. */
template <class E>
__global__ void __launch_bounds__(256) k_alltoalls(const char *src0, char *dst0, uint64_t step,
                                                   int P, uint64_t n, int64_t dst, int64_t sst) {
  const uint64_t pairs = (uint64_t)P * (uint64_t)P;
  for (uint64_t pr = blockIdx.y; pr < pairs; pr += gridDim.y) {
    const uint64_t k = pr / (uint64_t)P, l = pr % (uint64_t)P;
    const E *src = (const E *)(src0 + k * step) + l * n * (uint64_t)sst;
    E *d = (E *)(dst0 + l * step) + k * n * (uint64_t)dst;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (uint64_t)gridDim.x * blockDim.x)
      d[t * (uint64_t)dst] = src[t * (uint64_t)sst];
  }
}

/* strided alltoall with few elements per pair: one thread per element of
 * the flattened [pair][element] space */
template <class E>
__global__ void __launch_bounds__(256) k_alltoalls_flat(const char *src0, char *dst0,
                                                        uint64_t step, int P, uint64_t n,
                                                        int64_t dst, int64_t sst) {
  const uint64_t total = (uint64_t)P * (uint64_t)P * n;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t pr = i / n, t = i - pr * n;
    const uint64_t k = pr / (uint64_t)P, l = pr - k * (uint64_t)P;
    const E *src = (const E *)(src0 + k * step);
    E *d = (E *)(dst0 + l * step);
    d[(k * n + t) * (uint64_t)dst] = src[(l * n + t) * (uint64_t)sst];
  }
}

/* strided alltoall with an element size that is not 1/2/4/8/16 bytes */
__global__ void __launch_bounds__(256) k_alltoalls_bytes(const char *src0, char *dst0,
                                                         uint64_t step, int P, uint64_t n,
                                                         int64_t dst, int64_t sst, uint64_t es) {
  const uint64_t pairs = (uint64_t)P * (uint64_t)P;
  for (uint64_t pr = blockIdx.y; pr < pairs; pr += gridDim.y) {
    const uint64_t k = pr / (uint64_t)P, l = pr % (uint64_t)P;
    const char *src = src0 + k * step + l * n * (uint64_t)sst * es;
    char *d = dst0 + l * step + k * n * (uint64_t)dst * es;
    for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n * es;
         x += (uint64_t)gridDim.x * blockDim.x) {
      const uint64_t t = x / es, b = x % es;
      d[t * (uint64_t)dst * es + b] = src[t * (uint64_t)sst * es + b];
    }
  }
}

/* Pairs of an all-to-all beyond this many loop over blockIdx.y. */
constexpr uint64_t kMaxGridY = 65535;
/* Strided blocks of fewer elements than this per pair take the flattened kernel. */
constexpr uint64_t kFlatWords = 64;

/* CTAs along x for a per-pair / per-member extent of n work items, so that
 * the whole grid is about `want` CTAs. */
unsigned x_blocks(uint64_t n, uint64_t ypairs, uint64_t want) {
  uint64_t per = (n + 255) / 256;
  uint64_t cap = want / (ypairs ? ypairs : 1);
  if (cap < 1) cap = 1;
  if (per > cap) per = cap;
  return (unsigned)(per < 1 ? 1 : per);
}

/* Launch the copy of a row of len bytes to P members; grid16: its blocks and
 * the offsets are multiples of 16. */
template <class BLK>
void spread(const char *src, char *dst, uint64_t step, int P, uint64_t len, int nblk, int skip,
            bool grid16, const BLK &blk, cudaStream_t s) {
  const uint64_t sms = (uint64_t)st().sm_count;
  auto members_per_cta = [&](uint64_t split, uint64_t least) {
    split = std::max<uint64_t>(1, std::min<uint64_t>(split, ((uint64_t)P + least - 1) / least));
    return (int)((P + split - 1) / split);
  };
  /* Bytes against vectors, us in a graph: fcollect of 32 x 100 bytes 1.6 / 1.9,
   * 16 x 260 1.7 / 1.9, 6 x 4100 1.6 / 2.2, 128 x 64 (whole vectors) 1.8 / 1.9; a
   * broadcast of 4096 to 4 1.6 either way; an uneven collect, whose table every
   * byte searches, of 4 members and 129 KB 2.0 / 1.8. */
  constexpr bool table = !std::is_same<BLK, Even>::value && !std::is_same<BLK, Whole>::value;
  if (len <= (grid16 ? 1024 : 8192) || (!grid16 && !table && len * (uint64_t)P <= 1 << 20)) {
    const uint64_t gx = (len + 255) / 256;
    const int mpc = members_per_cta(2 * sms / gx, 2);
    k_spread_bytes<BLK><<<dim3((unsigned)gx, (unsigned)((P + mpc - 1) / mpc)), 256, 0, s>>>(
        Row<BLK>{src, dst, step, len, P, nblk, mpc, skip, blk, {}});
    count_launch();
    return;
  }
  /* The members are split over more CTAs where the row's vectors leave SMs
   * idle: short rows, two members to a CTA at least, into one wave of the six
   * CTAs an SM holds (128 x 260 bytes 2.9 us, 4.5 in the 1.3 waves that eight
   * an SM make), longer ones, four to a CTA, into eight an SM (128 x 8 KiB 21.9
   * against 24.6, 32 x 64 KiB 10.6 against 12.1: the SMs finish more evenly; 8 x
   * 64 KiB 2.3, with two to a CTA 2.6). */
  const uint64_t tiles = (((uintptr_t)dst & 15) + len + 4095) / 4096;
  const int mpc = tiles < 128 ? members_per_cta(6 * sms / tiles, 2)
                              : members_per_cta((8 * sms + tiles - 1) / tiles, 4);
  dim3 grid((unsigned)tiles, (unsigned)((P + mpc - 1) / mpc));
  /* Long rows of many members run two CTAs an SM, by a claim on shared
   * memory: fewer rows are written at a time, which DRAM likes better.  Two /
   * six CTAs, us in a graph: 128 members, 512 tiles 39.9 / 42.4, 1024 76.3 /
   * 81.2; 64 members, 512 20.8 / 21.9; 32 members, 512 10.7 / 10.6, 768 15.4 /
   * 15.7, an uneven collect of 512 11.4 / 10.8, 640 13.0 / 13.1; 16 members, 1024
   * 40.5 / 46; but a broadcast of 4096 tiles to 8 19.5 / 19.0, of 16384 100 / 84, to
   * 4 72 / 42.  (A resident serving loop leaves room for one such CTA an SM,
   * and takes nothing: 128 x 32 KiB 78.0 beside it, 82.8 with six.) */
  constexpr int kHalfSm = 100000;
  size_t smem = 0;
  if (tiles >= 640 && P >= 16 && /* the claim is the current device's: asked for on each launch */
      cudaFuncSetAttribute(k_spread<BLK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHalfSm) ==
          cudaSuccess)
    smem = kHalfSm;
  k_spread<BLK><<<grid, 256, smem, s>>>(Row<BLK>{src, dst, step, len, P, nblk, mpc, skip, blk, {}});
  count_launch();
}

}  // namespace

int fcollect_launch(int pe_start, int pe_stride, int P, uint64_t dest_off, uint64_t src_off,
                    uint64_t nbytes, cudaStream_t s) {
  int rc = check_team(pe_start, pe_stride, P);
  if (rc) return rc;
  if (nbytes > st().slice / (uint64_t)P) return fail(B200SHM_ERR_ARG, "fcollect: too large");
  if ((rc = check_extent(src_off, nbytes, "fcollect source"))) return rc;
  if ((rc = check_extent(dest_off, nbytes * (uint64_t)P, "fcollect dest"))) return rc;
  if (overlaps(dest_off, nbytes * (uint64_t)P, src_off, nbytes))
    return fail(B200SHM_ERR_ARG, "fcollect: dest and source overlap");
  if (nbytes == 0) return B200SHM_OK;
  if (P > 65535) return fail(B200SHM_ERR_UNSUPPORTED, "fcollect: more than 65535 members");
  Members m = members(pe_start, pe_stride, P);
  const bool vec = ((src_off | dest_off | nbytes | m.step) & 15u) == 0;
  static const bool bulk = getenv("B200SHM_FCOLLECT_BULK") && atoi(getenv("B200SHM_FCOLLECT_BULK")) > 0;
  if (vec && bulk) { /* the staged form, selected for measurement */
    const uint64_t ntiles = (nbytes + kFcBulkTile - 1) / kFcBulkTile;
    const uint64_t cap = (8ull * st().sm_count + P - 1) / (uint64_t)P;
    dim3 g((unsigned)(ntiles < cap ? ntiles : (cap ? cap : 1)), P);
    k_fcollect_bulk<<<g, 256, 0, s>>>(m.first + src_off, m.first + dest_off, m.step, P, nbytes,
                                      st().d_status);
    count_launch();
    return B200SHM_OK;
  }
  spread(m.first + src_off, m.first + dest_off, m.step, P, nbytes * (uint64_t)P, P, -1, vec,
         Even{nbytes}, s);
  return B200SHM_OK;
}

/* Where s is being captured, the upload of a table runs at each replay of the
 * graph: from a copy that the graph owns, not from the caller's. */
static int table_for_graph(const std::vector<uint64_t> &pre, cudaStream_t s,
                           const uint64_t **table) {
  cudaStreamCaptureStatus cap;
  cudaGraph_t graph = nullptr;
  B200_CK(cudaStreamGetCaptureInfo(s, &cap, nullptr, &graph));
  if (cap != cudaStreamCaptureStatusActive) return B200SHM_OK;
  auto *own = new std::vector<uint64_t>(pre);
  cudaUserObject_t obj;
  cudaError_t e = cudaUserObjectCreate(
      &obj, own, [](void *p) { delete (std::vector<uint64_t> *)p; }, 1,
      cudaUserObjectNoDestructorSync);
  if (e != cudaSuccess) {
    delete own;
    return cuda_fail(e, "collect: table of a captured call");
  }
  *table = own->data();
  e = cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(obj, 1);
    return cuda_fail(e, "collect: table of a captured call");
  }
  return B200SHM_OK;
}

int collect_launch(int pe_start, int pe_stride, int P, uint64_t dest_off, uint64_t src_off,
                   const uint64_t *nbytes, cudaStream_t s) {
  int rc = check_team(pe_start, pe_stride, P);
  if (rc) return rc;
  if (!nbytes) return fail(B200SHM_ERR_ARG, "collect: null size array");
  if (P > 65535) return fail(B200SHM_ERR_UNSUPPORTED, "collect: more than 65535 members");
  std::vector<uint64_t> pre((size_t)P + 1);
  uint64_t total = 0, biggest = 0;
  for (int k = 0; k < P; k++) {
    if (nbytes[k] > st().slice || total + nbytes[k] > st().slice)
      return fail(B200SHM_ERR_ARG, "collect: contributions larger than a heap slice");
    pre[k] = total;
    total += nbytes[k];
    if (nbytes[k] > biggest) biggest = nbytes[k];
  }
  pre[P] = total;
  if ((rc = check_extent(src_off, biggest, "collect source"))) return rc;
  if ((rc = check_extent(dest_off, total, "collect dest"))) return rc;
  if (overlaps(dest_off, total, src_off, biggest))
    return fail(B200SHM_ERR_ARG, "collect: dest and source overlap");
  if (total == 0) return B200SHM_OK;
  Members m = members(pe_start, pe_stride, P);
  const char *src = m.first + src_off;
  char *dst = m.first + dest_off;
  /* The table of positions as a kernel parameter, which takes an allocation,
   * an upload and a free from around the kernel; teams too large for one keep
   * it in device memory. */
  auto by_value = [&](auto blk) {
    memcpy(blk.pre, pre.data(), pre.size() * sizeof(uint64_t));
    spread(src, dst, m.step, P, total, P, -1, false, blk, s);
  };
  if (P < 136) {
    by_value(Uneven<136>{});
  } else if (P < 1032) {
    by_value(Uneven<1032>{});
  } else {
    const uint64_t *table = pre.data();
    if ((rc = table_for_graph(pre, s, &table))) return rc;
    uint64_t *dev = nullptr;
    B200_CK(cudaMallocAsync((void **)&dev, pre.size() * sizeof(uint64_t), s));
    B200_CK(cudaMemcpyAsync(dev, table, pre.size() * sizeof(uint64_t), cudaMemcpyHostToDevice, s));
    spread(src, dst, m.step, P, total, P, -1, false, Uneven<0>{dev}, s);
    B200_CK(cudaFreeAsync(dev, s));
  }
  return B200SHM_OK;
}

int alltoall_launch(int pe_start, int pe_stride, int P, uint64_t dest_off, uint64_t src_off,
                    uint64_t B, cudaStream_t s) {
  int rc = check_team(pe_start, pe_stride, P);
  if (rc) return rc;
  if (B > st().slice / (uint64_t)P) return fail(B200SHM_ERR_ARG, "alltoall: too large");
  if ((rc = check_extent(src_off, B * (uint64_t)P, "alltoall source"))) return rc;
  if ((rc = check_extent(dest_off, B * (uint64_t)P, "alltoall dest"))) return rc;
  if (overlaps(dest_off, B * (uint64_t)P, src_off, B * (uint64_t)P))
    return fail(B200SHM_ERR_ARG, "alltoall: dest and source overlap");
  if (B == 0) return B200SHM_OK;
  Members m = members(pe_start, pe_stride, P);
  const char *sp = m.first + src_off;
  char *dp = m.first + dest_off;
  const uint64_t bits = src_off | dest_off | B;
  const uint64_t nv = (((uintptr_t)dp & 15) + (uint64_t)P * B + 15) / 16; /* vectors of a row */
  const bool many = nv * (uint64_t)P >= 16ull * 256 * st().sm_count;
  /* Words of the common width of blocks and offsets, one a thread, in the
   * sources' order: for blocks of less than 16 bytes (more than two may meet
   * in a vector), and where a step has few words, or blocks so small that
   * most warps' vectors meet a block end.  Vectors / words in us, in a graph:
   * words of 8 bytes, 128 members x 456 bytes 6.5 / 5.3, x 1000 10.5 / 9.9,
   * x 2056 14.4 / 19.2, 24 x 2056 2.4 / 2.2; of 4, 128 x 36 2.5 / 2.2, x 100
   * 3.2 / 3.3, 24 x 228 1.9 / 1.7, 48 x 388 2.3 / 2.5; of 1, 24 x 101 2.2 /
   * 1.8, 48 x 101 2.0 / 2.5; whole vectors, 96 x 256 2.4 / 2.3, 48 x 256 1.7 /
   * 1.8, 128 x 1008 (four a thread) 5.1 / 5.8. */
  const uint64_t w = bits & 15 ? bits & 7 ? bits & 3 ? 1 : 4 : 8 : 16, nw = B / w;
  const uint64_t words = (uint64_t)P * P * nw;
  const bool flat = w == 16  ? nw >= 4 && words >= 70000 && !many
                    : w == 8 ? nw <= 128 || words <= 200000
                    : w == 4 ? (nw <= 12 && words <= 1500000) || words <= 130000
                             : words <= 120000;
  if (flat || B < 16) {
    const unsigned g = grid_for(words, 256, 8);
    switch (w) {
    case 16: k_alltoall_flat<uint4><<<g, 256, 0, s>>>(sp, dp, m.step, P, nw); break;
    case 8: k_alltoall_flat<unsigned long long><<<g, 256, 0, s>>>(sp, dp, m.step, P, nw); break;
    case 4: k_alltoall_flat<unsigned><<<g, 256, 0, s>>>(sp, dp, m.step, P, nw); break;
    default: k_alltoall_flat<unsigned char><<<g, 256, 0, s>>>(sp, dp, m.step, P, nw); break;
    }
    count_launch();
    return B200SHM_OK;
  }
  const unsigned gy = (unsigned)((uint64_t)P < kMaxGridY ? (uint64_t)P : kMaxGridY);
  auto grid = [&](int u) { return dim3((unsigned)((nv + 256 * u - 1) / (256 * u)), gy); };
  /* More vectors a thread once the grid fills the SMs four times over (below
   * that the fewer CTAs cost more than the loads in flight give).  Shifted
   * blocks: a warp in whose bytes a block ends takes about three times as
   * long, so small blocks want short runs.  128 members, U = 1 / 2 / 4:
   * 1004 bytes 12.4 / 12.4 us, 2052 18.6 / 16.5, 4100 37.0 / 29.1 / 35.0,
   * 9999 82 / 59.5 / 68, 16388 - / 90.5 / 96.3, 24580 - / 131 / 133,
   * 65532 (four) 321.  Blocks no larger than a CTA's bytes divide by a
   * reciprocal. */
  auto recip = [&](uint64_t u) { return B <= 4096 * u ? (unsigned)((1ull << 32) / B) + 1 : 0u; };
  if ((bits & 15) == 0) {
    if (many)
      k_alltoall<4><<<grid(4), 256, 0, s>>>(sp, dp, m.step, P, B, recip(4));
    else
      k_alltoall<1><<<grid(1), 256, 0, s>>>(sp, dp, m.step, P, B, recip(1));
  } else {
    if (many && B >= 32768)
      k_alltoall_shift<4><<<grid(4), 256, 0, s>>>(sp, dp, m.step, P, B, recip(4));
    else if (many && B >= 2048)
      k_alltoall_shift<2><<<grid(2), 256, 0, s>>>(sp, dp, m.step, P, B, recip(2));
    else
      k_alltoall_shift<1><<<grid(1), 256, 0, s>>>(sp, dp, m.step, P, B, recip(1));
  }
  count_launch();
  return B200SHM_OK;
}

int alltoalls_launch(int pe_start, int pe_stride, int P, uint64_t dest_off, uint64_t src_off,
                     int64_t dst, int64_t sst, uint64_t n, uint64_t es, cudaStream_t s) {
  int rc = check_team(pe_start, pe_stride, P);
  if (rc) return rc;
  if (dst < 1 || sst < 1 || es < 1)
    return fail(B200SHM_ERR_ARG, "alltoalls: strides and element size must be positive");
  const uint64_t lim = st().slice;
  /* extent touched: (P*n - 1)*stride + 1 elements */
  if (n > lim / es / (uint64_t)P) return fail(B200SHM_ERR_ARG, "alltoalls: too large");
  if (n == 0) return B200SHM_OK;
  const uint64_t cnt = (uint64_t)P * n;
  if ((uint64_t)dst > lim / cnt || (uint64_t)sst > lim / cnt)
    return fail(B200SHM_ERR_ARG, "alltoalls: stride too large");
  const uint64_t dbytes = ((cnt - 1) * (uint64_t)dst + 1) * es;
  const uint64_t sbytes = ((cnt - 1) * (uint64_t)sst + 1) * es;
  if ((rc = check_extent(src_off, sbytes, "alltoalls source"))) return rc;
  if ((rc = check_extent(dest_off, dbytes, "alltoalls dest"))) return rc;
  if (overlaps(dest_off, dbytes, src_off, sbytes))
    return fail(B200SHM_ERR_ARG, "alltoalls: dest and source overlap");
  Members m = members(pe_start, pe_stride, P);
  const uint64_t pairs = (uint64_t)P * P;
  const char *sp = m.first + src_off;
  char *dp = m.first + dest_off;
  const bool al = ((src_off | dest_off | m.step) % es) == 0;
  const bool typed = es == 1 || (al && (es == 2 || es == 4 || es == 8 || es == 16));
  if (typed && n < kFlatWords) {
    /* few elements per pair: threads over the flattened [pair][element] space */
    const unsigned g = grid_for(pairs * n, 256, 8);
    switch (es) {
    case 8: k_alltoalls_flat<uint64_t><<<g, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst); break;
    case 4: k_alltoalls_flat<uint32_t><<<g, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst); break;
    case 2: k_alltoalls_flat<uint16_t><<<g, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst); break;
    case 16: k_alltoalls_flat<uint4><<<g, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst); break;
    default: k_alltoalls_flat<uint8_t><<<g, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst); break;
    }
    count_launch();
    return B200SHM_OK;
  }
  const unsigned gy = (unsigned)(pairs < kMaxGridY ? pairs : kMaxGridY);
  dim3 grid(x_blocks(n, gy, 8ull * st().sm_count * 4), gy);
  if (al && es == 8)
    k_alltoalls<uint64_t><<<grid, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst);
  else if (al && es == 4)
    k_alltoalls<uint32_t><<<grid, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst);
  else if (al && es == 2)
    k_alltoalls<uint16_t><<<grid, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst);
  else if (es == 1)
    k_alltoalls<uint8_t><<<grid, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst);
  else if (al && es == 16)
    k_alltoalls<uint4><<<grid, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst);
  else {
    dim3 g2(x_blocks(n * es, gy, 8ull * st().sm_count * 4), gy);
    k_alltoalls_bytes<<<g2, 256, 0, s>>>(sp, dp, m.step, P, n, dst, sst, es);
  }
  count_launch();
  return B200SHM_OK;
}

int broadcast_launch(int root, int pe_start, int pe_stride, int P, uint64_t dest_off,
                     uint64_t src_off, uint64_t nbytes, cudaStream_t s) {
  int rc = check_team(pe_start, pe_stride, P);
  if (rc) return rc;
  if (root < 0 || root >= P) return fail(B200SHM_ERR_ARG, "broadcast: root %d not a member", root);
  if ((rc = check_extent(src_off, nbytes, "broadcast source"))) return rc;
  if ((rc = check_extent(dest_off, nbytes, "broadcast dest"))) return rc;
  if (dest_off != src_off && overlaps(dest_off, nbytes, src_off, nbytes))
    return fail(B200SHM_ERR_ARG, "broadcast: dest and source overlap");
  if (nbytes == 0 || P == 1) return B200SHM_OK;
  Members m = members(pe_start, pe_stride, P);
  const char *from = m.first + (uint64_t)root * m.step + src_off;
  const bool vec = ((src_off | dest_off | nbytes) & 15u) == 0;
  /* us in a graph, k_broadcast / k_spread (without its claim): to one member
   * 4 MiB 2.4 / 3.0, 64 MiB 18 / 28; to 3 1 MiB 2.0 / 2.5, 16 MiB 9.3 / 8.5; to 7 64
   * KiB 1.9 / 1.8, 1 MiB 2.6 / 3.0, 4 MiB 5.8 / 6.0, 16 MiB 25 / 19; to 15 1 MiB
   * 3.8 / 4.2; to 31 1 MiB 6.3 / 6.3. */
  const bool in_l2 = P <= 16 && nbytes >= (128 << 10) && nbytes * (uint64_t)P <= (32ull << 20);
  if (vec && (P == 2 || in_l2)) {
    k_broadcast<<<grid_for(nbytes / 16, 256, 8), 256, 0, s>>>(from, m.first + dest_off, m.step, P,
                                                             root, nbytes / 16);
    count_launch();
    return B200SHM_OK;
  }
  spread(from, m.first + dest_off, m.step, P, nbytes, 1, root, vec, Whole{nbytes}, s);
  return B200SHM_OK;
}

}  // namespace b200

using namespace b200;

extern "C" {

int b200shm_fcollect(int pe_start, int pe_stride, int pe_size, uint64_t dest_off,
                     uint64_t src_off, uint64_t nbytes, void *stream) {
  int rc = fcollect_launch(pe_start, pe_stride, pe_size, dest_off, src_off, nbytes,
                           pick_stream(stream));
  return rc ? rc : finish(stream, "b200shm_fcollect");
}

int b200shm_collect(int pe_start, int pe_stride, int pe_size, uint64_t dest_off,
                    uint64_t src_off, const uint64_t *nbytes, void *stream) {
  int rc = collect_launch(pe_start, pe_stride, pe_size, dest_off, src_off, nbytes,
                          pick_stream(stream));
  return rc ? rc : finish(stream, "b200shm_collect");
}

int b200shm_alltoall(int pe_start, int pe_stride, int pe_size, uint64_t dest_off,
                     uint64_t src_off, uint64_t nbytes, void *stream) {
  int rc = alltoall_launch(pe_start, pe_stride, pe_size, dest_off, src_off, nbytes,
                           pick_stream(stream));
  return rc ? rc : finish(stream, "b200shm_alltoall");
}

int b200shm_alltoalls(int pe_start, int pe_stride, int pe_size, uint64_t dest_off,
                      uint64_t src_off, int64_t dst, int64_t sst, uint64_t nelems,
                      uint64_t elem_size, void *stream) {
  int rc = alltoalls_launch(pe_start, pe_stride, pe_size, dest_off, src_off, dst, sst, nelems,
                            elem_size, pick_stream(stream));
  return rc ? rc : finish(stream, "b200shm_alltoalls");
}

int b200shm_broadcast(int root, int pe_start, int pe_stride, int pe_size, uint64_t dest_off,
                      uint64_t src_off, uint64_t nbytes, void *stream) {
  int rc = broadcast_launch(root, pe_start, pe_stride, pe_size, dest_off, src_off, nbytes,
                            pick_stream(stream));
  return rc ? rc : finish(stream, "b200shm_broadcast");
}

}  // extern "C"
