/*
 * reduce_kernels.cuh -- the one-pass all-reduce kernels and their launch
 * sequences, included by the translation units that instantiate them for
 * one family of element types each (reduce_int.cu, reduce_f32.cu,
 * reduce_f64.cu, reduce_c32.cu, reduce_c64.cu, and reduce_f80_<op>.cu for
 * long double, one op each), so the families compile in parallel.
 * Everything here has internal linkage.
 *
 * The reference moves O(N log P) bytes per PE through log2(P) rounds of
 * put + flag handshake (rec_dbl, src/shcoll/src/reduce.c:182-293) or
 * reduce-scatter + allgather (Rabenseifner, 306-724).  On one GPU every
 * member's slice is directly addressable, so each thread owns a 16-byte
 * column of elements, streams that column in from all P members' sources
 * with 128-bit loads, combines it in registers and streams the result out
 * to all P members' dests: 2*P*N*sizeof(T) bytes, the algorithmic minimum.
 *
 * Exactness.  The algorithm fixes the combine order and so the exact
 * floating-point result.  Three facts keep the kernel cheap:
 *  - integer AND/OR/XOR/SUM/PROD (wrapping) and MIN/MAX are associative
 *    and commutative bit for bit, so any order is exact: a running chain;
 *  - float and complex SUM/PROD are exactly commutative (a+b == b+a, and
 *    the naive complex product is symmetric), so only the tree SHAPE
 *    matters: linear = left fold (reduce.c:78-81); binomial = balanced
 *    binary tree over members combining op(upper block, lower block)
 *    (reduce.c:137-154, children in increasing mask order); rec_dbl and
 *    both Rabenseifner variants = butterfly over the power-of-two subset
 *    after folding the extra members (reduce.c:206-272, 338-454) -- the
 *    same tree for all three;
 *  - float MIN/MAX written a<b?a:b (reduce.c:731-732) is order dependent
 *    only when the operands include a NaN or both +0 and -0; columns with
 *    such operands are replayed in the algorithm's operand order, by their
 *    warp in the same launch (exact_columns; teams whose butterfly has more
 *    than 64 leaves: k_minmax_fix).  rec_dbl then gives different members
 *    different bits, exactly as the reference does.
 * Trees over more than 32 leaves in a lane are evaluated as a binary counter
 * over subtrees of 8, with one register slot per level, so leaves stream in
 * member order.
 *
 * What the kernel is bound by, and measured (GB/s of 2*P*N*sizeof(T); us in
 * a graph of back-to-back calls), against one launch for the packs with one
 * or two lanes a column, a second for the last elements, single elements
 * throughout where rows leave the 16-byte grid, and a replay launch after
 * every float MIN/MAX:
 *   64 members x 2^20, f32 SUM / f64 MAX / i64 XOR in a row: HBM, 6.15 TB/s
 *   before and after (437.0 and 435.4 us);
 *   100 members x 50001 doubles, one element off the grid, rabenseifner
 *   order: 0.62 -> 4.1 TB/s (129 -> 19.2 us), HBM and the loads in flight of
 *   a lane's 16 leaves and their extras;
 *   64 members x 4096: f32 SUM 5.6 -> 2.6 us, f64 MAX 10.9 -> 3.8 us, latency
 *   of the launch and of one or two rounds of loads;
 *   2 members x 65536 f64 MAX 4.5 -> 2.5 us; 64 members x 2^20 int16 SUM off
 *   the grid 144 -> 52 us; 100 x 2^16 complex double SUM 78 -> 52 us.
 * No fused multiply-add is ever formed: float ops use the _rn intrinsics.
 */
#pragma once
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "internal.cuh"
#include "reduce_core.cuh"

namespace b200 {
namespace {

/* Teams of more than 2 * kExactLeaves - 1 members only (smaller ones replay
 * such elements inside the streaming kernel, exact_columns): second pass
 * over the elements the streaming kernel deferred (it left their dests
 * untouched, so in-place sources are still intact): one CTA per element
 * stages the P inputs in shared memory, then replays the algorithm's
 * operand order from there.  Launched as a programmatic dependent of the
 * streaming kernel, whose CTAs let it start as they end (let_replay_start):
 * its launch then costs a call without such elements next to nothing (2 to 3
 * us otherwise), and its CTAs find the SMs empty.  (Let go as the streaming
 * CTAs began, they piled up on the SMs that had room and stayed there: 256
 * members x 20000 floats with NaNs throughout 16.1 ms, 6.2 so.)  The last CTA
 * to leave sets the counter back to zero for the next call (every CTA reads
 * it before it counts itself out), so no memset precedes the streaming
 * kernel. */
template <class T, int OP>
__global__ void __launch_bounds__(256) k_minmax_fix(const RArgs a,
                                                    const unsigned long long *list,
                                                    unsigned long long *count,
                                                    unsigned long long *done,
                                                    unsigned long long cap) {
  __shared__ T vals[fix_max_members<T>()];
  __shared__ T common;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const unsigned long long cnt = *(volatile unsigned long long *)count;
  const unsigned long long n = cnt < cap ? cnt : cap;
  for (unsigned long long k = blockIdx.x; k < n; k += gridDim.x) {
    const uint64_t e = list[k];
    for (int j = threadIdx.x; j < a.P; j += blockDim.x)
      memcpy(&vals[j], a.src + (uint64_t)j * a.sstep + e * sizeof(T), sizeof(T));
    __syncthreads();
    const uint64_t eg = a.g_off + e; /* the order depends on the position in the whole */
    const bool lower = eg < a.g_n / 2;
    if (a.algo == B200SHM_REC_DBL) {
      /* every p2s member (and the extra folded into it) keeps its own value */
      for (int q = threadIdx.x; q < a.p2s; q += blockDim.x) {
        const T v = exact_value<T, OP>([&](int j) { return vals[j]; }, a.P, a.p2s, a.logp2s,
                                       a.algo, lower, q);
        const int as = p2s_member(q, a.P, a.p2s);
        memcpy(a.dst + (uint64_t)as * a.dstep + e * sizeof(T), &v, sizeof(T));
        if (p2s_extra(q, a.P, a.p2s))
          memcpy(a.dst + (uint64_t)(as + 1) * a.dstep + e * sizeof(T), &v, sizeof(T));
      }
    } else {
      if (threadIdx.x == 0) {
        int q = 0;
        if (a.algo != B200SHM_LINEAR && a.algo != B200SHM_BINOMIAL)
          q = rev_bits(rab_block(eg, a.g_n, a.p2s), a.logp2s); /* owner of e's block */
        common = exact_value<T, OP>([&](int j) { return vals[j]; }, a.P, a.p2s, a.logp2s, a.algo,
                                    lower, q);
      }
      __syncthreads();
      for (int j = threadIdx.x; j < a.P; j += blockDim.x)
        memcpy(a.dst + (uint64_t)j * a.dstep + e * sizeof(T), &common, sizeof(T));
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(done, 1ull) == (unsigned long long)gridDim.x - 1) {
      *(volatile unsigned long long *)count = 0;
      *(volatile unsigned long long *)done = 0;
      __threadfence();
    }
  }
}

/* This CTA no longer holds up the replay kernel that follows a MIN/MAX launch
 * (which waits for this grid's results before it reads anything). */
__device__ __forceinline__ void let_replay_start() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

/* ---- the streaming kernel ----------------------------------------------
 * A column is V consecutive elements of every member (one 16-byte pack), or
 * one element where packs do not apply.  G lanes (a power of two) share a
 * column.  Lane g owns a contiguous share of the leaves -- for the
 * butterfly and for binomial trees over a power-of-two team that share is a
 * complete subtree -- and reduces it from loads it keeps up to 8 deep; the G
 * partial results are then combined across lanes with __shfl_xor over masks
 * 1, 2, ..., G/2, which is exactly the butterfly's remaining levels (mask m
 * pairs group g with g^m, lower group first: reduce.c:250-272).  Every lane
 * then stores the result to its own share of the members.
 *
 * How a column is accessed (MODE):
 *   kPacks    16-byte accesses: every row has the same offset from the
 *             16-byte grid, so the columns begin at the grid's first point
 *             in the dest rows (rows of 4 KiB or more: at the first 128-byte
 *             line) and the elements before it (fewer than a line's) and
 *             after the last whole pack (at most V - 1) are columns of one
 *             element, in the same launch;
 *   kElements one element each, at its own alignment: rows of different
 *             offsets (dest and source shifted against each other, member
 *             strides off the grid), and few elements of 1 or 2 bytes off
 *             the grid;
 *   kBytes    elements at any byte offset. */
enum { kPacks = 0, kElements = 1, kBytes = 2 };

template <class T, int V, int MODE>
__device__ __forceinline__ Pack<T, V> ld_col(const char *p) {
  if constexpr (MODE == kPacks && sizeof(T) == 16) {
    uint32_t w[4];
    asm(B200_LD_OP ".v4.u32 {%0,%1,%2,%3}, [%4];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
        : "l"(p));
    Pack<T, V> r;
    memcpy(&r, w, 16);
    return r;
  } else if constexpr (MODE == kElements) {
    static_assert(V == 1 && sizeof(T) <= 8, "one element at its own alignment");
    Pack<T, V> r;
    if constexpr (sizeof(T) == 8) {
      unsigned long long u;
      asm(B200_LD_OP ".u64 %0, [%1];" : "=l"(u) : "l"(p));
      memcpy(&r, &u, 8);
    } else if constexpr (sizeof(T) == 4) {
      unsigned u;
      asm(B200_LD_OP ".u32 %0, [%1];" : "=r"(u) : "l"(p));
      memcpy(&r, &u, 4);
    } else if constexpr (sizeof(T) == 2) {
      unsigned short u;
      asm(B200_LD_OP ".u16 %0, [%1];" : "=h"(u) : "l"(p));
      memcpy(&r, &u, 2);
    } else {
      unsigned u;
      asm(B200_LD_OP ".u8 %0, [%1];" : "=r"(u) : "l"(p));
      const unsigned char c = (unsigned char)u;
      memcpy(&r, &c, 1);
    }
    return r;
  } else {
    return ld_pack<T, V>(p);
  }
}
template <class T, int V, int MODE>
__device__ __forceinline__ void st_col(char *p, const Pack<T, V> &v) {
  if constexpr (MODE == kPacks && sizeof(T) == 16) {
    uint32_t w[4];
    memcpy(w, &v, 16);
    asm volatile(B200_ST_OP ".v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(w[0]), "r"(w[1]),
                 "r"(w[2]), "r"(w[3])
                 : "memory");
  } else if constexpr (MODE == kElements) {
    if constexpr (sizeof(T) == 8) {
      unsigned long long u;
      memcpy(&u, &v, 8);
      asm volatile(B200_ST_OP ".u64 [%0], %1;" ::"l"(p), "l"(u) : "memory");
    } else if constexpr (sizeof(T) == 4) {
      unsigned u;
      memcpy(&u, &v, 4);
      asm volatile(B200_ST_OP ".u32 [%0], %1;" ::"l"(p), "r"(u) : "memory");
    } else if constexpr (sizeof(T) == 2) {
      unsigned short u;
      memcpy(&u, &v, 2);
      asm volatile(B200_ST_OP ".u16 [%0], %1;" ::"l"(p), "h"(u) : "memory");
    } else {
      unsigned char c;
      memcpy(&c, &v, 1);
      asm volatile(B200_ST_OP ".u8 [%0], %1;" ::"l"(p), "r"((unsigned)c) : "memory");
    }
  } else {
    st_pack<T, V>(p, v);
  }
}

/* A lane's place: its column group, its leaves [l0, l1) and the members
 * [m0, m1) it stores to. */
struct Lane {
  int G, g, l0, l1, m0, m1;
};

/* One column group's work on the column whose first element is e0 (live:
 * the column exists; the whole warp enters, for the shuffles).  C: leaves a
 * lane of a tree holds -- 2, 4, 8: all loaded at once; 16 to 128: chunks of 8;
 * 0: any number of chunks of 8, a binary counter over them; kRagged<L>:
 * fewer than 2^L leaves, not a power of two (a binomial tree in one lane):
 * chunks of 8, then the last leaves one by one.  Chains: 0 where one lane
 * has all members, so that the loop's bounds are the same in all lanes and
 * slots beyond them cost nothing (f64 SUM in a linear order over 64 members x
 * 409600 93 -> 72 us, int16 SUM over 2 x 2^24 50 -> 33 us), else 1.
 * True for a MIN/MAX column whose bits depend on operand order: its dests
 * are left for the exact replay. */
template <int LEVELS>
constexpr int kRagged = -LEVELS;
template <class T, int OP, int ORDER, int V, bool MM, int C, bool POW2, int MODE>
__device__ __forceinline__ bool reduce_column(const RArgs &a, const Lane &ln, uint64_t e0,
                                              bool live) {
  typedef Pack<T, V> PK;
  const int P = a.P, l0 = ln.l0, l1 = ln.l1;
  auto member_of = [&](int q) -> int {
    /* trees have at most 2^13 members: no overflow */
    return ORDER == ORD_BUTTERFLY ? (q * P + a.p2s - 1) >> a.logp2s : q;
  };
  auto comb = [](const PK &lo, const PK &hi) {
    if constexpr (MM) return mm_combine<OP>(lo, hi);
    else if constexpr (ORDER == ORD_BINOMIAL) return papply<OP>(hi, lo);
    else return papply<OP>(lo, hi);
  };
  const char *src = a.src + e0 * sizeof(T);
  PK r;
  unsigned cls = 0;
  if (live) {
    if constexpr (ORDER == ORD_CHAIN) {
      constexpr bool kOne = C == 0; /* one lane: bounds that the whole launch shares */
      const char *p = src + (kOne ? 0 : (uint64_t)l0 * a.sstep);
      r = ld_col<T, V, MODE>(p);
      int j = kOne ? 1 : l0 + 1;
      const int end = kOne ? P : l1; /* at most kMaxMembers: j + 8 fits an int */
      do { /* once at least: a MIN/MAX lane looks at its first operand below the loads */
        PK x[8];
        const uint64_t step = opaque(a.sstep);
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (j + u < end) x[u] = ld_col<T, V, MODE>(p + (uint64_t)(u + 1) * step);
        p += 8 * step;
        if constexpr (MM)
          if (j == (kOne ? 1 : l0 + 1)) cls = mm_flags<OP>(r);
#pragma unroll
        for (int u = 0; u < 8; u++)
          if (j + u < end) {
            r = comb(r, x[u]);
            if constexpr (MM) cls |= mm_flags<OP>(x[u]);
          }
        j += 8;
      } while (j < end);
    } else {
      /* K leaves from q0 as a complete subtree, all loads before any use;
       * extra members folded in first as op(extra, own) (reduce.c:232-241) */
      auto chunk = [&](int q0, auto k_c) {
        constexpr int K = decltype(k_c)::value;
        PK x[K];
        if constexpr (POW2 || ORDER == ORD_BINOMIAL) { /* member == leaf */
          const uint64_t step = a.sstep;
          const char *p = src + (uint64_t)q0 * step;
#pragma unroll
          for (int u = 0; u < K; u++) x[u] = ld_col<T, V, MODE>(p + (uint64_t)u * step);
        } else {
#pragma unroll
          for (int h = 0; h < K; h += 4) { /* up to 4 leaves and their extras in flight */
            constexpr int E = K < 4 ? K : 4;
            const uint64_t step = opaque(a.sstep);
            const char *p = src + (uint64_t)member_of(q0 + h) * step;
            PK e[E];
            bool ex[E];
#pragma unroll
            for (int u = 0; u < E; u++, p += step) {
              x[h + u] = ld_col<T, V, MODE>(p);
              ex[u] = member_of(q0 + h + u + 1) - member_of(q0 + h + u) == 2;
              if (ex[u]) {
                p += step;
                e[u] = ld_col<T, V, MODE>(p);
              }
            }
#pragma unroll
            for (int u = 0; u < E; u++)
              if (ex[u]) x[h + u] = papply<OP>(e[u], x[h + u]);
          }
        }
#pragma unroll
        for (int w = K; w > 1; w >>= 1) {
#pragma unroll
          for (int i = 0; i < w / 2; i++) x[i] = comb(x[2 * i], x[2 * i + 1]);
        }
        return x[0];
      };
      typedef std::integral_constant<int, 8> k8;
      if constexpr (C >= 2 && C <= 8) {
        r = chunk(l0, std::integral_constant<int, C>{});
      } else if constexpr (C >= 16) {
        /* C / 8 chunks, one at a time (8 loads in flight, not C), each
         * combined with the finished subtrees of its size before it: a
         * binary counter whose carries are branches all lanes take alike */
        PK s0, s1, s2, s3;
#pragma unroll 1
        for (int c8 = 0; c8 < C / 8; c8++) {
          r = chunk(l0 + 8 * c8, k8{});
          if (c8 & 1) {
            r = comb(s0, r);
            if constexpr (C >= 32) {
              if (c8 & 2) {
                r = comb(s1, r);
                if constexpr (C >= 64) {
                  if (c8 & 4) {
                    r = comb(s2, r);
                    if constexpr (C >= 128) {
                      if (c8 & 8) r = comb(s3, r);
                      else s3 = r;
                    }
                  } else {
                    s2 = r;
                  }
                }
              } else {
                s1 = r;
              }
            }
          } else {
            s0 = r;
          }
        }
      } else {
        constexpr bool kRest = C < 0;
        /* the last leaves of complex PROD and long double trees one by one:
         * seven at a time take registers the operation needs (complex float
         * PROD over 15 members x 10^6 86 us, 79 so) */
        constexpr bool kOneByOne =
            C < -3 && (std::is_same<T, f80>::value ||
                       (OP == B200SHM_PROD && !std::is_floating_point<T>::value));
        constexpr int LV = kRest ? -C : kMaxLevels - 3; /* levels of 2^k leaves (chunks) */
        PK stk[LV];
        const int n = l1 - l0;
        int c = 0; /* subtrees of the lowest level pushed so far */
        auto push = [&](PK y, int lv) {
          const int t = lv + __ffs(~(c >> lv)) - 1;
#pragma unroll
          for (int L = 0; L < LV - 1; L++)
            if (L >= lv && L < t) y = comb(stk[L], y);
#pragma unroll
          for (int L = 0; L < LV; L++)
            if (L == t) stk[L] = y;
          c += 1 << lv;
        };
        int q = 0;
        if constexpr (LV > 3)
          for (; q + 8 <= n; q += 8) push(chunk(l0 + q, k8{}), kRest ? 3 : 0);
        if constexpr (kRest) {
          if constexpr (kOneByOne) {
#pragma unroll 1
            for (; q < n; q++) push(ld_col<T, V, MODE>(src + (uint64_t)q * a.sstep), 0);
          } else {
            PK x[7];
#pragma unroll
            for (int u = 0; u < 7; u++)
              if (q + u < n) x[u] = ld_col<T, V, MODE>(src + (uint64_t)(q + u) * a.sstep);
#pragma unroll
            for (int u = 0; u < 7; u++)
              if (q + u < n) push(x[u], 0);
          }
          bool have = false;
#pragma unroll
          for (int L = 0; L < LV; L++)
            if (n & (1 << L)) {
              r = have ? papply<OP>(r, stk[L]) : stk[L];
              have = true;
            }
        } else {
          const int top = __ffs(n >> 3) - 1; /* log2(n/8) */
#pragma unroll
          for (int L = 0; L < LV; L++)
            if (L == top) r = stk[L];
        }
      }
    }
  }
  /* butterfly levels across the G lanes of this column */
  for (int m = 1; m < ln.G; m <<= 1) {
    const PK o = shfl_xor_pack<T, V>(r, m);
    r = (ln.g & m) ? comb(o, r) : comb(r, o);
    if constexpr (MM) cls |= __shfl_xor_sync(0xffffffffu, cls, m);
  }
  if constexpr (MM) {
    const bool amb = live && mm_ambiguous<OP>(r, cls);
    if (amb && ln.g == 0 && a.fix_list != nullptr) { /* on the list of deferred elements */
      const unsigned long long slot = atomicAdd(a.fix_count, (unsigned long long)V);
      for (int i = 0; i < V; i++) {
        if (slot + i < a.fix_cap) a.fix_list[slot + i] = e0 + i;
        else atomicOr(a.status, (int)B200SHM_STATUS_FIX_OVERFLOW);
      }
    }
    if (amb) return true;
  }
  if (!live) return false;
  char *dst = a.dst + e0 * sizeof(T) + (uint64_t)ln.m0 * a.dstep;
  for (int j = ln.m0; j < ln.m1; j++, dst += a.dstep) st_col<T, V, MODE>(dst, r);
  return false;
}

/* The columns a warp left in its turns (see k_reduce), replayed exactly.
 * After the streaming loop and out of line, so that the loop's registers
 * and code are those of a kernel without it. */
template <class T, int OP, int V>
__device__ __noinline__ void exact_sweep(const RArgs &a, unsigned left, int lgG, uint64_t warp,
                                         uint64_t nwarps, uint64_t nb) {
  const int lgcols = 5 - lgG;
  unsigned turn = 1;
  for (uint64_t t = warp; t < nb; t += nwarps) {
    unsigned todo = __ballot_sync(0xffffffffu, (left & turn) != 0);
    for (; todo; todo &= todo - 1) {
      const uint64_t v = (t << lgcols) + ((__ffs(todo) - 1) >> lgG);
      if (v < a.nvec) exact_columns<T, OP, V>(a, a.head + v * V);
    }
    if (turn != 1u << 31) turn <<= 1;
  }
}

/* The elements before and after the packs, columns of one element, the last
 * warps first. */
template <class T, int OP, int ORDER, int V, bool MM, int C, bool POW2>
__device__ __forceinline__ void reduce_edges(const RArgs &a, const Lane &ln, int lgG,
                                             uint64_t warp, uint64_t nwarps) {
  const int c = (threadIdx.x & 31) >> lgG, lgcols = 5 - lgG;
  const unsigned ne = (a.nedge + (1u << lgcols) - 1) >> lgcols;
  for (uint64_t t = warp; t < ne; t += nwarps) {
    const unsigned i = (unsigned)(t << lgcols) + c;
    const bool live = i < a.nedge;
    const uint64_t e = !live ? 0 : i < a.head ? i : i + a.nvec * V;
    const bool amb = reduce_column<T, OP, ORDER, 1, MM, C, POW2, kElements>(a, ln, e, live);
    if constexpr (MM) {
      if (a.fix_list == nullptr) {
        unsigned todo = __ballot_sync(0xffffffffu, amb && ln.g == 0);
        for (; todo; todo &= todo - 1)
          exact_columns<T, OP, 1>(a, __shfl_sync(0xffffffffu, e, __ffs(todo) - 1));
      }
    }
  }
}

/* CTAs per SM an instance is held to, at least, by what its op needs (in
 * parentheses: the registers that leaves):
 *   trees over power-of-two teams 5 (48), with edges or long runs 4 (64: the
 *   code for single elements costs registers, so rows of whole packs, nedge
 *   == 0, have an instance without it), with extra members 3 (80), with a
 *   stack 2;
 *   complex PROD, four temporaries an element, 4 (at 48 registers its trees
 *   spill 160 to 250 bytes);
 *   chains in one lane 4, for 1- and 2-byte elements what their unpacking
 *   takes; chains in several lanes 5 for 8-byte elements, 4 for their MIN/MAX
 *   (a compare and two selects) and for 4-byte ones, 3 for MIN/MAX/PROD of
 *   2-byte elements, 2 for the others of 2 bytes and for bytes (which are
 *   unpacked into a register each: bytes' MIN/MAX and bit operations spill
 *   180 to 420 bytes there, and still ran 1.1 to 3 times as fast as the one
 *   CTA of 160 to 200 registers that does not, over 24 to 256 members);
 *   3 for the float MIN/MAX ones: holding those to 64 registers (4 CTAs, no
 *   spills) measured slower on the 64-PE headline (f64 MAX 5908-5912 against
 *   5938-5950 GB/s). */
template <class T, int OP, int ORDER, bool MM, int C, bool POW2, int MODE, bool EDGES>
constexpr int min_ctas() {
  constexpr bool order = OP == B200SHM_MIN || OP == B200SHM_MAX, prod = OP == B200SHM_PROD;
  constexpr bool cplx = std::is_same<T, cf32>::value || std::is_same<T, cf64>::value;
  constexpr int es = (int)sizeof(T);
  if (MODE == kBytes && (es < 16 || MM)) return 1;
  if (MM) return 3;
  if (ORDER == ORD_CHAIN && C == 0) {
    if (es == 1) return prod || OP == B200SHM_SUM ? 2 : 1;
    if (es == 2) return order || prod ? 3 : 2;
    if (MODE == kElements && cplx) return 5;
    return std::is_same<T, cf64>::value && prod ? 3 : 4;
  }
  if (ORDER == ORD_CHAIN) {
    if (es < 4) return es == 2 && (order || prod) ? 3 : 2;
    return es == 4 || EDGES || order ? 4 : 5;
  }
  if (C == 0 || C < -3 || (C < 0 && MODE == kBytes)) return 2;
  if (cplx && prod && POW2 && MODE != kElements) return 4;
  return !POW2 ? 3 : EDGES || C > 32 || MODE == kBytes ? 4 : 5;
}
template <class T, int OP, int ORDER, int V, bool MM, int C, bool POW2, int MODE, bool EDGES>
__global__ void __launch_bounds__(256, min_ctas<T, OP, ORDER, MM, C, POW2, MODE, EDGES>())
k_reduce(const __grid_constant__ RArgs a) {
  const int lane = threadIdx.x & 31, lgG = ORDER == ORD_CHAIN && C == 0 ? 0 : a.lgG;
  Lane ln;
  ln.G = 1 << lgG;
  ln.g = lane & (ln.G - 1);
  const int c = lane >> lgG, lgcols = 5 - lgG; /* columns per warp per iteration */
  const int P = a.P;
  const int nleaves = ORDER == ORD_BUTTERFLY ? a.p2s : P;
  ln.l0 = lane_leaf(ln.g, nleaves, lgG);
  ln.l1 = lane_leaf(ln.g + 1, nleaves, lgG);
  if (ORDER == ORD_BUTTERFLY) {
    ln.m0 = (ln.l0 * P + a.p2s - 1) >> a.logp2s;
    ln.m1 = (ln.l1 * P + a.p2s - 1) >> a.logp2s;
  } else {
    ln.m0 = ln.l0;
    ln.m1 = ln.l1;
  }
  /* grid-stride: all CTAs sweep one contiguous front of every member's
   * slice together, which keeps DRAM row locality (contiguous per-CTA
   * ranges measured ~20% slower) */
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t nb = (a.nvec + (1u << lgcols) - 1) >> lgcols;
  unsigned left = 0; /* bit i: this lane's column of turn i (the last bit: and of
                      * the turns after it) is left for the exact replay */
  unsigned turn = 1;
  for (uint64_t t = warp; t < nb; t += nwarps) {
    const uint64_t v = (t << lgcols) + c;
    const bool live = v < a.nvec;
    const bool amb = reduce_column<T, OP, ORDER, V, MM, C, POW2, MODE>(
        a, ln, a.head + (live ? v : 0) * V, live);
    if constexpr (MM) {
      if (amb && ln.g == 0) left |= turn;
      if (turn != 1u << 31) turn <<= 1;
    }
  }
  if constexpr (MM) {
    if (a.fix_list == nullptr && __any_sync(0xffffffffu, left != 0))
      exact_sweep<T, OP, V>(a, left, lgG, warp, nwarps, nb);
  }
  if constexpr (EDGES)
    reduce_edges<T, OP, ORDER, V, MM, C, POW2>(a, ln, lgG, nwarps - 1 - warp, nwarps);
  if constexpr (MM)
    if (a.fix_list != nullptr) let_replay_start();
}

/* CTAs of 256 threads of `kernel` that one SM holds at once (cached per
 * kernel). */
int resident_ctas(const void *kernel) {
  static std::mutex mu;
  static std::unordered_map<const void *, int> cache;
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(kernel);
  if (it != cache.end()) return it->second;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0) != cudaSuccess || n < 1) {
    (void)cudaGetLastError();
    n = 1;
  }
  cache[kernel] = n;
  return n;
}

/* Launch over `lanes` threads of work.  Grid: up to 8 waves of the CTAs one
 * SM holds at once (B200SHM_REDUCE_WAVES overrides it, or
 * B200SHM_REDUCE_CTAS_PER_SM gives a fixed count); for chains in one lane 8
 * CTAs an SM where the sources are less than 128 MiB (8 members x 2^21 int32:
 * 19.6 us, 21.3 with 8 waves; x 6.5 x 10^6 67.4 and 65.6).  On the 64-PE x
 * 2^20 workload one exact wave was slowest (5.27 TB/s over the six reductions):
 * CTAs of a grid-stride loop finish unevenly and leave their SM's slots
 * idle, while the CTAs of later waves backfill them.  4 waves gave 5.73,
 * 6-16 waves 5.78-5.80, one pack per lane 5.76.  CTAs of 256 threads, less
 * where that leaves SMs without one. */
template <class K>
void launch_one(K kernel, uint64_t lanes, bool small, cudaStream_t s, const RArgs &a) {
  static int per_sm_env = -1, waves = 8;
  if (per_sm_env < 0) {
    const char *e = getenv("B200SHM_REDUCE_CTAS_PER_SM");
    const char *w = getenv("B200SHM_REDUCE_WAVES");
    if (w && atoi(w) > 0) waves = atoi(w);
    per_sm_env = e && atoi(e) > 0 ? atoi(e) : 0;
  }
  const uint64_t sms = (uint64_t)grid_sms();
  int threads = 256;
  while (threads > 64 && lanes < sms * (uint64_t)threads) threads >>= 1;
  const int per_sm = per_sm_env ? per_sm_env
                     : small ? 8
                             : waves * resident_ctas((const void *)kernel);
  kernel<<<grid_for(lanes, threads, per_sm), threads, 0, s>>>(a);
  count_launch();
}

/* the instance with or without edges */
template <class T, int OP, int ORDER, int V, bool MM, int C, bool POW2, int MODE>
void launch_edges(uint64_t lanes, cudaStream_t s, const RArgs &a) {
  const bool small = ORDER == ORD_CHAIN && C == 0 &&
                     a.N * sizeof(T) * (uint64_t)a.P < (128ull << 20);
  if constexpr (V > 1) {
    if (a.nedge) {
      launch_one(k_reduce<T, OP, ORDER, V, MM, C, POW2, MODE, true>, lanes, small, s, a);
      return;
    }
  }
  launch_one(k_reduce<T, OP, ORDER, V, MM, C, POW2, MODE, false>, lanes, small, s, a);
}

/* Whether a lane has instances of 64 and 128 leaves (not long double, whose
 * software arithmetic bounds it, and takes minutes to compile). */
template <class T, int MODE>
constexpr bool kLongRuns = MODE == kPacks && !std::is_same<T, f80>::value;
/* leaves per lane n -> the instance */
template <class T, int OP, int ORDER, int V, bool POW2, int MODE>
void launch_tree(int n, uint64_t lanes, cudaStream_t s, const RArgs &a) {
  constexpr bool wide = MODE == kPacks || sizeof(T) == 16;
  constexpr int C16 = wide ? 16 : 0, C32 = wide ? 32 : 0;
  constexpr int C64 = kLongRuns<T, MODE> ? 64 : 0, C128 = kLongRuns<T, MODE> ? 128 : 0;
  switch (n) {
  case 2: launch_edges<T, OP, ORDER, V, false, 2, POW2, MODE>(lanes, s, a); break;
  case 4: launch_edges<T, OP, ORDER, V, false, 4, POW2, MODE>(lanes, s, a); break;
  case 8: launch_edges<T, OP, ORDER, V, false, 8, POW2, MODE>(lanes, s, a); break;
  case 16: launch_edges<T, OP, ORDER, V, false, C16, POW2, MODE>(lanes, s, a); break;
  case 32: launch_edges<T, OP, ORDER, V, false, C32, POW2, MODE>(lanes, s, a); break;
  case 64: launch_edges<T, OP, ORDER, V, false, C64, POW2, MODE>(lanes, s, a); break;
  case 128: launch_edges<T, OP, ORDER, V, false, C128, POW2, MODE>(lanes, s, a); break;
  default: launch_edges<T, OP, ORDER, V, false, 0, POW2, MODE>(lanes, s, a); break;
  }
}

/* Lanes per column (log2), for `cols` columns over `leaves` leaves.
 * Many columns: 2 lanes (1 where a lane would hold fewer than 8 leaves); for
 * float trees as many as give each lane `run` leaves (2 to 8): 128, the
 * most an instance without a stack takes, from 256 leaves on, and from 128
 * where every member is a leaf and every column a pack; else 32.  (f32 SUM,
 * 200 MiB: 256 members at 8 lanes of 32, a warp reading 64 bytes of each
 * member, 2.82 TB/s, at 2 of 128 5.50; 128 members at 4 of 32 4.89, at 2 of
 * 64 5.70; but 128 to 255 members with extras or edges at 2 lanes 1-8 %
 * slower.)  Long runs only where at least 256 threads an SM are left: 256
 * members x 65536 at 4 of 64 4.36 TB/s, at 8 of 32 2.6.  On the 64-PE
 * workload G = 2 with 32 leaves per lane ran the f32 tree at 5.6-5.9 TB/s, G =
 * 4 with 16 at 5.2-5.4 (a warp then reads 128 rather than 256 consecutive
 * bytes of each member per load).  Few columns: what counts is
 * how many rounds of loads a lane makes in turn, so lanes are added while a
 * lane holds more than 4 leaves and the columns are fewer than 128 per SM
 * over G^2 (each doubling halves the run of each member that a warp reads,
 * so it has to bring more each time: f32 SUM over 64 members of 1024 /
 * 4096 / 16384 / 65536 elements ran 2.3 / 2.8 / 3.3 / 6.2 us at the 16 / 8 /
 * 4 / 2 lanes this gives, and 4.3 / 5.5 / - / 6.0 at 2 before; at 16384 8
 * lanes take 4.6 and 16 take 7.0).
 * B200SHM_REDUCE_COOP sets the starting point (0 or 1 = one lane per
 * column). */
template <int ORDER>
int lanes_log2(uint64_t cols, int leaves, bool one, int run) {
  int G = one ? 1 : 2; /* 16-byte elements, say: a chain of one lane per element */
  if (ORDER != ORD_CHAIN) G = std::max(2, std::min(8, leaves / run));
  static const char *ec = getenv("B200SHM_REDUCE_COOP"); /* read once */
  if (ec) G = std::max(1, std::min(8, atoi(ec)));
  int lg = 31 - __builtin_clz((unsigned)G);
  while (lg > 0 && (8 << lg) > leaves) lg--;
  if (!ec && ORDER != ORD_CHAIN) /* long runs only where they fill the SMs */
    while (lg < 3 && (leaves >> lg) > 32 && (cols << lg) < (uint64_t)grid_sms() * 256) lg++;
  if (!ec)
    while (lg < 4 && (4 << (lg + 1)) <= leaves &&
           (cols << (2 * lg)) < (uint64_t)grid_sms() * 128)
      lg++;
  return lanes_within_int(lg, leaves);
}

template <class T, int OP, int ORDER, bool MM, int MODE>
void run_mode(RArgs &a, cudaStream_t s) {
  constexpr int V = MODE == kPacks && sizeof(T) < 16 ? (int)(16 / sizeof(T)) : 1;
  const int P = a.P, leaves = ORDER == ORD_BUTTERFLY ? a.p2s : P;
  const bool pow2 = (P & (P - 1)) == 0;
  a.nvec = (a.N - a.head) / V;
  a.nedge = (unsigned)(a.N - a.nvec * V);
  /* splitting the members over lanes is exact for any-order ops, for
   * butterflies, and for binomial trees over power-of-two teams */
  constexpr bool any_order = ORDER == ORD_CHAIN && (std::is_integral<T>::value || MM);
  const bool split = any_order || ORDER == ORD_BUTTERFLY || (ORDER == ORD_BINOMIAL && pow2);
  const bool long_runs = kLongRuns<T, MODE> && (leaves >= 256 || (pow2 && a.nedge == 0));
  /* single elements of 4 bytes: longer runs, and of 1 byte: one lane, else a
   * warp reads less than a sector of each member (250 members x 209715 floats
   * 218 -> 119 us, 130 x 1613193 bytes 316 -> 233) */
  const int run = long_runs ? 128 : MODE == kElements && sizeof(T) == 4 ? 64 : 32;
  const bool one = sizeof(T) == 16 || (MODE == kElements && sizeof(T) == 1);
  a.lgG = split ? lanes_log2<ORDER>(a.nvec + a.nedge, leaves, one, run) : 0;
  const uint64_t lanes = std::max<uint64_t>(a.nvec + a.nedge, 1) << a.lgG;
  if constexpr (ORDER == ORD_CHAIN && any_order) {
    if (MM || a.lgG) launch_edges<T, OP, ORDER, V, MM, 1, true, MODE>(lanes, s, a);
    else if constexpr (!MM) launch_edges<T, OP, ORDER, V, MM, 0, true, MODE>(lanes, s, a);
  } else if constexpr (ORDER == ORD_CHAIN) {
    launch_edges<T, OP, ORDER, V, MM, 0, true, MODE>(lanes, s, a);
  } else if constexpr (ORDER == ORD_BINOMIAL) {
    if (pow2) launch_tree<T, OP, ORDER, V, true, MODE>(leaves >> a.lgG, lanes, s, a);
    else if (P < 8) launch_edges<T, OP, ORDER, V, false, kRagged<3>, false, MODE>(lanes, s, a);
    else if (P < 256) launch_edges<T, OP, ORDER, V, false, kRagged<8>, false, MODE>(lanes, s, a);
    else launch_edges<T, OP, ORDER, V, false, kRagged<kMaxLevels>, false, MODE>(lanes, s, a);
  } else {
    if (pow2) launch_tree<T, OP, ORDER, V, true, MODE>(leaves >> a.lgG, lanes, s, a);
    else launch_tree<T, OP, ORDER, V, false, MODE>(leaves >> a.lgG, lanes, s, a);
  }
}

template <class T, int OP, int ORDER, bool MM>
int run(const RArgs &base, cudaStream_t s) {
  if constexpr (ORDER != ORD_CHAIN) { /* one member: nothing to combine, a copy */
    if (base.P == 1) return run<T, OP, ORD_CHAIN, false>(base, s);
  }
  RArgs a = base;
  const uint64_t steps = a.P > 1 ? a.sstep | a.dstep : 0;
  const uintptr_t sp = (uintptr_t)a.src, dp = (uintptr_t)a.dst;
  a.head = 0;
  if (!MM || a.p2s <= kExactLeaves) a.fix_list = nullptr;
  /* few narrow elements off the grid: what counts is lanes, and an element a
   * lane makes V times as many (bytes, MAX over 8 members x 8193: 2.1 us, 3.8
   * in packs; over 2 x 32769 2.0 and 2.6; 8 x 524289 the other way round) */
  const bool few = sizeof(T) <= 2 && (dp & 15) && a.N * (uint64_t)a.P <= 262144;
  if (((sp ^ dp) & 15) == 0 && (steps & 15) == 0 && dp % sizeof(T) == 0 && !few) {
    /* the packs begin at a 128-byte line of the dest, so that warps do not
     * share lines (vectors shorter than a few lines: at the 16-byte grid) */
    const uintptr_t grid = sizeof(T) < 16 && a.N * sizeof(T) >= 4096 ? 128 : 16;
    a.head = (unsigned)std::min<uint64_t>((grid - (dp & (grid - 1))) % grid / sizeof(T), a.N);
    run_mode<T, OP, ORDER, MM, kPacks>(a, s);
  } else if (sizeof(T) < 16 && ((sp | dp | steps) % sizeof(T)) == 0) {
    run_mode<T, OP, ORDER, MM, sizeof(T) < 16 ? kElements : kBytes>(a, s);
  } else {
    run_mode<T, OP, ORDER, MM, kBytes>(a, s);
  }
  if constexpr (MM) {
    if (a.fix_list == nullptr) return B200SHM_OK;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * grid_sms());
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    B200_CK(cudaLaunchKernelEx(&cfg, k_minmax_fix<T, OP>, base,
                               (const unsigned long long *)base.fix_list, base.fix_count,
                               base.fix_done, base.fix_cap));
    count_launch();
  }
  return B200SHM_OK;
}

template <class T, int OP>
int run_float(const RArgs &a, cudaStream_t s) {
  if constexpr (OP == B200SHM_MIN || OP == B200SHM_MAX) {
    /* the deferred count is zero here: the previous replay cleared it */
    return run<T, OP, ORD_CHAIN, true>(a, s);
  } else {
    switch (a.algo) {
    case B200SHM_LINEAR: return run<T, OP, ORD_CHAIN, false>(a, s);
    case B200SHM_BINOMIAL: return run<T, OP, ORD_BINOMIAL, false>(a, s);
    default: return run<T, OP, ORD_BUTTERFLY, false>(a, s);
    }
  }
}

template <class T, int OP>
int run_cplx(const RArgs &a, cudaStream_t s) {
  switch (a.algo) {
  case B200SHM_LINEAR: return run<T, OP, ORD_CHAIN, false>(a, s);
  case B200SHM_BINOMIAL: return run<T, OP, ORD_BINOMIAL, false>(a, s);
  default: return run<T, OP, ORD_BUTTERFLY, false>(a, s);
  }
}

/* Integer ops other than MIN/MAX give the same bits on signed and unsigned
 * views, so they run on the unsigned type of the same width. */
template <class S, class U>
int run_int(int op, const RArgs &a, cudaStream_t s) {
  switch (op) {
  case B200SHM_AND: return run<U, B200SHM_AND, ORD_CHAIN, false>(a, s);
  case B200SHM_OR: return run<U, B200SHM_OR, ORD_CHAIN, false>(a, s);
  case B200SHM_XOR: return run<U, B200SHM_XOR, ORD_CHAIN, false>(a, s);
  case B200SHM_MIN: return run<S, B200SHM_MIN, ORD_CHAIN, false>(a, s);
  case B200SHM_MAX: return run<S, B200SHM_MAX, ORD_CHAIN, false>(a, s);
  case B200SHM_SUM: return run<U, B200SHM_SUM, ORD_CHAIN, false>(a, s);
  default: return run<U, B200SHM_PROD, ORD_CHAIN, false>(a, s);
  }
}

}  // namespace
}  // namespace b200
