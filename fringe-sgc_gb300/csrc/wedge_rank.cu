// Wedge core with a fringe-free centre, counted in rank order.
//
// The reference evaluates wedge(dx, dy, adjacent, C - 1) once per wedge
// (src/fringeCount.cu:1381-1477); its value depends on the endpoint pair only,
// so the total is the sum over pairs of C * W(dx, dy, adjacent, C - 1), where
// C is the pair's number of common neighbours.  All sums are taken in a ring
// (mod 2^64 for the reference's arithmetic, mod 2^128 for exact counts whose
// total is bounded below 2^128 beforehand), so the total may be split:
//
//   linear      sum over wedges of W(dx, dy, no, 0): W with no second common
//               neighbour is P(dx) Q(dy) (+ P(dy) Q(dx)), P, Q binomials of the
//               degree, so it is a sum of products per centre: O(m) in all;
//   adjacent    sum over edges of C (W(.., yes, C-1) - W(.., no, C-1)), with C
//               the loader's edge support: O(m);
//   residual    sum over pairs with C >= 2 of C (W(.., no, C-1) - W(.., no, 0)).
//
// Only the residual needs the pairs' C.  When it is a multiple of C (C-1) (one
// fringe on each end, or one shared fringe: the 4-cycle) it is a multiple of
// the number of 4-cycles, and those are found from their highest-ranked vertex
// alone (ORD below): sum over edges of the smaller degree instead of the sum
// over vertices of C(deg, 2) wedges, 5.7e9 instead of 3.5e10 on RMAT scale 20.
//
// The graph is copied once into rank order: vertex r is the r-th by
// descending degree, lists sorted by rank.  Owners v count, for every w > v,
// the centres u in N(v) with w in N(u).  Heavy owners come first (the queue
// then balances the blocks), their partners sit in the lowest ids, and the
// ids of vertices too small to matter form one tail that is cut off.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "fsgc_formulas.cuh"
#include "fsgc_internal.h"

namespace fsgc {

void upload_div_magic_wedge() { upload_div_table(); }

namespace {

typedef unsigned __int128 u128;

// Exact binomials mod 2^128; the caller has checked that none reaches 2^128.
template <> __device__ __forceinline__ u128 nck_a<u128>(int n, int k) {
  const X128 r = nck_x(n, k);
  return ((u128)r.hi << 64) | r.lo;
}

// Sums mod 2^128 into slot[0..1]: every low-word carry moves on with its add.
__device__ __forceinline__ void slot_add(u128 v, u64* __restrict__ slot) {
  const u64 lo = (u64)v, hi = (u64)(v >> 64);
  const u64 old = atomicAdd(slot, lo);
  const u64 up = hi + (old + lo < old ? 1ULL : 0ULL);
  if (up) atomicAdd(slot + 1, up);
}
__device__ __forceinline__ void slot_add(u64 v, u64* __restrict__ slot) { atomicAdd(slot, v); }

__device__ __forceinline__ u64 shfl_down_a(u64 v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }
__device__ __forceinline__ u128 shfl_down_a(u128 v, int o) {
  const u64 lo = __shfl_down_sync(0xffffffffu, (u64)v, o), hi = __shfl_down_sync(0xffffffffu, (u64)(v >> 64), o);
  return ((u128)hi << 64) | lo;
}
__device__ __forceinline__ u64 shfl_up_a(u64 v, int o) { return __shfl_up_sync(0xffffffffu, v, o); }
__device__ __forceinline__ u128 shfl_up_a(u128 v, int o) {
  const u64 lo = __shfl_up_sync(0xffffffffu, (u64)v, o), hi = __shfl_up_sync(0xffffffffu, (u64)(v >> 64), o);
  return ((u128)hi << 64) | lo;
}

template <class A>
__device__ __forceinline__ A warp_sum_a(A v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += shfl_down_a(v, o);
  return v;
}

// One add per warp: the kernels here run a few thousand warps once, so the
// block-level step of block_sum_to is not worth its barriers.
template <class A>
__device__ __forceinline__ void warp_sum_to(A v, u64* __restrict__ slot) {
  v = warp_sum_a(v);
  if ((threadIdx.x & 31) == 0 && v) slot_add(v, slot);
}

// exclusive prefix over the lanes
template <class A>
__device__ __forceinline__ A warp_excl(A v) {
  const int lane = threadIdx.x & 31;
  A inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const A y = shfl_up_a(inc, o);
    if (lane >= o) inc += y;
  }
  return inc - v;
}

// wedge() with binomials of any order: out of line, the kernel calls it
// from several places and the inlined loops cost more registers than the call.
template <class A>
__device__ __noinline__ A wedge_value_any(int dx, int dy, bool adj, int f_x, int f_xy, int f_y, int c) {
  return wedge_formula_with<A>(dx, dy, adj, f_x, f_xy, f_y, c, NckA<A>());
}
template <class A>
__device__ __forceinline__ A wedge_value(int dx, int dy, bool adj, int f_x, int f_xy, int f_y, int c) {
  if ((unsigned)(f_x | f_xy | f_y) <= 1u) return wedge_formula_with<A>(dx, dy, adj, f_x, f_xy, f_y, c, Nck01<A>());
  return wedge_value_any<A>(dx, dy, adj, f_x, f_xy, f_y, c);
}

// ------------------------------------------------------------- linear term
// Per centre u: the sum over unordered pairs of neighbours of P_i Q_j + Q_i P_j
// (P Q when both ends carry the same number of fringes), P = C(deg - 1, f_v),
// Q = C(deg - 1, f_w).  Any partition of the list serves: a thread pairs each
// of its neighbours with the running sums of those before it, then the
// threads' sums are paired with each other.  One warp per centre; centres of
// degree above kLinBlock are taken by the whole block afterwards.  Bound by
// the degree gathers (4 bytes at random per list entry).
constexpr int kLinBlock = 2048;

template <class A>
__global__ void __launch_bounds__(kTPB) wedge_linear_kernel(GView g, int f_v, int f_w, u64* __restrict__ slot) {
  __shared__ int s_big[kTPB / 32];
  __shared__ A s_p[kTPB / 32], s_q[kTPB / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool same = f_v == f_w;
  A total = A(0);
  auto take = [&](int dx, A& p_sum, A& q_sum, A& acc) {
    const A p = nck_a<A>(dx, f_v), q = same ? p : nck_a<A>(dx, f_w);
    acc += same ? p * p_sum : p * q_sum + q * p_sum;
    p_sum += p;
    q_sum += q;
  };
  // consecutive vertices go to different blocks: hubs are often neighbours by id
  const int step = gridDim.x * (kTPB / 32);
  for (int v0 = 0; v0 < g.n; v0 += step) {
    const int v = v0 + warp * gridDim.x + blockIdx.x;
    int d = 0;
    if (v < g.n) d = g.deg[v];
    A acc = A(0);
    if (d >= 2 && d <= kLinBlock) {
      A p = A(0), q = A(0);
      const int* nb = g.adj + g.off[v];
      for (int t = lane; t < d; t += 32) take(g.deg[__ldg(nb + t)] - 1, p, q, acc);
      const A pe = warp_excl(p), qe = same ? pe : warp_excl(q);
      acc += same ? p * pe : p * qe + q * pe;
    }
    if (lane == 0) s_big[warp] = d > kLinBlock ? v : -1;
    if (g.comp && v < g.n) {
      acc = warp_sum_a(acc);
      if (lane == 0 && acc) slot_add(acc, g.comp_slots + g.comp[v]);
    } else {
      total += acc;
    }
    block_sync();
    for (int b = 0; b < kTPB / 32; b++) {
      const int h = s_big[b];
      if (h < 0) continue;
      A p = A(0), q = A(0), a2 = A(0);
      const int* nb = g.adj + g.off[h];
      const int dh = g.deg[h];
      for (int t0 = threadIdx.x; t0 < dh; t0 += 4 * kTPB) {
        int x[4], dx[4];  // four entries and their degrees in flight
#pragma unroll
        for (int k = 0; k < 4; k++) x[k] = t0 + k * kTPB < dh ? __ldg(nb + t0 + k * kTPB) : -1;
#pragma unroll
        for (int k = 0; k < 4; k++) dx[k] = x[k] >= 0 ? __ldg(g.deg + x[k]) - 1 : 0;
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (x[k] >= 0) take(dx[k], p, q, a2);
      }
      const A pe = warp_excl(p), qe = same ? pe : warp_excl(q);
      a2 += same ? p * pe : p * qe + q * pe;
      if (lane == 31) {
        s_p[warp] = pe + p;
        s_q[warp] = qe + q;
      }
      block_sync();
      if (threadIdx.x == 0) {
        A ps = A(0), qs = A(0);
        for (int w = 0; w < kTPB / 32; w++) {
          a2 += same ? s_p[w] * ps : s_p[w] * qs + s_q[w] * ps;
          ps += s_p[w];
          qs += s_q[w];
        }
      }
      block_sync();
      if (g.comp) {
        a2 = warp_sum_a(a2);
        if (lane == 0 && a2) slot_add(a2, g.comp_slots + g.comp[h]);
      } else {
        total += a2;
      }
    }
    block_sync();  // s_big is free again
  }
  warp_sum_to(total, slot);
}

// ------------------------------------------------------------- adjacent term
// Edges whose endpoints share a neighbour: the pair's formula with the
// adjacency correction instead of without.  One pass over the oriented edges.
template <class A>
__global__ void __launch_bounds__(kTPB) wedge_adjacent_kernel(GView g, WedgeParams p, u64* __restrict__ slot) {
  const long long me = g.m / 2;
  A acc = A(0);
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const int C = (int)g.osup[j];
    if (C == 0 || C <= p.f_vw) continue;
    const int a = g.osrc[j], b = g.oadj[j];
    const int dx = g.deg[max(a, b)], dy = g.deg[min(a, b)];
    const A x = A((u64)C) * (wedge_value<A>(dx, dy, true, p.f_v, p.f_vw, p.f_w, C - 1) -
                             wedge_value<A>(dx, dy, false, p.f_v, p.f_vw, p.f_w, C - 1));
    if (g.comp) {
      if (x) slot_add(x, g.comp_slots + g.comp[a]);
    } else {
      acc += x;
    }
  }
  warp_sum_to(acc, slot);
}

// ------------------------------------------------------------- residual
struct RankView {
  int n;
  const int* __restrict__ off;  // n+1
  const int* __restrict__ adj;  // m ranks, ascending per list
  const unsigned short* __restrict__ adj16;  // the ranks' low 16 bits
  const int* __restrict__ deg;  // n (descending, per member for packed graphs)
  const int* __restrict__ rev;  // per list entry (v, u): entries of N(u) up to and including v
  const int* __restrict__ oid;  // the vertex's id in the graph
  // lists of the first `rows` vertices: entries at or above boundary k *
  // kRGran, k = 0..K-1, so that a chunk's end is one load instead of a search
  const int* __restrict__ tab;
  int rows, K;
  const int* __restrict__ comp;  // packed graphs: member by id
  u64* comp_slots;
};

// How a pattern's residual is summed over an owner's pairs (see "Residual sums").
enum { kGeneral = 0, kSums = 1, kProduct = 2 };
struct PairForm {
  int kind;
  int s;             // shared fringes
  int kappa, delta;  // g(d) = C(d - delta, kappa); kappa < 0: g = 0
  int sign;          // kSums: total = sign (g(dv) B + A), or B where g = 0
};

struct RankSet {
  int np;                      // FULL: 1; ORD: patterns that are multiples of the 4-cycles
  int lim;                     // smallest endpoint degree that the residual needs
  int roles;                   // FULL: the binomials depend on which end has the larger id
  WedgeParams w;               // FULL
  PairForm form;               // FULL
  long long mult[kWedgeFuse];  // ORD: multiple of the number of 4-cycles
  u64* slot[kWedgeFuse];
};

constexpr int kRT = 512;         // threads; two blocks per SM overlap each other's barriers
constexpr int kRW = kRT / 32;    // warps
constexpr int kRWords = 16384;   // counter words: 64 KB
constexpr int kRCap = 2048;      // centres per batch
constexpr int kRGran = 16384;    // boundary spacing; every chunk width is a multiple
constexpr int kRStage = 160;     // staged pairs per warp: 31 left over and up to 128 of one step
constexpr int kLongSegment = 64;  // segment length from which a warp walks it by itself
constexpr int kSegmentCost = 64;  // what such a segment costs a warp beyond its entries, in entries
constexpr int kTinyCentres = 64, kTinyWedges = 256, kTinySlots = 512;
constexpr int kHashWedges = 4096, kHashSlots = 8192;
static_assert(kRW * 2 * kTinySlots == kRWords && 2 * kHashSlots == kRWords, "hash tables live in the counter words");

struct RankSmem {
  unsigned cnt[kRWords];
  int cur[kRCap];  // per centre: next entry
  int nxt[kRCap];  // and the rank there (kDone past the end)
  union {
    struct {
      int start[kRCap + 1];  // of the batch's non-empty segments: first entry
      int pre[kRCap + 2];    // and number of entries (long segments: padded) before
    };
    unsigned stage[kRW][kRStage];  // pairs on their way to evaluation; never live with the segments
  };
  unsigned long long wedges;
  int item, nlist, centres, last;
  int nlong, nshort;  // segments start[0..nlong) and start[nlong+1..nlong+nshort]
  int list[kRW];
  u64 warp_tmp[4 * kRW];
};
constexpr int kDone = 0x7fffffff;
static_assert(2 * (sizeof(RankSmem) + 1024) <= 233472, "two blocks per SM");

// number of ranks with degree >= d (ordinary graphs: degrees descend)
__device__ __forceinline__ int ranks_with_degree(const RankView& r, int d) {
  int lo = 0, hi = r.n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(r.deg + mid) >= d) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// first position of N(v) holding a rank above v
__device__ __forceinline__ int own_pos(const RankView& r, int v, int vb, int dv) {
  int lo = 0, hi = dv;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(r.adj + vb + mid) <= v) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The segment slots a thread serves in a batch: 2t, 2t+1, 1024+2t, 1025+2t.
__device__ __forceinline__ int slot_of(int k) { return (k >> 1) * 2 * kRT + 2 * (int)threadIdx.x + (k & 1); }

// Lists the non-empty segments of a batch of n slots, long ones first: segment
// i < S.nlong starts at entry S.start[i]; S.pre is the prefix sum of the
// lengths, kSegmentCost added to each, so that equal shares of it are equal
// work.  The short ones follow from index nlong + 1 with their own, unpadded
// prefix.  `st` and `len` are the thread's slots' first entries and lengths.
// Two barriers; the arrays may be written again once every warp has passed a
// barrier after its last read.
__device__ __forceinline__ void list_segments(RankSmem& S, int n, const int* st, const int* len) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto item = [&](int k, bool is_long) -> u64 {  // entries in the low word, segments in the high one
    if (len[k] <= 0 || (len[k] >= kLongSegment) != is_long) return 0ULL;
    return (1ULL << 32) + (unsigned)(len[k] + (is_long ? kSegmentCost : 0));
  };
  const int halves = n > 2 * kRT ? 2 : 1;
  u64 el[2] = {0, 0}, es[2] = {0, 0};
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (h >= halves) break;
    const u64 a = item(2 * h, true) + item(2 * h + 1, true), b = item(2 * h, false) + item(2 * h + 1, false);
    el[h] = warp_excl(a);
    es[h] = warp_excl(b);
    if (lane == 31) {
      S.warp_tmp[h * kRW + warp] = el[h] + a;
      S.warp_tmp[(2 + h) * kRW + warp] = es[h] + b;
    }
  }
  block_sync();
  // lanes 0..15: long totals of one half's warps, lanes 16..31: short totals
  u64 cl = 0, cs = 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (h >= halves) break;
    const u64 v = S.warp_tmp[(lane < kRW ? h : 2 + h) * kRW + (lane & (kRW - 1))];
    u64 inc = v;
#pragma unroll
    for (int o = 1; o < kRW; o <<= 1) {
      const u64 y = __shfl_up_sync(0xffffffffu, inc, o);
      if ((lane & (kRW - 1)) >= o) inc += y;
    }
    el[h] += cl + __shfl_sync(0xffffffffu, inc - v, warp);
    es[h] += cs + __shfl_sync(0xffffffffu, inc - v, kRW + warp);
    cl += __shfl_sync(0xffffffffu, inc, kRW - 1);
    cs += __shfl_sync(0xffffffffu, inc, 31);
  }
  const int nl = (int)(cl >> 32);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    if (h >= halves) break;
#pragma unroll
    for (int k = 2 * h; k < 2 * h + 2; k++) {
      const u64 a = item(k, true), b = item(k, false);
      if (a) {
        S.start[(int)(el[h] >> 32)] = st[k];
        S.pre[(int)(el[h] >> 32)] = (int)(unsigned)el[h];
      } else if (b) {
        S.start[nl + 1 + (int)(es[h] >> 32)] = st[k];
        S.pre[nl + 1 + (int)(es[h] >> 32)] = (int)(unsigned)es[h];
      }
      el[h] += a;
      es[h] += b;
    }
  }
  if (tid == 0) {
    S.nlong = nl;
    S.nshort = (int)(cs >> 32);
    S.pre[nl] = (int)(unsigned)cl;
    S.pre[nl + 1 + (int)(cs >> 32)] = (int)(unsigned)cs;
  }
  block_sync();
}

// index in [a, b) of the last prefix value <= e
__device__ __forceinline__ int seg_of(const int* pre, int e, int a, int b) {
  while (b - a > 1) {
    const int mid = (a + b) >> 1;
    if (pre[mid] <= e) a = mid;
    else b = mid;
  }
  return a;
}

// Calls f(w) for every entry of `n` listed segments, 0xffffffff for lanes
// without one (every caller's range check refuses it).  The warps take equal
// ranges of the concatenated segments, 32 entries at a time over at most 32
// segments: the starts among them, one bit each, number the segments.
template <class T, class F>
__device__ __forceinline__ void walk_short(const T* __restrict__ adj, const int* start, const int* pre, int n, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int L = n > 0 ? pre[n] : 0;
  const int per = (L + kRW - 1) / kRW;
  const int ws = warp * per, we = min(L, ws + per);
  if (ws >= we) return;
  int a = seg_of(pre, ws, 0, n);
  auto group = [&](int e0) {
    const int at = a + 1 + lane < n ? pre[a + 1 + lane] - e0 : 64;
    const unsigned starts = __reduce_or_sync(0xffffffffu, at < 32 ? 1u << at : 0u);
    const int t = a + __popc(starts & (0xffffffffu >> (31 - lane)));
    const int e = e0 + lane;
    const unsigned w = e < we ? (unsigned)__ldg(adj + start[t] + (e - pre[t])) : 0xffffffffu;
    a += __popc(starts) + __any_sync(0xffffffffu, at == 32);
    return w;
  };
  for (int e0 = ws; e0 < we; e0 += 128) {
    unsigned w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = e0 + 32 * k < we ? group(e0 + 32 * k) : 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (e0 + 32 * k < we) f(w[k]);
  }
}

// The long segments, over the lists' low 16 bits (the caller's entries lie in
// one 65,536-id window): f gets an entry's low 16 bits, or 0xffffffff for none.
// 128 entries are one 8-byte load a lane, three rounds of them in flight.
template <class F>
__device__ __forceinline__ void walk_long(const unsigned short* __restrict__ adj, const RankSmem& S, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int* pre = S.pre;
  const int n = S.nlong;
  const int L = n > 0 ? pre[n] : 0;
  const int per = (L + kRW - 1) / kRW;
  const int ws = warp * per, we = min(L, ws + per);
  if (ws >= we) return;
  struct Round {
    uint2 x;
    int g, gs, ge;  // first entry of the round, and the bounds of the segment's share
  };
  int a = seg_of(pre, ws, 0, n);
  int g = 0, gs = 0, ge = 0;
  auto open = [&](int from) {  // segment a from prefix position `from` to this warp's end
    const int b = pre[a], e = pre[a + 1] - kSegmentCost;
    gs = S.start[a] + min(from, e) - b;
    ge = S.start[a] + min(we, e) - b;
    g = gs & ~3;
  };
  open(ws);
  auto skip = [&]() {  // to the next segment with entries for this warp
    while (g >= ge && a + 1 < n && pre[a + 1] < we) {
      a++;
      open(pre[a]);
    }
  };
  skip();
  auto fetch = [&](Round& r) {
    if (g >= ge) return false;
    r.g = g;
    r.gs = gs;
    r.ge = ge;
    r.x = make_uint2(0, 0);
    if (g + 4 * lane < ge) r.x = __ldg(reinterpret_cast<const uint2*>(adj + g + 4 * lane));
    g += 128;
    skip();
    return true;
  };
  auto use = [&](const Round& r) {
    unsigned w[4] = {r.x.x & 0xffffu, r.x.x >> 16, r.x.y & 0xffffu, r.x.y >> 16};
    if (r.g < r.gs || r.g + 128 > r.ge) {
      const int g0 = r.g + 4 * lane;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (g0 + k < r.gs || g0 + k >= r.ge) w[k] = 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) f(w[k]);
  };
  Round r0, r1, r2;
  bool h0 = fetch(r0), h1 = fetch(r1);
  while (h0) {
    const bool h2 = fetch(r2);
    use(r0);
    r0 = r1;
    r1 = r2;
    h0 = h1;
    h1 = h2;
  }
}

// Adds `v` at a shared-memory word when o <= o_max (unsigned), as one
// predicated instruction; the second form returns the word before (0 if not).
__device__ __forceinline__ void shared_add_if(unsigned o, unsigned o_max, unsigned addr, unsigned v) {
  asm volatile("{\n .reg .pred p;\n setp.le.u32 p, %0, %1;\n @p red.shared.add.u32 [%2], %3;\n}\n" ::"r"(o), "r"(o_max),
               "r"(addr), "r"(v)
               : "memory");
}
__device__ __forceinline__ unsigned shared_add_if_old(unsigned o, unsigned o_max, unsigned addr, unsigned v) {
  unsigned old;
  asm volatile(
      "{\n .reg .pred p;\n setp.le.u32 p, %1, %2;\n mov.u32 %0, 0;\n @p atom.shared.add.u32 %0, [%3], %4;\n}\n"
      : "=r"(old)
      : "r"(o), "r"(o_max), "r"(addr), "r"(v)
      : "memory");
  return old;
}

// Residual sums.  When one end carries at most one fringe (lo = 0 or 1, the
// other k >= lo, s shared), choosing k fringes from N(x) and lo from N(y)
// disjointly, without the centre and the shared fringes, leaves
//   lo = 0:  C(dx-1-s, k),   lo = 1:  C(dx-1-s, k) (dy-1-s) - a C(dx-2-s, k-1)
// with a = C-1-s, which equals the sum in wedge() while no binomial of the
// graph's degrees wraps.  Over one owner's pairs the part that depends on the
// owner's degree is constant, so a pair only adds to two sums,
//   A += c_s g(dw)  and  B += c_s (or c_s a),  c_s = C C(C-1, s)  (s = 0: C (C-1)),
// and the owner's end combines them (owner_total).  Other patterns (kGeneral)
// evaluate wedge() per pair.
template <class A>
__device__ __forceinline__ A form_g(const PairForm& f, int d) {
  if (f.kappa < 0) return A(0);
  return f.kappa <= 1 ? A(nck01(d - f.delta, f.kappa)) : nck_a<A>(d - f.delta, f.kappa);
}

// wedge() for a pair by the general loop, C (W(C-1) - W(0)); dx: the end with
// the larger id
template <class A>
__device__ __noinline__ A residual_general(const WedgeParams p, int dx, int dy, int C) {
  if (C <= p.f_vw) return A(0);
  A x = wedge_value<A>(dx, dy, false, p.f_v, p.f_vw, p.f_w, C - 1);
  if (p.f_vw == 0) x -= wedge_value<A>(dx, dy, false, p.f_v, 0, p.f_w, 0);
  return A((u64)C) * x;
}

// What an owner's pairs add up to.
template <class A>
__device__ __forceinline__ A owner_total(const PairForm& f, int dv, A sa, A sb) {
  if (f.kind == kProduct) return A((u64)(dv - f.delta)) * sa - sb;
  const A t = f.kappa < 0 ? sb : form_g<A>(f, dv) * sb + sa;
  return f.sign < 0 ? A(0) - t : t;
}

// One pair by itself (owners counted in tables).
template <class A>
__device__ __noinline__ A pair_total(const RankView& r, const RankSet& rs, int v, int dv, int w, int C) {
  const int dw = __ldg(r.deg + w);
  const PairForm f = rs.form;
  if (f.kind == kGeneral) {
    const bool swap = rs.roles && __ldg(r.oid + w) > __ldg(r.oid + v);
    return residual_general<A>(rs.w, swap ? dw : dv, swap ? dv : dw, C);
  }
  const int c = C - 1, a = c - f.s;
  if (a < 0) return A(0);
  const A cs = f.s <= 1 ? A((u64)C * (u64)c) : A((u64)C) * nck_a<A>(c, f.s);
  return f.kind == kSums ? owner_total<A>(f, dv, cs * form_g<A>(f, dw), cs)
                         : owner_total<A>(f, dv, cs * A((u64)(dw - f.delta)), cs * A((u64)a));
}

__device__ __forceinline__ unsigned hash_slot(int w, int shift) { return ((unsigned)w * 0x9E3779B1u) >> shift; }

// Counts w in an open-addressed table of 2^(32 - shift) slots (keys w + 1);
// returns the count before.  The table is at most half full.
__device__ __forceinline__ unsigned hash_bump(unsigned* keys, unsigned* vals, int w, int shift) {
  const unsigned key = (unsigned)w + 1u, mask = 0xffffffffu >> shift;
  unsigned s = hash_slot(w, shift);
  for (unsigned probe = 0; probe <= mask; probe++) {
    const unsigned k = atomicCAS(keys + s, 0u, key);
    if (k == 0u || k == key) return atomicAdd(vals + s, 1u);
    s = (s + 1) & mask;
  }
  return 0;
}

// Counts the listed segments' entries of the chunk [lo, lo + CH) in S.cnt; ORD:
// returns the 4-cycles closed.  Out of line, like the scans: inlined into the
// kernel the walk spills (two local accesses per add were measured).
template <bool ORD>
__device__ __noinline__ u64 count_chunk(const unsigned short* __restrict__ adj16, RankSmem& S, int lo, int lbits,
                                        unsigned o_max) {
  const int lper = 5 - lbits;
  const unsigned cnt_addr = smem_u32(S.cnt);
  const unsigned cmask = lbits == 5 ? 0xffffffffu : (1u << (1 << lbits)) - 1u;
  u64 closed = 0;
  auto add = [&](unsigned o) {
    const unsigned at = cnt_addr + ((o >> lper) << 2), sh = (o << lbits) & 31u;
    if (ORD) closed += (shared_add_if_old(o, o_max, at, 1u << sh) >> sh) & cmask;
    else shared_add_if(o, o_max, at, 1u << sh);
  };
  const unsigned base = (unsigned)lo & 0xffffu;
  auto low16 = [&](unsigned w) { add(w > 0xffffu ? w : (w - base) & 0xffffu); };
  walk_long(adj16, S, low16);
  walk_short(adj16, S.start + S.nlong + 1, S.pre + S.nlong + 1, S.nshort, low16);
  return closed;
}

// bits above the lowest of every counter (2^lbits wide): non-zero there means 2 or more
__device__ __forceinline__ unsigned two_mask(int lbits) {
  return lbits == 2 ? 0xEEEEEEEEu : lbits == 3 ? 0xFEFEFEFEu : lbits == 4 ? 0xFFFEFFFEu : 0xFFFFFFFEu;
}
// One bit per counter of 2 or more: bit (k << lbits) + i for counter k of word
// i (counters are at least 4 bits wide).
__device__ __forceinline__ unsigned hit_bits(const uint4& x, int lbits) {
  const unsigned two = two_mask(lbits);
  const unsigned low = lbits == 2 ? 0x11111111u : lbits == 3 ? 0x01010101u : lbits == 4 ? 0x00010001u : 1u;
  auto hits = [&](unsigned word) {
    unsigned h = word & two;
    for (int s = 1 << (lbits - 1); s > 0; s >>= 1) h |= h >> s;
    return h & low;
  };
  return hits(x.x) | hits(x.y) << 1 | hits(x.z) << 2 | hits(x.w) << 3;
}

// Every counter of one thread's four words, 2 or more or not (a count of 0 or 1
// adds nothing), against the degrees of its consecutive ids: in dense words
// cheaper than finding the counters of 2 or more.
template <int LB, int KIND, int KAPPA, class A>
__device__ __forceinline__ void dense_words(const int* __restrict__ deg, int delta, int s, const uint4& x, A& sa, A& sb) {
  constexpr int BITS = 1 << LB, N = 32 / BITS;  // counters per word
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const unsigned word = i < 2 ? (i == 0 ? x.x : x.y) : (i == 2 ? x.z : x.w);
    int d[N];
    if constexpr (N >= 4) {
#pragma unroll
      for (int k = 0; k < N; k += 4) {
        const int4 t = __ldg(reinterpret_cast<const int4*>(deg + i * N + k));
        d[k] = t.x;
        d[k + 1] = t.y;
        d[k + 2] = t.z;
        d[k + 3] = t.w;
      }
    } else {
      const int2 t = __ldg(reinterpret_cast<const int2*>(deg + i * N));
      d[0] = t.x;
      d[1] = t.y;
    }
#pragma unroll
    for (int k = 0; k < N; k++) {
      const unsigned C = (word >> (k * BITS)) & ((1u << BITS) - 1u);
      const unsigned cc = C * (C - 1u);  // at most 65,535 * 65,534
      const unsigned g = (unsigned)(d[k] - delta);
      if (KIND == kProduct) {
        sa += A((u64)cc * g);
        sb += A((u64)cc * (C - 1u - (unsigned)s));
      } else {
        if (KAPPA == 1) sa += A((u64)cc * g);
        if (KAPPA == 2) sa += A((u64)cc) * A(((u64)g * (g - 1u)) >> 1);
        sb += A((u64)cc);
      }
    }
  }
}

// Reads and clears the chunk's counters (uint4 words below q1) and returns the
// residuals of every pair of 2 or more common neighbours (kSums, kProduct).
// KAPPA as in PairForm, 3 for any above 2.
template <int KIND, int KAPPA, class A>
__device__ __noinline__ A scan_sums(const int* __restrict__ deg, RankSmem& S, const PairForm f, int dv, int lo, int lbits,
                                    int q1) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lper = 5 - lbits;
  const unsigned cmask = lbits == 5 ? 0xffffffffu : (1u << (1 << lbits)) - 1u;
  const unsigned two = two_mask(lbits);
  // more counters of 2 or more than this in some lane's words: all of them
  const int dense = KAPPA > 2 || f.s > 1 || lbits == 5 ? 64 : lbits == 4 ? 2 : lbits == 3 ? 4 : 8;
  uint4* c4 = reinterpret_cast<uint4*>(S.cnt);
  A sa = A(0), sb = A(0);
  for (int qb = warp * 32; qb < q1; qb += kRT) {
    const int q = qb + lane;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (q < q1) x = c4[q];
    const unsigned all = x.x | x.y | x.z | x.w;
    if (all) c4[q] = make_uint4(0, 0, 0, 0);
    if (!__any_sync(0xffffffffu, (all & two) != 0)) continue;
    unsigned m = hit_bits(x, lbits);
    if (__reduce_max_sync(0xffffffffu, __popc(m)) > dense) {
      const int* d = deg + lo + ((q << 2) << lper);
      if (m) {
        if (lbits == 2) dense_words<2, KIND, KAPPA, A>(d, f.delta, f.s, x, sa, sb);
        else if (lbits == 3) dense_words<3, KIND, KAPPA, A>(d, f.delta, f.s, x, sa, sb);
        else dense_words<4, KIND, KAPPA, A>(d, f.delta, f.s, x, sa, sb);
      }
      continue;
    }
    const int* d = deg + lo + ((q << 2) << lper);
    for (; m; m &= m - 1) {
      const int bit = __ffs(m) - 1, i = bit & 3, k = bit >> lbits;
      const unsigned word = i < 2 ? (i == 0 ? x.x : x.y) : (i == 2 ? x.z : x.w);
      const int C = (int)((word >> (k << lbits)) & cmask);
      const int dw = __ldg(d + (i << lper) + k);
      const int a = C - 1 - f.s;
      if (a < 0) continue;
      const A cs = f.s <= 1 ? A((u64)C * (u64)(C - 1)) : A((u64)C) * nck_a<A>(C - 1, f.s);
      if (KIND == kProduct) {
        sa += cs * A((u64)(dw - f.delta));
        sb += cs * A((u64)a);
      } else {
        if (KAPPA == 1) sa += cs * A((u64)(dw - f.delta));
        else if (KAPPA > 1) sa += cs * nck_a<A>(dw - f.delta, f.kappa);
        sb += cs;
      }
    }
  }
  return owner_total<A>(f, dv, sa, sb);
}

// The same for patterns that evaluate wedge() per pair: the counters of 2 or
// more are staged per warp, so that all lanes evaluate.
template <class A>
__device__ __noinline__ A scan_general(const RankView& r, const RankSet& rs, RankSmem& S, int v, int dv, int lo, int lbits,
                                       int q1, int most) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lper = 5 - lbits;
  const unsigned cmask = lbits == 5 ? 0xffffffffu : (1u << (1 << lbits)) - 1u;
  const unsigned two = two_mask(lbits);
  const bool staged = most < (1 << 14);  // a staged pair: 18 bits of offset, 14 of count
  uint4* c4 = reinterpret_cast<uint4*>(S.cnt);
  unsigned* buf = S.stage[warp];
  int fill = 0;
  A acc = A(0);
  for (int qb = warp * 32; qb < q1; qb += kRT) {
    const int q = qb + lane;
    uint4 x = make_uint4(0, 0, 0, 0);
    if (q < q1) x = c4[q];
    const unsigned all = x.x | x.y | x.z | x.w;
    if (all) c4[q] = make_uint4(0, 0, 0, 0);
    if (!__any_sync(0xffffffffu, (all & two) != 0)) continue;
    unsigned m = hit_bits(x, lbits);
    const int c = __popc(m);
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const int sum = __shfl_sync(0xffffffffu, inc, 31);
    const bool stage = staged && sum <= kRStage - 32;
    int pos = fill + inc - c;
    for (; m; m &= m - 1) {
      const int bit = __ffs(m) - 1, i = bit & 3, k = bit >> lbits;
      const unsigned word = i < 2 ? (i == 0 ? x.x : x.y) : (i == 2 ? x.z : x.w);
      const unsigned C = (word >> (k << lbits)) & cmask;
      const int o = (((q << 2) + i) << lper) + k;
      if (stage) buf[pos++] = ((unsigned)o << 14) | C;
      else acc += pair_total<A>(r, rs, v, dv, lo + o, (int)C);
    }
    if (stage) fill += sum;
    __syncwarp();
    while (fill >= 32) {
      fill -= 32;
      const unsigned y = buf[fill + lane];
      acc += pair_total<A>(r, rs, v, dv, lo + (int)(y >> 14), (int)(y & 0x3fffu));
    }
    __syncwarp();
  }
  if (lane < fill) {
    const unsigned y = buf[lane];
    acc += pair_total<A>(r, rs, v, dv, lo + (int)(y >> 14), (int)(y & 0x3fffu));
  }
  __syncwarp();
  return acc;
}

// One block at a time per owner v (from a queue, heaviest first), w > v only:
//   tiny    (at most 64 centres and 256 wedges) one warp, a 512-slot table;
//   hash    (at most 4,096 wedges) the block, one table over the whole id range;
//   chunks  4- to 32-bit counters, the narrowest that holds the chunk's counts,
//           over at most 16,384 words: 65,536 to 16,384 ids per chunk.
// FULL: counters (table slots) of 2 or more go, 32 at a time and staged per
// warp, through the residual formula as the words are read and cleared.  ORD:
// the centres are restricted to u > v and every add returns the pairs it
// closes, so there is nothing to evaluate.
// What bounds it: instructions and list-read latency, not bytes or adds.  On RMAT
// n = 2^20, 31M entries, the schedulers issue in 62 (ORD) and 64 of 100 cycles with
// half the warps in flight, which wait for list reads (3.1 and 2.0 of a warp's cycles
// an instruction), dependent instructions (2.1, 2.3) and barriers (1.8, 2.5); the
// shared-memory adds, 2.9 cycles a warp and SM where they are random, are 13 and 12 %
// of the time, DRAM 6 and 1.5 % of its rate.  Whole counts there, before -> after, with
// the linear pass (2.3 to 3.2 ms) and the adjacent one (0.3 to 1.1 ms): one fringe on
// each end 344 -> 18 ms (ORD), 4-cycle with opposite fringes 327 -> 87 ms, three
// fringes and one 636 -> 99 ms.  The copy in rank order is built once per graph: 5 ms.
template <bool ORD, class A>
__global__ void __launch_bounds__(kRT, 2) wedge_rank_kernel(const __grid_constant__ RankView r,
                                                            const __grid_constant__ RankSet rs,
                                                            int* __restrict__ queue,
                                                            int* __restrict__ garena, int gstride) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  RankSmem& S = *reinterpret_cast<RankSmem*>(s_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kRWords; i += kRT) S.cnt[i] = 0;
  // ids from `cut` on cannot end a pair of two common neighbours; owners up to
  // `heavy` are taken one by one, the others up to sixteen at a time (fewer on a
  // small graph, where sixteen block-wide owners in a row would be its longest chain)
  const int cut = r.comp ? r.n : ranks_with_degree(r, max(2, rs.lim));
  const int heavy = r.comp ? 0 : min(cut, ranks_with_degree(r, kTinyCentres + 1));
  const int batch = min(kRW, max(1, (cut - heavy) / ((int)gridDim.x * 4)));
  A acc = A(0);
  u64 closed = 0;  // ORD: 4-cycles

  // packed graphs: an owner's sums go to its member's slot
  auto owner_end = [&](int v) {
    if (!r.comp) return;
    u64* slot = r.comp_slots + r.comp[r.oid[v]];
    const A c = warp_sum_a(ORD ? A(closed) * A(rs.mult[0]) : acc);
    if (lane == 0 && c) slot_add(c, slot);
    closed = 0;
    acc = A(0);
  };

  int next = 0;  // thread 0: the item after this one, fetched while this one runs
  if (tid == 0) next = atomicAdd(queue, 1);
  for (;;) {
    block_sync();
    if (tid == 0) {
      S.item = next;
      S.nlist = 0;
    }
    block_sync();
    const int item = S.item;
    if (tid == 0) next = atomicAdd(queue, 1);
    if (item < heavy) {
      if (tid == 0) {
        S.list[0] = item;
        S.nlist = 1;
      }
    } else {
      const long long b0 = (long long)heavy + (long long)(item - heavy) * batch;
      if (b0 >= cut) break;
      const int v = (int)b0 + warp;
      const int dv = warp < batch && v < cut ? r.deg[v] : 0;
      if (dv >= max(2, rs.lim)) {
        const int vb = r.off[v];
        const int cs = ORD ? own_pos(r, v, vb, dv) : 0;
        const int nc = dv - cs;
        bool block = nc > kTinyCentres;
        if (!block && nc >= 2) {
          int st[2] = {0, 0}, len[2] = {0, 0};
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int t = lane + 32 * h;
            if (t < nc) {
              const int u = __ldg(r.adj + vb + cs + t);
              const int ub = r.off[u], du = r.deg[u];
              const int p = min(du, __ldg(r.rev + vb + cs + t));
              st[h] = ub + p;
              len[h] = du - p;
            }
          }
          const int total = __reduce_add_sync(0xffffffffu, min(len[0] + len[1], 1 << 20));
          const int some = __popc(__ballot_sync(0xffffffffu, len[0] > 0)) + __popc(__ballot_sync(0xffffffffu, len[1] > 0));
          if (some >= 2) {
            if (total > kTinyWedges) {
              block = true;
            } else {
              unsigned* keys = S.cnt + warp * 2 * kTinySlots;
              unsigned* vals = keys + kTinySlots;
              int shift = 32 - 5;  // at least 32 slots and twice the wedges
              while ((1 << (32 - shift)) < 2 * total) shift--;
              int* seg = reinterpret_cast<int*>(S.stage[warp]);  // 65 prefix sums, then 64 starts
              const int ex = warp_excl<u64>((u64)(len[0] + len[1]));
              seg[2 * lane] = ex;
              seg[2 * lane + 1] = ex + len[0];
              seg[65 + 2 * lane] = st[0];
              seg[65 + 2 * lane + 1] = st[1];
              if (lane == 31) seg[64] = total;
              __syncwarp();
              for (int e = lane; e < total; e += 32) {
                int a = 0, b = 64;
                while (b - a > 1) {
                  const int mid = (a + b) >> 1;
                  if (seg[mid] <= e) a = mid;
                  else b = mid;
                }
                const int w = __ldg(r.adj + seg[65 + a] + (e - seg[a]));
                if ((unsigned)w < (unsigned)cut) {
                  const unsigned old = hash_bump(keys, vals, w, shift);
                  if (ORD) closed += old;
                }
              }
              __syncwarp();
              const int slots = 1 << (32 - shift);
              for (int i = lane; i < slots; i += 32) {
                const unsigned k = keys[i];
                if (k) {
                  const int C = (int)vals[i];
                  keys[i] = 0;
                  vals[i] = 0;
                  if (!ORD && C >= 2) acc += pair_total<A>(r, rs, v, dv, (int)k - 1, C);
                }
              }
              __syncwarp();
              owner_end(v);
            }
          }
        }
        if (block && lane == 0) S.list[atomicAdd(&S.nlist, 1)] = v;
      }
    }
    block_sync();
    const int nlist = S.nlist;
    for (int li = 0; li < nlist; li++) {
      const int v = S.list[li];
      const int dv = r.deg[v], vb = r.off[v];
      const int cs = ORD ? own_pos(r, v, vb, dv) : 0;
      const int nc = dv - cs;
      const bool big = nc > kRCap;
      int* cur = big ? garena + (size_t)blockIdx.x * 2 * gstride : S.cur;
      int* nxt = big ? cur + gstride : S.nxt;
      if (tid == 0) {
        S.wedges = 0;
        S.centres = 0;
        S.last = -1;
      }
      block_sync();
      {
        unsigned long long sum = 0;
        int some = 0, last = -1;
        for (int t = tid; t < nc; t += kRT) {
          const int u = __ldg(r.adj + vb + cs + t);
          const int ub = r.off[u], du = r.deg[u];
          const int p = min(du, __ldg(r.rev + vb + cs + t));
          cur[t] = ub + p;
          nxt[t] = kDone;
          if (p < du) {
            nxt[t] = __ldg(r.adj + ub + p);
            sum += (unsigned)(du - p);
            some++;
            last = max(last, __ldg(r.adj + ub + du - 1));
          }
        }
        sum = warp_sum_a((u64)sum);
        some = __reduce_add_sync(0xffffffffu, some);
        last = __reduce_max_sync(0xffffffffu, last);
        if (lane == 0 && some) {
          atomicAdd(&S.wedges, sum);
          atomicAdd(&S.centres, some);
          atomicMax(&S.last, last);
        }
      }
      block_sync();
      const unsigned long long wedges = S.wedges;
      const int top = S.last;  // the largest w any centre reaches
      if (S.centres >= 2) {
        if (!big && wedges <= kHashWedges) {
          unsigned* keys = S.cnt;
          unsigned* vals = S.cnt + kHashSlots;
          int shift = 32 - 6;
          while ((1 << (32 - shift)) < 2 * (int)wedges) shift--;
          int st[4], len[4];
#pragma unroll
          for (int k = 0; k < 4; k++) {
            const int t = slot_of(k);
            st[k] = len[k] = 0;
            if (t < nc && nxt[t] != kDone) {
              st[k] = cur[t];
              len[k] = r.off[__ldg(r.adj + vb + cs + t) + 1] - st[k];
            }
          }
          list_segments(S, nc, st, len);
          auto bump = [&](int w) {
            if ((unsigned)w < (unsigned)cut) {
              const unsigned old = hash_bump(keys, vals, w, shift);
              if (ORD) closed += old;
            }
          };
          for (int a = warp; a < S.nlong; a += kRW) {
            const int e = S.start[a] + S.pre[a + 1] - S.pre[a] - kSegmentCost;
            for (int i = S.start[a] + lane; i < e; i += 32) bump(__ldg(r.adj + i));
          }
          walk_short(r.adj, S.start + S.nlong + 1, S.pre + S.nlong + 1, S.nshort, [&](unsigned w) { bump((int)w); });
          block_sync();
          const int slots = 1 << (32 - shift);
          for (int i = tid; i < slots; i += kRT) {
            const unsigned k = keys[i];
            if (k) {
              const int C = (int)vals[i];
              keys[i] = 0;
              vals[i] = 0;
              if (!ORD && C >= 2) acc += pair_total<A>(r, rs, v, dv, (int)k - 1, C);
            }
          }
        } else {
          const int end = min(top, cut - 1);
          int CH = 0;
          for (int lo = (v + 1) / kRGran * kRGran; lo <= end; lo += CH) {
            // counter layout: 2^lbits bits per counter, 2^lper counters per
            // word, CH ids per chunk.  A count exceeds neither the number of
            // centres nor the partner's degree, and degrees descend with the id:
            // the chunks of a hub owner widen towards the low degrees.
            const int most = r.comp ? nc : min(nc, __ldg(r.deg + max(lo, v + 1)));
            const int lbits = most <= 15 ? 2 : most <= 255 ? 3 : most <= 65535 ? 4 : 5;
            const int lper = 5 - lbits;
            CH = min(kRWords << lper, 65536);  // at most one window of the 16-bit lists
            const int hi = lo + CH;
            const int o_max = min(hi - 1, top) - lo;  // the largest offset this chunk may touch
            int here = 0;
            for (int b0 = 0; b0 < nc; b0 += kRCap) {
              const int nb = min(kRCap, nc - b0);
              // Centres with an entry in the chunk, and the segments' ends: the
              // boundary table, or a search of a short list; four loads in
              // flight per step.  A centre whose next entry lies further on
              // costs one load.
              int st[4], len[4], to[4], from[4], x[4], u[4];
#pragma unroll
              for (int k = 0; k < 4; k++) {
                const int t = slot_of(k);
                const bool on = t < nb && nxt[b0 + t] < hi;
                st[k] = on ? cur[b0 + t] : 0;
                u[k] = on ? __ldg(r.adj + vb + cs + b0 + t) : -1;
              }
#pragma unroll
              for (int k = 0; k < 4; k++) {
                to[k] = u[k] >= 0 ? __ldg(r.off + u[k] + 1) : 0;
                x[k] = u[k] >= 0 && u[k] < r.rows && hi <= top ? __ldg(r.tab + (size_t)u[k] * r.K + hi / kRGran) : -1;
              }
              int end_of[4];
#pragma unroll
              for (int k = 0; k < 4; k++) {
                end_of[k] = to[k];
                from[k] = st[k];
                if (x[k] >= 0) to[k] = max(st[k], to[k] - x[k]);
                if (x[k] >= 0 || hi > top) from[k] = to[k];
              }
              while (from[0] < to[0] || from[1] < to[1] || from[2] < to[2] || from[3] < to[3]) {
#pragma unroll
                for (int k = 0; k < 4; k++) x[k] = from[k] < to[k] ? __ldg(r.adj + ((from[k] + to[k]) >> 1)) : hi;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                  const int mid = (from[k] + to[k]) >> 1;
                  if (x[k] < hi) from[k] = mid + 1;
                  else to[k] = mid;
                }
              }
#pragma unroll
              for (int k = 0; k < 4; k++) {
                len[k] = to[k] - st[k];
                // the next entry, for the next chunk: stored after the walk
                x[k] = u[k] >= 0 && to[k] < end_of[k] ? __ldg(r.adj + to[k]) : kDone;
              }
              list_segments(S, nb, st, len);
              here |= S.nlong | S.nshort;
              closed += count_chunk<ORD>(r.adj16, S, lo, lbits, (unsigned)o_max);
              block_sync();
#pragma unroll
              for (int k = 0; k < 4; k++) {
                const int t = slot_of(k);
                if (u[k] < 0) continue;
                cur[b0 + t] = st[k] + len[k];
                nxt[b0 + t] = x[k];
              }
            }
            if (here) {
              // read and clear the words this chunk may have touched
              const int q1 = ((o_max >> lper) >> 2) + 1;
              if (ORD) {
                for (int q = tid; q < q1; q += kRT) reinterpret_cast<uint4*>(S.cnt)[q] = make_uint4(0, 0, 0, 0);
              } else {
                const PairForm& f = rs.form;
                if (f.kind == kGeneral) acc += scan_general<A>(r, rs, S, v, dv, lo, lbits, q1, most);
                else if (f.kind == kProduct) acc += scan_sums<kProduct, 1, A>(r.deg, S, f, dv, lo, lbits, q1);
                else if (f.kappa < 0) acc += scan_sums<kSums, -1, A>(r.deg, S, f, dv, lo, lbits, q1);
                else if (f.kappa == 1) acc += scan_sums<kSums, 1, A>(r.deg, S, f, dv, lo, lbits, q1);
                else if (f.kappa == 2) acc += scan_sums<kSums, 2, A>(r.deg, S, f, dv, lo, lbits, q1);
                else acc += scan_sums<kSums, 3, A>(r.deg, S, f, dv, lo, lbits, q1);
              }
            }
            // the next chunk's (or owner's) first barrier comes before its first add
          }
        }
      }
      owner_end(v);
      block_sync();
    }
  }
  if (ORD) {
    for (int q = 0; q < rs.np; q++) warp_sum_to(A(closed) * A(rs.mult[q]), rs.slot[q]);
  } else {
    warp_sum_to(acc, rs.slot[0]);
  }
}

// ------------------------------------------------------------- rank order
__global__ void rank_degree_keys_kernel(GView g, int maxdeg, unsigned* __restrict__ key, int* __restrict__ val) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    key[v] = (unsigned)(maxdeg - g.deg[v]);
    val[v] = v;
  }
}

__global__ void rank_member_keys_kernel(GView g, const int* __restrict__ val, unsigned* __restrict__ key) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.n; i += gridDim.x * blockDim.x) key[i] = (unsigned)g.comp[val[i]];
}

__global__ void rank_assign_kernel(GView g, const int* __restrict__ oid, int* __restrict__ rank, int* __restrict__ rdeg) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= g.n; r += gridDim.x * blockDim.x) {
    if (r == g.n) {
      rdeg[r] = 0;
      continue;
    }
    const int v = oid[r];
    rank[v] = r;
    rdeg[r] = g.deg[v];
  }
}

// Calls f(r, first, step) for every rank r whose list the thread takes part in, from
// entry `first` on, every `step`-th: the whole grid for the leading ranks with long
// lists (all hubs of an ordinary graph), a warp for every other.  A warp alone took
// 40 ms for the two passes over a list of a million entries, 12 ns an entry and pass.
// The grid's turns take 1 to 2 us each, so rank r has one as long as its list takes
// a warp longer than the r turns before it: two hubs of 30,000 are two turns, a graph
// of lists of 9,000 has forty.
constexpr int kGridList = 4096, kGridTurn = 120;
template <class F>
__device__ __forceinline__ void each_list(const int* __restrict__ rdeg, int n, F f) {
  const int at = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
  int long_lists = 0;
  for (; long_lists < n && rdeg[long_lists] > kGridList + (long long)kGridTurn * long_lists; long_lists++)
    f(long_lists, at, all);
  for (int r = long_lists + (at >> 5); r < n; r += all >> 5) f(r, at & 31, 32);
}

// (neighbour's rank, own rank) per list entry, owners in rank order: a stable
// sort by the first gives every vertex its neighbours' ranks in ascending
// order, because a symmetric graph is its own transpose.
__global__ void rank_entries_kernel(GView g, const int* __restrict__ oid, const int* __restrict__ rank,
                                    const int* __restrict__ roff, const int* __restrict__ rdeg,
                                    unsigned* __restrict__ key, int* __restrict__ val) {
  each_list(rdeg, g.n, [&](int r, int first, int step) {
    const int o = roff[r], d = rdeg[r];
    const int* nb = g.adj + g.off[oid[r]];
    for (int t = first; t < d; t += step) {
      key[o + t] = (unsigned)rank[__ldg(nb + t)];
      val[o + t] = r;
    }
  });
}

// ranks with degree >= 2^(k + 4), k = 0..15 (degrees descend)
__global__ void rank_rows_kernel(const int* __restrict__ rdeg, int n, int* __restrict__ rows) {
  const int d = 1 << (threadIdx.x + 4);
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (rdeg[mid] >= d) lo = mid + 1;
    else hi = mid;
  }
  rows[threadIdx.x] = lo;
}

__global__ void rank_table_kernel(const int* __restrict__ roff, const int* __restrict__ radj, const int* __restrict__ rdeg,
                                  int rows, int K, int* __restrict__ tab) {
  const long long total = (long long)rows * K;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int u = (int)(i / K), k = (int)(i % K);
    const int d = rdeg[u];
    tab[i] = d - lower_bound_dev(radj + roff[u], d, k * kRGran);
  }
}

__global__ void rank_low16_kernel(const int* __restrict__ radj, int m, unsigned short* __restrict__ out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (long long)gridDim.x * blockDim.x)
    out[i] = (unsigned short)radj[i];
}

// entries of N(u) up to and including v, per list entry (v, u)
__global__ void rank_reverse_kernel(const int* __restrict__ roff, const int* __restrict__ radj, const int* __restrict__ rdeg,
                                    int n, const int* __restrict__ tab, int rows, int K, int* __restrict__ rev) {
  each_list(rdeg, n, [&](int v, int first, int step) {
    const int vb = roff[v], d = rdeg[v];
    for (int t = first; t < d; t += step) {
      const int u = __ldg(radj + vb + t), ub = roff[u], du = rdeg[u];
      int lo = 0, hi = du;
      if (u < rows) {  // the boundary table narrows the search
        const int* b = tab + (size_t)u * K + v / kRGran;
        lo = du - __ldg(b);
        hi = du - __ldg(b + 1);
      }
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(radj + ub + mid) <= v) lo = mid + 1;
        else hi = mid;
      }
      rev[vb + t] = lo;
    }
  });
}

int bits_for(unsigned x) {
  int b = 1;
  while (b < 32 && (x >> b)) b++;
  return b;
}

int grid_for(long long work, int tpb, int per_sm) {
  const long long want = (work + tpb - 1) / tpb;
  return (int)std::max(1LL, std::min(want, (long long)sm_count() * per_sm));
}

// log2 of an upper bound of the exact total: wedges times the largest pair formula
double exact_bound_log2(const DevGraph& G, const WedgeParams& p) {
  const double d = std::max(2, G.maxdeg);
  auto lb = [&](int k) { return k * std::log2(d) + 1.0; };  // C(d, k) <= d^k
  return std::log2((double)std::max(2LL, G.m)) + std::log2(d) + lb(p.f_v) + lb(p.f_vw) + lb(p.f_w) + 2.0;
}

PairForm pair_form(const WedgeParams& p, bool exact) {
  const int lo = std::min(p.f_v, p.f_w), k = std::max(p.f_v, p.f_w), s = p.f_vw;
  PairForm f{kGeneral, s, 0, 0, 1};
  if (!exact || lo > 1) return f;
  if (lo == 0) {
    f.kind = kSums;  // C(dx-1-s, k) + C(dy-1-s, k), once for k = 0
    f.kappa = k > 0 ? k : -1;
    f.delta = 1 + s;
  } else if (s == 0) {
    f.kind = kSums;  // -(C-1) (C(dx-2, k-1) + C(dy-2, k-1)), once for k = 1
    f.kappa = k > 1 ? k - 1 : -1;
    f.delta = 2;
    f.sign = -1;
  } else if (k == 1) {
    f.kind = kProduct;  // (dx-1-s) (dy-1-s) - a
    f.kappa = 1;
    f.delta = 1 + s;
  }
  return f;
}

// Binomials of the pattern's sums, the sums with C common neighbours among them.
bool pattern_fits(const DevGraph& G, const WedgeParams& p) {
  return binomials_fit(G.maxdeg, std::max(p.f_v, std::max(p.f_vw, p.f_w)));
}

// Whether the pattern's residual is a multiple of C (C - 1) alone.
bool counts_four_cycles(const WedgeParams& p, long long* mult) {
  if (p.f_v == 1 && p.f_w == 1 && p.f_vw == 0) *mult = -4;       // C ((dx-1)(dy-1) - (C-1))
  else if (p.f_v == 0 && p.f_w == 0 && p.f_vw == 1) *mult = 4;   // C (C-1)
  else return false;
  return true;
}

template <bool ORD, class A>
int launch_rank_set(const RankView& r, const RankSet& rs, const DevGraph& G, cudaStream_t s, uint64_t* launches,
                    DevWork& work) {
  int* queue = reinterpret_cast<int*>(work.small + 7);
  cudaMemsetAsync(queue, 0, sizeof(int), s);
  const size_t smem = sizeof(RankSmem);
  cudaFuncSetAttribute(wedge_rank_kernel<ORD, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  wedge_rank_kernel<ORD, A><<<2 * sm_count(), kRT, smem, s>>>(r, rs, queue, reinterpret_cast<int*>(work.tri.ptr),
                                                                  G.maxdeg);
  *launches += 1;
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

template <class A>
int enqueue_rank_a(DevGraph& G, const GView& gv, const WedgeParams* pats, u64* const* slots, int np, cudaStream_t s,
                   uint64_t* launches, DevWork& work) {
  for (int i = 0; i < np; i++) {
    const WedgeParams& p = pats[i];
    if (p.f_vw == 0) {
      wedge_linear_kernel<A><<<grid_for((long long)G.n * 32, kTPB, 8), kTPB, 0, s>>>(gv, p.f_v, p.f_w, slots[i]);
      *launches += 1;
    }
    wedge_adjacent_kernel<A><<<grid_for(G.m / 2, kTPB, 8), kTPB, 0, s>>>(gv, p, slots[i]);
    *launches += 1;
  }
  if (cudaGetLastError() != cudaSuccess) return FSGC_ECUDA;
  RankView r{G.n, G.roff, G.radj, G.radj16, G.rdeg, G.rrev, G.oid, G.rtab, G.rrows, G.rK, gv.comp, gv.comp_slots};
  RankSet ord;  // the patterns that share one 4-cycle pass
  memset(&ord, 0, sizeof(ord));
  ord.lim = 2;
  int st = FSGC_OK;
  for (int i = 0; i < np && st == FSGC_OK; i++) {
    const WedgeParams& p = pats[i];
    long long mult = 0;
    if (counts_four_cycles(p, &mult)) {
      ord.mult[ord.np] = mult;
      ord.slot[ord.np++] = slots[i];
      if (ord.np < kWedgeFuse) continue;
      st = launch_rank_set<true, A>(r, ord, G, s, launches, work);
      ord.np = 0;
      continue;
    }
    const bool fits = std::is_same<A, u128>::value || pattern_fits(G, p);
    // no shared fringe and none on one end: W does not depend on C, as long as
    // no binomial wraps before its division
    if (fits && p.f_vw == 0 && std::min(p.f_v, p.f_w) == 0) continue;
    RankSet rs;
    memset(&rs, 0, sizeof(rs));
    rs.np = 1;
    rs.w = p;
    rs.lim = p.lim;
    rs.slot[0] = slots[i];
    rs.form = pair_form(p, fits);
    rs.roles = !fits;  // the sum does not depend on which end is which unless a binomial wraps
    st = launch_rank_set<false, A>(r, rs, G, s, launches, work);
  }
  if (st == FSGC_OK && ord.np > 0) st = launch_rank_set<true, A>(r, ord, G, s, launches, work);
  return st;
}

}  // namespace

bool binomials_fit(int maxdeg, int k) {
  return k <= 2 || k * std::log2((double)std::max(2, maxdeg)) - std::lgamma((double)k) / std::log(2.0) < 63.0;
}

WedgePass wedge_pass(const DevGraph& G, const WedgeParams& p, bool exact) {
  long long mult = 0;
  const bool fits = exact || pattern_fits(G, p);
  if (counts_four_cycles(p, &mult) || (fits && p.f_vw == 0 && std::min(p.f_v, p.f_w) == 0)) return kNoPass;
  return pair_form(p, fits).kind == kGeneral ? kPairsPass : kSumsPass;
}

static double wedges_per_pair(const DevGraph& G) { return (double)G.m * G.mean_end_degree / ((double)G.n * (double)G.n); }

// A pair costs the residual two evaluations and the chunk kernel one, which counts up
// to four patterns in one pass: the better where most vertices are pairs with common
// neighbours and none is a large hub.  With R wedges a pair of ids and S the mean
// degree of an entry's vertex over the mean degree (ms, two and two fringes; three and
// three; a set of three such and one other; by chunks and in rank order):
//   uniform, n = 3,000, R = 0.09: 0.20 0.12; 0.22 0.16; 0.40 0.48
//   n = 16,000, R = 0.16: 1.38 1.20; 1.70 1.87; 4.4 5.7   n = 8,000, R = 0.32: 0.70 0.71; 0.86 1.15; 2.1 3.4
//   n = 5,000, R = 8: 0.84 0.97; 1.22 1.71; 2.7 4.8       n = 5,000, R = 0.055: 0.30 0.13; 0.34 0.16; 0.62 0.53
//   RMAT n = 1,024, R = 2, S = 4.7: 0.10 0.14; 0.13 0.22; 0.31 0.62
//   RMAT n = 4,096, R = 1.1, S = 8: 0.31 0.28; 0.42 0.44; 1.10 1.31
//   RMAT n = 16,384, R = 0.6, S = 14: 1.4 1.1; 1.9 1.6; 5.8 5.0
//   cliques of 600 and 1,200, R = n - 1: 0.39 0.26, 2.3 1.1; 0.40 0.29, 2.3 1.2; 0.47 1.03, 2.5 4.5
// Exact counts, one pattern each: uniform, n = 600, R = 4: 0.14 0.37; 0.23 0.70   clique of
// 300: 0.12 0.18; 0.13 0.24   RMAT n = 4,096, 52,000 entries, S = 8: 0.44 0.42; 0.64 0.70
bool pairs_by_chunks(const DevGraph& G, int count, bool exact) {
  if (count == 0 || G.ngraphs > 0 || G.m == 0) return false;
  const double R = wedges_per_pair(G), S = G.mean_end_degree * (double)G.n / (double)G.m;
  return count == 1 ? R >= 0.25 && R <= (exact ? 512 : 256) && S <= 6.5 : R >= 0.08 && S <= 9;
}

// From about 16 wedges a pair of ids (the set above, its fourth pattern in rank order and
// by chunks): cliques of 600 0.68 0.47, of 200 0.16 0.12; uniform R = 67 0.30 0.27,
// R = 27 0.66 0.64, R = 8 2.5 2.7.
bool sums_join_pairs(const DevGraph& G) { return wedges_per_pair(G) >= 16; }

int ensure_rank_order(DevGraph& G, cudaStream_t s, uint64_t* launches, DevWork& work) {
  if (G.radj) return FSGC_OK;
  if (G.lean || G.rank_failed || !wedge_rank_size_ok(G)) return FSGC_EUNSUPPORTED;
  const int n = G.n;
  const int m = (int)G.m;
  const GView gv = G.view();
  unsigned *k1 = nullptr, *k2 = nullptr;
  int *v1 = nullptr, *rank = nullptr, *rows_d = nullptr;
  void* temp = nullptr;
  auto drop = [&](int st) {
    for (void* p : {(void*)k1, (void*)k2, (void*)v1, (void*)rank, (void*)rows_d, temp}) cudaFreeAsync(p, s);
    if (st != FSGC_OK) {
      for (int* p : {G.roff, G.radj, G.rdeg, G.oid, G.rrev, G.rtab}) cudaFreeAsync(p, s);
      cudaFreeAsync(G.radj16, s);
      G.radj16 = nullptr;
      G.roff = G.radj = G.rdeg = G.oid = G.rrev = G.rtab = nullptr;
      G.rrows = G.rK = 0;
      cudaGetLastError();
    }
    return st;
  };
  const size_t big = (size_t)std::max(n + 1, m);
  auto get = [&](void** p, size_t bytes) { return cudaMallocAsync(p, bytes, s) == cudaSuccess; };
  // scratch of the sorts and the scan
  size_t t1 = 0, t2 = 0, t3 = 0;
  const int rank_bits = bits_for((unsigned)n);
  auto room = [&](size_t& bytes, int items, int bits) {
    return cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned*)nullptr, (unsigned*)nullptr, (const int*)nullptr,
                                           (int*)nullptr, items, 0, bits, s) == cudaSuccess;
  };
  if (!room(t1, n, 32) || !room(t2, m, rank_bits) ||
      cub::DeviceScan::ExclusiveSum(nullptr, t3, (const int*)nullptr, (int*)nullptr, n + 1, s) != cudaSuccess)
    return drop(FSGC_ECUDA);
  const size_t tb = std::max(t1, std::max(t2, t3));
  if (!get((void**)&k1, sizeof(unsigned) * big) || !get((void**)&k2, sizeof(unsigned) * big) ||
      !get((void**)&v1, sizeof(int) * big) || !get((void**)&rank, sizeof(int) * (size_t)n) ||
      !get((void**)&rows_d, sizeof(int) * 16) || !get(&temp, tb) || !get((void**)&G.oid, sizeof(int) * (size_t)n) ||
      !get((void**)&G.rdeg, sizeof(int) * ((size_t)n + 1 + 32)) || !get((void**)&G.roff, sizeof(int) * ((size_t)n + 1)) ||
      !get((void**)&G.radj, sizeof(int) * (size_t)m) || !get((void**)&G.rrev, sizeof(int) * (size_t)m) ||
      !get((void**)&G.radj16, sizeof(short) * ((size_t)m + 8))) {
    cudaStreamSynchronize(s);
    drop(FSGC_EUNSUPPORTED);  // no room: the count takes the path without this copy
    cudaStreamSynchronize(s);  // what was had is free again
    G.rank_failed = true;
    note_no_room(G, 3 * sizeof(int) * big + tb + sizeof(int) * ((size_t)4 * n + 64) + (2 * sizeof(int) + sizeof(short)) * (size_t)m);
    return FSGC_EUNSUPPORTED;
  }
  const int vg = grid_for((long long)n + 1, kTPB, 16);
  // every pass indexes with what the sort or scan before it wrote
  auto sort = [&](int* out, int items, int bits) {
    size_t tt = tb;
    return cub::DeviceRadixSort::SortPairs(temp, tt, k1, k2, v1, out, items, 0, bits, s) == cudaSuccess;
  };
  rank_degree_keys_kernel<<<vg, kTPB, 0, s>>>(gv, G.maxdeg, k1, v1);
  if (!sort(G.oid, n, bits_for((unsigned)G.maxdeg))) return drop(FSGC_ECUDA);
  *launches += 1;
  if (gv.comp) {
    if (cudaMemcpyAsync(v1, G.oid, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return drop(FSGC_ECUDA);
    rank_member_keys_kernel<<<vg, kTPB, 0, s>>>(gv, v1, k1);
    if (!sort(G.oid, n, bits_for((unsigned)G.ngraphs))) return drop(FSGC_ECUDA);
    *launches += 1;
  }
  rank_assign_kernel<<<vg, kTPB, 0, s>>>(gv, G.oid, rank, G.rdeg);
  size_t tt = tb;
  if (cub::DeviceScan::ExclusiveSum(temp, tt, G.rdeg, G.roff, n + 1, s) != cudaSuccess) return drop(FSGC_ECUDA);
  rank_entries_kernel<<<grid_for((long long)n * 32, kTPB, 16), kTPB, 0, s>>>(gv, G.oid, rank, G.roff, G.rdeg, k1, v1);
  if (!sort(G.radj, m, rank_bits)) return drop(FSGC_ECUDA);
  *launches += 2;
  // boundary table of the long lists (ordinary graphs; a packed graph's members
  // span few chunks), at most 256 MiB
  int rows[16] = {0};
  G.rK = n / kRGran + 2;
  if (!gv.comp) {
    rank_rows_kernel<<<1, 16, 0, s>>>(G.rdeg, n, rows_d);
    *launches += 1;
    cudaMemcpyAsync(rows, rows_d, sizeof(rows), cudaMemcpyDeviceToHost, s);
  }
  if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess) return drop(FSGC_ECUDA);
  int k = 0;
  while (k < 15 && (size_t)rows[k] * G.rK * sizeof(int) > ((size_t)256 << 20)) k++;
  G.rrows = (size_t)rows[k] * G.rK * sizeof(int) > ((size_t)256 << 20) ? 0 : rows[k];
  if (G.rrows > 0) {
    if (!get((void**)&G.rtab, sizeof(int) * (size_t)G.rrows * G.rK)) {
      cudaGetLastError();
      G.rrows = 0;  // searches instead
    } else {
      rank_table_kernel<<<grid_for((long long)G.rrows * G.rK, kTPB, 16), kTPB, 0, s>>>(G.roff, G.radj, G.rdeg, G.rrows,
                                                                                       G.rK, G.rtab);
      *launches += 1;
    }
  }
  rank_low16_kernel<<<grid_for(m, kTPB, 16), kTPB, 0, s>>>(G.radj, m, G.radj16);
  rank_reverse_kernel<<<grid_for((long long)n * 32, kTPB, 16), kTPB, 0, s>>>(G.roff, G.radj, G.rdeg, n, G.rtab, G.rrows,
                                                                            G.rK, G.rrev);
  *launches += 2;
  G.rank_bytes = sizeof(int) * ((size_t)3 * n + 2 + (size_t)2 * m + (size_t)G.rrows * G.rK) + sizeof(short) * (size_t)m;
  G.bytes += G.rank_bytes;
  drop(FSGC_OK);
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

void free_rank_order(DevGraph& G) {
  for (void* p : {(void*)G.roff, (void*)G.radj, (void*)G.rdeg, (void*)G.oid, (void*)G.rrev, (void*)G.radj16, (void*)G.rtab})
    cudaFree(p);
  G.roff = G.radj = G.rdeg = G.oid = G.rrev = G.rtab = nullptr;
  G.radj16 = nullptr;
  G.rrows = G.rK = 0;
  G.bytes -= G.rank_bytes;
  G.rank_bytes = 0;
}

size_t wedge_rank_scratch(const DevGraph& G) {
  return G.maxdeg > kRCap ? (size_t)2 * sm_count() * 2 * (size_t)G.maxdeg * sizeof(int) : 0;
}

int enqueue_wedge_rank(DevGraph& G, const GView& gv, const WedgeParams* pats, u64* const* slots, int np, bool exact,
                       cudaStream_t s, uint64_t* launches, DevWork& work) {
  if (exact)
    for (int i = 0; i < np; i++)
      if (exact_bound_log2(G, pats[i]) > 126.0) return FSGC_EUNSUPPORTED;
  const int st = ensure_rank_order(G, s, launches, work);
  if (st != FSGC_OK) return st;
  return exact ? enqueue_rank_a<u128>(G, gv, pats, slots, np, s, launches, work)
               : enqueue_rank_a<u64>(G, gv, pats, slots, np, s, launches, work);
}

}  // namespace fsgc
