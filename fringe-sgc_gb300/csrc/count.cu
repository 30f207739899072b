// Counting kernels: one family per core shape of the matching order.
//
// Every kernel evaluates, per core match, the reference's closed-form fringe
// count with the reference's u64 arithmetic (nck_ref) and the reference's
// vertex roles, and adds it into a u64 result slot through a warp -> block ->
// slot reduction.  The per-match formulas are fixed by the reference; what
// changes is how the matches and their Venn sizes are found:
//   vertex core   one pass over the degrees;
//   edge core     one pass over oriented edges, common-neighbour counts taken
//                 from the loader's per-edge triangle supports, binomials in
//                 chains;
//   triangle core bitmap rows per lowest vertex (triangle.cu); here only for
//                 out-degrees beyond its tables;
//   wedge core    (centre without fringes) aggregated per endpoint pair: the
//                 reference evaluates the same formula once per centre, and
//                 the formula does not depend on the centre, so each pair is
//                 evaluated once and multiplied by its number of centres: in
//                 rank order (wedge_rank.cu), here for graphs that do not take
//                 that path;
//                 (centre with fringes) one warp per centre-endpoint edge, on
//                 the bit matrix of a small graph;
//   general core  warp-cooperative depth-first matching of 4-6 core vertices,
//                 a Venn histogram per match and a per-lane placement sum.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "fsgc_formulas.cuh"
#include "fsgc_internal.h"

namespace fsgc {

void upload_div_magic() {
  upload_div_table();
  upload_div_magic_wedge();
  upload_div_magic_triangle();
}

namespace {

// ------------------------------------------------------------- vertex core
template <class A>
__global__ void star_kernel(GView g, int t, u64* __restrict__ slot) {
  A acc = A(0);
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    const int d = g.deg[v];
    if (d >= t) credit(g, acc, nck_a<A>(d, t), v);
  }
  block_sum_to(acc, slot);
}

// ------------------------------------------------------------- edge core
struct EdgeParams {
  int f_u, f_uv, f_v, lim1, lim2;
};


// C(n, 0..K) as nck_ref(n, k) gives them, in one chain: its r after step i is
// C(n, i) with the wrapping of every step, whatever k it is on the way to, and
// below n = 2 k, where it goes to n - k instead, nothing wraps.  n >= 0.
template <int K>
__device__ __forceinline__ void binomial_chain(int n, u64* c) {
  c[0] = 1;
  if constexpr (K >= 1) c[1] = (u64)n;
  if constexpr (K >= 2) c[2] = ((u64)n * (u64)(n - 1)) >> 1;
#pragma unroll
  for (int i = 3; i <= K; i++) c[i] = c[i - 1] * (u64)(n + 1 - i) / (u64)i;
}

// C(n - j, F) as nck_ref gives them, j = 0..J, n >= 0; where j > n any value.
// Up to n = nfit nothing below k = F wraps: C(n - j, k) then follows from
// C(n - j + 1, k) by a subtraction, and only the step to F is done as nck_ref
// does it.
template <int F, int J>
__device__ __forceinline__ void binomial_column(int n, int nfit, u64* t) {
  if constexpr (F <= 2) {
#pragma unroll
    for (int j = 0; j <= J; j++)
      t[j] = F == 0 ? 1ULL : F == 1 ? (u64)(n - j) : ((u64)(n - j) * (u64)(n - j - 1)) >> 1;
  } else if (n <= nfit) {
    u64 c[F];
    binomial_chain<F - 1>(n, c);
#pragma unroll
    for (int j = 0; j <= J; j++) {
      if (j > 0) {
#pragma unroll
        for (int k = 1; k < F; k++) c[k] -= c[k - 1];  // ascending: c[k - 1] is the new row's
      }
      t[j] = c[F - 1] * (u64)(n - j + 1 - F) / (u64)F;
    }
  } else {
    for (int j = 0; j <= J; j++) t[j] = nck(n - j, F);
  }
}

// edge_formula for few fringes, each binomial once: the formula's pool
// a_uv + c_v - j is deg v - 1 - f_uv - j.  Bound by instructions (350 a warp,
// 73 % of the SMs' issue rate; the 12 bytes an edge would take 28 us): five
// fringes on each end, RMAT n = 2^20, 15.7 M edges, 1.42 -> 0.29 ms against the
// loop of nck calls, which lanes leave at different steps.  More than six
// fringes on an end keep the loop: their columns' state would spill.
template <int FU, int FV>
__device__ __forceinline__ u64 edge_formula_chains(int du, int dv, int c_uv, int f_uv, int nfit) {
  const int a_uv = c_uv - f_uv;
  if (a_uv < 0) return 0;
  u64 ku[FU + 1], b[FU + 1], t[FU + 1];
  binomial_chain<FU>(a_uv, b);  // 0 beyond a_uv
  binomial_chain<FU>(du - 1 - c_uv, ku);
  binomial_column<FV, FU>(dv - 1 - f_uv, nfit, t);
  u64 acc = 0;
#pragma unroll
  for (int j = 0; j <= FU; j++) acc += ku[FU - j] * t[j] * b[j];
  if constexpr (FU != FV) {
    binomial_chain<FU>(dv - 1 - c_uv, ku);
    binomial_column<FV, FU>(du - 1 - f_uv, nfit, t);
#pragma unroll
    for (int j = 0; j <= FU; j++) acc += ku[FU - j] * t[j] * b[j];
  }
  return acc * nck(c_uv, f_uv);
}

constexpr int kEdgeChainMax = 6;  // fringes of one endpoint

template <int FU, int FV>
__global__ void __launch_bounds__(kTPB) edge_chain_kernel(GView g, EdgeParams p, int nfit, u64* __restrict__ slot) {
  const long long me = g.m / 2;
  u64 acc = 0;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const int a = g.osrc[j], b = g.oadj[j];
    const int u = max(a, b), v = min(a, b);  // the reference orients by id, v < u
    const int du = g.deg[u], dv = g.deg[v];
    if (!(du > p.lim1 && dv > p.lim1 && du + dv > p.lim2)) continue;  // init_wl_edge pruning
    credit(g, acc, edge_formula_chains<FU, FV>(du, dv, (int)g.osup[j], p.f_uv, nfit), a);
  }
  block_sum_to(acc, slot);
}

template <class A>
__global__ void edge_kernel(GView g, EdgeParams p, u64* __restrict__ slot) {
  const long long me = g.m / 2;
  A acc = A(0);
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const int a = g.osrc[j], b = g.oadj[j];
    const int u = max(a, b), v = min(a, b);  // the reference orients by id, v < u
    const int du = g.deg[u], dv = g.deg[v];
    if (!(du > p.lim1 && dv > p.lim1 && du + dv > p.lim2)) continue;  // init_wl_edge pruning
    credit(g, acc, edge_formula<A>(du, dv, (int)g.osup[j], p.f_u, p.f_uv, p.f_v), a);
  }
  block_sum_to(acc, slot);
}

// triangle with `tails` fringes on one vertex: sum over triangles of the three
// vertex terms = sum over vertices of (triangles at v) * C(deg v - 2, tails)
template <class A>
__global__ void tailed_triangle_kernel(GView g, const u64* __restrict__ vtri2, int tails, u64* __restrict__ slot) {
  A acc = A(0);
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    const u64 t2 = vtri2[v];
    if (t2) credit(g, acc, A(t2 >> 1) * nck_a<A>(g.deg[v] - 2, tails), v);
  }
  block_sum_to(acc, slot);
}

// packed graphs: per-member sum of a per-vertex value (6 x triangles from vtri2)
__global__ void packed_vertex_sum_kernel(GView g, const u64* __restrict__ vals, u64* __restrict__ slot) {
  u64 acc = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x)
    credit(g, acc, vals[v], v);
  block_sum_to(acc, slot);
}

// Vertex- and edge-pass patterns counted together: one pass over the vertices
// (stars, tailed triangles) or the oriented edges (edge-core formulas) adds
// every pattern of the set into its own slot; each term is the single-pattern
// kernel's.  Ordinary graphs and u64 counts only.
constexpr int kPassFuse = 8;
struct VertexSet {
  int np;
  int tailed[kPassFuse];  // 0: star, sum C(deg v, t); 1: tailed triangle, triangles(v) * C(deg v - 2, t)
  int t[kPassFuse];
  u64* slot[kPassFuse];
};

__global__ void vertex_set_kernel(GView g, const u64* __restrict__ vtri2, VertexSet p) {
  u64 acc[kPassFuse];
#pragma unroll
  for (int q = 0; q < kPassFuse; q++) acc[q] = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    const int d = g.deg[v];
    const u64 t2 = vtri2 ? vtri2[v] : 0;
#pragma unroll
    for (int q = 0; q < kPassFuse; q++) {
      if (q >= p.np) break;
      if (p.tailed[q]) {
        if (t2) acc[q] += (t2 >> 1) * nck(d - 2, p.t[q]);
      } else if (d >= p.t[q]) {
        acc[q] += nck(d, p.t[q]);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kPassFuse; q++)
    if (q < p.np) block_sum_to(acc[q], p.slot[q]);
}

struct EdgeSet {
  int np;
  EdgeParams e[kPassFuse];
  u64* slot[kPassFuse];
};

__global__ void edge_set_kernel(GView g, EdgeSet p) {
  const long long me = g.m / 2;
  u64 acc[kPassFuse];
#pragma unroll
  for (int q = 0; q < kPassFuse; q++) acc[q] = 0;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const int a = g.osrc[j], b = g.oadj[j];
    const int u = max(a, b), v = min(a, b);  // the reference orients by id, v < u
    const int du = g.deg[u], dv = g.deg[v];
    const int sup = (int)g.osup[j];
#pragma unroll
    for (int q = 0; q < kPassFuse; q++) {
      if (q >= p.np) break;
      const EdgeParams& e = p.e[q];
      if (du > e.lim1 && dv > e.lim1 && du + dv > e.lim2)  // init_wl_edge pruning
        acc[q] += edge_formula<u64>(du, dv, sup, e.f_u, e.f_uv, e.f_v);
    }
  }
#pragma unroll
  for (int q = 0; q < kPassFuse; q++)
    if (q < p.np) block_sum_to(acc[q], p.slot[q]);
}

// ------------------------------------------------------------- triangle core
// Graphs with out-degrees beyond triangle.cu's tables: triangles by merging
// out-lists, triple overlaps by a warp-cooperative intersection.

// Merge step over two sorted out-lists: advance (i,k) to the next common element.
__device__ __forceinline__ bool next_common(const int* A, int la, const int* B, int lb, int& i, int& k) {
  while (i < la && k < lb) {
    const int x = __ldg(A + i), y = __ldg(B + k);
    if (x < y) i++;
    else if (y < x) k++;
    else return true;
  }
  return false;
}

// warp-cooperative |L0 & L1 & L2| for three sorted lists, iterating the shortest
__device__ int warp_triple(const int* L0, int l0, const int* L1, int l1, const int* L2, int l2) {
  const int lane = threadIdx.x & 31;
  // put the shortest list first
  if (l1 < l0) { const int* t = L0; L0 = L1; L1 = t; int tl = l0; l0 = l1; l1 = tl; }
  if (l2 < l0) { const int* t = L0; L0 = L2; L2 = t; int tl = l0; l0 = l2; l2 = tl; }
  int c = 0;
  for (int i = lane; i < l0; i += 32) {
    const int x = __ldg(L0 + i);
    if (bsearch_has(L1, l1, x) && bsearch_has(L2, l2, x)) c++;
  }
  return __reduce_add_sync(0xffffffffu, c);
}

__device__ __forceinline__ long long tri_key(int x, int d, int relabel) {
  // larger key = later in the reference's vertex order (its new ids ascend
  // with descending (deg, id) after the relabel, with the id otherwise)
  return relabel ? -(((long long)d << 32) | (unsigned)x) : (long long)x;
}

// One lane per oriented edge (a -> b); triangles a < b < c are found by merging
// the out-lists.  Found triangles are served one at a time by the whole warp.
template <class Ar>  // (A and B name out-lists below)
__global__ void triangle_core_kernel(GView g, TrianglePattern p, u64* __restrict__ slot) {
  const int lane = threadIdx.x & 31;
  const long long me = g.m / 2;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  Ar acc = Ar(0);
  for (long long base = ((long long)blockIdx.x * blockDim.x + threadIdx.x - lane); base < me; base += nwarps * 32) {
    const long long j = base + lane;
    bool live = j < me;
    int a = 0, b = 0, la = 0, lb = 0, i = 0, k = 0;
    const int *A = nullptr, *B = nullptr;
    long long aoff = 0, boff = 0;
    if (live) {
      a = g.osrc[j];
      b = g.oadj[j];
      aoff = g.ooff[a];
      boff = g.ooff[b];
      la = (int)(g.ooff[a + 1] - aoff);
      lb = (int)(g.ooff[b + 1] - boff);
      A = g.oadj + aoff;
      B = g.oadj + boff;
    }
    while (__any_sync(0xffffffffu, live)) {
      bool found = false;
      int c = 0;
      if (live) {
        found = next_common(A, la, B, lb, i, k);
        if (!found) live = false;
        else c = A[i];
      }
      if (p.mode != 0) {
        // 4-cliques a < b < c < d: d in out(a) & out(b) & out(c)
        if (found) {
          const long long coff = g.ooff[c];
          const int lc = (int)(g.ooff[c + 1] - coff);
          const int* C = g.oadj + coff;
          for (int t = 0; t < lc; t++) {
            const int d = __ldg(C + t);
            if (bsearch_has(A, la, d) && bsearch_has(B, lb, d)) {
              if (p.mode == 1) credit(g, acc, Ar(1), a);
              else credit(g, acc, nck_a<Ar>(g.deg[a] - 3, p.tails) + nck_a<Ar>(g.deg[b] - 3, p.tails) +
                                  nck_a<Ar>(g.deg[c] - 3, p.tails) + nck_a<Ar>(g.deg[d] - 3, p.tails), a);
            }
          }
        }
      } else {
        // roles: u latest, w earliest in the reference's vertex order
        int x[3], dx[3];
        unsigned sx[3];  // support of the edge opposite... indexed by vertex pair below
        int venn[8];
        bool take = false;
        if (found) {
          x[0] = a; x[1] = b; x[2] = c;
          dx[0] = g.deg[a]; dx[1] = g.deg[b]; dx[2] = g.deg[c];
          // supports of edges ab, ac, bc
          const unsigned s_ab = g.osup[j], s_ac = g.osup[aoff + i], s_bc = g.osup[boff + k];
          // sort the three vertices by key descending: u, v, w
          const int rl = relabel_of(g, p.relabel, a);
          long long kx[3] = {tri_key(a, dx[0], rl), tri_key(b, dx[1], rl), tri_key(c, dx[2], rl)};
          int ord[3] = {0, 1, 2};
          if (kx[ord[0]] < kx[ord[1]]) { int t = ord[0]; ord[0] = ord[1]; ord[1] = t; }
          if (kx[ord[1]] < kx[ord[2]]) { int t = ord[1]; ord[1] = ord[2]; ord[2] = t; }
          if (kx[ord[0]] < kx[ord[1]]) { int t = ord[0]; ord[0] = ord[1]; ord[1] = t; }
          // pair support lookup
          auto sup = [&](int p0, int p1) -> unsigned {
            const int lo = min(p0, p1), hi = max(p0, p1);
            return (lo == 0) ? (hi == 1 ? s_ab : s_ac) : s_bc;
          };
          const int iu = ord[0], iv = ord[1], iw = ord[2];
          const int du = dx[iu], dv = dx[iv], dw = dx[iw];
          // the reference's pruning (init_wl_triangle, common3_triangle)
          const int th1 = max(p.sum1, p.sum2 - du);
          const int th2 = max(max(p.sum1, p.sum3 - du - dv), max(p.sum2 - du, p.sum2 - dv));
          take = (du >= p.sum1) && (dv >= th1) && (dw >= th2);
          venn[IUV] = (int)sup(iu, iv);
          venn[IUW] = (int)sup(iu, iw);
          venn[IVW] = (int)sup(iv, iw);
          venn[IU] = du; venn[IV] = dv; venn[IW] = dw;
          sx[0] = x[iu]; sx[1] = x[iv]; sx[2] = x[iw];
        }
        // triple overlaps, one triangle at a time across the warp
        unsigned bal = __ballot_sync(0xffffffffu, take);
        int c123 = 0;
        while (bal) {
          const int who = __ffs(bal) - 1;
          bal &= bal - 1;
          const int q0 = __shfl_sync(0xffffffffu, (int)sx[0], who);
          const int q1 = __shfl_sync(0xffffffffu, (int)sx[1], who);
          const int q2 = __shfl_sync(0xffffffffu, (int)sx[2], who);
          const long long o0 = g.off[q0], o1 = g.off[q1], o2 = g.off[q2];
          const int r = warp_triple(g.adj + o0, (int)(g.off[q0 + 1] - o0), g.adj + o1, (int)(g.off[q1 + 1] - o1),
                                    g.adj + o2, (int)(g.off[q2 + 1] - o2));
          if (lane == who) c123 = r;
        }
        if (take) {
          // com3 (src/fringeCount.cu:934-964): exclusive regions without the
          // triangle's own vertices
          const int p12 = venn[IUV], t13 = venn[IUW], t23 = venn[IVW];
          const int c12 = p12 - (c123 + 1), c13 = t13 - (c123 + 1), c23 = t23 - (c123 + 1);
          const int du = venn[IU], dv = venn[IV], dw = venn[IW];
          venn[0] = 0;
          venn[IU] = du - (c12 + c13 + (c123 + 2));
          venn[IV] = dv - (c12 + c23 + (c123 + 2));
          venn[IW] = dw - (c13 + c23 + (c123 + 2));
          venn[IUV] = c12; venn[IUW] = c13; venn[IVW] = c23; venn[IUVW] = c123;
          Ar t = Ar(0);
          for (int r = 0; r < p.rot.count; r++) t += fc3<Ar>(p.rot.fr[r], venn);
          credit(g, acc, t, a);
        }
      }
      if (found) { i++; k++; }
    }
  }
  block_sum_to(acc, slot);
}

// ------------------------------------------------------------- wedge core
// Centre without fringes (wedgecore_specialized, src/fringeCount.cu:1409-1477).
// The reference evaluates wedge() once per (centre u, endpoints v > w); the
// value depends only on the endpoints and their centre count C = |N(v) & N(w)|,
// so here each endpoint pair is evaluated once and weighted by C: one block per
// endpoint v (from a queue) counts, for every w < v, the centres u in N(v) with
// w in N(u), with the counts kept in shared memory.  The ids w < v are swept in chunks of CH ids; per chunk every
// centre u in N(v) contributes the segment of N(u) inside the chunk (a cursor
// per centre walks each sorted list once; segment ends are found by galloping
// from the cursor).  The segment lengths are prefix-summed and every warp takes
// a contiguous range of the chunk's elements, following segment boundaries as
// it goes.  Counts go to shared-memory counters; the counters are then scanned,
// the non-zero ones compacted per warp so that every lane evaluates one pair,
// and cleared.  Chunks no centre reaches are skipped.
//
// SMALL (deg v <= kWDvMax): two 16-bit counters per word (a centre count never
// exceeds deg v < 2^16) and the per-centre cursors in shared memory.
// BIG (hub endpoints): 32-bit counters, cursors in a per-block global array.
constexpr int kWDvMax = 2048;
constexpr int kWThreads = 1024;
constexpr int kWGran = 32768;  // ids between the chunk boundaries in the boundary table

// SMALL packs counters of 16, 8 or 4 bits into 32-bit words, the narrowest
// that holds the owner's degree (a count C(v, w) never exceeds deg v), so one
// chunk covers 65,536, 131,072 or 262,144 ids; BIG uses 32-bit counters.
template <bool BIG>
struct WedgeCfg {
  static constexpr int CH = BIG ? 32768 : 65536;   // ids per chunk at 16-bit (BIG: 32-bit) counters
  static constexpr int WORDS = BIG ? CH : CH / 2;  // counter words
  static constexpr int TW = WORDS / 32;            // touched-bitmap words (= kWThreads)
  static constexpr int CH_MAX = BIG ? CH : 4 * CH; // widest chunk (4-bit counters)
};

// One bit, the lowest of the counter, for every non-zero `bits`-wide counter of
// `word` (bits = 4, 8, 16 or 32): each counter's bits are OR-folded into its
// lowest bit.
__device__ __forceinline__ unsigned nonzero_counter_bits(unsigned word, int bits) {
  if (bits == 32) return word != 0u ? 1u : 0u;
  unsigned t = word;
  for (int s = bits >> 1; s > 0; s >>= 1) t |= t >> s;
  return t & (bits == 16 ? 0x00010001u : (bits == 8 ? 0x01010101u : 0x11111111u));
}

// Position of the n-th (from 0) set bit of mask, which has more than n set
// bits: a halving search on the population counts of the low halves.
__device__ __forceinline__ int nth_set_bit(unsigned mask, int n) {
  int pos = 0;
  for (int w = 16; w >= 1; w >>= 1) {
    const int c = __popc(mask & ((1u << w) - 1u));
    if (n >= c) {
      n -= c;
      mask >>= w;
      pos += w;
    }
  }
  return pos;
}

// counter width for an owner of degree dv (SMALL kernel)
__device__ __forceinline__ int wedge_counter_bits(int dv) { return dv <= 15 ? 4 : (dv <= 255 ? 8 : 16); }
static_assert(WedgeCfg<false>::TW == kWThreads && WedgeCfg<true>::TW == kWThreads, "one bitmap word per thread");

// One non-zero counter handed from the counter words to the evaluation: its
// offset o in the chunk and its centre count C.  SMALL: o < 2^18 and
// C <= kWDvMax pack into 32 bits; BIG: 32-bit counts take 64.
template <bool BIG>
struct WedgePair {
  using T = unsigned;
  __device__ static T pack(int o, unsigned c) { return ((unsigned)o << 12) | c; }
  __device__ static int off(T x) { return (int)(x >> 12); }
  __device__ static unsigned count(T x) { return x & 0xfffu; }
};
template <>
struct WedgePair<true> {
  using T = unsigned long long;
  __device__ static T pack(int o, unsigned c) { return ((unsigned long long)o << 32) | c; }
  __device__ static int off(T x) { return (int)(x >> 32); }
  __device__ static unsigned count(T x) { return (unsigned)x; }
};
static_assert(kWDvMax < 4096 && WedgeCfg<false>::CH_MAX <= (1 << 20), "SMALL pairs pack into 32 bits");
constexpr int kPairBuf = 128;  // pairs staged per warp and pass

template <bool BIG>
struct WedgeSmem {
  unsigned cnt[WedgeCfg<BIG>::WORDS];
  unsigned touched[WedgeCfg<BIG>::TW];  // counter words that became non-zero
  int tpre[WedgeCfg<BIG>::TW + 1];      // prefix of touched popcounts
  unsigned adjbits[WedgeCfg<BIG>::CH_MAX / 32];
  long long cur[BIG ? 1 : kWDvMax];
  long long lim[BIG ? 1 : kWDvMax];
  typename WedgePair<BIG>::T pairs[kWThreads / 32][kPairBuf];
  int pre[BIG ? 1 : kWDvMax + 1];
  int warp_tmp[33];
  int v;
  int lo;
  int grab;  // next touched word to evaluate
};
// dynamic shared memory of one block, with 1 KB left for the reductions' static arrays
static_assert(sizeof(WedgeSmem<false>) + 1024 <= 232448 && sizeof(WedgeSmem<true>) + 1024 <= 232448,
              "wedge kernel shared memory");

// Per high-degree vertex u: offsets in N(u) of the first neighbour >= k *
// kWGran, for every k.  A chunk that ends on such a boundary finds the end of
// u's segment with one load instead of a search.
struct ChunkTable {
  const int* id;   // n entries: row of u, or -1
  const int* pos;  // rows of K offsets
  int K;
};

// first index i in [from, to) with a[i] >= x, searching outward from `from`
__device__ __forceinline__ long long gallop_lb(const int* __restrict__ a, long long from, long long to, int x) {
  if (from >= to || __ldg(a + from) >= x) return from;
  long long p = from, step = 1;  // invariant: a[p] < x
  while (p + step < to && __ldg(a + p + step) < x) {
    p += step;
    step <<= 1;
  }
  long long l = p + 1, r = min(p + step, to);  // answer in [l, r]
  while (l < r) {
    const long long m = (l + r) >> 1;
    if (__ldg(a + m) < x) l = m + 1;
    else r = m;
  }
  return l;
}

// block-wide exclusive scan of x[0..n) in place (x[n] = total); every thread calls
template <bool BIG>
__device__ void block_scan_inplace(int* x, int n, WedgeSmem<BIG>& S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  int carry = 0;
  for (int base = 0; base < n; base += 2 * blockDim.x) {
    const int i0 = base + 2 * tid, i1 = i0 + 1;
    const int x0 = (i0 < n) ? x[i0] : 0, x1 = (i1 < n) ? x[i1] : 0;
    const int sum = x0 + x1;
    int inc = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (lane == 31) S.warp_tmp[warp] = inc;
    block_sync();
    if (warp == 0) {
      const int wv = (lane < nwarp) ? S.warp_tmp[lane] : 0;
      int wi = wv;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += y;
      }
      if (lane < nwarp) S.warp_tmp[lane] = wi - wv;
      if (lane == 31) S.warp_tmp[32] = wi;
    }
    block_sync();
    const int ex = carry + S.warp_tmp[warp] + inc - sum;
    if (i0 < n) x[i0] = ex;
    if (i1 < n) x[i1] = ex + x0;
    carry += S.warp_tmp[32];
    block_sync();
  }
  if (tid == 0) x[n] = carry;
}

// Patterns of this core shape counted together: the centre counts C(v, w)
// do not depend on the pattern, so one counting pass serves every pattern of
// the set and each pair is evaluated once per pattern.  lim is the smallest
// endpoint degree any of them takes.
struct WedgeSet {
  int np;
  int lim;
  int small_max;  // endpoints up to this degree go to the SMALL kernel (<= kWDvMax)
  WedgeParams w[kWedgeFuse];
  u64* slot[kWedgeFuse];
};

template <bool BIG, int NP, class A>
__device__ __forceinline__ void eval_pair(const GView& g, const WedgeSet& ws, WedgeSmem<BIG>& S, int o, unsigned C,
                                          int dw, int v, int dv, A* acc) {
  const bool vw = (S.adjbits[o >> 5] >> (o & 31)) & 1u;
#pragma unroll
  for (int q = 0; q < NP; q++) {
    if (q >= ws.np) break;
    const WedgeParams& p = ws.w[q];
    if (dv >= p.lim && dw >= max(p.lim, p.minsum - dv))
      credit(g, acc[q], A((u64)C) * wedge_formula<A>(dv, dw, vw, p.f_v, p.f_vw, p.f_w, (int)C - 1), v);
  }
}

template <bool BIG, int NP, class A>
__global__ void __launch_bounds__(kWThreads, 1) wedge_chunk_kernel(GView g, WedgeSet ws, int* __restrict__ queue,
                                                                   long long* __restrict__ gcur, int* __restrict__ gpre,
                                                                   long long gstride, ChunkTable tab) {
  constexpr int WORDS = WedgeCfg<BIG>::WORDS;
  constexpr int TW = WedgeCfg<BIG>::TW;
  extern __shared__ unsigned char s_raw[];
  WedgeSmem<BIG>& S = *reinterpret_cast<WedgeSmem<BIG>*>(s_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  long long* cur = BIG ? gcur + (size_t)blockIdx.x * 2 * gstride : S.cur;
  long long* lim = BIG ? cur + gstride : S.lim;
  int* pre = BIG ? gpre + (size_t)blockIdx.x * (gstride + 1) : S.pre;
  for (int i = tid; i < WORDS; i += blockDim.x) S.cnt[i] = 0;
  for (int i = tid; i < TW; i += blockDim.x) S.touched[i] = 0;
  for (int i = tid; i < WedgeCfg<BIG>::CH_MAX / 32; i += blockDim.x) S.adjbits[i] = 0;
  A acc[NP];
#pragma unroll
  for (int q = 0; q < NP; q++) acc[q] = A(0);
  for (;;) {
    block_sync();  // every warp has read S.v and, to leave the loop below, S.lo
    if (tid == 0) {
      S.v = atomicAdd(queue, 1);
      S.lo = 0;
    }
    block_sync();
    const int v = S.v;
    if (v >= g.n) break;
    const int dv = g.deg[v];
    if (dv < ws.lim || (BIG ? dv <= ws.small_max : dv > ws.small_max)) continue;
    // counter layout: `bits` per counter, 2^lper counters per word, CH ids per chunk
    const int bits = BIG ? 32 : wedge_counter_bits(dv);
    const int lper = BIG ? 0 : (bits == 16 ? 1 : (bits == 8 ? 2 : 3));
    const int CH = WORDS << lper;
    const long long vb = g.off[v];
    const int* Nv = g.adj + vb;
    for (int t = tid; t < dv; t += blockDim.x) {
      const int u = __ldg(Nv + t);
      cur[t] = g.off[u];
      lim[t] = g.off[u + 1];
    }
    int cv = 0;  // cursor into N(v) for the adjacency marks
    block_sync();
    while (S.lo < v) {
      const int lo = S.lo;  // a multiple of CH
      const int hi = min(lo + CH, v);
      const bool aligned = (hi % kWGran) == 0;
      // segment of each centre's list inside [lo, hi): table lookup for
      // high-degree centres at aligned chunk ends, a gallop from the cursor otherwise
      for (int t = tid; t < dv; t += blockDim.x) {
        const long long c = cur[t];
        long long e = -1;
        if (aligned && tab.id) {
          const int u = __ldg(Nv + t);
          const int row = __ldg(tab.id + u);
          if (row >= 0) e = g.off[u] + __ldg(tab.pos + (size_t)row * tab.K + hi / kWGran);
        }
        if (e < 0) e = gallop_lb(g.adj, c, lim[t], hi);
        pre[t] = (int)(e - c);
      }
      const int cs = cv + lower_bound_dev(Nv + cv, dv - cv, lo);
      const int cend = cs + lower_bound_dev(Nv + cs, dv - cs, hi);
      for (int i = cs + tid; i < cend; i += blockDim.x) {
        const int o = __ldg(Nv + i) - lo;
        atomicOr(&S.adjbits[o >> 5], 1u << (o & 31));
      }
      block_sync();
      block_scan_inplace<BIG>(pre, dv, S);
      block_sync();
      // count: warp-contiguous ranges of the chunk's elements
      {
        const int L = pre[dv];
        const int ws = (int)(((long long)L * warp) / nwarp), we = (int)(((long long)L * (warp + 1)) / nwarp);
        if (ws < we) {
          int a = 0, b = dv;  // last segment with pre <= ws
          while (b - a > 1) {
            const int mid = (a + b) >> 1;
            if (pre[mid] <= ws) a = mid;
            else b = mid;
          }
          for (int e0 = ws; e0 < we; e0 += 32) {
            const int e = e0 + lane;
            int al = a;
            if (e < we) {
              while (pre[al + 1] <= e) al++;
              const int o = __ldg(g.adj + cur[al] + (e - pre[al])) - lo;
              const int wd = o >> lper;
              const unsigned old = atomicAdd(&S.cnt[wd], BIG ? 1u : (1u << ((o & ((1 << lper) - 1)) * bits)));
              if (old == 0) atomicOr(&S.touched[wd >> 5], 1u << (wd & 31));
            }
            a = __shfl_sync(0xffffffffu, al, 31);
          }
        }
      }
      block_sync();
      // evaluate: the chunk's touched counter words are numbered by a prefix
      // over the touched-bitmap words; a warp takes 32 words at a time, one
      // per lane, prefix-sums their non-zero counters, writes
      // them as (offset, centre count) pairs into its shared-memory buffer and
      // then evaluates one pair per lane per step, so the lanes evaluate in
      // lockstep and adjacent lanes take adjacent endpoints.
      {
        const int nw = (hi - lo + (1 << lper) - 1) >> lper;
        const int ntw = (nw + 31) >> 5;
        const int c0 = (tid < ntw) ? __popc(S.touched[tid]) : 0;
        int inc = c0;
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, inc, o);
          if (lane >= o) inc += y;
        }
        if (lane == 31) S.warp_tmp[warp] = inc;
        block_sync();
        if (warp == 0) {
          const int wv = (lane < nwarp) ? S.warp_tmp[lane] : 0;
          int wi = wv;
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
          }
          if (lane < nwarp) S.warp_tmp[lane] = wi - wv;
          if (lane == 31) S.warp_tmp[32] = wi;
        }
        block_sync();
        S.tpre[tid] = S.warp_tmp[warp] + inc - c0;
        const int T = S.warp_tmp[32];
        if (tid == 0) S.grab = 0;
        block_sync();
        const int lbits = BIG ? 5 : (lper == 1 ? 4 : (lper == 2 ? 3 : 2));  // log2(bits)
        const unsigned cmask = BIG ? 0xffffffffu : ((1u << bits) - 1);
        using PT = WedgePair<BIG>;
        typename PT::T* buf = S.pairs[warp];
        // warps take the touched words 32 at a time from a shared counter, so
        // a warp whose words hold more pairs takes fewer of them
        for (;;) {
          int W = 0;
          if (lane == 0) W = atomicAdd(&S.grab, 32);
          W = __shfl_sync(0xffffffffu, W, 0);
          if (W >= T) break;
          const int W1 = min(W + 32, T);
          const int idx = W + lane;
          int wd = 0, c = 0;
          unsigned word = 0, nz = 0;
          if (idx < W1) {
            int a = 0, b = ntw;  // bitmap word holding touched word `idx`: last with tpre <= idx
            while (b - a > 1) {
              const int mid = (a + b) >> 1;
              if (S.tpre[mid] <= idx) a = mid;
              else b = mid;
            }
            wd = (a << 5) + nth_set_bit(S.touched[a], idx - S.tpre[a]);
            word = S.cnt[wd];
            nz = nonzero_counter_bits(word, bits);
            c = __popc(nz);
          }
          int incl = c;
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
          }
          const int excl = incl - c;
          const int P = __shfl_sync(0xffffffffu, incl, 31);
          // pairs excl .. excl + c - 1 are this lane's; a pass stages the
          // pairs [base, base + kPairBuf) and evaluates them
          for (int base = 0; base < P; base += kPairBuf) {
            unsigned mk = nz;
            for (int t = 0; t < c; t++) {
              const int kbit = __ffs(mk) - 1;  // low bit of the counter
              mk &= mk - 1;
              const int pos = excl + t - base;
              if (pos >= 0 && pos < kPairBuf) buf[pos] = PT::pack((wd << lper) + (kbit >> lbits), (word >> kbit) & cmask);
            }
            __syncwarp();
            const int np = min(kPairBuf, P - base);
            for (int i = lane; i < np; i += 32) {
              const typename PT::T x = buf[i];
              const int o = PT::off(x);
              eval_pair<BIG, NP, A>(g, ws, S, o, PT::count(x), __ldg(g.deg + lo + o), v, dv, acc);
            }
            __syncwarp();
          }
        }
      }
      // advance the cursors and find the next id any centre still reaches
      int nxt = 0x7fffffff;
      for (int t = tid; t < dv; t += blockDim.x) {
        const long long c = cur[t] + (pre[t + 1] - pre[t]);
        cur[t] = c;
        if (c < lim[t]) nxt = min(nxt, __ldg(g.adj + c));
      }
      nxt = __reduce_min_sync(0xffffffffu, nxt);
      if (tid == 0) S.lo = v;
      block_sync();  // touched, adjbits, pre and S.lo are free again
      for (int i = tid; i < TW; i += blockDim.x) {
        for (unsigned mk = S.touched[i]; mk; mk &= mk - 1) S.cnt[(i << 5) + __ffs(mk) - 1] = 0;
        S.touched[i] = 0;
      }
      for (int i = cs + tid; i < cend; i += blockDim.x) S.adjbits[(__ldg(Nv + i) - lo) >> 5] = 0;
      cv = cend;
      if (lane == 0 && nxt < v) atomicMin(&S.lo, max(hi, (nxt / CH) * CH));
      block_sync();
    }
  }
#pragma unroll
  for (int q = 0; q < NP; q++)
    if (q < ws.np) block_sum_to(acc[q], ws.slot[q]);
}

// boundary table: pass 1 gives each vertex of degree >= min_deg a row
__global__ void chunk_table_rows_kernel(GView g, int min_deg, int* __restrict__ id, int* __restrict__ rows,
                                        int* __restrict__ nrows) {
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < g.n; u += gridDim.x * blockDim.x) {
    int r = -1;
    if (g.deg[u] >= min_deg) {
      r = atomicAdd(nrows, 1);
      rows[r] = u;
    }
    id[u] = r;
  }
}

// pass 2: row r, column k = first position in N(rows[r]) with neighbour >= k * kWGran
__global__ void chunk_table_fill_kernel(GView g, const int* __restrict__ rows, int nrows, int K, int* __restrict__ pos) {
  const long long total = (long long)nrows * K;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / K), k = (int)(i % K);
    const int u = rows[r];
    const long long b = g.off[u];
    const long long x = (long long)k * kWGran;
    pos[i] = (x > 0x7fffffffLL) ? (int)(g.off[u + 1] - b) : lower_bound_dev(g.adj + b, (int)(g.off[u + 1] - b), (int)x);
  }
}

struct GWedgeParams {
  int min_u, lim, sum1, sum2, sum3;
  Rot3 rot;
  u64 packed[6];  // the rotations' counts, a byte each
};

// Centre with fringes (general_wedge_core, src/fringeCount.cu:1480-1650): one
// warp per centre u, looping over endpoints v in N(u); lanes take w in N(u),
// w < v; open wedges use rotations 0 (and 3), triangles (counted once, with
// u < w < v) use all rotations.
template <class A>
__global__ void wedge_general_kernel(GView g, GWedgeParams p, const unsigned* __restrict__ esup,
                                     u64* __restrict__ slot) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  A acc = A(0);
  // one warp per list entry (u, v): a hub centre's pairs spread over as many
  // warps as it has neighbours
  for (long long j = wid; j < g.m; j += nw) {
    int lo = 0, hi = g.n;  // u = the last vertex with off[u] <= j
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (g.off[mid] <= j) lo = mid;
      else hi = mid;
    }
    const int u = lo;
    const int du = g.deg[u];
    if (du < p.sum1) continue;
    const long long ub = g.off[u];
    const int* Nu = g.adj + ub;
    const int th1u = max(p.sum1, p.sum2 - du);
    {
      const int v = __ldg(g.adj + j);
      const int dv = g.deg[v];
      if (dv < th1u) continue;  // init_wl_wedge
      const int* Nv = g.adj + g.off[v];
      const int p12 = (int)__ldg(esup + j);  // |N(u) & N(v)|
      const bool cond = (du >= p.min_u) && (dv >= p.lim);
      const int thres1 = max(p.lim, p.sum2 - dv);
      const int thres2 = max(max(p.sum1, p.sum3 - du - dv), max(p.sum2 - du, p.sum2 - dv));
      for (int t0 = 0; t0 < du; t0 += 32) {
        const int t = t0 + lane;
        bool active = false, tri = false;
        int w = 0, dw = 0;
        if (t < du) {
          w = __ldg(Nu + t);
          if (w < v) {
            dw = g.deg[w];
            if (dw >= thres2) {
              tri = bsearch_has(Nv, dv, w);
              active = tri ? (u < w) : (cond && dw >= thres1);
            }
          }
        }
        if (!__any_sync(0xffffffffu, t < du && w < v)) break;
        unsigned bal = __ballot_sync(0xffffffffu, active);
        // |N(u) & N(w)| is the support of the entry (u, w); |N(v) & N(w)|
        // and the triple overlap walk the shorter of N(v), N(w)
        const int t13 = active ? (int)__ldg(esup + ub + t) : 0;
        int t23 = 0, t123 = 0;
        while (bal) {
          const int who = __ffs(bal) - 1;
          bal &= bal - 1;
          const int ww = __shfl_sync(0xffffffffu, w, who);
          const int dww = __shfl_sync(0xffffffffu, dw, who);
          const int* Nw = g.adj + g.off[ww];
          const int* S = (dww <= dv) ? Nw : Nv;
          const int* L = (dww <= dv) ? Nv : Nw;
          const int ls = min(dww, dv), ll = max(dww, dv);
          int a23 = 0, a123 = 0;
          for (int q = lane; q < ls; q += 32) {
            const int x = __ldg(S + q);
            if (bsearch_has(L, ll, x)) {
              a23++;
              a123 += bsearch_has(Nu, du, x);
            }
          }
          a23 = __reduce_add_sync(0xffffffffu, a23);
          a123 = __reduce_add_sync(0xffffffffu, a123);
          if (lane == who) { t23 = a23; t123 = a123; }
        }
        if (active) {
          // common3_wedge (src/fringeCount.cu:1480-1510) + corrections
          int venn[8];
          const int c123 = t123, c12 = p12 - c123, c13 = t13 - c123, c23 = t23 - c123;
          venn[0] = 0;
          venn[IU] = du - (p12 + c13);
          venn[IV] = dv - (p12 + c23);
          venn[IW] = dw - (c13 + c23 + c123);
          venn[IUV] = c12; venn[IUW] = c13; venn[IVW] = c23; venn[IUVW] = c123;
          A t = A(0);
          if (tri) {
            venn[IUV]--; venn[IUW]--; venn[IVW]--;
            for (int r = 0; r < p.rot.count; r++) t += fc3<A>(p.rot.fr[r], venn);
          } else {
            venn[IU] -= 2; venn[IVW]--;
            t += fc3<A>(p.rot.fr[0], venn);
            if (p.rot.count > 3) t += fc3<A>(p.rot.fr[3], venn);
          }
          credit(g, acc, t, u);
        }
      }
    }
  }
  block_sum_to(acc, slot);
}

// ------------------------------------------------------------- general core
constexpr int kMaxSlots = 665;  // 3^6 - 2^6: (anchor set, region) pairs for 6 anchors

struct GenParams {
  int k;           // core vertices
  int anchors;     // bitmask of anchoring core vertices
  int nonanchors;  // the other core vertices
  int startdeg;
  uint8_t destdeg[5];
  uint8_t list[5];
  int nslots;
  int lane_venn_max;  // a lane builds its own match's Venn row up to this many list entries
  int grab;           // list entries a warp takes from the queue at a time (1..32)
  uint8_t slot_idx[kMaxSlots];  // region bitmap of each placement step
  uint8_t slot_set[kMaxSlots];  // anchor set index of each step
  uint8_t slot_top[kMaxSlots];  // 1 if the step takes all remaining fringes
  uint8_t fcnt[63];
  uint8_t anch[63];
  int nsets;
  int exact;  // 1: exact placement sum; 0: the reference's functionX
};

// Placement sum over the precomputed step list (exact count of placements):
// step s puts a fringes of its anchor set into region slot_idx[s]; the last
// step of each set takes all its remaining fringes.  Each complete placement
// adds the product of nck(remaining region size, fringes placed).  D bounds
// the number of steps (the host picks the smallest D >= nslots); per step the
// walk keeps the fringes placed, those left and the partial product.
template <int D, class A>
__device__ A placement_sum(const GenParams& p, int* venn) {
  int8_t a_[D];
  uint8_t rem_[D];
  A pre_[D];
  const int S = p.nslots;
  A sum = A(0);
  int s = 0;
  rem_[0] = p.fcnt[p.slot_set[0]];
  pre_[0] = A(1);
  a_[0] = (int8_t)(p.slot_top[0] ? rem_[0] : min(venn[p.slot_idx[0]], (int)rem_[0]));
  while (s >= 0) {
    if (a_[s] < 0) {  // this step is exhausted: back up
      s--;
      if (s >= 0) {
        venn[p.slot_idx[s]] += a_[s];
        a_[s] = p.slot_top[s] ? -1 : a_[s] - 1;
      }
      continue;
    }
    const int idx = p.slot_idx[s];
    const A w = pre_[s] * nck_a<A>(venn[idx], a_[s]);
    if (a_is_zero(w) || s == S - 1) {
      sum += w;
      a_[s] = p.slot_top[s] ? -1 : a_[s] - 1;
      continue;
    }
    venn[idx] -= a_[s];
    const int ns = s + 1;
    pre_[ns] = w;
    rem_[ns] = (uint8_t)(p.slot_top[s] ? (int)p.fcnt[p.slot_set[ns]] : rem_[s] - a_[s]);
    a_[ns] = (int8_t)(p.slot_top[ns] ? rem_[ns] : min(venn[p.slot_idx[ns]], (int)rem_[ns]));
    s = ns;
  }
  return sum;
}

// functionX with the reference's own control flow (src/fringeCount.cu:408-486),
// the default: a flat depth-first walk that saves (a, prod, venn[region],
// fr[set]) per level and, when it backs up, restores only the level it returns
// to.  A region changed by the step it abandons keeps that change, so later
// alternatives can see it reduced; for anchor sets with two or more fringes
// the sum then differs from placement_sum (the exact count), and the
// reference's counts are these sums.  Level s is step s of the host's step
// list, so the region and anchor set of a level come from the table instead of
// the saved state, and D (>= nslots, chosen on the host) bounds the depth:
// 14 bytes of state per level instead of the reference's 21 x 665.
template <int D>
__device__ u64 placement_sum_reference(const GenParams& p, int* venn) {
  int8_t savea[D];
  uint8_t savefr[D];
  int savevenn[D];
  u64 saveprod[D];
  uint8_t fr[64];
  for (int i = 0; i < 64; i++) fr[i] = 0;
  for (int i = 0; i < p.nsets; i++) fr[p.anch[i]] = p.fcnt[i];
  u64 sum = 0, prod = 1;
  int level = 0;
  int a = min(venn[p.slot_idx[0]], (int)fr[p.anch[p.slot_set[0]]]);
  for (;;) {
    const int idx = p.slot_idx[level];
    const int anch = p.anch[p.slot_set[level]];
    const bool top = p.slot_top[level] != 0;
    savea[level] = (int8_t)a; saveprod[level] = prod;
    savevenn[level] = venn[idx]; savefr[level] = fr[anch];
    if (a < 0) {
      prod = 0;
    } else if (top) {
      prod *= nck(venn[idx], fr[anch]);
      venn[idx] -= fr[anch];
      fr[anch] = 0;
      if (p.slot_set[level] == 0) { sum += prod; prod = 0; }
    } else {
      prod *= nck(venn[idx], a);
      venn[idx] -= a;
      fr[anch] = (uint8_t)(fr[anch] - a);
    }
    if (prod == 0) {
      level--;
      if (level < 0) break;
      a = savea[level] - 1;
      prod = saveprod[level];
      venn[p.slot_idx[level]] = savevenn[level];
      fr[p.anch[p.slot_set[level]]] = savefr[level];
    } else {
      level++;
      const int nidx = p.slot_idx[level];
      a = p.slot_top[level] ? 0 : min(venn[nidx], (int)fr[p.anch[p.slot_set[level]]]);
    }
  }
  return sum;
}

constexpr int kGenWarps = 4;  // warps per block in the general-core kernel

struct GenWarp {
  int stack[6];
  int venn[32][65];  // one Venn row per lane (the lane that owns the match); padded against bank conflicts
};

// Exclusive Venn regions of one core match: row[S] = number of vertices whose
// set of adjacent anchor core vertices is exactly S, minus the core vertices
// themselves (commonX, src/fringeCount.cu:345-405, computes the same sizes by
// inclusion-exclusion over every anchor's full list).  Here the anchor with the
// longest list, M, is never walked: every vertex adjacent to M and to another
// anchor is counted from the first other anchor (in core order) it touches,
// and row[{M}] = deg M - those.  Each walked entry needs one membership test
// per other anchor.  `vert(i)` gives the match's vertex at core position i.
// Warp-cooperative (LANES = 32, atomics into row) or by one lane (LANES = 1).
template <int LANES, class VertOf>
__device__ void venn_exclusive(const GView& g, const GenParams& p, VertOf vert, int* row) {
  const int lane = (LANES == 1) ? 0 : (threadIdx.x & 31);
  for (int i = lane; i < 64; i += LANES) row[i] = 0;
  if (LANES > 1) __syncwarp();
  int big = -1, bigdeg = -1;
  for (int i = 0; i < p.k; i++)
    if (p.anchors & (1 << i)) {
      const int d = g.deg[vert(i)];
      if (d >= bigdeg) { big = i; bigdeg = d; }
    }
  for (int i = 0; i < p.k; i++) {
    if (!(p.anchors & (1 << i)) || i == big) continue;
    const int vi = vert(i);
    const long long b = g.off[vi];
    const int d = (int)(g.off[vi + 1] - b);
    for (int t = lane; t < d; t += LANES) {
      const int x = __ldg(g.adj + b + t);
      int bmp = 1 << i;
      bool first = true;
      for (int q = 0; q < p.k && first; q++) {
        if (q == i || !(p.anchors & (1 << q))) continue;
        const int vq = vert(q);
        const long long qb = g.off[vq];
        if (bsearch_has(g.adj + qb, (int)(g.off[vq + 1] - qb), x)) {
          if (q < i && q != big) first = false;  // counted from anchor q
          else bmp |= 1 << q;
        }
      }
      if (first) {
        if (LANES > 1) atomicAdd(row + bmp, 1);
        else row[bmp]++;
      }
    }
  }
  if (LANES > 1) __syncwarp();
  if (lane == 0) {
    int shared_with_big = 0;
    for (int s = 1; s < 64; s++)
      if ((s & (1 << big)) && s != (1 << big)) shared_with_big += row[s];
    row[1 << big] = bigdeg - shared_with_big;
  }
  if (LANES > 1) __syncwarp();
  // core vertices themselves are not fringe candidates
  for (int c = lane; c < p.k; c += LANES) {
    const int x = vert(c);
    int bmp = 0;
    for (int q = 0; q < p.k; q++) {
      if (!(p.anchors & (1 << q))) continue;
      const int vq = vert(q);
      const long long qb = g.off[vq];
      if (bsearch_has(g.adj + qb, (int)(g.off[vq + 1] - qb), x)) bmp |= 1 << q;
    }
    if (bmp) {
      if (LANES > 1) atomicSub(row + bmp, 1);
      else row[bmp]--;
    }
  }
  if (LANES > 1) __syncwarp();
}

// Entries a Venn row walks: the anchors' lists except the longest.
template <class VertOf>
__device__ __forceinline__ int venn_walk_len(const GView& g, const GenParams& p, VertOf vert) {
  int sum = 0, big = 0;
  for (int i = 0; i < p.k; i++)
    if (p.anchors & (1 << i)) {
      const int d = g.deg[vert(i)];
      sum += d;
      big = max(big, d);
    }
  return sum - big;
}

template <int D, class A>
__device__ __forceinline__ A placement_of(const GenParams& p, int* row) {
  if constexpr (std::is_same<A, u64>::value)
    return p.exact ? placement_sum<D, u64>(p, row) : placement_sum_reference<D>(p, row);
  else
    return placement_sum<D, A>(p, row);  // exact counts: exact placements
}

template <int L, int D, class A>
__device__ A gen_level(const GView& g, const GenParams& p, GenWarp& w) {
  // choose stack[L+1] among the neighbours of the first core vertex it must touch
  const int lane = threadIdx.x & 31;
  const int list = p.list[L];
  const int first = __ffs(list) - 1;
  const int src = w.stack[first];
  const long long sb = g.off[src];
  const int sd = (int)(g.off[src + 1] - sb);
  const bool last = (L + 1 == p.k - 1);
  A acc = A(0);
  for (int t0 = 0; t0 < sd; t0 += 32) {
    const int t = t0 + lane;
    bool ok = false;
    int x = -1;
    if (t < sd) {
      x = __ldg(g.adj + sb + t);
      ok = g.deg[x] >= p.destdeg[L];
      for (int q = 0; q <= L && ok; q++) {
        if (list & (1 << q)) {
          if (q != first) {
            const int vq = w.stack[q];
            const long long qb = g.off[vq];
            ok = bsearch_has(g.adj + qb, (int)(g.off[vq + 1] - qb), x);
          }
        } else {
          ok = (w.stack[q] != x);
        }
      }
    }
    if (last) {
      // Venn rows: a lane builds its own when its lists are short, the warp
      // builds the long ones together, one match at a time
      auto vert = [&](int i) { return i == L + 1 ? x : w.stack[i]; };
      const bool alone = ok && venn_walk_len(g, p, vert) <= p.lane_venn_max;
      if (alone) venn_exclusive<1>(g, p, vert, w.venn[lane]);
      unsigned rows = __ballot_sync(0xffffffffu, ok && !alone);
      while (rows) {
        const int who = __ffs(rows) - 1;
        rows &= rows - 1;
        const int xx = __shfl_sync(0xffffffffu, x, who);
        auto vw = [&](int i) { return i == L + 1 ? xx : w.stack[i]; };
        venn_exclusive<32>(g, p, vw, w.venn[who]);
      }
      __syncwarp();
      if (ok) credit(g, acc, placement_of<D, A>(p, w.venn[lane]), w.stack[0]);
      __syncwarp();
    } else {
      unsigned bal = __ballot_sync(0xffffffffu, ok);
      while (bal) {
        const int who = __ffs(bal) - 1;
        bal &= bal - 1;
        const int xx = __shfl_sync(0xffffffffu, x, who);
        if (lane == 0) w.stack[L + 1] = xx;
        __syncwarp();
        if constexpr (L < 4) acc += gen_level<L + 1, D, A>(g, p, w);
        __syncwarp();
      }
    }
  }
  return acc;
}

// One warp per directed edge (u, v) at a time, u = core vertex A and v = core
// vertex B (the reference's worklist of general_core_level0,
// src/fringeCount.cu:567-663, with its degree pruning): warps take p.grab
// (1..32) consecutive list entries from a queue, find their owners in
// parallel and then walk each entry's matches.  Work is spread per edge, so a
// hub's edges go to many warps; on small graphs a warp takes one edge at a
// time, so that every warp of the GPU has work.
template <int D, class A>
__global__ void __launch_bounds__(kGenWarps * 32) general_core_kernel(GView g, const __grid_constant__ GenParams p,
                                                                       unsigned long long* __restrict__ queue,
                                                                       u64* __restrict__ slot) {
  __shared__ GenWarp sw[kGenWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  GenWarp& w = sw[warp];
  A acc = A(0);
  const unsigned long long m = (unsigned long long)g.m;
  for (;;) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(queue, (unsigned long long)p.grab);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= m) break;
    const long long j = (long long)base + lane;
    bool ok = lane < p.grab && j < (long long)m;
    int u = 0, v = 0;
    if (ok) {
      int lo = 0, hi = g.n;  // owner: the last vertex with off[u] <= j
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (g.off[mid] <= j) lo = mid;
        else hi = mid;
      }
      u = lo;
      v = __ldg(g.adj + j);
      ok = g.deg[u] >= p.startdeg && g.deg[v] >= p.destdeg[0];  // init_wl_general
    }
    unsigned bal = __ballot_sync(0xffffffffu, ok);
    while (bal) {
      const int who = __ffs(bal) - 1;
      bal &= bal - 1;
      const int uu = __shfl_sync(0xffffffffu, u, who), vv = __shfl_sync(0xffffffffu, v, who);
      if (lane == 0) { w.stack[0] = uu; w.stack[1] = vv; }
      __syncwarp();
      acc += gen_level<1, D, A>(g, p, w);
      __syncwarp();
    }
  }
  block_sum_to(acc, slot);
}

// ---- general core on a bit matrix (graphs of at most kBitsMaxN vertices)
//
// Row v of the matrix is N(v), one bit per vertex.  A candidate is then checked
// with one bit per core vertex it must (not) touch, where the lists need a
// binary search each, and the number of vertices adjacent to a set of anchors is
// a popcount of their rows' AND.  The rows of the anchors before the last core
// vertex are ANDed once per partial match (without the core vertices), so a
// match costs one pass over its own row per set that its formula needs:
//   few     at most three fringes, one per anchor set: the sets and their
//           unions, F1 F2 - F12 and its three-set counterpart;
//   others  all sets of anchors (at most four), turned into exclusive regions
//           for the placement walk.
// Bound by instructions (popcounts, the walk).  RMAT n = 512, 14,000 entries: a
// five-vertex core with a chord fringe 45 -> 0.5 ms, a 4-path with three
// fringes 57 -> 0.5 ms; n = 1,500: 45 -> 0.95 ms.  Up to 4,096 vertices the matrix
// stays under 2 MiB and a row within the four words a lane that the wedge core
// keeps in registers.
constexpr int kBitsMaxN = 4096;
constexpr int kBitsMaxAnchors = 4;  // for the placement walk
constexpr int kBitsMaxSets = 15;

struct BitSets {
  int few;                       // fringes counted by inclusion-exclusion (0: placement walk)
  int twice;                     // few: the reference's walk starts with its all-anchor step and repeats it
  int nsets;                     // anchor sets whose common neighbours are counted
  uint8_t set[kBitsMaxSets];     // as core bitmaps
  int8_t term[7];                // few: index of F1, F2, F12, F3, F13, F23, F123
  int parts;                     // ways a list entry's third vertices are split over tasks
  int words;                     // matrix words per row (a multiple of 4)
};

struct BitWarp {
  int stack[6];
  int before[kBitsMaxSets];  // common neighbours of a set's earlier anchors
  int venn[32][65];
};

template <int L, int D, class A>
__device__ A bits_level(const GView& g, const GenParams& p, const BitSets& bs, const unsigned* __restrict__ mat, BitWarp& w,
                        unsigned* rows, int part) {
  const int lane = threadIdx.x & 31;
  const int words = bs.words;
  const int list = p.list[L];
  const int src = w.stack[__ffs(list) - 1];
  const long long sb = g.off[src];
  const int sd = (int)(g.off[src + 1] - sb);
  const bool last = (L + 1 == p.k - 1);
  const int xbit = 1 << (L + 1);
  A acc = A(0);
  if (last) {
    // per set: the AND of its earlier anchors' rows without the core vertices
    for (int q = 0; q < bs.nsets; q++) {
      const int early = bs.set[q] & ~xbit;
      int c = 0;
      if (early) {
        for (int i = lane; i < words; i += 32) {
          unsigned x = 0xffffffffu;
          for (int a = 0; a <= L; a++) {
            const int va = w.stack[a];
            if (early >> a & 1) x &= __ldg(mat + (size_t)va * words + i);
            if (va >> 5 == i) x &= ~(1u << (va & 31));
          }
          rows[q * words + i] = x;
          c += __popc(x);
        }
      }
      c = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0) w.before[q] = c;
    }
    __syncwarp();
  }
  for (int t0 = 0; t0 < sd; t0 += 32) {
    const int t = t0 + lane;
    bool ok = false;
    int x = 0;
    if (t < sd && (L > 1 || t % bs.parts == part)) {
      x = __ldg(g.adj + sb + t);
      ok = g.deg[x] >= p.destdeg[L];
      for (int q = 0; q <= L && ok; q++) {
        const int vq = w.stack[q];
        ok = (list >> q & 1) ? (__ldg(mat + (size_t)vq * words + (x >> 5)) >> (x & 31)) & 1u : vq != x;
      }
    }
    if (last) {
      if (ok) {
        const uint4* mx = reinterpret_cast<const uint4*>(mat + (size_t)x * words);
        int* row = w.venn[lane];
        for (int q = 0; q < bs.nsets; q++) {
          const int set = bs.set[q], early = set & ~xbit;
          int c;
          if (!(set & xbit)) {
            c = w.before[q] - (int)((rows[q * words + (x >> 5)] >> (x & 31)) & 1u);
          } else if (early == 0) {
            c = g.deg[x];
            for (int a = 0; a <= L; a++) {
              const int va = w.stack[a];
              c -= (int)((__ldg(mat + (size_t)x * words + (va >> 5)) >> (va & 31)) & 1u);
            }
          } else {
            const uint4* r4 = reinterpret_cast<const uint4*>(rows + q * words);
            c = 0;
            for (int i = 0; i < words / 4; i++) {
              const uint4 a = __ldg(mx + i), b = r4[i];
              c += (__popc(a.x & b.x) + __popc(a.y & b.y)) + (__popc(a.z & b.z) + __popc(a.w & b.w));
            }
          }
          row[set] = c;
        }
        A f;
        if (bs.few > 0) {
          // below 2^36, and never negative: exact in any arithmetic
          auto at = [&](int i) { return (u64)row[bs.set[bs.term[i]]]; };
          u64 few = at(0);
          if (bs.few == 2) few = at(0) * at(1) - at(2);
          if (bs.few == 3) few = at(0) * at(1) * at(3) - at(0) * at(5) - at(1) * at(4) - at(3) * at(2) + 2 * at(6);
          f = A(bs.twice ? 2 * few : few);
        } else {
          // common neighbours of every set -> exclusive regions
          row[0] = 0;
          for (int a = 0; a < p.k; a++) {
            if (!(p.anchors >> a & 1)) continue;
            for (int q = 0; q < bs.nsets; q++) {
              const int set = bs.set[q];
              if (!(set >> a & 1)) row[set] -= row[set | 1 << a];
            }
          }
          f = placement_of<D, A>(p, row);
        }
        credit(g, acc, f, w.stack[0]);
      }
      __syncwarp();
    } else {
      unsigned bal = __ballot_sync(0xffffffffu, ok);
      while (bal) {
        const int who = __ffs(bal) - 1;
        bal &= bal - 1;
        const int xx = __shfl_sync(0xffffffffu, x, who);
        if (lane == 0) w.stack[L + 1] = xx;
        __syncwarp();
        if constexpr (L < 4) acc += bits_level<L + 1, D, A>(g, p, bs, mat, w, rows, part);
        __syncwarp();
      }
    }
  }
  return acc;
}

// One warp per (list entry, part) task, from a queue.
template <int D, class A>
__global__ void __launch_bounds__(kGenWarps * 32) general_bits_kernel(GView g, const __grid_constant__ GenParams p,
                                                                       const __grid_constant__ BitSets bs,
                                                                       const unsigned* __restrict__ mat,
                                                                       unsigned long long* __restrict__ queue,
                                                                       u64* __restrict__ slot) {
  extern __shared__ __align__(16) unsigned s_rows[];
  __shared__ BitWarp sw[kGenWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  BitWarp& w = sw[warp];
  unsigned* rows = s_rows + (size_t)warp * bs.nsets * bs.words;
  A acc = A(0);
  const unsigned long long tasks = (unsigned long long)g.m * (unsigned)bs.parts;
  for (;;) {
    unsigned long long task = 0;
    if (lane == 0) task = atomicAdd(queue, 1ULL);
    task = __shfl_sync(0xffffffffu, task, 0);
    if (task >= tasks) break;
    const long long j = (long long)(task / (unsigned)bs.parts);
    int lo = 0, hi = g.n;  // owner: the last vertex with off[u] <= j
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (g.off[mid] <= j) lo = mid;
      else hi = mid;
    }
    const int v = __ldg(g.adj + j);
    if (g.deg[lo] < p.startdeg || g.deg[v] < p.destdeg[0]) continue;  // init_wl_general
    if (lane == 0) {
      w.stack[0] = lo;
      w.stack[1] = v;
    }
    __syncwarp();
    acc += bits_level<1, D, A>(g, p, bs, mat, w, rows, (int)(task % (unsigned)bs.parts));
    __syncwarp();
  }
  block_sum_to(acc, slot);
}

__global__ void bit_matrix_kernel(GView g, int words, unsigned* __restrict__ mat) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
  for (int v = wid; v < g.n; v += nw) {
    const long long b = g.off[v];
    for (int t = lane; t < g.deg[v]; t += 32) {
      const int x = __ldg(g.adj + b + t);
      if ((unsigned)x < (unsigned)g.n) atomicOr(mat + (size_t)v * words + (x >> 5), 1u << (x & 31));
    }
  }
}

int bit_matrix_words(int n) { return ((n + 31) / 32 + 3) & ~3; }
size_t bit_matrix_bytes(const DevGraph& G) { return sizeof(unsigned) * (size_t)G.n * bit_matrix_words(G.n); }

// The adjacency bit matrix of a small graph, once per graph (at most 2 MiB).
// FSGC_EUNSUPPORTED when the graph is larger or there was no room for it: the
// caller takes the lists.
int ensure_bit_matrix(DevGraph& G, cudaStream_t s, uint64_t* launches) {
  if (G.bits) return FSGC_OK;
  if (G.lean || G.bits_failed || G.n > kBitsMaxN) return FSGC_EUNSUPPORTED;
  const size_t bytes = bit_matrix_bytes(G);
  if (cudaMallocAsync((void**)&G.bits, bytes, s) != cudaSuccess) {
    cudaGetLastError();
    G.bits = nullptr;
    G.bits_failed = true;
    note_no_room(G, bytes);
    return FSGC_EUNSUPPORTED;
  }
  cudaMemsetAsync(G.bits, 0, bytes, s);
  bit_matrix_kernel<<<std::max(1, std::min(G.n / 8 + 1, sm_count() * 8)), 256, 0, s>>>(G.view(), bit_matrix_words(G.n), G.bits);
  *launches += 1;
  G.bytes += bytes;
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

// The sets a pattern needs counted, or false when it takes the list kernel.  With
// one fringe per set the reference's walk is exact but for one case: when its
// first step is the all-anchor one and other sets follow, that step's saved
// alternative starts at 1 instead of 0 and the walk below it runs twice.
bool bit_sets_for(const GenParams& p, bool exact, int n, BitSets& bs) {
  if (n > kBitsMaxN) return false;
  memset(&bs, 0, sizeof(bs));
  bs.words = bit_matrix_words(n);
  bool ones = p.nsets <= 3;
  for (int i = 0; i < p.nsets; i++) ones = ones && p.fcnt[i] == 1;
  auto need = [&](int set) {
    for (int q = 0; q < bs.nsets; q++)
      if (bs.set[q] == set) return q;
    bs.set[bs.nsets] = (uint8_t)set;
    return bs.nsets++;
  };
  if (ones) {
    bs.few = p.nsets;
    bs.twice = !exact && p.nsets > 1 && p.slot_top[0];
    const int a = p.anch[0], b = p.nsets > 1 ? p.anch[1] : 0, c = p.nsets > 2 ? p.anch[2] : 0;
    const int sets[7] = {a, b, a | b, c, a | c, b | c, a | b | c};
    const bool used[7] = {true, p.nsets > 1, p.nsets > 1, p.nsets > 2, p.nsets > 2, p.nsets > 2, p.nsets > 2};
    for (int i = 0; i < 7; i++)
      if (used[i]) bs.term[i] = (int8_t)need(sets[i]);
    return true;
  }
  if (__builtin_popcount(p.anchors) > kBitsMaxAnchors) return false;
  for (int set = 1; set < 64; set++)
    if ((set & ~p.anchors) == 0) need(set);
  return true;
}

// Parts that a list entry's third vertices are split into: enough tasks for the
// warps to end together, but fewer than the longest list has entries and than four
// times those of the lists that entries lie in on average, where most parts are
// empty.  Split 32 ways whatever the lists, a path of 4,096 took 0.20 ms (searching
// lists 0.03 ms, now 0.03 ms), a square grid 0.27 ms (0.21, now 0.12).
int bits_parts(const DevGraph& G, long long warps) {
  const double most = std::min((double)G.maxdeg, 4 * G.mean_end_degree);
  int parts = 1;
  while (parts < 32 && 2 * parts < most && G.m * parts < warps * 32) parts *= 2;
  return parts;
}

template <int D, class A>
int launch_bits(const GView& gv, const GenParams& gp, BitSets bs, const unsigned* mat, unsigned long long* queue, u64* slot,
                int blocks, cudaStream_t s) {
  const size_t smem = sizeof(unsigned) * (size_t)kGenWarps * bs.nsets * bs.words;
  cudaFuncSetAttribute(general_bits_kernel<D, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  general_bits_kernel<D, A><<<blocks, kGenWarps * 32, smem, s>>>(gv, gp, bs, mat, queue, slot);
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

// ---- wedge core with a fringed centre on the bit matrix
//
// The matches, thresholds and values of wedge_general_kernel, whose time went
// into walking the shorter of N(v), N(w) with two binary searches per entry for
// every match.  Here the warp of a list entry (u, v) keeps the rows of v and of
// N(u) & N(v) in registers, and a match costs its row once, read together, and
// two popcounts a word; the lanes' matches are then evaluated at one place.
// Bound by instructions (60 % of the issue rate, 44 % of the warps in flight).
// One fringe on each of the three, RMAT n = 3,001, 16 entries a vertex: 3.93 ms
// -> 0.39 ms by fc3_ring in line, 0.25 ms by the products.
// NW: words of a row per lane.  FORM: 0 fc3; while no binomial wraps, 1 when the
// fringes on single core vertices are at most one each and there are none on
// pairs (products), 2 fc3_ring otherwise, out of line: its loops spill.
__device__ __noinline__ u64 fc3_ring_call(u64 fr, int r, int uv, int uw, int vw, int xu, int xv, int xw) {
  int f[8];
#pragma unroll
  for (int i = 0; i < 8; i++) f[i] = (int)(fr >> (8 * i) & 0xff);
  return fc3_ring(f, r, uv, uw, vw, xu, xv, xw);
}

// fc3_ring with at most one fringe on each core vertex and none on pairs.
__device__ __forceinline__ u64 fc3_ones(const int* fr, int r, int uv, int uw, int vw, int xu, int xv, int xw) {
  const int fuvw = fr[IUVW];
  if (r < fuvw) return 0;
  const u64 base = nck(r, fuvw);
  r -= fuvw;
  const u64 a = (u64)(unsigned)(r + uv + uw + xu), b = (u64)(unsigned)(r + uv + vw + xv), c = (u64)(unsigned)(r + uw + vw + xw);
  const u64 ab = (u64)(unsigned)(r + uv), ac = (u64)(unsigned)(r + uw), bc = (u64)(unsigned)(r + vw);
  u64 x = fr[IU] ? a : 1;
  if (fr[IV]) x *= b;
  if (fr[IW]) x *= c;
  // less the choices that coincide
  if (fr[IU] & fr[IV]) x -= ab * (fr[IW] ? c : 1);
  if (fr[IU] & fr[IW]) x -= ac * (fr[IV] ? b : 1);
  if (fr[IV] & fr[IW]) x -= bc * (fr[IU] ? a : 1);
  if (fr[IU] & fr[IV] & fr[IW]) x += 2ULL * (u64)(unsigned)r;
  return base * x;
}

template <int NW, int FORM, class A>
__global__ void __launch_bounds__(kTPB) wedge_bits_kernel(GView g, const __grid_constant__ GWedgeParams p, const unsigned* __restrict__ esup,
                                                           const unsigned* __restrict__ mat, int words,
                                                           u64* __restrict__ slot) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  A acc = A(0);
  for (long long j = wid; j < g.m; j += nw) {
    int lo = 0, hi = g.n;  // u = the last vertex with off[u] <= j
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (g.off[mid] <= j) lo = mid;
      else hi = mid;
    }
    const int u = lo, v = __ldg(g.adj + j);
    const int du = g.deg[u], dv = g.deg[v];
    if (du < p.sum1 || dv < max(p.sum1, p.sum2 - du)) continue;  // init_wl_wedge
    const long long ub = g.off[u];
    const unsigned* row_v = mat + (size_t)v * words;
    unsigned bv[NW], buv[NW];
#pragma unroll
    for (int i = 0; i < NW; i++) {
      const int word = i * 32 + lane;
      bv[i] = word < words ? __ldg(row_v + word) : 0;
      buv[i] = word < words ? bv[i] & __ldg(mat + (size_t)u * words + word) : 0;
    }
    const int p12 = (int)__ldg(esup + j);  // |N(u) & N(v)|
    const bool cond = (du >= p.min_u) && (dv >= p.lim);
    const int thres1 = max(p.lim, p.sum2 - dv);
    const int thres2 = max(max(p.sum1, p.sum3 - du - dv), max(p.sum2 - du, p.sum2 - dv));
    const int ahead = (int)(j - ub);  // w < v: the entries before v's
    for (int t0 = 0; t0 < ahead; t0 += 32) {
      const int t = t0 + lane;
      bool active = false, tri = false;
      int w = 0, dw = 0, t13 = 0;
      if (t < ahead) {
        w = __ldg(g.adj + ub + t);
        dw = g.deg[w];
        if (dw >= thres2) {
          tri = (__ldg(row_v + (w >> 5)) >> (w & 31)) & 1u;
          active = tri ? (u < w) : (cond && dw >= thres1);
        }
        t13 = (int)__ldg(esup + ub + t);
      }
      unsigned bal = __ballot_sync(0xffffffffu, active);
      int both = 0;  // |N(v) & N(w)| and, above 16 bits, |N(u) & N(v) & N(w)|
      while (bal) {
        const int who = __ffs(bal) - 1;
        bal &= bal - 1;
        const unsigned* row_w = mat + (size_t)__shfl_sync(0xffffffffu, w, who) * words;
        int c = 0;
#pragma unroll
        for (int i = 0; i < NW; i++) {
          const int word = i * 32 + lane;
          const unsigned x = word < words ? __ldg(row_w + word) : 0;
          c += __popc(x & bv[i]) + (__popc(x & buv[i]) << 16);
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == who) both = c;
      }
      if (!__any_sync(0xffffffffu, active)) continue;
      // common3_wedge (src/fringeCount.cu:1480-1510) + corrections
      const int c123 = both >> 16, c12 = p12 - c123, c13 = t13 - c123, c23 = (both & 0xffff) - c123;
      int xu = du - (p12 + c13), xv = dv - (p12 + c23), xw = dw - (c13 + c23 + c123);
      int uv = c12, uw = c13, vw = c23;
      if (tri) {
        uv--; uw--; vw--;
      } else {
        xu -= 2; vw--;
      }
      A sum = A(0);
#pragma unroll 1
      for (int r = 0; r < p.rot.count; r++) {
        if (!active || !(tri || r == 0 || r == 3)) continue;
        if constexpr (FORM == 1) {
          sum += fc3_ones(p.rot.fr[r], c123, uv, uw, vw, xu, xv, xw);
        } else if constexpr (FORM == 2) {
          sum += fc3_ring_call(p.packed[r], c123, uv, uw, vw, xu, xv, xw);
        } else {
          const int venn[8] = {0, xu, xv, uv, xw, uw, vw, c123};
          sum += fc3<A>(p.rot.fr[r], venn);
        }
      }
      if (active) credit(g, acc, sum, u);
    }
  }
  block_sum_to(acc, slot);
}

template <int NW, class A>
void launch_wedge_bits(const GView& gv, const GWedgeParams& gp, const unsigned* esup, const unsigned* mat, int words,
                       int form, u64* slot, int blocks, cudaStream_t s) {
  if constexpr (std::is_same<A, u64>::value) {
    if (form == 1) wedge_bits_kernel<NW, 1, A><<<blocks, kTPB, 0, s>>>(gv, gp, esup, mat, words, slot);
    if (form == 2) wedge_bits_kernel<NW, 2, A><<<blocks, kTPB, 0, s>>>(gv, gp, esup, mat, words, slot);
    if (form != 0) return;
  }
  wedge_bits_kernel<NW, 0, A><<<blocks, kTPB, 0, s>>>(gv, gp, esup, mat, words, slot);
}

// ------------------------------------------------------------- host helpers
void rotations3(const int f[8], bool wedge, Rot3& r) {
  auto rot = [](const int* q, int* o) {
    o[0] = 0; o[IUVW] = q[IUVW]; o[IUV] = q[IVW]; o[IUW] = q[IUV]; o[IVW] = q[IUW];
    o[IU] = q[IV]; o[IV] = q[IW]; o[IW] = q[IU];
  };
  auto rot2 = [](const int* q, int* o) {
    o[0] = 0; o[IUVW] = q[IUVW]; o[IUV] = q[IUW]; o[IUW] = q[IVW]; o[IVW] = q[IUV];
    o[IU] = q[IW]; o[IV] = q[IU]; o[IW] = q[IV];
  };
  for (int i = 0; i < 8; i++) r.fr[0][i] = (i == 0) ? 0 : f[i];
  r.count = 1;
  // triangleRotations (src/fringeCount.cu:1291-1317) / wedgeRotations (:1754-1780)
  const bool any = wedge || f[IU] != f[IV] || f[IU] != f[IW] || f[IUV] != f[IUW] || f[IUV] != f[IVW];
  if (!any) return;
  rot(r.fr[0], r.fr[1]);
  rot2(r.fr[0], r.fr[2]);
  r.count = 3;
  const bool fl = wedge ? (f[IV] != f[IW] || f[IUV] != f[IUW])
                        : ((f[IV] != f[IW] || f[IUV] != f[IUW]) && (f[IU] != f[IW] || f[IUV] != f[IVW]) &&
                           (f[IU] != f[IV] || f[IUW] != f[IVW]));
  if (!fl) return;
  int* q = r.fr[3];
  q[0] = 0; q[IUVW] = f[IUVW]; q[IUV] = f[IUW]; q[IUW] = f[IUV]; q[IVW] = f[IVW];
  q[IU] = f[IU]; q[IV] = f[IW]; q[IW] = f[IV];
  rot(r.fr[3], r.fr[4]);
  rot2(r.fr[3], r.fr[5]);
  r.count = 6;
}

int grid_for(long long work, int tpb, int per_sm) {
  const long long want = (work + tpb - 1) / tpb;
  const long long cap = (long long)sm_count() * per_sm;
  return (int)std::max(1LL, std::min(want, cap));
}

// The instantiation of the pattern's fringe counts, f_u <= f_v <= kEdgeChainMax.
template <int FU, int FV>
void launch_edge_chains(const GView& gv, const EdgeParams& ep, u64* slot, cudaStream_t s) {
  if (ep.f_u > FU) {
    if constexpr (FU < kEdgeChainMax) launch_edge_chains<FU + 1, FU + 1>(gv, ep, slot, s);
  } else if (ep.f_v > FV) {
    if constexpr (FV < kEdgeChainMax) launch_edge_chains<FU, FV + 1>(gv, ep, slot, s);
  } else {
    int nfit = 0;  // the largest n without wrapping below FV
    for (int bit = 30; bit >= 0; bit--)
      if (binomials_fit(nfit | 1 << bit, FV - 1)) nfit |= 1 << bit;
    edge_chain_kernel<FU, FV><<<grid_for(gv.m / 2, kTPB, 8), kTPB, 0, s>>>(gv, ep, nfit, slot);
  }
}

// Builds the wedge core's chunk-boundary table once per graph (vertices of
// degree >= 512, fewer when the table would pass 512 MiB).
int ensure_chunk_table(DevGraph& G, cudaStream_t s, uint64_t* launches, u64* d_small) {
  if (G.ctab_K > 0) return FSGC_OK;
  const int K = (int)(((long long)G.n + kWGran - 1) / kWGran) + 1;
  int min_deg = 512;
  GView gv = G.view();
  int* nrows_d = reinterpret_cast<int*>(d_small);
  if (cudaMalloc((void**)&G.ctab_id, sizeof(int) * (size_t)std::max(1, G.n)) != cudaSuccess ||
      cudaMalloc((void**)&G.ctab_rows, sizeof(int) * (size_t)std::max(1, G.n)) != cudaSuccess) {
    cudaGetLastError();
    return FSGC_ENOMEM;
  }
  int nrows = 0;
  for (;;) {
    cudaMemsetAsync(nrows_d, 0, sizeof(int), s);
    chunk_table_rows_kernel<<<grid_for(G.n, 256, 8), 256, 0, s>>>(gv, min_deg, G.ctab_id, G.ctab_rows, nrows_d);
    *launches += 1;
    if (cudaMemcpyAsync(&nrows, nrows_d, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return FSGC_ECUDA;
    if ((size_t)nrows * K * sizeof(int) <= ((size_t)512 << 20)) break;
    min_deg *= 2;
  }
  if (cudaMalloc((void**)&G.ctab_pos, sizeof(int) * std::max<size_t>(1, (size_t)nrows * K)) != cudaSuccess) {
    cudaGetLastError();
    return FSGC_ENOMEM;
  }
  if (nrows > 0) {
    chunk_table_fill_kernel<<<grid_for((long long)nrows * K, 256, 8), 256, 0, s>>>(gv, G.ctab_rows, nrows, K, G.ctab_pos);
    *launches += 1;
  }
  G.ctab_K = K;
  G.bytes += sizeof(int) * ((size_t)2 * G.n + (size_t)nrows * K);
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

}  // namespace

// Stream-ordered, so that growing one stream's arena neither waits for nor
// stalls work queued on other streams.
int ensure_plain_scratch(Scratch& sc, size_t need, cudaStream_t s) {
  if (sc.bytes >= need) return FSGC_OK;
  if (sc.ptr) {
    cudaFreeAsync(sc.ptr, s);
    sc.ptr = nullptr;
    sc.bytes = 0;
  }
  if (cudaMallocAsync(&sc.ptr, need, s) != cudaSuccess) {
    cudaGetLastError();
    sc.ptr = nullptr;
    return FSGC_ENOMEM;
  }
  sc.bytes = need;
  sc.gen++;
  return FSGC_OK;
}

// What a count of `mo` on `G` needs beyond the resident graph.  The shape
// tests repeat enqueue_count's dispatch.
namespace {
struct Needs {
  bool chunk_table = false;  // wedge core with a fringe-free centre
  bool pairs = false;        // which evaluates its pairs one by one in rank order
  bool vertex_triangles = false;
  bool entry_supports = false;  // general wedge core
  bool bit_matrix = false;      // general cores and that one, on a small graph
  size_t scratch = 0;        // arena bytes (hub cursors, triangle bitmaps)
};

Needs needs_of(const fsgc_matching_order& mo, const DevGraph& G, const fsgc_tuning& t) {
  Needs nd;
  if (mo.nodes < 2 || mo.nodes > FSGC_MAX_CORE) return nd;
  if (mo.nodes == 2) {
    int f[4] = {0, 0, 0, 0};
    for (int i = 0; i < mo.anchorsets; i++) f[mo.anch[i] & 3] = mo.fcnt[i];
    const int f_u = std::min(f[1], f[2]), f_uv = f[3], f_v = std::max(f[1], f[2]);
    if (f_uv == 1 && (f_u == 0 || f_v == 0)) nd.vertex_triangles = !(f_u == 0 && f_v == 0) || G.ngraphs > 0;
    return nd;
  }
  if (mo.nodes > 3) {
    nd.bit_matrix = true;
    return nd;
  }
  int f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = 0; i < mo.anchorsets; i++) f[mo.anch[i] & 7] = mo.fcnt[i];
  if (__builtin_popcount(mo.list[1]) == 1) {
    if (mo.list[1] == 2) {
      std::swap(f[IU], f[IV]);
      std::swap(f[IUW], f[IVW]);
    }
    if (f[IUVW] == 0 && f[IUV] == 0 && f[IUW] == 0 && f[IU] == 0) {
      nd.chunk_table = true;
      nd.pairs = wedge_pass(G, WedgeParams{f[IV], f[IVW], f[IW], 0, 0}, false) == kPairsPass;
      if (G.maxdeg > std::min(kWDvMax, std::max(16, t.wedge_small_max_degree))) {
        const long long gs = G.maxdeg;
        nd.scratch = (size_t)sm_count() * ((size_t)2 * gs * sizeof(long long) + (size_t)(gs + 1) * sizeof(int));
      }
    } else {
      nd.entry_supports = true;
      nd.bit_matrix = true;
    }
    return nd;
  }
  const bool clique = (f[IUVW] == 1) && (f[IUV] + f[IUW] + f[IVW] == 0) &&
                      ((f[IU] == 0) + (f[IV] == 0) + (f[IW] == 0) >= 2);
  if (!clique && triangle_by_tables(G, clique)) nd.scratch = triangle_scratch(G);
  return nd;
}
}  // namespace

size_t count_scratch_bytes(const fsgc_matching_order& mo, const DevGraph& G, const fsgc_tuning& t) {
  return needs_of(mo, G, t).scratch;
}

int check_tuning(const fsgc_tuning& t) {
  const bool ok = t.wedge_small_max_degree >= 16 && t.wedge_small_max_degree <= kWDvMax && t.triangle_walk_ratio >= 0 &&
                  t.triangle_walk_ratio <= (1 << 20) && t.triangle_stage_max >= 0 && t.triangle_stage_max <= 8192 &&
                  t.triangle_stage_max % 32 == 0 && t.general_lane_venn_max >= 0 &&
                  t.general_lane_venn_max <= (1 << 20) && t.general_blocks_per_sm >= 1 && t.general_blocks_per_sm <= 16;
  return ok ? FSGC_OK : FSGC_EINVAL;
}

void note_no_room(DevGraph& G, size_t need) {
  size_t free_now = 0, total = 0;
  if (cudaMemGetInfo(&free_now, &total) != cudaSuccess) cudaGetLastError();
  // more than was free, by a page, and enough for it
  G.room_from = std::max(std::max(need, free_now + ((size_t)2 << 20)), G.room_from);
}

bool room_again(DevGraph& G) {
  if (!G.rank_failed && !G.bits_failed) return false;
  size_t free_now = 0, total = 0;
  if (cudaMemGetInfo(&free_now, &total) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (free_now < G.room_from) return false;
  G.rank_failed = G.bits_failed = false;
  G.room_from = 0;
  return true;
}

size_t fast_structure_bytes(const DevGraph& G) { return G.rank_bytes + (G.bits ? bit_matrix_bytes(G) : 0); }

void free_fast_structures(DevGraph& G) {
  if (G.bits) G.bytes -= bit_matrix_bytes(G);
  free_rank_order(G);
  cudaFree(G.bits);
  G.bits = nullptr;
}

int prepare_for_count(const fsgc_matching_order& mo, DevGraph& G, cudaStream_t s, uint64_t* launches,
                      DevWork& work) {
  if (mo.nodes < 2) return FSGC_OK;
  int st = prepare_graph(G, s, launches, work.small);
  if (st != FSGC_OK) return st;
  const Needs nd = needs_of(mo, G, work.tune);
  if (nd.chunk_table) {
    st = nd.pairs && pairs_by_chunks(G, 1, false) ? FSGC_EUNSUPPORTED : ensure_rank_order(G, s, launches, work);
    if (st == FSGC_EUNSUPPORTED) st = ensure_chunk_table(G, s, launches, work.small + 9);
    if (st != FSGC_OK) return st;
  }
  if (nd.vertex_triangles) {
    st = ensure_vertex_triangles(G, s, launches);
    if (st != FSGC_OK) return st;
  }
  if (nd.entry_supports) {
    st = ensure_entry_supports(G, s, launches);
    if (st != FSGC_OK) return st;
  }
  if (nd.bit_matrix) {
    st = ensure_bit_matrix(G, s, launches);
    if (st != FSGC_OK && st != FSGC_EUNSUPPORTED) return st;
  }
  return cudaStreamSynchronize(s) == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

// The chunk table is for graphs without a copy in rank order and dense ones: beside
// a copy, only exact counts beyond its bound read it elsewhere, and they build it.
int prepare_all(DevGraph& G, cudaStream_t s, uint64_t* launches, DevWork& work) {
  int st = prepare_graph(G, s, launches, work.small);
  if (st == FSGC_OK) {
    st = ensure_rank_order(G, s, launches, work);
    if (st == FSGC_EUNSUPPORTED || (st == FSGC_OK && pairs_by_chunks(G, 1, false)))
      st = G.ngraphs == 0 ? ensure_chunk_table(G, s, launches, work.small + 9) : FSGC_OK;
  }
  if (st == FSGC_OK) st = ensure_vertex_triangles(G, s, launches);
  if (st == FSGC_OK && G.ngraphs == 0) st = ensure_entry_supports(G, s, launches);
  if (st == FSGC_OK) {
    st = ensure_bit_matrix(G, s, launches);
    if (st == FSGC_EUNSUPPORTED) st = FSGC_OK;
  }
  if (st != FSGC_OK) return st;
  return cudaStreamSynchronize(s) == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

namespace {
// The fringe-free-centre wedge core for a set of patterns by both pair kernels:
// endpoints of degree <= kWDvMax, then hub endpoints (cursors and segment offsets in
// the work arena).
template <int NP, class A>
int launch_wedge_chunks(DevGraph& G, const GView& gv, const WedgeSet& ws0, cudaStream_t s, uint64_t* launches,
                        DevWork& work) {
  int* q1 = reinterpret_cast<int*>(work.small + 7);
  int* q2 = reinterpret_cast<int*>(work.small + 8);
  int st = ensure_chunk_table(G, s, launches, work.small + 9);
  if (st != FSGC_OK) return st;
  const ChunkTable tab{G.ctab_id, G.ctab_pos, G.ctab_K};
  cudaMemsetAsync(q1, 0, 2 * sizeof(u64), s);
  const int blocks = sm_count();
  WedgeSet ws = ws0;
  ws.small_max = std::min(kWDvMax, std::max(16, work.tune.wedge_small_max_degree));
  {
    const size_t smem = sizeof(WedgeSmem<false>);
    cudaFuncSetAttribute(wedge_chunk_kernel<false, NP, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    wedge_chunk_kernel<false, NP, A><<<blocks, kWThreads, smem, s>>>(gv, ws, q1, nullptr, nullptr, 0, tab);
    *launches += 1;
  }
  if (G.maxdeg > ws.small_max) {
    // hub endpoints: cursors (2 x int64) and segment offsets (int32) per block
    const long long gs = G.maxdeg;
    const size_t need = (size_t)blocks * ((size_t)2 * gs * sizeof(long long) + (size_t)(gs + 1) * sizeof(int));
    st = ensure_plain_scratch(work.tri, std::max(need, work.tri.bytes), s);
    if (st != FSGC_OK) return st;
    long long* gcur = reinterpret_cast<long long*>(work.tri.ptr);
    int* gpre = reinterpret_cast<int*>(gcur + (size_t)blocks * 2 * gs);
    const size_t smem = sizeof(WedgeSmem<true>);
    cudaFuncSetAttribute(wedge_chunk_kernel<true, NP, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    wedge_chunk_kernel<true, NP, A><<<blocks, kWThreads, smem, s>>>(gv, ws, q2, gcur, gpre, gs, tab);
    *launches += 1;
  }
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

// The fringe-free-centre wedge core for a set of patterns: in rank order where the
// graph takes that path, but patterns whose pairs are evaluated one by one by chunks
// where that is the better path for as many of them.
template <int NP, class A>
int launch_wedge_set(DevGraph& G, const GView& gv, const WedgeSet& ws, cudaStream_t s, uint64_t* launches, DevWork& work) {
  const bool none = !wedge_rank_size_ok(G) || (!G.radj && (G.lean || G.rank_failed));  // no copy, nor will there be
  if (none) return launch_wedge_chunks<NP, A>(G, gv, ws, s, launches, work);
  int evaluated = 0;
  constexpr bool exact = std::is_same<A, X128>::value;
  for (int i = 0; i < ws.np; i++) evaluated += wedge_pass(G, ws.w[i], exact) == kPairsPass;
  const int from = !pairs_by_chunks(G, evaluated, exact) ? kPairsPass + 1 : sums_join_pairs(G) ? kSumsPass : kPairsPass;
  WedgeSet rank = ws, pairs = ws;
  rank.np = pairs.np = 0;
  for (int i = 0; i < ws.np; i++) {
    WedgeSet& to = wedge_pass(G, ws.w[i], exact) >= from ? pairs : rank;
    to.w[to.np] = ws.w[i];
    to.slot[to.np++] = ws.slot[i];
  }
  int st = FSGC_OK;
  if (pairs.np > 0) st = launch_wedge_chunks<NP, A>(G, gv, pairs, s, launches, work);
  if (st != FSGC_OK || rank.np == 0) return st;
  const size_t arena = wedge_rank_scratch(G);
  if (arena > 0) st = ensure_plain_scratch(work.tri, std::max(arena, work.tri.bytes), s);
  if (st != FSGC_OK) return st;
  st = enqueue_wedge_rank(G, gv, rank.w, rank.slot, rank.np, exact, s, launches, work);
  return st == FSGC_EUNSUPPORTED ? launch_wedge_chunks<NP, A>(G, gv, rank, s, launches, work) : st;
}

template <class A>
int enqueue_count_a(CountJob& job, cudaStream_t s, uint64_t* launches, DevWork& work) {
  const fsgc_matching_order& mo = *job.mo;
  DevGraph& G = *job.g;
  job.host_only = false;
  job.host_value = 0;
  job.per_member_div = 1;
  if (mo.nodes < 1 || mo.nodes > FSGC_MAX_CORE || mo.anchorsets > 63) return FSGC_EINVAL;
  const int TPB = kTPB;
  const bool packed = G.ngraphs > 0;

  // ---- vertex core (vertexCore, src/fringeCount.cu:2172-2191)
  if (mo.nodes == 1) {
    job.core_type = FSGC_CORE_VERTEX;
    // single vertex: n; single edge: m/2 (per member graph for packed graphs, on the host)
    if (mo.anchorsets == 0) { job.host_only = true; job.host_value = (u64)G.n; return FSGC_OK; }
    if (mo.fcnt[0] == 1) { job.host_only = true; job.host_value = (u64)(G.m / 2); return FSGC_OK; }
    GView gv0 = G.view();
    gv0.comp_slots = job.d_comp_slots;
    star_kernel<A><<<grid_for(G.n, TPB, 8), TPB, 0, s>>>(gv0, mo.fcnt[0], job.d_slot);
    *launches += 1;
    return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
  }

  int st = prepare_graph(G, s, launches, work.small);
  if (st != FSGC_OK) return st;
  GView gv = G.view();
  gv.comp_slots = job.d_comp_slots;
  const long long me = G.m / 2;

  // ---- edge core (edgeCore, src/fringeCount.cu:2106-2144)
  if (mo.nodes == 2) {
    job.core_type = FSGC_CORE_EDGE;
    int f[4] = {0, 0, 0, 0};
    for (int i = 0; i < mo.anchorsets; i++) f[mo.anch[i] & 3] = mo.fcnt[i];
    const int f_u = std::min(f[1], f[2]), f_uv = f[3], f_v = std::max(f[1], f[2]);
    if (f_uv == 1 && (f_u == 0 || f_v == 0)) {
      if (f_u == 0 && f_v == 0) {  // triangle
        if (!packed) {
          job.host_only = true;
          job.host_value = (u64)G.triangles;
          return FSGC_OK;
        }
        // per member: sum of 2 x (triangles at v) over its vertices = 6 x triangles
        st = ensure_vertex_triangles(G, s, launches);
        if (st != FSGC_OK) return st;
        packed_vertex_sum_kernel<<<grid_for(G.n, TPB, 8), TPB, 0, s>>>(gv, G.vtri2, job.d_slot);
        *launches += 1;
        job.per_member_div = 6;
        return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
      }
      st = ensure_vertex_triangles(G, s, launches);
      if (st != FSGC_OK) return st;
      tailed_triangle_kernel<A><<<grid_for(G.n, TPB, 8), TPB, 0, s>>>(gv, G.vtri2, f_v, job.d_slot);
      *launches += 1;
      return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
    }
    EdgeParams ep{f_u, f_uv, f_v, f_u + f_uv, f_u + f_uv + f_v};
    if (me > 0) {
      if (std::is_same<A, u64>::value && f_v <= kEdgeChainMax)
        launch_edge_chains<0, 0>(gv, ep, job.d_slot, s);
      else
        edge_kernel<A><<<grid_for(me, TPB, 8), TPB, 0, s>>>(gv, ep, job.d_slot);
      *launches += 1;
    }
    return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
  }

  int f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (mo.nodes == 3)
    for (int i = 0; i < mo.anchorsets; i++) f[mo.anch[i] & 7] = mo.fcnt[i];

  // ---- wedge core (wedgeCore, src/fringeCount.cu:1783-1825)
  if (mo.nodes == 3 && __builtin_popcount(mo.list[1]) == 1) {
    job.core_type = FSGC_CORE_WEDGE;
    if (mo.list[1] == 2) {  // centre is B: swap roles of A and B
      std::swap(f[IU], f[IV]);
      std::swap(f[IUW], f[IVW]);
    }
    const int min_u = f[IUVW] + f[IUV] + f[IUW] + f[IU] + 2;
    const int min_v = f[IUVW] + f[IUV] + f[IVW] + f[IV] + 1;
    const int min_w = f[IUVW] + f[IUW] + f[IVW] + f[IW] + 1;
    const int sum3 = min_u + min_v + min_w;
    const int sum2 = sum3 - std::max(std::max(min_u, min_v), min_w);
    const int sum1 = std::min(std::min(min_u, min_v), min_w);
    const int lim = std::min(min_v, min_w);
    if (f[IUVW] == 0 && f[IUV] == 0 && f[IUW] == 0 && f[IU] == 0) {
      WedgeSet ws;
      memset(&ws, 0, sizeof(ws));
      ws.np = 1;
      ws.lim = lim;
      ws.w[0] = WedgeParams{f[IV], f[IVW], f[IW], lim, min_v + min_w};
      ws.slot[0] = job.d_slot;
      return launch_wedge_set<1, A>(G, gv, ws, s, launches, work);
    }
    GWedgeParams gp;
    gp.min_u = min_u; gp.lim = lim; gp.sum1 = sum1; gp.sum2 = sum2; gp.sum3 = sum3;
    rotations3(f, true, gp.rot);
    for (int r = 0; r < gp.rot.count; r++) {
      gp.packed[r] = 0;
      for (int i = 1; i < 8; i++) gp.packed[r] |= (u64)gp.rot.fr[r][i] << (8 * i);
    }
    st = ensure_entry_supports(G, s, launches);
    if (st != FSGC_OK) return st;
    const int blocks = grid_for(G.m * 32, TPB, 8);
    st = ensure_bit_matrix(G, s, launches);
    if (st != FSGC_OK && st != FSGC_EUNSUPPORTED) return st;
    if (st == FSGC_OK) {
      int k = 0;
      for (int i = 0; i < 8; i++) k = std::max(k, f[i]);
      const bool ones = std::max(f[IU], std::max(f[IV], f[IW])) <= 1 && f[IUV] + f[IUW] + f[IVW] == 0;
      const int ring = !binomials_fit(G.maxdeg, k) ? 0 : ones ? 1 : 2;
      const int words = bit_matrix_words(G.n);
      if (words <= 32) launch_wedge_bits<1, A>(gv, gp, G.esup, G.bits, words, ring, job.d_slot, blocks, s);
      else if (words <= 64) launch_wedge_bits<2, A>(gv, gp, G.esup, G.bits, words, ring, job.d_slot, blocks, s);
      else launch_wedge_bits<4, A>(gv, gp, G.esup, G.bits, words, ring, job.d_slot, blocks, s);
    } else {
      wedge_general_kernel<A><<<blocks, TPB, 0, s>>>(gv, gp, G.esup, job.d_slot);
    }
    *launches += 1;
    return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
  }

  // ---- triangle core (triangleCore, src/fringeCount.cu:1320-1373)
  if (mo.nodes == 3) {
    job.core_type = FSGC_CORE_TRIANGLE;
    const int min_u = f[IUVW] + f[IUV] + f[IUW] + f[IU];
    const int min_v = f[IUVW] + f[IUV] + f[IVW] + f[IV];
    const int min_w = f[IUVW] + f[IUW] + f[IVW] + f[IW];
    TrianglePattern tp;
    tp.sum3 = min_u + min_v + min_w + 6;
    tp.sum2 = tp.sum3 - (std::max(std::max(min_u, min_v), min_w) + 2);
    tp.sum1 = std::min(std::min(min_u, min_v), min_w) + 2;
    const bool clique = (f[IUVW] == 1) && (f[IUV] + f[IUW] + f[IVW] == 0) &&
                        ((f[IU] == 0) + (f[IV] == 0) + (f[IW] == 0) >= 2);
    tp.tails = f[IU] + f[IV] + f[IW];
    tp.mode = clique ? (tp.tails == 0 ? 1 : 2) : 0;
    tp.relabel = G.tri_relabel ? 1 : 0;
    rotations3(f, false, tp.rot);
    if (me == 0) return FSGC_OK;
    if (triangle_by_tables(G, clique))
      return enqueue_triangle(G, gv, tp, std::is_same<A, X128>::value, job.d_slot, s, launches, work);
    triangle_core_kernel<A><<<grid_for(me, TPB, 8), TPB, 0, s>>>(gv, tp, job.d_slot);
    *launches += 1;
    return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
  }

  // ---- general core (generalCore, src/fringeCount.cu:666-692)
  job.core_type = FSGC_CORE_GENERAL;
  if (mo.anchorsets == 0) return FSGC_EINVAL;
  GenParams* gp = new GenParams();
  memset(gp, 0, sizeof(GenParams));
  gp->k = mo.nodes;
  for (int i = 0; i < mo.anchorsets; i++) gp->anchors |= mo.anch[i];
  gp->nonanchors = gp->anchors ^ ((1 << mo.nodes) - 1);
  gp->startdeg = mo.startdeg;
  for (int i = 0; i < 5; i++) { gp->destdeg[i] = mo.destdeg[i]; gp->list[i] = mo.list[i]; }
  for (int i = 0; i < 63; i++) gp->fcnt[i] = mo.fcnt[i];
  for (int i = 0; i < 63; i++) gp->anch[i] = mo.anch[i];
  gp->nsets = mo.anchorsets;
  gp->exact = job.exact_placements;
  // placement steps: anchor sets from the last to the first; within a set the
  // regions containing it in increasing bitmap order, the all-anchor region last
  int ns = 0;
  for (int asi = mo.anchorsets - 1; asi >= 0; asi--) {
    const int anch = mo.anch[asi];
    int idx = anch;
    for (;;) {
      if (ns >= kMaxSlots) { delete gp; return FSGC_EUNSUPPORTED; }
      gp->slot_idx[ns] = (uint8_t)idx;
      gp->slot_set[ns] = (uint8_t)asi;
      gp->slot_top[ns] = (idx == gp->anchors) ? 1 : 0;
      ns++;
      if (idx == gp->anchors) break;
      idx = (((idx | gp->nonanchors) + 1) | anch) & ~gp->nonanchors;
    }
  }
  gp->nslots = ns;
  gp->lane_venn_max = std::max(0, work.tune.general_lane_venn_max);
  auto* queue = reinterpret_cast<unsigned long long*>(work.small + 5);
  cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
  const int blocks = sm_count() * std::min(16, std::max(1, work.tune.general_blocks_per_sm));
  // one edge per grab until there are many more edges than warps
  gp->grab = (int)std::max(1LL, std::min(32LL, G.m / ((long long)blocks * kGenWarps * 64)));
  BitSets bs;
  if (bit_sets_for(*gp, gp->exact || !std::is_same<A, u64>::value, G.n, bs)) {
    st = ensure_bit_matrix(G, s, launches);
    if (st == FSGC_OK) {
      bs.parts = bits_parts(G, (long long)blocks * kGenWarps);
      if (ns <= 32) st = launch_bits<32, A>(gv, *gp, bs, G.bits, queue, job.d_slot, blocks, s);
      else if (ns <= 64) st = launch_bits<64, A>(gv, *gp, bs, G.bits, queue, job.d_slot, blocks, s);
      else st = launch_bits<128, A>(gv, *gp, bs, G.bits, queue, job.d_slot, blocks, s);
      *launches += 1;
      delete gp;
      return st;
    }
    if (st != FSGC_EUNSUPPORTED) {
      delete gp;
      return st;
    }
    st = FSGC_OK;  // no room for the matrix: the lists
  }
  // the placement walk's state is sized by the step count
  if (ns <= 32) general_core_kernel<32, A><<<blocks, kGenWarps * 32, 0, s>>>(gv, *gp, queue, job.d_slot);
  else if (ns <= 64) general_core_kernel<64, A><<<blocks, kGenWarps * 32, 0, s>>>(gv, *gp, queue, job.d_slot);
  else if (ns <= 128) general_core_kernel<128, A><<<blocks, kGenWarps * 32, 0, s>>>(gv, *gp, queue, job.d_slot);
  else general_core_kernel<kMaxSlots, A><<<blocks, kGenWarps * 32, 0, s>>>(gv, *gp, queue, job.d_slot);
  *launches += 1;
  delete gp;
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}
}  // namespace

int enqueue_count(CountJob& job, cudaStream_t s, uint64_t* launches, DevWork& work) {
  return job.exact_count ? enqueue_count_a<X128>(job, s, launches, work) : enqueue_count_a<u64>(job, s, launches, work);
}

// Many patterns on one graph: patterns whose kernels share their match
// enumeration run as sets -- stars and tailed triangles in one vertex pass,
// edge-core formulas in one pass over the oriented edges, fringe-free-centre
// wedges together -- and every other pattern as a count of its own.  Each job's
// result goes to its own slot; the values equal the single-pattern kernels'.
int enqueue_count_set(std::vector<CountJob*>& jobs, cudaStream_t s, uint64_t* launches, DevWork& work) {
  if (jobs.empty()) return FSGC_OK;
  DevGraph& G = *jobs[0]->g;
  for (CountJob* j : jobs)
    if (j->g != &G || j->exact_count || G.ngraphs > 0) return FSGC_EINVAL;
  int st = prepare_graph(G, s, launches, work.small);
  if (st != FSGC_OK) return st;
  GView gv = G.view();
  std::vector<std::pair<CountJob*, std::pair<int, int>>> verts;  // (job, (tailed, t))
  std::vector<std::pair<CountJob*, EdgeParams>> edges;
  std::vector<std::pair<CountJob*, WedgeParams>> wedges;
  std::vector<CountJob*> single;
  for (CountJob* jp : jobs) {
    CountJob& job = *jp;
    const fsgc_matching_order& mo = *job.mo;
    job.host_only = false;
    job.host_value = 0;
    job.per_member_div = 1;
    if (mo.nodes == 1 && mo.anchorsets > 0 && mo.fcnt[0] > 1) {
      job.core_type = FSGC_CORE_VERTEX;
      verts.push_back({jp, {0, (int)mo.fcnt[0]}});
      continue;
    }
    if (mo.nodes == 2) {
      int f[4] = {0, 0, 0, 0};
      for (int i = 0; i < mo.anchorsets; i++) f[mo.anch[i] & 3] = mo.fcnt[i];
      const int f_u = std::min(f[1], f[2]), f_uv = f[3], f_v = std::max(f[1], f[2]);
      job.core_type = FSGC_CORE_EDGE;
      if (f_uv == 1 && (f_u == 0 || f_v == 0)) {
        if (f_u == 0 && f_v == 0) { single.push_back(jp); continue; }  // the triangle total
        verts.push_back({jp, {1, f_v}});
      } else {
        edges.push_back({jp, EdgeParams{f_u, f_uv, f_v, f_u + f_uv, f_u + f_uv + f_v}});
      }
      continue;
    }
    if (mo.nodes == 3) {
      int f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int i = 0; i < mo.anchorsets; i++) f[mo.anch[i] & 7] = mo.fcnt[i];
      if (__builtin_popcount(mo.list[1]) == 1) {
        if (mo.list[1] == 2) {
          std::swap(f[IU], f[IV]);
          std::swap(f[IUW], f[IVW]);
        }
        if (f[IUVW] == 0 && f[IUV] == 0 && f[IUW] == 0 && f[IU] == 0) {
          const int min_v = f[IUVW] + f[IUV] + f[IVW] + f[IV] + 1;
          const int min_w = f[IUVW] + f[IUW] + f[IVW] + f[IW] + 1;
          job.core_type = FSGC_CORE_WEDGE;
          wedges.push_back({jp, WedgeParams{f[IV], f[IVW], f[IW], std::min(min_v, min_w), min_v + min_w}});
          continue;
        }
      }
    }
    single.push_back(jp);
  }
  const int TPB = kTPB;
  for (size_t b = 0; b < verts.size(); b += kPassFuse) {
    VertexSet vs;
    memset(&vs, 0, sizeof(vs));
    bool tailed = false;
    for (size_t i = b; i < std::min(verts.size(), b + kPassFuse); i++) {
      const int q = vs.np++;
      vs.tailed[q] = verts[i].second.first;
      vs.t[q] = verts[i].second.second;
      vs.slot[q] = verts[i].first->d_slot;
      tailed |= vs.tailed[q] != 0;
    }
    if (tailed) {
      st = ensure_vertex_triangles(G, s, launches);
      if (st != FSGC_OK) return st;
    }
    vertex_set_kernel<<<grid_for(G.n, TPB, 8), TPB, 0, s>>>(gv, tailed ? G.vtri2 : nullptr, vs);
    *launches += 1;
  }
  // patterns that no edge of the graph has degrees for count nothing
  const long long most = G.maxdeg;
  edges.erase(std::remove_if(edges.begin(), edges.end(),
                             [&](const std::pair<CountJob*, EdgeParams>& e) {
                               return most <= e.second.lim1 || 2 * most <= e.second.lim2;
                             }),
              edges.end());
  // few fringes: a kernel each.  A pass for two patterns takes 32 us over 8,000
  // edges and 127 us over 3.2 M in the fused kernel's nck loops, 27 and 101 us in
  // two kernels (whole calls).  Eight patterns, of which a path of 10,000 has degrees
  // for two: 30 us fused, 43 us in eight kernels, 30 us without the other six; where
  // all eight run but few edges have the degrees, the launches cost what is left: a
  // square grid of 10,000 32 and 43 us, uniform with 11,000 edges 34 and 42 us.
  auto fused = edges.begin();
  for (auto& e : edges) {
    if (e.second.f_v > kEdgeChainMax || G.m == 0) {
      *fused++ = e;
      continue;
    }
    launch_edge_chains<0, 0>(gv, e.second, e.first->d_slot, s);
    *launches += 1;
  }
  edges.erase(fused, edges.end());
  for (size_t b = 0; b < edges.size(); b += kPassFuse) {
    EdgeSet es;
    memset(&es, 0, sizeof(es));
    for (size_t i = b; i < std::min(edges.size(), b + kPassFuse); i++) {
      const int q = es.np++;
      es.e[q] = edges[i].second;
      es.slot[q] = edges[i].first->d_slot;
    }
    if (G.m / 2 > 0) {
      edge_set_kernel<<<grid_for(G.m / 2, TPB, 8), TPB, 0, s>>>(gv, es);
      *launches += 1;
    }
  }
  for (size_t b = 0; b < wedges.size(); b += kWedgeFuse) {
    WedgeSet ws;
    memset(&ws, 0, sizeof(ws));
    ws.lim = 1 << 30;
    for (size_t i = b; i < std::min(wedges.size(), b + kWedgeFuse); i++) {
      const int q = ws.np++;
      ws.w[q] = wedges[i].second;
      ws.slot[q] = wedges[i].first->d_slot;
      ws.lim = std::min(ws.lim, ws.w[q].lim);
    }
    st = ws.np == 1 ? launch_wedge_set<1, u64>(G, gv, ws, s, launches, work)
                    : launch_wedge_set<kWedgeFuse, u64>(G, gv, ws, s, launches, work);
    if (st != FSGC_OK) return st;
  }
  for (CountJob* jp : single) {
    st = enqueue_count(*jp, s, launches, work);
    if (st != FSGC_OK) return st;
  }
  return FSGC_OK;
}

// Launchers for callers that bring their own device memory (noalloc.cu): the
// wedge-core pair kernels on a view whose deg[] the caller filled.
namespace {
WedgeSet single_wedge(int f_v, int f_vw, int f_w, int lim, int minsum, u64* slot) {
  WedgeSet ws;
  memset(&ws, 0, sizeof(ws));
  ws.np = 1;
  ws.lim = lim;
  ws.small_max = kWDvMax;
  ws.w[0] = WedgeParams{f_v, f_vw, f_w, lim, minsum};
  ws.slot[0] = slot;
  return ws;
}
}  // namespace

int launch_wedge_small(const GView& gv, int f_v, int f_vw, int f_w, int lim, int minsum, int* queue, u64* slot,
                       cudaStream_t s) {
  const WedgeSet ws = single_wedge(f_v, f_vw, f_w, lim, minsum, slot);
  const size_t smem = sizeof(WedgeSmem<false>);
  cudaFuncSetAttribute(wedge_chunk_kernel<false, 1, u64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  wedge_chunk_kernel<false, 1, u64><<<sm_count(), kWThreads, smem, s>>>(gv, ws, queue, nullptr, nullptr, 0,
                                                                   ChunkTable{nullptr, nullptr, 0});
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

int launch_wedge_big(const GView& gv, int f_v, int f_vw, int f_w, int lim, int minsum, int* queue, long long* gcur,
                     int* gpre, long long gstride, int blocks, u64* slot, cudaStream_t s) {
  const WedgeSet ws = single_wedge(f_v, f_vw, f_w, lim, minsum, slot);
  const size_t smem = sizeof(WedgeSmem<true>);
  cudaFuncSetAttribute(wedge_chunk_kernel<true, 1, u64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  wedge_chunk_kernel<true, 1, u64><<<blocks, kWThreads, smem, s>>>(gv, ws, queue, gcur, gpre, gstride,
                                                              ChunkTable{nullptr, nullptr, 0});
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

int wedge_small_max_degree() { return kWDvMax; }

}  // namespace fsgc
