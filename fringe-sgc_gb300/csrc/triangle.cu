// Triangle core: counts by fc3 over every triangle (src/fringeCount.cu:1320-1373),
// and the reference's 4-clique and tailed 4-clique special cases.
//
// The triangles whose lowest (deg, id) vertex is a are counted together.  For
// each out-neighbour b_j of a (above it in the degree order) a bitmap row over
// the positions of N(a) holds N(a) & N(b_j); then a pair (b_i, b_j) is a
// triangle iff b_j is in the oriented list of b_i, the pairwise overlaps are
// the loader's edge supports, and the triple overlap is a popcount of two rows.
// (4-cliques: the rows run over the out-neighbours alone.)
//
// The rows are filled through a hash table of a's out-neighbours in shared
// memory: every neighbour x of a looks up its oriented list -- at most O(sqrt m)
// entries -- and a hit b_j means that x is in N(a) & N(b_j).  That is
// sum over x of deg(x) * outdeg(x) lookups in all, read as contiguous lists,
// where testing N(a) against N(b_j) entry by entry costs a binary search each.
// The same lookups of the out-neighbours alone then list the triangles with
// their edge slots, and are staged per warp so that every lane evaluates one.
//
// Small vertices (at most 32 out-neighbours, 768 row words and, in rows over
// N(a), 256 neighbours) take one warp each; most others a block of four warps;
// the triangle_wide ones, listed when the graph is prepared, a block of twelve,
// one at a time, with rows that do not fit in shared memory in a per-block part
// of the work arena.
//
// What bounds it: the lookups' instructions (a hash probe, five shuffles and a
// share of a list load per entry, 20 to 22 of 32 lanes busy) and their latency: on
// RMAT n = 2^20 the schedulers issue in 43 (narrow blocks) and 38 of 100 cycles with
// 36 % of the warps in flight, which wait for list reads and for shared memory; DRAM
// runs at 1 % of its rate.  RMAT n = 600,011 (192M triangles), 4-clique with three
// fringes: rows by binary searches in the arena 167 ms -> 57 ms; RMAT n = 65,536:
// 4-clique (one lane per triangle, before) 129 -> 2.3 ms, with two tails 201 -> 2.6 ms,
// a mixed triangle pattern (six rotations) 77 -> 18 ms, of which the placement sums
// (fc3_ring instead of fc3) are half.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "fsgc_formulas.cuh"
#include "fsgc_internal.h"

namespace fsgc {

void upload_div_magic_triangle() { upload_div_table(); }

namespace {

// Two launches: blocks of 4 warps (37 KB of shared memory, six an SM) for the
// vertices whose rows fit there, then blocks of 12 (112 KB, two an SM) for the
// rest.  Half of RMAT's larger vertices have 53 out-neighbours and 400 row
// words, the largest 700 and 20,000: one block size for both left three warps in
// four waiting at barriers.
constexpr int kNarrow = 128, kWide = 384;
// Kernel modes: the pattern's, and kRing for the triangle core by fc3_ring.
constexpr int kRing = 3;
constexpr int kSmallK = 32;             // out-neighbours of a warp-sized vertex
constexpr int kSmallRows = 768;         // and its row words
constexpr int kSmallLists = 256;        // and its neighbours, in rows over N(a): their lists are read by that warp
constexpr int kSmallSlots = 64;
constexpr int kSmallWords = kSmallRows + kSmallSlots + kSmallSlots / 2 + 4 * kSmallK;
constexpr int kStage = 96;              // staged triangles per warp: 31 left over and two steps' worth
constexpr int kMaxOut = 8192;           // largest out-degree (table and arrays in shared memory)
constexpr int kArraysMax = 2048;        // up to here degrees, ids and supports sit beside the table

// What the evaluation reads, in shared memory: it is called out of line, where
// the launch parameters would be generic loads.
struct TriShared {
  int sum1, sum2, sum3;  // pruning thresholds (init_wl_triangle, common3_triangle)
  Rot3 rot;
};

struct TriLaunch {
  TriShared eval;
  int tails;
  int relabel;           // roles by (deg, id) order (1) or by id (0)
  int slots;             // table slots of the largest vertex
  int kmax;
  int arrays;            // ints per out-neighbour kept in shared memory (4 or 1)
  int rows;              // row words that fit in shared memory
  const int* list;       // the vertices to look at (null: all of them)
  int items;             // and their number
  long long gstride;     // arena words per block
};

// A table of out-neighbours: key = id, val = index; empty keys are -1.
struct OutTable {
  int* key;
  unsigned short* val;
  int shift;  // 32 - log2(slots)
};
__device__ __forceinline__ unsigned out_hash(int id, int shift) { return ((unsigned)id * 0x9E3779B1u) >> shift; }
__device__ __forceinline__ int out_find(const OutTable& t, int id) {
  const unsigned mask = 0xffffffffu >> t.shift;
  unsigned s = out_hash(id, t.shift);
  for (unsigned probe = 0; probe <= mask; probe++) {  // at most half full: an empty slot ends the probes
    const int k = t.key[s];
    if (k == id) return t.val[s];
    if (k < 0) break;
    s = (s + 1) & mask;
  }
  return -1;
}

__device__ __forceinline__ long long role_key(int x, int d, int relabel) {
  // larger key = later in the reference's vertex order (its new ids ascend with
  // descending (deg, id) after the relabel, with the id otherwise)
  return relabel ? -(((long long)d << 32) | (unsigned)x) : (long long)x;
}

// fc3 summed over the rotations for the triangle (x, y, z) with the given
// degrees, pairwise supports and triple overlap; 0 where the reference prunes it.
template <bool RING, class A>
__device__ __forceinline__ A triangle_value(const TriShared& p, int rl, int x, int y, int z, int dx, int dy, int dz, int s_xy,
                                            int s_xz, int s_yz, int c123) {
  // u latest, w earliest in the reference's vertex order
  long long kx = role_key(x, dx, rl), ky = role_key(y, dy, rl), kz = role_key(z, dz, rl);
  auto swap_ll = [](long long& a, long long& b) { const long long t = a; a = b; b = t; };
  auto swap_i = [](int& a, int& b) { const int t = a; a = b; b = t; };
  auto order_xy = [&]() {
    if (kx < ky) { swap_ll(kx, ky); swap_i(dx, dy); swap_i(s_xz, s_yz); }
  };
  order_xy();
  if (ky < kz) { swap_ll(ky, kz); swap_i(dy, dz); swap_i(s_xy, s_xz); }
  order_xy();
  const int du = dx, dv = dy, dw = dz;
  const int th1 = max(p.sum1, p.sum2 - du);
  const int th2 = max(max(p.sum1, p.sum3 - du - dv), max(p.sum2 - du, p.sum2 - dv));
  const bool take = du >= p.sum1 && dv >= th1 && dw >= th2;
  // com3 (src/fringeCount.cu:934-964): exclusive regions without the triangle
  const int c12 = s_xy - (c123 + 1), c13 = s_xz - (c123 + 1), c23 = s_yz - (c123 + 1);
  const int u = du - (c12 + c13 + (c123 + 2)), v = dv - (c12 + c23 + (c123 + 2)), w = dw - (c13 + c23 + (c123 + 2));
  A t = A(0);
  if constexpr (RING) {
    for (int i = 0; i < p.rot.count; i++) t += fc3_ring(p.rot.fr[i], c123, c12, c13, c23, u, v, w);
  } else {
    const int venn[8] = {0, u, v, c12, w, c13, c23, c123};
    for (int i = 0; i < p.rot.count; i++) t += fc3<A>(p.rot.fr[i], venn);
  }
  return take ? t : A(0);
}

// The entries of the 32 lists [first, first + len) that a warp's lanes hold, 32
// at a time.  Every call is the whole warp's.
struct ListWalk {
  long long first_;
  int len_, inc_, total_ = 0, at_ = 0;
  __device__ __forceinline__ bool done() const { return at_ >= total_; }
  __device__ __forceinline__ void open(long long first, int len) {
    const int lane = threadIdx.x & 31;
    first_ = first;
    len_ = len;
    inc_ = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, inc_, o);
      if (lane >= o) inc_ += y;
    }
    total_ = __shfl_sync(0xffffffffu, inc_, 31);
    at_ = 0;
  }
  // The lane whose list this lane's entry is in (-1: no entry left) and the entry.
  __device__ __forceinline__ int step(long long& entry) {
    const int e = at_ + (int)(threadIdx.x & 31);
    int own = 0;  // lanes whose inclusive prefix does not exceed e
#pragma unroll
    for (int h = 16; h >= 1; h >>= 1) {
      const int v = __shfl_sync(0xffffffffu, inc_, own + h - 1);
      if (v <= e) own += h;
    }
    own = min(own, 31);
    const int before = __shfl_sync(0xffffffffu, inc_ - len_, own);
    entry = __shfl_sync(0xffffffffu, first_, own) + (e - before);
    at_ += 32;
    return e < total_ ? own : -1;
  }
};

// The vertex a group of warps is counting, in shared memory.
struct VertexCtx {
  int a, da, k, rl;
  int stride, w0, w1;      // rows: words a row, first and past the last position word
  unsigned* rows;
  const int* oadj;         // oriented list of a
  const unsigned* osup;    // its supports
  const int* deg;
  const int *ids, *degs, *sups;  // per out-neighbour; null when they are not kept
};

// One triangle (a, b_i, b_j), t = (i | j << 16, support of (b_i, b_j)).
template <int MODE, class A>
__device__ __forceinline__ A triangle_of(const VertexCtx& c, const TriShared& p, int tails, uint2 t) {
  const int i = (int)(t.x & 0xffffu), j = (int)(t.x >> 16);
  const int w0 = c.w0, w1 = c.w1;
  const unsigned *mi = c.rows + (size_t)i * c.stride - w0, *mj = c.rows + (size_t)j * c.stride - w0;
  if (MODE % 3 == 0) {
    int n = 0, w = 0;
    for (; w + 4 <= w1; w += 4) {
      const unsigned x0 = mi[w] & mj[w], x1 = mi[w + 1] & mj[w + 1], x2 = mi[w + 2] & mj[w + 2], x3 = mi[w + 3] & mj[w + 3];
      n += (__popc(x0) + __popc(x1)) + (__popc(x2) + __popc(x3));
    }
    for (; w < w1; w++) n += __popc(mi[w] & mj[w]);
    const int bi = c.ids ? c.ids[i] : c.oadj[i], bj = c.ids ? c.ids[j] : c.oadj[j];
    const int di = c.degs ? c.degs[i] : c.deg[bi], dj = c.degs ? c.degs[j] : c.deg[bj];
    const int si = c.sups ? c.sups[i] : (int)c.osup[i], sj = c.sups ? c.sups[j] : (int)c.osup[j];
    return triangle_value<MODE == kRing, A>(p, c.rl, c.a, bi, bj, c.da, di, dj, si, sj, (int)t.y, n);
  }
  // each 4-clique a < {i, j, l} once, from its two smallest indices: l above
  // both; its largest vertex's tails from the pair that leaves out the middle
  const int lo = min(i, j), hi = max(i, j);
  int above = 0, between = 0;
  for (int w = max(w0, MODE == 2 ? lo >> 5 : hi >> 5); w < w1; w++) {
    const unsigned x = mi[w] & mj[w];
    const int b = w << 5;
    const unsigned up = hi < b ? 0xffffffffu : (hi - b >= 31 ? 0u : 0xfffffffeu << (hi - b));
    above += __popc(x & up);
    if (MODE == 2) {
      const unsigned ul = lo < b ? 0xffffffffu : (lo - b >= 31 ? 0u : 0xfffffffeu << (lo - b));
      between += __popc(x & ul & ~up);  // hi itself is not its own neighbour
    }
  }
  if (MODE == 1) return A((u64)above);
  if ((above | between) == 0) return A(0);
  const A th = nck_a<A>(c.deg[c.oadj[hi]] - 3, tails);
  A s = A((u64)between) * th;
  if (above) s += A((u64)above) * (nck_a<A>(c.da - 3, tails) + nck_a<A>(c.deg[c.oadj[lo]] - 3, tails) + th);
  return s;
}

// The vertex of `c` (its rows and arrays allotted), by one warp or (NT > 32) the
// whole block of NT threads.  The triangle core needs all position words at
// once; the 4-cliques are sums over words, so a vertex whose rows do not fit is
// counted slab by slab.  Warps take `grab` lists at a time from `next`.
template <int MODE, int NT, class A>
__device__ __forceinline__ void count_vertex(const GView& g, const VertexCtx& c, const TriShared& ps, int tails,
                                             const OutTable& tab, int* arr, unsigned* rows, uint2* stage, int* next,
                                             A& acc) {
  constexpr bool BLOCK = NT > 32;
  const int lane = threadIdx.x & 31;
  const int gt = BLOCK ? (int)threadIdx.x : lane;
  auto sync = [&]() {
    __syncwarp();
    if (BLOCK) block_sync();
  };
  auto take = [&](int* from, int grab) {  // the warp's next lists
    int b = 0;
    if (lane == 0) b = atomicAdd(from, grab);
    return __shfl_sync(0xffffffffu, b, 0);
  };
  const int k = c.k;
  const int slots = 1 << (32 - tab.shift);
  const int words = k * c.stride;
  for (int i = gt; i < slots; i += NT) tab.key[i] = -1;
  for (int i = gt; i < words; i += NT) rows[i] = 0u;
  if (gt == 0) next[0] = next[1] = 0;
  sync();
  const int* nb = g.adj + g.off[c.a];
  for (int j = gt; j < k; j += NT) {
    const int b = __ldg(c.oadj + j);
    unsigned s = out_hash(b, tab.shift);
    const unsigned mask = (unsigned)slots - 1u;
    for (unsigned probe = 0; probe <= mask && atomicCAS(tab.key + s, -1, b) != -1; probe++) s = (s + 1) & mask;
    tab.val[s] = (unsigned short)j;
    arr[j] = MODE % 3 == 0 ? min(lower_bound_dev(nb, c.da, b), c.da - 1) : j;
    if (c.ids) {
      arr[k + j] = b;
      arr[2 * k + j] = __ldg(c.deg + b);
      arr[3 * k + j] = (int)__ldg(c.osup + j);
    }
  }
  sync();
  // rows
  {
    const int* list = MODE % 3 == 0 ? nb : c.oadj;
    const int len = MODE % 3 == 0 ? c.da : k;
    const int grab = BLOCK ? min(32, max(1, len / (NT / 32 * 4))) : 32;
    const int stride = c.stride, w0 = c.w0, span = c.w1 - c.w0;
    for (int base = take(next, grab); base < len; base = take(next, grab)) {
      const int q = base + lane;
      long long first = 0;
      int n = 0, own = -1;
      if (lane < grab && q < len) {
        const int x = __ldg(list + q);
        first = g.ooff[x];
        n = (int)(g.ooff[x + 1] - first);
        own = MODE % 3 == 0 ? out_find(tab, x) : q;
        if (own < 0 && n == 1) n = 0;  // the one entry is a
      }
      __syncwarp();
      ListWalk lists;
      lists.open(first, n);
      while (!lists.done()) {
        // four steps' entries in flight
        int who[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          who[u] = -1;
          y[u] = -1;
          if (!lists.done()) {
            long long e;
            who[u] = lists.step(e);
            if (who[u] >= 0) y[u] = __ldg(g.oadj + e);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int i = __shfl_sync(0xffffffffu, own, max(who[u], 0));
          const int j = y[u] >= 0 ? out_find(tab, y[u]) : -1;
          if (j >= 0) {
            auto mark = [&](int row, int at) {
              const int w = (at >> 5) - w0;
              if (MODE % 3 == 0 || (unsigned)w < (unsigned)span) atomicOr(rows + row * stride + w, 1u << (at & 31));
            };
            mark(j, base + who[u]);
            if (i >= 0) mark(i, MODE % 3 == 0 ? arr[j] : j);
          }
          __syncwarp();
        }
      }
    }
  }
  sync();
  // triangles: entries of the out-neighbours' lists that are out-neighbours of a
  // themselves, gathered until there is one per lane
  const int grab = BLOCK ? min(32, max(1, k / (NT / 32 * 4))) : 32;
  ListWalk lists;
  int fill = 0, base = 0;
  bool more = true;
  for (;;) {
    while (fill < 32 && more) {
      if (lists.done()) {
        base = take(next + 1, grab);
        more = base < k;
        const int i = base + lane;
        long long first = 0;
        int n = 0;
        if (lane < grab && i < k && __ldg(c.osup + i) != 0) {
          const int b = __ldg(c.oadj + i);
          first = g.ooff[b];
          n = (int)(g.ooff[b + 1] - first);
        }
        lists.open(first, n);
        continue;
      }
      // two steps at a time: their entries and supports are in flight together
      int who[2], y[2];
      unsigned sup[2];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        who[u] = -1;
        y[u] = -1;
        sup[u] = 0;
        if (!lists.done()) {
          long long e;
          who[u] = lists.step(e);
          if (who[u] >= 0) {
            y[u] = __ldg(g.oadj + e);
            if (MODE % 3 == 0) sup[u] = __ldg(g.osup + e);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int j = y[u] >= 0 ? out_find(tab, y[u]) : -1;
        __syncwarp();
        const unsigned hit = __ballot_sync(0xffffffffu, j >= 0);
        if (j >= 0)
          stage[fill + __popc(hit & ((1u << lane) - 1u))] = make_uint2((unsigned)(base + who[u]) | ((unsigned)j << 16), sup[u]);
        fill += __popc(hit);
      }
      __syncwarp();
    }
    if (fill == 0) break;
    const int now = min(fill, 32);
    fill -= now;
    const bool on = lane < now;
    const uint2 t = on ? stage[fill + lane] : make_uint2(0u, 0u);
    __syncwarp();
    if (on) acc += triangle_of<MODE, A>(c, ps, tails, t);
    __syncwarp();
  }
  sync();
}

// Whether a 4-clique can have its lowest vertex where these out-edges start: three
// of them must be in two triangles or more.  Called by a warp; four loads a lane
// in flight, and most vertices with cliques are known after the first.  Tables
// for every vertex of three out-neighbours cost 487 ms on two complete sides of
// 6,000 with seven edges inside them, now 1.0 ms (lists merged: 1.7 ms); uniform, 16
// entries a vertex, n = 100,000: 0.17 ms, now 0.05 ms (0.12 ms).
__device__ __forceinline__ bool may_hold_clique(const unsigned* __restrict__ osup, int k) {
  const int lane = threadIdx.x & 31;
  int found = 0;
  for (int j0 = 0; j0 < k && found < 3; j0 += 128) {
    unsigned s[4];
#pragma unroll
    for (int u = 0; u < 4; u++) s[u] = j0 + 32 * u + lane < k ? __ldg(osup + j0 + 32 * u + lane) : 0;
#pragma unroll
    for (int u = 0; u < 4; u++) found += __popc(__ballot_sync(0xffffffffu, s[u] >= 2));
  }
  return found >= 3;
}

// The narrow blocks look at every vertex and take those that are not
// triangle_wide (warp-sized ones among them); the wide ones take the graph's
// list of wide vertices one at a time.
template <int MODE, int NT, class A>
__global__ void __launch_bounds__(NT, NT == kNarrow ? 6 : 2)
    triangle_kernel(GView g, TriLaunch p, int batch, int* __restrict__ queue,
                    unsigned* __restrict__ arena, u64* __restrict__ slot) {
  constexpr int NW = NT / 32;
  extern __shared__ __align__(16) unsigned s_tri[];
  __shared__ int s_item, s_nlist, s_list[32], s_next[NW][2];
  __shared__ TriShared s_p;
  __shared__ VertexCtx s_ctx[NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // [stage][table keys][table values][arrays][rows]; warp-sized vertices carve
  // their own pieces out of the rows
  uint2* stage = reinterpret_cast<uint2*>(s_tri) + warp * kStage;
  int* keys = reinterpret_cast<int*>(s_tri + NW * kStage * 2);
  unsigned short* vals = reinterpret_cast<unsigned short*>(keys + p.slots);
  int* arrays = keys + p.slots + p.slots / 2;
  unsigned* rows = reinterpret_cast<unsigned*>(arrays + p.arrays * p.kmax);
  unsigned* mine = rows + warp * kSmallWords;
  if (threadIdx.x == 0) {
    s_p.sum1 = p.eval.sum1;
    s_p.sum2 = p.eval.sum2;
    s_p.sum3 = p.eval.sum3;
    s_p.rot.count = p.eval.rot.count;
#pragma unroll
    for (int r = 0; r < 6; r++)
#pragma unroll
      for (int q = 0; q < 8; q++) s_p.rot.fr[r][q] = p.eval.rot.fr[r][q];
  }
  A acc = A(0);
  auto flush_member = [&](int a) {  // packed graphs: the sums of one vertex go to its member's slot
    if constexpr (std::is_same<A, u64>::value) {
      if (g.comp == nullptr) return;
      const u64 s = warp_sum_u64(acc);
      if (lane == 0 && s) atomicAdd(g.comp_slots + g.comp[a], s);
      acc = 0;
    }
  };
  auto shift_for = [](int k, int least) {
    int b = least;
    while ((1 << b) < 2 * k) b++;
    return 32 - b;
  };
  auto open = [&](VertexCtx& c, int a, int k, int da, long long ob, int* arr, bool all, unsigned* m, int stride, int w0, int w1) {
    c.a = a;
    c.da = da;
    c.k = k;
    c.rl = relabel_of(g, p.relabel, a);
    c.stride = stride;
    c.w0 = w0;
    c.w1 = w1;
    c.rows = m;
    c.oadj = g.oadj + ob;
    c.osup = g.osup + ob;
    c.deg = g.deg;
    c.ids = all ? arr + k : nullptr;
    c.degs = all ? arr + 2 * k : nullptr;
    c.sups = all ? arr + 3 * k : nullptr;
  };
  for (;;) {
    block_sync();
    if (threadIdx.x == 0) {
      s_item = atomicAdd(queue, batch);
      s_nlist = 0;
    }
    block_sync();
    const int v0 = s_item;
    if (v0 >= p.items) break;
    for (int i = warp; i < batch; i += NW) {
      if (v0 + i >= p.items) break;
      const int a = p.list ? p.list[v0 + i] : v0 + i;
      const long long ob = g.ooff[a];
      const int k = (int)(g.ooff[a + 1] - ob), da = g.deg[a];
      if (k < (MODE % 3 == 0 ? 2 : 3) || (MODE % 3 == 0 && da < p.eval.sum1)) continue;
      const int W = ((MODE % 3 == 0 ? da : k) + 31) >> 5, stride = W | 1;
      const int lists = MODE % 3 == 0 ? da : k;
      if ((NT == kNarrow) == triangle_wide(k, lists)) continue;
      if (MODE % 3 != 0 && !may_hold_clique(g.osup + ob, k)) continue;
      if (k > kSmallK || k * stride > kSmallRows || lists > kSmallLists) {
        if (lane == 0) s_list[atomicAdd(&s_nlist, 1)] = a;
        continue;
      }
      OutTable t;
      t.key = reinterpret_cast<int*>(mine + kSmallRows);
      t.val = reinterpret_cast<unsigned short*>(mine + kSmallRows + kSmallSlots);
      t.shift = shift_for(k, 3);
      int* arr = reinterpret_cast<int*>(mine + kSmallRows + kSmallSlots + kSmallSlots / 2);
      if (lane == 0) open(s_ctx[warp], a, k, da, ob, arr, true, mine, stride, 0, W);
      __syncwarp();
      count_vertex<MODE, 32, A>(g, s_ctx[warp], s_p, p.tails, t, arr, mine, stage, s_next[warp], acc);
      flush_member(a);
    }
    block_sync();
    const int nlist = s_nlist;
    for (int li = 0; li < nlist; li++) {
      const int a = s_list[li];
      const long long ob = g.ooff[a];
      const int k = (int)(g.ooff[a + 1] - ob), da = g.deg[a];
      const int W = ((MODE % 3 == 0 ? da : k) + 31) >> 5;
      OutTable t;
      t.key = keys;
      t.val = vals;
      t.shift = shift_for(k, 6);
      const bool fits = (long long)k * (W | 1) <= p.rows;
      const int slab = MODE % 3 == 0 || fits ? W : max(1, (p.rows / k - 1) | 1);
      for (int w0 = 0; w0 < W; w0 += slab) {
        // rows in the arena: only the wide blocks' triangle core
        unsigned* far = MODE % 3 == 0 && NT == kWide && !fits ? arena + (size_t)blockIdx.x * (size_t)p.gstride : nullptr;
        if (threadIdx.x == 0)
          open(s_ctx[0], a, k, da, ob, arrays, p.arrays == 4, far ? far : rows, fits ? W | 1 : MODE % 3 == 0 ? W : slab, w0,
               min(W, w0 + slab));
        block_sync();
        if (MODE % 3 == 0 && NT == kWide && far)
          count_vertex<MODE, NT, A>(g, s_ctx[0], s_p, p.tails, t, arrays, far, stage, s_next[0], acc);
        else
          count_vertex<MODE, NT, A>(g, s_ctx[0], s_p, p.tails, t, arrays, rows, stage, s_next[0], acc);
      }
      flush_member(a);
    }
  }
  block_sum_to(acc, slot);
}

// Shared memory of one block: tables and arrays for `kmax` out-neighbours, the
// rest row words.
size_t shape_block(TriLaunch& p, int kmax, int warps, size_t smem) {
  p.kmax = kmax;
  p.slots = 64;
  while (p.slots < 2 * kmax) p.slots *= 2;
  p.arrays = kmax <= kArraysMax ? 4 : 1;
  const size_t fixed = sizeof(unsigned) * ((size_t)warps * kStage * 2 + (size_t)p.slots + p.slots / 2 + (size_t)p.arrays * kmax);
  const size_t least = sizeof(unsigned) * (size_t)warps * kSmallWords;
  const size_t bytes = std::max(fixed + least, smem);
  p.rows = (int)((bytes - fixed) / sizeof(unsigned));
  return bytes;
}

constexpr size_t kWideSmem = 111 * 1024;

// Rows of the triangle core that do not fit in a wide block's shared memory (each
// with at most one pad word) go to the arena: unpadded, at most 8 GiB in all.
bool rows_fit(const DevGraph& G, int rows) { return G.max_bitmap_words + G.max_outdeg <= rows; }
long long arena_words(const DevGraph& G) { return std::max(1LL, G.max_bitmap_words); }
int arena_blocks(const DevGraph& G) {
  const size_t per = sizeof(unsigned) * (size_t)arena_words(G);
  return (int)std::max<size_t>(1, std::min<size_t>((size_t)2 * sm_count(), ((size_t)8 << 30) / per));
}

template <int MODE, int NT, class A>
int launch_blocks(DevGraph& G, const GView& gv, const TriLaunch& p, size_t smem, u64* slot, cudaStream_t s, int blocks,
                  uint64_t* launches, DevWork& work) {
  int* queue = reinterpret_cast<int*>(work.small + 6);
  cudaMemsetAsync(queue, 0, sizeof(int), s);
  cudaFuncSetAttribute(triangle_kernel<MODE, NT, A>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  // vertices a block takes at a time: one per warp at least, few enough that the
  // blocks end together
  const int batch = p.list ? 1 : std::max(NT / 32, std::min(32, p.items / (blocks * 24)));
  triangle_kernel<MODE, NT, A><<<blocks, NT, smem, s>>>(gv, p, batch, queue, reinterpret_cast<unsigned*>(work.tri.ptr), slot);
  *launches += 1;
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

template <int MODE, class A>
int launch_mode(DevGraph& G, const GView& gv, TriLaunch p, u64* slot, cudaStream_t s, uint64_t* launches, DevWork& work) {
  const int kmax = (int)std::max(1LL, G.max_outdeg);
  TriLaunch n = p;
  const size_t nsmem = shape_block(n, std::min(kmax, kTriNarrowK), kNarrow / 32, 35 * 1024);
  const size_t wsmem = shape_block(p, kmax, kWide / 32, kWideSmem);
  if (n.rows < kTriNarrowRows) return FSGC_EINVAL;  // the block holds what triangle_wide leaves to it
  n.items = G.n;
  p.list = G.wide;
  p.items = G.nwide;
  int st = launch_blocks<MODE, kNarrow, A>(G, gv, n, nsmem, slot, s, 6 * sm_count(), launches, work);
  if (st != FSGC_OK || G.nwide == 0) return st;
  int blocks = 2 * sm_count();
  if (MODE % 3 == 0 && !rows_fit(G, p.rows)) {
    blocks = arena_blocks(G);
    p.gstride = arena_words(G);
    st = ensure_plain_scratch(work.tri, triangle_scratch(G), s);
    if (st != FSGC_OK) return st;
  }
  return launch_blocks<MODE, kWide, A>(G, gv, p, wsmem, slot, s, blocks, launches, work);
}

}  // namespace

size_t triangle_scratch(const DevGraph& G) {
  TriLaunch p;
  shape_block(p, (int)std::max(1LL, G.max_outdeg), kWide / 32, kWideSmem);
  if (G.nwide == 0 || rows_fit(G, p.rows)) return 0;
  return sizeof(unsigned) * (size_t)arena_words(G) * (size_t)arena_blocks(G);
}

// 4-cliques of graphs whose lists all hold a few entries are found by merging them
// (triangle_core_kernel): the blocks' turns over the vertices cost more.  Rings of
// cliques of 4, 6, 7, 8 and 9, merged and by tables: 0.04 and 0.15 ms, 0.05 and 0.09,
// 0.06 and 0.09, 0.09 and 0.10, 0.11 and 0.09; a path of 2^20 0.04 and 0.10, uniform
// with 3 entries a vertex, n = 2 M (5 out-neighbours at most), 0.13 and 0.19, with 8,
// n = 20,000 (9), 0.03 and 0.03.
constexpr int kMergeOut = 8;

bool triangle_by_tables(const DevGraph& G, bool clique) {
  return G.max_outdeg <= kMaxOut && G.m / 2 > 0 && !(clique && G.max_outdeg <= kMergeOut);
}

int enqueue_triangle(DevGraph& G, const GView& gv, const TrianglePattern& tp, bool exact, u64* slot, cudaStream_t s,
                     uint64_t* launches, DevWork& work) {
  TriLaunch p;
  memset(&p, 0, sizeof(p));
  p.eval.sum1 = tp.sum1;
  p.eval.sum2 = tp.sum2;
  p.eval.sum3 = tp.sum3;
  p.tails = tp.tails;
  p.relabel = tp.relabel;
  p.eval.rot = tp.rot;
  int k = 0;
  for (int i = 0; i < 8; i++) k = std::max(k, tp.rot.fr[0][i]);
  const bool ring = !exact && binomials_fit(G.maxdeg, k);
#define FSGC_TRI(MODE)                                                                          \
  return exact ? launch_mode<MODE, X128>(G, gv, p, slot, s, launches, work)                 \
               : launch_mode<MODE, u64>(G, gv, p, slot, s, launches, work)
  if (tp.mode == 1) FSGC_TRI(1);
  if (tp.mode == 2) FSGC_TRI(2);
  if (ring) return launch_mode<kRing, u64>(G, gv, p, slot, s, launches, work);
  FSGC_TRI(0);
#undef FSGC_TRI
}

}  // namespace fsgc
