// Graph loader on the GPU: degrees, the degree-ordered orientation of every
// undirected edge, and per-edge triangle supports.
//
// The reference relabels vertices by degree with CUB radix sorts inside the
// triangle-core count (relabelByDegree, src/fringeCount.cu:1221-1288) and builds
// a fresh degree-pruned worklist with one global atomic per edge for every count
// (init_wl_*, :617-663, 1167-1218, 1653-1751, 2054-2103).  Here a graph is
// prepared once when it becomes resident: the orientation (lower (deg, id)
// endpoint -> higher) bounds out-degrees by O(sqrt m), and one pass over the
// oriented edges computes |N(x) & N(y)| for every edge, which the edge,
// triangle and wedge cores all consume.  No relabel is needed: kernels compare
// (deg, id) pairs directly, which is the order the reference's relabel induces.
#include <algorithm>
#include <cstdio>

#include <cub/cub.cuh>

#include "fsgc_internal.h"

namespace fsgc {

namespace {

constexpr int kTPB = 256;

__device__ __forceinline__ bool above(int w, int dw, int v, int dv) {  // (dw, w) > (dv, v)
  return (dw > dv) || (dw == dv && w > v);
}

__global__ void degree_kernel(int n, const long long* __restrict__ off, int* __restrict__ deg,
                              int* __restrict__ maxdeg) {
  int local = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int d = (int)(off[v + 1] - off[v]);
    deg[v] = d;
    local = max(local, d);
  }
  local = __reduce_max_sync(0xffffffffu, local);
  if ((threadIdx.x & 31) == 0) atomicMax(maxdeg, local);
}

// One warp per vertex; lists are read kOrientRun entries a lane at a time, all
// loads before their uses: a warp's time is the latency of entry and degree, and
// a hub's list is one warp's.  RMAT n = 2^20, 31 M entries, hub of 65,000:
// filling 2.7 -> 0.67 ms; the out-degrees stay at 0.85 ms, most of it the random
// reads of degrees.
constexpr int kOrientRun = 8;

// Whether entries j, j + 32, ... of v's list stand above v; w: the entries.
__device__ __forceinline__ unsigned orient_run(const GView& g, long long j, long long e, int v, int dv, int* w) {
  unsigned up = 0;
#pragma unroll
  for (int i = 0; i < kOrientRun; i++) w[i] = j + i * 32 < e ? __ldg(g.adj + j + i * 32) : -1;
  int dw[kOrientRun];
#pragma unroll
  for (int i = 0; i < kOrientRun; i++) dw[i] = w[i] >= 0 ? __ldg(g.deg + w[i]) : -1;
#pragma unroll
  for (int i = 0; i < kOrientRun; i++) up |= (unsigned)above(w[i], dw[i], v, dv) << i;
  return up;
}

// number of neighbours above each vertex in degree order
__global__ void outdeg_kernel(GView g, long long* __restrict__ odeg) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int v = wid; v < g.n; v += nw) {
    const int dv = g.deg[v];
    const long long e = g.off[v + 1];
    int c = 0;
    for (long long j0 = g.off[v]; j0 < e; j0 += 32 * kOrientRun) {
      int w[kOrientRun];
      c += __popc(orient_run(g, j0 + lane, e, v, dv, w));
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) odeg[v] = c;
  }
}

__global__ void orient_fill_kernel(GView g, int* __restrict__ oadj, int* __restrict__ osrc) {
  const int lane = threadIdx.x & 31;
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int v = wid; v < g.n; v += nw) {
    const int dv = g.deg[v];
    const long long e = g.off[v + 1];
    long long o = g.ooff[v];
    for (long long j0 = g.off[v]; j0 < e; j0 += 32 * kOrientRun) {
      int w[kOrientRun];
      const unsigned up = orient_run(g, j0 + lane, e, v, dv, w);
#pragma unroll
      for (int i = 0; i < kOrientRun; i++) {
        if (j0 + i * 32 >= e) break;
        const bool p = up >> i & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, p);
        if (p) {
          const long long pos = o + __popc(bal & lt);
          oadj[pos] = w[i];
          osrc[pos] = v;
        }
        o += __popc(bal);
      }
    }
  }
}

// ---- exclusive scan of n int64 values into out[0..n] (out[n] = total)
constexpr int kScanTile = 2048;  // 256 threads x 8

__device__ __forceinline__ long long block_excl_scan(long long x, long long* s_warp, long long& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long inc = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) s_warp[w] = inc;
  block_sync();
  if (w == 0) {
    long long t = (lane < (int)(blockDim.x >> 5)) ? s_warp[lane] : 0;
    long long ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti += y;
    }
    if (lane < (int)(blockDim.x >> 5)) s_warp[lane] = ti - t;
    if (lane == 31) s_warp[32] = ti;
  }
  block_sync();
  const long long r = s_warp[w] + inc - x;
  total = s_warp[32];
  block_sync();
  return r;
}

__global__ void scan_tiles_kernel(const long long* __restrict__ in, long long n, long long* __restrict__ tile_sum) {
  __shared__ long long s_warp[33];
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * 8;
  long long x = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) x += (base + i < n) ? in[base + i] : 0;
  long long tot;
  block_excl_scan(x, s_warp, tot);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

__global__ void scan_sums_kernel(long long* __restrict__ sums, long long nt) {  // one block, in place
  __shared__ long long s_warp[33];
  long long carry = 0;
  for (long long b = 0; b < nt; b += blockDim.x) {
    const long long i = b + threadIdx.x;
    const long long x = (i < nt) ? sums[i] : 0;
    long long tot;
    const long long ex = block_excl_scan(x, s_warp, tot);
    if (i < nt) sums[i] = carry + ex;
    carry += tot;
  }
}

__global__ void scan_apply_kernel(const long long* __restrict__ in, long long n, const long long* __restrict__ tile_off,
                                  long long* __restrict__ out) {
  __shared__ long long s_warp[33];
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * 8;
  long long v[8];
  long long x = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    v[i] = (base + i < n) ? in[base + i] : 0;
    x += v[i];
  }
  long long tot;
  long long run = block_excl_scan(x, s_warp, tot) + tile_off[blockIdx.x];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = run;
}

// ---- triangle supports: thread per oriented edge (a -> b); the common
// out-neighbours c of a and b close the triangles a < b < c, each found once.
__device__ __forceinline__ void tri_found(unsigned* __restrict__ osup, long long sa, long long sb) {
  atomicAdd(osup + sa, 1u);
  atomicAdd(osup + sb, 1u);
}

__global__ void triangle_support_kernel(GView g, unsigned* __restrict__ osup, u64* __restrict__ tri_total) {
  const long long me = g.m / 2;
  u64 tot = 0;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const int a = g.osrc[j], b = g.oadj[j];
    const long long ab = g.ooff[a], bb = g.ooff[b];
    const int la = (int)(g.ooff[a + 1] - ab), lb = (int)(g.ooff[b + 1] - bb);
    if (lb == 0) continue;
    const int* A = g.oadj + ab;
    const int* B = g.oadj + bb;
    unsigned cnt = 0;
    if ((long long)la * 16 < lb) {
      for (int i = 0; i < la; i++) {
        const int p = bsearch_pos(B, lb, A[i]);
        if (p >= 0) { cnt++; tri_found(osup, ab + i, bb + p); }
      }
    } else if ((long long)lb * 16 < la) {
      for (int k = 0; k < lb; k++) {
        const int p = bsearch_pos(A, la, B[k]);
        if (p >= 0) { cnt++; tri_found(osup, ab + p, bb + k); }
      }
    } else {
      int i = 0, k = 0;
      while (i < la && k < lb) {
        const int x = __ldg(A + i), y = __ldg(B + k);
        if (x < y) i++;
        else if (y < x) k++;
        else { cnt++; tri_found(osup, ab + i, bb + k); i++; k++; }
      }
    }
    if (cnt) atomicAdd(osup + j, cnt);
    tot += cnt;
  }
  block_sum_to(tot, tri_total);
}

// ---- triangle supports of larger graphs, every list in rank order
//
// With a's list ordered by rank, its entries behind b are the candidates c of
// the edge (a, b): each pair of a's out-neighbours is looked up once, in b's
// out-neighbours, and two in five are triangles (RMAT), where merging the two
// lists reads every entry of both.  b's out-neighbours stand in a hash table in
// shared memory behind a filter of 16 bits a slot; the rests of its
// in-neighbours' lists are read as one run of entries, 32 at a time whatever
// their lengths, and those that pass the filter queue until 32 can be looked up
// together.  A hit adds to (a, c) in memory, next to the entry read, and to
// (a, b) and (b, c) in shared memory.  Up to kSupSmall out-neighbours and
// kSupPiece in-edges a warp does it, beyond that blocks, a piece at a time.
// Bound by the lookups' instructions, 3 a candidate.  RMAT n = 2^20, 15.7 M edges:
// merges 13.6 ms; here 4.0 ms in blocks, 0.8 ms in warps, 0.7 ms for the sorts and
// 0.4 ms for the passes around them.
constexpr int kSupWarps = 8;
constexpr int kSupSmall = 128;
constexpr int kSupChunk = 1024;
constexpr int kSupPiece = 1024;  // in-edges of a block's turn

// The oriented edges with every list in rank order, for the supports.
struct OrderedEdges {
  const unsigned* __restrict__ rank;   // per position: rank of the edge's upper end
  const int* __restrict__ into;        // edges (slots) by their upper end's rank
  const int* __restrict__ place;       // position of each slot
  const int* __restrict__ start;       // per rank: its first in `into`
  const int* __restrict__ rank_of;     // per vertex
  unsigned* __restrict__ sup;          // per position
};

struct SupLists {      // of one warp: the lists being read, those with entries first
  int base[32];        // entry of the run -> its position
  unsigned hits[32];
  int at[64];          // entries that passed the filter
  int id[64];
  unsigned char list[64];
};

template <class Pos>
struct SupTable {
  int* key;        // -1 where empty; at most half full
  Pos* pos;
  unsigned* hits;  // by position
  unsigned* bits;  // filter: 16 bits a slot
  int shift;       // 32 - log2 of the slots

  __device__ void insert(int id, int position) {
    const unsigned mask = 0xffffffffu >> shift;
    const unsigned f = ((unsigned)id * 0x9E3779B1u) >> (shift - 4);
    atomicOr(bits + (f >> 5), 1u << (f & 31));
    unsigned s = f >> 4;
    for (unsigned probe = 0; probe <= mask && atomicCAS(key + s, -1, id) != -1; probe++) s = (s + 1) & mask;
    pos[s] = (Pos)position;
  }
  __device__ __forceinline__ bool may_hold(int id) const {
    const unsigned f = ((unsigned)id * 0x9E3779B1u) >> (shift - 4);
    return bits[f >> 5] >> (f & 31) & 1u;
  }
  __device__ __forceinline__ int find(int id) const {
    const unsigned mask = 0xffffffffu >> shift;
    unsigned s = ((unsigned)id * 0x9E3779B1u) >> shift;
    for (unsigned probe = 0; probe <= mask; probe++) {
      const int k = key[s];
      if (k == id) return pos[s];
      if (k < 0) break;
      s = (s + 1) & mask;
    }
    return -1;
  }
};

// Slots, as a power of two of at least 32, for k keys.
__device__ __forceinline__ int sup_log2(int k) { return max(5, 33 - __clz(k - 1)); }

// One warp looks up the rest of up to 32 in-neighbours' lists, one per lane: the
// edge (a, b) stands at position p of the ordered entries (-1 for none), the
// entries of a's list above b behind it, up to `stop`.
template <class Pos>
__device__ __forceinline__ unsigned support_lists(const OrderedEdges& o, int p, int stop, const SupTable<Pos>& tab,
                                                  SupLists& w) {
  const int lane = threadIdx.x & 31;
  const int lb = p + 1, len = p >= 0 ? stop - lb : 0;
  int end = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= o) end += y;
  }
  const int start = end - len;
  const int total = __shfl_sync(0xffffffffu, end, 31);
  if (total == 0) return 0;
  const unsigned has = __ballot_sync(0xffffffffu, len > 0);
  const int rank = __popc(has & ((1u << lane) - 1u));
  if (len > 0) w.base[rank] = lb - start;
  w.hits[lane] = 0;
  __syncwarp();
  unsigned found = 0;
  int before = -1;  // lists begun, less one
  int queued = 0;
  auto drain = [&](int first, int count) {
    if (lane < count) {
      const int q = first + lane;
      const int p = tab.find(w.id[q]);
      if (p >= 0) {
        atomicAdd(tab.hits + p, 1u);
        atomicAdd(w.hits + w.list[q], 1u);
        atomicAdd(o.sup + w.at[q], 1u);
        found++;
      }
    }
    __syncwarp();
  };
  int r = 0, id = -1;
  int at = 0;
  auto fetch = [&](int t0) {
    const unsigned d = (unsigned)(start - t0);
    const unsigned begun = __reduce_or_sync(0xffffffffu, len > 0 && d < 32u ? 1u << d : 0u);
    r = before + __popc(begun & (0xffffffffu >> (31 - lane)));
    before += __popc(begun);
    id = -1;
    if (t0 + lane < total) {
      at = w.base[r] + t0 + lane;
      id = (int)__ldg(o.rank + at);
    }
  };
  fetch(0);
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int r0 = r, id0 = id;
    const int at0 = at;
    if (t0 + 32 < total) fetch(t0 + 32);
    const bool pass = id0 >= 0 && tab.may_hold(id0);
    const unsigned bal = __ballot_sync(0xffffffffu, pass);
    if (pass) {
      const int q = queued + __popc(bal & ((1u << lane) - 1u));
      w.at[q] = at0;
      w.id[q] = id0;
      w.list[q] = (unsigned char)r0;
    }
    queued += __popc(bal);
    __syncwarp();
    if (queued >= 32) {
      queued -= 32;
      drain(queued, 32);
    }
  }
  drain(0, queued);
  if (len > 0 && w.hits[rank]) atomicAdd(o.sup + p, w.hits[rank]);
  __syncwarp();
  return found;
}

// Work of the two support kernels: the queues' heads, and behind them the pieces
// (vertex, first in-edge) left to the blocks.
struct SupWork {
  unsigned next_small, next_wide, nwide, pad;
  __device__ int2* wide() { return reinterpret_cast<int2*>(this + 1); }
};

// In-neighbours of one piece, by one warp: positions p and ends of their lists.
template <class Pos>
__device__ __forceinline__ unsigned support_piece(const GView& g, const OrderedEdges& o, int i, int last,
                                                  const SupTable<Pos>& tab, SupLists& w) {
  int p = -1, stop = 0;
  if (i < last) {
    const int e = __ldg(o.into + i);
    p = __ldg(o.place + e);
    stop = (int)__ldg(g.ooff + __ldg(g.osrc + e) + 1);
  }
  return support_lists(o, p, stop, tab, w);
}

__global__ void __launch_bounds__(kSupWarps * 32) support_warp_kernel(GView g, OrderedEdges o, int grab,
                                                                      SupWork* __restrict__ work,
                                                                      u64* __restrict__ tri_total) {
  __shared__ int s_key[kSupWarps][2 * kSupSmall];
  __shared__ unsigned char s_pos[kSupWarps][2 * kSupSmall];
  __shared__ unsigned s_hits[kSupWarps][kSupSmall];
  __shared__ unsigned s_bits[kSupWarps][kSupSmall];
  __shared__ SupLists s_lists[kSupWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u64 tot = 0;
  for (;;) {
    unsigned base = 0;
    if (lane == 0) base = atomicAdd(&work->next_small, (unsigned)grab);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= (unsigned)g.n) break;
    int bb_l = 0, k_l = 0, in_l = 0, last_l = 0;
    if (lane < grab && base + lane < (unsigned)g.n) {
      const int b = (int)base + lane;
      bb_l = (int)g.ooff[b];
      k_l = (int)g.ooff[b + 1] - bb_l;
      const int r = o.rank_of[b];
      in_l = o.start[r];
      last_l = o.start[r + 1];
      if (k_l > 0 && last_l > in_l && (k_l > kSupSmall || last_l - in_l > kSupPiece)) {
        const int pieces = (last_l - in_l + kSupPiece - 1) / kSupPiece;
        const unsigned at = atomicAdd(&work->nwide, (unsigned)pieces);
        for (int q = 0; q < pieces; q++) work->wide()[at + q] = make_int2(b, in_l + q * kSupPiece);
        k_l = 0;
      }
    }
    unsigned bal = __ballot_sync(0xffffffffu, k_l > 0 && last_l > in_l);
    while (bal) {
      const int who = __ffs(bal) - 1;
      bal &= bal - 1;
      const int bb = __shfl_sync(0xffffffffu, bb_l, who), k = __shfl_sync(0xffffffffu, k_l, who);
      const int in = __shfl_sync(0xffffffffu, in_l, who), last = __shfl_sync(0xffffffffu, last_l, who);
      const int log2 = sup_log2(k);
      SupTable<unsigned char> tab{s_key[warp], s_pos[warp], s_hits[warp], s_bits[warp], 32 - log2};
      for (int i = lane; i < 1 << log2; i += 32) tab.key[i] = -1;
      for (int i = lane; i < 1 << (log2 - 1); i += 32) tab.bits[i] = 0;
      for (int i = lane; i < k; i += 32) tab.hits[i] = 0;
      __syncwarp();
      for (int i = lane; i < k; i += 32) tab.insert((int)__ldg(o.rank + bb + i), i);
      __syncwarp();
      for (int i0 = in; i0 < last; i0 += 32) tot += support_piece(g, o, i0 + lane, last, tab, s_lists[warp]);
      for (int i = lane; i < k; i += 32)
        if (tab.hits[i]) atomicAdd(o.sup + bb + i, tab.hits[i]);
      __syncwarp();
    }
  }
  block_sum_to(tot, tri_total);
}

constexpr int kSupBlock = 256;

__global__ void __launch_bounds__(kSupBlock) support_block_kernel(GView g, OrderedEdges o, SupWork* __restrict__ work,
                                                                  u64* __restrict__ tri_total) {
  __shared__ int s_key[2 * kSupChunk];
  __shared__ unsigned short s_pos[2 * kSupChunk];
  __shared__ unsigned s_hits[kSupChunk];
  __shared__ unsigned s_bits[kSupChunk];
  __shared__ SupLists s_lists[kSupBlock / 32];
  __shared__ int s_turn, s_next;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned nwide = work->nwide;  // the warps' kernel has ended
  u64 tot = 0;
  for (;;) {
    if (threadIdx.x == 0) s_turn = (int)min(atomicAdd(&work->next_wide, 1u), nwide);
    block_sync();
    const unsigned turn = (unsigned)s_turn;
    if (turn >= nwide) break;
    const int2 piece = work->wide()[turn];
    const int bb = (int)g.ooff[piece.x], k = (int)g.ooff[piece.x + 1] - bb;
    const int last = min(o.start[o.rank_of[piece.x] + 1], piece.y + kSupPiece);
    for (int c0 = 0; c0 < k; c0 += kSupChunk) {
      const int kc = min(kSupChunk, k - c0);
      const int log2 = sup_log2(kc);
      SupTable<unsigned short> tab{s_key, s_pos, s_hits, s_bits, 32 - log2};
      for (int i = threadIdx.x; i < 1 << log2; i += kSupBlock) s_key[i] = -1;
      for (int i = threadIdx.x; i < 1 << (log2 - 1); i += kSupBlock) s_bits[i] = 0;
      for (int i = threadIdx.x; i < kc; i += kSupBlock) s_hits[i] = 0;
      if (threadIdx.x == 0) s_next = piece.y;
      block_sync();
      for (int i = threadIdx.x; i < kc; i += kSupBlock) tab.insert((int)__ldg(o.rank + bb + c0 + i), i);
      block_sync();
      for (;;) {
        int i0 = 0;
        if (lane == 0) i0 = atomicAdd(&s_next, 32);
        i0 = __shfl_sync(0xffffffffu, i0, 0);
        if (i0 >= last) break;
        tot += support_piece(g, o, i0 + lane, last, tab, s_lists[warp]);
      }
      block_sync();
      for (int i = threadIdx.x; i < kc; i += kSupBlock)
        if (s_hits[i]) atomicAdd(o.sup + bb + c0 + i, s_hits[i]);
      block_sync();
    }
  }
  block_sum_to(tot, tri_total);
}

__global__ void degree_keys_kernel(GView g, unsigned* __restrict__ key, int* __restrict__ id) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    key[v] = (unsigned)g.deg[v];
    id[v] = v;
  }
}
__global__ void rank_scatter_kernel(int n, const int* __restrict__ by_rank, int* __restrict__ rank_of) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) rank_of[by_rank[r]] = r;
}
__global__ void upper_keys_kernel(GView g, int me, const int* __restrict__ rank_of, unsigned* __restrict__ key,
                                  int* __restrict__ slot) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < me; e += gridDim.x * blockDim.x) {
    key[e] = (unsigned)rank_of[g.oadj[e]];
    slot[e] = e;
  }
}
__global__ void into_starts_kernel(int n, const unsigned* __restrict__ key, int me, int* __restrict__ start) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= n; r += gridDim.x * blockDim.x) {
    int lo = 0, hi = me;
    while (lo < hi) {
      const int mid = lo + (hi - lo) / 2;
      if (key[mid] < (unsigned)r) lo = mid + 1;
      else hi = mid;
    }
    start[r] = lo;
  }
}
__global__ void lower_keys_kernel(GView g, int me, const int* __restrict__ into, unsigned* __restrict__ key) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < me; i += gridDim.x * blockDim.x) key[i] = (unsigned)g.osrc[into[i]];
}
__global__ void places_kernel(GView g, int me, const int* __restrict__ slot, const int* __restrict__ rank_of,
                              unsigned* __restrict__ rank, int* __restrict__ place) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < me; p += gridDim.x * blockDim.x) {
    const int e = slot[p];
    rank[p] = (unsigned)rank_of[g.oadj[e]];
    place[e] = p;
  }
}
__global__ void supports_back_kernel(int me, const int* __restrict__ place, const unsigned* __restrict__ sup,
                                     unsigned* __restrict__ osup) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < me; e += gridDim.x * blockDim.x) osup[e] = sup[place[e]];
}

// Largest out-degree, largest out-degree * ceil(deg / 32) (bitmap rows), the
// number of vertices whose triangles take a wide block, and the sums of squares of
// out-degrees and (stats[5]) of degrees.
__global__ void outdeg_stats_kernel(GView g, unsigned long long* __restrict__ stats) {
  unsigned long long k1 = 0, k2 = 0, wide = 0, squares = 0, ends = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    const unsigned long long k = (unsigned long long)(g.ooff[v + 1] - g.ooff[v]);
    k1 = max(k1, k);
    k2 = max(k2, k * (unsigned long long)((g.deg[v] + 31) >> 5));
    wide += k >= 2 && triangle_wide((int)k, g.deg[v]);
    squares += k * k;
    ends += (unsigned long long)g.deg[v] * (unsigned long long)g.deg[v];
  }
  for (int o = 16; o > 0; o >>= 1) {
    k1 = max(k1, __shfl_down_sync(0xffffffffu, k1, o));
    k2 = max(k2, __shfl_down_sync(0xffffffffu, k2, o));
    wide += __shfl_down_sync(0xffffffffu, wide, o);
    squares += __shfl_down_sync(0xffffffffu, squares, o);
    ends += __shfl_down_sync(0xffffffffu, ends, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(stats, k1);
    atomicMax(stats + 1, k2);
    if (wide) atomicAdd(stats + 2, wide);
    if (squares) atomicAdd(stats + 4, squares);
    if (ends) atomicAdd(stats + 5, ends);
  }
}

__global__ void wide_list_kernel(GView g, int* __restrict__ list, int* __restrict__ count) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < g.n; v += gridDim.x * blockDim.x) {
    const int k = (int)(g.ooff[v + 1] - g.ooff[v]);
    if (k >= 2 && triangle_wide(k, g.deg[v])) list[atomicAdd(count, 1)] = v;
  }
}

__global__ void vertex_triangle_kernel(GView g, u64* __restrict__ vtri2) {
  const long long me = g.m / 2;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const unsigned s = g.osup[j];
    if (s) {
      atomicAdd(vtri2 + g.osrc[j], (u64)s);
      atomicAdd(vtri2 + g.oadj[j], (u64)s);
    }
  }
}

// The support of each oriented edge, written to both of its list entries.
__global__ void entry_support_kernel(GView g, unsigned* __restrict__ esup) {
  const long long me = g.m / 2;
  for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < me; j += (long long)gridDim.x * blockDim.x) {
    const int a = g.osrc[j], b = g.oadj[j];
    const unsigned s = g.osup[j];
    const long long oa = g.off[a], ob = g.off[b];
    const int pa = bsearch_pos(g.adj + oa, (int)(g.off[a + 1] - oa), b);
    const int pb = bsearch_pos(g.adj + ob, (int)(g.off[b + 1] - ob), a);
    if (pa >= 0) esup[oa + pa] = s;
    if (pb >= 0) esup[ob + pb] = s;  // absent only in a non-symmetric input
  }
}

// The ordered lists cost two sorts and a few passes; merging costs what the lists
// are long, for which the mean square of the out-degrees over the edges stands.
// Whole loads, merged and ordered: RMAT (86 to 157 squares an edge) with 1.9 M
// edges 2.2 and 2.6 ms, 3.8 M 4.1 and 3.3, 15.7 M 19.5 and 12.3; power law with 30
// an edge, 16 M edges, 10.5 and 10.4, with 16, 8 M edges, 5.3 and 6.4; uniform
// with 19, 16.8 M edges, 5.7 and 8.1.
constexpr long long kOrderedMin = 2500000;
constexpr int kOrderedSquares = 40;

int g_sms = 0;

}  // namespace

// Whether the supports of `me` oriented edges between n vertices, `squares` the
// sum of the squared out-degrees, are found through lists in rank order.
bool supports_ordered(long long me, int n, u64 squares) {
  return me >= kOrderedMin && me <= kMaxItems32 && n <= kMaxItems32 && squares >= (u64)kOrderedSquares * (u64)me;
}

int sm_count() {
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 1;
  }
  return g_sms;
}

static int grid_for(long long work, int tpb, int per_sm) {
  const long long want = (work + tpb - 1) / tpb;
  const long long cap = (long long)sm_count() * per_sm;
  return (int)std::max(1LL, std::min(want, cap));
}

#define FSGC_TRY(x)                               \
  do {                                            \
    cudaError_t e__ = (x);                        \
    if (e__ != cudaSuccess) return FSGC_ECUDA;    \
  } while (0)

// Degrees and the maximum degree into caller-provided device memory.
int launch_degrees(int n, const long long* off, int* deg, int* maxdeg, cudaStream_t s) {
  degree_kernel<<<grid_for(n, kTPB, 8), kTPB, 0, s>>>(n, off, deg, maxdeg);
  return cudaGetLastError() == cudaSuccess ? FSGC_OK : FSGC_ECUDA;
}

// Degrees and the maximum degree; run when a graph becomes resident.
int graph_degrees(DevGraph& g, cudaStream_t s, uint64_t* launches, u64* d_u64) {
  int* d_max = reinterpret_cast<int*>(d_u64);
  FSGC_TRY(cudaMemsetAsync(d_max, 0, sizeof(int), s));
  degree_kernel<<<grid_for(g.n, kTPB, 8), kTPB, 0, s>>>(g.n, g.off, g.deg, d_max);
  *launches += 1;
  int maxd = 0;
  FSGC_TRY(cudaMemcpyAsync(&maxd, d_max, sizeof(int), cudaMemcpyDeviceToHost, s));
  FSGC_TRY(cudaStreamSynchronize(s));
  FSGC_TRY(cudaGetLastError());
  g.maxdeg = maxd;
  return FSGC_OK;
}

// Supports through lists in rank order; FSGC_EUNSUPPORTED, with nothing added,
// when there is no room.  32-bit positions (supports_ordered).
static int ordered_supports(DevGraph& g, const GView& v, cudaStream_t s, uint64_t* launches, u64* d_tri) {
  const int n = g.n;
  const int me = (int)(g.m / 2);
  auto bits_for = [](unsigned x) { int b = 1; while (b < 32 && x >> b) b++; return b; };
  unsigned *k1 = nullptr, *k2 = nullptr, *sup = nullptr;
  int *v1 = nullptr, *into = nullptr, *slot = nullptr, *rank_of = nullptr, *start = nullptr;
  SupWork* work = nullptr;
  void* temp = nullptr;
  auto done = [&](int st) {
    for (void* p : {(void*)k1, (void*)k2, (void*)sup, (void*)v1, (void*)into, (void*)slot, (void*)rank_of, (void*)start,
                    (void*)work, temp})
      if (p) cudaFreeAsync(p, s);
    if (st != FSGC_OK) cudaGetLastError();
    return st;
  };
  auto get = [&](void** p, size_t bytes) { return cudaMallocAsync(p, bytes, s) == cudaSuccess; };
  const size_t words = sizeof(int) * (size_t)std::max(me, n);
  const int rank_bits = bits_for((unsigned)n - 1);
  size_t t1 = 0, t2 = 0;
  auto room = [&](size_t& bytes, int items, int bits) {
    return cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const unsigned*)nullptr, (unsigned*)nullptr, (const int*)nullptr,
                                           (int*)nullptr, items, 0, bits, s) == cudaSuccess;
  };
  if (!room(t1, n, 32) || !room(t2, me, rank_bits)) return done(FSGC_EUNSUPPORTED);
  const size_t tb = std::max(t1, t2);
  // a vertex left to the blocks has more than kSupSmall out-edges or kSupPiece in-edges
  const size_t pieces = (size_t)me / (kSupSmall + 1) + 2 * ((size_t)me / kSupPiece) + 2;
  if (!get((void**)&k1, words) || !get((void**)&k2, words) || !get((void**)&v1, words) || !get((void**)&into, words) ||
      !get((void**)&slot, words) || !get((void**)&sup, words) || !get((void**)&rank_of, sizeof(int) * (size_t)n) ||
      !get((void**)&start, sizeof(int) * ((size_t)n + 1)) || !get((void**)&work, sizeof(SupWork) + sizeof(int2) * pieces) ||
      !get(&temp, tb))
    return done(FSGC_EUNSUPPORTED);
  const int vg = grid_for((long long)n + 1, kTPB, 16), eg = grid_for(me, kTPB, 16);
  // every pass indexes with what the sort before it wrote
  auto sort = [&](const int* values, int* out, int items, int bits) {
    size_t tt = tb;
    return cub::DeviceRadixSort::SortPairs(temp, tt, k1, k2, values, out, items, 0, bits, s) == cudaSuccess;
  };
  degree_keys_kernel<<<vg, kTPB, 0, s>>>(v, k1, v1);
  if (!sort(v1, into, n, bits_for((unsigned)g.maxdeg))) return done(FSGC_EUNSUPPORTED);
  rank_scatter_kernel<<<vg, kTPB, 0, s>>>(n, into, rank_of);
  upper_keys_kernel<<<eg, kTPB, 0, s>>>(v, me, rank_of, k1, v1);
  if (!sort(v1, into, me, rank_bits)) return done(FSGC_EUNSUPPORTED);
  into_starts_kernel<<<vg, kTPB, 0, s>>>(n, k2, me, start);
  lower_keys_kernel<<<eg, kTPB, 0, s>>>(v, me, into, k1);
  if (!sort(into, slot, me, rank_bits)) return done(FSGC_EUNSUPPORTED);
  places_kernel<<<eg, kTPB, 0, s>>>(v, me, slot, rank_of, k1, v1);
  cudaMemsetAsync(sup, 0, sizeof(unsigned) * (size_t)me, s);
  cudaMemsetAsync(work, 0, sizeof(SupWork), s);
  const OrderedEdges o{k1, into, v1, start, rank_of, sup};
  // a few vertices a turn where there are many more of them than warps
  const int grab = (int)std::max(1LL, std::min(32LL, n / ((long long)sm_count() * 64 * 32)));
  support_warp_kernel<<<grid_for(n, kSupWarps * grab, 8), kSupWarps * 32, 0, s>>>(v, o, grab, work, d_tri);
  support_block_kernel<<<grid_for((long long)pieces, 1, 8), kSupBlock, 0, s>>>(v, o, work, d_tri);
  supports_back_kernel<<<eg, kTPB, 0, s>>>(me, v1, sup, g.osup);
  *launches += 9;
  return done(FSGC_OK);
}

int prepare_graph(DevGraph& g, cudaStream_t s, uint64_t* launches, u64* d_u64) {
  if (g.prepared) return FSGC_OK;
  const int n = g.n;
  const long long me = g.m / 2;
  const int maxd = g.maxdeg;
  // oriented CSR
  long long* odeg = nullptr;
  const long long ntiles = ((long long)n + kScanTile - 1) / kScanTile;
  long long* tiles = nullptr;
  FSGC_TRY(cudaMallocAsync((void**)&odeg, sizeof(long long) * ((size_t)n + 1), s));
  FSGC_TRY(cudaMallocAsync((void**)&tiles, sizeof(long long) * (size_t)std::max(1LL, ntiles), s));
  FSGC_TRY(cudaMallocAsync((void**)&g.ooff, sizeof(long long) * ((size_t)n + 1), s));
  FSGC_TRY(cudaMallocAsync((void**)&g.oadj, sizeof(int) * (size_t)std::max(1LL, me), s));
  FSGC_TRY(cudaMallocAsync((void**)&g.osrc, sizeof(int) * (size_t)std::max(1LL, me), s));
  FSGC_TRY(cudaMallocAsync((void**)&g.osup, sizeof(unsigned) * (size_t)std::max(1LL, me), s));
  GView v = g.view();
  const int wgrid = grid_for((long long)n * 32, kTPB, 16);
  outdeg_kernel<<<wgrid, kTPB, 0, s>>>(v, odeg);
  scan_tiles_kernel<<<(int)ntiles, kTPB, 0, s>>>(odeg, n, tiles);
  scan_sums_kernel<<<1, 1024, 0, s>>>(tiles, ntiles);
  scan_apply_kernel<<<(int)ntiles, kTPB, 0, s>>>(odeg, n, tiles, g.ooff);
  v = g.view();
  orient_fill_kernel<<<wgrid, kTPB, 0, s>>>(v, g.oadj, g.osrc);
  *launches += 5;
  u64* d_stats = d_u64 + 2;
  // after the first three: the list's fill count, sums of squares of out-degrees and degrees
  FSGC_TRY(cudaMemsetAsync(d_stats, 0, 6 * sizeof(u64), s));
  outdeg_stats_kernel<<<grid_for(n, kTPB, 8), kTPB, 0, s>>>(v, d_stats);
  *launches += 1;
  // supports and triangle total
  FSGC_TRY(cudaMemsetAsync(g.osup, 0, sizeof(unsigned) * (size_t)std::max(1LL, me), s));
  u64* d_tri = d_u64 + 1;
  FSGC_TRY(cudaMemsetAsync(d_tri, 0, sizeof(u64), s));
  bool ordered = false;
  if (me >= kOrderedMin) {
    u64 squares = 0;
    FSGC_TRY(cudaMemcpyAsync(&squares, d_stats + 4, sizeof(u64), cudaMemcpyDeviceToHost, s));
    FSGC_TRY(cudaStreamSynchronize(s));
    ordered = supports_ordered(me, n, squares) && ordered_supports(g, v, s, launches, d_tri) == FSGC_OK;
  }
  if (me > 0 && !ordered) {
    triangle_support_kernel<<<grid_for(me, kTPB, 8), kTPB, 0, s>>>(v, g.osup, d_tri);
    *launches += 1;
  }
  u64 stats[7] = {0};
  FSGC_TRY(cudaMemcpyAsync(stats, d_tri, sizeof(stats), cudaMemcpyDeviceToHost, s));
  FSGC_TRY(cudaFreeAsync(odeg, s));
  FSGC_TRY(cudaFreeAsync(tiles, s));
  FSGC_TRY(cudaStreamSynchronize(s));
  FSGC_TRY(cudaGetLastError());
  g.triangles = (long long)stats[0];
  g.max_outdeg = (long long)stats[1];
  g.max_bitmap_words = (long long)stats[2];
  g.mean_end_degree = g.m > 0 ? (double)stats[6] / (double)g.m : 0;
  if (stats[3] > 0) {
    FSGC_TRY(cudaMallocAsync((void**)&g.wide, sizeof(int) * (size_t)stats[3], s));
    wide_list_kernel<<<grid_for(n, kTPB, 8), kTPB, 0, s>>>(v, g.wide, reinterpret_cast<int*>(d_stats + 3));
    *launches += 1;
    FSGC_TRY(cudaStreamSynchronize(s));
    g.nwide = (int)stats[3];
    g.bytes += sizeof(int) * (size_t)stats[3];
  }
  // the reference relabels (and so orders triangle roles by degree) only for
  // n > 10000, n <= m/10 and maximum degree > 16
  g.tri_relabel = (n > 10000) && !((long long)n > g.m / 10) && (maxd > 16);
  g.bytes += sizeof(long long) * ((size_t)n + 1) + (sizeof(int) * 2 + sizeof(unsigned)) * (size_t)std::max(1LL, me);
  g.prepared = true;
  return FSGC_OK;
}

int ensure_entry_supports(DevGraph& g, cudaStream_t s, uint64_t* launches) {
  if (g.esup) return FSGC_OK;
  FSGC_TRY(cudaMallocAsync((void**)&g.esup, sizeof(unsigned) * (size_t)std::max(1LL, g.m), s));
  FSGC_TRY(cudaMemsetAsync(g.esup, 0, sizeof(unsigned) * (size_t)std::max(1LL, g.m), s));
  const long long me = g.m / 2;
  if (me > 0) {
    entry_support_kernel<<<grid_for(me, kTPB, 8), kTPB, 0, s>>>(g.view(), g.esup);
    *launches += 1;
  }
  g.bytes += sizeof(unsigned) * (size_t)std::max(1LL, g.m);
  FSGC_TRY(cudaGetLastError());
  return FSGC_OK;
}

int ensure_vertex_triangles(DevGraph& g, cudaStream_t s, uint64_t* launches) {
  if (g.vtri2) return FSGC_OK;
  FSGC_TRY(cudaMallocAsync((void**)&g.vtri2, sizeof(u64) * (size_t)std::max(1, g.n), s));
  FSGC_TRY(cudaMemsetAsync(g.vtri2, 0, sizeof(u64) * (size_t)std::max(1, g.n), s));
  const long long me = g.m / 2;
  if (me > 0) {
    vertex_triangle_kernel<<<grid_for(me, kTPB, 8), kTPB, 0, s>>>(g.view(), g.vtri2);
    *launches += 1;
  }
  g.bytes += sizeof(u64) * (size_t)std::max(1, g.n);
  FSGC_TRY(cudaGetLastError());
  return FSGC_OK;
}

}  // namespace fsgc
