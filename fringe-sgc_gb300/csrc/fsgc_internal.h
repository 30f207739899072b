// Internal types shared by the library's translation units.
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "fsgc.h"
#include "fsgc_device.cuh"

namespace fsgc {

// Graph resident in HBM.  Full CSR (int64 offsets, int32 sorted lists) plus the
// loader's derived structures:
//  - degree order:  x < y  iff  (deg x, x) < (deg y, y); every undirected edge
//    is stored once, from its lower to its higher endpoint ("oriented" CSR);
//  - osrc: the lower endpoint of each oriented slot (edge-parallel kernels);
//  - osup: per oriented slot, |N(x) & N(y)| (triangles through the edge);
//  - vtri2: per vertex, twice its triangle count (lazily).
struct GView {
  int n;
  long long m;                       // directed entries
  const long long* __restrict__ off;  // n+1
  const int* __restrict__ adj;        // m
  const int* __restrict__ deg;        // n
  const long long* __restrict__ ooff; // n+1
  const int* __restrict__ oadj;       // m/2
  const int* __restrict__ osrc;       // m/2
  const unsigned* __restrict__ osup;  // m/2
  // packed graphs (many member graphs in one CSR): member of each vertex,
  // the triangle-core relabel gate of each member, and one result slot per
  // member that kernels add each match into; comp == nullptr for one graph
  const int* __restrict__ comp;
  const unsigned char* __restrict__ comp_relabel;
  u64* comp_slots;
};

struct DevGraph {
  int n = 0;
  long long m = 0;
  long long* off = nullptr;
  int* adj = nullptr;
  int* deg = nullptr;
  int maxdeg = 0;
  // orientation + supports (built by prepare_graph)
  bool prepared = false;
  long long* ooff = nullptr;
  int* oadj = nullptr;
  int* osrc = nullptr;
  unsigned* osup = nullptr;
  long long triangles = -1;
  long long max_outdeg = 0;        // largest oriented out-degree
  int* wide = nullptr;             // vertices whose triangles take a wide block each (triangle_wide)
  int nwide = 0;
  long long max_bitmap_words = 0;  // max over v of outdeg(v) * ceil(deg(v) / 32)
  double mean_end_degree = 0;      // over the list entries: mean degree of their vertices
  u64* vtri2 = nullptr;  // lazily
  unsigned* esup = nullptr;  // lazily: per list entry (u, v), |N(u) & N(v)|
  // wedge core: offsets of chunk boundaries in the lists of high-degree vertices (lazily)
  int* ctab_id = nullptr;
  int* ctab_rows = nullptr;
  int* ctab_pos = nullptr;
  int ctab_K = 0;
  // wedge core: copy of the graph in rank order (lazily; wedge_rank.cu)
  int* roff = nullptr;
  int* radj = nullptr;
  unsigned short* radj16 = nullptr;  // the lists' low 16 bits
  int* rdeg = nullptr;
  int* oid = nullptr;   // id of each rank
  int* rrev = nullptr;  // per list entry (v, u): entries of N(u) up to v
  int* rtab = nullptr;  // boundary table of the first rrows lists, rK columns
  int rrows = 0, rK = 0;
  size_t rank_bytes = 0;     // of the copy (0: there is none)
  bool rank_failed = false;  // no room for the copy: not tried again before room_again()
  unsigned* bits = nullptr;  // lazily: adjacency bit matrix of a small graph (general cores)
  bool bits_failed = false;  // no room for it, likewise
  size_t room_from = 0;      // free device bytes at which what failed is tried again
  bool lean = false;  // neither of the two is built: counts take the paths without them
  // the reference's degree-relabel gate for the triangle core
  // (src/fringeCount.cu:1237, 1342-1344): vertex roles follow (deg, id) order
  // when it fires, vertex ids otherwise
  bool tri_relabel = false;
  size_t bytes = 0;
  // packed graphs
  int ngraphs = 0;                 // 0 for an ordinary graph
  int* comp = nullptr;             // member of each vertex (device)
  unsigned char* comp_relabel = nullptr;  // per member (device)
  std::vector<int> member_n;       // per member: vertices, directed entries
  std::vector<long long> member_m;

  GView view() const {
    GView g;
    g.n = n; g.m = m; g.off = off; g.adj = adj; g.deg = deg;
    g.ooff = ooff; g.oadj = oadj; g.osrc = osrc; g.osup = osup;
    g.comp = comp; g.comp_relabel = comp_relabel; g.comp_slots = nullptr;
    return g;
  }
};

// Device scratch arena owned by a context; grows on demand, never shrinks.
struct Scratch {
  void* ptr = nullptr;
  size_t bytes = 0;
  int layout_n = -1, layout_rows = -1;
  uint64_t gen = 0;  // bumped whenever ptr changes (captured launch sequences hold the pointer)
};

// Per-context device work areas: a few u64 counters/queues (kernel work
// queues, loader results) and a growable scratch arena (triangle-core bitmaps,
// wedge-core hub cursors).
struct DevWork {
  u64* small = nullptr;  // 32 u64; small[kErrWord] collects kernel error bits
  Scratch tri;
  u64* h_err = nullptr;  // pinned host copy of small[kErrWord], refreshed after kernels that can set it
  fsgc_tuning tune = {2048, 16, 8192, 96, 8};
};
constexpr int kErrWord = 10;
// Items that a kernel may walk with 32-bit indices: a grid-stride step (at most 16
// blocks of 256 on each of up to 1,024 SMs) or a piece beyond the last one still
// fits an int.
constexpr int kMaxItems32 = 0x7fffffff - (1 << 22);
// Wedge pairs in rank order from this many list entries: RMAT with 21,000 entries
// counts in 0.11 ms either way, with 45,000 in 0.09 instead of 0.16 ms; below,
// the copy only costs (pattern graphs, counted in themselves, stay there too).
constexpr long long kWedgeRankMin = 20000;

// FSGC_ETIMEDOUT when a kernel of this work area gave up a bounded wait since
// the last call (its count is void), FSGC_OK otherwise; clears the bits.
// Call after the stream has been synchronised.
int take_kernel_error(DevWork& w, cudaStream_t s);

struct Launcher;  // forward

// Structural checks of a matching order shared by every entry point (api.cu).
bool matching_order_valid(const fsgc_matching_order& mo);

// Entry points implemented in prep.cu / count.cu.
int graph_degrees(DevGraph& g, cudaStream_t s, uint64_t* launches, u64* d_scratch_u64);
int prepare_graph(DevGraph& g, cudaStream_t s, uint64_t* launches, u64* d_scratch_u64);
bool supports_ordered(long long me, int n, u64 squares);  // prep.cu: the rule
int ensure_vertex_triangles(DevGraph& g, cudaStream_t s, uint64_t* launches);
int ensure_entry_supports(DevGraph& g, cudaStream_t s, uint64_t* launches);
void upload_div_magic();
void upload_div_magic_wedge();
void upload_div_magic_triangle();
int sm_count();

struct CountJob {
  const fsgc_matching_order* mo;
  DevGraph* g;
  u64* d_slot;        // result slot (zeroed by the caller)
  int core_type;      // out
  u64 host_value;     // used when the result needs no device work (n, m/2, T)
  bool host_only;
  int exact_placements;  // general core: exact placement sum instead of the reference's
  u64* d_comp_slots;     // packed graphs: per-member result slots (zeroed by the caller)
  int per_member_div;    // packed graphs: divide each member's total by this on the host (1 = none)
  bool exact_count = false;  // exact 128-bit sums: d_slot holds (lo, hi, saturated); ordinary graphs only
};

// Fringe counts of a 3-vertex core's anchor sets, one row per rotation.
struct Rot3 {
  int fr[6][8];
  int count;
};

// Whether no C(n, i), n <= maxdeg, i <= k, wraps in u64 before its division:
// C(n, i) i <= n^i / (i-1)! < 2^63.  Sums of products of them may then be
// regrouped mod 2^64.
bool binomials_fit(int maxdeg, int k);

// Triangle core (triangle.cu).
struct TrianglePattern {
  int sum1, sum2, sum3;  // pruning thresholds
  int mode;              // 0 general, 1 4-clique, 2 tailed 4-clique
  int tails;
  int relabel;           // roles by (deg, id) order (1) or by id (0)
  Rot3 rot;
};
// Vertices with `k` out-neighbours and rows over `lists` positions that need the
// larger blocks: more row words or a larger table than a narrow block holds, or
// more lists than its four warps should read.
constexpr int kTriNarrowK = 256, kTriNarrowRows = 6400, kTriNarrowLists = 4096;
__host__ __device__ inline bool triangle_wide(int k, int lists) {
  return k > kTriNarrowK || lists > kTriNarrowLists || (long long)k * (((lists + 31) >> 5) | 1) > kTriNarrowRows;
}
bool triangle_by_tables(const DevGraph& G, bool clique);  // out-degrees for which that path is taken
size_t triangle_scratch(const DevGraph& G);  // work-arena bytes of its modes other than the 4-cliques
int enqueue_triangle(DevGraph& G, const GView& gv, const TrianglePattern& tp, bool exact, u64* slot, cudaStream_t s,
                     uint64_t* launches, DevWork& work);
// Grows a work arena, stream-ordered.
int ensure_plain_scratch(Scratch& sc, size_t need, cudaStream_t s);

// Wedge core with a fringe-free centre: fringes of the larger-id endpoint, of
// both and of the other, and the endpoint degrees below which it counts nothing.
struct WedgeParams {
  int f_v, f_vw, f_w;
  int lim, minsum;  // min(min_v, min_w) and min_v + min_w
};
constexpr int kWedgeFuse = 4;  // patterns counted in one pass

// The rank-order path (wedge_rank.cu).  Graphs it takes: 32-bit list offsets,
// and enough entries that a copy in rank order pays.
inline bool wedge_rank_size_ok(const DevGraph& G) {
  return G.m >= kWedgeRankMin && G.m <= (1LL << 30) && G.n <= (1 << 30);
}
// FSGC_EUNSUPPORTED when the graph does not take this path or has no room for
// the copy, or (exact) the total is not bounded below 2^128: nothing is
// enqueued then and the caller counts another way.
int ensure_rank_order(DevGraph& G, cudaStream_t s, uint64_t* launches, DevWork& work);
void free_rank_order(DevGraph& G);  // no work that reads it in flight
// What a pattern's residual takes there: nothing of its own (none, or the pass over
// the 4-cycles), a pass with sums per owner, or one that evaluates wedge() per pair.
enum WedgePass { kNoPass = 0, kSumsPass = 1, kPairsPass = 2 };
WedgePass wedge_pass(const DevGraph& G, const WedgeParams& p, bool exact);
// Whether `count` patterns of the last kind on an ordinary graph are better counted by
// chunks, in one pass, and whether those with sums then join them.
bool pairs_by_chunks(const DevGraph& G, int count, bool exact);
bool sums_join_pairs(const DevGraph& G);
int enqueue_wedge_rank(DevGraph& G, const GView& gv, const WedgeParams* pats, u64* const* slots, int np, bool exact,
                       cudaStream_t s, uint64_t* launches, DevWork& work);
size_t wedge_rank_scratch(const DevGraph& G);  // work-arena bytes (cursors of hub owners)

// Launchers over caller-provided device memory (used by noalloc.cu).
int launch_degrees(int n, const long long* off, int* deg, int* maxdeg, cudaStream_t s);
int launch_wedge_small(const GView& gv, int f_v, int f_vw, int f_w, int lim, int minsum, int* queue, u64* slot,
                       cudaStream_t s);
int launch_wedge_big(const GView& gv, int f_v, int f_vw, int f_w, int lim, int minsum, int* queue, long long* gcur,
                     int* gpre, long long gstride, int blocks, u64* slot, cudaStream_t s);
int wedge_small_max_degree();

// Enqueue the kernels that add the raw total of `mo` on `g` into *d_slot.
int enqueue_count(CountJob& job, cudaStream_t s, uint64_t* launches, DevWork& work);
// Many jobs on one ordinary graph (u64 counts): patterns whose kernels share
// their match enumeration are counted in shared passes (count.cu).
int enqueue_count_set(std::vector<CountJob*>& jobs, cudaStream_t s, uint64_t* launches, DevWork& work);
// Builds, on `s` and synchronously, every per-graph structure a count of `mo`
// would otherwise build on first use, so that counts enqueued afterwards on
// other streams only read the graph.
int prepare_for_count(const fsgc_matching_order& mo, DevGraph& g, cudaStream_t s, uint64_t* launches,
                      DevWork& work);
// Edge list (device pairs) -> cleaned CSR on the device (ingest.cu).  The
// arrays are the caller's to keep (stream-ordered allocations); the list
// array is padded by 16 bytes.  FSGC_EINVAL for an id outside [0, n).
int csr_from_device_edges(int n, long long E, const int* d_pairs, cudaStream_t s, long long** off_out, int** adj_out,
                          long long* m_out, u64* d_small);
// Builds every per-graph structure any count could need, synchronously.
int prepare_all(DevGraph& g, cudaStream_t s, uint64_t* launches, DevWork& work);
// What DevGraph::lean leaves out: its bytes, and freeing it (nothing that reads it
// is in flight).
size_t fast_structure_bytes(const DevGraph& g);
void free_fast_structures(DevGraph& g);
// Notes that a structure which takes `need` bytes to build found no room.
void note_no_room(DevGraph& g, size_t need);
// Whether structures that found no room may be tried again, which the caller then
// lets happen on the context's stream; false as long as no more is free than then.
bool room_again(DevGraph& g);
// Scratch-arena bytes a count of `mo` on the prepared graph `g` grows to.
size_t count_scratch_bytes(const fsgc_matching_order& mo, const DevGraph& g, const fsgc_tuning& t);
// FSGC_EINVAL unless every field of `t` is in its documented range.
int check_tuning(const fsgc_tuning& t);

}  // namespace fsgc
