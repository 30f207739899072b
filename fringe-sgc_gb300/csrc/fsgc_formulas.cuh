// Per-match formulas of the counting kernels, shared by the counting
// translation units.  Each unit that includes this file has its own copy of
// the division table and fills it with upload_div_table().
#pragma once
#include "fsgc_internal.h"

namespace fsgc {
namespace {

__constant__ DivMagic c_div[kMaxDiv];

inline void upload_div_table() {
  DivMagic t[kMaxDiv];
  t[0] = DivMagic{0, 1};
  t[1] = DivMagic{0, 1};
  for (int d = 2; d < kMaxDiv; d++) t[d] = make_div_magic((unsigned)d);
  cudaMemcpyToSymbol(c_div, t, sizeof(t));
}

constexpr int kTPB = 256;
enum { IU = 1, IV = 2, IW = 4, IUV = 3, IUW = 5, IVW = 6, IUVW = 7 };

// Most fringe counts are 0, 1 or 2: closed forms there, without nck_ref's
// min(k, n - k), which would send the lanes of a warp different ways.  Equal to
// nck_ref for every n: n (n - 1) stays below 2^62.
__device__ __forceinline__ u64 nck(int n, int k) {
  if (k <= 2) {
    if (n < k || k < 0) return 0;
    return k == 0 ? 1ULL : k == 1 ? (u64)n : ((u64)n * (u64)(n - 1)) >> 1;
  }
  return nck_ref(n, k, c_div);
}

// Arithmetic of a count: u64 with the reference's wrapping binomials (A = u64),
// or exact saturating 128-bit values (A = X128).
template <class A> __device__ __forceinline__ A nck_a(int n, int k);
template <> __device__ __forceinline__ u64 nck_a<u64>(int n, int k) { return nck(n, k); }
template <> __device__ __forceinline__ X128 nck_a<X128>(int n, int k) { return nck_x(n, k); }
__device__ __forceinline__ bool a_is_zero(u64 x) { return x == 0; }
__device__ __forceinline__ bool a_is_zero(const X128& x) { return x.is_zero(); }

// Adds one match's value: into the thread's running sum for an ordinary graph,
// into the result slot of the match's member graph for a packed graph.
__device__ __forceinline__ void credit(const GView& g, u64& acc, u64 x, int vertex) {
  if (g.comp == nullptr) acc += x;
  else if (x) atomicAdd(g.comp_slots + g.comp[vertex], x);
}
// exact counts run on ordinary graphs only
__device__ __forceinline__ void credit(const GView&, X128& acc, X128 x, int) { acc += x; }
__device__ __forceinline__ int relabel_of(const GView& g, int relabel, int vertex) {
  return g.comp ? (int)g.comp_relabel[g.comp[vertex]] : relabel;
}

// ------------------------------------------------------------- shared formulas
// Edge-core formula (src/fringeCount.cu:2030-2049) for an edge (u, v), where
// u is the endpoint with the larger vertex id and c_uv = |N(u) & N(v)|.
template <class A>
__device__ A edge_formula(int du, int dv, int c_uv, int f_u, int f_uv, int f_v) {
  const int a_uv = c_uv - f_uv;
  if (a_uv < 0) return 0;
  const int c_u = du - 1 - c_uv, c_v = dv - 1 - c_uv;
  const int bound = min(f_u, a_uv);
  A acc = 0;
  for (int j = 0; j <= bound; j++) {
    const int k = f_u - j;
    A term = nck_a<A>(c_u, k) * nck_a<A>(a_uv + c_v - j, f_v);
    if (f_u != f_v) term += nck_a<A>(c_v, k) * nck_a<A>(a_uv + c_u - j, f_v);
    acc += term * nck_a<A>(a_uv, j);
  }
  return acc * nck_a<A>(c_uv, f_uv);
}

// Binomials for wedge_formula_with: the count's arithmetic in general, and
// the two-case form when every k is 0 or 1 (nck01, equal for those k).
template <class A>
struct NckA {
  __device__ A operator()(int n, int k) const { return nck_a<A>(n, k); }
};
template <class A>
struct Nck01 {
  __device__ A operator()(int n, int k) const { return A(nck01(n, k)); }
};

// wedge() (src/fringeCount.cu:1381-1406) for endpoints x (larger id) and y.
template <class A>
__device__ __forceinline__ A wedge_formula(int dx, int dy, bool adj, int f_x, int f_xy, int f_y, int c) {
  if ((unsigned)(f_x | f_xy | f_y) <= 1u) return wedge_formula_with<A>(dx, dy, adj, f_x, f_xy, f_y, c, Nck01<A>());
  return wedge_formula_with<A>(dx, dy, adj, f_x, f_xy, f_y, c, NckA<A>());
}

// fc3 (src/fringeCount.cu:233-327): placements of the seven anchor-set types of
// a 3-vertex core into its seven exclusive Venn regions.  Same summation
// indices and the same nck factors per term as the reference.
template <class A>
__device__ A fc3(const int* fr, const int* venn) {
  const int fuvw = fr[IUVW], fuv = fr[IUV], fuw = fr[IUW], fvw = fr[IVW];
  const int fu = fr[IU], fv = fr[IV], fw = fr[IW];
  int x_uvw = venn[IUVW];
  const int x_uv = venn[IUV], x_uw = venn[IUW], x_vw = venn[IVW];
  const int x_u = venn[IU], x_v = venn[IV], x_w = venn[IW];
  if (x_uvw < fuvw) return 0;
  const A base = nck_a<A>(x_uvw, fuvw);
  x_uvw -= fuvw;
  A total = 0;
  for (int i = min(x_uvw, fuv); i >= 0; i--) {
    if (x_uv < fuv - i) break;
    const A t1 = base * nck_a<A>(x_uvw, i) * nck_a<A>(x_uv, fuv - i);
    const int r1 = x_uvw - i, r_uv = x_uv - (fuv - i);
    for (int j = min(r1, fuw); j >= 0; j--) {
      if (x_uw < fuw - j) break;
      const A t2 = t1 * nck_a<A>(r1, j) * nck_a<A>(x_uw, fuw - j);
      const int r2 = r1 - j, r_uw = x_uw - (fuw - j);
      for (int k = min(r2, fvw); k >= 0; k--) {
        if (x_vw < fvw - k) break;
        const A t3 = t2 * nck_a<A>(r2, k) * nck_a<A>(x_vw, fvw - k);
        const int r3 = r2 - k, r_vw = x_vw - (fvw - k);
        for (int a = min(r3, fu); a >= 0; a--) {
          const A ta = t3 * nck_a<A>(r3, a);
          const int pool_v = (r3 - a) + r_vw;
          for (int b = min(r_uv, fu - a); b >= 0; b--) {
            const A tb = ta * nck_a<A>(r_uv, b);
            const int r_uv2 = r_uv - b;
            for (int c = min(r_uw, fu - a - b); c >= 0; c--) {
              if (x_u < fu - a - b - c) break;
              const A tc = tb * nck_a<A>(r_uw, c) * nck_a<A>(x_u, fu - a - b - c);
              const int r_uw2 = r_uw - c;
              for (int d = min(pool_v, fv); d >= 0; d--) {
                if (r_uv2 + x_v < fv - d) break;
                const A td = tc * nck_a<A>(pool_v, d) * nck_a<A>(r_uv2 + x_v, fv - d);
                const int pool_w = (pool_v - d) + r_uw2 + x_w;
                if (pool_w >= fw) total += td * nck_a<A>(pool_w, fw);
              }
            }
          }
        }
      }
    }
  }
  return total;
}

// ---- fc3 in a ring: the same number of placements with fewer terms.
// Disjoint choices of fa out of A and fb out of B, |A & B| = both.
__device__ __forceinline__ u64 choose_two(int fa, int fb, int na, int nb, int both) {
  if (fa > fb) {
    int t = fa; fa = fb; fb = t;
    t = na; na = nb; nb = t;
  }
  if (fa == 0) return nck(nb, fb);
  if (fa == 1) {
    if (fb == 1) return (u64)(unsigned)na * (u64)(unsigned)nb - (u64)(unsigned)both;
    return (u64)(unsigned)both * nck(nb - 1, fb) + (u64)(unsigned)(na - both) * nck(nb, fb);
  }
  u64 sum = 0;
  for (int t = 0; t <= fa; t++) sum += nck(both, t) * nck(na - both, fa - t) * nck(nb - t, fb);
  return sum;
}

// Disjoint choices of fu, fv, fw (each at least 1, not all 1) out of U, V, W by
// their exclusive regions: one vertex's fringes, the fewest, are split over its
// regions.
__device__ __forceinline__ u64 choose_three_split(int fu, int fv, int fw, int r, int uv, int uw, int vw, int xu, int xv, int xw) {
  if (fv < fu && fv <= fw) {
    int t = fu; fu = fv; fv = t;
    t = uw; uw = vw; vw = t;
    t = xu; xu = xv; xv = t;
  } else if (fw < fu) {
    int t = fu; fu = fw; fw = t;
    t = uv; uv = vw; vw = t;
    t = xu; xu = xw; xw = t;
  }
  const int nv = r + uv + vw + xv, nw = r + uw + vw + xw, i_vw = r + vw;
  u64 sum = 0;
  for (int a = 0; a <= fu; a++) {
    const u64 ta = nck(r, a);
    if (ta == 0) break;
    for (int b = 0; a + b <= fu; b++) {
      const u64 tb = ta * nck(uv, b);
      for (int c = 0; a + b + c <= fu; c++) {
        const u64 tc = tb * nck(uw, c) * nck(xu, fu - a - b - c);
        if (tc) sum += tc * choose_two(fv, fw, nv - a - b, nw - a - c, i_vw - a);
      }
    }
  }
  return sum;
}

// Disjoint choices of fu, fv, fw out of U, V, W.
__device__ __forceinline__ u64 choose_three(int fu, int fv, int fw, int r, int uv, int uw, int vw, int xu, int xv, int xw) {
  const int nu = r + uv + uw + xu, nv = r + uv + vw + xv, nw = r + uw + vw + xw;
  if (fu == 0 || fv == 0 || fw == 0) {  // at most two vertices have fringes of their own
    int fa = fu, fb = fv, na = nu, nb = nv, both = r + uv;
    if (fu == 0) { fa = fw; na = nw; both = r + vw; }
    else if (fv == 0) { fb = fw; nb = nw; both = r + uw; }
    return choose_two(fa, fb, na, nb, both);
  }
  if (fu + fv + fw == 3) {  // one each: inclusion-exclusion over coinciding choices
    const u64 a = (u64)(unsigned)nu, b = (u64)(unsigned)nv, c = (u64)(unsigned)nw;
    return a * b * c - a * (u64)(unsigned)(r + vw) - b * (u64)(unsigned)(r + uw) - c * (u64)(unsigned)(r + uv) +
           2ULL * (u64)(unsigned)r;
  }
  return choose_three_split(fu, fv, fw, r, uv, uw, vw, xu, xv, xw);
}

// Equal to fc3<u64> while no binomial of the graph's degrees wraps before its
// division (the sums regrouped are then equal mod 2^64).
__device__ __forceinline__ u64 fc3_ring(const int* fr, int r, int uv, int uw, int vw, int xu, int xv, int xw) {
  const int fuvw = fr[IUVW], fuv = fr[IUV], fuw = fr[IUW], fvw = fr[IVW];
  if (r < fuvw) return 0;
  const u64 base = nck(r, fuvw);
  r -= fuvw;
  if ((fuv | fuw | fvw) == 0) return base * choose_three(fr[IU], fr[IV], fr[IW], r, uv, uw, vw, xu, xv, xw);
  u64 sum = 0;
  for (int i = 0; i <= fuv; i++) {
    const u64 ti = nck(r, i) * nck(uv, fuv - i);
    if (ti == 0) continue;
    for (int j = 0; j <= fuw; j++) {
      const u64 tj = ti * nck(r - i, j) * nck(uw, fuw - j);
      if (tj == 0) continue;
      for (int k = 0; k <= fvw; k++) {
        const u64 tk = tj * nck(r - i - j, k) * nck(vw, fvw - k);
        if (tk)
          sum += tk * choose_three(fr[IU], fr[IV], fr[IW], r - i - j - k, uv - (fuv - i), uw - (fuw - j), vw - (fvw - k),
                                   xu, xv, xw);
      }
    }
  }
  return base * sum;
}

}  // namespace
}  // namespace fsgc
