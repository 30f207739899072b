// Edge-list ingestion on the device: an arbitrary list of undirected pairs
// becomes the cleaned, symmetric CSR the counting kernels take (self loops
// dropped, duplicates merged, both directions, lists sorted ascending) -- the
// reference's documented input preconditions (src/fringeCount.cu:50-56), which
// its own loader only assumes (src/ECLgraph.h:58-85).  The host-side
// equivalent is fsgc_csr_from_edges.
//
// A pair becomes one key, low id above high id in twice the bits of n - 1, radix
// sorted over those bits alone and made unique.  A vertex's list is its lower
// neighbours, then its higher ones: the higher ones stand in order in the keys,
// the lower ones in the same edges sorted by their high ids, which is stable and
// takes half the bits, so both go straight to their places and nothing is sorted
// in both directions.  Sorting uses CUB's device radix sort (this runs once per
// graph, off the counting path).
// Bound by memory, the sorts' passes: 2^20 vertices and 16.7 M pairs take five
// passes over 8-byte keys and three over 4 + 4 bytes, 8 x 134 MB read and
// written, where full 64-bit keys of both directions took 24 of them.
#include <cub/cub.cuh>

#include "fsgc_internal.h"

namespace fsgc {
namespace {

// key of (a, b): low id << bits | high id; loops and bad pairs take the largest
// key, which is itself the loop of the largest id.  flags: 1 an id is out of
// range, 2 the largest key was given out.
__global__ void edge_keys_kernel(const int* __restrict__ pairs, long long E, int n, int bits,
                                 unsigned long long* __restrict__ keys, int* __restrict__ flags) {
  const unsigned long long loop_key = (1ULL << (2 * bits)) - 1;
  int seen = 0;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (long long)gridDim.x * blockDim.x) {
    const int a = pairs[2 * e], b = pairs[2 * e + 1];
    unsigned long long k = loop_key;
    if (a < 0 || b < 0 || a >= n || b >= n) {
      seen |= 3;
    } else if (a != b) {
      const unsigned long long lo = (unsigned)min(a, b), hi = (unsigned)max(a, b);
      k = (lo << bits) | hi;
    } else {
      seen |= 2;
    }
    keys[e] = k;
  }
  if (seen) atomicOr(flags, seen);
}

__global__ void split_keys_kernel(const unsigned long long* __restrict__ und, long long U, int bits,
                                  unsigned* __restrict__ hi, unsigned* __restrict__ lo) {
  const unsigned long long mask = (1ULL << bits) - 1;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < U; i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = und[i];
    hi[i] = (unsigned)(k & mask);
    lo[i] = (unsigned)(k >> bits);
  }
}

template <class T>
__device__ __forceinline__ long long first_at_least(const T* __restrict__ a, long long len, T x) {
  long long lo = 0, hi = len;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// below[v]: edges whose high id is under v; off[v]: those and the edges whose low id is under v
__global__ void csr_offsets_kernel(const unsigned long long* __restrict__ und, const unsigned* __restrict__ hi, long long U,
                                   int bits, int n, long long* __restrict__ below, long long* __restrict__ off) {
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += (long long)gridDim.x * blockDim.x) {
    const long long b = first_at_least(hi, U, (unsigned)v);
    below[v] = b;
    off[v] = b + first_at_least(und, U, (unsigned long long)v << bits);
  }
}

__global__ void csr_lists_kernel(const unsigned long long* __restrict__ und, const unsigned* __restrict__ hi,
                                 const unsigned* __restrict__ lo, long long U, int bits,
                                 const long long* __restrict__ below, const long long* __restrict__ off,
                                 int* __restrict__ adj) {
  const unsigned long long mask = (1ULL << bits) - 1;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < U; i += (long long)gridDim.x * blockDim.x) {
    const unsigned long long k = und[i];
    adj[below[(k >> bits) + 1] + i] = (int)(k & mask);
    const unsigned h = hi[i];
    adj[off[h] - below[h] + i] = (int)lo[i];
  }
}

int grid_of(long long work) { return (int)std::max(1LL, std::min((work + 255) / 256, (long long)sm_count() * 16)); }

// Grows the sorts' temporary storage.
cudaError_t grow(void*& temp, size_t& temp_bytes, size_t need, cudaStream_t s) {
  if (need <= temp_bytes) return cudaSuccess;
  cudaFreeAsync(temp, s);
  temp = nullptr;
  temp_bytes = 0;
  const cudaError_t e = cudaMallocAsync(&temp, need, s);
  if (e == cudaSuccess) temp_bytes = need;
  return e;
}

}  // namespace

int csr_from_device_edges(int n, long long E, const int* d_pairs, cudaStream_t s, long long** off_out, int** adj_out,
                          long long* m_out, u64* d_small) {
  *off_out = nullptr;
  *adj_out = nullptr;
  *m_out = 0;
  unsigned long long *a = nullptr, *b = nullptr;
  unsigned *hi1 = nullptr, *hi2 = nullptr, *lo1 = nullptr, *lo2 = nullptr;
  long long *off = nullptr, *below = nullptr;
  int* adj = nullptr;
  void* temp = nullptr;
  size_t temp_bytes = 0;
  int* flags = reinterpret_cast<int*>(d_small + 11);
  long long* nsel = reinterpret_cast<long long*>(d_small + 12);
  auto drop = [&] {
    for (void* p : {(void*)a, (void*)b, (void*)hi1, (void*)hi2, (void*)lo1, (void*)lo2, (void*)below, temp})
      cudaFreeAsync(p, s);
    a = b = nullptr;
    hi1 = hi2 = lo1 = lo2 = nullptr;
    below = nullptr;
    temp = nullptr;
  };
  auto fail = [&](int st) {
    drop();
    cudaFreeAsync(off, s);
    cudaFreeAsync(adj, s);
    cudaStreamSynchronize(s);
    cudaGetLastError();
    return st;
  };
  auto fail_e = [&](cudaError_t e) { return fail(e == cudaErrorMemoryAllocation ? FSGC_ENOMEM : FSGC_ECUDA); };
  int bits = 1;
  while (bits < 31 && ((long long)n - 1) >> bits) bits++;
  const size_t kbytes = sizeof(unsigned long long) * (size_t)std::max(1LL, E);
  if (cudaMallocAsync((void**)&a, kbytes, s) != cudaSuccess || cudaMallocAsync((void**)&b, kbytes, s) != cudaSuccess)
    return fail(FSGC_ENOMEM);
  long long U = 0;
  if (E > 0) {
    cudaMemsetAsync(flags, 0, sizeof(int), s);
    edge_keys_kernel<<<grid_of(E), 256, 0, s>>>(d_pairs, E, n, bits, a, flags);
    cub::DoubleBuffer<unsigned long long> db(a, b);
    size_t need = 0;
    cudaError_t e = cub::DeviceRadixSort::SortKeys(nullptr, need, db, E, 0, 2 * bits, s);
    if (e == cudaSuccess) e = grow(temp, temp_bytes, need, s);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortKeys(temp, need, db, E, 0, 2 * bits, s);
    if (e != cudaSuccess) return fail_e(e);
    a = db.Current();
    b = db.Alternate();
    need = 0;
    e = cub::DeviceSelect::Unique(nullptr, need, a, b, nsel, E, s);
    if (e == cudaSuccess) e = grow(temp, temp_bytes, need, s);
    if (e == cudaSuccess) e = cub::DeviceSelect::Unique(temp, need, a, b, nsel, E, s);
    if (e != cudaSuccess) return fail_e(e);
    int h_flags = 0;
    cudaMemcpyAsync(&U, nsel, sizeof(long long), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&h_flags, flags, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (cudaStreamSynchronize(s) != cudaSuccess) return fail(FSGC_ECUDA);
    if (h_flags & 1) return fail(FSGC_EINVAL);
    if (h_flags & 2) U--;  // the loops' key, the last
    std::swap(a, b);  // a: the unique undirected keys
  }
  cudaFreeAsync(b, s);
  b = nullptr;
  const size_t wbytes = sizeof(unsigned) * (size_t)std::max(1LL, U);
  for (unsigned** w : {&hi1, &hi2, &lo1, &lo2})
    if (cudaMallocAsync((void**)w, wbytes, s) != cudaSuccess) return fail(FSGC_ENOMEM);
  // the lists are padded by 16 bytes, as every resident graph's
  if (cudaMallocAsync((void**)&below, sizeof(long long) * ((size_t)n + 1), s) != cudaSuccess ||
      cudaMallocAsync((void**)&off, sizeof(long long) * ((size_t)n + 1), s) != cudaSuccess ||
      cudaMallocAsync((void**)&adj, sizeof(int) * (size_t)std::max(1LL, 2 * U) + 16, s) != cudaSuccess)
    return fail(FSGC_ENOMEM);
  if (U > 0) {
    split_keys_kernel<<<grid_of(U), 256, 0, s>>>(a, U, bits, hi1, lo1);
    cub::DoubleBuffer<unsigned> dk(hi1, hi2), dv(lo1, lo2);
    size_t need = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, need, dk, dv, U, 0, bits, s);
    if (e == cudaSuccess) e = grow(temp, temp_bytes, need, s);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(temp, need, dk, dv, U, 0, bits, s);
    if (e != cudaSuccess) return fail_e(e);
    hi1 = dk.Current();
    hi2 = dk.Alternate();
    lo1 = dv.Current();
    lo2 = dv.Alternate();
  }
  csr_offsets_kernel<<<grid_of((long long)n + 1), 256, 0, s>>>(a, hi1, U, bits, n, below, off);
  if (U > 0) csr_lists_kernel<<<grid_of(U), 256, 0, s>>>(a, hi1, lo1, U, bits, below, off, adj);
  drop();
  if (cudaStreamSynchronize(s) != cudaSuccess || cudaGetLastError() != cudaSuccess) return fail(FSGC_ECUDA);
  *off_out = off;
  *adj_out = adj;
  *m_out = 2 * U;
  return FSGC_OK;
}

}  // namespace fsgc
