// sort.cu -- device scans and stable LSD radix sort used by the scene builder
// (Morton-ordered LBVH leaves, half-edge grouping for the edge list).
#include <algorithm>

#include "psdr_internal.h"

namespace psdr {

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;  // elements per thread per block
constexpr int kScanBlock = kScanThreads * kScanPer;

template <class T>
__device__ T block_exclusive_scan(T v, T* smem_warp, T& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem_warp[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    T w = lane < nw ? smem_warp[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) smem_warp[lane] = w;
  }
  __syncthreads();
  T base = wid > 0 ? smem_warp[wid - 1] : T(0);
  total = smem_warp[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

// Inputs of the scans: an array; the first of each run of equal sorted keys; floats widened
// to double, zero past a device-side count.
struct FirstOfRun {
  const uint64_t* k64;
  const uint32_t* k32;
  __device__ int operator()(int i) const {
    if (i == 0) return 1;
    return k32 ? k32[i] != k32[i - 1] : k64[i] != k64[i - 1];
  }
};
struct PrefixOf {
  const float* v;
  const int* n;  // entries (device); zero beyond
  __device__ double operator()(int i) const { return i < *n ? (double)v[i] : 0.0; }
};
template <class T>
struct Plain {
  const T* v;
  __device__ T operator()(int i) const { return v[i]; }
};

template <class T, class In>
__global__ void k_reduce(In in, int n, T* __restrict__ sums) {
  __shared__ T sw[32];
  const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
  T acc = T(0);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k)
    if (base + k < n) acc += in(base + k);
  T tot;
  block_exclusive_scan<T>(acc, sw, tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Single block: exclusive scan of `n` block sums in place (n <= kScanBlock * 64).
template <class T>
__global__ void k_scan_sums(T* data, int n) {
  __shared__ T sw[32];
  T carry = T(0);
  for (int start = 0; start < n; start += kScanBlock) {
    const int base = start + threadIdx.x * kScanPer;
    T loc[kScanPer];
    T acc = T(0);
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      loc[k] = base + k < n ? data[base + k] : T(0);
      acc += loc[k];
    }
    T tot;
    T ex = block_exclusive_scan<T>(acc, sw, tot);
    T run = carry + ex;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
      if (base + k < n) data[base + k] = run;
      run += loc[k];
    }
    carry += tot;
    __syncthreads();
  }
}

template <class T, bool INCL, class In>
__global__ void k_scan_apply(In in, T* __restrict__ out, int n, const T* __restrict__ offs) {
  __shared__ T sw[32];
  const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanPer;
  T loc[kScanPer];
  T acc = T(0);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    loc[k] = base + k < n ? in(base + k) : T(0);
    acc += loc[k];
  }
  T tot;
  T run = offs[blockIdx.x] + block_exclusive_scan<T>(acc, sw, tot);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (INCL) run += loc[k];
    if (base + k < n) out[base + k] = run;
    if (!INCL) run += loc[k];
  }
}

template <class T, bool INCL, class In>
void scan_impl(In in, T* out, int n, T* tmp, cudaStream_t st) {
  if (n <= 0) return;
  const int nb = (n + kScanBlock - 1) / kScanBlock;
  k_reduce<T, In><<<nb, kScanThreads, 0, st>>>(in, n, tmp);
  k_scan_sums<T><<<1, kScanThreads, 0, st>>>(tmp, nb);
  k_scan_apply<T, INCL, In><<<nb, kScanThreads, 0, st>>>(in, out, n, tmp);
  PSDR_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------- radix sort
// Stable LSD sort over 8-bit digits. One kernel counts the digits of every pass; each pass
// is then a single kernel: a tile ranks its keys, publishes its digit counts and adds up its
// predecessors' (decoupled look-back, Merrill and Garland 2016), so a pass reads and writes the
// pairs once and needs no scan kernels between. The sorts of a scene of a few thousand
// triangles are bound by their launches, not by bytes: 2 + passes launches instead of 5 per
// pass. Building a scene of 1,284 triangles: the two sorts took 10 passes and 50 launches,
// now 7 passes (the half-edge keys are packed) and 11 launches.
constexpr int kSortThreads = 256;
constexpr int kSortItems = 8;                           // keys per thread
constexpr int kSortTile = kSortThreads * kSortItems;    // 2048
constexpr int kSortMaxPasses = 8;
constexpr unsigned kSortCount = (1u << 30) - 1;         // tile status: 2 flag bits, 30-bit count
constexpr unsigned kSortTileOnly = 1u << 30, kSortPrefix = 2u << 30;
// Look-back polls before a tile counts a predecessor's keys itself (tiles start in the order
// of their tickets and publish before they wait, so this is not expected to happen).
constexpr int kSortPolls = 1 << 16;

template <class K>
__global__ void k_sort_counts(const K* __restrict__ keys, int n, int passes, int* __restrict__ counts) {
  __shared__ int h[kSortMaxPasses * 256];
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) h[i] = 0;
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const K k = keys[i];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p * 256 + (int)((k >> (8 * p)) & 255u)], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
    if (h[i]) atomicAdd(&counts[i], h[i]);
}

template <class K>
__global__ void __launch_bounds__(kSortThreads) k_sort_pass(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                            K* __restrict__ kout, uint32_t* __restrict__ vout, int n,
                                                            int shift, const int* __restrict__ counts,
                                                            int* __restrict__ ticket, unsigned* __restrict__ status) {
  constexpr int kWarps = kSortThreads / 32;
  __shared__ int wcnt[kWarps][256];
  __shared__ int offs[256];
  __shared__ int warp_sum[kWarps];
  __shared__ int tile_sh;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (tid == 0) tile_sh = atomicAdd(ticket, 1);
  for (int w = 0; w < kWarps; ++w) wcnt[w][tid] = 0;
  __syncthreads();
  const int tile = tile_sh;
  const int base = tile * kSortTile + wid * (32 * kSortItems) + lane;
  K key[kSortItems];
  int rank[kSortItems];
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) key[j] = base + 32 * j < n ? kin[base + 32 * j] : K(0);
  // ranks among the warp's equal digits, in order
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const bool ok = base + 32 * j < n;
    const int dig = ok ? (int)((key[j] >> shift) & 255u) : 256;
    const unsigned peers = __match_any_sync(0xffffffffu, dig);
    const int leader = __ffs(peers) - 1;
    int before = 0;
    if (ok && lane == leader) {
      before = wcnt[wid][dig];
      wcnt[wid][dig] = before + __popc(peers);
    }
    rank[j] = __shfl_sync(0xffffffffu, before, leader) + __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
  }
  __syncthreads();
  // digit `tid`: exclusive counts over the warps, the tile's total, then the tiles before
  int total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int c = wcnt[w][tid];
    wcnt[w][tid] = total;
    total += c;
  }
  volatile unsigned* st = status;
  st[(size_t)tile * 256 + tid] = (tile == 0 ? kSortPrefix : kSortTileOnly) | (unsigned)total;
  int before = 0;
  for (int t = tile - 1; t >= 0; --t) {
    unsigned s = 0;
    for (int k = 0; k < kSortPolls && !(s >> 30); ++k) s = st[(size_t)t * 256 + tid];
    if (!(s >> 30)) {
      const int hi = min(n, (t + 1) * kSortTile);
      for (int i = t * kSortTile; i < hi; ++i) before += (int)((kin[i] >> shift) & 255u) == tid;
      continue;
    }
    before += (int)(s & kSortCount);
    if (s & kSortPrefix) break;
  }
  if (tile > 0) st[(size_t)tile * 256 + tid] = kSortPrefix | (unsigned)(before + total);
  // first position of the digit: exclusive scan of the digit counts of all keys
  int x = counts[tid];
  const int own = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sum[wid] = x;
  __syncthreads();
  int first = x - own;
#pragma unroll
  for (int w = 0; w < kWarps; ++w)
    if (w < wid) first += warp_sum[w];
  offs[tid] = first + before;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSortItems; ++j) {
    const int i = base + 32 * j;
    if (i >= n) continue;
    const int dig = (int)((key[j] >> shift) & 255u);
    const int pos = offs[dig] + wcnt[wid][dig] + rank[j];
    kout[pos] = key[j];
    vout[pos] = vin[i];
  }
}

}  // namespace

size_t scan_tmp_ints(int n) { return (size_t)((n + kScanBlock - 1) / kScanBlock + 1); }
size_t scan_tmp_doubles(int n) { return scan_tmp_ints(n); }

void exclusive_scan_runs(const SortedKeys& k, int* out, int n, int* tmp, cudaStream_t st) {
  scan_impl<int, false>(FirstOfRun{k.k64, k.k32}, out, n, tmp, st);
}
void inclusive_scan_double(const double* in, double* out, int n, double* tmp, cudaStream_t st) {
  scan_impl<double, true>(Plain<double>{in}, out, n, tmp, st);
}
void inclusive_scan_widen(const float* in, const int* n_dev, double* out, int n, double* tmp, cudaStream_t st) {
  scan_impl<double, true>(PrefixOf{in, n_dev}, out, n, tmp, st);
}

size_t sort_hist_ints(int n, int bits) {
  const size_t passes = (bits + 7) / 8, nt = ((size_t)n + kSortTile - 1) / kSortTile;
  return passes * (256 + 1) + passes * nt * 256;
}

template <class K>
static SortedKeys sort_impl(K* keys, uint32_t* vals, int n, int bits, SortTmp& tmp, cudaStream_t st) {
  const int passes = (bits + 7) / 8;
  K* ka = keys;
  uint32_t* va = vals;
  if (n > 1) {
    const int nt = (n + kSortTile - 1) / kSortTile;
    // digit counts and tickets of every pass, then the tiles' status words
    const size_t ints = sort_hist_ints(n, bits);
    tmp.keys2.alloc(sizeof(K) * n, st);
    tmp.vals2.alloc(sizeof(uint32_t) * n, st);
    tmp.hist.alloc(sizeof(int) * ints, st);
    int* counts = tmp.hist.as<int>();
    int* tickets = counts + passes * 256;
    unsigned* status = reinterpret_cast<unsigned*>(tickets + passes);
    PSDR_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * ints, st));
    k_sort_counts<K><<<std::min(nt, 2 * num_sms()), kSortThreads, 0, st>>>(ka, n, passes, counts);
    K* kb = tmp.keys2.as<K>();
    uint32_t* vb = tmp.vals2.as<uint32_t>();
    for (int p = 0; p < passes; ++p) {
      k_sort_pass<K><<<nt, kSortThreads, 0, st>>>(ka, va, kb, vb, n, 8 * p, counts + 256 * p, tickets + p,
                                                  status + (size_t)p * nt * 256);
      std::swap(ka, kb);
      std::swap(va, vb);
    }
    PSDR_CUDA(cudaGetLastError());
    count_launches(1 + passes);
  }
  SortedKeys out;
  if (sizeof(K) == 8) out.k64 = reinterpret_cast<uint64_t*>(ka);
  else out.k32 = reinterpret_cast<uint32_t*>(ka);
  out.vals = va;
  return out;
}

SortedKeys radix_sort_pairs(uint64_t* keys, uint32_t* vals, int n, int bits, SortTmp& tmp, cudaStream_t st) {
  return sort_impl(keys, vals, n, bits, tmp, st);
}
SortedKeys radix_sort_pairs(uint32_t* keys, uint32_t* vals, int n, int bits, SortTmp& tmp, cudaStream_t st) {
  return sort_impl(keys, vals, n, bits, tmp, st);
}

}  // namespace psdr
