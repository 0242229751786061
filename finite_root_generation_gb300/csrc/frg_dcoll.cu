// Device-resident root collection with duplicate marking (include/frg_gb300.h,
// frg_dcoll_*): the reference's SortingDeletingMerging (frgsupport.cu:10-215) with the
// driver's thrust ordering (frg.cu:432-435) done on the GPU, across rounds, for many
// tasks at once (one collection per key, e.g. per task).
//
// The duplicate rule is the host merge's (frg_collect.cpp), which restates the
// reference's: a success (code 0) becomes a duplicate (code 6) when every real
// component is within tol of a collected root of its key, or of a lower-index success
// of the same batch and key that is itself not a duplicate. Two roots within tol have
// Re(root[0]) in the same or adjacent cells of width 2 tol (the doubled width keeps that
// true after rounding x / (2 tol)), so candidates come from a hash table keyed by
// (key, cell) instead of the reference's sorted neighbour scan; every candidate is
// compared in all 42 components, so the marks are the same.
//
// One merge, all on the caller's stream:
//   1. check_insert   each success against the collection (read-only table); the
//                     remaining successes into a batch table
//   2. check_append   a success with no earlier in-batch match is kept and joins the
//                     collection; one with an earlier match is "dependent" (its status
//                     depends on the earlier roots' statuses)
//   3. resolve        one block: dependent roots that match an independent one are
//                     duplicates; the others are walked in index order, the host rule
//                     applied sequentially, and those that are kept join the collection
// Bound by the latency of the probes and by the launches; the rows, 336 bytes each, are
// copied by whole warps. A call merging 65,536 roots, host side included: new roots
// 158 -> 86 us, all known 114 -> 66 us; four rounds of 65,536 with 20 % repeats, creation
// and release of the collection included, 2.00 -> 0.89 ms.
// Roots whose first component is not finite never match (the host merge would let
// NaN compare equal); a success with a residual check has finite components. Every
// table probe is bounded by the table size.
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <new>

#include "../../include/frg_gb300.h"

namespace {

constexpr int kReals = 2 * FRG_NV;
constexpr unsigned long long kEmpty = ~0ull;
constexpr int kThreads = 256;
constexpr int64_t kMost = (int64_t)1 << 48;  // roots: more fit no GPU, and their bytes may not fit 64 bits

struct DcollDev {
  double* roots;                  // capacity x 42
  int32_t* keys;                  // capacity collection keys
  unsigned long long* tkey;       // table: packed (key, cell) or kEmpty
  int64_t* tval;                  // table: root index
  unsigned long long tmask;       // table size - 1 (power of two)
  unsigned long long* size;       // [0] roots in the collection, [1] overflow flag
  int64_t capacity;
};

// (key, cell) packed into 64 bits: key in the top 20 bits, cell (clamped) in the low 44
__device__ __forceinline__ unsigned long long pack(int32_t key, long long cell) {
  const long long lim = (1ll << 43) - 1;
  cell = cell > lim ? lim : (cell < -lim ? -lim : cell);
  return ((unsigned long long)(uint32_t)key << 44) | ((unsigned long long)cell & ((1ull << 44) - 1));
}

__device__ __forceinline__ unsigned long long mix(unsigned long long x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  x ^= x >> 33;
  return x;
}

// cell of width 2 tol of Re(root[0]); false if it is not finite
__device__ __forceinline__ bool cell_of(const double* r, double tol, long long* cell) {
  const double x = r[0];
  if (!(x - x == 0.0)) return false;
  *cell = (long long)floor(x * (0.5 / tol));
  return true;
}

// a success that takes part in the merge: code 0 and, when residuals are given, a
// residual of at most resid_max (a NaN residual fails)
__device__ __forceinline__ bool takes_part(const int32_t* codes, const double* resid, double resid_max, int64_t t) {
  return codes[t] == 0 && (!resid || resid[t] <= resid_max);
}

// every component within tol; seven at a time, so that a true match waits for memory six
// times and not 42
__device__ __forceinline__ bool same_root(const double* a, const double* b, double tol) {
  for (int k0 = 0; k0 < kReals; k0 += 7) {
    double x[7], y[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) { x[k] = a[k0 + k]; y[k] = b[k0 + k]; }
    bool same = true;
#pragma unroll
    for (int k = 0; k < 7; ++k) same = same && fabs(x[k] - y[k]) <= tol;
    if (!same) return false;
  }
  return true;
}

__device__ void table_insert(unsigned long long* tkey, int64_t* tval, unsigned long long tmask,
                             unsigned long long k, int64_t v) {
  unsigned long long h = mix(k) & tmask;
  for (unsigned long long probe = 0; probe <= tmask; ++probe) {
    const unsigned long long prev = atomicCAS(&tkey[h], kEmpty, k);
    if (prev == kEmpty) {
      tval[h] = v;
      return;
    }
    h = (h + 1) & tmask;
  }
}

// 1. successes matching a collected root of their key become duplicates, the others join
//    the batch table
__global__ void __launch_bounds__(kThreads) check_insert(DcollDev c, const double* roots, int32_t* codes,
                                                        const double* resid, double resid_max, const int32_t* keys,
                                                        int64_t n, double tol, unsigned long long* bkey,
                                                        int64_t* bval, unsigned long long bmask,
                                                        unsigned long long* ndep) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) *ndep = 0;
  if (t >= n || !takes_part(codes, resid, resid_max, t)) return;
  const double* rt = roots + (size_t)t * kReals;
  long long cell;
  if (!cell_of(rt, tol, &cell)) return;
  const int32_t key = keys ? keys[t] : 0;
  for (int dc = -1; dc <= 1; ++dc) {
    const unsigned long long k = pack(key, cell + dc);
    unsigned long long h = mix(k) & c.tmask;
    for (unsigned long long probe = 0; probe <= c.tmask; ++probe) {
      const unsigned long long e = c.tkey[h];
      if (e == kEmpty) break;
      if (e == k && same_root(rt, c.roots + (size_t)c.tval[h] * kReals, tol)) {
        codes[t] = FRG_CODE_DUPLICATE;
        return;
      }
      h = (h + 1) & c.tmask;
    }
  }
  table_insert(bkey, bval, bmask, pack(key, cell), t);
}

// 2. a success with an earlier matching success of the batch depends on it; the others
//    are kept. The warp copies its kept rows together.
__global__ void __launch_bounds__(kThreads) check_append(DcollDev c, const double* roots, const int32_t* codes,
                                                        const double* resid, double resid_max, const int32_t* keys,
                                                        int64_t n, double tol, const unsigned long long* bkey,
                                                        const int64_t* bval, unsigned long long bmask,
                                                        unsigned char* dep, int64_t* deps,
                                                        unsigned long long* ndep) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool part = t < n && takes_part(codes, resid, resid_max, t);
  const double* rt = roots + (size_t)t * kReals;
  const int32_t key = part && keys ? keys[t] : 0;
  long long cell = 0;
  const bool finite = part && cell_of(rt, tol, &cell);
  bool depends = false;
  for (int dc = -1; dc <= 1 && finite && !depends; ++dc) {
    const unsigned long long k = pack(key, cell + dc);
    unsigned long long h = mix(k) & bmask;
    for (unsigned long long probe = 0; probe <= bmask; ++probe) {
      const unsigned long long e = bkey[h];
      if (e == kEmpty) break;
      const int64_t u = bval[h];
      if (e == k && u < t && same_root(rt, roots + (size_t)u * kReals, tol)) {
        depends = true;
        break;
      }
      h = (h + 1) & bmask;
    }
  }
  if (t < n) dep[t] = depends;
  if (depends) deps[atomicAdd(ndep, 1ull)] = t;
  const bool keep = part && !depends;
  const unsigned kept = __ballot_sync(0xffffffffu, keep);
  if (!kept) return;
  // one reservation for the warp; roots past the capacity are not collected
  const int cnt = __popc(kept), rank = __popc(kept & ((1u << lane) - 1));
  unsigned long long first = 0;
  if (lane == 0) first = atomicAdd(&c.size[0], (unsigned long long)cnt);
  first = __shfl_sync(0xffffffffu, first, 0);
  const int64_t room = c.capacity - (int64_t)first;
  const int rows = room <= 0 ? 0 : (room < cnt ? (int)room : cnt);
  if (rows < cnt && lane == 0) c.size[1] = 1;
  __shared__ unsigned char from[kThreads];  // lane of the warp's r-th kept root
  unsigned char* src = from + (threadIdx.x & ~31);
  if (keep) src[rank] = (unsigned char)lane;
  __syncwarp();
  // the rows lie one after another in the collection: 8 loads in flight per lane
  double* dst = c.roots + first * kReals;
  const double* base = roots + (size_t)(t - lane) * kReals;
  for (int i0 = lane; i0 < rows * kReals; i0 += 32 * 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + 32 * u;
      if (i < rows * kReals) v[u] = base[src[i / kReals] * kReals + i % kReals];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + 32 * u;
      if (i < rows * kReals) dst[i] = v[u];
    }
  }
  if (keep && rank < rows) {
    const int64_t slot = (int64_t)first + rank;
    c.keys[slot] = key;
    if (finite) table_insert(c.tkey, c.tval, c.tmask, pack(key, cell), slot);
  }
}

// Is an earlier success of the batch that matches root t kept? With `sure`, only those that
// depend on nothing count (they are kept whatever the others are).
__device__ __forceinline__ bool kept_match(const double* roots, const int32_t* codes, const int32_t* keys, int64_t t,
                                           double tol, const unsigned long long* bkey, const int64_t* bval,
                                           unsigned long long bmask, const unsigned char* dep, bool sure) {
  const double* rt = roots + (size_t)t * kReals;
  long long cell = 0;
  cell_of(rt, tol, &cell);
  const int32_t key = keys ? keys[t] : 0;
  for (int dc = -1; dc <= 1; ++dc) {
    const unsigned long long k = pack(key, cell + dc);
    unsigned long long h = mix(k) & bmask;
    for (unsigned long long probe = 0; probe <= bmask; ++probe) {
      const unsigned long long e = bkey[h];
      if (e == kEmpty) break;
      const int64_t u = bval[h];
      if (e == k && u < t && (sure ? !dep[u] : codes[u] == 0) && same_root(rt, roots + (size_t)u * kReals, tol))
        return true;
      h = (h + 1) & bmask;
    }
  }
  return false;
}

// A dependent root, once those before it are settled: a duplicate when an earlier matching
// success is still a success (the host merge's sequential rule), collected otherwise.
__device__ void settle(const DcollDev& c, const double* roots, int32_t* codes, const int32_t* keys, int64_t t,
                       double tol, const unsigned long long* bkey, const int64_t* bval, unsigned long long bmask,
                       const unsigned char* dep) {
  if (kept_match(roots, codes, keys, t, tol, bkey, bval, bmask, dep, false)) {
    codes[t] = FRG_CODE_DUPLICATE;
    return;
  }
  const unsigned long long slot = atomicAdd(&c.size[0], 1ull);
  if ((int64_t)slot >= c.capacity) {
    c.size[1] = 1;  // overflow: the root is not collected
    return;
  }
  const double* rt = roots + (size_t)t * kReals;
  for (int k = 0; k < kReals; ++k) c.roots[slot * kReals + k] = rt[k];
  const int32_t key = keys ? keys[t] : 0;
  c.keys[slot] = key;
  long long cell;
  if (cell_of(rt, tol, &cell)) table_insert(c.tkey, c.tval, c.tmask, pack(key, cell), (int64_t)slot);
}

// 3. dependent roots. One block. A root that matches an independent one is a duplicate
//    whatever the others are, and all threads look for those; the rest is settled by thread 0
//    in index order, 8 us each: a list that fits is ordered by rank, a longer one found again
//    from the flags by the whole block, 1,024 at a time (262,144 roots, 1,000 / 1,100 / 5,000 to
//    settle: 8.8 / 9.6 / 41 ms; with thread 0 walking the flags 8.8 / 40 / 74).
__global__ void __launch_bounds__(1024) resolve(DcollDev c, const double* roots, int32_t* codes, const int32_t* keys,
                                                int64_t n, double tol, const unsigned long long* bkey,
                                                const int64_t* bval, unsigned long long bmask, unsigned char* dep,
                                                const int64_t* deps, const unsigned long long* ndep) {
  __shared__ int64_t open_[1024], order[1024];
  __shared__ unsigned long long count;
  __shared__ int before[33];
  const unsigned long long all = *ndep;
  if (all == 0) return;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  for (unsigned long long i = threadIdx.x; i < all; i += blockDim.x) {
    const int64_t t = deps[i];
    if (kept_match(roots, codes, keys, t, tol, bkey, bval, bmask, dep, true)) {
      codes[t] = FRG_CODE_DUPLICATE;
    } else {
      const unsigned long long slot = atomicAdd(&count, 1ull);
      if (slot < 1024) open_[slot] = t;
    }
  }
  __syncthreads();
  const unsigned long long left = count;
  if (left <= 1024) {
    if (threadIdx.x < left) {
      int rank = 0;
      for (unsigned long long i = 0; i < left; ++i) rank += open_[i] < open_[threadIdx.x];
      order[rank] = open_[threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < (int)left; ++i) settle(c, roots, codes, keys, order[i], tol, bkey, bval, bmask, dep);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t base = 0; base < n; base += 1024) {
    const int64_t t = base + threadIdx.x;
    const bool open = t < n && dep[t] && codes[t] == 0;
    const unsigned ballot = __ballot_sync(0xffffffffu, open);
    if (!__syncthreads_or(open)) continue;
    if (lane == 0) before[warp + 1] = __popc(ballot);
    __syncthreads();
    if (threadIdx.x == 0) {
      before[0] = 0;
      for (int w = 1; w <= 32; ++w) before[w] += before[w - 1];
    }
    __syncthreads();
    if (open) order[before[warp] + __popc(ballot & ((1u << lane) - 1))] = t;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < before[32]; ++i) settle(c, roots, codes, keys, order[i], tol, bkey, bval, bmask, dep);
    __syncthreads();
  }
}

unsigned long long pow2_at_least(unsigned long long x) {
  unsigned long long p = 1024;
  while (p < x) p <<= 1;
  return p;
}

}  // namespace

struct frg_dcoll {
  int device = 0;
  double tol = 1e-6;
  DcollDev d{};
  void* mem = nullptr;  // the collection's arrays, one allocation
  // batch scratch (grown on demand), one allocation: table keys, then the count of dependent
  // roots, table values, dependent roots
  // and their flags
  void* bmem = nullptr;
  unsigned long long* bkey = nullptr;
  int64_t* bval = nullptr;
  unsigned char* dep = nullptr;
  int64_t* deps = nullptr;  // the dependent roots, in no order
  unsigned long long* ndep = nullptr;
  unsigned long long bsize = 0;
  int64_t bn = 0;
};

static void dcoll_free_batch(frg_dcoll* c) {
  cudaFree(c->bmem);
  c->bmem = nullptr;
  c->bkey = nullptr;
  c->bval = nullptr;
  c->dep = nullptr;
  c->deps = nullptr;
  c->ndep = nullptr;
  c->bsize = 0;
  c->bn = 0;
}

extern "C" void frg_dcoll_destroy(frg_dcoll* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaDeviceSynchronize();
  cudaFree(c->mem);
  dcoll_free_batch(c);
  delete c;
}

extern "C" frg_status frg_dcoll_create(frg_dcoll** out, int device, int64_t capacity, double dup_tol) {
  if (!out) return FRG_ERR_ARG;
  *out = nullptr;
  if (capacity < 1 || !(dup_tol > 0) || !std::isfinite(dup_tol)) return FRG_ERR_ARG;
  if (capacity > kMost) return FRG_ERR_CUDA;
  frg_dcoll* c = new (std::nothrow) frg_dcoll();
  if (!c) return FRG_ERR_ALLOC;
  c->device = device;
  c->tol = dup_tol;
  c->d.capacity = capacity;
  const unsigned long long tsize = pow2_at_least((unsigned long long)capacity * 2);
  c->d.tmask = tsize - 1;
  // table keys, size, table values, roots, keys: every array starts 8-byte aligned
  const size_t kb = sizeof(unsigned long long) * tsize, sb = sizeof(unsigned long long) * 2,
               vb = sizeof(int64_t) * tsize, rb = sizeof(double) * kReals * (size_t)capacity,
               ib = sizeof(int32_t) * (size_t)capacity;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaMalloc(&c->mem, kb + sb + vb + rb + ib);
  if (e == cudaSuccess) {
    char* m = (char*)c->mem;
    c->d.tkey = (unsigned long long*)m;
    c->d.size = (unsigned long long*)(m + kb);
    c->d.tval = (int64_t*)(m + kb + sb);
    c->d.roots = (double*)(m + kb + sb + vb);
    c->d.keys = (int32_t*)(m + kb + sb + vb + rb);
    e = cudaMemset(c->d.tkey, 0xff, kb);
  }
  if (e == cudaSuccess) e = cudaMemset(c->d.size, 0, sb);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    frg_dcoll_destroy(c);
    return FRG_ERR_CUDA;
  }
  *out = c;
  return FRG_OK;
}

extern "C" frg_status frg_dcoll_merge(frg_dcoll* c, const double* roots, int32_t* codes, const double* resid,
                                      double resid_max, const int32_t* keys, int64_t n, void* stream) {
  if (!c || n < 0 || (n > 0 && (!roots || !codes))) return FRG_ERR_ARG;
  if (n == 0) return FRG_OK;
  if (n > kMost) return FRG_ERR_ALLOC;
  if (cudaSetDevice(c->device) != cudaSuccess) return FRG_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  if (n > c->bn) {
    if (cudaStreamSynchronize(st) != cudaSuccess) return FRG_ERR_CUDA;
    dcoll_free_batch(c);
    const unsigned long long bs = pow2_at_least((unsigned long long)n * 2);
    const size_t kb = sizeof(unsigned long long) * bs;
    const size_t bytes = kb + sizeof(unsigned long long) + sizeof(int64_t) * bs + (sizeof(int64_t) + 1) * (size_t)n;
    if (cudaMalloc(&c->bmem, bytes) != cudaSuccess) {
      dcoll_free_batch(c);
      return FRG_ERR_ALLOC;
    }
    char* m = (char*)c->bmem;
    c->bkey = (unsigned long long*)m;
    c->ndep = (unsigned long long*)(m + kb);
    c->bval = (int64_t*)(m + kb + sizeof(unsigned long long));
    c->deps = (int64_t*)(m + kb + sizeof(unsigned long long) + sizeof(int64_t) * bs);
    c->dep = (unsigned char*)(c->deps + n);
    c->bsize = bs;
    c->bn = n;
  }
  const unsigned long long bmask = c->bsize - 1;
  if (cudaMemsetAsync(c->bkey, 0xff, sizeof(unsigned long long) * c->bsize, st) != cudaSuccess) return FRG_ERR_CUDA;
  const unsigned grid = (unsigned)((n + kThreads - 1) / kThreads);
  check_insert<<<grid, kThreads, 0, st>>>(c->d, roots, codes, resid, resid_max, keys, n, c->tol, c->bkey, c->bval,
                                          bmask, c->ndep);
  check_append<<<grid, kThreads, 0, st>>>(c->d, roots, codes, resid, resid_max, keys, n, c->tol, c->bkey, c->bval,
                                          bmask, c->dep, c->deps, c->ndep);
  resolve<<<1, 1024, 0, st>>>(c->d, roots, codes, keys, n, c->tol, c->bkey, c->bval, bmask, c->dep, c->deps, c->ndep);
  return cudaGetLastError() == cudaSuccess ? FRG_OK : FRG_ERR_CUDA;
}

extern "C" frg_status frg_dcoll_size(frg_dcoll* c, void* stream, int64_t* size) {
  if (!c || !size) return FRG_ERR_ARG;
  if (cudaSetDevice(c->device) != cudaSuccess) return FRG_ERR_CUDA;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned long long h[2] = {0, 0};
  if (cudaMemcpyAsync(h, c->d.size, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return FRG_ERR_CUDA;
  if (h[1]) return FRG_ERR_ALLOC;  // a merge ran out of capacity
  *size = (int64_t)h[0];
  return FRG_OK;
}

extern "C" frg_status frg_dcoll_get(frg_dcoll* c, double* roots, int32_t* keys, int64_t capacity) {
  if (!c) return FRG_ERR_ARG;
  if (cudaSetDevice(c->device) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return FRG_ERR_CUDA;
  int64_t n = 0;
  frg_status s = frg_dcoll_size(c, nullptr, &n);
  if (s != FRG_OK) return s;
  if (capacity < n || (n > 0 && !roots)) return FRG_ERR_ARG;
  if (n == 0) return FRG_OK;
  if (cudaMemcpy(roots, c->d.roots, sizeof(double) * kReals * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess)
    return FRG_ERR_CUDA;
  if (keys && cudaMemcpy(keys, c->d.keys, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost) != cudaSuccess)
    return FRG_ERR_CUDA;
  return FRG_OK;
}
