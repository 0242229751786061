// Stand-in for the CUDA headers with which g++ compiles the kernels' sources, so that the
// CPU tests can run the device code itself: every thread of a block is a fiber, and a warp
// collective or a barrier hands over to the next fiber until all the threads it names have
// arrived. Arithmetic is the host's, without contraction.
#pragma once

#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <ucontext.h>

#include <cmath>
#include <functional>
#include <map>
#include <utility>
#include <vector>

#define __host__
#define __device__
#define __global__
#define __constant__
#define __shared__ static
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

using std::fabs;
using std::floor;
using std::fma;
using std::fmax;
using std::fmin;
using std::log10;
using std::pow;
using std::sqrt;

struct uint3 { unsigned x, y, z; };
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
inline float2 make_float2(float x, float y) { return {x, y}; }
typedef int cudaError_t;
typedef void* cudaStream_t;
enum { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
template <class F>
cudaError_t cudaFuncSetAttribute(F, int, int) { return cudaSuccess; }
template <class F>
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, F, int, size_t) { *n = 1; return cudaSuccess; }

inline uint3 threadIdx{}, blockIdx{}, blockDim{}, gridDim{};

namespace emu {
struct Barrier { int arrived = 0; unsigned turn = 0; };
struct Block {
  std::vector<ucontext_t> fibers;
  std::vector<bool> done;
  std::vector<std::vector<char>> stacks;
  std::map<std::pair<int, unsigned>, Barrier> bars;  // by warp (-1: the block) and lane mask
  unsigned char slot[32][32][16];                    // a warp's exchanged values
  std::vector<unsigned char> smem;                   // dynamic shared memory
  std::function<void()> body;
  int cur = 0;
  ucontext_t home;
};
inline Block* B = nullptr;

inline unsigned char* smem() { return (unsigned char*)(((uintptr_t)B->smem.data() + 15) & ~(uintptr_t)15); }
inline void yield() {
  const int from = B->cur, n = (int)B->done.size();
  for (int k = 1; k <= n; ++k) {
    const int to = (from + k) % n;
    if (B->done[to]) continue;
    B->cur = to;
    threadIdx.x = to;
    if (to != from) swapcontext(&B->fibers[from], &B->fibers[to]);
    return;
  }
  setcontext(&B->home);
}
inline void entry() {
  B->body();
  B->done[B->cur] = true;
  yield();
}
inline void arrive(int warp, unsigned mask, int count) {
  Barrier& b = B->bars[{warp, mask}];
  const unsigned turn = b.turn;
  if (++b.arrived == count) {
    b.arrived = 0;
    ++b.turn;
    return;
  }
  for (long spin = 0; b.turn == turn; ++spin) {
    if (spin > 10000000) { fprintf(stderr, "a barrier waits for threads that never come\n"); exit(3); }
    yield();
  }
}
// One block of n threads; launch(grid, n, smem, f) runs the blocks one after the other.
inline void launch(int grid, int n, size_t smem, std::function<void()> f) {
  for (int b = 0; b < grid; ++b) {
    Block blk;
    B = &blk;
    blk.fibers.resize(n);
    blk.done.assign(n, false);
    blk.stacks.assign(n, std::vector<char>(1 << 18));
    blk.smem.assign(smem + 16, 0);
    blk.body = f;
    blockIdx.x = b; gridDim.x = grid; blockDim.x = n; threadIdx.x = 0;
    for (int i = 0; i < n; ++i) {
      getcontext(&blk.fibers[i]);
      blk.fibers[i].uc_stack.ss_sp = blk.stacks[i].data();
      blk.fibers[i].uc_stack.ss_size = blk.stacks[i].size();
      blk.fibers[i].uc_link = nullptr;
      makecontext(&blk.fibers[i], entry, 0);
    }
    swapcontext(&blk.home, &blk.fibers[0]);
    B = nullptr;
  }
}
inline int lane() { return threadIdx.x & 31; }
inline int warp() { return threadIdx.x >> 5; }
template <class V, class R>
R collect(unsigned mask, V v, R (*read)(const V*, unsigned, int, int), int arg) {
  static_assert(sizeof(V) <= 16, "");
  const int w = warp(), l = lane();
  memcpy(B->slot[w][l], &v, sizeof(V));
  arrive(w, mask, __builtin_popcount(mask));
  V all[32];
  for (int i = 0; i < 32; ++i)
    if (mask >> i & 1) memcpy(&all[i], B->slot[w][i], sizeof(V));
  const R r = read(all, mask, l, arg);
  arrive(w, mask, __builtin_popcount(mask));
  return r;
}
}  // namespace emu

inline void __syncthreads() { emu::arrive(-1, 0, (int)emu::B->done.size()); }
inline void __syncwarp(unsigned mask = 0xffffffffu) { emu::arrive(emu::warp(), mask, __builtin_popcount(mask)); }
template <class T>
T __shfl_sync(unsigned mask, T v, int src, int width = 32) {
  return emu::collect<T, T>(mask, v, [](const T* a, unsigned, int l, int arg) {
    const int w = arg >> 8, s = arg & 255;
    return a[(l & ~(w - 1)) + (s & (w - 1))];
  }, width << 8 | (src & 31));
}
template <class T>
T __shfl_xor_sync(unsigned mask, T v, int off, int = 32) {
  return emu::collect<T, T>(mask, v, [](const T* a, unsigned, int l, int arg) { return a[l ^ arg]; }, off);
}
inline unsigned __ballot_sync(unsigned mask, bool p) {
  return emu::collect<bool, unsigned>(mask, p, [](const bool* a, unsigned m, int, int) {
    unsigned r = 0;
    for (int i = 0; i < 32; ++i)
      if ((m >> i & 1) && a[i]) r |= 1u << i;
    return r;
  }, 0);
}
inline bool __any_sync(unsigned mask, bool p) { return __ballot_sync(mask, p) != 0; }
template <class T>
T __reduce_max_sync(unsigned mask, T v) {
  return emu::collect<T, T>(mask, v, [](const T* a, unsigned m, int, int) {
    T r = a[__builtin_ctz(m)];
    for (int i = 0; i < 32; ++i)
      if ((m >> i & 1) && a[i] > r) r = a[i];
    return r;
  }, 0);
}
template <class T>
T __reduce_min_sync(unsigned mask, T v) {
  return emu::collect<T, T>(mask, v, [](const T* a, unsigned m, int, int) {
    T r = a[__builtin_ctz(m)];
    for (int i = 0; i < 32; ++i)
      if ((m >> i & 1) && a[i] < r) r = a[i];
    return r;
  }, 0);
}
inline int __ffs(int x) { return __builtin_ffs(x); }
inline int __popc(unsigned x) { return __builtin_popcount(x); }
inline int __clz(int x) { return x ? __builtin_clz(x) : 32; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __expf(float x) { return expf(x); }
inline double cospi(double x) { return cos(3.14159265358979323846 * x); }
template <class To, class From>
To emu_bits(From v) { To r; static_assert(sizeof(r) == sizeof(v), ""); memcpy(&r, &v, sizeof(r)); return r; }
inline int __float_as_int(float v) { return emu_bits<int>(v); }
inline long long __double_as_longlong(double v) { return emu_bits<long long>(v); }
inline double __longlong_as_double(long long v) { return emu_bits<double>(v); }
inline int __double2hiint(double v) { return (int)(emu_bits<unsigned long long>(v) >> 32); }
inline int __double2loint(double v) { return (int)emu_bits<unsigned long long>(v); }
inline double __hiloint2double(int hi, int lo) {
  return emu_bits<double>((unsigned long long)(unsigned)hi << 32 | (unsigned)lo);
}
template <class T>
T __ldg(const T* p) { return *p; }
template <class T>
T atomicAdd(T* p, T v) { const T old = *p; *p = old + v; return old; }
inline long long clock64() { return 0; }
