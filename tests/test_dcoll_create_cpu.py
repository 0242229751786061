"""The device collection's allocations, its source compiled with stand-ins for the CUDA calls
(tests/warp_emu): a capacity or a batch that no GPU holds is refused, also where the sizes of
the arrays add up past 64 bits, and nothing is cleared outside what was allocated."""
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "finite_root_generation_gb300", "csrc")

MAIN = r"""
#include "cuda_runtime.h"
static char* base = nullptr;
static size_t held = 0;
static bool outside = false;
enum { cudaMemcpyDeviceToHost = 2, cudaErrorMemoryAllocation = 2 };
static cudaError_t cudaSetDevice(int) { return 0; }
static cudaError_t cudaDeviceSynchronize() { return 0; }
static cudaError_t cudaStreamSynchronize(cudaStream_t) { return 0; }
template <class T> cudaError_t cudaMalloc(T** p, size_t n) {
  if (n > (size_t)1 << 30) return cudaErrorMemoryAllocation;
  *p = (T*)malloc(n ? n : 1);
  base = (char*)*p;
  held = n;
  return 0;
}
static cudaError_t cudaFree(void* p) { free(p); return 0; }
static cudaError_t cudaMemset(void* p, int v, size_t n) {
  if ((char*)p < base || n > held || (size_t)((char*)p - base) > held - n) { outside = true; return 1; }
  memset(p, v, n);
  return 0;
}
static cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
static cudaError_t cudaMemcpy(void*, const void*, size_t, int) { return 1; }
static cudaError_t cudaMemcpyAsync(void*, const void*, size_t, int, cudaStream_t) { return 1; }
static int __syncthreads_or(int v) { return v; }
static unsigned long long atomicCAS(unsigned long long*, unsigned long long, unsigned long long) { return 0; }
#include "dcoll.inc"
int main() {
  setvbuf(stdout, nullptr, _IONBF, 0);
  const int64_t kib = 1024;
  int bad = 0;
  // 340 c + 16 t + 16 bytes with a table of t = 2^57 slots: 2^64 + 48 KiB or so at the third
  for (int64_t c : {(int64_t)1, kib * kib, (int64_t)((7ull << 61) / 340) + kib * 48 / 340, ((int64_t)1) << 52,
                    ((int64_t)1) << 60, INT64_MAX}) {
    frg_dcoll* d = nullptr;
    const frg_status s = frg_dcoll_create(&d, 0, c, 1e-6);
    if (outside || s != (c <= kib * kib ? FRG_OK : FRG_ERR_CUDA) || (d != nullptr) != (s == FRG_OK)) {
      printf("capacity %lld: status %d, outside %d\n", (long long)c, (int)s, (int)outside);
      ++bad;
    }
    outside = false;
    if (s != FRG_OK) continue;
    for (uint64_t n : {~0ull / 9 + 2, 1ull << 62})
      if (frg_dcoll_merge(d, (double*)8, (int32_t*)8, nullptr, 0.0, nullptr, (int64_t)n, nullptr) != FRG_ERR_ALLOC) {
        printf("a batch of %llu accepted\n", (unsigned long long)n);
        ++bad;
      }
    frg_dcoll_destroy(d);
  }
  return bad;
}
"""


def test_capacity_beyond_any_gpu_is_refused(tmp_path):
    src = open(os.path.join(CSRC, "frg_dcoll.cu")).read()
    src = re.sub(r"\w+<<<.*?>>>\(.*?\);", ";", src, flags=re.S).replace('"../../include/', '"')
    (tmp_path / "dcoll.inc").write_text(src)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-w", f"-I{tmp_path}", f"-I{os.path.join(HERE, 'warp_emu')}",
                    f"-I{os.path.join(HERE, '..', 'include')}", str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run(["timeout", "20", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
