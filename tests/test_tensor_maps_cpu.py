"""The cache of tensor maps (csrc/host.cu) against stand-ins for the CUDA calls it makes, on the CPU: a map that a launcher holds stays
what it was while later calls, its own or another thread's, fill the cache until it is dropped."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"

CUDA_H = r"""
#pragma once
#include <cstddef>
#include <cstdint>
typedef int CUresult; typedef int CUtensorMapDataType, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill;
typedef uint32_t cuuint32_t; typedef uint64_t cuuint64_t;
struct alignas(64) CUtensorMap { uint64_t opaque[16]; };
enum { CUDA_SUCCESS = 0, CU_TENSOR_MAP_SWIZZLE_NONE = 0, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_SWIZZLE_128B,
       CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 = 9, CU_TENSOR_MAP_INTERLEAVE_NONE = 0, CU_TENSOR_MAP_L2_PROMOTION_L2_256B = 3,
       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE = 0 };
"""

RUNTIME_H = r"""
#pragma once
#include "cuda.h"
#include <cstring>
#define __device__
typedef int cudaError_t; typedef void* cudaStream_t;
enum { cudaSuccess = 0, cudaEnableDefault = 0, cudaMemcpyDeviceToHost = 2, cudaDevAttrMultiProcessorCount = 16 };
enum cudaDriverEntryPointQueryResult { cudaDriverEntryPointSuccess = 0 };
struct dim3 { unsigned x, y, z; dim3(unsigned a = 1, unsigned b = 1, unsigned c = 1) : x(a), y(b), z(c) {} };
enum { cudaLaunchAttributeClusterDimension = 4, cudaLaunchAttributeProgrammaticStreamSerialization = 6 };
struct cudaLaunchAttribute { int id; struct { struct { unsigned x, y, z; } clusterDim; int programmaticStreamSerializationAllowed; } val; };
struct cudaLaunchConfig_t { dim3 gridDim, blockDim; size_t dynamicSmemBytes; cudaStream_t stream; cudaLaunchAttribute* attrs; unsigned numAttrs; };
template <typename... P, typename... A> int cudaLaunchKernelEx(const cudaLaunchConfig_t*, void (*)(P...), A...) { return 0; }
inline int cudaGetDevice(int* d) { *d = 0; return 0; }
inline int cudaSetDevice(int) { return 0; }
inline int cudaFree(void*) { return 0; }
inline int cudaMemset(void*, int, size_t) { return 0; }
inline int cudaMemcpy(void*, const void*, size_t, int) { return 0; }
inline int cudaDeviceGetAttribute(int* v, int, int) { *v = 148; return 0; }
template <typename T> int cudaGetSymbolAddress(void** p, const T& s) { *p = (void*)&s; return 0; }
// the map is its base address over and over, so that any other content shows
inline CUresult fake_encode(CUtensorMap* m, int, cuuint32_t, void* base, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                            int, int, int, int) {
  for (auto& w : m->opaque) w = (uint64_t)base;
  return (uint64_t)base % 16 ? 1 : CUDA_SUCCESS;
}
inline int cudaGetDriverEntryPoint(const char*, void** p, int, cudaDriverEntryPointQueryResult* q) {
  *p = (void*)fake_encode; *q = cudaDriverEntryPointSuccess; return 0;
}
"""

MAIN = r"""
#include "host.h"
#include <cstdio>
#include <thread>
#include <vector>
static bool holds(const CUtensorMap& m, uint64_t base) { for (auto w : m.opaque) if (w != base) return false; return true; }
static void fill(uint64_t from, int n) { for (int i = 0; i < n; ++i) b2::tensor_map_2d_bf16((void*)(from + 16ull * i), 8, 64, 64, 8, 64); }
int main() {
  if (b2::tensor_map_2d_bf16((void*)0x1008, 8, 64, 64, 8, 64)) return 1;            // refused: not aligned
  auto held = b2::tensor_map_2d_bf16((void*)0x1000, 8, 64, 64, 8, 64);
  auto again = b2::tensor_map_2d_bf16((void*)0x1000, 8, 64, 64, 8, 64);             // from the cache
  if (!held || !again || !holds(*again, 0x1000)) return 2;
  fill(1ull << 32, 70000);
  if (!holds(*held, 0x1000)) return 3;
  int bad = 0;
  std::vector<std::thread> others;
  for (int t = 0; t < 4; ++t) others.emplace_back([t] { fill((2ull + t) << 36, 70000); });
  for (int i = 0; i < 20000; ++i) {
    const uint64_t a = (9ull << 36) + 64 * i, b = a + 32;
    auto ta = b2::tensor_map_2d_bf16((void*)a, 8, 64, 64, 8, 64);
    auto tb = b2::tensor_map_2d_bf16((void*)b, 8, 64, 64, 8, 64);
    if (!ta || !tb || !holds(*ta, a) || !holds(*tb, b)) ++bad;
  }
  for (auto& t : others) t.join();
  return bad ? 4 : 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_maps_outlive_the_cache(tmp_path):
    (tmp_path / "cuda.h").write_text(CUDA_H)
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME_H)
    (tmp_path / "main.cpp").write_text(MAIN)
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-pthread", "-I", str(tmp_path), "-I", str(CSRC), "-x", "c++",
           str(CSRC / "host.cu"), str(tmp_path / "main.cpp"), "-o", str(tmp_path / "maps")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(tmp_path / "maps")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-3000:])
