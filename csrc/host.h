// Host-side helpers shared by the launchers: status word access and TMA tensor-map encoding.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdlib>

#define B2_EXPORT extern "C" __attribute__((visibility("default")))

namespace b2 {

// activations a matrix product can apply to its first output columns
constexpr int GEMM_ACT_SILU = 1;
constexpr int GEMM_ACT_RELU2 = 2;    // the square of relu

// Makes the process's device (b2_set_device) current on the calling thread.  Launchers call this
// first: autograd runs backward passes on worker threads that this library's runtime has never
// seen, and driver entry points such as the tensor-map encoder need a current context.
void ensure_thread_context();

// Device address of this device's status word (one int; 0 = no error).
int* status_ptr();

// Last host-side error text (argument checks, CUDA runtime failures).
void set_error(const char* fmt, ...);

// A tensor map, or none (with the reason in set_error's text).  By value: the cache behind the two functions below may drop its
// entries in any later call, of this launcher or of another thread's.
struct TensorMap {
  CUtensorMap map;
  bool ok = false;
  explicit operator bool() const { return ok; }
  const CUtensorMap& operator*() const { return map; }
};

// Encode (and cache) a 2-D tiled tensor map over a row-major [rows, cols] matrix of 2-byte
// elements with row stride `ld` elements; box = [box_rows, box_cols], 128-byte swizzle.
// box_cols * 2 must be 128.
TensorMap tensor_map_2d_bf16(const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, uint32_t box_cols);

// Generic N-D (<=4) tiled tensor map for 2-byte elements.  dims/strides innermost first; strides in
// bytes for dims 1..n-1.  swizzle: 0 none, 1 32B, 2 64B, 3 128B.
TensorMap tensor_map_nd_bf16(const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                             int swizzle);

inline int num_sms() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (n[dev] == 0) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev];
}

// B200FW_BATCH_INVARIANT=1: products and paged decode attention take a row's sums in one order, however many rows or sequences
// there are beside it: nothing dealt to a cluster or cut into slices, which the dispatch does by how many there are.
inline bool batch_invariant() {
  static const bool on = [] {
    const char* e = std::getenv("B200FW_BATCH_INVARIANT");
    return e != nullptr && e[0] == '1';
  }();
  return on;
}

// Steps of few rows (decoding, single short examples) are chains of short kernels: the launch, barrier set-up and first copies
// of each are a large part of its time.  Up to this many rows a kernel is launched so that it may start before its
// predecessor has ended (see chain_wait).  Larger ones run long enough to hide it, and keep the ordinary order of
// launches, in which CTAs of one kernel never wait on an SM while another stream's kernel could use it.
constexpr int CHAIN_ROWS = 512;

// chained: allow the overlap described above; the kernel has to call chain_wait.  cluster_x, cluster_z: cluster shape (1: none).
template <typename... P, typename... A>
cudaError_t launch_chained(bool chained, void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, int cluster_x,
                           int cluster_z, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster_x * cluster_z > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n++].val.clusterDim.z = cluster_z;
  }
  if (chained) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace b2
