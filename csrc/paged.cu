// Paged KV-cache kernels: block-segment KV store (bf16 and fp8-e4m3 with one scale per block and kv
// head), gather / dequantise into contiguous bf16, paged decode attention with split-KV partitions
// and the exact log-sum-exp merge.
//
// Cache layout for one layer and one of {K, V}: [num_blocks, 16 tokens, Hkv, 128] (bf16 or fp8 bytes);
// scales [num_blocks, Hkv] fp32 (value = stored * scale).
#include <cuda_fp8.h>

#include "common.cuh"
#include "host.h"

namespace b2 {

constexpr int PAGE = 16;
constexpr int HD = 128;
constexpr float FP8_MAX = 448.f;

__device__ __forceinline__ float fp8_to_float(uint8_t v) {
  __nv_fp8_e4m3 t;
  t.__x = v;
  return static_cast<float>(t);
}
__device__ __forceinline__ uint8_t float_to_fp8(float v) {
  __nv_fp8_e4m3 t(v);
  return t.__x;
}

// ---------------------------------------------------------------------------------------------
// KV store.  A segment is a run of `count` consecutive new tokens (rows tok0.. of k / v) that land in
// one cache block starting at slot `off`: seg = {block, tok0, count, off}.  Grid (nseg, Hkv, 2) —
// z = 0 stores K, z = 1 stores V; 128 threads = one per head dimension.
// fp8: the block's scale only ever grows; when a new token raises it, the tokens already in the block
// are requantised by the same CTA (a block's tail is owned by one sequence, so no one else writes it).
// ---------------------------------------------------------------------------------------------
template <bool FP8>
__global__ void __launch_bounds__(128) kv_store_kernel(
    const __nv_bfloat16* k, const __nv_bfloat16* v, int ld_k, int ld_v,
    void* k_cache, void* v_cache, float* k_scale,
    float* v_scale, const int* segs, int Hkv) {
  __shared__ float red[4];
  chain_wait();
  chain_release();
  const int seg = blockIdx.x, h = blockIdx.y, which = blockIdx.z;
  const int block = segs[seg * 4 + 0], tok0 = segs[seg * 4 + 1], count = segs[seg * 4 + 2],
            off = segs[seg * 4 + 3];
  if (block < 0 || count <= 0) return;
  const __nv_bfloat16* src = which ? v : k;
  const int ld = which ? ld_v : ld_k;
  const int d = threadIdx.x;
  const size_t base = (static_cast<size_t>(block) * PAGE) * Hkv * HD + static_cast<size_t>(h) * HD + d;
  const size_t tok_stride = static_cast<size_t>(Hkv) * HD;
  if (!FP8) {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(which ? v_cache : k_cache);
    __nv_bfloat16 rows[PAGE];   // all loads before the first store: the compiler may not move one over the other
#pragma unroll
    for (int t = 0; t < PAGE; ++t)
      if (t < count) rows[t] = src[static_cast<size_t>(tok0 + t) * ld + h * HD + d];
#pragma unroll
    for (int t = 0; t < PAGE; ++t)
      if (t < count) dst[base + (off + t) * tok_stride] = rows[t];
    return;
  }
  uint8_t* dst = reinterpret_cast<uint8_t*>(which ? v_cache : k_cache);
  float* scale_p = (which ? v_scale : k_scale) + static_cast<size_t>(block) * Hkv + h;
  float vals[PAGE];
  float amax = 0.f;
  for (int t = 0; t < count; ++t) {
    vals[t] = __bfloat162float(src[static_cast<size_t>(tok0 + t) * ld + h * HD + d]);
    amax = fmaxf(amax, fabsf(vals[t]));
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
  const float old_scale = off > 0 ? *scale_p : 0.f;
  float new_scale = fmaxf(old_scale, amax / FP8_MAX);
  if (new_scale <= 0.f) new_scale = 1.f / FP8_MAX;
  if (off > 0 && new_scale > old_scale) {
    const float r = old_scale / new_scale;
    for (int t = 0; t < off; ++t) {
      const size_t a = base + t * tok_stride;
      dst[a] = float_to_fp8(fp8_to_float(dst[a]) * r);
    }
  }
  const float inv = 1.f / new_scale;
  for (int t = 0; t < count; ++t) dst[base + (off + t) * tok_stride] = float_to_fp8(vals[t] * inv);
  __syncthreads();
  if (threadIdx.x == 0) *scale_p = new_scale;
}

// ---------------------------------------------------------------------------------------------
// Gather cache rows into contiguous bf16 K / V [rows, Hkv*128]; slot[r] = block*16 + offset.
// ---------------------------------------------------------------------------------------------
template <bool FP8>
__global__ void kv_gather_kernel(const void* __restrict__ k_cache, const void* __restrict__ v_cache,
                                 const float* __restrict__ k_scale, const float* __restrict__ v_scale,
                                 const int* __restrict__ slot, __nv_bfloat16* __restrict__ k_out,
                                 __nv_bfloat16* __restrict__ v_out, int rows, int Hkv) {
  const int W = Hkv * HD;
  const long long total = static_cast<long long>(rows) * W;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(i / W), c = static_cast<int>(i % W);
    const int s = slot[r];
    const size_t a = static_cast<size_t>(s) * W + c;
    if (FP8) {
      const size_t sc = static_cast<size_t>(s / PAGE) * Hkv + c / HD;
      k_out[i] = __float2bfloat16(fp8_to_float(reinterpret_cast<const uint8_t*>(k_cache)[a]) * k_scale[sc]);
      v_out[i] = __float2bfloat16(fp8_to_float(reinterpret_cast<const uint8_t*>(v_cache)[a]) * v_scale[sc]);
    } else {
      k_out[i] = reinterpret_cast<const __nv_bfloat16*>(k_cache)[a];
      v_out[i] = reinterpret_cast<const __nv_bfloat16*>(v_cache)[a];
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Paged decode attention: one query token per sequence.  Grid (B, Hkv, parts of the context).
//
// Bound by the bytes of the cache.  With scalar FMAs it was not: every cache row cost G dot products, their shuffles over the
// lanes of the row and (fp8) a conversion per byte in every head group, 86 us for 98 MB of fp8 cache with four query
// heads per kv head (32 sequences of ~1500 tokens, 8 kv heads), and a single sequence kept 8 CTAs busy (25 us at 1024
// tokens).  Here both products run on the tensor cores (mma.m16n8k16: the query heads of one kv head are too few rows for
// a tcgen05 tile) and the parts of a context that a cluster of CTAs works through are merged over distributed shared
// memory, so the split needs neither a plan on the host nor a workspace nor a second kernel.
//
// A warp takes pages (16 tokens) in turn; its K and V rows arrive in a ring of its own by 16-byte cp.async copies.
//   scores:  A = the query heads, one per row (rows r and r + GP hold the same head), B = the page's keys.
//   output:  A = the probabilities, B = the page's values.  Probabilities keep 24 bits: p = hi + mid + lo in the 16-bit type,
//            and rows r, r + GP, r + 2 GP of A are those three parts of the same head, so the split costs no product of its
//            own up to four heads (GP = 8: a second one).  The rows of a head are added up once, at the end; where the first
//            is infinite (16-bit values may be), it alone counts.
// Contraction indices may be permuted freely, so both operands are read from shared memory 16 bytes per lane: lane
// (r = lane / 4, c = lane % 4) owns the dims of chunks c, c + 4, .. of key r, and dims 16 r .. 16 r + 15 of the values of
// tokens 2 c, 2 c + 1, 2 c + 8, 2 c + 9.  The chunk swizzle below makes both patterns free of bank conflicts.
// fp8 rows become fp16 (exact).  The page's key scale multiplies the score; its value scale, less its largest exponent
// so far (a power of two, divided out at the end), the probability, which carries a factor 2^14 to stay clear of
// fp16's subnormals.  Queries of fp8 caches are scaled by a power of two per head to lie in [2^13, 2^14) at most.
// ---------------------------------------------------------------------------------------------
constexpr int DEC_CHUNK = 64;   // partitions are multiples of this many tokens
constexpr int DEC_MAX_G = 8;
constexpr int DEC_MAX_CLUSTER = 8;
constexpr float DEC_LOG2E = 1.4426950408889634f;
constexpr float DEC_LN2 = 0.6931471805599453f;

template <bool FP8>
struct DecCfg {
  static constexpr int ROW = HD * (FP8 ? 1 : 2);      // bytes of a cache row
  static constexpr int CPR = ROW / 16;                // 16-byte chunks per row
  static constexpr int TILE = PAGE * ROW;             // one page of K or V
  static constexpr int STAGES = FP8 ? 4 : 3;
  static constexpr int RING = STAGES * 2 * TILE;      // per warp
  // chunk of row t is stored at chunk ^ swz(t): keys of two neighbouring tokens differ in bit 2, values of four tokens
  // two apart differ in the two bits that the two chunks of a quarter warp leave free
  static __device__ __forceinline__ int swz(int t) {
    const int b2 = ((t >> 2) ^ t) & 1, b1 = (t >> 1) & 1;
    return (b2 << 2) | (FP8 ? b1 << 1 : b1);
  }
};

template <bool FP8>
__device__ __forceinline__ void dec_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  if (FP8)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// two floats as halves (first one in the low half), and back
__device__ __forceinline__ uint32_t dec_pack(float x, float y) {
  const __half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float2 dec_unpack(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
// Part `part` of the pair (x, y): 0 the leading bits, 1 the leading ones of the rest, 2 what is left after both; none beyond.
// fp16 parts are rounded.  bf16 parts are cut off, 8 bits each: of a probability none is negative, and three are all of it.
template <bool FP8>
__device__ __forceinline__ uint32_t dec_part(float x, float y, int part) {
  if (!FP8) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (part > i) {
        x -= __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
        y -= __uint_as_float(__float_as_uint(y) & 0xFFFF0000u);
      }
    }
    return part > 2 ? 0u : __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632u);
  }
  uint32_t u = dec_pack(x, y);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (part > i) {
      const float2 f = dec_unpack(u);
      x -= f.x;
      y -= f.y;
      u = dec_pack(x, y);
    }
  }
  return part > 2 ? 0u : u;
}
// The last part where it has no rows of its own and is added to the first one's (eight heads).  A bf16 value may be infinite: the
// part is then not 0 unless the probability is, so that both rows' products are the same infinity.
template <bool FP8>
__device__ __forceinline__ uint32_t dec_last_part(float x, float y) {
  if (FP8) return dec_part<FP8>(x, y, 2);
  const uint32_t u = dec_part<FP8>(x, y, 2);
  const float2 f = unpack_bf16x2(u);
  const float tiny = 7.888609e-31f;   // 2^-100
  return __byte_perm(__float_as_uint(fmaxf(f.x, fminf(x, tiny))), __float_as_uint(fmaxf(f.y, fminf(y, tiny))), 0x7632u);
}
// two e4m3 bytes (the low half of w) as two halves
__device__ __forceinline__ uint32_t dec_fp8x2(uint32_t w) {
  const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(w & 0xFFFFu), __NV_E4M3);
  return static_cast<uint32_t>(r.x) | (static_cast<uint32_t>(r.y) << 16);
}
__device__ __forceinline__ uint4 dec_lds(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float dec_ld_cluster(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}
__device__ __forceinline__ void dec_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// GP: query heads per kv head, rounded up to a power of two.  clustered: the CTAs along z are one cluster and share a context;
// otherwise CTA z takes tokens [z * partition, (z + 1) * partition) and, with several, writes its partial result.
template <bool FP8, int GP, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) paged_decode_kernel(
    const __nv_bfloat16* __restrict__ q, const void* __restrict__ k_cache, const void* __restrict__ v_cache,
    const float* __restrict__ k_scale, const float* __restrict__ v_scale,
    const int* __restrict__ block_tables, const int* __restrict__ context_lens, int max_blocks,
    __nv_bfloat16* __restrict__ out, float* __restrict__ part_o, float* __restrict__ part_ml, int Hq, int Hkv,
    int partition, float scale, int clustered) {
  using Cfg = DecCfg<FP8>;
  extern __shared__ __align__(128) uint8_t dec_ring[];   // [warp][stage][K | V][16 rows]
  __shared__ float sO[GP][HD], sM[GP], sL[GP];
  const int G = Hq / Hkv;
  const int b = blockIdx.x, kvh = blockIdx.y, z = blockIdx.z, nz = gridDim.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, c = lane & 3;
  // The query, the first page numbers (a context that is not split starts at page 0) and the context's length are requested
  // together: one after the other their latencies are most of what a short context takes.
  const int* table = block_tables + static_cast<size_t>(b) * max_blocks;
  int my_block = nz == 1 && warp + WARPS * lane < max_blocks ? table[warp + WARPS * lane] : 0;
  uint32_t qa[16];   // the query head of rows r and r + 8 (both r % GP), in the order of the lane's key chunks
  {
    const int g = r % GP;
    const __nv_bfloat16* qp = q + (static_cast<size_t>(b) * Hq + kvh * G + g) * HD;
    const bool aligned = (reinterpret_cast<uintptr_t>(q) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // bf16 rows: chunk c + 4 i is 8 dims; fp8 rows: chunk c + 4 (i / 2) is 16 dims, two vectors
      const int v = FP8 ? (c + 4 * (i >> 1)) * 2 + (i & 1) : c + 4 * i;
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (g < G) {
        if (aligned) {
          w = *reinterpret_cast<const uint4*>(qp + 8 * v);
        } else {
          const unsigned short* h = reinterpret_cast<const unsigned short*>(qp + 8 * v);
          w = make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
        }
      }
      qa[4 * i] = w.x;
      qa[4 * i + 1] = w.y;
      qa[4 * i + 2] = w.z;
      qa[4 * i + 3] = w.w;
    }
  }
  int ctx = context_lens[b], t_begin, t_end;
  if (clustered) {
    ctx = min(ctx, partition);
    const int per = ((ctx + PAGE - 1) / PAGE + nz - 1) / nz * PAGE;
    t_begin = min(z * per, ctx);
    t_end = min(t_begin + per, ctx);
  } else {
    t_begin = z * partition;
    t_end = min(ctx, t_begin + partition);
  }
  const int tiles = t_end > t_begin ? (t_end - t_begin + PAGE - 1) / PAGE : 0;
  table += t_begin / PAGE;
  const size_t tok_stride = static_cast<size_t>(Hkv) * Cfg::ROW;
  const uint8_t* kc = static_cast<const uint8_t*>(k_cache) + static_cast<size_t>(kvh) * Cfg::ROW;
  const uint8_t* vc = static_cast<const uint8_t*>(v_cache) + static_cast<size_t>(kvh) * Cfg::ROW;
  const uint32_t ring = smem_u32(dec_ring) + warp * Cfg::RING;

  // copies of this warp's i-th page (tile warp + 4 i); the table entries of 32 pages are read together
  auto issue = [&](int i) {
    const int tile = warp + WARPS * i;
    if ((i & 31) == 0 && (i > 0 || nz > 1)) {
      const int ahead = tile + WARPS * lane;
      my_block = ahead < tiles ? table[ahead] : 0;
    }
    const int blk = __shfl_sync(0xffffffffu, my_block, i & 31);
    if (tile < tiles) {
      const uint32_t dst0 = ring + (i % Cfg::STAGES) * (2 * Cfg::TILE);
      const size_t page = static_cast<size_t>(blk) * PAGE * tok_stride;
#pragma unroll
      for (int u = 0; u < PAGE * Cfg::CPR / 32; ++u) {
        const int row = (u * 32 + lane) / Cfg::CPR, ch = lane % Cfg::CPR;
        const bool valid = t_begin + tile * PAGE + row < t_end;   // rows past the end become zeros
        const size_t src = page + (valid ? row : 0) * tok_stride + ch * 16;
        const uint32_t dst = dst0 + row * Cfg::ROW + ((ch ^ Cfg::swz(row)) << 4);
        const int bytes = valid ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(kc + src), "r"(bytes) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + Cfg::TILE), "l"(vc + src), "r"(bytes) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // one group per page, empty ones included
  };
#pragma unroll
  for (int i = 0; i < Cfg::STAGES - 1; ++i) issue(i);

  float qscale = scale * DEC_LOG2E;
  {
    if (FP8) {
      float amax = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 f = unpack_bf16x2(qa[i]);
        amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
      }
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      const int e = min(max(static_cast<int>(__float_as_uint(amax) >> 23), 127 - 100), 254);   // biased exponent
      const float to = __uint_as_float(static_cast<uint32_t>(127 + 13 + 127 - e) << 23);             // 2^(13 - (e - 127))
      qscale *= __uint_as_float(static_cast<uint32_t>(e - 13) << 23);                               // its reciprocal
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float2 f = unpack_bf16x2(qa[i]);
        qa[i] = dec_pack(f.x * to, f.y * to);
      }
    }
  }
  const int part_a = r / GP, part_b = part_a + 8 / GP;
  float acc[16][4];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
  float m = -INFINITY, l = 0.f, my_ks = 1.f, my_vs = 1.f;
  // fp8: largest biased exponent of the value scales so far (acc is scaled by its inverse).  It starts where 2^14 times the
  // inverse is still finite and the last factor, 2^(ev - 127) / 2^14, still normal: a page may have the scale 0.
  int ev = 16;

  for (int i = 0; warp + WARPS * i < tiles; ++i) {
    issue(i + Cfg::STAGES - 1);
    float ks = 1.f, vs = 1.f;
    if (FP8) {
      if ((i & 31) == 0) {
        const int ahead = warp + WARPS * (i + lane);
        if (ahead < tiles) {
          const size_t at = static_cast<size_t>(table[ahead]) * Hkv + kvh;
          my_ks = k_scale[at];
          my_vs = v_scale[at];
        }
      }
      ks = __shfl_sync(0xffffffffu, my_ks, i & 31);
      vs = __shfl_sync(0xffffffffu, my_vs, i & 31);
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(Cfg::STAGES - 1) : "memory");
    __syncwarp();
    const uint32_t kt = ring + (i % Cfg::STAGES) * (2 * Cfg::TILE), vt = kt + Cfg::TILE;
    const int left = t_end - t_begin - (warp + WARPS * i) * PAGE;   // valid tokens of the page, from 1
    // ---- scores of tokens 2c, 2c+1 (s[0], s[1]) and 2c+8, 2c+9 (s[2], s[3])
    float s[4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      const int t = nt * 8 + r;
#pragma unroll
      for (int u = 0; u < Cfg::CPR / 4; ++u) {
        const uint4 w4 = dec_lds(kt + t * Cfg::ROW + (((c + 4 * u) ^ Cfg::swz(t)) << 4));
        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
        if (FP8) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int j = 4 * u + k;
            dec_mma<FP8>(d, qa[2 * j], qa[2 * j], qa[2 * j + 1], qa[2 * j + 1], dec_fp8x2(w[k]), dec_fp8x2(w[k] >> 16));
          }
        } else {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int j = 2 * u + k;
            dec_mma<FP8>(d, qa[2 * j], qa[2 * j], qa[2 * j + 1], qa[2 * j + 1], w[2 * k], w[2 * k + 1]);
          }
        }
      }
      s[2 * nt] = d[0];
      s[2 * nt + 1] = d[1];
    }
    const float f = qscale * ks;
    float mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int t = 2 * c + (k & 1) + (k >> 1) * 8;
      s[k] = t < left ? s[k] * f : -INFINITY;
      mx = fmaxf(mx, s[k]);
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx);
    float back = 1.f;
    if (FP8) {
      const int e = min(max(static_cast<int>((__float_as_uint(vs) >> 23) & 255u), ev), 253);
      back = e - ev > 126 ? 0.f : __uint_as_float(static_cast<uint32_t>(127 - (e - ev)) << 23);
      ev = e;
      vs *= 16384.f * __uint_as_float(static_cast<uint32_t>(254 - e) << 23);
    }
    if (__any_sync(0xffffffffu, mn != m || back != 1.f)) {
      const float alpha = mn == -INFINITY ? 0.f : fast_exp2(m - mn);
      l *= alpha;
#pragma unroll
      for (int j = 0; j < 16; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[j][k] *= alpha * back;
      m = mn;
    }
    const float base = mn == -INFINITY ? 0.f : mn;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s[k] = fast_exp2(s[k] - base);
      l += s[k];
      s[k] *= vs;
    }
    const uint32_t a0 = dec_part<FP8>(s[0], s[1], part_a), a2 = dec_part<FP8>(s[2], s[3], part_a);
    const uint32_t a1 = GP >= 4 ? dec_part<FP8>(s[0], s[1], part_b) : 0u, a3 = GP >= 4 ? dec_part<FP8>(s[2], s[3], part_b) : 0u;
    const uint32_t x0 = GP == 8 ? dec_last_part<FP8>(s[0], s[1]) : 0u, x2 = GP == 8 ? dec_last_part<FP8>(s[2], s[3]) : 0u;
    // ---- output dims 16 n + j of n-tile j
#pragma unroll
    for (int h = 0; h < Cfg::CPR / 8; ++h) {
      uint32_t w[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = 2 * c + (k & 1) + (k >> 1) * 8;
        const uint4 w4 = dec_lds(vt + t * Cfg::ROW + (((r * (Cfg::CPR / 8) + h) ^ Cfg::swz(t)) << 4));
        w[k][0] = w4.x;
        w[k][1] = w4.y;
        w[k][2] = w4.z;
        w[k][3] = w4.w;
      }
#pragma unroll
      for (int jj = 0; jj < (FP8 ? 16 : 8); ++jj) {
        uint32_t b0, b1;
        if (FP8) {   // byte jj of tokens 2c and 2c+1, of 2c+8 and 2c+9
          const uint32_t pick = (jj & 3) | ((4 + (jj & 3)) << 4);
          b0 = dec_fp8x2(__byte_perm(w[0][jj >> 2], w[1][jj >> 2], pick));
          b1 = dec_fp8x2(__byte_perm(w[2][jj >> 2], w[3][jj >> 2], pick));
        } else {     // half jj
          const uint32_t pick = (jj & 1) ? 0x7632u : 0x5410u;
          b0 = __byte_perm(w[0][jj >> 1], w[1][jj >> 1], pick);
          b1 = __byte_perm(w[2][jj >> 1], w[3][jj >> 1], pick);
        }
        const int j = h * 8 + jj;
        dec_mma<FP8>(acc[j], a0, a1, a2, a3, b0, b1);
        if (GP == 8) dec_mma<FP8>(acc[j], x0, 0u, x2, 0u, b0, b1);
      }
    }
    __syncwarp();   // every lane has read the stage before its next copies are issued
  }
  chain_release();
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();

  // ---- the parts of a head: rows r and r + 8, then rows GP apart; then the warps through shared memory
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  const float unit = FP8 ? __uint_as_float(static_cast<uint32_t>(ev) << 23) * (1.f / 16384.f) : 1.f;
  // per warp [GP][PITCH], channel 16 n + j at 8 j + n (what the lanes of a row hold is then adjacent), then maxima and sums
  constexpr int PITCH = HD + 8;
  float* wo = reinterpret_cast<float*>(dec_ring + warp * Cfg::RING);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float o0 = acc[j][0] + acc[j][2], o1 = acc[j][1] + acc[j][3];
#pragma unroll
    for (int d = 16; d >= 4 * GP; d >>= 1) {
      o0 += __shfl_xor_sync(0xffffffffu, o0, d);
      o1 += __shfl_xor_sync(0xffffffffu, o1, d);
    }
    if (r < GP) {   // this lane's row r is the high part of head r: where it is infinite, the other parts are 0 * inf or -inf
      o0 = fabsf(acc[j][0]) < INFINITY ? o0 : acc[j][0];
      o1 = fabsf(acc[j][1]) < INFINITY ? o1 : acc[j][1];
      *reinterpret_cast<float2*>(wo + r * PITCH + 8 * j + 2 * c) = make_float2(o0 * unit, o1 * unit);
    }
  }
  if (r < GP && c == 0) {
    wo[GP * PITCH + r] = m;
    wo[GP * PITCH + GP + r] = l;
  }
  __syncthreads();
  for (int e = tid; e < G * HD; e += (WARPS * 32)) {
    const int g = e / HD, at = e % HD, d = (at & 7) * 16 + (at >> 3);
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) M = fmaxf(M, reinterpret_cast<const float*>(dec_ring + w * Cfg::RING)[GP * PITCH + g]);
    float L = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float* p = reinterpret_cast<const float*>(dec_ring + w * Cfg::RING);
      const float mw = p[GP * PITCH + g];
      const float wgt = mw == -INFINITY ? 0.f : fast_exp2(mw - M);
      L += p[GP * PITCH + GP + g] * wgt;
      o += p[g * PITCH + at] * wgt;
    }
    const int head = kvh * G + g;
    if (nz == 1) {
      out[(static_cast<size_t>(b) * Hq + head) * HD + d] = __float2bfloat16(L > 0.f ? o / L : 0.f);
    } else if (clustered) {
      sO[g][d] = o;
      if (d == 0) {
        sM[g] = M;
        sL[g] = L;
      }
    } else {
      part_o[((static_cast<size_t>(b) * Hq + head) * nz + z) * HD + d] = o;
      if (d == 0) {
        float* ml = part_ml + ((static_cast<size_t>(b) * Hq + head) * nz + z) * 2;
        ml[0] = M * DEC_LN2;   // natural-log domain for the merge kernel
        ml[1] = L;
      }
    }
  }
  if (!clustered || nz == 1) return;
  // ---- the heads' channels are dealt to the CTAs, which add up the cluster's parts
  dec_cluster_sync();
  for (int e = z * (WARPS * 32) + tid; e < G * HD; e += nz * (WARPS * 32)) {
    const int g = e / HD, d = e % HD;
    float M = -INFINITY, mz[DEC_MAX_CLUSTER], lz[DEC_MAX_CLUSTER], oz[DEC_MAX_CLUSTER], L = 0.f, o = 0.f;
#pragma unroll
    for (int k = 0; k < DEC_MAX_CLUSTER; ++k) {
      mz[k] = k < nz ? dec_ld_cluster(smem_u32(&sM[g]), k) : -INFINITY;
      lz[k] = k < nz ? dec_ld_cluster(smem_u32(&sL[g]), k) : 0.f;
      oz[k] = k < nz ? dec_ld_cluster(smem_u32(&sO[g][d]), k) : 0.f;
      M = fmaxf(M, mz[k]);
    }
#pragma unroll
    for (int k = 0; k < DEC_MAX_CLUSTER; ++k) {
      const float wgt = mz[k] == -INFINITY ? 0.f : fast_exp2(mz[k] - M);
      L += lz[k] * wgt;
      o += oz[k] * wgt;
    }
    out[(static_cast<size_t>(b) * Hq + kvh * G + g) * HD + d] = __float2bfloat16(L > 0.f ? o / L : 0.f);
  }
  dec_cluster_sync();   // nobody leaves while its shared memory is read
}

// Exact merge of split-KV partials: out = sum_i acc_i e^{m_i - M} / sum_i l_i e^{m_i - M}.
__global__ void __launch_bounds__(HD) paged_merge_kernel(const float* __restrict__ part_o,
                                                        const float* __restrict__ part_ml,
                                                        __nv_bfloat16* __restrict__ out,
                                                        float* __restrict__ lse_out, int nsplit) {
  const size_t bh = blockIdx.x;
  const int d = threadIdx.x;
  float M = -INFINITY;
  for (int i = 0; i < nsplit; ++i) M = fmaxf(M, part_ml[(bh * nsplit + i) * 2]);
  float L = 0.f, o = 0.f;
  for (int i = 0; i < nsplit; ++i) {
    const float m = part_ml[(bh * nsplit + i) * 2], l = part_ml[(bh * nsplit + i) * 2 + 1];
    if (m == -INFINITY) continue;
    const float w = __expf(m - M);
    L += l * w;
    o += part_o[(bh * nsplit + i) * HD + d] * w;
  }
  out[bh * HD + d] = __float2bfloat16(L > 0.f ? o / L : 0.f);
  if (lse_out && d == 0) lse_out[bh] = M + __logf(L);
}

}  // namespace b2

using namespace b2;

#define B2_LAUNCH_CHECK(name)                                        \
  do {                                                               \
    cudaError_t e_ = cudaGetLastError();                             \
    if (e_ != cudaSuccess) {                                         \
      set_error(name " launch failed: %s", cudaGetErrorString(e_)); \
      return 4;                                                      \
    }                                                                \
  } while (0)

B2_EXPORT int b2_kv_store(const void* k, const void* v, int ld_k, int ld_v, void* k_cache, void* v_cache,
                          float* k_scale, float* v_scale, const int* segs, int nseg, int Hkv, int head_dim,
                          int fp8, void* stream) {
  b2::ensure_thread_context();
  if (head_dim != HD) { set_error("kv_store: head_dim must be 128"); return 10; }
  if (nseg <= 0) return 0;
  dim3 grid(nseg, Hkv, 2);
  if (fp8)
    launch_chained(nseg <= CHAIN_ROWS, kv_store_kernel<true>, grid, 128, 0, static_cast<cudaStream_t>(stream), 1, 1,
        static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), ld_k, ld_v, k_cache, v_cache,
        k_scale, v_scale, segs, Hkv);
  else
    launch_chained(nseg <= CHAIN_ROWS, kv_store_kernel<false>, grid, 128, 0, static_cast<cudaStream_t>(stream), 1, 1,
        static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v), ld_k, ld_v, k_cache, v_cache,
        k_scale, v_scale, segs, Hkv);
  B2_LAUNCH_CHECK("kv_store");
  return 0;
}

B2_EXPORT int b2_kv_gather(const void* k_cache, const void* v_cache, const float* k_scale, const float* v_scale,
                           const int* slot, void* k_out, void* v_out, int rows, int Hkv, int head_dim, int fp8,
                           void* stream) {
  b2::ensure_thread_context();
  if (head_dim != HD) { set_error("kv_gather: head_dim must be 128"); return 10; }
  if (rows <= 0) return 0;
  const long long total = static_cast<long long>(rows) * Hkv * HD;
  long long blocks = (total + 255) / 256;
  const long long cap = static_cast<long long>(num_sms()) * 16;
  if (blocks > cap) blocks = cap;
  if (fp8)
    kv_gather_kernel<true><<<static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        k_cache, v_cache, k_scale, v_scale, slot, static_cast<__nv_bfloat16*>(k_out),
        static_cast<__nv_bfloat16*>(v_out), rows, Hkv);
  else
    kv_gather_kernel<false><<<static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        k_cache, v_cache, k_scale, v_scale, slot, static_cast<__nv_bfloat16*>(k_out),
        static_cast<__nv_bfloat16*>(v_out), rows, Hkv);
  B2_LAUNCH_CHECK("kv_gather");
  return 0;
}

// partition: tokens per split (multiple of 64); nsplit = ceil(max_ctx / partition) chosen by the caller.
// part_o: fp32 [B, Hq, nsplit, 128]; part_ml: fp32 [B, Hq, nsplit, 2] (only read when nsplit > 1).
B2_EXPORT int b2_paged_decode(const void* q, const void* k_cache, const void* v_cache, const float* k_scale,
                              const float* v_scale, const int* block_tables, const int* context_lens,
                              int max_blocks, void* out, float* part_o, float* part_ml, float* lse, int B,
                              int Hq, int Hkv, int head_dim, int partition, int nsplit, float scale, int fp8,
                              void* stream_) {
  b2::ensure_thread_context();
  if (head_dim != HD || Hq % Hkv != 0 || Hq / Hkv > DEC_MAX_G || partition % DEC_CHUNK != 0 || nsplit < 1) {
    set_error("paged_decode: head_dim 128, Hq/Hkv <= 8, partition %% 64 == 0 required");
    return 10;
  }
  if (B <= 0) return 0;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int G = Hq / Hkv, GP = G > 4 ? 8 : G > 2 ? 4 : G;
  // Without a split from the caller, the CTAs of a cluster share a context: as many (up to 8) as keep the grid within two CTAs
  // per SM, i.e. in one wave, and no more than the table has pieces of 64 tokens.  Clusters of 1 / 2 / 4 / 8, us: 8 (sequence, kv
  // head) pairs of 1024 tokens 12.9 / 9.6 / 7.6 / 6.3; 64 pairs of up to 8192 80.3 / 45.5 / 41.8 / 45.5; 256 pairs of up to 2000
  // 41.3 / 48.2 / 58.5 / 87.4.
  int cluster = 1;
  if (nsplit == 1 && !batch_invariant())
    while (cluster < DEC_MAX_CLUSTER && static_cast<long long>(B) * Hkv * cluster * 2 <= 2LL * num_sms() && cluster * 2 * (DEC_CHUNK / PAGE) <= max_blocks)
      cluster *= 2;
  // Two warps per CTA where there are many pairs anyway: CTAs of short contexts come and go faster.  256 sequences, 8 kv
  // heads, two / four warps, us: 128 tokens 31 / 39, 1024 tokens 130 / 125; 32 sequences of 2000 tokens 53 / 41.
  const int warps = static_cast<long long>(B) * Hkv >= 8LL * num_sms() && !batch_invariant() ? 2 : 4;
#define B2_DECODE_LAUNCH_W(F8, GPV, WV)                                                                                   \
  do {                                                                                                              \
    auto kern = paged_decode_kernel<F8, GPV, WV>;                                                                   \
    static bool attr_set[64] = {};                                                                                  \
    int dev = 0;                                                                                                    \
    cudaGetDevice(&dev);                                                                                            \
    if (!attr_set[dev & 63]) {                                                                                      \
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, WV * DecCfg<F8>::RING);                \
      attr_set[dev & 63] = true;                                                                                    \
    }                                                                                                               \
    /* not chained: waiting CTAs of this kernel hold shared memory that the products before it could use */ \
    launch_chained(false, kern, dim3(B, Hkv, nsplit == 1 ? cluster : nsplit), WV * 32, WV * DecCfg<F8>::RING, stream, 1, \
                   cluster, static_cast<const __nv_bfloat16*>(q), k_cache, v_cache, k_scale, v_scale, block_tables,  \
                   context_lens, max_blocks, static_cast<__nv_bfloat16*>(out), part_o, part_ml, Hq, Hkv, partition, \
                   scale, nsplit == 1 ? 1 : 0);                                                                     \
  } while (0)
#define B2_DECODE_LAUNCH(F8, GPV)                     \
  do {                                                \
    if (warps == 2) B2_DECODE_LAUNCH_W(F8, GPV, 2);   \
    else B2_DECODE_LAUNCH_W(F8, GPV, 4);              \
  } while (0)
#define B2_DECODE_GROUP(F8)                       \
  do {                                            \
    if (GP == 8) B2_DECODE_LAUNCH(F8, 8);         \
    else if (GP == 4) B2_DECODE_LAUNCH(F8, 4);    \
    else if (GP == 2) B2_DECODE_LAUNCH(F8, 2);    \
    else B2_DECODE_LAUNCH(F8, 1);                 \
  } while (0)
  if (fp8) B2_DECODE_GROUP(true);
  else B2_DECODE_GROUP(false);
#undef B2_DECODE_GROUP
#undef B2_DECODE_LAUNCH
#undef B2_DECODE_LAUNCH_W
  B2_LAUNCH_CHECK("paged_decode");
  if (nsplit > 1) {
    paged_merge_kernel<<<B * Hq, HD, 0, stream>>>(part_o, part_ml, static_cast<__nv_bfloat16*>(out), lse, nsplit);
    B2_LAUNCH_CHECK("paged_merge");
  }
  return 0;
}
