// Row movement of the mixture-of-experts block around its grouped GEMMs: token rows into the expert-grouped matrix,
// weighted expert rows back to their tokens, and the two backward passes.
//
// `row[t * k + j]` is the row of the grouped matrix that holds token t's j-th expert (expert layout, router_ops.cu);
// every expert's segment ends with up to tile_m - 1 padding rows.
//
// All four are bound by HBM: one block per token reads or writes k rows of H bf16 in 16-byte pieces.  They replace
// repeat_interleave + index_copy + index + fp32 multiply + sum and their autograd counterparts (an index_put with
// accumulation among them).  32,768 routed rows of 2048, all passes together, weights and GEMMs aside:
// 1.97 ms before, 0.15 ms now.
#include "ptx.cuh"

namespace cvb {

constexpr int MOE_THREADS = 256;
constexpr int MOE_MAX_K = 32;

__device__ __forceinline__ void moe_unpack(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = __bfloat1622float2(h[i]);
    f[2 * i] = v.x;
    f[2 * i + 1] = v.y;
  }
}
__device__ __forceinline__ uint4 moe_pack(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]);
  u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]);
  u.w = pack_bf16x2(f[6], f[7]);
  return u;
}

// xp[row[t, j]] = x[t]
__global__ void __launch_bounds__(MOE_THREADS)
moe_dispatch_kernel(const uint4* __restrict__ x, const long long* __restrict__ row, uint4* __restrict__ xp, int k,
                    int chunks) {
  const long long t = blockIdx.x;
  for (int c = threadIdx.x; c < chunks; c += MOE_THREADS) {
    const uint4 v = x[t * chunks + c];
    for (int j = 0; j < k; ++j) xp[row[t * k + j] * chunks + c] = v;
  }
}

// zeroes the padding rows of every expert's segment (the weight-gradient GEMM's K range runs over them)
__global__ void __launch_bounds__(MOE_THREADS)
moe_zero_pad_kernel(const int* __restrict__ offsets, const int* __restrict__ totals, uint4* __restrict__ m, int chunks) {
  const int e = blockIdx.x;
  const long long first = static_cast<long long>(offsets[e] + totals[e]) * chunks;
  const long long last = static_cast<long long>(offsets[e + 1]) * chunks;
  for (long long i = first + static_cast<long long>(blockIdx.y) * MOE_THREADS + threadIdx.x; i < last;
       i += static_cast<long long>(gridDim.y) * MOE_THREADS)
    m[i] = make_uint4(0u, 0u, 0u, 0u);
}

// out[t] = sum_j w[t, j] * y[row[t, j]]   (w = nullptr: plain sum), fp32 accumulation, one rounding
__global__ void __launch_bounds__(MOE_THREADS)
moe_combine_kernel(const uint4* __restrict__ y, const long long* __restrict__ row, const float* __restrict__ w,
                   uint4* __restrict__ out, int k, int chunks) {
  const long long t = blockIdx.x;
  for (int c = threadIdx.x; c < chunks; c += MOE_THREADS) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll 8
    for (int j = 0; j < k; ++j) {
      float v[8];
      moe_unpack(y[row[t * k + j] * chunks + c], v);
      const float wj = w ? w[t * k + j] : 1.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += wj * v[i];
    }
    out[t * chunks + c] = moe_pack(acc);
  }
}

// dy[row[t, j]] = w[t, j] * dout[t];  dw[t, j] = <dout[t], y[row[t, j]]>
__global__ void __launch_bounds__(MOE_THREADS)
moe_combine_bwd_kernel(const uint4* __restrict__ dout, const uint4* __restrict__ y, const long long* __restrict__ row,
                       const float* __restrict__ w, uint4* __restrict__ dy, float* __restrict__ dw, int k, int chunks) {
  __shared__ float part[MOE_MAX_K][MOE_THREADS / 32];
  const long long t = blockIdx.x;
  const int warp = threadIdx.x >> 5;
  for (int j = 0; j < k; ++j) {
    const long long r = row[t * k + j];
    const float wj = w[t * k + j];
    float dot = 0.f;
    for (int c = threadIdx.x; c < chunks; c += MOE_THREADS) {
      float g[8], v[8];
      moe_unpack(dout[t * chunks + c], g);
      moe_unpack(y[r * chunks + c], v);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        dot += g[i] * v[i];
        g[i] *= wj;
      }
      dy[r * chunks + c] = moe_pack(g);
    }
    dot = warp_sum(dot);
    if ((threadIdx.x & 31) == 0) part[j][warp] = dot;
  }
  __syncthreads();
  if (threadIdx.x < k) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < MOE_THREADS / 32; ++i) s += part[threadIdx.x][i];
    dw[t * k + threadIdx.x] = s;
  }
}

static bool moe_bad(const void* a, const void* b, long long T, int k, int H) {
  return T > 0x7fffffffLL || k <= 0 || k > MOE_MAX_K || H <= 0 || H % 8 != 0 ||
         (reinterpret_cast<uintptr_t>(a) & 15) != 0 || (reinterpret_cast<uintptr_t>(b) & 15) != 0;
}
static void moe_zero_pad(const int* offsets, const int* totals, void* m, int E, int H, cudaStream_t st) {
  moe_zero_pad_kernel<<<dim3(E, 8), MOE_THREADS, 0, st>>>(offsets, totals, static_cast<uint4*>(m), H / 8);
}

}  // namespace cvb

using namespace cvb;

// x bf16 [T, H], row int64 [T, k] with every entry inside the grouped matrix, xp bf16 [m_pad, H]; offsets int32 [E + 1]
// and totals int32 [E] of the expert layout: padding rows are zeroed, rows of unused tiles are left as they are.
extern "C" int cvb_moe_dispatch(const void* x, const long long* row, void* xp, const int* offsets, const int* totals,
                                long long T, int k, int H, int E, void* stream) {
  if (T <= 0) return 0;
  if (moe_bad(x, xp, T, k, H) || E <= 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  moe_dispatch_kernel<<<static_cast<unsigned>(T), MOE_THREADS, 0, st>>>(static_cast<const uint4*>(x), row,
                                                                        static_cast<uint4*>(xp), k, H / 8);
  moe_zero_pad(offsets, totals, xp, E, H, st);
  return static_cast<int>(cudaGetLastError());
}

// y bf16 [m_pad, H]; w fp32 [T, k] or NULL (plain sum: the dispatch's backward); out bf16 [T, H]
extern "C" int cvb_moe_combine(const void* y, const long long* row, const float* w, void* out, long long T, int k,
                               int H, void* stream) {
  if (T <= 0) return 0;
  if (moe_bad(y, out, T, k, H)) return -1;
  moe_combine_kernel<<<static_cast<unsigned>(T), MOE_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(y), row, w, static_cast<uint4*>(out), k, H / 8);
  return static_cast<int>(cudaGetLastError());
}

// dout bf16 [T, H]; y as in the forward; dy bf16 [m_pad, H] (padding rows zeroed); dw fp32 [T, k]
extern "C" int cvb_moe_combine_bwd(const void* dout, const void* y, const long long* row, const float* w, void* dy,
                                   float* dw, const int* offsets, const int* totals, long long T, int k, int H, int E,
                                   void* stream) {
  if (T <= 0) return 0;
  if (moe_bad(dout, dy, T, k, H) || (reinterpret_cast<uintptr_t>(y) & 15) || E <= 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  moe_combine_bwd_kernel<<<static_cast<unsigned>(T), MOE_THREADS, 0, st>>>(
      static_cast<const uint4*>(dout), static_cast<const uint4*>(y), row, w, static_cast<uint4*>(dy), dw, k, H / 8);
  moe_zero_pad(offsets, totals, dy, E, H, st);
  return static_cast<int>(cudaGetLastError());
}
