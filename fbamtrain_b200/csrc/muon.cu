// The element-wise part of a Muon step around the Newton–Schulz products: momentum and cast, normalisation, update.
//
// Bound by DRAM.  As separate tensor operations (cast of the gradient, decay and add of the momentum, Nesterov
// combination, cast, cast back, norm, division, cast; scale, decay, add, cast into the parameter) one step of a
// 4096 x 2048 matrix moves about 60 bytes per element in sixteen launches; the three kernels move 28, with fp32 gradient and
// parameter (4 + 8 + 2, 2 + 2, 2 + 8) as with 16-bit ones and a master (2 + 8 + 2, 2 + 2, 2 + 8 + 2).  The one-billion-parameter model with two action blocks: 95.3 -> 87.3 ms of GPU time per
// step, 1315 -> 924 launches (with the affine terms of the iterations moved into the GEMM epilogue).
//
// Sums of squares go through per-block partial sums that every block of the next kernel adds in the same order: no
// atomics, so ranks that run the same step on the same values get the same bits.
//
// Algorithm: the reference's Muon (reference: src/optimizers.cpp:825-1434).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 592;  // partial sums of one matrix

__device__ __forceinline__ float to_f(float x) { return x; }
__device__ __forceinline__ float to_f(__nv_bfloat16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float to_f(__half x) { return __half2float(x); }
__device__ __forceinline__ void from_f(float v, float& o) { o = v; }
__device__ __forceinline__ void from_f(float v, __nv_bfloat16& o) { o = __float2bfloat16(v); }
__device__ __forceinline__ void from_f(float v, __half& o) { o = __float2half_rn(v); }

template <typename T>
struct alignas(4 * sizeof(T)) Four { T v[4]; };

// Sum over the block in a fixed order; valid in every thread.
__device__ __forceinline__ float block_sum(float v) {
  __shared__ float s[kThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.0f;
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) t += s[i];
  return t;
}

// buf = mu * buf + nu * g;  x = bf16(nesterov ? nu * g + mu * buf : buf);  partial[block] = sum of x^2.
// nu = 1 - mu comes from the host, rounded once: 1.0f - (float)mu carries the rounding of mu, which is a relative error of
// 2.4e-7 of every update at mu = 0.95 and 1.3e-5 at 0.999, always to the same side, in a buffer that is kept.
// n is a multiple of 4 (rows and columns are multiples of 8).
template <typename G>
__global__ void __launch_bounds__(kThreads) muon_momentum_kernel(const G* __restrict__ grad, float* __restrict__ buf,
                                                                 __nv_bfloat16* __restrict__ x, float* __restrict__ partial,
                                                                 long long n, float mu, float nu, int nesterov) {
  float sum = 0.0f;
  const long long step = (long long)gridDim.x * kThreads * 4;
  for (long long i = ((long long)blockIdx.x * kThreads + threadIdx.x) * 4; i < n; i += step) {
    const Four<G> g = *reinterpret_cast<const Four<G>*>(grad + i);
    Four<float> b = *reinterpret_cast<const Four<float>*>(buf + i);
    Four<__nv_bfloat16> o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float gf = to_f(g.v[j]);
      b.v[j] = fmaf(nu, gf, mu * b.v[j]);
      o.v[j] = __float2bfloat16(nesterov ? fmaf(mu, b.v[j], nu * gf) : b.v[j]);
      const float r = __bfloat162float(o.v[j]);
      sum = fmaf(r, r, sum);
    }
    *reinterpret_cast<Four<float>*>(buf + i) = b;
    *reinterpret_cast<Four<__nv_bfloat16>*>(x + i) = o;
  }
  sum = block_sum(sum);
  if (threadIdx.x == 0) partial[blockIdx.x] = sum;
}

__device__ __forceinline__ float norm_of(const float* partial, int blocks) {
  float s = 0.0f;
  for (int i = threadIdx.x; i < blocks; i += kThreads) s += partial[i];
  return sqrtf(block_sum(s)) + 1e-7f;
}

// out = x / (norm + 1e-7), with rows and columns exchanged when TRANSPOSE (32 x 32 tiles through shared memory).
template <bool TRANSPOSE>
__global__ void __launch_bounds__(kThreads) muon_normalise_kernel(const __nv_bfloat16* __restrict__ x,
                                                                  const float* __restrict__ partial, int blocks,
                                                                  __nv_bfloat16* __restrict__ out, int rows, int cols) {
  const float norm = norm_of(partial, blocks);
  if (!TRANSPOSE) {
    const long long n = (long long)rows * cols, step = (long long)gridDim.x * kThreads * 4;
    for (long long i = ((long long)blockIdx.x * kThreads + threadIdx.x) * 4; i < n; i += step) {
      Four<__nv_bfloat16> v = *reinterpret_cast<const Four<__nv_bfloat16>*>(x + i);
#pragma unroll
      for (int j = 0; j < 4; ++j) v.v[j] = __float2bfloat16(__bfloat162float(v.v[j]) / norm);
      *reinterpret_cast<Four<__nv_bfloat16>*>(out + i) = v;
    }
  } else {
    __shared__ __nv_bfloat16 tile[32][34];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int tiles_c = (cols + 31) / 32;
    const long long tiles = (long long)((rows + 31) / 32) * tiles_c;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
      const int r0 = (int)(t / tiles_c) * 32, c0 = (int)(t % tiles_c) * 32;
      __syncthreads();
      for (int j = ty; j < 32; j += 8)
        if (r0 + j < rows && c0 + tx < cols)
          tile[j][tx] = __float2bfloat16(__bfloat162float(x[(long long)(r0 + j) * cols + c0 + tx]) / norm);
      __syncthreads();
      for (int j = ty; j < 32; j += 8)
        if (c0 + j < cols && r0 + tx < rows) out[(long long)(c0 + j) * rows + r0 + tx] = tile[tx][j];
    }
  }
}

// w = decay * w - lr * (scale * u);  param = rounded w.  u is (rows, cols), or (cols, rows) when TRANSPOSE.
template <bool TRANSPOSE, typename P>
__global__ void __launch_bounds__(kThreads) muon_apply_kernel(const __nv_bfloat16* __restrict__ u, float* __restrict__ w,
                                                              P* __restrict__ param, int rows, int cols, float decay,
                                                              float lr, float scale) {
  if (!TRANSPOSE) {
    const long long n = (long long)rows * cols, step = (long long)gridDim.x * kThreads * 4;
    for (long long i = ((long long)blockIdx.x * kThreads + threadIdx.x) * 4; i < n; i += step) {
      const Four<__nv_bfloat16> uv = *reinterpret_cast<const Four<__nv_bfloat16>*>(u + i);
      Four<float> wv = *reinterpret_cast<const Four<float>*>(w + i);
      Four<P> pv;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        wv.v[j] = fmaf(-lr, __bfloat162float(uv.v[j]) * scale, decay * wv.v[j]);
        from_f(wv.v[j], pv.v[j]);
      }
      *reinterpret_cast<Four<float>*>(w + i) = wv;
      if (param != nullptr) *reinterpret_cast<Four<P>*>(param + i) = pv;
    }
  } else {
    __shared__ __nv_bfloat16 tile[32][34];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int tiles_c = (cols + 31) / 32;
    const long long tiles = (long long)((rows + 31) / 32) * tiles_c;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
      const int r0 = (int)(t / tiles_c) * 32, c0 = (int)(t % tiles_c) * 32;
      __syncthreads();
      for (int j = ty; j < 32; j += 8)
        if (c0 + j < cols && r0 + tx < rows) tile[j][tx] = u[(long long)(c0 + j) * rows + r0 + tx];
      __syncthreads();
      for (int j = ty; j < 32; j += 8)
        if (r0 + j < rows && c0 + tx < cols) {
          const long long i = (long long)(r0 + j) * cols + c0 + tx;
          const float v = fmaf(-lr, __bfloat162float(tile[tx][j]) * scale, decay * w[i]);
          w[i] = v;
          if (param != nullptr) from_f(v, param[i]);
        }
    }
  }
}

unsigned grid_for(long long items) {
  const long long b = (items + kThreads * 4 - 1) / (kThreads * 4);
  return (unsigned)(b < kMaxBlocks ? b : kMaxBlocks);
}
bool aligned(const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }
int launched() { return cudaGetLastError() == cudaSuccess ? 0 : 5; }

}  // namespace

extern "C" {

// Number of partial sums the caller provides room for.
int fbam_muon_partials() { return kMaxBlocks; }

// type: 0 bf16, 1 half, 2 fp32 gradient (rows, cols) contiguous; buf: fp32, updated; x: bf16 scratch like grad; partial:
// fbam_muon_partials() floats; out: bf16 normalised update with the shorter side first (transposed when rows > cols).
// rows and cols are multiples of 8.  mu: momentum; nu: 1 - momentum.
int fbam_muon_prepare(const void* grad, int type, float* buf, void* x, float* partial, void* out, int rows, int cols,
                      float mu, float nu, int nesterov, void* stream) {
  if (rows < 8 || cols < 8 || rows % 8 || cols % 8 || type < 0 || type > 2) return 1;
  if (!aligned(grad, 16) || !aligned(buf, 16) || !aligned(x, 16) || !aligned(out, 16)) return 2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const long long n = (long long)rows * cols;
  const unsigned grid = grid_for(n);
  __nv_bfloat16* xb = (__nv_bfloat16*)x;
  if (type == 0) muon_momentum_kernel<<<grid, kThreads, 0, s>>>((const __nv_bfloat16*)grad, buf, xb, partial, n, mu, nu, nesterov);
  else if (type == 1) muon_momentum_kernel<<<grid, kThreads, 0, s>>>((const __half*)grad, buf, xb, partial, n, mu, nu, nesterov);
  else muon_momentum_kernel<<<grid, kThreads, 0, s>>>((const float*)grad, buf, xb, partial, n, mu, nu, nesterov);
  if (rows > cols)
    muon_normalise_kernel<true><<<grid, kThreads, 0, s>>>(xb, partial, (int)grid, (__nv_bfloat16*)out, rows, cols);
  else
    muon_normalise_kernel<false><<<grid, kThreads, 0, s>>>(xb, partial, (int)grid, (__nv_bfloat16*)out, rows, cols);
  return launched();
}

// u: bf16, the result of the iterations in the orientation of fbam_muon_prepare's out; w: fp32 master, updated; param
// (type 0 bf16, 1 half) receives the rounded master, or null.
int fbam_muon_apply(const void* u, float* w, void* param, int type, int rows, int cols, float decay, float lr, float scale,
                    void* stream) {
  if (rows < 8 || cols < 8 || rows % 8 || cols % 8 || type < 0 || type > 1) return 1;
  if (!aligned(u, 16) || !aligned(w, 16) || !aligned(param, 8)) return 2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const unsigned grid = grid_for((long long)rows * cols);
  const __nv_bfloat16* ub = (const __nv_bfloat16*)u;
  if (type == 0) {
    if (rows > cols) muon_apply_kernel<true><<<grid, kThreads, 0, s>>>(ub, w, (__nv_bfloat16*)param, rows, cols, decay, lr, scale);
    else muon_apply_kernel<false><<<grid, kThreads, 0, s>>>(ub, w, (__nv_bfloat16*)param, rows, cols, decay, lr, scale);
  } else {
    if (rows > cols) muon_apply_kernel<true><<<grid, kThreads, 0, s>>>(ub, w, (__half*)param, rows, cols, decay, lr, scale);
    else muon_apply_kernel<false><<<grid, kThreads, 0, s>>>(ub, w, (__half*)param, rows, cols, decay, lr, scale);
  }
  return launched();
}

}  // extern "C"
