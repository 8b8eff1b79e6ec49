// Elementwise kernels of the warm-start surrogate (a small MLP with a learned
// low-rank field basis): the GELU backward, column sums, the masked MSE
// gradient and an Adam step.  Its GEMM is in dsmc_gemm.cu.
#include <cuda_bf16.h>

#include <cstdint>

#include "dsmc_b200.h"
#include "dsmc_kernels.cuh"

namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678f)) + z * 0.39894228f * expf(-0.5f * z * z);
}

__global__ void k_gelu_backward(const float* z, const float* dh, float* dz, bf16* dzb, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float d = dh[i] * gelu_grad(z[i]);
    if (dz) dz[i] = d;
    if (dzb) dzb[i] = __float2bfloat16(d);
  }
}

// out[col] = sum over rows of x[row * ld + col], every column added row by row
// in FP32.  A block takes 32 columns: its eight warps stage kColRows rows at a
// time in shared memory, so that hundreds of loads are in flight, and the
// first warp adds them (one thread per column straight from memory waited
// for each group of loads in turn, on two blocks for a layer's 512 columns:
// 1024 x 512 61 us, now 10 us).
constexpr int kColWarps = 8, kColRows = 128;
__global__ void __launch_bounds__(32 * kColWarps) k_colsum(const float* x, int rows, int cols, int ld, float* out,
                                                           bool beside) {
  dsmcb::beside_entry(beside);
  __shared__ float st[2][kColRows][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  constexpr int per = kColRows / kColWarps;
  float v[per];
  auto load = [&](int r0) {
#pragma unroll
    for (int i = 0; i < per; i++) {
      const int r = r0 + w + kColWarps * i;
      v[i] = (r < rows && col < cols) ? x[(size_t)r * ld + col] : 0.f;
    }
  };
  load(0);
  float s = 0.f;
  int b = 0;
  for (int r0 = 0; r0 < rows; r0 += kColRows, b ^= 1) {
#pragma unroll
    for (int i = 0; i < per; i++) st[b][w + kColWarps * i][lane] = v[i];
    __syncthreads();
    load(r0 + kColRows);  // the next rows, while the first warp adds these
    if (w == 0) {
      const int n = min(kColRows, rows - r0);
      if (n == kColRows) {
#pragma unroll 32
        for (int i = 0; i < kColRows; i++) s += st[b][i][lane];
      } else {
        for (int i = 0; i < n; i++) s += st[b][i][lane];
      }
    }
  }
  if (w == 0 && col < cols) out[col] = s;
  dsmcb::beside_exit(beside);
}

// The same sums, a thread per column straight from memory: few rows, or so
// many columns that they fill the GPU by themselves (the staged form's blocks
// then come in many waves: 16 x 327680 37 us, here 5; 128 x 81920 15 and 8; but
// 128 x 8192 5 and 7, 1024 x 81920 65 and 80).
__global__ void k_colsum_wide(const float* x, int rows, int cols, int ld, float* out) {
  const int col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= cols) return;
  float s = 0.f;
  for (int r = 0; r < rows; r++) s += x[(size_t)r * ld + col];
  out[col] = s;
}

// Masked MSE: targets that are NaN carry no loss.  dy = scale * 2 (y - t).
__global__ void k_mse_grad(const float* y, const bf16* t, size_t n, float scale, bf16* dyb, float* dy,
                           double* loss, unsigned long long* count) {
  __shared__ double red[32];
  __shared__ unsigned long long cnt[32];
  double s = 0.0;
  unsigned long long c = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float tv = __bfloat162float(t[i]);
    float g = 0.f;
    if (tv == tv) {
      const float e = y[i] - tv;
      s += (double)e * e;
      c++;
      g = scale * 2.f * e;
    }
    if (dyb) dyb[i] = __float2bfloat16(g);
    if (dy) dy[i] = g;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = s;
    cnt[threadIdx.x >> 5] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    unsigned long long b = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      a += red[w];
      b += cnt[w];
    }
    if (loss) atomicAdd(loss, a);
    if (count) atomicAdd(count, b);
  }
}

struct AdamArgs {
  float lr, b1, b2, eps, c1, c2, wd;
};

__device__ __forceinline__ void adam_one(const AdamArgs& a, float gi, float& w, float& m, float& v) {
  m = a.b1 * m + (1.f - a.b1) * gi;
  v = a.b2 * v + (1.f - a.b2) * gi * gi;
  const float upd = (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
  w = w - a.lr * (upd + a.wd * w);
}

// Adam with decoupled weight decay; also refreshes the BF16 copy.  30 bytes
// per weight: memory bounds it, so four weights per thread move as 16-byte
// accesses (VEC: every array aligned for them; the n % 4 last ones singly):
// 84M weights 558 -> 400 us, 0.96 of the copy bandwidth.
template <bool VEC>
__global__ void __launch_bounds__(256) k_adam(float* w, const float* g, float* m, float* v, bf16* wb, size_t n,
                                              const AdamArgs a,
                                              bool beside) {
  dsmcb::beside_entry(beside);
  const size_t t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
  size_t done = 0;
  if (VEC) {
    done = n & ~(size_t)3;
    for (size_t i = 4 * t0; i < done; i += 4 * nt) {
      const float4 gv = __ldcs(reinterpret_cast<const float4*>(g + i));
      float4 wv = *reinterpret_cast<const float4*>(w + i);
      float4 mv = __ldcs(reinterpret_cast<const float4*>(m + i));
      float4 vv = __ldcs(reinterpret_cast<const float4*>(v + i));
      adam_one(a, gv.x, wv.x, mv.x, vv.x);
      adam_one(a, gv.y, wv.y, mv.y, vv.y);
      adam_one(a, gv.z, wv.z, mv.z, vv.z);
      adam_one(a, gv.w, wv.w, mv.w, vv.w);
      __stcs(reinterpret_cast<float4*>(m + i), mv);
      __stcs(reinterpret_cast<float4*>(v + i), vv);
      *reinterpret_cast<float4*>(w + i) = wv;
      if (wb) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(wv.x, wv.y), hi = __floats2bfloat162_rn(wv.z, wv.w);
        *reinterpret_cast<uint2*>(wb + i) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
      }
    }
  }
  for (size_t i = done + t0; i < n; i += nt) {
    const float gi = g[i];  // all four loads before the first store
    float wi = w[i], mi = m[i], vi = v[i];
    adam_one(a, gi, wi, mi, vi);
    m[i] = mi;
    v[i] = vi;
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16(wi);
  }
  dsmcb::beside_exit(beside);
}

__global__ void k_to_bf16(const float* x, bf16* y, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

unsigned grid_1d(size_t n) {
  size_t b = (n + 255) / 256;
  return (unsigned)(b < 4096 ? (b ? b : 1) : 4096);
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

}  // namespace

cudaError_t dsmcb::launch_colsum_beside(const float* x, int rows, int cols, int ld, float* out, cudaStream_t stream) {
  return launch_chained(k_colsum, (uint32_t)(cols + 31) / 32, 32 * kColWarps, 0, stream, true, x, rows, cols, ld, out,
                        true);
}

extern "C" {

int dsmc_gelu_backward(const float* z, const float* dh, float* dz, void* dz_bf16, size_t n,
                       void* stream) {
  if (!z || !dh || (!dz && !dz_bf16)) return DSMC_ERR_ARG;
  k_gelu_backward<<<grid_1d(n), 256, 0, (cudaStream_t)stream>>>(z, dh, dz, static_cast<bf16*>(dz_bf16), n);
  return cudaGetLastError() == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

int dsmc_colsum(const float* x, int rows, int cols, int ld, float* out, void* stream) {
  if (!x || !out || rows < 0 || cols <= 0) return DSMC_ERR_ARG;
  // measured between 1 and 1024 rows of 512 to 327,680 columns: the forms meet
  // at about one row per 150 columns
  cudaStream_t s = (cudaStream_t)stream;
  if (rows <= 16 || (int64_t)rows * 150 <= cols) k_colsum_wide<<<(cols + 255) / 256, 256, 0, s>>>(x, rows, cols, ld, out);
  else k_colsum<<<(cols + 31) / 32, 32 * kColWarps, 0, s>>>(x, rows, cols, ld, out, false);
  return cudaGetLastError() == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

int dsmc_mse_grad(const float* y, const void* t_bf16, size_t n, float scale, void* dy_bf16, float* dy,
                  double* loss, unsigned long long* count, void* stream) {
  if (!y || !t_bf16) return DSMC_ERR_ARG;
  k_mse_grad<<<grid_1d(n), 256, 0, (cudaStream_t)stream>>>(y, static_cast<const bf16*>(t_bf16), n, scale,
                                                           static_cast<bf16*>(dy_bf16), dy, loss, count);
  return cudaGetLastError() == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

static int adam(float* w, const float* g, float* m, float* v, void* w_bf16, size_t n, float lr, float b1, float b2,
                float eps, int t, float weight_decay, bool beside, void* stream) {
  if (!w || !g || !m || !v || t < 1) return DSMC_ERR_ARG;
  AdamArgs a{lr, b1, b2, eps, 1.f - powf(b1, (float)t), 1.f - powf(b2, (float)t), weight_decay};
  bf16* wb = static_cast<bf16*>(w_bf16);
  cudaStream_t s = (cudaStream_t)stream;
  const bool vec = aligned16(w) && aligned16(g) && aligned16(m) && aligned16(v) && ((uintptr_t)wb & 7u) == 0;
  const cudaError_t e = dsmcb::launch_chained(vec ? k_adam<true> : k_adam<false>, grid_1d(vec ? (n + 3) / 4 : n), 256, 0, s,
                                              beside, w, g, m, v, wb, n, a, beside);
  return e == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

int dsmc_adam_step(float* w, const float* g, float* m, float* v, void* w_bf16, size_t n, float lr,
                   float b1, float b2, float eps, int t, float weight_decay, void* stream) {
  return adam(w, g, m, v, w_bf16, n, lr, b1, b2, eps, t, weight_decay, false, stream);
}

int dsmc_adam_steps(const dsmc_adam_param* params, int count, float lr, float b1, float b2, float eps, int t,
                    void* stream) {
  if (!params || count < 0) return DSMC_ERR_ARG;
  for (int i = 0; i < count; i++) {
    const dsmc_adam_param& p = params[i];
    const int st = adam(p.w, p.g, p.m, p.v, p.w_bf16, p.n, lr, b1, b2, eps, t, p.weight_decay, i > 0, stream);
    if (st != DSMC_OK) return st;
  }
  return DSMC_OK;
}

int dsmc_to_bf16(const float* x, void* y, size_t n, void* stream) {
  if (!x || !y) return DSMC_ERR_ARG;
  k_to_bf16<<<grid_1d(n), 256, 0, (cudaStream_t)stream>>>(x, static_cast<bf16*>(y), n);
  return cudaGetLastError() == cudaSuccess ? DSMC_OK : DSMC_ERR_CUDA;
}

}  // extern "C"
