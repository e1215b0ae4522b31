// Element-wise kernels of the decode step around the attention op: RMSNorm, rotary embedding of
// the new query, SiLU(gate) * up.  In the accuracy pipeline these are chains of small torch ops
// (fake_quant/svd_utils.py:1628-1674: LlamaRMSNorm, apply_rotary_pos_emb, the MLP's act_fn); a
// decode step of batch 64 spends a third of its time launching them, so each chain is one kernel
// here.  f16 in and out, fp32 arithmetic, rounding at the same places as the torch chains.
#include "common.cuh"

namespace wsvd {
namespace {

// y[r, :] = f16( x[r, :] * rsqrt(mean(x[r, :]^2) + eps) ), one block per row
__global__ void __launch_bounds__(256) rms_norm_kernel(const __half* __restrict__ x, __half* __restrict__ y, int cols,
                                                       float eps) {
  const __half* xr = x + (int64_t)blockIdx.x * cols;
  __half* yr = y + (int64_t)blockIdx.x * cols;
  float ss = 0.f;
  for (int i = threadIdx.x; i < cols; i += 256) {
    const float v = __half2float(xr[i]);
    ss = fmaf(v, v, ss);
  }
  ss = warp_sum(ss);
  __shared__ float part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) tot += part[w];
  const float scale = rsqrtf(tot / (float)cols + eps);
  for (int i = threadIdx.x; i < cols; i += 256) yr[i] = __float2half_rn(__half2float(xr[i]) * scale);
}

// x_out[r, :] = f16(x[r, :] + delta[r, :]) (the residual add), y[r, :] = RMSNorm of the rounded sum:
// the residual update and the next block's normalisation in one pass over the row
__global__ void __launch_bounds__(256) add_rms_norm_kernel(const __half* __restrict__ x, const __half* __restrict__ delta,
                                                           __half* __restrict__ x_out, __half* __restrict__ y, int cols,
                                                           float eps) {
  const int64_t off = (int64_t)blockIdx.x * cols;
  float ss = 0.f;
  for (int i = threadIdx.x; i < cols; i += 256) {
    const __half sum = __float2half_rn(__half2float(x[off + i]) + __half2float(delta[off + i]));
    x_out[off + i] = sum;
    const float v = __half2float(sum);
    ss = fmaf(v, v, ss);
  }
  ss = warp_sum(ss);
  __shared__ float part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < 8; ++w) tot += part[w];
  const float scale = rsqrtf(tot / (float)cols + eps);
  // each thread re-reads the elements it wrote itself
  for (int i = threadIdx.x; i < cols; i += 256) y[off + i] = __float2half_rn(__half2float(x_out[off + i]) * scale);
}

// The two kernels above for rows of whole 16-byte vectors: a row stays in registers between the two passes (up to
// kRowVecs vectors a thread), so it is read once, eight values a load.  The squares are added in the order of the
// scalar kernels (a thread takes every 256th value, handed over through shared memory), so that the results have the
// same bits: an int8 latent two GEMMs later must not depend on which of the kernels ran.  A decode step's 16 rows of 4096
// are bound by latency (one block a row): add + norm 5.5 us with scalar loads and a second read of the row, 3.3 us here.
constexpr int kRowThreads = 256, kRowVecs = 8;

template <bool kAdd>
__global__ void __launch_bounds__(kRowThreads) rms_norm_vec_kernel(const uint4* x, const uint4* delta, uint4* x_out, uint4* y,
                                                                   int vecs, float eps) {  // x_out may be x
  const int64_t off = (int64_t)blockIdx.x * vecs;
  extern __shared__ uint4 row_sm[];
  uint4 v[kRowVecs];
#pragma unroll
  for (int k = 0; k < kRowVecs; ++k) {
    const int i = threadIdx.x + k * kRowThreads;
    if (i < vecs) v[k] = x[off + i];
  }
#pragma unroll
  for (int k = 0; k < kRowVecs; ++k) {
    const int i = threadIdx.x + k * kRowThreads;
    if (i >= vecs) continue;
    if (kAdd) {
      const uint4 d = delta[off + i];
      __half2* h = reinterpret_cast<__half2*>(&v[k]);
      const __half2* e = reinterpret_cast<const __half2*>(&d);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h[j]), g = __half22float2(e[j]);
        h[j] = __floats2half2_rn(f.x + g.x, f.y + g.y);
      }
      x_out[off + i] = v[k];
    }
    row_sm[i] = v[k];
  }
  __syncthreads();
  float ss = 0.f;
  const __half* row = reinterpret_cast<const __half*>(row_sm);
#pragma unroll 8
  for (int i = threadIdx.x; i < vecs * 8; i += kRowThreads) {
    const float f = __half2float(row[i]);
    ss = fmaf(f, f, ss);
  }
  ss = warp_sum(ss);
  __shared__ float part[kRowThreads / 32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < kRowThreads / 32; ++w) tot += part[w];
  const float scale = rsqrtf(tot / (float)(vecs * 8) + eps);
#pragma unroll
  for (int k = 0; k < kRowVecs; ++k) {
    const int i = threadIdx.x + k * kRowThreads;
    if (i >= vecs) continue;
    __half2* h = reinterpret_cast<__half2*>(&v[k]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __half22float2(h[j]);
      h[j] = __floats2half2_rn(f.x * scale, f.y * scale);
    }
    y[off + i] = v[k];
  }
}

// whether rows of `cols` values at these addresses can be taken as 16-byte vectors by the kernel above
bool row_vectors(int cols, const void* a, const void* b, const void* c, const void* d) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
                        reinterpret_cast<uintptr_t>(d);
  return cols % 8 == 0 && cols <= kRowThreads * kRowVecs * 8 && (all & 15) == 0;
}

// half-split rotary embedding in place: q[b, h, i], q[b, h, i + D/2] rotated by pos[b] * inv_freq[i]
__global__ void rope_half_kernel(__half* __restrict__ q, int64_t q_stride_b, const int32_t* __restrict__ pos,
                                 const float* __restrict__ inv_freq, int heads, int half_dim, int64_t total) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int i = (int)(idx % half_dim);
  const int64_t bh = idx / half_dim;
  const int b = (int)(bh / heads);
  float sn, cs;
  sincosf((float)pos[b] * inv_freq[i], &sn, &cs);
  __half* row = q + (int64_t)b * q_stride_b + (bh - (int64_t)b * heads) * (2 * half_dim);
  const float lo = __half2float(row[i]), hi = __half2float(row[i + half_dim]);
  row[i] = __float2half_rn(lo * cs - hi * sn);
  row[i + half_dim] = __float2half_rn(hi * cs + lo * sn);
}

// out = up * f16(silu(gate)), the product rounded to f16 (the two roundings of the torch chain)
__global__ void silu_mul_kernel(const __half* __restrict__ up, int64_t up_ld, const __half* __restrict__ gate,
                                int64_t gate_ld, __half* __restrict__ out, int cols, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t r = i / cols, c = i - r * cols;
  const float g = __half2float(gate[r * gate_ld + c]);
  const __half s = __float2half_rn(g / (1.f + expf(-g)));
  out[i] = __float2half_rn(__half2float(up[r * up_ld + c]) * __half2float(s));
}

// The same, eight values a thread (rows of whole 16-byte vectors)
__global__ void silu_mul_vec_kernel(const uint4* __restrict__ up, int64_t up_ld, const uint4* __restrict__ gate, int64_t gate_ld,
                                    uint4* __restrict__ out, int vecs, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t r = i / vecs, c = i - r * vecs;
  uint4 u = up[r * up_ld + c];
  const uint4 gv = gate[r * gate_ld + c];
  __half2* uh = reinterpret_cast<__half2*>(&u);
  const __half2* gh = reinterpret_cast<const __half2*>(&gv);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 g = __half22float2(gh[j]), a = __half22float2(uh[j]);
    const float2 s = __half22float2(__floats2half2_rn(g.x / (1.f + expf(-g.x)), g.y / (1.f + expf(-g.y))));
    uh[j] = __floats2half2_rn(a.x * s.x, a.y * s.y);
  }
  out[i] = u;
}

}  // namespace
}  // namespace wsvd

extern "C" {

int wsvd_rms_norm_f16(const void* x, void* y, int32_t rows, int32_t cols, float eps, void* stream) {
  if (!x || !y) return WSVD_ERR_NULL_POINTER;
  if (rows < 0 || cols <= 0) return WSVD_ERR_BAD_SHAPE;
  if (rows == 0) return WSVD_OK;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (wsvd::row_vectors(cols, x, y, nullptr, nullptr))
    wsvd::rms_norm_vec_kernel<false><<<rows, wsvd::kRowThreads, (size_t)cols * 2, s>>>(reinterpret_cast<const uint4*>(x), nullptr, nullptr,
                                                                        reinterpret_cast<uint4*>(y), cols / 8, eps);
  else
    wsvd::rms_norm_kernel<<<rows, 256, 0, s>>>(reinterpret_cast<const __half*>(x), reinterpret_cast<__half*>(y), cols, eps);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WSVD_OK : wsvd::record_cuda_error(e);
}

int wsvd_add_rms_norm_f16(const void* x, const void* delta, void* x_out, void* y, int32_t rows, int32_t cols, float eps,
                          void* stream) {
  if (!x || !delta || !x_out || !y) return WSVD_ERR_NULL_POINTER;
  if (rows < 0 || cols <= 0) return WSVD_ERR_BAD_SHAPE;
  if (rows == 0) return WSVD_OK;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (wsvd::row_vectors(cols, x, delta, x_out, y))
    wsvd::rms_norm_vec_kernel<true><<<rows, wsvd::kRowThreads, (size_t)cols * 2, s>>>(
        reinterpret_cast<const uint4*>(x), reinterpret_cast<const uint4*>(delta), reinterpret_cast<uint4*>(x_out),
        reinterpret_cast<uint4*>(y), cols / 8, eps);
  else
    wsvd::add_rms_norm_kernel<<<rows, 256, 0, s>>>(reinterpret_cast<const __half*>(x), reinterpret_cast<const __half*>(delta),
                                                   reinterpret_cast<__half*>(x_out), reinterpret_cast<__half*>(y), cols, eps);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WSVD_OK : wsvd::record_cuda_error(e);
}

int wsvd_rope_half_f16(void* q, int64_t q_stride_b, const int32_t* pos, const float* inv_freq, int32_t batch,
                       int32_t heads, int32_t head_dim, void* stream) {
  if (!q || !pos || !inv_freq) return WSVD_ERR_NULL_POINTER;
  if (batch < 0 || heads <= 0 || head_dim <= 0 || head_dim % 2) return WSVD_ERR_BAD_SHAPE;
  if (q_stride_b < (int64_t)heads * head_dim) return WSVD_ERR_BAD_STRIDE;
  const int64_t total = (int64_t)batch * heads * (head_dim / 2);
  if (total == 0) return WSVD_OK;
  wsvd::rope_half_kernel<<<(unsigned)((total + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<__half*>(q), q_stride_b, pos, inv_freq, heads, head_dim / 2, total);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WSVD_OK : wsvd::record_cuda_error(e);
}

int wsvd_silu_mul_f16(const void* up, int64_t up_ld, const void* gate, int64_t gate_ld, void* out, int32_t rows,
                      int32_t cols, void* stream) {
  if (!up || !gate || !out) return WSVD_ERR_NULL_POINTER;
  if (rows < 0 || cols <= 0) return WSVD_ERR_BAD_SHAPE;
  if (up_ld < cols || gate_ld < cols) return WSVD_ERR_BAD_STRIDE;
  const int64_t n = (int64_t)rows * cols;
  if (n == 0) return WSVD_OK;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const uintptr_t all = reinterpret_cast<uintptr_t>(up) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(out);
  if (cols % 8 == 0 && up_ld % 8 == 0 && gate_ld % 8 == 0 && (all & 15) == 0)
    wsvd::silu_mul_vec_kernel<<<(unsigned)((n / 8 + 127) / 128), 128, 0, s>>>(
        reinterpret_cast<const uint4*>(up), up_ld / 8, reinterpret_cast<const uint4*>(gate), gate_ld / 8,
        reinterpret_cast<uint4*>(out), cols / 8, n / 8);
  else
    wsvd::silu_mul_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
        reinterpret_cast<const __half*>(up), up_ld, reinterpret_cast<const __half*>(gate), gate_ld,
        reinterpret_cast<__half*>(out), cols, n);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? WSVD_OK : wsvd::record_cuda_error(e);
}

}  // extern "C"
