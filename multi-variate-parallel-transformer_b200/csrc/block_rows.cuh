// Row kernels of the block: RMSNorm (with the residual sum), the SwiGLU gate, and their backwards.  Included by
// mvpa_block.cu, which runs them on bf16, and by mvpa_rows_f32.cu, which runs them on fp32 and is compiled without
// approximate arithmetic: in 16 bits the result's rounding hides what `expf` and the divisions lose there, in fp32 it does not.
#pragma once
#include <cuda_bf16.h>

#include "mvpa_common.cuh"
#include "tc_ptx.cuh"

namespace mvpa {
namespace {

constexpr int kWarpsPerCta = 8;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename T>
struct Vec;  // 16 bytes of T
template <>
struct Vec<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void load(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 r = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  __device__ static void unpack(const uint4& r, float (&f)[8]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
  __device__ static uint4 pack(const float (&f)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 v = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&v);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
  __device__ static void store(__nv_bfloat16* p, const float (&f)[8]) { *reinterpret_cast<uint4*>(p) = pack(f); }
  __device__ static float round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
};
template <>
struct Vec<float> {
  static constexpr int N = 4;
  __device__ static void load(const float* p, float (&f)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    f[0] = r.x; f[1] = r.y; f[2] = r.z; f[3] = r.w;
  }
  __device__ static void unpack(const uint4& r, float (&f)[4]) {
    f[0] = __uint_as_float(r.x); f[1] = __uint_as_float(r.y); f[2] = __uint_as_float(r.z); f[3] = __uint_as_float(r.w);
  }
  __device__ static uint4 pack(const float (&f)[4]) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
  __device__ static void store(float* p, const float (&f)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
  }
  __device__ static float round(float x) { return x; }
};

// Sum over a row's vectors of a[e] b[e]: bf16 rows in one chain, fp32 rows a sum per vector and then by halves (as few
// roundings at the size of the whole sum as eager PyTorch's reduction has).
template <typename T, int NV>
struct RowSum {
  static constexpr bool kSplit = sizeof(T) == 4;
  float part[kSplit ? NV : 1] = {};
  template <int N>
  __device__ __forceinline__ void add(int i, const float (&a)[N], const float (&b)[N]) {
    float& t = part[kSplit ? i : 0];
#pragma unroll
    for (int e = 0; e < N; ++e) t += a[e] * b[e];
  }
  __device__ __forceinline__ float total();
};

// The sum of N partial sums: fp32 rows by halves, bf16 rows one after the other.
template <typename T, int N>
__device__ __forceinline__ float sum_of(float (&s)[N]) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int h = N / 2; h > 0; h >>= 1)
#pragma unroll
      for (int k = 0; k < h; ++k) s[k] += s[k + h];
  } else {
#pragma unroll
    for (int k = 1; k < N; ++k) s[0] += s[k];
  }
  return s[0];
}

template <typename T, int NV>
__device__ __forceinline__ float RowSum<T, NV>::total() {
  return sum_of<T>(part);
}

// y = rmsnorm(h) * w with h = x (+ a), h optionally written out.  One warp per row; the row stays in
// registers, in its storage format (NV 16-byte vectors per lane: half the registers of an fp32 copy for
// bf16, which doubles the rows in flight per multiprocessor), between the sum of squares and the scaling.
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) rmsnorm_kernel(const T* __restrict__ x, const T* __restrict__ a,
                                                                    const T* __restrict__ w, T* __restrict__ h_out,
                                                                    T* __restrict__ y, int64_t rows, int E, float eps) {
  constexpr int N = Vec<T>::N;
  ptx::griddep_wait();
  const int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  const T* xr = x + row * E;
  uint4 raw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (i * 32 + lane) * N;
    if (col < E) raw[i] = *reinterpret_cast<const uint4*>(xr + col);
  }
  RowSum<T, NV> ss;
  if (a != nullptr) {
    uint4 rawa[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * 32 + lane) * N;
      if (col < E) rawa[i] = *reinterpret_cast<const uint4*>(a + row * E + col);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * 32 + lane) * N;
      if (col < E) {
        float v[N], b[N];
        Vec<T>::unpack(raw[i], v);
        Vec<T>::unpack(rawa[i], b);
#pragma unroll
        for (int e = 0; e < N; ++e) v[e] = Vec<T>::round(v[e] + b[e]);  // the sum lives in T, as in eager PyTorch
        ss.add(i, v, v);
        raw[i] = Vec<T>::pack(v);
        if (h_out != nullptr) *reinterpret_cast<uint4*>(h_out + row * E + col) = raw[i];
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * 32 + lane) * N;
      if (col < E) {
        float v[N];
        Vec<T>::unpack(raw[i], v);
        ss.add(i, v, v);
      }
    }
  }
  const float rstd = rsqrtf(warp_sum(ss.total()) / (float)E + eps);
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (i * 32 + lane) * N;
    if (col < E) {
      float v[N], g[N];
      Vec<T>::unpack(raw[i], v);
      Vec<T>::load(w + col, g);
#pragma unroll
      for (int e = 0; e < N; ++e) g[e] = v[e] * rstd * g[e];
      Vec<T>::store(y + row * E + col, g);
    }
  }
}

// Backward of rmsnorm_kernel without the residual add:  with g = dy w and xh = x rstd,
//   dx = rstd (g - xh mean(g xh)) (+ add),   dw = sum_rows dy xh.
// One warp per row at a time, rows strided over the grid; x and dy are read once, the row stays in registers;
// each lane keeps the dw of its columns over all its rows, the warps of a CTA meet in shared memory and one
// fp32 row per CTA goes to `dw_part` (summed in a fixed order by colsum_kernel: deterministic).  Bound by memory at many
// rows: 65536 x 768 without `add`, both kernels, L2 flushed, 73 us in bf16 (302 MB) and 126 us in fp32 (604 MB; 122 with
// approximate division and one chain per sum); 6400 x 768 bf16 takes 21.5 us, most of it the latency of two short kernels.
template <typename T, int NV>
__global__ void __launch_bounds__(kWarpsPerCta * 32) rmsnorm_bwd_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                                        const T* __restrict__ dy, const T* __restrict__ add,
                                                                        T* __restrict__ dx, float* __restrict__ dw_part,
                                                                        int64_t rows, int E, float eps) {
  constexpr int N = Vec<T>::N;
  extern __shared__ __align__(16) float s_dw[];  // [kWarpsPerCta][E]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float acc[NV][N];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int e = 0; e < N; ++e) acc[i][e] = 0.f;
  for (int64_t row = (int64_t)blockIdx.x * kWarpsPerCta + warp; row < rows; row += (int64_t)gridDim.x * kWarpsPerCta) {
    uint4 rx[NV], rg[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * 32 + lane) * N;
      if (col < E) {
        rx[i] = *reinterpret_cast<const uint4*>(x + row * E + col);
        rg[i] = *reinterpret_cast<const uint4*>(dy + row * E + col);
      }
    }
    RowSum<T, NV> ss, sg;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * 32 + lane) * N;
      if (col < E) {
        float v[N], g[N], wv[N];
        Vec<T>::unpack(rx[i], v);
        Vec<T>::unpack(rg[i], g);
        Vec<T>::load(w + col, wv);
        ss.add(i, v, v);
#pragma unroll
        for (int e = 0; e < N; ++e) wv[e] = g[e] * wv[e];
        sg.add(i, wv, v);
      }
    }
    const float rstd = rsqrtf(warp_sum(ss.total()) / (float)E + eps);
    const float c = warp_sum(sg.total()) * rstd / (float)E;  // mean(g xh)
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int col = (i * 32 + lane) * N;
      if (col < E) {
        float v[N], g[N], wv[N], r[N] = {};
        if (add != nullptr) Vec<T>::load(add + row * E + col, r);
        Vec<T>::unpack(rx[i], v);
        Vec<T>::unpack(rg[i], g);
        Vec<T>::load(w + col, wv);
#pragma unroll
        for (int e = 0; e < N; ++e) {
          const float xh = v[e] * rstd;
          acc[i][e] += g[e] * xh;
          r[e] += rstd * (g[e] * wv[e] - xh * c);
        }
        Vec<T>::store(dx + row * E + col, r);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int col = (i * 32 + lane) * N;
    if (col < E) {
#pragma unroll
      for (int e = 0; e < N; e += 4)
        *reinterpret_cast<float4*>(s_dw + warp * E + col + e) = make_float4(acc[i][e], acc[i][e + 1], acc[i][e + 2], acc[i][e + 3]);
    }
  }
  __syncthreads();
  for (int col = threadIdx.x; col < E; col += kWarpsPerCta * 32) {
    float s[kWarpsPerCta];
#pragma unroll
    for (int k = 0; k < kWarpsPerCta; ++k) s[k] = s_dw[k * E + col];
    dw_part[(int64_t)blockIdx.x * E + col] = sum_of<T>(s);
  }
}

// out[col] = sum_r part[r][col] in a fixed order: 32 columns per CTA, eight row strides; fp32 rows in eight chains a stride.
template <typename T>
__global__ void __launch_bounds__(256) colsum_kernel(const float* __restrict__ part, T* __restrict__ out, int n, int E) {
  constexpr int CH = sizeof(T) == 4 ? 8 : 1;
  __shared__ float s[8][33];
  const int col = blockIdx.x * 32 + (threadIdx.x & 31), k = threadIdx.x >> 5;
  float acc[CH] = {};
  if (col < E) {
#pragma unroll 8 / CH
    for (int r = k; r < n; r += 8 * CH)
#pragma unroll
      for (int c = 0; c < CH; ++c)
        if (CH == 1 || r + 8 * c < n) acc[c] += part[(int64_t)(r + 8 * c) * E + col];
  }
  s[k][threadIdx.x & 31] = sum_of<T>(acc);
  __syncthreads();
  if (k == 0 && col < E) {
    float part8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) part8[q] = s[q][threadIdx.x];
    out[col] = from_f32<T>(sum_of<T>(part8));
  }
}

// out = silu(gate) * up, elementwise, rows of `width` elements at independent leading dimensions.
template <typename T>
__global__ void __launch_bounds__(256) silu_mul_kernel(const T* __restrict__ gate, const T* __restrict__ up, int64_t ld_in,
                                                       T* __restrict__ out, int64_t ld_out, int64_t rows, int width) {
  ptx::griddep_wait();
  constexpr int N = Vec<T>::N;
  const int vec_per_row = width / N;
  const int64_t total = rows * vec_per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / vec_per_row;
    const int c = (int)(i % vec_per_row) * N;
    float g[N], u[N];
    Vec<T>::load(gate + r * ld_in + c, g);
    Vec<T>::load(up + r * ld_in + c, u);
#pragma unroll
    for (int e = 0; e < N; ++e) g[e] = Vec<T>::round(g[e] / (1.f + expf(-g[e]))) * u[e];
    Vec<T>::store(out + r * ld_out + c, g);
  }
}

// Backward of silu_mul_kernel for out = silu(gate) * up: with s = sigmoid(gate),
//   dgate = dout up s (1 + gate (1 - s)),  dup = dout silu(gate)   (silu rounded to T as in the forward).
// Bound by memory: L2 flushed, 65536 x 768 takes 92 us in bf16 (503 MB) and 178 us in fp32 (1007 MB; 168 with approximate
// exponentials and divisions, whose error grows with the gate: 1.8e-6 against 2.3e-7 at gates of standard deviation 8).
template <typename T>
__global__ void __launch_bounds__(256) silu_mul_bwd_kernel(const T* __restrict__ gate, const T* __restrict__ up, int64_t ld_in,
                                                           const T* __restrict__ dout, int64_t ld_dout,
                                                           T* __restrict__ dgate, T* __restrict__ dup, int64_t ld_g,
                                                           int64_t rows, int width) {
  constexpr int N = Vec<T>::N;
  const int vec_per_row = width / N;
  const int64_t total = rows * vec_per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / vec_per_row;
    const int c = (int)(i % vec_per_row) * N;
    float g[N], u[N], d[N];
    Vec<T>::load(gate + r * ld_in + c, g);
    Vec<T>::load(up + r * ld_in + c, u);
    Vec<T>::load(dout + r * ld_dout + c, d);
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const float s = 1.f / (1.f + expf(-g[e]));
      const float silu = Vec<T>::round(g[e] / (1.f + expf(-g[e])));
      const float du = d[e] * silu;
      const float ds = 1.f + g[e] * (1.f - s);
      g[e] = sizeof(T) == 4 ? d[e] * u[e] * s * ds : d[e] * u[e] * (s * ds);  // (the products in eager PyTorch's order)
      u[e] = du;
    }
    Vec<T>::store(dgate + r * ld_g + c, g);
    Vec<T>::store(dup + r * ld_g + c, u);
  }
}

template <typename T>
int launch_rmsnorm(const void* x, const void* a, const void* w, void* h_out, void* y, int64_t rows, int E, float eps,
                   cudaStream_t s) {
  constexpr int N = Vec<T>::N;
  const unsigned grid = (unsigned)((rows + kWarpsPerCta - 1) / kWarpsPerCta);
  const int nv = (E / N + 31) / 32;
#define MVPA_RMS(NV)                                                                                             \
  MVPA_CUDA_CHECK(launch_dependent(1, rmsnorm_kernel<T, NV>, grid, kWarpsPerCta * 32, 0, s, (const T*)x, (const T*)a, (const T*)w, \
                                   (T*)h_out, (T*)y, rows, E, eps))
  if (nv <= 2) MVPA_RMS(2);
  else if (nv <= 4) MVPA_RMS(4);
  else if (nv <= 8) MVPA_RMS(8);
  else MVPA_RMS(16);
#undef MVPA_RMS
  count_launch();
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

inline int rmsnorm_bwd_blocks(int64_t rows) {
  const int64_t want = (rows + kWarpsPerCta - 1) / kWarpsPerCta, most = 2 * (int64_t)device_sm_count();
  return (int)(want < most ? want : most);
}

template <typename T, int NV>
int run_rmsnorm_bwd(const void* x, const void* w, const void* dy, const void* add, void* dx, void* dw, float* ws, int64_t rows, int E,
                    float eps, cudaStream_t s) {
  const size_t smem = sizeof(float) * kWarpsPerCta * E;
  if (smem > 48 * 1024)
    MVPA_CUDA_CHECK(cudaFuncSetAttribute(rmsnorm_bwd_kernel<T, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = rmsnorm_bwd_blocks(rows);
  rmsnorm_bwd_kernel<T, NV><<<grid, kWarpsPerCta * 32, smem, s>>>((const T*)x, (const T*)w, (const T*)dy, (const T*)add, (T*)dx, ws, rows, E, eps);
  colsum_kernel<T><<<(E + 31) / 32, 256, 0, s>>>(ws, (T*)dw, grid, E);
  count_launch(2);
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

template <typename T>
int launch_rmsnorm_bwd(const void* x, const void* w, const void* dy, const void* add, void* dx, void* dw, float* ws, int64_t rows, int E,
                       float eps, cudaStream_t s) {
  const int nv = (E / Vec<T>::N + 31) / 32;
  if (nv <= 2) return run_rmsnorm_bwd<T, 2>(x, w, dy, add, dx, dw, ws, rows, E, eps, s);
  if (nv <= 4) return run_rmsnorm_bwd<T, 4>(x, w, dy, add, dx, dw, ws, rows, E, eps, s);
  if (nv <= 8) return run_rmsnorm_bwd<T, 8>(x, w, dy, add, dx, dw, ws, rows, E, eps, s);
  return run_rmsnorm_bwd<T, 16>(x, w, dy, add, dx, dw, ws, rows, E, eps, s);
}

template <typename T>
int launch_silu_mul(const void* gate, const void* up, int64_t ld_in, void* out, int64_t ld_out, int64_t rows, int width,
                    cudaStream_t s) {
  const int64_t ctas = (rows * (width / Vec<T>::N) + 255) / 256, most = (int64_t)device_sm_count() * 16;
  MVPA_CUDA_CHECK(launch_dependent(1, silu_mul_kernel<T>, (unsigned)(ctas < most ? ctas : most), 256, 0, s, (const T*)gate, (const T*)up,
                                   ld_in, (T*)out, ld_out, rows, width));
  count_launch();
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

template <typename T>
int launch_silu_mul_bwd(const void* gate, const void* up, int64_t ld_in, const void* dout, int64_t ld_dout, void* dgate, void* dup,
                        int64_t ld_grad, int64_t rows, int width, cudaStream_t s) {
  const int64_t ctas = (rows * (width / Vec<T>::N) + 255) / 256, most = (int64_t)device_sm_count() * 16;
  silu_mul_bwd_kernel<T><<<(unsigned)(ctas < most ? ctas : most), 256, 0, s>>>((const T*)gate, (const T*)up, ld_in, (const T*)dout,
                                                                               ld_dout, (T*)dgate, (T*)dup, ld_grad, rows, width);
  count_launch();
  MVPA_CUDA_CHECK(cudaGetLastError());
  return MVPA_OK;
}

}  // namespace

// The fp32 forms (mvpa_rows_f32.cu).
int rmsnorm_f32(const void* x, const void* a, const void* w, void* h_out, void* y, int64_t rows, int E, float eps, cudaStream_t s);
int rmsnorm_bwd_f32(const void* x, const void* w, const void* dy, const void* add, void* dx, void* dw, float* ws, int64_t rows,
                    int E, float eps, cudaStream_t s);
int silu_mul_f32(const void* gate, const void* up, int64_t ld_in, void* out, int64_t ld_out, int64_t rows, int width,
                 cudaStream_t s);
int silu_mul_bwd_f32(const void* gate, const void* up, int64_t ld_in, const void* dout, int64_t ld_dout, void* dgate, void* dup,
                     int64_t ld_grad, int64_t rows, int width, cudaStream_t s);

}  // namespace mvpa
