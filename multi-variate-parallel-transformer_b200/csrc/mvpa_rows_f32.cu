// The block's row kernels on fp32 rows, compiled without --use_fast_math: expf within one unit in the last place, divisions
// correctly rounded, small values kept.  What that costs is hidden by memory: see the kernels' figures in block_rows.cuh.
#include "block_rows.cuh"

namespace mvpa {

int rmsnorm_f32(const void* x, const void* a, const void* w, void* h_out, void* y, int64_t rows, int E, float eps, cudaStream_t s) {
  return launch_rmsnorm<float>(x, a, w, h_out, y, rows, E, eps, s);
}

int rmsnorm_bwd_f32(const void* x, const void* w, const void* dy, const void* add, void* dx, void* dw, float* ws, int64_t rows,
                    int E, float eps, cudaStream_t s) {
  return launch_rmsnorm_bwd<float>(x, w, dy, add, dx, dw, ws, rows, E, eps, s);
}

int silu_mul_f32(const void* gate, const void* up, int64_t ld_in, void* out, int64_t ld_out, int64_t rows, int width,
                 cudaStream_t s) {
  return launch_silu_mul<float>(gate, up, ld_in, out, ld_out, rows, width, s);
}

int silu_mul_bwd_f32(const void* gate, const void* up, int64_t ld_in, const void* dout, int64_t ld_dout, void* dgate, void* dup,
                     int64_t ld_grad, int64_t rows, int width, cudaStream_t s) {
  return launch_silu_mul_bwd<float>(gate, up, ld_in, dout, ld_dout, dgate, dup, ld_grad, rows, width, s);
}

}  // namespace mvpa
