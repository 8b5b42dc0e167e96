// Cloud-in-cell deposit of the particle store onto a complex mesh, and the
// complex-to-complex 3D FFT over device grids.  No counterpart in the
// reference (its mesh quantities are per-cell multipoles, src/particle.cpp:
// 180-209); these serve callers that want a plain density mesh and its
// spectrum, in FP32 on the CUDA cores or with the y and x passes on the
// tensor cores (ct2g_set_fft_mode).
//
// Deposit: a particle at x (box units) sits between mesh points
// m = floor(x N - 1/2) and m + 1 along each axis, at fraction
// f = x N - 1/2 - m; it adds weight w = prod_d (f_d or 1 - f_d) to the 8
// surrounding points (periodic), and the four grids receive, at every point,
//   grid 0: sum_p w            (the CIC mass, unit particle mass)
//   grid 1..3: sum_p w * s_d   (the first moment about the point, s_d the
//                                particle's offset from it, in mesh units)
// as the real parts of complex values (imaginary parts zero), so that a
// batch of four complex transforms of N^3 points follows.
#include "ct2g_internal.cuh"

namespace {

__global__ void cic_deposit_kernel(const uint32_t *__restrict__ x, const uint32_t *__restrict__ y,
                                   const uint32_t *__restrict__ z, size_t n, int N,
                                   float2 *__restrict__ grid, bool aligned) {
  const size_t N3 = (size_t)N * N * N;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n;
       p += (size_t)gridDim.x * blockDim.x) {
    const uint32_t c[3] = {x[p], y[p], z[p]};
    int m[3];
    float f[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      // x N - 1/2 in mesh units, exact in FP64 for N <= 2^20
      const double u = (double)c[d] * CT2G_TWO_M32 * (double)N - 0.5;
      const double fl = floor(u);
      m[d] = (int)fl;
      f[d] = (float)(u - fl);
    }
    // the two corners of a z pair at once: where the lower point is even (and the
    // grid on a 16-byte boundary) they are one aligned 16 bytes (their imaginary parts get + 0), added by one vector
    // atomic: a quarter of the L2 atomics less (2.1 M particles onto 4 x 512^3:
    // 1.63 -> 1.10 ms)
    const int z0 = m[2] & (N - 1), z1 = (m[2] + 1) & (N - 1);
    const float wz0 = 1.f - f[2], wz1 = f[2];
#pragma unroll
    for (int corner = 0; corner < 4; corner++) {
      const int bx = corner >> 1, by = corner & 1;
      const float wxy = (bx ? f[0] : 1.f - f[0]) * (by ? f[1] : 1.f - f[1]);
      const float s0 = bx ? f[0] - 1.f : f[0], s1 = by ? f[1] - 1.f : f[1];
      const size_t row = ((size_t)((m[0] + bx) & (N - 1)) * N + ((m[1] + by) & (N - 1))) * N;
      const float w0 = wxy * wz0, w1 = wxy * wz1;
      const float v[4][2] = {{w0, w1}, {w0 * s0, w1 * s0}, {w0 * s1, w1 * s1},
                             {w0 * f[2], w1 * (f[2] - 1.f)}};
#pragma unroll
      for (int g = 0; g < 4; g++) {
        float2 *p0 = grid + g * N3 + row;
        if (aligned && (z0 & 1) == 0) {
          atomicAdd(reinterpret_cast<float4 *>(p0 + z0), make_float4(v[g][0], 0.f, v[g][1], 0.f));
        } else {
          atomicAdd(&p0[z0].x, v[g][0]);
          atomicAdd(&p0[z1].x, v[g][1]);
        }
      }
    }
  }
}

bool pow2(int n) { return n >= 1 && (n & (n - 1)) == 0; }

}  // namespace

extern "C" int ct2g_cic_deposit(ct2g_ctx *ctx, int N, void *d_grid) {
  CT2G_TRY(ct2g_check(ctx));
  if (!d_grid || !pow2(N) || N < 4 || N > 512)
    return ct2g_fail(ctx, CT2G_EINVAL, "cic_deposit: N a power of two in [4, 512], grid non-null");
  if (((uintptr_t)d_grid & 3) != 0)
    return ct2g_fail(ctx, CT2G_EINVAL, "cic_deposit: the grid must be 4-byte aligned");
  if (!ctx->has_particles) return ct2g_fail(ctx, CT2G_ESTATE, "no particles uploaded");
  const size_t N3 = (size_t)N * N * N;
  float2 *g = reinterpret_cast<float2 *>(d_grid);
  CT2G_CUDA(ctx, cudaMemsetAsync(g, 0, sizeof(float2) * 4 * N3, ctx->stream));
  if (ctx->n == 0) return CT2G_OK;
  const unsigned blocks = (unsigned)std::min<size_t>((ctx->n + 255) / 256, (size_t)ctx->num_sms * 8);
  cic_deposit_kernel<<<blocks, 256, 0, ctx->stream>>>(ctx->x, ctx->y, ctx->z, ctx->n, N, g,
                                                  ((uintptr_t)g & 15) == 0);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

extern "C" int ct2g_fft3d_c2c_f32_dev(ct2g_ctx *ctx, int dir, void *d_data, int N, int batch) {
  CT2G_TRY(ct2g_check(ctx));
  if (!d_data || batch < 1 || !pow2(N) || N < 4 || N > 512 || (dir != 1 && dir != -1))
    return ct2g_fail(ctx, CT2G_EINVAL, "fft3d_c2c_f32_dev: bad arguments");
  if ((reinterpret_cast<uintptr_t>(d_data) & 15) != 0)
    return ct2g_fail(ctx, CT2G_EINVAL, "fft3d_c2c_f32_dev: the grid must be 16-byte aligned");
  if (ctx->fft_tc && N != ctx->M)
    return ct2g_fail(ctx, CT2G_EINVAL,
                     "fft3d_c2c_f32_dev: the tensor-core passes are prepared for the context's mesh");
  return ct2g_fft_c2c_f32(ctx, reinterpret_cast<float2 *>(d_data), N, batch, dir < 0);
}
