// In-register and shared-memory FFT building blocks, shared by the FFT entry
// points (ct2g_fft.cu) and the mesh-solve kernels (ct2g_fft_mesh.cuh).
#pragma once

#include <type_traits>

#include <cuda.h>  // CUtensorMap and the cuTensorMapEncodeTiled signature (called through the runtime's entry point)

#include "ct2g_internal.cuh"
#include "ct2g_tc.cuh"

namespace {

template <typename T> struct Cplx;
template <> struct Cplx<float> { using type = float2; };
template <> struct Cplx<double> { using type = double2; };

// exp(-2 pi i k/32), k < 32, set at context creation from host FP64 cos/sin
__constant__ float2 c_w32f[32];
__constant__ double2 c_w32d[32];

template <typename C2> __device__ __forceinline__ C2 w32(int k);
template <> __device__ __forceinline__ float2 w32<float2>(int k) { return c_w32f[k]; }
template <> __device__ __forceinline__ double2 w32<double2>(int k) { return c_w32d[k]; }

template <typename C2>
__device__ __forceinline__ C2 cmul(C2 a, C2 b) {
  C2 r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename C2>
__device__ __forceinline__ C2 cadd(C2 a, C2 b) {
  C2 r;
  r.x = a.x + b.x;
  r.y = a.y + b.y;
  return r;
}
template <typename C2>
__device__ __forceinline__ C2 csub(C2 a, C2 b) {
  C2 r;
  r.x = a.x - b.x;
  r.y = a.y - b.y;
  return r;
}
// FP32 complex sums as one packed f32x2 instruction (two round-to-nearest
// FP32 operations, the same results as the scalar pair)
template <>
__device__ __forceinline__ float2 cadd<float2>(float2 a, float2 b) {
  unsigned long long pa, pb, pr;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b.x), "f"(b.y));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(pr) : "l"(pa), "l"(pb));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(pr));
  return r;
}
template <>
__device__ __forceinline__ float2 csub<float2>(float2 a, float2 b) {
  unsigned long long pa, pb, pr;
  asm("mov.b64 %0, {%1, %2};" : "=l"(pa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(pb) : "f"(b.x), "f"(b.y));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(pr) : "l"(pa), "l"(pb));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(pr));
  return r;
}

constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n / 2); }
constexpr int brevc(int v, int bits) {
  int r = 0;
  for (int i = 0; i < bits; i++) r |= ((v >> i) & 1) << (bits - 1 - i);
  return r;
}

// In-register R-point DFT (R <= 32), natural order in and out.
// Radix-2 DIF: span h from R/2 down to 1, butterfly (a, b) ->
// (a + b, (a - b) W_{2h}^j); the result lands in bit-reversed order and is
// permuted back at compile time.  W = -i (a quarter turn) is a swap and a
// sign, not a complex product.
template <int R, typename C2, bool INV>
__device__ __forceinline__ void reg_dft(C2 (&v)[R]) {
#pragma unroll
  for (int h = R / 2; h >= 1; h >>= 1) {
#pragma unroll
    for (int blk = 0; blk < R; blk += 2 * h) {
#pragma unroll
      for (int j = 0; j < h; j++) {
        const C2 a = v[blk + j], b = v[blk + j + h];
        v[blk + j] = cadd(a, b);
        C2 d = csub(a, b);
        if (j * (32 / (2 * h)) == 8) {  // W = -i (forward), +i (inverse): a swap
          const C2 e = d;
          d.x = INV ? -e.y : e.y;
          d.y = INV ? e.x : -e.x;
        } else if (j != 0) {
          C2 w = w32<C2>(j * (32 / (2 * h)));
          if (INV) w.y = -w.y;
          d = cmul(d, w);
        }
        v[blk + j + h] = d;
      }
    }
  }
  C2 t[R];
#pragma unroll
  for (int k = 0; k < R; k++) t[k] = v[brevc(k, ilog2c(R))];
#pragma unroll
  for (int k = 0; k < R; k++) v[k] = t[k];
}

// Line FFTs on smem lines.  Layout ROWS: element (l, r) at
// l*(N + N/R1 + 1) + r + r/R1 (one pad every R1 points); layout COLS: element
// (l, r) at r*W + l.
template <int N, bool ROWS>
struct LineLayout {
  static constexpr int R2 = N >= 4 ? (1 << (ilog2c(N) / 2)) : 1;
  static constexpr int R1 = N / R2;  // R1 >= R2
  // odd in complex units, so that the same point of consecutive lines falls
  // in different banks
  static constexpr int LS = N + N / R1 + 1;
  __device__ __forceinline__ static int at(int l, int r, int W) {
    return ROWS ? l * LS + r + r / R1 : r * W + l;
  }
};

// Transform `nlines` lines (nlines*R1 and nlines*R2 jobs spread over the block).
// stw: the step-1 twiddles in smem (load_twiddles).
template <int N, bool ROWS, typename C2, bool INV>
__device__ __forceinline__ void tile_fft(C2 *s, int nlines, int W, const C2 *stw) {
  using LL = LineLayout<N, ROWS>;
  constexpr int R1 = LL::R1, R2 = LL::R2;
  // step 1: job (line, n1): R2-point DFT over r = n1 + R1*n2, twiddle.  The
  // block has 256 threads.
  for (int job = threadIdx.x; job < nlines * R1; job += blockDim.x) {
    int l, n1;
    if (ROWS) {
      n1 = job % R1;
      l = job / R1;
    } else {
      l = job % nlines;
      n1 = job / nlines;
    }
    C2 v[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) v[n2] = s[LL::at(l, n1 + R1 * n2, W)];
    reg_dft<R2, C2, INV>(v);
#pragma unroll
    for (int k2 = 1; k2 < R2; k2++) {
      C2 w = stw[R1 * k2 + n1];
      if (INV) w.y = -w.y;
      v[k2] = cmul(v[k2], w);
    }
    // Y[n1][k2] back into the slots just read (slot n1 + R1*k2)
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) s[LL::at(l, n1 + R1 * k2, W)] = v[k2];
  }
  __syncthreads();
  // step 2: job (line, k2): R1-point DFT over n1 -> X[k2 + R2*k1].  Jobs go
  // in rounds of whole lines (LW lines per round), so a round's writes never
  // touch slots that a later round still has to read.
  constexpr int LW = 256 / R2;
  for (int l0 = 0; l0 < nlines; l0 += LW) {
    int l, k2;
    if (ROWS) {
      k2 = threadIdx.x % R2;
      l = l0 + threadIdx.x / R2;
    } else {
      l = l0 + threadIdx.x % LW;
      k2 = threadIdx.x / LW;
    }
    const bool on = l < nlines;
    C2 v[R1];
    if (on) {
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) v[n1] = s[LL::at(l, n1 + R1 * k2, W)];
      reg_dft<R1, C2, INV>(v);
    }
    __syncthreads();  // all reads of this round before any write
    if (on) {
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) s[LL::at(l, k2 + R2 * k1, W)] = v[k1];
    }
    __syncthreads();
  }
}

// exp(-2 pi i n1 k2/N) at R1 k2 + n1: the threads of a warp that differ in n1
// read consecutive values at offsets known at compile time (the table of
// exp(-2 pi i k/N) itself put them k2 apart: 2.1 shared-memory cycles a load on
// average over k2 < 16, 8 at k2 = 8, and an index to compute: inverse z pass
// of a 256^3 mesh 954 -> 900 us, y passes 840 -> 826)
template <int N, typename C2>
__device__ __forceinline__ void load_twiddles(C2 *stw, const C2 *tw) {
  constexpr int R1 = LineLayout<N, true>::R1;
  for (int i = threadIdx.x; i < N; i += blockDim.x) stw[i] = tw[((i % R1) * (i / R1)) & (N - 1)];
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int NPEND>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(NPEND) : "memory");
}

template <typename C2>
const C2 *twiddle_ptr(ct2g_ctx *ctx);
template <>
inline const float2 *twiddle_ptr<float2>(ct2g_ctx *ctx) { return ctx->tw32; }
template <>
inline const double2 *twiddle_ptr<double2>(ct2g_ctx *ctx) { return ctx->tw64; }

// polls of a bounded wait for a bulk copy
constexpr uint32_t kTmaWaitLimit = 1u << 22;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                  const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the driver's tensor-map encoder, looked up once through the runtime
inline int tensor_map_encoder(ct2g_ctx *ctx, EncodeTiledFn *out) {
  static EncodeTiledFn encode = nullptr;
  if (!encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      cudaGetLastError();
      return ct2g_fail(ctx, CT2G_ECUDA, "cuTensorMapEncodeTiled not available");
    }
    encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  *out = encode;
  return CT2G_OK;
}

// the constant twiddles of the in-register DFTs (every file that includes this
// has its own)
inline int set_consts(ct2g_ctx *ctx) {
  float2 wf[32];
  double2 wd[32];
  const double twopi = 6.283185307179586476925286766559;
  for (int k = 0; k < 32; k++) {
    const double a = -twopi * (double)k / 32.0;
    wd[k] = make_double2(std::cos(a), std::sin(a));
    wf[k] = make_float2((float)wd[k].x, (float)wd[k].y);
  }
  CT2G_CUDA(ctx, cudaMemcpyToSymbol(c_w32f, wf, sizeof(wf)));
  CT2G_CUDA(ctx, cudaMemcpyToSymbol(c_w32d, wd, sizeof(wd)));
  return CT2G_OK;
}

}  // namespace
