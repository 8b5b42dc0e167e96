// Batched 3D real-to-complex / complex-to-real FFTs (FP32 and FP64).
//
// Replaces the reference's FP64 radix-2/4 FFT family (src/fft/*.cpp,
// cosmictiger/fft.hpp:18-29) and its 3D drivers fft_r2c_3d / fft_c2r_3d,
// whose bodies are empty or commented out in the reference
// (src/fft/fft_r2c_3d.cpp:4-31, src/fft/fft_c2r_3d.cpp:4-40).
//
// Layout: real grid x[b][i][j][k] (k contiguous), spectrum
// X[b][qi][qj][qk] with qk in [0, N/2] (k is the halved axis).  Forward sign
// exp(-2 pi i q.r/N) (the reference's twiddles cos(-2 pi n/N), sin(-2 pi n/N),
// src/fft/twiddles.cpp:6-38); c2r is the unnormalised inverse.
//
// Three passes, each one read and one write of the array:
//   Z: r2c along the contiguous axis, two real lines packed as one complex line
//   Y: complex FFT along j, tiles of W contiguous qk columns
//   X: complex FFT along i, tiles of W contiguous (qj,qk) columns
// A tile is staged in shared memory with coalesced loads.  Each line of
// N = R1*R2 points is transformed in two register stages (the "four-step"
// factorisation): R1 threads each do an R2-point DFT in registers over a
// stride-R1 subsequence, multiply by exp(-2 pi i n1 k2/N), and exchange
// through shared memory; R2 threads each then do an R1-point DFT.  The
// in-register DFTs are radix-2 decimation-in-frequency butterflies with
// compile-time twiddles.  Row tiles pad one word pair every R1 points so both
// exchange patterns are free of bank conflicts.
#include "ct2g_fft_core.cuh"

namespace {

// ---- pass Z forward: pairs of real lines -> half spectra -------------------
// LP complex (packed) lines per block; npairs = number of real-line pairs;
// output rows hold ld >= N/2+1 complex (the rest is written as zero).  VEC:
// ld*sizeof(complex) is a multiple of 16 bytes.
// (FP32 up to N = 256: four blocks per SM, whose loads and stores then overlap
// the others' transforms, at 64 registers, which spill 40 bytes a thread at N = 256; larger
// in-register DFTs and FP64 need the registers)
template <typename T, int N, bool VEC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 && N <= 256 ? 4 : 3) fftz_r2c_kernel(const T *__restrict__ in,
                                                          typename Cplx<T>::type *__restrict__ out,
                                                          size_t npairs, int LP, int ld,
                                                          const typename Cplx<T>::type *__restrict__ tw) {
  using C2 = typename Cplx<T>::type;
  using LL = LineLayout<N, true>;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int NH = N / 2 + 1;
  constexpr int RC = 16 / sizeof(T);  // reals per 16-byte chunk
  using RV = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  C2 *stw = reinterpret_cast<C2 *>(smraw);
  C2 *s = stw + N;
  T *sr = reinterpret_cast<T *>(s);
  load_twiddles<N>(stw, tw);
  const size_t pair0 = (size_t)blockIdx.x * LP;
  const int np = (int)min((size_t)LP, npairs - pair0);
  const T *src = in + pair0 * 2 * N;
  // real line 2l -> .x of complex line l, real line 2l+1 -> .y
  for (int c = threadIdx.x; c < np * 2 * N / RC; c += 256) {
    const int e = c * RC, rl = e / N, r = e % N;
    const RV v = *reinterpret_cast<const RV *>(src + e);
    const T *vv = reinterpret_cast<const T *>(&v);
#pragma unroll
    for (int q = 0; q < RC; q++) sr[2 * LL::at(rl >> 1, r + q, 0) + (rl & 1)] = vv[q];
  }
  __syncthreads();
  tile_fft<N, true, C2, false>(s, np, 0, stw);
  C2 *dst = out + pair0 * 2 * (size_t)ld;
  constexpr int CC = (VEC && sizeof(C2) == 8) ? 2 : 1;  // complex per store
  const int nchunk = ld / CC;
  for (int c = threadIdx.x; c < np * nchunk; c += 256) {
    const int l = c / nchunk, k0 = (c % nchunk) * CC;
    C2 a[CC], b[CC];
#pragma unroll
    for (int q = 0; q < CC; q++) {
      const int k = k0 + q;
      if (k < NH) {
        const C2 zk = s[LL::at(l, k & (N - 1), 0)];
        const C2 zc = s[LL::at(l, (N - k) & (N - 1), 0)];
        // A_k = (Z_k + conj Z_{N-k})/2, B_k = (Z_k - conj Z_{N-k})/(2i)
        a[q].x = (T)0.5 * (zk.x + zc.x);
        a[q].y = (T)0.5 * (zk.y - zc.y);
        b[q].x = (T)0.5 * (zk.y + zc.y);
        b[q].y = (T)0.5 * (zc.x - zk.x);
      } else {
        a[q].x = a[q].y = b[q].x = b[q].y = (T)0;
      }
    }
    if (CC == 2) {
      *reinterpret_cast<float4 *>(dst + (size_t)(2 * l) * ld + k0) = *reinterpret_cast<float4 *>(a);
      *reinterpret_cast<float4 *>(dst + (size_t)(2 * l + 1) * ld + k0) = *reinterpret_cast<float4 *>(b);
    } else {
      dst[(size_t)(2 * l) * ld + k0] = a[0];
      dst[(size_t)(2 * l + 1) * ld + k0] = b[0];
    }
  }
}

// ---- pass Z inverse: pairs of half spectra -> real lines --------------------
template <typename T, int N, bool VEC>
__global__ void __launch_bounds__(256, sizeof(T) == 4 && N <= 256 ? 4 : 3) fftz_c2r_kernel(const typename Cplx<T>::type *__restrict__ in,
                                                          T *__restrict__ out, size_t npairs, int LP,
                                                          int ld,
                                                          const typename Cplx<T>::type *__restrict__ tw) {
  using C2 = typename Cplx<T>::type;
  using LL = LineLayout<N, true>;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int NH = N / 2 + 1;
  constexpr int RC = 16 / sizeof(T);
  using RV = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
  C2 *stw = reinterpret_cast<C2 *>(smraw);
  C2 *s = stw + N;
  const T *sr = reinterpret_cast<const T *>(s);
  load_twiddles<N>(stw, tw);
  const size_t pair0 = (size_t)blockIdx.x * LP;
  const int np = (int)min((size_t)LP, npairs - pair0);
  const C2 *src = in + pair0 * 2 * (size_t)ld;
  constexpr int CC = (VEC && sizeof(C2) == 8) ? 2 : 1;
  constexpr int NCH = (NH + CC - 1) / CC;  // chunks covering k = 0..N/2
  for (int c = threadIdx.x; c < np * NCH; c += 256) {
    const int l = c / NCH, k0 = (c % NCH) * CC;
    C2 a[CC], b[CC];
    if (CC == 2) {
      *reinterpret_cast<float4 *>(a) = *reinterpret_cast<const float4 *>(src + (size_t)(2 * l) * ld + k0);
      *reinterpret_cast<float4 *>(b) = *reinterpret_cast<const float4 *>(src + (size_t)(2 * l + 1) * ld + k0);
    } else {
      a[0] = src[(size_t)(2 * l) * ld + k0];
      b[0] = src[(size_t)(2 * l + 1) * ld + k0];
    }
#pragma unroll
    for (int q = 0; q < CC; q++) {
      const int k = k0 + q;
      if (k >= NH) continue;
      // Z_k = A_k + i B_k; Z_{N-k} = conj(A_k) + i conj(B_k)
      C2 z;
      z.x = a[q].x - b[q].y;
      z.y = a[q].y + b[q].x;
      s[LL::at(l, k, 0)] = z;
      if (k > 0 && k < N / 2) {
        C2 w;
        w.x = a[q].x + b[q].y;
        w.y = -a[q].y + b[q].x;
        s[LL::at(l, N - k, 0)] = w;
      }
    }
  }
  __syncthreads();
  tile_fft<N, true, C2, true>(s, np, 0, stw);
  T *dst = out + pair0 * 2 * N;
  for (int c = threadIdx.x; c < np * 2 * N / RC; c += 256) {
    const int e = c * RC, rl = e / N, r = e % N;
    RV v;
    T *vv = reinterpret_cast<T *>(&v);
#pragma unroll
    for (int q = 0; q < RC; q++) vv[q] = sr[2 * LL::at(rl >> 1, r + q, 0) + (rl & 1)];
    *reinterpret_cast<RV *>(dst + e) = v;
  }
}

// ---- strided passes: FFT along rows for tiles of W contiguous columns -------
// array: outer blocks of `ostride` elements; inside, rows of `rstride`; ncols
// valid columns per row.  grid.x = nouter * ntiles.  VEC: rows start on
// 16-byte boundaries, so the tile moves in 16-byte chunks.
template <typename C2, int N, int W, bool INV, bool VEC>
__global__ void __launch_bounds__(256, 3) fft_cols_kernel(C2 *__restrict__ a, size_t ostride,
                                                          size_t rstride, size_t ncols,
                                                          int ntiles, const C2 *__restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smraw[];
  C2 *stw = reinterpret_cast<C2 *>(smraw);
  C2 *s = stw + N;
  load_twiddles<N>(stw, tw);
  const size_t outer = blockIdx.x / ntiles;
  const size_t col0 = (size_t)(blockIdx.x % ntiles) * W;
  const int wv = (int)min((size_t)W, ncols - col0);
  C2 *base = a + outer * ostride + col0;
  // complex elements per 16-byte chunk
  constexpr int CPC = (VEC && sizeof(C2) == 8) ? 2 : 1;
  constexpr int CH = W / CPC;  // chunks per row
  using V = typename std::conditional<CPC == 2, float4, C2>::type;
#pragma unroll 4
  for (int e = threadIdx.x; e < N * CH; e += 256) {
    const int r = e / CH, c = (e % CH) * CPC;
    if (c < wv) *reinterpret_cast<V *>(s + r * W + c) = *reinterpret_cast<const V *>(base + (size_t)r * rstride + c);
  }
  __syncthreads();
  // (the last tile of a half spectrum holds one column: its own, not W)
  if (wv == W) tile_fft<N, false, C2, INV>(s, W, W, stw);
  else tile_fft<N, false, C2, INV>(s, wv, W, stw);
#pragma unroll 4
  for (int e = threadIdx.x; e < N * CH; e += 256) {
    const int r = e / CH, c = (e % CH) * CPC;
    if (c < wv) *reinterpret_cast<V *>(base + (size_t)r * rstride + c) = *reinterpret_cast<const V *>(s + r * W + c);
  }
}

// Persistent, double-buffered form of the column pass for 16-byte aligned
// rows: each block walks tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the
// next tile is copied into the second smem buffer with cp.async while the
// current one is transformed and written back.
template <typename C2, int N, int W, bool INV>
__global__ void __launch_bounds__(256, 2) fft_cols_pipe_kernel(C2 *__restrict__ a, size_t ostride,
                                                               size_t rstride, size_t ncols,
                                                               int ntiles, size_t ntot,
                                                               const C2 *__restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smraw[];
  C2 *stw = reinterpret_cast<C2 *>(smraw);
  C2 *buf[2] = {stw + N, stw + N + N * W};
  load_twiddles<N>(stw, tw);
  constexpr int CPC = 16 / sizeof(C2);  // complex per 16-byte chunk
  constexpr int CH = W / CPC;           // chunks per row
  auto issue = [&](size_t tile, C2 *s) {
    const size_t outer = tile / ntiles;
    const size_t col0 = (size_t)(tile % ntiles) * W;
    const int wv = (int)min((size_t)W, ncols - col0);
    const C2 *base = a + outer * ostride + col0;
#pragma unroll 4
    for (int e = threadIdx.x; e < N * CH; e += 256) {
      const int r = e / CH, c = (e % CH) * CPC;
      if (c < wv) cp_async16(s + r * W + c, base + (size_t)r * rstride + c);
    }
  };
  size_t tile = blockIdx.x;
  if (tile < ntot) issue(tile, buf[0]);
  cp_async_commit();
  for (int it = 0; tile < ntot; it++, tile += gridDim.x) {
    C2 *s = buf[it & 1];
    const size_t next = tile + gridDim.x;
    if (next < ntot) issue(next, buf[(it + 1) & 1]);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    tile_fft<N, false, C2, INV>(s, W, W, stw);
    const size_t outer = tile / ntiles;
    const size_t col0 = (size_t)(tile % ntiles) * W;
    const int wv = (int)min((size_t)W, ncols - col0);
    C2 *base = a + outer * ostride + col0;
#pragma unroll 4
    for (int e = threadIdx.x; e < N * CH; e += 256) {
      const int r = e / CH, c = (e % CH) * CPC;
      if (c < wv) *reinterpret_cast<float4 *>(base + (size_t)r * rstride + c) = *reinterpret_cast<const float4 *>(s + r * W + c);
    }
    __syncthreads();  // this buffer is refilled two tiles later
  }
  cp_async_wait<0>();
}

template <typename C2, int N, int W, bool INV>
int launch_pipe(ct2g_ctx *ctx, C2 *spec, size_t nouter, size_t ostride, size_t rstride,
                size_t ncols) {
  const size_t smem = sizeof(C2) * ((size_t)N + 2 * (size_t)N * W);
  auto k = fft_cols_pipe_kernel<C2, N, W, INV>;
  CT2G_TRY(ct2g_smem_attrs(ctx, k, smem));
  int per_sm = 0;
  CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, smem));
  // the query can miss the maximum carveout the attributes ask for: count
  // from the kernel's registers and shared memory as well, keep the larger
  per_sm = std::max(per_sm, ct2g_blocks_per_sm(ctx, (const void *)k, 256, smem));
  const int ntiles = (int)((ncols + W - 1) / W);
  const size_t ntot = nouter * ntiles;
  const size_t grid = std::min(ntot, (size_t)std::max(1, per_sm) * ctx->num_sms);
  k<<<(unsigned)grid, 256, smem, ctx->stream>>>(spec, ostride, rstride, ncols, ntiles, ntot,
                                                twiddle_ptr<C2>(ctx));
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

// ---- y pass with tiles moved by TMA --------------------------------------------
// The same column transform as fft_cols_pipe_kernel on the spectrum's y pass,
// with each tile (N rows x W complex columns of one plane) brought into shared
// memory by one tiled bulk tensor copy and written back by another: a
// persistent block keeps S tiles in flight (S - 1 loading while one is
// transformed), completion through one mbarrier per stage (bounded waits), and
// no thread spends issue slots on addresses or copies.  The tensor map views
// the spectrum as floats [plane][y][2 * ldk * NC]; x coordinates are
// multiples of 2W floats (16-byte aligned), and the last tile of a row reads
// zeros past its end and stores nothing there.
template <int N, int W, bool INV, int S>
__global__ void __launch_bounds__(256, 1) fft_cols_tma_kernel(
    const __grid_constant__ CUtensorMap map, uint32_t ntiles, uint32_t ntot,
    const float2 *__restrict__ tw, uint32_t *__restrict__ status) {
  // the tensor copies need 128-byte aligned shared memory: the tiles start at
  // the first 128-byte boundary of the dynamic region (128 bytes reserved for
  // it), whatever offset the static variables leave that region at
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t pad = (128u - (tc::smem_addr(smraw) & 127u)) & 127u;
  float2 *buf = reinterpret_cast<float2 *>(smraw + pad);  // S tiles of N * W
  float2 *stw = buf + S * N * W;
  __shared__ uint64_t bar[S];
  const int tid = threadIdx.x;
  if (tc::smem_addr(buf) & 127u) {  // not reached: checked before any copy
    if (tid == 0) atomicExch(status, (uint32_t)CT2G_ECUDA);
    return;
  }
  load_twiddles<N>(stw, tw);
  if (tid == 0)
    for (int k = 0; k < S; k++) tc::mbar_init(&bar[k], 1);
  __syncthreads();
  // a tensor copy's box holds at most 256 rows: N = 512 moves as two boxes
  constexpr int NB = (N + 255) / 256, BR = N / NB;
  auto issue = [&](uint32_t t, int k) {  // thread 0
    tc::mbar_arrive_expect_tx(&bar[k], (uint32_t)(N * W * sizeof(float2)));
#pragma unroll
    for (int b = 0; b < NB; b++)
      tc::tma_load_3d(buf + k * N * W + b * BR * W, &map, (int)(2 * W * (t % ntiles)), b * BR,
                      (int)(t / ntiles), &bar[k]);
  };
  uint32_t t = blockIdx.x;
  if (tid == 0)
    for (int k = 0; k < S - 1; k++)
      if (t + k * gridDim.x < ntot) issue(t + k * gridDim.x, k);
  uint32_t parity = 0;
  bool ok = true;
  for (int it = 0; t < ntot; t += gridDim.x, it++) {
    const int k = it % S;
    if (tid == 0) {
      // the next tile goes into the previous tile's stage once its store has
      // read it
      const uint32_t tn = t + (S - 1) * gridDim.x;
      if (tn < ntot) {
        tc::bulk_wait_read();
        issue(tn, (it + S - 1) % S);
      }
    }
    ok = tc::mbar_wait(&bar[k], (parity >> k) & 1u, kTmaWaitLimit);
    parity ^= 1u << k;
    if (!__syncthreads_and(ok)) break;
    float2 *s = buf + k * N * W;
    tile_fft<N, false, float2, INV>(s, W, W, stw);
    tc::fence_async_smem();  // this thread's writes, before the bulk store reads them
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int b = 0; b < NB; b++)
        tc::tma_store_3d(&map, (int)(2 * W * (t % ntiles)), b * BR, (int)(t / ntiles),
                         s + b * BR * W);
      tc::bulk_commit();
    }
  }
  if (tid == 0) {
    if (!ok) {
      atomicExch(status, (uint32_t)CT2G_ETIMEOUT);
      // loads still in flight land before the block's shared memory goes away
      for (int k = 0; k < S; k++) tc::mbar_wait(&bar[k], (parity >> k) & 1u, kTmaWaitLimit);
    }
    tc::bulk_wait_all();
  }
}

// The tensor map of a column pass over complex FP32 data: `nouter` blocks
// (ostride complex apart) of N rows (rstride complex apart), seen as floats
// [outer][row][2 * rstride]; a box is W complex columns x N / NB rows.
int cols_map(ct2g_ctx *ctx, void *base, size_t nouter, size_t ostride, size_t rstride, int N,
             int W, CUtensorMap *m) {
  EncodeTiledFn encode = nullptr;
  CT2G_TRY(tensor_map_encoder(ctx, &encode));
  const cuuint64_t dims[3] = {2 * (cuuint64_t)rstride, (cuuint64_t)N, (cuuint64_t)nouter};
  const cuuint64_t strides[2] = {rstride * sizeof(float2), ostride * sizeof(float2)};
  const cuuint32_t box[3] = {(cuuint32_t)(2 * W), (cuuint32_t)(N > 256 ? 256 : N), 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  if (encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return ct2g_fail(ctx, CT2G_ECUDA, "column-pass tensor map");
  return CT2G_OK;
}

// a column pass (y pass, or an x pass over whole planes) with its tiles moved
// by TMA: N rows x W columns per tile (W 32, or 16 with fft_tile 16 and at
// N = 512), three tiles in flight per block; the data 16-byte aligned with
// rstride and ostride even (the callers' vector condition)
template <int N, bool INV>
int launch_cols_tma(ct2g_ctx *ctx, float2 *data, size_t nouter, size_t ostride, size_t rstride,
                    size_t ncols) {
  if constexpr (N < 64 || N > 512) {
    return ct2g_fail(ctx, CT2G_EINVAL, "TMA column pass: sizes 64-512");
  } else {
    const bool narrow = N > 256 || ctx->fft_tile == 16;
    const int W = narrow ? 16 : 32;
    alignas(64) CUtensorMap map;
    CT2G_TRY(cols_map(ctx, data, nouter, ostride, rstride, N, W, &map));
    const uint32_t ntiles = (uint32_t)((ncols + W - 1) / W), ntot = ntiles * (uint32_t)nouter;
    auto k = fft_cols_tma_kernel<N, 16, INV, 3>;
    if constexpr (N <= 256)
      if (!narrow) k = fft_cols_tma_kernel<N, 32, INV, 3>;
    const size_t smem = sizeof(float2) * (3 * (size_t)N * W + N) + 128;
    CT2G_TRY(ct2g_smem_attrs(ctx, k, smem));
    const int per_sm = ct2g_blocks_per_sm(ctx, (const void *)k, 256, smem);
    const uint32_t grid = std::min(ntot, (uint32_t)(per_sm * ctx->num_sms));
    k<<<grid, 256, smem, ctx->stream>>>(map, ntiles, ntot, twiddle_ptr<float2>(ctx),
                                        ctx->d_counts + 6);
    CT2G_LAUNCHED(ctx);
    return CT2G_OK;
  }
}

// column tile widths: the default W, and W/2 or 2W (FP32 only) when the
// context's tuning asks for them and the double buffer fits in shared memory
template <typename T, int N, bool INV, bool VEC>
int launch_cols(ct2g_ctx *ctx, typename Cplx<T>::type *spec, size_t nouter, size_t ostride,
                size_t rstride, size_t ncols) {
  using C2 = typename Cplx<T>::type;
  if constexpr (sizeof(C2) == 8 && N >= 64 && N <= 512) {
    // FP32 columns with 16-byte aligned rows: tiles moved by TMA (tuning cols_tma)
    if (VEC && ctx->cols_tma)
      return launch_cols_tma<N, INV>(ctx, spec, nouter, ostride, rstride, ncols);
  }
  // 16-column tiles from N = 256 on; FP64 at N = 512 takes 8 so that the
  // double-buffered tile fits in shared memory
  constexpr int W = N >= 256 ? (sizeof(C2) == 16 && N >= 512 ? 8 : 16) : 4096 / N;
  if (VEC && N >= 64) {
    if constexpr (sizeof(C2) == 8) {
      if (ctx->fft_tile == W / 2)
        return launch_pipe<C2, N, W / 2, INV>(ctx, spec, nouter, ostride, rstride, ncols);
      if constexpr (sizeof(C2) * ((size_t)N + 4 * (size_t)N * W) <= 200 * 1024)
        if (ctx->fft_tile == 2 * W)
          return launch_pipe<C2, N, 2 * W, INV>(ctx, spec, nouter, ostride, rstride, ncols);
    }
    return launch_pipe<C2, N, W, INV>(ctx, spec, nouter, ostride, rstride, ncols);
  }
  const size_t smem = sizeof(C2) * ((size_t)N + (size_t)N * W);
  auto k = fft_cols_kernel<C2, N, W, INV, VEC>;
  CT2G_TRY(ct2g_smem_attrs(ctx, k, smem));
  const int ntiles = (int)((ncols + W - 1) / W);
  k<<<(unsigned)(nouter * ntiles), 256, smem, ctx->stream>>>(spec, ostride, rstride, ncols, ntiles,
                                                             twiddle_ptr<C2>(ctx));
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

// Y and X passes over a spectrum whose qk rows hold ld >= N/2+1 elements (a
// half spectrum: the Y pass transforms its first N/2+1 columns) or, `full`,
// N elements (a complex grid: every column)
template <typename T, int N>
int run_cols(ct2g_ctx *ctx, typename Cplx<T>::type *spec, int batch, bool inv, size_t ld,
             bool full = false) {
  using C2 = typename Cplx<T>::type;
  const size_t NH = full ? (size_t)N : (size_t)N / 2 + 1;
  for (int pass = 0; pass < 2; pass++) {
    const bool ypass = (pass == 0) != inv;
    size_t nouter, ostride, rstride, ncols;
    if (ypass) {
      nouter = (size_t)batch * N;
      ostride = (size_t)N * ld;
      rstride = ld;
      ncols = NH;
    } else {
      nouter = (size_t)batch;
      ostride = (size_t)N * N * ld;
      rstride = (size_t)N * ld;
      ncols = (size_t)N * ld;
    }
    // rows on 16-byte boundaries: the x pass's always are (N rows of ld values
    // apart), the y pass's where ld is even (FP32), if the grid itself is.  (The x
    // passes of 3 x 256^3 half spectra moved their tiles by plain 8-byte loads like the
    // y passes, 117 us each; by TMA 74 us.  Feeding the y passes by 8-byte cp.async
    // or in tiles of 32 columns measured 136 and 119 us.)
    const bool vec = (rstride * sizeof(C2)) % 16 == 0 && ((uintptr_t)spec & 15) == 0;
    if constexpr (sizeof(C2) == 8 && (N == 256 || N == 512)) {
      if (ctx->fft_tc) {
        CT2G_TRY(ct2g_fft_cols_tc(ctx, spec, N, nouter, ostride, rstride, ncols, inv));
        continue;
      }
    }
    if (inv) {
      if (vec) CT2G_TRY((launch_cols<T, N, true, true>(ctx, spec, nouter, ostride, rstride, ncols)));
      else CT2G_TRY((launch_cols<T, N, true, false>(ctx, spec, nouter, ostride, rstride, ncols)));
    } else {
      if (vec) CT2G_TRY((launch_cols<T, N, false, true>(ctx, spec, nouter, ostride, rstride, ncols)));
      else CT2G_TRY((launch_cols<T, N, false, false>(ctx, spec, nouter, ostride, rstride, ncols)));
    }
  }
  return CT2G_OK;
}

template <typename T, int N>
int fft_r2c_n(ct2g_ctx *ctx, const T *in, typename Cplx<T>::type *out, int batch, int ld) {
  using C2 = typename Cplx<T>::type;
  const size_t npairs = (size_t)batch * N * N / 2;
  const int LP = std::max(1, 4096 / N);
  const size_t smem = sizeof(C2) * ((size_t)N + (size_t)LP * LineLayout<N, true>::LS);
  const bool vec = ((size_t)ld * sizeof(C2)) % 16 == 0;
  auto kern = vec ? fftz_r2c_kernel<T, N, true> : fftz_r2c_kernel<T, N, false>;
  CT2G_TRY(ct2g_smem_attrs(ctx, kern, smem));
  kern<<<ct2g_div_up(npairs, LP), 256, smem, ctx->stream>>>(in, out, npairs, LP, ld,
                                                            twiddle_ptr<C2>(ctx));
  CT2G_LAUNCHED(ctx);
  return run_cols<T, N>(ctx, out, batch, false, ld);
}

template <typename T, int N>
int fft_c2r_n(ct2g_ctx *ctx, typename Cplx<T>::type *in, T *out, int batch, int ld) {
  using C2 = typename Cplx<T>::type;
  CT2G_TRY((run_cols<T, N>(ctx, in, batch, true, ld)));
  const size_t npairs = (size_t)batch * N * N / 2;
  const int LP = std::max(1, 4096 / N);
  const size_t smem = sizeof(C2) * ((size_t)N + (size_t)LP * LineLayout<N, true>::LS);
  const bool vec = ((size_t)ld * sizeof(C2)) % 16 == 0;
  auto kern = vec ? fftz_c2r_kernel<T, N, true> : fftz_c2r_kernel<T, N, false>;
  CT2G_TRY(ct2g_smem_attrs(ctx, kern, smem));
  kern<<<ct2g_div_up(npairs, LP), 256, smem, ctx->stream>>>(in, out, npairs, LP, ld,
                                                            twiddle_ptr<C2>(ctx));
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

template <typename T>
int fft_r2c(ct2g_ctx *ctx, const T *in, typename Cplx<T>::type *out, int N, int batch, int ld) {
  CT2G_TRY(ct2g_twiddles(ctx, N));
  switch (N) {
    case 4: return fft_r2c_n<T, 4>(ctx, in, out, batch, ld);
    case 8: return fft_r2c_n<T, 8>(ctx, in, out, batch, ld);
    case 16: return fft_r2c_n<T, 16>(ctx, in, out, batch, ld);
    case 32: return fft_r2c_n<T, 32>(ctx, in, out, batch, ld);
    case 64: return fft_r2c_n<T, 64>(ctx, in, out, batch, ld);
    case 128: return fft_r2c_n<T, 128>(ctx, in, out, batch, ld);
    case 256: return fft_r2c_n<T, 256>(ctx, in, out, batch, ld);
    case 512: return fft_r2c_n<T, 512>(ctx, in, out, batch, ld);
  }
  return ct2g_fail(ctx, CT2G_EINVAL, "FFT size must be a power of two in [4, 512]");
}

template <typename T>
int fft_c2r(ct2g_ctx *ctx, typename Cplx<T>::type *in, T *out, int N, int batch, int ld) {
  CT2G_TRY(ct2g_twiddles(ctx, N));
  switch (N) {
    case 4: return fft_c2r_n<T, 4>(ctx, in, out, batch, ld);
    case 8: return fft_c2r_n<T, 8>(ctx, in, out, batch, ld);
    case 16: return fft_c2r_n<T, 16>(ctx, in, out, batch, ld);
    case 32: return fft_c2r_n<T, 32>(ctx, in, out, batch, ld);
    case 64: return fft_c2r_n<T, 64>(ctx, in, out, batch, ld);
    case 128: return fft_c2r_n<T, 128>(ctx, in, out, batch, ld);
    case 256: return fft_c2r_n<T, 256>(ctx, in, out, batch, ld);
    case 512: return fft_c2r_n<T, 512>(ctx, in, out, batch, ld);
  }
  return ct2g_fail(ctx, CT2G_EINVAL, "FFT size must be a power of two in [4, 512]");
}

// ---- complex-to-complex 3D FFT ------------------------------------------------
// Pass Z of a complex grid a[b][i][j][k] (k contiguous, N per row): LP rows
// per block through shared memory, moved in 16-byte chunks (two complex
// values); the Y and X passes are the column passes of the real transforms
// over every column (run_cols, `full`).
template <int N, bool INV>
__global__ void __launch_bounds__(256, 3) fftz_c2c_kernel(float2 *__restrict__ a, size_t nrows,
                                                          int LP, const float2 *__restrict__ tw) {
  using LL = LineLayout<N, true>;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *stw = reinterpret_cast<float2 *>(smraw);
  float2 *s = stw + N;
  load_twiddles<N>(stw, tw);
  const size_t row0 = (size_t)blockIdx.x * LP;
  const int nr = (int)min((size_t)LP, nrows - row0);
  float2 *g = a + row0 * N;
  for (int c = threadIdx.x; c < nr * N / 2; c += 256) {
    const int e = 2 * c, l = e / N, r = e % N;
    const float4 v = *reinterpret_cast<const float4 *>(g + e);
    s[LL::at(l, r, 0)] = make_float2(v.x, v.y);
    s[LL::at(l, r + 1, 0)] = make_float2(v.z, v.w);
  }
  __syncthreads();
  tile_fft<N, true, float2, INV>(s, nr, 0, stw);
  for (int c = threadIdx.x; c < nr * N / 2; c += 256) {
    const int e = 2 * c, l = e / N, r = e % N;
    const float2 u = s[LL::at(l, r, 0)], w = s[LL::at(l, r + 1, 0)];
    *reinterpret_cast<float4 *>(g + e) = make_float4(u.x, u.y, w.x, w.y);
  }
}

template <int N>
int fft_c2c_n(ct2g_ctx *ctx, float2 *a, int batch, bool inv) {
  const size_t nrows = (size_t)batch * N * N;
  const int LP = std::max(1, 4096 / N);
  const size_t smem = sizeof(float2) * ((size_t)N + (size_t)LP * LineLayout<N, true>::LS);
  auto kern = inv ? fftz_c2c_kernel<N, true> : fftz_c2c_kernel<N, false>;
  if (inv) CT2G_TRY((run_cols<float, N>(ctx, a, batch, true, N, true)));
  CT2G_TRY(ct2g_smem_attrs(ctx, kern, smem));
  kern<<<ct2g_div_up(nrows, LP), 256, smem, ctx->stream>>>(a, nrows, LP, twiddle_ptr<float2>(ctx));
  CT2G_LAUNCHED(ctx);
  if (!inv) CT2G_TRY((run_cols<float, N>(ctx, a, batch, false, N, true)));
  return CT2G_OK;
}

int fft_c2c(ct2g_ctx *ctx, float2 *a, int N, int batch, bool inv) {
  CT2G_TRY(ct2g_twiddles(ctx, N));
  switch (N) {
    case 4: return fft_c2c_n<4>(ctx, a, batch, inv);
    case 8: return fft_c2c_n<8>(ctx, a, batch, inv);
    case 16: return fft_c2c_n<16>(ctx, a, batch, inv);
    case 32: return fft_c2c_n<32>(ctx, a, batch, inv);
    case 64: return fft_c2c_n<64>(ctx, a, batch, inv);
    case 128: return fft_c2c_n<128>(ctx, a, batch, inv);
    case 256: return fft_c2c_n<256>(ctx, a, batch, inv);
    case 512: return fft_c2c_n<512>(ctx, a, batch, inv);
  }
  return ct2g_fail(ctx, CT2G_EINVAL, "FFT size must be a power of two in [4, 512]");
}

}  // namespace

extern const Ct2gOrderFns ct2g_order_fns_p1, ct2g_order_fns_p2, ct2g_order_fns_p3,
    ct2g_order_fns_p4, ct2g_order_fns_p5, ct2g_order_fns_p6;

namespace {

// the mesh-solve kernels of order p (1 .. CT2G_MAX_ORDER)
const Ct2gOrderFns &order_fns(int p) {
  static const Ct2gOrderFns *const f[] = {&ct2g_order_fns_p1, &ct2g_order_fns_p2,
                                          &ct2g_order_fns_p3, &ct2g_order_fns_p4,
                                          &ct2g_order_fns_p5, &ct2g_order_fns_p6};
  return *f[p - 1];
}

// the Y pass (tiles of the (qk, c) columns of each (box, qi) plane) or the
// split X pass (tiles of the (qj, qk, c) columns of each box)
template <int N>
int spec_cols(ct2g_ctx *ctx, bool inv, bool xpass) {
  const size_t RS = (size_t)ctx->ldk * ctx->nc, nb = (size_t)ctx->nbox;
  size_t nouter, ostride, rstride, ncols;
  if (!xpass) {
    nouter = nb * N;
    ostride = (size_t)N * RS;
    rstride = RS;
    ncols = (size_t)(N / 2 + 1) * ctx->nc;
  } else {
    nouter = nb;
    ostride = (size_t)N * N * RS;
    rstride = (size_t)N * RS;
    ncols = (size_t)N * RS;
  }
  if constexpr (N == 256 || N == 512) {
    if (ctx->fft_tc)
      return ct2g_fft_cols_tc(ctx, ctx->spec, N, nouter, ostride, rstride, ncols, inv);
  }
  if (inv) return launch_cols<float, N, true, true>(ctx, ctx->spec, nouter, ostride, rstride, ncols);
  return launch_cols<float, N, false, true>(ctx, ctx->spec, nouter, ostride, rstride, ncols);
}

int spec_cols_n(ct2g_ctx *ctx, bool inv, bool xpass) {
  switch (ctx->M) {
    case 8: return spec_cols<8>(ctx, inv, xpass);
    case 16: return spec_cols<16>(ctx, inv, xpass);
    case 32: return spec_cols<32>(ctx, inv, xpass);
    case 64: return spec_cols<64>(ctx, inv, xpass);
    case 128: return spec_cols<128>(ctx, inv, xpass);
    case 256: return spec_cols<256>(ctx, inv, xpass);
    case 512: return spec_cols<512>(ctx, inv, xpass);
  }
  return ct2g_fail(ctx, CT2G_EINVAL, "mesh must be a power of two in [8, 512]");
}

// stage 0: z pass (mode: CT2G_P2M_*); 1: fused X + MG2L; 2: inverse
// z pass (mode 0/1/2 as fftz_c2r_l2p_kernel); 3: Y pass (mode 0) or X pass
// (mode 1), inverse when flag
int spec_run(ct2g_ctx *ctx, int stage, bool flag, int mode) {
  if (stage == 3) return spec_cols_n(ctx, flag, mode != 0);
  return order_fns(ctx->p).stage(ctx, stage, mode);
}

// the z and y passes of one direction as the plane pipeline, when the
// context's configuration has one (*done tells)
int spec_pipe(ct2g_ctx *ctx, bool inverse, int mode, bool *done) {
  return order_fns(ctx->p).pipe(ctx, inverse, mode, done);
}

}  // namespace

// constant twiddles of the in-register DFTs, once per context (device), in this
// file and in those of the orders
int ct2g_fft_init(ct2g_ctx *ctx) {
  CT2G_TRY(set_consts(ctx));
  for (int p = 1; p <= CT2G_MAX_ORDER; p++) CT2G_TRY(order_fns(p).consts(ctx));
  return CT2G_OK;
}

// twiddles exp(-2 pi i k/N), k < N, computed on the host in FP64
int ct2g_twiddles(ct2g_ctx *ctx, int N) {
  if (ctx->tw_n == N) return CT2G_OK;
  if (ctx->capturing) return ct2g_fail(ctx, CT2G_ESTATE, "FFT twiddles not set up before recording");
  ctx->epoch++;  // twiddle pointers are part of a recorded graph
  if (ctx->tw32) cudaFree(ctx->tw32);
  if (ctx->tw64) cudaFree(ctx->tw64);
  ctx->tw32 = nullptr;
  ctx->tw64 = nullptr;
  ctx->tw_n = 0;
  std::vector<float2> t32(N);
  std::vector<double2> t64(N);
  const double twopi = 6.283185307179586476925286766559;
  for (int k = 0; k < N; k++) {
    const double a = -twopi * (double)k / (double)N;
    t64[k] = make_double2(std::cos(a), std::sin(a));
    t32[k] = make_float2((float)t64[k].x, (float)t64[k].y);
  }
  CT2G_CUDA(ctx, cudaMalloc(&ctx->tw32, sizeof(float2) * N));
  CT2G_CUDA(ctx, cudaMalloc(&ctx->tw64, sizeof(double2) * N));
  CT2G_CUDA(ctx, cudaMemcpyAsync(ctx->tw32, t32.data(), sizeof(float2) * N,
                                 cudaMemcpyHostToDevice, ctx->stream));
  CT2G_CUDA(ctx, cudaMemcpyAsync(ctx->tw64, t64.data(), sizeof(double2) * N,
                                 cudaMemcpyHostToDevice, ctx->stream));
  CT2G_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->tw_n = N;
  return CT2G_OK;
}

int ct2g_fft_r2c_f32(ct2g_ctx *ctx, const float *in, float2 *out, int N, int batch, int ld) {
  return fft_r2c<float>(ctx, in, out, N, batch, ld);
}
int ct2g_fft_c2r_f32(ct2g_ctx *ctx, float2 *in, float *out, int N, int batch, int ld) {
  return fft_c2r<float>(ctx, in, out, N, batch, ld);
}
int ct2g_fft_c2c_f32(ct2g_ctx *ctx, float2 *a, int N, int batch, bool inv) {
  return fft_c2c(ctx, a, N, batch, inv);
}
int ct2g_fft_r2c_f64(ct2g_ctx *ctx, const double *in, double2 *out, int N, int batch, int ld) {
  return fft_r2c<double>(ctx, in, out, N, batch, ld);
}
int ct2g_fft_c2r_f64(ct2g_ctx *ctx, double2 *in, double *out, int N, int batch, int ld) {
  return fft_c2r<double>(ctx, in, out, N, batch, ld);
}

bool ct2g_mg2l_fused(const ct2g_ctx *ctx) {
  if (ctx->fft_tc || ctx->split_mg2l || !ctx->greens_x) return false;
  return order_fns(ctx->p).fx_fits(ctx->M);
}

// z pass (P2M inside it, or from the moment grid), Y pass, X pass when split
int ct2g_spec_forward(ct2g_ctx *ctx, int src) {
  CT2G_TRY(ct2g_twiddles(ctx, ctx->M));
  bool piped = false;
  CT2G_TRY(spec_pipe(ctx, false, src, &piped));
  if (!piped) {
    // P2M into compact per-cell records first, read by the z pass
    if (src == CT2G_P2M_FUSED && ctx->p2m_compact && ctx->cmom) src = CT2G_P2M_COMPACT;
    CT2G_TRY(spec_run(ctx, 0, false, src));
    CT2G_TRY(spec_run(ctx, 3, false, 0));
  }
  if (!ct2g_mg2l_fused(ctx)) CT2G_TRY(spec_run(ctx, 3, false, 1));
  return CT2G_OK;
}

int ct2g_spec_mg2l(ct2g_ctx *ctx) {
  if (ct2g_mg2l_fused(ctx)) return spec_run(ctx, 1, false, 0);
  return ct2g_mg2l_split(ctx);
}

// inverse X pass when split, Y pass, z pass (L2P inside it, or into the
// expansion grid)
int ct2g_spec_inverse(ct2g_ctx *ctx, bool l2p, bool pot) {
  CT2G_TRY(ct2g_twiddles(ctx, ctx->M));
  if (!ct2g_mg2l_fused(ctx)) CT2G_TRY(spec_run(ctx, 3, true, 1));
  const int mode = l2p ? (pot ? 1 : 0) : 2;
  bool piped = false;
  CT2G_TRY(spec_pipe(ctx, true, mode, &piped));
  if (piped) return CT2G_OK;
  CT2G_TRY(spec_run(ctx, 3, true, 0));
  return spec_run(ctx, 2, false, mode);
}
