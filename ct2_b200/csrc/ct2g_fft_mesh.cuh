// The mesh solve's z and x passes (with P2M, MG2L and L2P) and its plane
// pipeline, templates over the order and the mesh; each order is compiled in a
// file of its own (ct2g_fft_p1.cu ... p6.cu).
#pragma once

#include <type_traits>
#include <utility>

#include "ct2g_fft_core.cuh"

namespace {

// ---- the mesh solve's spectrum ------------------------------------------------
// ctx->spec keeps the NC components of a k-point side by side,
// [box][qi][qj][qk][NC] with qk < ldk, so that a (qi, qj) row is RS = ldk*NC
// complex values (16-byte aligned rows: ldk is even; slots qk > N/2 hold
// zeros).  The z passes write and read whole rows; the Y pass transforms tiles
// of W contiguous (qk, c) columns; the X pass runs inside the MG2L kernel,
// whose block holds every component of one (qj, qk) column.

// (x, y) lines per block of a z pass that reads or writes the moment grid:
// enough packed lines for a block's transform to fill its threads (one line
// when the components alone give 16 packed lines or more)
template <int P>
constexpr int z_lines() {
  constexpr int NL = (ct2g_ncomp(P) + 1) / 2;
  return NL >= 8 ? 1 : NL >= 4 ? 2 : NL >= 2 ? 4 : 8;
}

// ---- forward z pass fused with P2M -----------------------------------------
// One block per (x, y) line of one box: the moments of the line's N cells
// (FP64 sums about the cell centres, as p2m_kernel) go straight into shared
// memory as FP32, components paired into complex lines (2l -> .x, 2l+1 ->
// .y), are transformed along z and split into the half spectra of the two
// components.  The moment grid is never written to HBM.  A thread sums a
// cell of up to kWarpCell particles; bigger cells are summed by a warp
// (lanes stride over the particles, partial moments reduced by shuffles), so
// no block waits on one thread's long loop: a thread's FP64 sums are a serial
// chain, and a block's transform waits for its slowest cell.  GRID: the moments are read from
// the moment grid (component k of box b at grid + (k * nbox + b) * N^3).
constexpr uint32_t kWarpCell = 6;
constexpr uint32_t kBlockCell = 256;

// components [K0, K1) of one particle's moments about the cell centre u
template <int P, int K0, int K1>
__device__ __forceinline__ void p2m_accumulate(const uint32_t *__restrict__ px,
                                               const uint32_t *__restrict__ py,
                                               const uint32_t *__restrict__ pz, uint32_t i,
                                               uint32_t ux, uint32_t uy, uint32_t uz,
                                               double *acc) {
  constexpr MiTable<P> T{};
  const double sx = -(double)(int32_t)(px[i] - ux) * CT2G_TWO_M32;
  const double sy = -(double)(int32_t)(py[i] - uy) * CT2G_TWO_M32;
  const double sz = -(double)(int32_t)(pz[i] - uz) * CT2G_TWO_M32;
  double qx[P + 1], qy[P + 1], qz[P + 1];
  qx[0] = qy[0] = qz[0] = 1.0;
#pragma unroll
  for (int q = 1; q <= P; q++) {
    qx[q] = qx[q - 1] * sx * (1.0 / q);
    qy[q] = qy[q - 1] * sy * (1.0 / q);
    qz[q] = qz[q - 1] * sz * (1.0 / q);
  }
#pragma unroll
  for (int k = K0; k < K1; k++) acc[k - K0] += qx[T.nx[k]] * qy[T.ny[k]] * qz[T.nz[k]];
}

// v[k] summed over the warp, k < K <= 32: each lane ends with the sum of the one k
// it returns (-1: none) in v[0].  At each step a lane hands half of its values to
// its partner and adds what it is handed to the others, so K values take about
// K + 4 exchanges instead of 5 K (each two shuffles, the pipe that held a warp's
// cell); each sum is the same tree as a butterfly per value.
template <int K>
__device__ __forceinline__ int warp_sums(double (&v)[K], int lane) {
  static_assert(K <= 32, "a value per lane at most");
  int base = 0, cnt = K;
#pragma unroll
  for (int s = 0; s < 5; s++) {
    const int n = (K + (1 << s) - 1) >> s, h = (n + 1) >> 1, o = 16 >> s;
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < (K + 1) / 2; k++) {
      if (k < h) {
        const double lo = v[k], hi = k + h < n ? v[k + h < K ? k + h : 0] : 0.0;
        v[k] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
      }
    }
    base += up ? h : 0;
    cnt = up ? max(cnt - h, 0) : min(cnt, h);
  }
  return cnt > 0 ? base : -1;
}

// the moments of cell particles b, b + step, ... < e (a thread: step 1; a
// warp: lane offset, step 32 or more, then summed over the warp) for components
// [K0, K1): the components go in pieces so that only one's FP64 sums are live at
// once.  st(k, sum) by the lane that has it.
template <int P, int K0, int K1, typename ST>
__device__ __forceinline__ void p2m_sum(const uint32_t *__restrict__ px,
                                        const uint32_t *__restrict__ py,
                                        const uint32_t *__restrict__ pz, uint32_t b, uint32_t e,
                                        uint32_t step, bool warp_sum, int lane, uint32_t ux,
                                        uint32_t uy, uint32_t uz, ST st) {
  double acc[K1 - K0];
#pragma unroll
  for (int k = 0; k < K1 - K0; k++) acc[k] = 0.0;
  for (uint32_t i = b; i < e; i += step) p2m_accumulate<P, K0, K1>(px, py, pz, i, ux, uy, uz, acc);
  if (warp_sum) {
    const int k = warp_sums<K1 - K0>(acc, lane);
    if (k >= 0) st(K0 + k, acc[0]);
  } else {
#pragma unroll
    for (int k = K0; k < K1; k++) st(k, acc[k - K0]);
  }
}

// f(0), f(1), ... of NP pieces, as compile-time constants
template <typename F, int... I>
__device__ __forceinline__ void each_piece(F f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}

// all the components in NP pieces; st(piece, k, sum)
template <int P, int NP, typename ST>
__device__ __forceinline__ void p2m_all(const uint32_t *__restrict__ px,
                                        const uint32_t *__restrict__ py,
                                        const uint32_t *__restrict__ pz, uint32_t b, uint32_t e,
                                        uint32_t step, bool warp_sum, int lane, uint32_t ux,
                                        uint32_t uy, uint32_t uz, ST st) {
  constexpr int NC = ct2g_ncomp(P);
  each_piece(
      [&](auto i) {
        constexpr int I = decltype(i)::value;
        p2m_sum<P, I * NC / NP, (I + 1) * NC / NP>(px, py, pz, b, e, step, warp_sum, lane, ux, uy,
                                                   uz, [&](int k, double v) { st(I, k, v); });
      },
      std::make_integer_sequence<int, NP>{});
}

// ---- P2M into compact per-cell records ---------------------------------------
// The moments of every occupied cell (the same FP64 sums about the cell
// centre as the fused z pass, term for term, stored FP32) as NC floats at
// cmom + rank * NC, where rank is the cell's index among the occupied cells
// in key order: blk_rank[block] (an exclusive scan of the occupancy words'
// populations) plus the occupied cells before it in its 4x4x4 block's word.
// A thread per particle of the binned range: the first particle of each
// cell's run (in the sorted keys) sums the cell; cells of more than
// kWarpCell particles are listed (by key) for p2m_compact_big_kernel, a warp
// each.  The z pass then reads the records instead of summing particles, so
// its blocks no longer wait on the slowest cell of a line.
__device__ __forceinline__ uint32_t occ_rank(const unsigned long long *__restrict__ occ,
                                             const uint32_t *__restrict__ blk_rank, uint32_t key,
                                             bool &on) {
  const unsigned long long w = occ[key >> 6];
  on = (w >> (key & 63u)) & 1ull;
  return blk_rank[key >> 6] + (uint32_t)__popcll(w & ((1ull << (key & 63u)) - 1ull));
}

__global__ void occ_popc_kernel(const unsigned long long *__restrict__ occ, size_t nw,
                                uint32_t *__restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nw) out[i] = (uint32_t)__popcll(occ[i]);
}

// the cell coordinates of a Morton key's low 3 * mbits bits (the inverse of
// ct2g_morton: bit 3b + 2 is x's bit b, 3b + 1 y's, 3b z's)
__device__ __forceinline__ void demorton(uint32_t key, int mbits, uint32_t &x, uint32_t &y,
                                         uint32_t &z) {
  x = y = z = 0;
  for (int b = 0; b < mbits; b++) {
    z |= ((key >> (3 * b)) & 1u) << b;
    y |= ((key >> (3 * b + 1)) & 1u) << b;
    x |= ((key >> (3 * b + 2)) & 1u) << b;
  }
}

// the moments of the cell `key` (particles b .. e) into out (a thread: step
// 1; a warp: lanes strided, summed over the warp)
template <int P>
__device__ __forceinline__ void p2m_cell(const uint32_t *__restrict__ px,
                                         const uint32_t *__restrict__ py,
                                         const uint32_t *__restrict__ pz, uint32_t key, int mbits,
                                         uint32_t b, uint32_t e, bool warp, int lane,
                                         float *out) {
  uint32_t cx, cy, cz;
  demorton(key, mbits, cx, cy, cz);
  const int sh = 32 - mbits;
  const uint32_t halfc = 1u << (sh - 1);
  const uint32_t ux = (cx << sh) + halfc, uy = (cy << sh) + halfc, uz = (cz << sh) + halfc;
  p2m_all<P, 3>(px, py, pz, warp ? b + (uint32_t)lane : b, e, warp ? 32u : 1u, warp, lane, ux, uy,
                uz, [&](int, int k, double v) { out[k] = (float)v; });
}

// a thread per particle j of the range (absolute index rbegin + j, key
// skeys[j]); the first of its cell's run sums the cell
template <int P>
__global__ void __launch_bounds__(256) p2m_compact_kernel(
    const uint32_t *__restrict__ px, const uint32_t *__restrict__ py,
    const uint32_t *__restrict__ pz, const uint32_t *__restrict__ cs,
    const unsigned long long *__restrict__ occ, const uint32_t *__restrict__ blk_rank, int mbits,
    const uint32_t *__restrict__ skeys, uint32_t rbegin, uint32_t nr, float *__restrict__ cmom,
    uint32_t *__restrict__ big) {
  const uint32_t j = blockIdx.x * 256 + threadIdx.x;
  if (j >= nr) return;
  const uint32_t key = skeys[j];
  if (j > 0 && skeys[j - 1] == key) return;  // not the first of its cell
  const uint32_t b = rbegin + j, e = cs[key + 1];
  if (e - b > kWarpCell) {
    big[1 + atomicAdd(big, 1u)] = key;
    return;
  }
  bool on;
  float *out = cmom + (size_t)occ_rank(occ, blk_rank, key, on) * ct2g_ncomp(P);
  p2m_cell<P>(px, py, pz, key, mbits, b, e, false, 0, out);
}

template <int P>
__global__ void __launch_bounds__(256) p2m_compact_big_kernel(
    const uint32_t *__restrict__ px, const uint32_t *__restrict__ py,
    const uint32_t *__restrict__ pz, const uint32_t *__restrict__ cs,
    const unsigned long long *__restrict__ occ, const uint32_t *__restrict__ blk_rank, int mbits,
    float *__restrict__ cmom, const uint32_t *__restrict__ big) {
  const uint32_t nbig = big[0];
  const int lane = threadIdx.x & 31;
  for (uint32_t q = (blockIdx.x * 256 + threadIdx.x) >> 5; q < nbig; q += gridDim.x * 8) {
    const uint32_t key = big[1 + q];
    bool on;
    float *out = cmom + (size_t)occ_rank(occ, blk_rank, key, on) * ct2g_ncomp(P);
    const uint32_t b = cs[key], e = cs[key + 1];
    if (e - b <= kBlockCell) {
      p2m_cell<P>(px, py, pz, key, mbits, b, e, true, lane, out);
      continue;
    }
    // a crowded cell: the parts that the fused pass gives its eight warps, one
    // after another, added in the same order (each lane its components, one a piece)
    uint32_t cx, cy, cz;
    demorton(key, mbits, cx, cy, cz);
    const int sh = 32 - mbits;
    const uint32_t halfc = 1u << (sh - 1);
    double acc[3] = {0.0, 0.0, 0.0};
    int at[3] = {-1, -1, -1};
    for (uint32_t v = 0; v < 8; v++)
      p2m_all<P, 3>(px, py, pz, b + 32u * v + (uint32_t)lane, e, 256, true, lane,
                    (cx << sh) + halfc, (cy << sh) + halfc, (cz << sh) + halfc,
                    [&](int piece, int k, double w) {
                      acc[piece] += w;
                      at[piece] = k;
                    });
#pragma unroll
    for (int q3 = 0; q3 < 3; q3++)
      if (at[q3] >= 0) out[at[q3]] = (float)acc[q3];
  }
}

// The moments of the N cells of line `line` (x * N + y) of box `box`, from
// the particles, into the packed smem lines sr (line l = components 2l, 2l+1
// as .x, .y).  Ends with the block synchronised.
// The pieces of the components: at N = 256 a thread has a cell and three pieces fit
// the registers of 4 blocks per SM.  Shorter lines leave threads without a cell, so
// the pieces are dealt to groups of N threads (4 pieces, 2 or 4 groups); 6 at order 6
// for its registers.  With warp_sums and 3 blocks per SM instead of 2 at orders 5 and
// 6: 12 boxes of a 64^3 mesh, order 5, 620 -> 447 us; one such mesh 69 -> 52; 64^3,
// order 4, 41 -> 31; 256^3 (warp_sums alone) 1105 -> 1080.
template <int P, int N>
constexpr int p2m_pieces() {
  return N >= 256 ? 3 : P <= 5 ? 4 : 6;
}
template <int P, int N>
struct P2mSmem {
  uint32_t big[N];        // cells for a warp from the front, for the block from the back
  uint32_t nbig, ncrowd;  // zero on entry
  double part[8][ct2g_ncomp(P)];  // a crowded cell's parts
};
template <int P, int N>
__device__ __forceinline__ void p2m_line(const uint32_t *__restrict__ px,
                                         const uint32_t *__restrict__ py,
                                         const uint32_t *__restrict__ pz,
                                         const uint32_t *__restrict__ cs, int mbits, uint32_t box,
                                         size_t line, float *sr, P2mSmem<P, N> &sm) {
  using LL = LineLayout<N, true>;
  constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2;
  const uint32_t cx = (uint32_t)(line / N), cy = (uint32_t)(line % N);
  const int sh = 32 - mbits;
  const uint32_t halfc = 1u << (sh - 1);
  const uint32_t ux = (cx << sh) + halfc, uy = (cy << sh) + halfc;
  // lines of fewer cells than threads: GW threads' worth of cells, the pieces dealt
  // to TG such groups
  constexpr int NP = p2m_pieces<P, N>(), GW = N < 32 ? 32 : N;
  constexpr int TG = 256 / GW < 1 ? 1 : 256 / GW < NP ? 256 / GW : NP;
  const int tg = TG == 1 ? 0 : (int)threadIdx.x / GW;
  for (int zc = TG == 1 ? threadIdx.x : threadIdx.x % GW; zc < N && tg < TG; zc += 256) {
    const uint32_t key = (box << (3 * mbits)) | ct2g_morton(cx, cy, (uint32_t)zc);
    const uint32_t b = cs[key], e = cs[key + 1];
    if (e - b > kWarpCell) {
      if (tg) continue;
      if (e - b > kBlockCell)
        sm.big[N - 1 - atomicAdd(&sm.ncrowd, 1u)] = (uint32_t)zc;
      else
        sm.big[atomicAdd(&sm.nbig, 1u)] = (uint32_t)zc;
      continue;
    }
    const uint32_t uz = ((uint32_t)zc << sh) + halfc;
    each_piece(
        [&](auto i) {
          constexpr int I = decltype(i)::value;
          if (I % TG == tg)
            p2m_sum<P, I * NC / NP, (I + 1) * NC / NP>(
                px, py, pz, b, e, 1, false, 0, ux, uy, uz, [&](int k, double v) {
                  sr[2 * LL::at(k >> 1, zc, 0) + (k & 1)] = (float)v;
                });
        },
        std::make_integer_sequence<int, NP>{});
    if ((NC & 1) && tg == 0) sr[2 * LL::at(NL - 1, zc, 0) + 1] = 0.f;
  }
  __syncthreads();
  {  // the big cells, a warp each, then the crowded ones, a part per warp: one loop
     // with one copy of the sums (two copies, the crowded one's out of line, cost the
     // pass registers: mesh 256, 128^3 particles, 1164 us; 1105 so; 980 -> 930 with
     // 2.5 M in halos)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nbig = sm.nbig, rounds = (nbig + 7) / 8;
    for (uint32_t q = 0; q < rounds + sm.ncrowd; q++) {
      const bool crowd = q >= rounds;
      const uint32_t at = crowd ? N - 1 - (q - rounds) : 8 * q + (uint32_t)warp;
      uint32_t zc = 0;
      if (crowd || at < nbig) {
        zc = sm.big[at];
        const uint32_t key = (box << (3 * mbits)) | ct2g_morton(cx, cy, zc);
        const uint32_t b = cs[key] + (uint32_t)lane + (crowd ? 32u * (uint32_t)warp : 0u),
                       e = cs[key + 1], step = crowd ? 256u : 32u;
        const uint32_t uz = (zc << sh) + halfc;
        auto st = [&](int, int k, double v) {
          if (crowd) sm.part[warp][k] = v;
          else sr[2 * LL::at(k >> 1, (int)zc, 0) + (k & 1)] = (float)v;
        };
        p2m_all<P, (N < 256 && P > 4) ? NP : 3>(px, py, pz, b, e, step, true, lane, ux, uy, uz,
                                                st);
        if ((NC & 1) && lane == 0 && !crowd) sr[2 * LL::at(NL - 1, (int)zc, 0) + 1] = 0.f;
      }
      if (crowd) {  // the parts added in order
        __syncthreads();
        for (int k = threadIdx.x; k < 2 * NL; k += 256) {
          double acc = 0.0;
          if (k < NC)
            for (int v = 0; v < 8; v++) acc += sm.part[v][k];
          sr[2 * LL::at(k >> 1, (int)zc, 0) + (k & 1)] = (float)acc;
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
}

// The moments of the N cells of line `line` of box `box` from the compact
// per-cell records (zeros for empty cells) into the packed smem lines sr.
// Ends with the block synchronised.
template <int P, int N>
__device__ __forceinline__ void cmom_line(const float *__restrict__ cmom,
                                          const unsigned long long *__restrict__ occ,
                                          const uint32_t *__restrict__ blk_rank, int mbits,
                                          uint32_t box, size_t line, float *sr) {
  using LL = LineLayout<N, true>;
  constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2;
  const uint32_t cx = (uint32_t)(line / N), cy = (uint32_t)(line % N);
  for (int zc = threadIdx.x; zc < N; zc += 256) {
    const uint32_t key = (box << (3 * mbits)) | ct2g_morton(cx, cy, (uint32_t)zc);
    bool on;
    const uint32_t rank = occ_rank(occ, blk_rank, key, on);
    float v[NC];
    if (on) {
      const float *m = cmom + (size_t)rank * NC;
#pragma unroll
      for (int k = 0; k < NC; k++) v[k] = __ldg(m + k);
    } else {
#pragma unroll
      for (int k = 0; k < NC; k++) v[k] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < NC; k++) sr[2 * LL::at(k >> 1, zc, 0) + (k & 1)] = v[k];
    if (NC & 1) sr[2 * LL::at(NL - 1, zc, 0) + 1] = 0.f;
  }
  __syncthreads();
}

// The transformed packed lines of LB mesh lines, split into the half spectra
// of their two components, written as LB spectrum rows from `rows` on (row
// lb at rows + lb * ldk * NC; k-point k's components at k * NC; the slots
// k > N/2 get zeros).
template <int P, int N, int LB>
__device__ __forceinline__ void store_half_spectra(const float2 *s, float2 *rows, int ldk) {
  using LL = LineLayout<N, true>;
  constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2, NH = N / 2 + 1;
  const int64_t RS = (int64_t)ldk * NC;
  for (int e = threadIdx.x; e < LB * ldk * NL; e += 256) {
    const int lb = LB == 1 ? 0 : e / (ldk * NL), r = e - lb * ldk * NL;
    const int k = r / NL, l = r - k * NL;
    float2 *row = rows + lb * RS;
    float2 a = make_float2(0.f, 0.f), bb = make_float2(0.f, 0.f);
    if (k < NH) {
      const float2 zk = s[LL::at(lb * NL + l, k & (N - 1), 0)];
      const float2 zn = s[LL::at(lb * NL + l, (N - k) & (N - 1), 0)];
      // A_k = (Z_k + conj Z_{N-k})/2, B_k = (Z_k - conj Z_{N-k})/(2i)
      a = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
      bb = make_float2(0.5f * (zk.y + zn.y), 0.5f * (zn.x - zk.x));
    }
    row[k * NC + 2 * l] = a;
    if (2 * l + 1 < NC) row[k * NC + 2 * l + 1] = bb;
  }
}

// occupancy: 4 blocks per SM up to order 4 (64 registers), 3 beyond on short lines
// (80 registers; from compact records order 6 spills 72-76 bytes there; 2 where the lines fill the
// shared memory); at N = 512 the
// 32-point in-register DFTs need more registers than that, so 2
template <int P, int N, int SRC>
__global__ void __launch_bounds__(256, N >= 512 ? 2 : P <= 4 ? 4 : N <= 128 ? 3 : 2) fftz_p2m_r2c_kernel(
    const uint32_t *__restrict__ px, const uint32_t *__restrict__ py,
    const uint32_t *__restrict__ pz, const uint32_t *__restrict__ cs, int mbits,
    float *__restrict__ grid, int64_t CB, float2 *__restrict__ spec, int ldk,
    const float2 *__restrict__ tw, const float *__restrict__ cmom,
    const unsigned long long *__restrict__ occ, const uint32_t *__restrict__ blk_rank) {
  using LL = LineLayout<N, true>;
  constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2, NH = N / 2 + 1;
  constexpr bool GRID = SRC == CT2G_P2M_GRID;
  constexpr int LB = GRID ? z_lines<P>() : 1;  // lines of this block
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *stw = reinterpret_cast<float2 *>(smraw);
  float2 *s = stw + N;
  float *sr = reinterpret_cast<float *>(s);
  constexpr bool FROM_PARTICLES = SRC == CT2G_P2M_FUSED || SRC == CT2G_P2M_FUSED_STORE;
  __shared__ P2mSmem<P, FROM_PARTICLES ? N : 1> sm;
  if (threadIdx.x == 0) sm.nbig = sm.ncrowd = 0;
  load_twiddles<N>(stw, tw);
  __syncthreads();
  const size_t L0 = (size_t)blockIdx.x * LB;  // first line (box * N^2 + line)
  const size_t line = L0 % ((size_t)N * N);
  const uint32_t box = (uint32_t)(L0 / ((size_t)N * N));
  if constexpr (GRID) {
    // line lb of the block: packed lines lb * NL ...; its grid rows follow
    const float *g = grid + ((int64_t)box * N * N + (int64_t)line) * N;
    for (int e = threadIdx.x; e < LB * NC * N; e += 256) {
      const int lb = LB == 1 ? 0 : e / (NC * N), r = e - lb * NC * N;
      const int k = r / N, z = r % N;
      sr[2 * LL::at(lb * NL + (k >> 1), z, 0) + (k & 1)] = g[(int64_t)k * CB + lb * N + z];
    }
    if (NC & 1)
      for (int e = threadIdx.x; e < LB * N; e += 256)
        sr[2 * LL::at((e / N) * NL + NL - 1, e % N, 0) + 1] = 0.f;
  } else if constexpr (SRC == CT2G_P2M_COMPACT) {
    cmom_line<P, N>(cmom, occ, blk_rank, mbits, box, line, sr);
  } else {
    p2m_line<P, N>(px, py, pz, cs, mbits, box, line, sr, sm);
  }
  __syncthreads();
  if constexpr (SRC == CT2G_P2M_FUSED_STORE) {
    // the moments also go to the moment grid (for passes that read it)
    float *g = grid + ((int64_t)box * N * N + (int64_t)line) * N;
    for (int e = threadIdx.x; e < NC * N; e += 256) {
      const int k = e / N, z = e % N;
      g[(int64_t)k * CB + z] = sr[2 * LL::at(k >> 1, z, 0) + (k & 1)];
    }
    __syncthreads();
  }
  tile_fft<N, true, float2, false>(s, LB * NL, 0, stw);
  store_half_spectra<P, N, LB>(s, spec + (int64_t)L0 * ldk * NC, ldk);
}

// the compact per-cell moment records of the current binning: the occupied
// cells' ranks, then a thread per small cell and a warp per listed big cell
template <int P>
int launch_p2m_compact(ct2g_ctx *ctx) {
  const size_t nw = (size_t)ctx->CB / 64;
  occ_popc_kernel<<<ct2g_div_up(nw, 256), 256, 0, ctx->stream>>>(ctx->occ, nw, ctx->blk_rank);
  CT2G_LAUNCHED(ctx);
  CT2G_TRY(ct2g_scan_exclusive(ctx, ctx->blk_rank, ctx->blk_rank, nw, nullptr, 0));
  CT2G_CUDA(ctx, cudaMemsetAsync(ctx->p2m_big, 0, sizeof(uint32_t), ctx->stream));
  const size_t nr = ctx->n - ctx->rung_begin;  // the binned range, as ct2g_bin_range sorted it
  p2m_compact_kernel<P><<<(unsigned)std::max<size_t>(1, ct2g_div_up(nr, 256)), 256, 0,
                          ctx->stream>>>(ctx->x, ctx->y, ctx->z, ctx->cell_start, ctx->occ,
                                         ctx->blk_rank, ctx->mbits, ctx->keys,
                                         (uint32_t)ctx->rung_begin, (uint32_t)nr, ctx->cmom,
                                         ctx->p2m_big);
  CT2G_LAUNCHED(ctx);
  p2m_compact_big_kernel<P><<<(unsigned)(4 * ctx->num_sms), 256, 0, ctx->stream>>>(
      ctx->x, ctx->y, ctx->z, ctx->cell_start, ctx->occ, ctx->blk_rank, ctx->mbits, ctx->cmom,
      ctx->p2m_big);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

template <int P, int N>
int launch_p2m_r2c(ct2g_ctx *ctx, int src) {
  constexpr int NL = (ct2g_ncomp(P) + 1) / 2;
  const int LB = src == CT2G_P2M_GRID ? z_lines<P>() : 1;
  const size_t smem = sizeof(float2) * ((size_t)N + (size_t)LB * NL * LineLayout<N, true>::LS);
  auto k = src == CT2G_P2M_GRID      ? fftz_p2m_r2c_kernel<P, N, CT2G_P2M_GRID>
           : src == CT2G_P2M_FUSED   ? fftz_p2m_r2c_kernel<P, N, CT2G_P2M_FUSED>
           : src == CT2G_P2M_COMPACT ? fftz_p2m_r2c_kernel<P, N, CT2G_P2M_COMPACT>
                                     : fftz_p2m_r2c_kernel<P, N, CT2G_P2M_FUSED_STORE>;
  CT2G_TRY(ct2g_smem_attrs(ctx, k, smem));
  k<<<(unsigned)((size_t)N * N * ctx->nbox / LB), 256, smem, ctx->stream>>>(
      ctx->x, ctx->y, ctx->z, ctx->cell_start, ctx->mbits, ctx->grid, ctx->CB, ctx->spec,
      ctx->ldk, twiddle_ptr<float2>(ctx), ctx->cmom, ctx->occ, ctx->blk_rank);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

// ---- inverse z pass fused with L2P ------------------------------------------
// LB spectrum rows from `rows` on (layout as store_half_spectra) unpacked
// into packed complex lines in smem: Z = A + iB for the components 2l, 2l+1,
// both halves of the line from the k <= N/2 slots.  ld(q) loads one value
// (a plain load, or one that bypasses L1).  The row's loads go out in batches
// of RB per thread before any of them is used, so that their latencies
// overlap.
template <int P, int N, int LB, typename LD>
__device__ __forceinline__ void load_half_spectra(const float2 *rows, int ldk, float2 *s, LD ld) {
  using LL = LineLayout<N, true>;
  constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2, NH = N / 2 + 1;
  const int64_t RS = (int64_t)ldk * NC;
  constexpr int RB = 5;
  for (int e0 = threadIdx.x; e0 < LB * NH * NL; e0 += RB * 256) {
    float2 a[RB], b[RB];
#pragma unroll
    for (int u = 0; u < RB; u++) {
      const int e = e0 + 256 * u;
      const int lb = LB == 1 ? 0 : e / (NH * NL), r = e - lb * NH * NL;
      const int k = r / NL, l = r - k * NL;
      a[u] = b[u] = make_float2(0.f, 0.f);
      if (e < LB * NH * NL) {
        a[u] = ld(rows + lb * RS + k * NC + 2 * l);
        if (2 * l + 1 < NC) b[u] = ld(rows + lb * RS + k * NC + 2 * l + 1);
      }
    }
#pragma unroll
    for (int u = 0; u < RB; u++) {
      const int e = e0 + 256 * u;
      const int lb = LB == 1 ? 0 : e / (NH * NL), r = e - lb * NH * NL;
      const int k = r / NL, l = r - k * NL;
      if (e < LB * NH * NL) {
        // Z_k = A_k + i B_k; Z_{N-k} = conj(A_k) + i conj(B_k)
        s[LL::at(lb * NL + l, k, 0)] = make_float2(a[u].x - b[u].y, a[u].y + b[u].x);
        if (k > 0 && k < N / 2)
          s[LL::at(lb * NL + l, N - k, 0)] = make_float2(a[u].x + b[u].y, b[u].x - a[u].y);
      }
    }
  }
}

// Inverse transform of one line's packed expansion lines in smem (s, loaded
// and synchronised), then the far field of every particle of the line's
// cells: cb / ce hold the cells' particle ranges (smem, written before the
// caller's last barrier), off is smem scratch of N + 1 words.
template <int P, int N, bool POT>
__device__ __forceinline__ void l2p_line(float2 *s, const float2 *stw, const uint32_t *cb,
                                         const uint32_t *ce, uint32_t *off,
                                         const float4 *__restrict__ src, float GM,
                                         float *__restrict__ ofx, float *__restrict__ ofy,
                                         float *__restrict__ ofz, float *__restrict__ opot) {
  using LL = LineLayout<N, true>;
  constexpr int NL = (ct2g_ncomp(P) + 1) / 2;
  // offsets of the cells' particles in the line's particle list (inclusive
  // scan of the counts, off[0] = 0): thread t holds cells [t ZT, t ZT + ZT),
  // scans its sum across its warp by shuffles before the transform and
  // across the block's warps after it (one barrier of its own)
  constexpr int ZT = (N + 255) / 256;  // cells per thread
  static_assert(N % 256 == 0 || N < 256, "cells per thread");
  __shared__ uint32_t wsum[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t c[ZT], tsum = 0;
#pragma unroll
  for (int q = 0; q < ZT; q++) {
    const int z = threadIdx.x * ZT + q;
    c[q] = z < N ? ce[z] - cb[z] : 0u;
    tsum += c[q];
  }
  uint32_t inc = tsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) wsum[warp] = inc;
  tile_fft<N, true, float2, true>(s, NL, 0, stw);
  __syncthreads();
  {
    uint32_t run = inc - tsum;
    for (int w = 0; w < warp; w++) run += wsum[w];
#pragma unroll
    for (int q = 0; q < ZT; q++) {
      const int z = threadIdx.x * ZT + q;
      run += c[q];
      if (z < N) off[z + 1] = run;
    }
    if (threadIdx.x == 0) off[0] = 0;
  }
  __syncthreads();
  // every particle of the line, one per thread: its cell is the last z with
  // off[z] <= q (that cell holds it: off[z] <= q < off[z + 1])
  const uint32_t total = off[N];
  for (uint32_t q = threadIdx.x; q < total; q += 256) {
    int lo = 0, hi = N;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (off[mid] <= q) lo = mid; else hi = mid;
    }
    const int z = lo;
    const uint32_t i = cb[z] + (q - off[z]);
    const auto acc = [&](int k) {
      const float2 v = s[LL::at(k >> 1, z, 0)];
      return (k & 1) ? v.y : v.x;
    };
    const float4 t = src[i];
    float fx, fy, fz, ph;
    ct2g_l2p<P>(acc, t.x, t.y, t.z, fx, fy, fz, ph);
    ofx[i] = GM * fx;
    ofy[i] = GM * fy;
    ofz[i] = GM * fz;
    if (POT) opot[i] = GM * ph;
  }
}


// One block per (x, y) line of the mesh, all NC expansion components: pairs of
// components are packed into complex lines (A + iB), transformed back along z
// in shared memory, and the block then evaluates the far field of every
// particle of the line's cells from the expansions in shared memory.  The
// expansion grid itself is never written to HBM.  Block b is line b % N^2
// of box b / N^2.  MODE 0: forces, 1: forces and potentials, 2: no L2P, the
// expansions go to the expansion grid (layout as the moment grid).
// occupancy: 5 blocks per SM (48 registers) below N = 512, whose 32-point
// in-register DFTs need more
template <int P, int N, int MODE>
__global__ void __launch_bounds__(256, N >= 512 ? 1 : 5) fftz_c2r_l2p_kernel(
    const float2 *__restrict__ spec, int ldk, const uint32_t *__restrict__ cs,
    const float4 *__restrict__ src, int mbits, const float *__restrict__ box_gm,
    float *__restrict__ ofx, float *__restrict__ ofy, float *__restrict__ ofz,
    float *__restrict__ opot, float *__restrict__ grid, int64_t CB,
    const float2 *__restrict__ tw) {
  using LL = LineLayout<N, true>;
  constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2, NH = N / 2 + 1;
  constexpr bool L2P = MODE < 2;
  constexpr int LB = L2P ? 1 : z_lines<P>();  // lines of this block
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *stw = reinterpret_cast<float2 *>(smraw);
  float2 *s = stw + N;
  __shared__ uint32_t cb[L2P ? N + 1 : 1], ce[L2P ? N : 1];  // particle ranges of the line's cells
  load_twiddles<N>(stw, tw);
  const size_t L0 = (size_t)blockIdx.x * LB;  // first line (box * N^2 + line)
  const size_t line = L0 % ((size_t)N * N);
  const uint32_t box = (uint32_t)(L0 / ((size_t)N * N));
  const uint32_t x = (uint32_t)(line / N), y = (uint32_t)(line % N);
  if constexpr (L2P) {
    // issue the range loads first: their latency hides behind the transform
    for (int z = threadIdx.x; z < N; z += 256) {
      const uint32_t key = (box << (3 * mbits)) | ct2g_morton(x, y, (uint32_t)z);
      cb[z] = cs[key];
      ce[z] = cs[key + 1];
    }
  }
  load_half_spectra<P, N, LB>(spec + (int64_t)L0 * ldk * NC, ldk, s,
                              [](const float2 *q) { return *q; });
  __syncthreads();
  if constexpr (!L2P) {
    tile_fft<N, true, float2, true>(s, LB * NL, 0, stw);
    float *g = grid + ((int64_t)box * N * N + (int64_t)line) * N;
    for (int e = threadIdx.x; e < LB * NC * N; e += 256) {
      const int lb = LB == 1 ? 0 : e / (NC * N), r = e - lb * NC * N;
      const int k = r / N, z = r % N;
      const float2 v = s[LL::at(lb * NL + (k >> 1), z, 0)];
      g[(int64_t)k * CB + lb * N + z] = (k & 1) ? v.y : v.x;
    }
    return;
  } else {
    __shared__ uint32_t off[N + 1];
    l2p_line<P, N, MODE == 1>(s, stw, cb, ce, off, src, __ldg(box_gm + box), ofx, ofy, ofz,
                              opot);
  }
}

template <int P, int N>
int launch_c2r_l2p(ct2g_ctx *ctx, int mode) {
  constexpr int NL = (ct2g_ncomp(P) + 1) / 2;
  const int LB = mode == 2 ? z_lines<P>() : 1;
  const size_t smem = sizeof(float2) * ((size_t)N + (size_t)LB * NL * LineLayout<N, true>::LS);
  auto k = mode == 0 ? fftz_c2r_l2p_kernel<P, N, 0>
           : mode == 1 ? fftz_c2r_l2p_kernel<P, N, 1> : fftz_c2r_l2p_kernel<P, N, 2>;
  CT2G_TRY(ct2g_smem_attrs(ctx, k, smem));
  k<<<(unsigned)((size_t)N * N * ctx->nbox / LB), 256, smem, ctx->stream>>>(
      ctx->spec, ctx->ldk, ctx->cell_start, ctx->src, ctx->mbits, ctx->box_gm, ctx->fx, ctx->fy,
      ctx->fz, ctx->pot, ctx->grid, ctx->CB, twiddle_ptr<float2>(ctx));
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

// ---- z and y passes plane by plane: one persistent kernel per direction -----
// The z pass and the y pass both work plane by plane (an x plane of a box is
// N spectrum rows, N * ldk * NC complex values: 9.3 MB at N = 256, order 4),
// so the y pass of a plane can start as soon as the z pass has written the
// plane, while it is still in L2.  One persistent kernel hands out the items
// of both passes in plane order from a device counter: the z lines of plane
// t, then the y tiles of plane t - 1, then the z lines of plane t + 1, ...;
// a y tile first waits (bounded) for the count of finished z lines of its
// plane.  The spectrum then crosses HBM once per direction instead of three
// times: forward, the y tiles read the rows from L2 and overwrite them in
// place, so only the final values are written back; inverse, the z lines
// read the y pass's output from L2 and (`discard`) drop the lines they have
// read, which nothing reads again, without writing them back.
//
// Waiting is deadlock free whatever the number of resident blocks: a block
// takes an item only while it runs, items are taken in order, and a waiting
// item waits only for items of the other pass taken before it, which never
// wait themselves.

// Item order of a plane pipeline over T planes with a lag of D planes: A(t),
// the first pass's NA items of plane t, and B(t), the second pass's NB items,
// in the order A(0) ... A(D-1), then A(t) B(t-D) for t = D ... T-1, then
// B(T-D) ... B(T-1).  The lag is how long a plane's first-pass items have
// to finish before its second-pass items are handed out; D + 1 planes are in
// flight at a time.
struct PipeOrder {
  uint32_t NA, NB, T, D;  // 1 <= D <= T
  __device__ __forceinline__ uint32_t total() const { return T * (NA + NB); }
  // true for an item of the first pass
  __device__ __forceinline__ bool decode(uint32_t i, uint32_t &plane, uint32_t &sub) const {
    if (i < D * NA) {
      plane = i / NA;
      sub = i - plane * NA;
      return true;
    }
    i -= D * NA;
    const uint32_t R = NA + NB;
    if (i < (T - D) * R) {
      const uint32_t t = i / R, o = i - t * R;
      plane = o < NA ? t + D : t;
      sub = o < NA ? o : o - NA;
      return o < NA;
    }
    i -= (T - D) * R;
    plane = T - D + i / NB;
    sub = i - (plane - (T - D)) * NB;
    return false;
  }
};

constexpr uint32_t kPipeWaitLimit = 1u << 21;  // polls of a plane count (about a second)
constexpr int kPipeW = 16;                     // y tile width (complex columns)

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Thread 0 waits until *count reaches target (the producers' row stores are
// then visible to the block); false for every thread when the wait gave up,
// after the status word was set to CT2G_ETIMEOUT.
__device__ __forceinline__ bool pipe_wait(const uint32_t *count, uint32_t target,
                                          uint32_t *status) {
  int good = 1;
  if (threadIdx.x == 0) {
    uint32_t polls = 0;
    while (ld_acquire(count) < target) {
      if (++polls > kPipeWaitLimit) {
        atomicExch(status, (uint32_t)CT2G_ETIMEOUT);
        good = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
  }
  return __syncthreads_and(good) != 0;
}

// After the block's stores: the item is counted as finished in *count.
__device__ __forceinline__ void pipe_done(uint32_t *count) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(count, 1u);
  }
}

// One y tile: columns [c0, c0 + wv) of the N rows of a plane (row r at
// plane + r * RS), copied into smem by cp.async past L1 (other blocks of the
// kernel wrote them; the whole tile is in flight at once, without staging
// registers), transformed along y in smem (column layout, W columns) and
// written back.  Columns go in 16-byte pairs; a pair that starts below wv
// moves whole (its second column, when past the last one, is a zero slot of
// the row); the smem columns of pairs past wv are left as they are (columns
// transform independently).
template <int N, int W, bool INV>
__device__ __forceinline__ void y_tile(float2 *plane, int64_t RS, int c0, int wv, float2 *s,
                                       const float2 *stw) {
  constexpr int CH = W / 2;  // 16-byte chunks per tile row
  static_assert(N * CH % 256 == 0, "tile chunks per thread");
#pragma unroll 4
  for (int e = threadIdx.x; e < N * CH; e += 256) {
    const int r = e / CH, c = (e % CH) * 2;
    if (c < wv) cp_async16(s + r * W + c, plane + r * RS + c0 + c);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  tile_fft<N, false, float2, INV>(s, W, W, stw);
#pragma unroll 4
  for (int e = threadIdx.x; e < N * CH; e += 256) {
    const int r = e / CH, c = (e % CH) * 2;
    if (c < wv)
      *reinterpret_cast<float4 *>(plane + r * RS + c0 + c) =
          *reinterpret_cast<const float4 *>(s + r * W + c);
  }
}

template <int P, int N>
struct PipeShape {
  static constexpr int NC = ct2g_ncomp(P), NL = (NC + 1) / 2, NH = N / 2 + 1;
  static constexpr size_t ZS = (size_t)NL * LineLayout<N, true>::LS;  // a z line's packed lines
  static constexpr size_t YS = (size_t)N * kPipeW;                    // a y tile
  static constexpr size_t SMEM = sizeof(float2) * ((size_t)N + (ZS > YS ? ZS : YS));
  // the z kernels' register budgets: 64 per thread up to order 4 (the y tiles' DFTs on top
  // spill 8-228 bytes there)
  static constexpr int MINB = P <= 4 ? 4 : 2;
  static constexpr bool OK = N >= 64 && N <= 256;
};

// Forward: z lines (P2M from the particles + r2c along z, store_half_spectra)
// and y tiles.  sync[0]: item counter; sync[2 + t]: finished z lines of plane t.
template <int P, int N>
__global__ void __launch_bounds__(256, PipeShape<P, N>::MINB) zy_forward_kernel(
    const uint32_t *__restrict__ px, const uint32_t *__restrict__ py,
    const uint32_t *__restrict__ pz, const uint32_t *__restrict__ cs, int mbits,
    float2 *__restrict__ spec, int ldk, const float2 *__restrict__ tw, uint32_t nplanes,
    uint32_t lag, uint32_t *__restrict__ sync, uint32_t *__restrict__ status) {
  using S = PipeShape<P, N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *stw = reinterpret_cast<float2 *>(smraw);
  float2 *s = stw + N;
  __shared__ P2mSmem<P, N> sm;
  __shared__ uint32_t item_s;
  load_twiddles<N>(stw, tw);
  const int64_t RS = (int64_t)ldk * S::NC;
  const uint32_t ncols = (uint32_t)(S::NH * S::NC);
  const PipeOrder ord{(uint32_t)N, (ncols + kPipeW - 1) / kPipeW, nplanes, min(lag, nplanes)};
  if (threadIdx.x == 0) item_s = atomicAdd(sync, 1u);
  __syncthreads();
  for (;;) {
    const uint32_t item = item_s;
    if (item >= ord.total()) break;
    uint32_t next = 0;
    if (threadIdx.x == 0) {
      next = atomicAdd(sync, 1u);  // the next item, asked for early
      sm.nbig = sm.ncrowd = 0;
    }
    __syncthreads();
    uint32_t plane, sub;
    if (ord.decode(item, plane, sub)) {
      const size_t L0 = (size_t)plane * N + sub;  // box * N^2 + x * N + y
      p2m_line<P, N>(px, py, pz, cs, mbits, plane / N, L0 % ((size_t)N * N),
                     reinterpret_cast<float *>(s), sm);
      tile_fft<N, true, float2, false>(s, S::NL, 0, stw);
      store_half_spectra<P, N, 1>(s, spec + (int64_t)L0 * RS, ldk);
      pipe_done(sync + 2 + plane);
    } else {
      if (!pipe_wait(sync + 2 + plane, (uint32_t)N, status)) break;
      const int c0 = (int)sub * kPipeW;
      y_tile<N, kPipeW, false>(spec + (int64_t)plane * N * RS, RS, c0,
                               (int)min((uint32_t)kPipeW, ncols - (uint32_t)c0), s, stw);
    }
    if (threadIdx.x == 0) item_s = next;
    __syncthreads();
  }
}

// Inverse: y tiles and z lines (c2r along z + L2P); with `discard` a z line
// drops the L2 lines that lie wholly inside the row it has read.  sync[0]:
// item counter; sync[2 + t]: finished y tiles of plane t.
template <int P, int N, bool POT>
__global__ void __launch_bounds__(256, PipeShape<P, N>::MINB) yz_inverse_kernel(
    float2 *__restrict__ spec, int ldk, const uint32_t *__restrict__ cs,
    const float4 *__restrict__ src, int mbits, const float *__restrict__ box_gm,
    float *__restrict__ ofx, float *__restrict__ ofy, float *__restrict__ ofz,
    float *__restrict__ opot, const float2 *__restrict__ tw, uint32_t nplanes, uint32_t lag,
    int discard, uint32_t *__restrict__ sync, uint32_t *__restrict__ status) {
  using S = PipeShape<P, N>;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *stw = reinterpret_cast<float2 *>(smraw);
  float2 *s = stw + N;
  __shared__ uint32_t cb[N + 1], ce[N], off[N + 1], item_s;
  load_twiddles<N>(stw, tw);
  const int64_t RS = (int64_t)ldk * S::NC;
  const uint32_t ncols = (uint32_t)(S::NH * S::NC), NT = (ncols + kPipeW - 1) / kPipeW;
  const PipeOrder ord{NT, (uint32_t)N, nplanes, min(lag, nplanes)};
  if (threadIdx.x == 0) item_s = atomicAdd(sync, 1u);
  __syncthreads();
  for (;;) {
    const uint32_t item = item_s;
    if (item >= ord.total()) break;
    uint32_t next = 0;
    if (threadIdx.x == 0) next = atomicAdd(sync, 1u);
    uint32_t plane, sub;
    if (ord.decode(item, plane, sub)) {
      const int c0 = (int)sub * kPipeW;
      y_tile<N, kPipeW, true>(spec + (int64_t)plane * N * RS, RS, c0,
                              (int)min((uint32_t)kPipeW, ncols - (uint32_t)c0), s, stw);
      pipe_done(sync + 2 + plane);
    } else {
      const size_t L0 = (size_t)plane * N + sub;
      const uint32_t box = plane / N, x = plane % N, y = sub;
      // the cells' particle ranges first: their latency hides behind the wait
      for (int z = threadIdx.x; z < N; z += 256) {
        const uint32_t key = (box << (3 * mbits)) | ct2g_morton(x, y, (uint32_t)z);
        cb[z] = cs[key];
        ce[z] = cs[key + 1];
      }
      if (!pipe_wait(sync + 2 + plane, NT, status)) break;
      const float2 *row = spec + (int64_t)L0 * RS;
      load_half_spectra<P, N, 1>(row, ldk, s, [](const float2 *q) { return __ldcg(q); });
      __syncthreads();
      if (discard) {
        // the row's own 128-byte lines: every value of them is in smem now
        const uintptr_t a = reinterpret_cast<uintptr_t>(row), e = a + (uintptr_t)RS * 8;
        for (uintptr_t q = ((a + 127) & ~(uintptr_t)127) + 128 * threadIdx.x; q + 128 <= e;
             q += 128 * 256)
          asm volatile("discard.global.L2 [%0], 128;" ::"l"(q) : "memory");
      }
      l2p_line<P, N, POT>(s, stw, cb, ce, off, src, __ldg(box_gm + box), ofx, ofy, ofz, opot);
    }
    if (threadIdx.x == 0) item_s = next;
    __syncthreads();
  }
}

// the plane pipeline of one direction, when the configuration has one
// (FP32 passes, the meshes it is built for, P2M from the particles or L2P
// into the forces); *done = false otherwise, nothing launched
template <int P, int N>
int launch_plane_pipe(ct2g_ctx *ctx, bool inverse, int mode, bool *done) {
  using S = PipeShape<P, N>;
  *done = false;
  if constexpr (!S::OK) {
    return CT2G_OK;
  } else {
    if (!ctx->plane_pipe || ctx->fft_tc || !ctx->pipe_sync) return CT2G_OK;
    if (inverse ? mode > 1 : mode != CT2G_P2M_FUSED) return CT2G_OK;
    const uint32_t nplanes = (uint32_t)(ctx->nbox * N);
    const void *kf = inverse ? (mode == 1 ? (const void *)yz_inverse_kernel<P, N, true>
                                          : (const void *)yz_inverse_kernel<P, N, false>)
                             : (const void *)zy_forward_kernel<P, N>;
    CT2G_TRY(ct2g_smem_attrs(ctx, kf, S::SMEM));
    const unsigned grid = (unsigned)(ct2g_blocks_per_sm(ctx, kf, 256, S::SMEM) * ctx->num_sms);
    uint32_t *sync = ctx->pipe_sync + (inverse ? 2 + nplanes : 0);
    CT2G_CUDA(ctx, cudaMemsetAsync(sync, 0, sizeof(uint32_t) * (2 + nplanes), ctx->stream));
    if (inverse) {
      auto k = mode == 1 ? yz_inverse_kernel<P, N, true> : yz_inverse_kernel<P, N, false>;
      k<<<grid, 256, S::SMEM, ctx->stream>>>(ctx->spec, ctx->ldk, ctx->cell_start, ctx->src,
                                             ctx->mbits, ctx->box_gm, ctx->fx, ctx->fy, ctx->fz,
                                             ctx->pot, twiddle_ptr<float2>(ctx), nplanes,
                                             (uint32_t)ctx->plane_pipe, ctx->pipe_discard, sync,
                                             ctx->d_counts + 6);
    } else {
      zy_forward_kernel<P, N><<<grid, 256, S::SMEM, ctx->stream>>>(
          ctx->x, ctx->y, ctx->z, ctx->cell_start, ctx->mbits, ctx->spec, ctx->ldk,
          twiddle_ptr<float2>(ctx), nplanes, (uint32_t)ctx->plane_pipe, sync, ctx->d_counts + 6);
    }
    CT2G_LAUNCHED(ctx);
    *done = true;
    return CT2G_OK;
  }
}

// ---- X pass + MG2L + inverse X pass ------------------------------------------
// One block per spectrum column (box, qj, qk): the column's N k-points with all
// NC components, s[qi * NC + c], are transformed along x, contracted with the
// Green's tensor (L_a = sum_b G_{a+b} M_b, src/particle.cpp:244-250) and
// transformed back, so neither the transformed moments nor the expansions
// make a round trip through HBM between the three steps.  The first transform
// step reads the column's moments from HBM into registers, the last one
// writes the expansions back from registers; the Green's values ([c][qi], one
// contiguous run of the column-ordered table) arrive by cp.async meanwhile.
// GD: the Green's values are read straight from HBM by the contraction (no
// shared-memory copy of the Green's column, so one more block fits per SM).
// Rows are an odd number of complex values apart: the contraction's threads
// read a row each, and with NC apart (56 at order 5) sixteen of them met in two
// banks.
template <int P, int N, bool GD = false>
struct FxShape {
  static constexpr int NC = ct2g_ncomp(P), NH = N / 2 + 1;
  static constexpr int PITCH = NC | 1;
  static constexpr int GCOL = NC * N;  // floats per Green's column (a multiple of 8)
  static constexpr size_t SMEM = sizeof(float2) * (size_t)N + sizeof(float2) * (size_t)N * PITCH +
                                 (GD ? 0 : sizeof(float) * (size_t)GCOL);
  static constexpr bool FITS = SMEM <= 227 * 1024;
  // three blocks per SM only where the contraction fits 85 registers
  // (orders up to 4 with the Green's values read directly)
  static constexpr int MINB = (GD && NC <= 35 && SMEM <= 75 * 1024) ? 3
                              : SMEM <= 112 * 1024                  ? 2
                                                                    : 1;
  static constexpr bool GREG = !GD && NC <= 35;  // Green's values in registers
  // (a persistent form with one 512-thread block per SM and the next
  // column's data arriving by cp.async in a second buffer measured slower:
  // 2.45 against 1.90 ms at N = 256, order 4)
};

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}

// The two steps of tile_fft for NL lines in the COLS layout s[r * NL + l],
// with the first step's input and the second step's output going through
// functors, so that a line can come straight from HBM or go straight back
// without a pass through shared memory.  cols_step1: jobs (l, n1), input
// ld(l, r), Y[n1][k2] to smem.  cols_step2: jobs (l, k2), X[k2 + R2*k1] to
// st(l, r, v); INPLACE when st writes the smem slots the step reads.
template <int N, int NL, bool INV, int NT, int PITCH = NL, typename LD>
__device__ __forceinline__ void cols_step1(float2 *s, const float2 *stw, LD ld, int off = 0) {
  using LL = LineLayout<N, false>;
  constexpr int R1 = LL::R1, R2 = LL::R2;
  for (int job = threadIdx.x; job < NL * R1; job += NT) {
    const int l = job % NL, n1 = job / NL;
    float2 v[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; n2++) v[n2] = ld(l, n1 + R1 * n2);
    reg_dft<R2, float2, INV>(v);
#pragma unroll
    for (int k2 = 1; k2 < R2; k2++) {
      float2 w = stw[R1 * k2 + n1];
      if (INV) w.y = -w.y;
      v[k2] = cmul(v[k2], w);
    }
#pragma unroll
    for (int k2 = 0; k2 < R2; k2++) s[(n1 + R1 * k2) * PITCH + off + l] = v[k2];
  }
}

template <int N, int NL, bool INV, bool INPLACE, int NT, int PITCH = NL, typename ST>
__device__ __forceinline__ void cols_step2(const float2 *s, ST st, int off = 0) {
  using LL = LineLayout<N, false>;
  constexpr int R1 = LL::R1, R2 = LL::R2;
  static_assert(NT % R2 == 0, "block size must be a multiple of R2");
  constexpr int LW = NT / R2;
  for (int l0 = 0; l0 < NL; l0 += LW) {
    const int l = l0 + threadIdx.x % LW, k2 = threadIdx.x / LW;
    const bool on = l < NL;
    float2 v[R1];
    if (on) {
#pragma unroll
      for (int n1 = 0; n1 < R1; n1++) v[n1] = s[(n1 + R1 * k2) * PITCH + off + l];
      reg_dft<R1, float2, INV>(v);
    }
    if (INPLACE) __syncthreads();  // all reads of this round before any write
    if (on) {
#pragma unroll
      for (int k1 = 0; k1 < R1; k1++) st(l, k2 + R2 * k1, v[k1]);
    }
    if (INPLACE) __syncthreads();
  }
}

// The contraction of a spectrum column in shared memory (row qi of the tile at
// s + qi * PITCH + off): L_a = sum_b G_{a+b} M_b in place.  From 256 rows on a
// thread takes a row.  Below that the outputs of a row are split over groups of
// max(N, 32) threads by the degree of a, so that every thread has work: with a
// thread per row, 64 of 256 did order 5's 462 complex terms each (fused x pass
// of twelve boxes at mesh 64, order 5: 842 -> 475 us, with the odd row pitch).  A group reads what its
// outputs need, and all groups write after the block's one barrier, which stands outside
// their branches; so that the registers across it are the largest group's and not all the
// outputs', each keeps output A as its rank(A)-th.
template <int P>
struct Mg2lSplit {
  static constexpr MiTable<P> mi{};
  // the group (of NG = 2 or 4) of the outputs of degree d, evened out by their
  // terms (of order 5: 56, 105, 120, 100, 60, 21 for d = 0 .. 5)
  static constexpr int group(int d, int NG) {
    if (NG == 4) return d <= 3 ? d : d == 4 ? 0 : d == 5 ? 3 : 1;
    if (P <= 3) return d & 1;
    if (P == 6) return d >= 3 && d <= 5;  // (434 of 924 terms, and 46 outputs of 84)
    return d == 2 || d == 3 || d == 5;
  }
  static constexpr int of(int a, int NG) { return group(mi.deg[a], NG); }
  // outputs of a's group before a, and the outputs of the largest group
  static constexpr int rank(int a, int NG) {
    int r = 0;
    for (int b = 0; b < a; b++) r += of(b, NG) == of(a, NG);
    return r;
  }
  static constexpr int most(int NG) {
    int m = 0;
    for (int a = 0; a < ct2g_ncomp(P); a++) m = rank(a, NG) >= m ? rank(a, NG) + 1 : m;
    return m;
  }
};
template <int P, int GS, int NG, int G, int I, int K>
__device__ __forceinline__ void mg2l_group_term(const float2 *m, const float *g, float2 (&L)[K]) {
  constexpr int A = Mg2lTab<P>::t.a[I], B = Mg2lTab<P>::t.b[I], AB = Mg2lTab<P>::t.ab[I];
  if constexpr (Mg2lSplit<P>::of(A, NG) == G) {
    constexpr int R = Mg2lSplit<P>::rank(A, NG);
    if constexpr (Mg2lTab<P>::t.first[I] != 0) L[R] = make_float2(0.f, 0.f);
    const float gv = g[AB * GS];
    const float2 mb = m[B];
    if constexpr (Mg2lTab<P>::t.odd[I] == 0) {
      L[R].x = fmaf(gv, mb.x, L[R].x);
      L[R].y = fmaf(gv, mb.y, L[R].y);
    } else {  // i*g*(mx + i my) = (-g my, g mx)
      L[R].x = fmaf(-gv, mb.y, L[R].x);
      L[R].y = fmaf(gv, mb.x, L[R].y);
    }
  }
}
template <int P, int GS, int NG, int G, int K, int... I>
__device__ __forceinline__ void mg2l_group_sums(const float2 *m, const float *g, float2 (&L)[K],
                                                std::integer_sequence<int, I...>) {
  (mg2l_group_term<P, GS, NG, G, I>(m, g, L), ...);
}
template <int P, int NG, int G, int A, int K>
__device__ __forceinline__ void mg2l_group_put(float2 *row, const float2 (&L)[K]) {
  if constexpr (Mg2lSplit<P>::of(A, NG) == G) row[A] = L[Mg2lSplit<P>::rank(A, NG)];
}
template <int P, int NG, int G, int K, int... A>
__device__ __forceinline__ void mg2l_group_store(float2 *row, const float2 (&L)[K],
                                                 std::integer_sequence<int, A...>) {
  (mg2l_group_put<P, NG, G, A>(row, L), ...);
}
template <int P, int N, int PITCH, bool GREG, int GS>
__device__ __forceinline__ void contract_column(float2 *s, int off, const float *g) {
  constexpr int NC = ct2g_ncomp(P), NP = Mg2lPairs<P>::NP;
  constexpr int TG = N < 32 ? 32 : N;  // threads per group
  constexpr int NG = N >= 256 ? 1 : TG == 128 ? 2 : 4;
  if constexpr (NG == 1) {
    for (int qi = threadIdx.x; qi < N; qi += 256) {
      float2 *row = s + qi * PITCH + off;
      float2 m[NC];
#pragma unroll
      for (int k = 0; k < NC; k++) m[k] = row[k];
      if constexpr (GREG) {
        float gr[NC];
#pragma unroll
        for (int k = 0; k < NC; k++) gr[k] = g[k * GS + qi];
        ct2g_mg2l_all<P, 1>(m, gr, row, std::make_integer_sequence<int, NP>{});
      } else {
        ct2g_mg2l_all<P, GS>(m, g + qi, row, std::make_integer_sequence<int, NP>{});
      }
    }
  } else {
    const int qi = threadIdx.x % TG, gr = threadIdx.x / TG;
    const int G = qi < N ? gr : NG;  // (threads past the rows or the groups: none)
    float2 *row = s + qi * PITCH + off;
    const std::make_integer_sequence<int, NP> I{};
    const std::make_integer_sequence<int, NC> A{};
    float2 L[Mg2lSplit<P>::most(NG)];
    if (G == 0) mg2l_group_sums<P, GS, NG, 0>(row, g + qi, L, I);
    else if (G == 1) mg2l_group_sums<P, GS, NG, 1>(row, g + qi, L, I);
    else if (NG == 4 && G == 2) mg2l_group_sums<P, GS, NG, 2>(row, g + qi, L, I);
    else if (NG == 4 && G == 3) mg2l_group_sums<P, GS, NG, 3>(row, g + qi, L, I);
    __syncthreads();
    if (G == 0) mg2l_group_store<P, NG, 0>(row, L, A);
    else if (G == 1) mg2l_group_store<P, NG, 1>(row, L, A);
    else if (NG == 4 && G == 2) mg2l_group_store<P, NG, 2>(row, L, A);
    else if (NG == 4 && G == 3) mg2l_group_store<P, NG, 3>(row, L, A);
  }
}

template <int P, int N, bool GD>
__global__ void __launch_bounds__(256, FxShape<P, N, GD>::MINB) fftx_mg2l_kernel(
    float2 *__restrict__ spec, int ldk, const float *__restrict__ gx,
    const float2 *__restrict__ tw) {
  using S = FxShape<P, N, GD>;
  constexpr int NC = S::NC, NH = S::NH;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2 *stw = reinterpret_cast<float2 *>(smraw);
  float2 *s = stw + N;
  constexpr int PITCH = S::PITCH;
  float *sg = reinterpret_cast<float *>(s + N * PITCH);
  const int qk = (int)(blockIdx.x % NH);
  const int qj = (int)((blockIdx.x / NH) % N);
  const int box = (int)(blockIdx.x / ((unsigned)NH * N));
  const int64_t RS = (int64_t)ldk * NC, XS = (int64_t)N * RS;
  float2 *col = spec + (int64_t)box * N * XS + (int64_t)qj * RS + (int64_t)qk * NC;
  // the Green's values arrive while the forward transform runs (or, GD, are
  // read by the contraction itself)
  const float *gcol = gx + ((int64_t)qj * NH + qk) * S::GCOL;
  if constexpr (!GD) {
    for (int e = threadIdx.x; e < S::GCOL / 4; e += 256) cp_async16(sg + 4 * e, gcol + 4 * e);
    cp_async_commit();
  }
  load_twiddles<N>(stw, tw);
  __syncthreads();
  // forward: the first step reads the column from HBM
  cols_step1<N, NC, false, 256, PITCH>(s, stw, [&](int l, int r) { return col[r * XS + l]; });
  __syncthreads();
  cols_step2<N, NC, false, true, 256, PITCH>(s, [&](int l, int r, float2 v) { s[r * PITCH + l] = v; });
  if constexpr (!GD) cp_async_wait<0>();
  __syncthreads();
  contract_column<P, N, PITCH, S::GREG, N>(s, 0, GD ? gcol : sg);
  __syncthreads();
  // inverse: the second step writes the column back to HBM
  cols_step1<N, NC, true, 256, PITCH>(s, stw, [&](int l, int r) { return s[r * PITCH + l]; });
  __syncthreads();
  cols_step2<N, NC, true, false, 256, PITCH>(s, [&](int l, int r, float2 v) { col[r * XS + l] = v; });
}

// The fused x pass + MG2L with its inputs brought in by bulk copies: the
// column (every qi row's NC components) by one tiled tensor copy, its rows
// PITCH complex apart (the copy starts on the 16-byte boundary at or below
// the column: `off` = 0 or 1 complex into each row), and, unless GD, the
// Green's column (contiguous) by one bulk copy, completing on one mbarrier
// (bounded wait) while the twiddles load; GD: the contraction reads the
// Green's values from HBM, and the smaller block (no Green's column, no
// static shared memory, so the dynamic region starts 128-byte aligned) fits
// three to an SM.  CPA: the column arrives instead by per-thread 8-byte
// cp.async copies, all in flight at once, into rows NC | 1 complex apart: the
// tensor copy's rows are a 16-byte multiple apart (36 complex at order 4),
// which puts the rows that the contraction's threads read (a k-point each,
// all NC components) into only four bank groups (an 8-way conflict on every
// component); an odd number apart they spread over all banks.  The
// transforms run in place in the copied tile; the inverse's last step
// writes the column back from registers (a tensor store would also write the
// neighbouring column's element that the tile carries, which another block
// owns).
template <int P, int N, bool GD, bool CPA = false>
struct FxTma {
  static constexpr int NC = ct2g_ncomp(P), NH = N / 2 + 1;
  static constexpr int BW = (2 * NC + 3) / 4 * 4;    // floats per tensor-copy row (16-byte multiple)
  static constexpr int PITCH = CPA ? (NC | 1) : BW / 2;  // complex per tile row
  static constexpr int GCOL = NC * N;
  // GD: tile, twiddles, the mbarrier; else 128 bytes of alignment slack,
  // tile, Green's column, twiddles, the mbarrier
  static constexpr size_t SMEM = (GD ? 0 : 128) + sizeof(float2) * (size_t)N * PITCH +
                                 (GD ? 0 : sizeof(float) * (size_t)GCOL) +
                                 sizeof(float2) * (size_t)N + 16;
  static constexpr bool OK = N >= 64 && N <= 256 && SMEM <= 227 * 1024;
  // three blocks per SM where the contraction fits 85 registers (GD, orders
  // up to 4) and three blocks' shared memory fit
  static constexpr int MINB = (GD && NC <= 35 && 3 * (SMEM + 1024) <= 228 * 1024) ? 3
                              : 2 * (SMEM + 1024) <= 228 * 1024               ? 2
                                                                              : 1;
};

template <int P, int N, bool GD, bool CPA>
__global__ void __launch_bounds__(256, FxTma<P, N, GD, CPA>::MINB) fftx_mg2l_tma_kernel(
    const __grid_constant__ CUtensorMap xmap, float2 *__restrict__ spec, int ldk,
    const float *__restrict__ gx, const float2 *__restrict__ tw, uint32_t *__restrict__ status) {
  using S = FxTma<P, N, GD, CPA>;
  constexpr int NC = S::NC, NH = S::NH, PITCH = S::PITCH;
  // the tensor copy needs a 128-byte aligned destination
  extern __shared__ __align__(128) unsigned char smraw[];
  const uint32_t pad = GD ? 0u : (128u - (tc::smem_addr(smraw) & 127u)) & 127u;
  float2 *s = reinterpret_cast<float2 *>(smraw + pad);  // N rows of PITCH
  float *sg = reinterpret_cast<float *>(s + N * PITCH);
  float2 *stw = reinterpret_cast<float2 *>(sg + (GD ? 0 : S::GCOL));
  uint64_t *bar = reinterpret_cast<uint64_t *>(stw + N);
  const int qk = (int)(blockIdx.x % NH);
  const int qj = (int)((blockIdx.x / NH) % N);
  const int box = (int)(blockIdx.x / ((unsigned)NH * N));
  const int64_t RS = (int64_t)ldk * NC, XS = (int64_t)N * RS;
  const int f0 = 2 * qk * NC, x0 = f0 & ~3, off = CPA ? 0 : (f0 - x0) / 2;
  const float *gcol = gx + ((int64_t)qj * NH + qk) * S::GCOL;
  float2 *col = spec + (int64_t)box * N * XS + (int64_t)qj * RS + (int64_t)qk * NC;
  if (!CPA && (tc::smem_addr(s) & 127u)) {  // checked before any tensor copy
    if (threadIdx.x == 0) atomicExch(status, (uint32_t)CT2G_ECUDA);
    return;
  }
  if (threadIdx.x == 0) tc::mbar_init(bar, 1);
  __syncthreads();  // the barrier is initialised before any thread polls it
  if (threadIdx.x == 0) {
    tc::mbar_arrive_expect_tx(bar, (uint32_t)((CPA ? 0 : sizeof(float2) * N * PITCH) +
                                              (GD ? 0 : sizeof(float) * S::GCOL)));
    if constexpr (!CPA) tc::tma_load_4d(s, &xmap, x0, qj, 0, box, bar);
    if constexpr (!GD) tc::bulk_load(sg, gcol, (uint32_t)(sizeof(float) * S::GCOL), bar);
  }
  if constexpr (CPA) {
    for (int e = threadIdx.x; e < N * NC; e += 256) {
      const int r = e / NC, l = e - r * NC;
      const unsigned sa = tc::smem_addr(s + r * PITCH + l);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(col + r * XS + l)
                   : "memory");
    }
    cp_async_commit();
  }
  load_twiddles<N>(stw, tw);
  if constexpr (CPA) cp_async_wait<0>();
  const bool ok = tc::mbar_wait(bar, 0, kTmaWaitLimit);
  if (!__syncthreads_and(ok)) {
    if (threadIdx.x == 0) {
      atomicExch(status, (uint32_t)CT2G_ETIMEOUT);
      tc::mbar_wait(bar, 0, kTmaWaitLimit);  // copies in flight land before the block exits
    }
    return;
  }
  // forward transform in place in the tile
  cols_step1<N, NC, false, 256, PITCH>(
      s, stw, [&](int l, int r) { return s[r * PITCH + off + l]; }, off);
  __syncthreads();
  cols_step2<N, NC, false, true, 256, PITCH>(
      s, [&](int l, int r, float2 v) { s[r * PITCH + off + l] = v; }, off);
  __syncthreads();
  contract_column<P, N, PITCH, !GD && FxShape<P, N>::GREG, N>(s, off, GD ? gcol : sg);
  __syncthreads();
  // inverse: the second step writes the column back to HBM
  cols_step1<N, NC, true, 256, PITCH>(
      s, stw, [&](int l, int r) { return s[r * PITCH + off + l]; }, off);
  __syncthreads();
  cols_step2<N, NC, true, false, 256, PITCH>(
      s, [&](int l, int r, float2 v) { col[r * XS + l] = v; }, off);
}

template <int P, int N, bool GD>
int launch_fx_mg2l_g(ct2g_ctx *ctx) {
  using S = FxShape<P, N, GD>;
  if constexpr (!S::FITS) {
    return ct2g_fail(ctx, CT2G_EINVAL, "fused X pass + MG2L does not fit in shared memory");
  } else {
    const size_t ncol = (size_t)ctx->nbox * N * S::NH;
    auto k = fftx_mg2l_kernel<P, N, GD>;
    CT2G_TRY(ct2g_smem_attrs(ctx, k, S::SMEM));
    k<<<(unsigned)ncol, 256, S::SMEM, ctx->stream>>>(ctx->spec, ctx->ldk, ctx->greens_x,
                                                     twiddle_ptr<float2>(ctx));
    CT2G_LAUNCHED(ctx);
    return CT2G_OK;
  }
}

// the x-pass tensor map: the spectrum as floats [box][qi][qj][2 * ldk * NC],
// a box of BW floats x all N rows qi of one (qj, box)
int xmap_build(ct2g_ctx *ctx, int BW) {
  if (ctx->xmap_bw == BW) return CT2G_OK;
  EncodeTiledFn encode = nullptr;
  CT2G_TRY(tensor_map_encoder(ctx, &encode));
  const cuuint64_t RS = (cuuint64_t)ctx->ldk * ctx->nc, N = (cuuint64_t)ctx->M;
  const cuuint64_t dims[4] = {2 * RS, N, N, (cuuint64_t)ctx->nbox};
  const cuuint64_t strides[3] = {RS * sizeof(float2), N * RS * sizeof(float2),
                                 N * N * RS * sizeof(float2)};
  const cuuint32_t box[4] = {(cuuint32_t)BW, 1, (cuuint32_t)N, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUtensorMap *m = reinterpret_cast<CUtensorMap *>(ctx->xmap);
  if (encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ctx->spec, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return ct2g_fail(ctx, CT2G_ECUDA, "x-pass tensor map");
  ctx->xmap_bw = BW;
  return CT2G_OK;
}

template <int P, int N, bool GD, bool CPA>
int launch_fx_mg2l_tma(ct2g_ctx *ctx) {
  using S = FxTma<P, N, GD, CPA>;
  if constexpr (!S::OK) {
    return ct2g_fail(ctx, CT2G_EINVAL, "TMA x pass: meshes 64-256");
  } else {
    CT2G_TRY(xmap_build(ctx, S::BW));
    const size_t ncol = (size_t)ctx->nbox * N * S::NH;
    auto k = fftx_mg2l_tma_kernel<P, N, GD, CPA>;
    CT2G_TRY(ct2g_smem_attrs(ctx, k, S::SMEM));
    const CUtensorMap *m = reinterpret_cast<const CUtensorMap *>(ctx->xmap);
    k<<<(unsigned)ncol, 256, S::SMEM, ctx->stream>>>(*m, ctx->spec, ctx->ldk, ctx->greens_x,
                                                     twiddle_ptr<float2>(ctx), ctx->d_counts + 6);
    CT2G_LAUNCHED(ctx);
    return CT2G_OK;
  }
}

template <int P, int N>
int launch_fx_mg2l(ct2g_ctx *ctx) {
  if (ctx->x_tma == 1) {
    if constexpr (FxTma<P, N, true>::OK) {
      if (ctx->mg2l_greens_direct) return launch_fx_mg2l_tma<P, N, true, false>(ctx);
    }
    if constexpr (FxTma<P, N, false>::OK) return launch_fx_mg2l_tma<P, N, false, false>(ctx);
  }
  if (ctx->x_tma == 2) {
    if constexpr (FxTma<P, N, true, true>::OK) {
      if (ctx->mg2l_greens_direct) return launch_fx_mg2l_tma<P, N, true, true>(ctx);
    }
    if constexpr (FxTma<P, N, false, true>::OK) return launch_fx_mg2l_tma<P, N, false, true>(ctx);
  }
  return ctx->mg2l_greens_direct ? launch_fx_mg2l_g<P, N, true>(ctx)
                                 : launch_fx_mg2l_g<P, N, false>(ctx);
}

template <int P>
bool fx_fits(int N) {
  switch (N) {
    case 8: return FxShape<P, 8>::FITS;
    case 16: return FxShape<P, 16>::FITS;
    case 32: return FxShape<P, 32>::FITS;
    case 64: return FxShape<P, 64>::FITS;
    case 128: return FxShape<P, 128>::FITS;
    case 256: return FxShape<P, 256>::FITS;
    case 512: return FxShape<P, 512>::FITS;
  }
  return false;
}

// order x mesh dispatch of the mesh-solve kernels
template <int P>
int spec_stage(ct2g_ctx *ctx, int stage, int mode) {
  switch (ctx->M) {
#define CT2G_SPEC_CASE(NN)                                                  \
  case NN:                                                                  \
    if (stage == 0 && mode == CT2G_P2M_COMPACT)                             \
      CT2G_TRY(launch_p2m_compact<P>(ctx));                                 \
    if (stage == 0) return launch_p2m_r2c<P, NN>(ctx, mode);                \
    if (stage == 1) return launch_fx_mg2l<P, NN>(ctx);                      \
    return launch_c2r_l2p<P, NN>(ctx, mode);
    CT2G_SPEC_CASE(8)
    CT2G_SPEC_CASE(16)
    CT2G_SPEC_CASE(32)
    CT2G_SPEC_CASE(64)
    CT2G_SPEC_CASE(128)
    CT2G_SPEC_CASE(256)
    CT2G_SPEC_CASE(512)
#undef CT2G_SPEC_CASE
  }
  return ct2g_fail(ctx, CT2G_EINVAL, "mesh must be a power of two in [8, 512]");
}

template <int P>
int spec_pipe_p(ct2g_ctx *ctx, bool inverse, int mode, bool *done) {
  switch (ctx->M) {
    case 64: return launch_plane_pipe<P, 64>(ctx, inverse, mode, done);
    case 128: return launch_plane_pipe<P, 128>(ctx, inverse, mode, done);
    case 256: return launch_plane_pipe<P, 256>(ctx, inverse, mode, done);
  }
  *done = false;
  return CT2G_OK;
}

}  // namespace

// the entry points of one order
#define CT2G_FFT_ORDER_FNS(P)                                                        \
  extern const Ct2gOrderFns ct2g_order_fns_p##P;                                     \
  const Ct2gOrderFns ct2g_order_fns_p##P = {set_consts, spec_stage<P>, spec_pipe_p<P>, \
                                            fx_fits<P>};
