// Particle binning (particle_to_grid, src/particle.cpp:69-114,349-362):
// Morton cell keys from the top mesh bits of the fixed-point positions, a
// stable LSD radix sort of (key, index) pairs, one pass over the cells for
// their ranges and the near field's sink chunks, the gather of the SoA into
// cell order and per-particle float offsets from the cell centre for the
// direct sum.
//
// The reference partitions recursively (a Hoare partition per level,
// dimension depth%3); for a power-of-two mesh every particle lands in the
// same leaf as here, because the split point fixed32((I+N/2)/Ncell) equals
// (I+N/2) << (32-mbits), and the leaves come out in the same (Morton) order.
// Only the order inside a cell differs: the reference's partition leaves it
// arbitrary, here it is the stable (previous) order, so the sort is
// deterministic.
#include "ct2g_internal.cuh"

namespace {

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;  // per thread
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// block-wide exclusive scan of one value per thread; returns block total
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *smem32,
                                                    uint32_t &total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t inc = warp_incl_scan(v);
  if (lane == 31) smem32[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t s = lane < nw ? smem32[lane] : 0;
    uint32_t si = warp_incl_scan(s);
    if (lane < nw) smem32[lane] = si - s;
    if (lane == nw - 1) smem32[32] = si;
  }
  __syncthreads();
  uint32_t res = inc - v + smem32[w];
  total = smem32[32];
  __syncthreads();
  return res;
}

__global__ void scan_reduce_kernel(const uint32_t *__restrict__ in, size_t n,
                                   uint32_t *__restrict__ bsum) {
  __shared__ uint32_t sm[33];
  size_t base = (size_t)blockIdx.x * kScanTile;
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    size_t i = base + (size_t)k * kScanThreads + threadIdx.x;
    if (i < n) s += in[i];
  }
  uint32_t tot;
  block_excl_scan(s, sm, tot);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

// single block: exclusive scan of bsum[nb] in place (nb arbitrary)
__global__ void scan_single_kernel(uint32_t *__restrict__ a, size_t nb, uint32_t *total) {
  __shared__ uint32_t sm[33];
  uint32_t carry = 0;
  for (size_t base = 0; base < nb; base += blockDim.x) {
    size_t i = base + threadIdx.x;
    uint32_t v = i < nb ? a[i] : 0;
    uint32_t tot;
    uint32_t ex = block_excl_scan(v, sm, tot);
    if (i < nb) a[i] = ex + carry;
    carry += tot;
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void scan_apply_kernel(const uint32_t *__restrict__ in, size_t n,
                                  const uint32_t *__restrict__ boff, uint32_t offset,
                                  uint32_t *__restrict__ out) {
  __shared__ uint32_t sm[33];
  size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  uint32_t tot;
  uint32_t ex = block_excl_scan(s, sm, tot) + boff[blockIdx.x] + offset;
#pragma unroll
  for (int k = 0; k < kScanItems; k++) {
    if (base + k < n) out[base + k] = ex;
    ex += v[k];
  }
}

// ---------------------------------------------------------------------------
// radix sort: digits of up to 9 bits (as even as the key allows: 2 x 9 at mesh
// 64, 3 x 8 at 256), tiles of 256 threads x ITEMS items (striped per warp).
// Up to kFusedTiles tiles the scatter adds up its tile's digit offsets from the
// histograms itself (a thread reads one or two digits' rows), so that a pass is
// two launches; beyond, the histograms (digit-major) are scanned in between, three
// launches more.  Tiles of 1024 below kSmallSort particles: 13 tiles of
// 4096 left a pass of 50 k particles 11 us in each of its two kernels.
// ---------------------------------------------------------------------------
constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kMaxBins = 512;
constexpr uint32_t kFusedTiles = 128;
constexpr size_t kSmallSort = 65536;

template <int ITEMS>
__device__ __forceinline__ size_t radix_item(int slot) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  return (size_t)blockIdx.x * (kRadixThreads * ITEMS) + (size_t)w * 32 * ITEMS + slot * 32 + lane;
}

// where the keys of the first pass come from: key = (box << 3*mbits) | Morton
// index of the cell; the box of a particle is found by bisection of the box
// offsets (boxes never exchange particles)
struct KeySource {
  const uint32_t *x, *y, *z;
  size_t begin;
  int mbits;
  const uint32_t *box_off;
  int nbox;
  __device__ __forceinline__ uint32_t operator()(size_t i) const {
    const int sh = 32 - mbits;
    const size_t g = begin + i;
    uint32_t box = 0;
    if (nbox > 1) {
      uint32_t lo = 0, hi = (uint32_t)nbox;  // box_off[lo] <= g < box_off[hi]
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(box_off + mid) <= (uint32_t)g) lo = mid; else hi = mid;
      }
      box = lo << (3 * mbits);
    }
    return box | ct2g_morton(x[g] >> sh, y[g] >> sh, z[g] >> sh);
  }
};

// digit histogram of each tile, hist[digit * ntiles + tile]; FIRST: the keys
// are formed (and stored) here
template <int ITEMS, bool FIRST>
__global__ void __launch_bounds__(kRadixThreads) radix_hist_kernel(
    const KeySource src, uint32_t *__restrict__ keys, size_t n, int shift, int bits,
    uint32_t ntiles, uint32_t *__restrict__ hist) {
  __shared__ uint32_t cnt[kMaxBins];
  const int nb = 1 << bits;
  for (int d = threadIdx.x; d < nb; d += kRadixThreads) cnt[d] = 0;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const size_t i = radix_item<ITEMS>(k);
    if (i < n) {
      const uint32_t key = FIRST ? src(i) : keys[i];
      if (FIRST) keys[i] = key;
      atomicAdd(&cnt[(key >> shift) & (uint32_t)(nb - 1)], 1u);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < nb; d += kRadixThreads)
    hist[(size_t)d * ntiles + blockIdx.x] = cnt[d];
}

// stable scatter by the digit; FIRST: the values are the particles' indices.
// FUSED: hist holds the tiles' counts, else their exclusive scan
template <int ITEMS, bool FIRST, bool FUSED>
__global__ void __launch_bounds__(kRadixThreads) radix_scatter_kernel(
    const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals, size_t n, int shift,
    int bits, uint32_t ntiles, const uint32_t *__restrict__ hist, uint32_t *__restrict__ okeys,
    uint32_t *__restrict__ ovals) {
  __shared__ uint32_t wcnt[kRadixWarps][kMaxBins];
  __shared__ uint32_t base[kMaxBins];
  __shared__ uint32_t sm[33];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = 1 << bits;
  const uint32_t mask = (uint32_t)(nb - 1);
  for (int i = threadIdx.x; i < kRadixWarps * kMaxBins; i += kRadixThreads) (&wcnt[0][0])[i] = 0;
  if constexpr (FUSED) {
    // digits 2 t and 2 t + 1: items in tiles before this one, and in all
    uint32_t before[2] = {0, 0}, all[2] = {0, 0};
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int d = 2 * threadIdx.x + q;
      if (d < nb) {
        const uint32_t *row = hist + (size_t)d * ntiles;
#pragma unroll 8
        for (uint32_t t = 0; t < ntiles; t++) {
          const uint32_t c = row[t];
          all[q] += c;
          if (t < blockIdx.x) before[q] += c;
        }
      }
    }
    uint32_t tot;
    const uint32_t ex = block_excl_scan(all[0] + all[1], sm, tot);
    base[2 * threadIdx.x] = ex + before[0];
    base[2 * threadIdx.x + 1] = ex + all[0] + before[1];
  } else {
    for (int d = threadIdx.x; d < nb; d += kRadixThreads)
      base[d] = hist[(size_t)d * ntiles + blockIdx.x];
  }
  __syncthreads();
  uint32_t k_[ITEMS], v_[ITEMS], r_[ITEMS];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const size_t i = radix_item<ITEMS>(k);
    const bool valid = i < n;
    const uint32_t key = valid ? keys[i] : 0u;
    const uint32_t d = (key >> shift) & mask;
    k_[k] = key;
    v_[k] = FIRST ? (uint32_t)i : valid ? vals[i] : 0u;
    const unsigned act = __ballot_sync(0xffffffffu, valid);
    const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : kMaxBins + lane) & act;
    const uint32_t before = valid ? wcnt[w][d] : 0u;
    __syncwarp();
    if (valid) {
      r_[k] = before + __popc(peers & lt);
      if ((peers & lt) == 0) wcnt[w][d] = before + __popc(peers);
    }
    __syncwarp();
  }
  __syncthreads();
  for (int d = threadIdx.x; d < nb; d += kRadixThreads) {  // exclusive prefix over warps
    uint32_t run = 0;
#pragma unroll
    for (int ww = 0; ww < kRadixWarps; ww++) {
      const uint32_t t = wcnt[ww][d];
      wcnt[ww][d] = run;
      run += t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const size_t i = radix_item<ITEMS>(k);
    if (i < n) {
      const uint32_t d = (k_[k] >> shift) & mask;
      const uint32_t pos = base[d] + wcnt[w][d] + r_[k];
      okeys[pos] = k_[k];
      ovals[pos] = v_[k];
    }
  }
}

// ---------------------------------------------------------------------------
// The cells' ranges, their occupancy bits and the near field's work lists in one
// pass over the sorted keys: a block per 2048 consecutive cells (32 blocks of
// 4x4x4).  Two warps find the tile's keys (32 probes a step); the first particle
// of each run of equal keys marks its cell, and an empty cell begins where the next
// occupied one does (crowded tiles: a lower bound per cell instead of a walk
// over their particles), so no count is scanned over the mesh.  (Counting and scanning, then flagging and scanning the particles three
// times for the lists, were 19 launches of some 170 us at 128^3 particles on a
// 256^3 mesh, now 122; at 12^3 on 16^3 a step takes 201 us instead of 246, at 50 k
// on 64^3 740 instead of 883.)
//
// Sink lists, in warp chunks: cells with at least dense_cell particles are
// split into chunks of one cell (every 64th particle of the cell starts one: two
// sinks a lane); the particles of sparser cells are listed (sparse_list, cell
// order within a 4x4x4 block, which is 64 consecutive Morton keys) and chunked
// per block, every kSparseChunk-th sparse particle of a block starting a
// chunk.  A tile takes its places in the lists with three atomics; the order of
// the tiles in them does not matter.
// counts: [0] dense chunks, [1] sparse sinks, [2] sparse chunks, zero on entry.
// ---------------------------------------------------------------------------
constexpr uint32_t kSparseChunk = 32;  // sinks per sparse chunk
constexpr int kCellTile = 2048, kCellThreads = 256;
constexpr uint32_t kMarkMax = 16384;  // particles of a tile that mark their cells' starts

// first index in [lo, hi) whose key is >= k (hi if none), by a whole warp
__device__ __forceinline__ size_t warp_lower_bound(const uint32_t *__restrict__ keys, size_t lo,
                                                   size_t hi, uint32_t k) {
  const int lane = threadIdx.x & 31;
  while (lo < hi) {
    // probes at the ends of 32 equal steps; the answer lies in the first step whose end is >= k
    const size_t step = (hi - lo + 31) / 32;
    const size_t p = min(lo + step * (size_t)(lane + 1), hi) - 1;
    const unsigned ge = __ballot_sync(0xffffffffu, keys[p] >= k);
    if (!ge) return hi;
    const int f = __ffs((int)ge) - 1;
    const size_t nhi = min(lo + step * (size_t)(f + 1), hi) - 1;  // its key is >= k
    lo = lo + step * (size_t)f;
    if (lo > nhi) lo = nhi;
    hi = nhi;
    if (lo == hi) return hi;
  }
  return lo;
}

__global__ void __launch_bounds__(kCellThreads, 6) cells_kernel(
    const uint32_t *__restrict__ skeys, size_t begin, size_t nr, size_t CB, uint32_t dense_cell,
    uint32_t *__restrict__ cs, unsigned long long *__restrict__ occ, uint32_t *__restrict__ counts,
    uint2 *__restrict__ chunks, uint2 *__restrict__ schunks, uint32_t *__restrict__ sparse_list) {
  __shared__ uint32_t first[kCellTile + 1];  // particles of the tile before each cell
  __shared__ uint32_t bits[kCellTile / 32];  // occupied cells
  __shared__ uint32_t after[kCellTile / 32];  // first[] of the next occupied cell past a word
  __shared__ size_t range[2];
  __shared__ uint32_t blk[3][64], base[3];   // per 4x4x4 block: dense chunks, sparse sinks, sparse chunks
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t c0 = (size_t)blockIdx.x * kCellTile;
  const int ncell = (int)min((size_t)kCellTile, CB - c0);  // a multiple of 64
  if (warp < 2) {
    // (the end of the key space may not be a 32-bit key: every key is below it)
    const size_t kc = c0 + (warp ? (size_t)ncell : 0);
    const size_t r = kc >= CB ? nr : warp_lower_bound(skeys, 0, nr, (uint32_t)kc);
    if (lane == 0) range[warp] = r;
  }
  if (tid < kCellTile / 32) bits[tid] = 0;
  __syncthreads();
  const size_t lo = range[0];
  const uint32_t m = (uint32_t)(range[1] - lo);
  const uint32_t *tk = skeys + lo;
  if (m <= kMarkMax) {
    // the first particle of each run of equal keys marks its cell
#pragma unroll 4
    for (uint32_t i = tid; i < m; i += kCellThreads) {
      const uint32_t k = tk[i];
      if (i == 0 || tk[i - 1] != k) {
        const uint32_t c = k - (uint32_t)c0;
        first[c] = i;
        atomicOr(&bits[c >> 5], 1u << (c & 31u));
      }
    }
    __syncthreads();
    if (warp == 0) {  // words WL lane .. WL lane + WL - 1, from the last
      constexpr int WL = kCellTile / 1024;
      uint32_t nx[WL + 1];  // first[] of the first occupied cell at or past each word
      nx[WL] = 0xffffffffu;
#pragma unroll
      for (int q = WL - 1; q >= 0; q--) {
        const uint32_t w = bits[WL * lane + q];
        nx[q] = w ? first[32 * (WL * lane + q) + __ffs((int)w) - 1] : nx[q + 1];
      }
      uint32_t r = nx[0];  // and at or past each lane's words
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_down_sync(0xffffffffu, r, d);
        if (lane + d < 32) r = min(r, v);  // (positions grow with the cell)
      }
      uint32_t past = __shfl_down_sync(0xffffffffu, r, 1);
      if (lane == 31 || past == 0xffffffffu) past = m;
#pragma unroll
      for (int q = 0; q < WL; q++) after[WL * lane + q] = nx[q + 1] != 0xffffffffu ? nx[q + 1] : past;
    }
    __syncthreads();
    // an empty cell begins where the next occupied one does
    for (int c = tid; c < ncell; c += kCellThreads) {
      const uint32_t w = bits[c >> 5], b = (uint32_t)c & 31u;
      if ((w >> b) & 1u) continue;
      const uint32_t up = w & ~(0xffffffffu >> (31u - b));
      first[c] = up ? first[(c & ~31) + __ffs((int)up) - 1] : after[c >> 5];
    }
    if (tid == 0) first[ncell] = m;
  } else {
    for (int c = tid; c <= ncell; c += kCellThreads) {
      uint32_t a = 0, e = c == ncell ? 0u : m;
      const uint32_t k = (uint32_t)(c0 + (size_t)c);
      while (a < e) {
        const uint32_t h = (a + e) >> 1;
        if (tk[h] < k) a = h + 1; else e = h;
      }
      first[c] = c == ncell ? m : a;
    }
  }
  __syncthreads();
  const uint32_t b0 = (uint32_t)(begin + lo);
  for (int c = tid; c < ncell; c += kCellThreads) cs[c0 + c] = b0 + first[c];
  if (c0 + ncell == CB && tid == 0) cs[CB] = (uint32_t)(begin + nr);
  // a warp per 4x4x4 block, two cells per lane (2 lane, 2 lane + 1)
  const int nblk = ncell / 64;
  for (int q = warp; q < nblk; q += kCellThreads / 32) {
    const int c = 64 * q + 2 * lane;
    const uint32_t f0 = first[c], f1 = first[c + 1], f2 = first[c + 2];
    unsigned long long w = (unsigned long long)((f1 > f0 ? 1u : 0u) | (f2 > f1 ? 2u : 0u)) << (2 * lane);
    const uint32_t wl = __reduce_or_sync(0xffffffffu, (uint32_t)w),
                   wh = __reduce_or_sync(0xffffffffu, (uint32_t)(w >> 32));
    if (lane == 0) occ[c0 / 64 + q] = (unsigned long long)wh << 32 | wl;
    const uint32_t n0 = f1 - f0, n1 = f2 - f1;
    const uint32_t dn = (n0 >= dense_cell ? (n0 + 63) / 64 : 0u) + (n1 >= dense_cell ? (n1 + 63) / 64 : 0u);
    const uint32_t sn = (n0 >= dense_cell ? 0u : n0) + (n1 >= dense_cell ? 0u : n1);
    const uint32_t dt = __reduce_add_sync(0xffffffffu, dn), st = __reduce_add_sync(0xffffffffu, sn);
    if (lane == 0) {
      blk[0][q] = dt;
      blk[1][q] = st;
      blk[2][q] = (st + kSparseChunk - 1) / kSparseChunk;
    }
  }
  if (m == 0) return;
  __syncthreads();
  if (warp < 3) {  // exclusive scans over the tile's blocks, and the tile's places
    const uint32_t v0 = 2 * lane < nblk ? blk[warp][2 * lane] : 0u;
    const uint32_t v1 = 2 * lane + 1 < nblk ? blk[warp][2 * lane + 1] : 0u;
    const uint32_t inc = warp_incl_scan(v0 + v1), ex = inc - v0 - v1;
    if (lane == 31) base[warp] = inc ? atomicAdd(counts + warp, inc) : 0u;
    blk[warp][2 * lane] = ex;
    blk[warp][2 * lane + 1] = ex + v0;
  }
  __syncthreads();
  for (int q = warp; q < nblk; q += kCellThreads / 32) {
    const int c = 64 * q + 2 * lane;
    const uint32_t f[3] = {first[c], first[c + 1], first[c + 2]};
    if (__ballot_sync(0xffffffffu, f[2] > f[0]) == 0) continue;
    uint32_t dn[2], sn[2];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t n = f[u + 1] - f[u];
      dn[u] = n >= dense_cell ? (n + 63) / 64 : 0u;
      sn[u] = n >= dense_cell ? 0u : n;
    }
    const uint32_t di = warp_incl_scan(dn[0] + dn[1]), si = warp_incl_scan(sn[0] + sn[1]);
    const uint32_t st = __shfl_sync(0xffffffffu, si, 31);
    uint32_t d = base[0] + blk[0][q] + di - dn[0] - dn[1];
    const uint32_t s0 = base[1] + blk[1][q];
    uint32_t s = s0 + si - sn[0] - sn[1];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t g = b0 + f[u], n = f[u + 1] - f[u];
      for (uint32_t k = 0; k < dn[u]; k++) chunks[d++] = make_uint2(g + 64 * k, min(64u, n - 64 * k));
      for (uint32_t k = 0; k < sn[u]; k++) sparse_list[s++] = g + k;
    }
    for (uint32_t k = lane; k * kSparseChunk < st; k += 32)
      schunks[base[2] + blk[2][q] + k] =
          make_uint2(s0 + k * kSparseChunk, min(kSparseChunk, st - k * kSparseChunk));
  }
}

// gather the active range into cell order; write the direct-sum source records
__global__ void gather_kernel(const uint32_t *__restrict__ perm, size_t begin, size_t nr,
                              int mbits, const uint32_t *__restrict__ x,
                              const uint32_t *__restrict__ y, const uint32_t *__restrict__ z,
                              const float *__restrict__ vx, const float *__restrict__ vy,
                              const float *__restrict__ vz, const int8_t *__restrict__ rung,
                              const uint32_t *__restrict__ id, uint32_t *__restrict__ x2,
                              uint32_t *__restrict__ y2, uint32_t *__restrict__ z2,
                              float *__restrict__ vx2, float *__restrict__ vy2,
                              float *__restrict__ vz2, int8_t *__restrict__ rung2,
                              uint32_t *__restrict__ id2, float4 *__restrict__ src,
                              bool vel) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nr) return;
  size_t s = begin + perm[i], d = begin + i;
  uint32_t px = x[s], py = y[s], pz = z[s];
  x2[d] = px;
  y2[d] = py;
  z2[d] = pz;
  if (vel) {
    vx2[d] = vx[s];
    vy2[d] = vy[s];
    vz2[d] = vz[s];
    rung2[d] = rung[s];
  } else {
    // velocities and rungs follow later (gather_vel_kernel): keep the source
    // index in their gather target
    reinterpret_cast<uint32_t *>(vx2)[d] = (uint32_t)s;
  }
  id2[d] = id[s];
  // offset from the cell centre: low (32-mbits) bits minus half a cell,
  // exact in float (|value| < 2^(31-mbits) <= 2^24)
  const int sh = 32 - mbits;
  const uint32_t mask = (sh == 32) ? 0xffffffffu : ((1u << sh) - 1u);
  const int32_t half = (int32_t)(1u << (sh - 1));
  const float sc = (float)CT2G_TWO_M32;
  src[d] = make_float4((float)((int32_t)(px & mask) - half) * sc,
                       (float)((int32_t)(py & mask) - half) * sc,
                       (float)((int32_t)(pz & mask) - half) * sc, 0.f);
}

// the gathered (cell-ordered) store goes back into the primary buffers, so
// that every step reads and writes the same addresses (a recorded graph
// replays with fixed pointers)
__global__ void copy_back_kernel(size_t begin, size_t nr, const uint32_t *__restrict__ x2,
                                 const uint32_t *__restrict__ y2, const uint32_t *__restrict__ z2,
                                 const float *__restrict__ vx2, const float *__restrict__ vy2,
                                 const float *__restrict__ vz2, const int8_t *__restrict__ rung2,
                                 const uint32_t *__restrict__ id2, uint32_t *__restrict__ x,
                                 uint32_t *__restrict__ y, uint32_t *__restrict__ z,
                                 float *__restrict__ vx, float *__restrict__ vy,
                                 float *__restrict__ vz, int8_t *__restrict__ rung,
                                 uint32_t *__restrict__ id, bool vel) {
  const size_t i = begin + (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= begin + nr) return;
  x[i] = x2[i];
  y[i] = y2[i];
  z[i] = z2[i];
  if (vel) {
    vx[i] = vx2[i];
    vy[i] = vy2[i];
    vz[i] = vz2[i];
    rung[i] = rung2[i];
  }
  id[i] = id2[i];
}

// the deferred half of the gather: velocities and rungs into cell order,
// from the source indices the position gather left in vx2
__global__ void gather_vel_kernel(size_t begin, size_t nr, const float *__restrict__ vx,
                                  const float *__restrict__ vy, const float *__restrict__ vz,
                                  const int8_t *__restrict__ rung, float *__restrict__ vx2,
                                  float *__restrict__ vy2, float *__restrict__ vz2,
                                  int8_t *__restrict__ rung2) {
  const size_t d = begin + (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= begin + nr) return;
  const uint32_t s = reinterpret_cast<const uint32_t *>(vx2)[d];
  if (s < begin || s >= begin + nr) return;  // the position gather wrote every index in range
  vx2[d] = vx[s];
  vy2[d] = vy[s];
  vz2[d] = vz[s];
  rung2[d] = rung[s];
}

__global__ void copy_back_vel_kernel(size_t begin, size_t nr, const float *__restrict__ vx2,
                                     const float *__restrict__ vy2,
                                     const float *__restrict__ vz2,
                                     const int8_t *__restrict__ rung2, float *__restrict__ vx,
                                     float *__restrict__ vy, float *__restrict__ vz,
                                     int8_t *__restrict__ rung) {
  const size_t i = begin + (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= begin + nr) return;
  vx[i] = vx2[i];
  vy[i] = vy2[i];
  vz[i] = vz2[i];
  rung[i] = rung2[i];
}

__global__ void fill_kernel(uint32_t *__restrict__ a, size_t n, uint32_t v) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = v;
}

}  // namespace

size_t ct2g_scan_scratch_words(size_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

// exclusive scan of n uint32 values (in may equal out); the sum optionally
// goes to the device word total_dev
int ct2g_scan_exclusive(ct2g_ctx *ctx, const uint32_t *in, uint32_t *out, size_t n,
                        uint32_t *total_dev, uint32_t offset) {
  if (n == 0) {
    if (total_dev) CT2G_CUDA(ctx, cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), ctx->stream));
    return CT2G_OK;
  }
  unsigned nb = ct2g_div_up(n, kScanTile);
  if (ctx->scan_tmp_words < (size_t)nb + 1) {
    if (ctx->capturing) return ct2g_fail(ctx, CT2G_ESTATE, "scan scratch too small while recording");
    ctx->epoch++;
    if (ctx->scan_tmp) cudaFree(ctx->scan_tmp);
    ctx->scan_tmp = nullptr;
    ctx->scan_tmp_words = 0;
    CT2G_CUDA(ctx, cudaMalloc(&ctx->scan_tmp, sizeof(uint32_t) * ((size_t)nb + 1)));
    ctx->scan_tmp_words = (size_t)nb + 1;
  }
  uint32_t *bsum = ctx->scan_tmp;
  scan_reduce_kernel<<<nb, kScanThreads, 0, ctx->stream>>>(in, n, bsum);
  CT2G_LAUNCHED(ctx);
  scan_single_kernel<<<1, 1024, 0, ctx->stream>>>(bsum, nb, total_dev ? total_dev : bsum + nb);
  CT2G_LAUNCHED(ctx);
  scan_apply_kernel<<<nb, kScanThreads, 0, ctx->stream>>>(in, n, bsum, offset, out);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

// The range's (key, index) pairs sorted by key, in ctx->keys and ctx->vals
template <int ITEMS>
static int radix_sort(ct2g_ctx *ctx, const KeySource &src, size_t nr, int bits) {
  cudaStream_t st = ctx->stream;
  const uint32_t ntiles = ct2g_div_up(nr, kRadixThreads * ITEMS);
  const bool fused = ntiles <= kFusedTiles;
  const int npass = (bits + 8) / 9;
  uint32_t *ka = ctx->keys, *va = ctx->vals, *kb = ctx->keys2, *vb = ctx->vals2;
  for (int pass = 0, shift = 0; pass < npass; pass++) {
    const int db = (bits - shift + npass - pass - 1) / (npass - pass);  // this digit's bits
    const bool first = pass == 0;
    auto hist = first ? radix_hist_kernel<ITEMS, true> : radix_hist_kernel<ITEMS, false>;
    hist<<<ntiles, kRadixThreads, 0, st>>>(src, ka, nr, shift, db, ntiles, ctx->hist);
    CT2G_LAUNCHED(ctx);
    if (!fused)
      CT2G_TRY(ct2g_scan_exclusive(ctx, ctx->hist, ctx->hist, ((size_t)1 << db) * ntiles, nullptr, 0));
    auto scatter = first ? (fused ? radix_scatter_kernel<ITEMS, true, true>
                                  : radix_scatter_kernel<ITEMS, true, false>)
                         : (fused ? radix_scatter_kernel<ITEMS, false, true>
                                  : radix_scatter_kernel<ITEMS, false, false>);
    scatter<<<ntiles, kRadixThreads, 0, st>>>(ka, va, nr, shift, db, ntiles, ctx->hist, kb, vb);
    CT2G_LAUNCHED(ctx);
    std::swap(ka, kb);
    std::swap(va, vb);
    shift += db;
  }
  // (the number of passes is fixed per context, so a replay ends in the same
  // buffers)
  if (ka != ctx->keys) {
    std::swap(ctx->keys, ctx->keys2);
    std::swap(ctx->vals, ctx->vals2);
  }
  return CT2G_OK;
}

// Sort the current range [rung_begin, n) by cell; build cell ranges, source
// records and sink chunks.  Every size a later kernel needs stays on the
// device (ctx->d_counts), so the sequence can be recorded into a graph.
int ct2g_bin_range(ct2g_ctx *ctx) {
  const size_t begin = ctx->rung_begin, nr = ctx->n - ctx->rung_begin;
  const int mbits = ctx->mbits;
  cudaStream_t st = ctx->stream;
  const unsigned T = 256;
  if (!ctx->boxes_set) return ct2g_fail(ctx, CT2G_ESTATE, "box sizes not set since the upload");
  uint32_t *counts = ctx->d_counts;
  CT2G_CUDA(ctx, cudaMemsetAsync(counts, 0, sizeof(uint32_t) * 6, st));
  if (nr > 0) {
    const int bits = 3 * mbits + ctx->boxbits;
    const KeySource src{ctx->x, ctx->y, ctx->z, begin, mbits, ctx->box_off, ctx->nbox};
    if (nr <= kSmallSort) CT2G_TRY(radix_sort<4>(ctx, src, nr, bits));
    else CT2G_TRY(radix_sort<16>(ctx, src, nr, bits));
    gather_kernel<<<ct2g_div_up(nr, T), T, 0, st>>>(
        ctx->vals, begin, nr, mbits, ctx->x, ctx->y, ctx->z, ctx->vx, ctx->vy, ctx->vz,
        ctx->rung, ctx->id, ctx->x2, ctx->y2, ctx->z2, ctx->vx2, ctx->vy2, ctx->vz2, ctx->rung2,
        ctx->id2, ctx->src, !ctx->defer_vel);
    CT2G_LAUNCHED(ctx);
    copy_back_kernel<<<ct2g_div_up(nr, T), T, 0, st>>>(
        begin, nr, ctx->x2, ctx->y2, ctx->z2, ctx->vx2, ctx->vy2, ctx->vz2, ctx->rung2, ctx->id2,
        ctx->x, ctx->y, ctx->z, ctx->vx, ctx->vy, ctx->vz, ctx->rung, ctx->id, !ctx->defer_vel);
    CT2G_LAUNCHED(ctx);
    ctx->vel_pending = ctx->defer_vel;
    cells_kernel<<<ct2g_div_up((size_t)ctx->CB, kCellTile), kCellThreads, 0, st>>>(
        ctx->keys, begin, nr, (size_t)ctx->CB, ctx->dense_cell, ctx->cell_start, ctx->occ, counts,
        ctx->chunks, ctx->schunks, ctx->sparse_list);
    CT2G_LAUNCHED(ctx);
  } else {
    // empty range: every cell empty
    fill_kernel<<<ct2g_div_up(ctx->CB + 1, T), T, 0, st>>>(ctx->cell_start, ctx->CB + 1,
                                                          (uint32_t)begin);
    CT2G_LAUNCHED(ctx);
    CT2G_CUDA(ctx, cudaMemsetAsync(ctx->occ, 0, sizeof(unsigned long long) * (ctx->CB / 64), st));
  }
  ctx->grid_valid = true;
  ctx->moments_valid = false;
  ctx->expansions_valid = false;
  ctx->forces_valid = false;
  return CT2G_OK;
}

// The second half of a deferred gather (ctx->defer_vel at binning): the
// velocities and rungs of the binned range into cell order, after `stream`
// has waited for ctx->ev_vel (the host-state step's velocity upload; a no-op
// wait otherwise).  Bitwise the same store as the one-pass gather.
int ct2g_gather_velocities(ct2g_ctx *ctx) {
  if (!ctx->vel_pending) return CT2G_OK;
  ctx->vel_pending = false;
  const size_t begin = ctx->rung_begin, nr = ctx->n - ctx->rung_begin;
  cudaStream_t st = ctx->stream;
  CT2G_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_vel,
                                     ctx->capturing ? cudaEventWaitExternal : 0));
  if (nr == 0) return CT2G_OK;
  const unsigned T = 256;
  gather_vel_kernel<<<ct2g_div_up(nr, T), T, 0, st>>>(begin, nr, ctx->vx, ctx->vy, ctx->vz,
                                                      ctx->rung, ctx->vx2, ctx->vy2, ctx->vz2,
                                                      ctx->rung2);
  CT2G_LAUNCHED(ctx);
  copy_back_vel_kernel<<<ct2g_div_up(nr, T), T, 0, st>>>(begin, nr, ctx->vx2, ctx->vy2,
                                                         ctx->vz2, ctx->rung2, ctx->vx, ctx->vy,
                                                         ctx->vz, ctx->rung);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}
