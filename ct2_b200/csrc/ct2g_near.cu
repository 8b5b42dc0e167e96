// Direct-sum near field (kick_cell, src/kick.cpp:3-74) and the order of the
// force stages.
//
// Defects of the reference fixed here: the source loop advanced by one but
// loaded eight sources (kick.cpp:38-43), and the near-field force was reduced
// from the far-field accumulator (kick.cpp:72).
#include "ct2g_internal.cuh"

namespace {

// ---------------------------------------------------------------------------
// Near-field neighbour walk.  The stencil (offsets |o|^2 <= bwidth^2, bwidth
// <= 4) of a cell touches the 27 4x4x4 cell blocks around its own; a block
// is 64 consecutive Morton keys, so its occupancy is one 64-bit word.  For
// the cell at in-block position p and block offset o, stmask[p*27+o] holds
// the stencil cells of that block; occ & stmask lists exactly the occupied
// stencil cells.  Neighbour block keys come from dilated (bit-interleaved)
// addition, which wraps periodically by itself.
// ---------------------------------------------------------------------------
struct Walk {
  uint32_t mx, my, mz;  // block-key masks of the x, y, z bits; the bits above
                        // them are the box index, which the walk keeps
  // neighbouring block o = 9 (dx + 1) + 3 (dy + 1) + (dz + 1): a dilated step
  // of -1 is every bit of the axis' mask, +1 its lowest bit (from the masks
  // of this launch's own mesh: contexts of several meshes share the GPU)
  __device__ __forceinline__ static uint32_t step(uint32_t sb, uint32_t m, int d) {
    const uint32_t off = d == 0 ? m : d == 2 ? (m & (0u - m)) : 0u;
    return ((sb | ~m) + off) & m;
  }
  __device__ __forceinline__ uint32_t add(uint32_t sb, int o) const {
    return step(sb, mx, o / 9) | step(sb, my, (o / 3) % 3) | step(sb, mz, o % 3) |
           (sb & ~(mx | my | mz));
  }
};

// ---------------------------------------------------------------------------
// Packed pairs: Blackwell's f32x2 add/mul/fma do two FP32 operations per
// issued instruction.  A warp's source batch is staged as arrays of x, y and z
// (and, sparse, of cell bits), so that one 16-byte broadcast load of each
// feeds four interactions of every sink a lane holds.
// ---------------------------------------------------------------------------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(f32x2 v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ void inblock(int b, int &x, int &y, int &z) {
  x = ((b >> 2) & 1) | ((b >> 4) & 2);
  y = ((b >> 1) & 1) | ((b >> 3) & 2);
  z = (b & 1) | ((b >> 2) & 2);
}

// index of the r-th set bit (r < popcount) of w
__device__ __forceinline__ int nth_set_bit(unsigned long long w, uint32_t r) {
  int base = 0;
  uint32_t c = __popc((uint32_t)w);
  if (r >= c) {
    r -= c;
    w >>= 32;
    base = 32;
  }
  uint32_t v = (uint32_t)w;
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
    c = __popc(v & ((1u << h) - 1u));
    if (r >= c) {
      r -= c;
      v >>= h;
      base += h;
    }
  }
  return base;
}

// ---------------------------------------------------------------------------
// Streamed near field.  A chunk is sinks of one cell (dense: up to 64, one or two
// per lane) or the sparse cells' sinks of one 4x4x4 block (sparse: up to 32, one per lane).  Its
// candidate cells (occupancy & the union of its sinks' stencil masks, lane o <
// 27 holding neighbouring block o's word) go in windows of 32, a cell per
// lane; the sources of a window form one stream, staged in batches of 32 and
// evaluated by every lane, two sources per packed instruction.
//
// A dense chunk's candidates all lie in its stencil.  In a sparse chunk a
// lane keeps a 32-bit mask of the window's cells in its own stencil: the
// lanes of one in-block position share it, so it is one ballot of "cell
// (lane) is in the stencil of position p" per distinct position (3-4 per
// chunk); a staged source carries its cell's bit, and a lane outside zeroes
// 1/r with a select.
//
// Staging: the source at stream position g belongs to the last cell whose
// first position is <= g.  The cells' first positions inside the batch are
// OR-reduced into one word of head bits, so the owner is a population count,
// and a table of the window in shared memory gives its (first particle - first
// position) and its centre in the chunk's frame (the sink cell's centre; that of the
// block's first cell for a sparse chunk).  Sources are staged negated, so that
// the inner loop adds.
//
// What bounds it: 11 packed FP32 instructions and two MUFU operations per two
// interactions (22 and 16 cycles of their pipes per warp and SM sub-partition), so
// 11.6 interactions per clock and SM, 3.4e12 per second, when nothing else
// is issued.  A packed instruction takes two issue slots, so what else a pair
// needs (two shared loads, two MUFU, its share of the staging) counts against
// it: FMA pipe 71%, all issue slots used; two sinks per lane halve that share.
// Against one warp per chunk, cells' sources in batches of their own half
// blocks (dense), a table of stencil entries per lane in shared memory (sparse)
// and scalar arithmetic cell by cell (sphere kernel), the near field of 2.5 M particles in halos
// (mesh 256, 7.7e10 interactions) takes 38.5 -> 33.2 ms, of 50 k in spheres (mesh 64) 478 -> 178
// us, of 12 boxes of 30 k 1054 -> 686, of 128^3 in Plummer spheres (256) 3.48 -> 3.34 ms;
// forces and potentials of 300 k in halos with the sphere kernel 7.7 -> 5.0 to
// 12.6 -> 7.9 ms a call, by the particles.
// Register bounds: 64 (sparse, four blocks of eight warps per SM) and 80 (three, dense and
// heavy) spill 4-24 and 8-16 bytes a thread, the sparse sphere kernel with potentials 152;
// three blocks per SM instead (28 bytes) measured the same, 6.16 and 6.15 ms a call of the above.
// ---------------------------------------------------------------------------
struct NearArgs {
  const uint2 *dchunks;     // dense chunks (first particle, sinks), *ndense of them
  const uint32_t *ndense;
  const uint2 *schunks;     // sparse chunks (first sparse_list entry, sinks),
  const uint32_t *nsparse;  // *nsparse of them (null: none)
  const uint32_t *slist;
  const uint32_t *cs;
  const unsigned long long *occ, *stm;
  Walk walk;
  const uint32_t *skeys;
  uint32_t rbegin;
  const float4 *src;        // offsets from the own cell's centre
  int mbits;
  float soft;
  int lo2, hi2;             // sparse: source cells with lo2 < |o|^2 <= hi2 of a lane's own
  const float *box_gm;
  float *ofx, *ofy, *ofz, *opot;
  bool store;               // store into the buffers instead of adding to them
  uint32_t *work;           // [0] sparse chunks taken, [1] heavy ones among them,
                            // [2] dense and heavy chunks taken
  uint32_t *heavy;          // list of the heavy chunks
  uint32_t heavy_min;       // sources a sparse chunk may have to stay with one warp
  uint32_t warps;           // warps the launch may spread few chunks over
  uint32_t maxch;
  unsigned long long *inter;
};

// A sparse chunk whose 27 neighbouring blocks hold more sources than A.heavy_min is
// left to the cooperative launch: one warp on its own walks 1000 sources in
// about 10 us, and clustered sets have sparse chunks beside cells of 10^5 (2.5 ms
// on a single warp while the rest of the GPU idled, at 400 k particles in 48
// halos).  A block per chunk costs its eight warps the setup, so that it only
// pays where a warp's chunk is long against the launch: a mesh of M has (M/4)^3
// blocks, under one round of the GPU's warps up to 64, 7 at 128, 55 at 256.
// Near field in ms at limits of 1024 / 4096 / 8192 / 16384 / none: 50 k particles, mesh
// 64, 0.180 / 0.287 / 0.351 / 0.358 / 0.354; 12 such boxes of 30 k (the boxes' blocks in all
// do not matter: each box has its long chunks) 0.68 / 0.76 / 0.85 / 0.91 / 0.91; 2.1 M in
// spheres, 256, 3.66 / 3.42 / 3.35 / 3.35 / 3.35; 4 M in spheres, 512, 6.07 / 4.74 / 4.56 / 4.56 / 4.57;
// 4 M in halos, 512, 29.96 / 29.95 / 30.00 / 29.99 / 29.93.  Steps with the learned
// correction (262 k, 128) 2.75 / 2.82 (3072) / 2.96 / 2.96.  From 256 on any limit of 8192 or
// more measures the same; 8192 keeps one warp below some 80 us in sets that were not measured.
uint32_t heavy_min(int M) { return M <= 128 ? 1024u : 8192u; }
// SPLIT: the sparse sinks of the sphere kernel.  A coordinate in the frame of a
// 4-cell block has lost up to three bits of the offset from its own cell's centre, so that
// the separation of two particles of one cell was off by up to 4 ulp of a
// cell (forces 1e-6 to 3e-6 rms off where the cell-by-cell form is 1e-7); so sinks and sources
// keep offset and cell centre apart, and a separation is (offset - offset) + (centre - centre):
// exact inside a cell, rounded at the size of a cell and of itself beyond.  Two
// more packed additions and half a broadcast load per coordinate and pair.  (The dense
// chunks' frame is the sink cell itself, where the pairs of the cell are exact as they are;
// the Plummer kernel's sparse sinks are staged in the block's frame.)
template <int KERNEL, bool SPARSE>
constexpr bool kSplit = KERNEL == CT2G_SOFT_SPHERE && SPARSE;
// floats of staging per warp: two batches (x, y, z and cell bits of 32
// sources; SPLIT: their cells' centres), then the window's table
template <bool SPLIT>
constexpr int kBatch = SPLIT ? 224 : 128;
template <bool SPLIT>
constexpr int kStage = 2 * kBatch<SPLIT> + 128;
// a coordinate that makes r^2 infinite: an empty slot of the last batch adds 0
constexpr float kFar = 3e19f;

// g = the softened 1/r^3 and pp = 1/r of two sources at separation (dx, dy, dz);
// a source that is off gives zeros
template <int KERNEL, bool POT, bool MASKED>
__device__ __forceinline__ void pair_weights(f32x2 dx, f32x2 dy, f32x2 dz, f32x2 H2, float h2,
                                             float hinv, float hinv3, bool on0, bool on1,
                                             f32x2 &g, f32x2 &pp) {
  if constexpr (KERNEL == CT2G_SOFT_PLUMMER) {
    const f32x2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, H2)));
    float r0, r1;
    f2_unpack(r2, r0, r1);
    r0 = rsqrtf(r0);
    r1 = rsqrtf(r1);
    if (MASKED) {
      r0 = on0 ? r0 : 0.f;
      r1 = on1 ? r1 : 0.f;
    }
    pp = f2_pack(r0, r1);
    g = f2_mul(f2_mul(pp, pp), pp);
  } else {
    // 1/h^3 inside r = h, 1/r^3 outside (continuous, so the smaller of the two)
    const f32x2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx)));
    float r0, r1, g0, g1;
    f2_unpack(r2, r0, r1);
    float p0 = rsqrtf(r0), p1 = rsqrtf(r1);
    const f32x2 ri = f2_pack(p0, p1);
    f2_unpack(f2_mul(f2_mul(ri, ri), ri), g0, g1);
    g0 = fminf(g0, hinv3);
    g1 = fminf(g1, hinv3);
    if (POT) {
      p0 = r0 < h2 ? fmaf(-0.5f * r0, hinv3, 1.5f * hinv) : p0;
      p1 = r1 < h2 ? fmaf(-0.5f * r1, hinv3, 1.5f * hinv) : p1;
    }
    if (MASKED) {
      g0 = on0 ? g0 : 0.f;
      g1 = on1 ? g1 : 0.f;
      p0 = on0 ? p0 : 0.f;
      p1 = on1 ? p1 : 0.f;
    }
    g = f2_pack(g0, g1);
    pp = f2_pack(p0, p1);
  }
}

// a lane's sink (coordinates in both halves; SPLIT: its offset, and its cell's
// centre in CX, CY, CZ) and its packed sums +d g, +1/r (the caller negates)
struct Sink {
  f32x2 X, Y, Z, ax, ay, az, ap, CX, CY, CZ;
};

// interactions of NS sinks with the four sources of quad qd (negated
// coordinates in the staged arrays)
template <int KERNEL, bool POT, bool MASKED, int NS>
__device__ __forceinline__ void quad_term(const float *sb, int qd, uint32_t bits, Sink (&k)[NS],
                                          f32x2 H2, float h2, float hinv, float hinv3) {
  const float4 x = reinterpret_cast<const float4 *>(sb)[qd];
  const float4 y = reinterpret_cast<const float4 *>(sb + 32)[qd];
  const float4 z = reinterpret_cast<const float4 *>(sb + 64)[qd];
  bool on[4] = {true, true, true, true};
  if (MASKED) {
    const uint4 m = reinterpret_cast<const uint4 *>(sb + 96)[qd];
    on[0] = (m.x & bits) != 0u;
    on[1] = (m.y & bits) != 0u;
    on[2] = (m.z & bits) != 0u;
    on[3] = (m.w & bits) != 0u;
  }
  const f32x2 px[2] = {f2_pack(x.x, x.y), f2_pack(x.z, x.w)};
  const f32x2 py[2] = {f2_pack(y.x, y.y), f2_pack(y.z, y.w)};
  const f32x2 pz[2] = {f2_pack(z.x, z.y), f2_pack(z.z, z.w)};
  f32x2 cx[2], cy[2], cz[2];
  if constexpr (kSplit<KERNEL, MASKED>) {
    const float4 a = reinterpret_cast<const float4 *>(sb + 128)[qd];
    const float4 b = reinterpret_cast<const float4 *>(sb + 160)[qd];
    const float4 c = reinterpret_cast<const float4 *>(sb + 192)[qd];
    cx[0] = f2_pack(a.x, a.y), cx[1] = f2_pack(a.z, a.w);
    cy[0] = f2_pack(b.x, b.y), cy[1] = f2_pack(b.z, b.w);
    cz[0] = f2_pack(c.x, c.y), cz[1] = f2_pack(c.z, c.w);
  }
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int u = 0; u < NS; u++) {
      f32x2 dx = f2_add(k[u].X, px[h]), dy = f2_add(k[u].Y, py[h]), dz = f2_add(k[u].Z, pz[h]);
      if constexpr (kSplit<KERNEL, MASKED>) {
        dx = f2_add(dx, f2_add(k[u].CX, cx[h]));
        dy = f2_add(dy, f2_add(k[u].CY, cy[h]));
        dz = f2_add(dz, f2_add(k[u].CZ, cz[h]));
      }
      f32x2 g, pp;
      pair_weights<KERNEL, POT, MASKED>(dx, dy, dz, H2, h2, hinv, hinv3, on[2 * h], on[2 * h + 1],
                                        g, pp);
      k[u].ax = f2_fma(dx, g, k[u].ax);
      k[u].ay = f2_fma(dy, g, k[u].ay);
      k[u].az = f2_fma(dz, g, k[u].az);
      if (POT) k[u].ap = f2_add(k[u].ap, pp);
    }
}

// the NS sinks per lane of a chunk and what its warp walks
template <bool SPARSE, int NS>
struct Chunk {
  uint32_t idx[NS];         // this lane's sinks (an inactive one repeats the first)
  uint32_t key, p;          // of the first; its position in the block
  unsigned long long pm;    // in-block positions present in the chunk
  unsigned long long word;  // lane o < 27: candidate cells of neighbouring block o,
  uint32_t nblk;            // and its block key
  uint32_t ex1, C;          // candidate cells before block o's, and in all
  int fx, fy, fz;           // the frame's cell in the block: the sink cell, or (sparse) 0
  __device__ __forceinline__ void open(const NearArgs &A, const uint2 cd, int lane) {
#pragma unroll
    for (int u = 0; u < NS; u++) {
      const uint32_t e = (uint32_t)(lane + 32 * u);
      const uint32_t slot = cd.x + (e < cd.y ? e : 0u);
      idx[u] = SPARSE ? A.slist[slot] : slot;
    }
    key = A.skeys[idx[0] - A.rbegin];
    p = key & 63u;
    const uint32_t blk = key >> 6;  // the same for the whole chunk
    pm = 1ull << p;
    if (SPARSE)
      pm = ((unsigned long long)__reduce_or_sync(0xffffffffu, (uint32_t)(pm >> 32)) << 32) |
           __reduce_or_sync(0xffffffffu, (uint32_t)pm);
    word = 0;
    nblk = 0;
    if (lane < 27) {
      nblk = A.walk.add(blk, lane);
      unsigned long long m = 0, q = pm;
      while (q) {
        const int pp = __ffsll((long long)q) - 1;
        q &= q - 1;
        m |= __ldg(A.stm + pp * 27 + lane);
      }
      word = A.occ[nblk] & m;
    }
    const uint32_t c1 = (uint32_t)__popcll(word);
    uint32_t in1 = c1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, in1, d);
      if (lane >= d) in1 += t;
    }
    ex1 = in1 - c1;
    C = __shfl_sync(0xffffffffu, in1, 31);
    fx = fy = fz = 0;
    if (!SPARSE) inblock((int)p, fx, fy, fz);
  }
  // sources of the neighbouring blocks that hold candidates (an upper bound)
  __device__ __forceinline__ uint32_t sources(const NearArgs &A) const {
    const uint32_t w = word ? A.cs[(size_t)(nblk + 1) << 6] - A.cs[(size_t)nblk << 6] : 0u;
    return __reduce_add_sync(0xffffffffu, w);
  }
  template <bool SPLIT>
  __device__ __forceinline__ void sinks(const NearArgs &A, float hc, Sink (&k)[NS]) const {
    int ix, iy, iz;
    inblock((int)p, ix, iy, iz);
    const float cx = (float)(ix - fx) * hc, cy = (float)(iy - fy) * hc, cz = (float)(iz - fz) * hc;
#pragma unroll
    for (int u = 0; u < NS; u++) {
      const float4 q = A.src[idx[u]];
      const float sx = SPLIT ? q.x : cx + q.x, sy = SPLIT ? q.y : cy + q.y,
                  sz = SPLIT ? q.z : cz + q.z;
      k[u] = Sink{f2_pack(sx, sx), f2_pack(sy, sy), f2_pack(sz, sz), 0ull, 0ull, 0ull, 0ull,
                  f2_pack(cx, cx), f2_pack(cy, cy), f2_pack(cz, cz)};
    }
  }
  // The window of candidate cells w0 ..: its table (a cell per lane: its centre
  // from the frame's, negated, and its first particle less its first stream position) into
  // win, its first stream position in `excl` (~0 past the last cell), the
  // sources in `total`, and (sparse) this lane's mask of the cells in its own
  // stencil in `bits`; nsrc counts the sources of a lane's stencil.
  __device__ __forceinline__ void window(const NearArgs &A, uint32_t w0, float hc, int lane,
                                         float4 *win, uint32_t &excl, uint32_t &total,
                                         uint32_t &bits, uint32_t &nsrc) const {
    const bool valid = w0 + (uint32_t)lane < C;
    // the (g - ex1[o])-th candidate cell of block o
    const uint32_t g = min(w0 + (uint32_t)lane, C - 1);
    int o = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const uint32_t e = __shfl_sync(0xffffffffu, ex1, o + step);
      if (e <= g) o += step;
    }
    const unsigned long long wo = __shfl_sync(0xffffffffu, word, o);
    const uint32_t nbo = __shfl_sync(0xffffffffu, nblk, o);
    const uint32_t exo = __shfl_sync(0xffffffffu, ex1, o);
    const int q = nth_set_bit(wo, g - exo);
    uint32_t jb = 0, c = 0;
    if (valid) {
      const uint32_t ck = (nbo << 6) | (uint32_t)q;
      jb = A.cs[ck];
      c = A.cs[ck + 1] - jb;
    }
    uint32_t incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    total = __shfl_sync(0xffffffffu, incl, 31);
    excl = valid ? incl - c : 0xffffffffu;
    int bx, by, bz;
    inblock(q, bx, by, bz);
    const int cx = 4 * (o / 9 - 1) + bx, cy = 4 * ((o / 3) % 3 - 1) + by, cz = 4 * (o % 3 - 1) + bz;
    win[lane] = make_float4((float)(fx - cx) * hc, (float)(fy - cy) * hc, (float)(fz - cz) * hc,
                            __uint_as_float(jb - (incl - c)));
    bits = 0xffffffffu;
    if (SPARSE) {
      bits = 0u;
      unsigned long long pq = pm;
      while (pq) {
        const int pp = __ffsll((long long)pq) - 1;
        pq &= pq - 1;
        int qx, qy, qz;
        inblock(pp, qx, qy, qz);
        const int d2 = (cx - qx) * (cx - qx) + (cy - qy) * (cy - qy) + (cz - qz) * (cz - qz);
        const bool in = valid && d2 > A.lo2 && d2 <= A.hi2;
        const uint32_t bal = __ballot_sync(0xffffffffu, in);
        const uint32_t sum = __reduce_add_sync(0xffffffffu, in ? c : 0u);
        if ((int)p == pp) {
          bits = bal;
          nsrc += sum;
        }
      }
    } else {
      nsrc += total;
    }
  }
};

// the window slot of stream position b + lane (clamped to the last), and its source
__device__ __forceinline__ uint32_t stream_slot(uint32_t excl, uint32_t b, uint32_t g1) {
  const uint32_t before = __ballot_sync(0xffffffffu, excl < b);
  const uint32_t rel = excl - b;
  const uint32_t heads = __reduce_or_sync(0xffffffffu, rel < 32u ? 1u << rel : 0u);
  return __popc(before) + __popc(heads & (0xffffffffu >> (31u - (g1 - b)))) - 1;
}

// a fetched source (offset q from its cell's centre, slot t of the window) into
// a staged batch; off: an empty slot
template <bool SPARSE, bool SPLIT>
__device__ __forceinline__ void stage_source(float *sb, const float4 &w, const float4 &q,
                                             uint32_t t, bool on, int lane) {
  sb[lane] = !on ? kFar : SPLIT ? -q.x : w.x - q.x;
  sb[32 + lane] = SPLIT ? -q.y : w.y - q.y;
  sb[64 + lane] = SPLIT ? -q.z : w.z - q.z;
  if (SPARSE) sb[96 + lane] = __uint_as_float(on ? 1u << t : 0u);
  if (SPLIT) {
    sb[128 + lane] = w.x;
    sb[160 + lane] = w.y;
    sb[192 + lane] = w.z;
  }
}

struct Soft {
  f32x2 H2;
  float h2, hinv, hinv3;
  __device__ __forceinline__ explicit Soft(float h)
      : H2(f2_pack(h * h, h * h)), h2(h * h), hinv(1.f / h), hinv3(0.f) {
    hinv3 = hinv * hinv * hinv;
  }
};

// a staged batch of n <= 32 sources
template <int KERNEL, bool POT, bool SPARSE, int NS>
__device__ __forceinline__ void eval_batch(const float *sb, uint32_t n, uint32_t bits,
                                           Sink (&k)[NS], const Soft &h) {
  if (n >= 32) {
#pragma unroll 4
    for (int qd = 0; qd < 8; qd++)
      quad_term<KERNEL, POT, SPARSE, NS>(sb, qd, bits, k, h.H2, h.h2, h.hinv, h.hinv3);
  } else {
    const int nq = (int)(n + 3) >> 2;
#pragma unroll 1
    for (int qd = 0; qd < nq; qd++)
      quad_term<KERNEL, POT, SPARSE, NS>(sb, qd, bits, k, h.H2, h.h2, h.hinv, h.hinv3);
  }
}

// a sink's packed sums so far, and back to zero
template <bool POT>
__device__ __forceinline__ float4 take(Sink &k) {
  float a0, a1;
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  f2_unpack(k.ax, a0, a1);
  v.x = a0 + a1;
  f2_unpack(k.ay, a0, a1);
  v.y = a0 + a1;
  f2_unpack(k.az, a0, a1);
  v.z = a0 + a1;
  if (POT) {
    f2_unpack(k.ap, a0, a1);
    v.w = a0 + a1;
  }
  k.ax = k.ay = k.az = k.ap = 0ull;
  return v;
}
__device__ __forceinline__ void add(float4 &n, const float4 &v) {
  n.x += v.x;
  n.y += v.y;
  n.z += v.z;
  n.w += v.w;
}

// The sums (negated) times GM, added to the far field (L2P, with GM) already in
// the force buffers, or stored into the near-field buffers when the two run
// side by side; the product is rounded on its own (no fused multiply-add into
// the far field), so that both forms add the same two values.
template <bool POT>
__device__ __forceinline__ void write_sink(const NearArgs &A, uint32_t i, uint32_t key,
                                           const float4 &n) {
  const float GM = __ldg(A.box_gm + (key >> (3 * A.mbits)));
  const float gx = __fmul_rn(GM, -n.x), gy = __fmul_rn(GM, -n.y), gz = __fmul_rn(GM, -n.z);
  if (A.store) {
    A.ofx[i] = gx;
    A.ofy[i] = gy;
    A.ofz[i] = gz;
    if (POT) A.opot[i] = __fmul_rn(GM, -n.w);
  } else {
    A.ofx[i] += gx;
    A.ofy[i] += gy;
    A.ofz[i] += gz;
    if (POT) A.opot[i] += __fmul_rn(GM, -n.w);
  }
}

// the barrier of the S warps (a power of two) that share a chunk
__device__ __forceinline__ void group_sync(int S, int group) {
  if (S > 1) asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(32 * S) : "memory");
}

// One sparse chunk by the S warps that share it: warp s takes the windows s,
// s + S, ..., and warp 0 adds each round's S sums in order, so the result does
// not depend on S.  stage: this warp's kStage floats (the group's warps' lie
// one after another).  A heavy chunk is left alone (false returned).
template <int KERNEL, bool POT>
__device__ __forceinline__ bool sparse_chunk(const NearArgs &A, const uint2 cd, int s, int S,
                                             int group, float *stage, int lane) {
  constexpr bool SPLIT = kSplit<KERNEL, true>;
  Chunk<true, 1> k;
  k.open(A, cd, lane);
  if (k.sources(A) > A.heavy_min) return false;
  const float hc = 1.0f / (float)(1 << A.mbits);
  Sink sink[1];
  k.template sinks<SPLIT>(A, hc, sink);
  const Soft soft(A.soft);
  float4 tot = make_float4(0.f, 0.f, 0.f, 0.f);
  uint32_t nsrc = 0;
  float4 *win = reinterpret_cast<float4 *>(stage + 2 * kBatch<SPLIT>);
  for (uint32_t r0 = 0; r0 < k.C; r0 += 32u * (uint32_t)S) {
    const uint32_t w0 = r0 + 32u * (uint32_t)s;
    if (w0 < k.C) {
      uint32_t excl, total, bits, t = 0;
      __syncwarp();  // the previous window's table and last batch are read
      k.window(A, w0, hc, lane, win, excl, total, bits, nsrc);
      __syncwarp();
      float4 nq = make_float4(0.f, 0.f, 0.f, 0.f);
      auto fetch = [&](uint32_t b) {
        const uint32_t g1 = min(b + (uint32_t)lane, total - 1);
        t = stream_slot(excl, b, g1);
        nq = __ldg(A.src + (__float_as_uint(win[t].w) + g1));
      };
      float *sb = stage;
      if (total) fetch(0u);
      for (uint32_t b = 0; b < total; b += 32u) {
        stage_source<true, SPLIT>(sb, win[t], nq, t, b + (uint32_t)lane < total, lane);
        __syncwarp();
        if (b + 32u < total) fetch(b + 32u);
        eval_batch<KERNEL, POT, true, 1>(sb, total - b, bits, sink, soft);
        sb = sb == stage ? stage + kBatch<SPLIT> : stage;
      }
    }
    const float4 v = take<POT>(sink[0]);
    if (S == 1) {
      add(tot, v);
    } else {
      __syncwarp();  // every lane is done with this warp's staging
      if (s > 0) reinterpret_cast<float4 *>(stage)[lane] = v;
      group_sync(S, group);
      if (s == 0) {
        add(tot, v);
        const int nw = (int)min((uint32_t)S, (k.C - r0 + 31u) / 32u);
        for (int u = 1; u < nw; u++) add(tot, reinterpret_cast<const float4 *>(stage + u * kStage<SPLIT>)[lane]);
      }
      group_sync(S, group);
    }
  }
  if (A.inter) {
    const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)lane < cd.y ? nsrc : 0u);
    if (lane == 0 && c) atomicAdd(A.inter, (unsigned long long)c);
  }
  if (s == 0 && (uint32_t)lane < cd.y) write_sink<POT>(A, k.idx[0], k.key, tot);
  return true;
}

// The sparse chunks, taken from a device counter by groups of S warps; blocks
// are persistent.  S = 1 wherever the chunks alone fill the warps the GPU
// holds (A.warps); fewer are shared by 2, 4 or 8 warps each (12^3 particles on
// a 16^3 mesh are 64 chunks: 48 us with one warp each on 7 blocks).  The sums
// do not depend on S.
template <int KERNEL, bool POT>
__global__ void __launch_bounds__(256, 4) near_sparse_kernel(const NearArgs A) {
  constexpr int ST = kStage<kSplit<KERNEL, true>>;
  __shared__ __align__(16) float stage[8 * ST];
  __shared__ uint32_t taken_s[2][8];  // by the parity of the turn: one barrier a turn
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t nch = *A.nsparse;
  const uint2 *list = A.schunks;
  int S = 8;
  while (S > 1 && (size_t)nch * S > A.warps) S >>= 1;
  const int s = wib & (S - 1), group = wib / S;
  // maxch > 0: a group takes at most maxch chunks and the block then exits,
  // so that blocks of kernels on other streams get the SM in between
  for (uint32_t taken = 0; A.maxch == 0 || taken < A.maxch; taken++) {
    uint32_t ch = 0;
    if (S > 1) {
      if (s == 0 && lane == 0) taken_s[taken & 1][group] = atomicAdd(A.work, 1u);
      group_sync(S, group);
      ch = taken_s[taken & 1][group];
    } else {
      if (lane == 0) ch = atomicAdd(A.work, 1u);
      ch = __shfl_sync(0xffffffffu, ch, 0);
    }
    if (ch >= nch) break;
    if (!sparse_chunk<KERNEL, POT>(A, list[ch], s, S, group, stage + wib * ST, lane) &&
        s == 0 && lane == 0)
      A.heavy[atomicAdd(A.work + 1, 1u)] = ch;
  }
}

// Dense chunks and heavy sparse ones: a block each.  The eight warps tabulate
// eight windows at a time, one each, and take the segments of kSeg sources of these
// windows in turn; their sums are added in warp order at the end.  A chunk
// then takes a few us, so that the last ones leave no tail (a warp each: 64^3
// particles in Plummer spheres had 2200 dense chunks for 3552 warps, and the
// launch half idle).  NS sinks per lane: a dense chunk of more than 32 sinks
// holds two, so that each staged quad feeds eight interactions.
constexpr uint32_t kSeg = 256;
template <int KERNEL>
struct CoopSmem {
  float stage[8][2 * kBatch<kSplit<KERNEL, true>>];
  float4 win[8][32];
  uint32_t excl[8][32], bits[8][32], total[8];
  uint32_t chunk[2];
};

template <int KERNEL, bool POT, bool SPARSE, int NS>
__device__ __forceinline__ void coop_chunk(const NearArgs &A, const uint2 cd,
                                           CoopSmem<KERNEL> &sm, int wib, int lane) {
  constexpr bool SPLIT = kSplit<KERNEL, SPARSE>;
  Chunk<SPARSE, NS> k;
  k.open(A, cd, lane);
  const float hc = 1.0f / (float)(1 << A.mbits);
  Sink sink[NS];
  k.template sinks<SPLIT>(A, hc, sink);
  const Soft soft(A.soft);
  uint32_t nsrc = 0;
  for (uint32_t r0 = 0; r0 < k.C; r0 += 256u) {
    const uint32_t w0 = r0 + 32u * (uint32_t)wib;
    uint32_t excl = 0xffffffffu, total = 0, bits = 0;
    if (r0) __syncthreads();  // the previous round's tables are read
    if (w0 < k.C) k.window(A, w0, hc, lane, sm.win[wib], excl, total, bits, nsrc);
    sm.excl[wib][lane] = excl;
    if (SPARSE) sm.bits[wib][lane] = bits;
    if (lane == 0) sm.total[wib] = total;
    __syncthreads();
    // this warp's place: window w, batch at b of its tot sources; segments
    // are numbered through the windows, this warp's are wib, wib + 8, ...
    uint32_t w = 0, b = 0, tot = sm.total[0], skip = (uint32_t)wib;
    auto seek = [&]() {  // to the segment `skip` segments on from (w, b); w = 8: none
      for (;;) {
        const uint32_t left = b < tot ? (tot - b + kSeg - 1) / kSeg : 0u;
        if (skip < left) {
          b += skip * kSeg;
          break;
        }
        skip -= left;
        b = 0;
        if (++w == 8) break;
        tot = sm.total[w];
      }
      if (w < 8) {
        excl = sm.excl[w][lane];
        if (SPARSE) bits = sm.bits[w][lane];
      }
    };
    seek();
    uint32_t t = 0;
    float4 nq = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&]() {
      const uint32_t g1 = min(b + (uint32_t)lane, tot - 1);
      t = stream_slot(excl, b, g1);
      nq = __ldg(A.src + (__float_as_uint(sm.win[w][t].w) + g1));
    };
    float *sb = sm.stage[wib];
    if (w < 8) fetch();
    __syncwarp();  // the last batch of the round before is read
    while (w < 8) {
      stage_source<SPARSE, SPLIT>(sb, sm.win[w][t], nq, t, b + (uint32_t)lane < tot, lane);
      __syncwarp();
      const uint32_t n = tot - b, eb = bits;
      b += 32u;
      if (b % kSeg == 0u || b >= tot) {  // the segment's end: seven segments on
        skip = 7u;
        if (b >= tot) b = tot;
        seek();
      }
      if (w < 8) fetch();
      eval_batch<KERNEL, POT, SPARSE, NS>(sb, n, eb, sink, soft);
      sb = sb == sm.stage[wib] ? sm.stage[wib] + kBatch<SPLIT> : sm.stage[wib];
    }
  }
  // the eight warps' sums, in order
  __syncwarp();
#pragma unroll
  for (int u = 0; u < NS; u++)
    reinterpret_cast<float4 *>(sm.stage[wib])[32 * u + lane] = take<POT>(sink[u]);
  if (A.inter) {  // (each warp has counted its own windows)
    unsigned long long c;
    if (SPARSE)
      c = __reduce_add_sync(0xffffffffu, (uint32_t)lane < cd.y ? nsrc : 0u);
    else
      c = (unsigned long long)nsrc * cd.y;
    if (lane == 0 && c) atomicAdd(A.inter, c);
  }
  __syncthreads();
  if (wib < NS) {  // warp u: the lanes' sinks u
    float4 n = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int v = 0; v < 8; v++) add(n, reinterpret_cast<const float4 *>(sm.stage[v])[32 * wib + lane]);
    const uint32_t e = (uint32_t)(lane + 32 * wib);
    if (e < cd.y) write_sink<POT>(A, SPARSE ? k.idx[0] : cd.x + e, k.key, n);
  }
}

template <int KERNEL, bool POT>
__global__ void __launch_bounds__(256, 3) near_coop_kernel(const NearArgs A) {
  __shared__ __align__(16) CoopSmem<KERNEL> sm;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t nh = A.nsparse ? A.work[1] : 0u, nch = nh + *A.ndense;
  if (threadIdx.x == 0) sm.chunk[0] = atomicAdd(A.work + 2, 1u);
  for (uint32_t taken = 0; A.maxch == 0 || taken < 8 * A.maxch; taken++) {
    __syncthreads();  // the chunk's number is there, the previous chunk's sums are read
    const uint32_t ch = sm.chunk[taken & 1];
    if (ch >= nch) break;
    // the next one, asked for early (none that this block would not take)
    if (threadIdx.x == 0 && (A.maxch == 0 || taken + 1 < 8 * A.maxch))
      sm.chunk[(taken + 1) & 1] = atomicAdd(A.work + 2, 1u);
    if (ch < nh) {
      coop_chunk<KERNEL, POT, true, 1>(A, A.schunks[A.heavy[ch]], sm, wib, lane);
    } else {
      const uint2 cd = A.dchunks[ch - nh];
      if (cd.y <= 32)
        coop_chunk<KERNEL, POT, false, 1>(A, cd, sm, wib, lane);
      else
        coop_chunk<KERNEL, POT, false, 2>(A, cd, sm, wib, lane);
    }
  }
}

// Sparse chunks cell by cell (tuning sparse_path 1): one warp per chunk; each
// candidate cell's sources are staged as their own batch, and a lane takes part only
// where the cell lies in its own stencil window (lo2 < |o|^2 <= hi2).
template <int KERNEL, bool POT>
__device__ __forceinline__ void cells_chunk(const NearArgs &A, const uint2 cd, float4 *sb,
                                            int lane) {
  const int M = 1 << A.mbits;
  const bool act = (uint32_t)lane < cd.y;
  const uint32_t slot = cd.x + (act ? (uint32_t)lane : 0u);
  const uint32_t i = A.slist[slot];
  const uint32_t key = A.skeys[i - A.rbegin];
  const float4 si = A.src[i];
  const uint32_t p = key & 63u, blk = key >> 6;  // blk is the same for the whole chunk
  const float GM = __ldg(A.box_gm + (key >> (3 * A.mbits)));
  int px, py, pz;
  inblock((int)p, px, py, pz);
  // cells of the block present in the chunk
  unsigned long long pm = 1ull << p;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pm |= __shfl_xor_sync(0xffffffffu, pm, o);
  unsigned long long word = 0;
  uint32_t nblk = 0;
  if (lane < 27) {
    nblk = A.walk.add(blk, lane);
    unsigned long long m = 0, q = pm;
    while (q) {
      const int pp = __ffsll((long long)q) - 1;
      q &= q - 1;
      m |= __ldg(A.stm + pp * 27 + lane);
    }
    word = A.occ[nblk] & m;
  }
  const float hc = 1.0f / (float)M;
  const float h2 = A.soft * A.soft, hinv = 1.f / A.soft, hinv3 = hinv * hinv * hinv;
  float nx = 0.f, ny = 0.f, nz = 0.f, np = 0.f;
  uint32_t nsrc = 0;
  for (int o = 0; o < 27; o++) {
    unsigned long long bits = __shfl_sync(0xffffffffu, word, o);
    const uint32_t nb = __shfl_sync(0xffffffffu, nblk, o);
    const int dX = 4 * (o / 9 - 1) - px, dY = 4 * ((o / 3) % 3 - 1) - py, dZ = 4 * (o % 3 - 1) - pz;
    while (bits) {
      const int t = __ffsll((long long)bits) - 1;
      bits &= bits - 1;
      const uint32_t ck = (nb << 6) | (uint32_t)t;
      const uint32_t j0 = A.cs[ck], j1 = A.cs[ck + 1];
      int bx, by, bz;
      inblock(t, bx, by, bz);
      const int ox = dX + bx, oy = dY + by, oz = dZ + bz;  // cells, from this lane's cell
      const int d2 = ox * ox + oy * oy + oz * oz;
      const bool in = act && d2 > A.lo2 && d2 <= A.hi2;
      if (in) nsrc += j1 - j0;
      // sink position relative to the neighbour cell's centre
      const float xs = si.x - (float)ox * hc, ys = si.y - (float)oy * hc,
                  zs = si.z - (float)oz * hc;
      float4 nxt = __ldg(A.src + min(j0 + lane, j1 - 1));
      for (uint32_t jj = j0; jj < j1; jj += 32) {
        const int cnt = (int)min(32u, j1 - jj);
        __syncwarp();
        sb[lane] = nxt;
        __syncwarp();
        if (jj + 32 < j1) nxt = __ldg(A.src + min(jj + 32 + lane, j1 - 1));
#pragma unroll 4
        for (int u = 0; u < cnt; u++) {
          const float4 q = sb[u];
          ct2g_pair_term<KERNEL, POT>(xs - q.x, ys - q.y, zs - q.z, h2, hinv, hinv3, nx, ny, nz,
                                      np, in);
        }
      }
    }
  }
  if (act) {  // as write_sink
    const float gx = __fmul_rn(GM, nx), gy = __fmul_rn(GM, ny), gz = __fmul_rn(GM, nz);
    if (A.store) {
      A.ofx[i] = gx;
      A.ofy[i] = gy;
      A.ofz[i] = gz;
      if (POT) A.opot[i] = __fmul_rn(GM, np);
    } else {
      A.ofx[i] += gx;
      A.ofy[i] += gy;
      A.ofz[i] += gz;
      if (POT) A.opot[i] += __fmul_rn(GM, np);
    }
  }
  const uint32_t c = __reduce_add_sync(0xffffffffu, nsrc);
  if (lane == 0 && c && A.inter) atomicAdd(A.inter, (unsigned long long)c);
}

template <int KERNEL, bool POT>
__global__ void __launch_bounds__(256, 4) near_cells_kernel(const NearArgs A) {
  __shared__ float4 sbuf[8][32];  // one batch of 32 sources per warp
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t nch = *A.nsparse;
  const uint2 *list = A.schunks;
  for (uint32_t taken = 0; A.maxch == 0 || taken < A.maxch; taken++) {
    uint32_t ch = 0;
    if (lane == 0) ch = atomicAdd(A.work, 1u);
    ch = __shfl_sync(0xffffffffu, ch, 0);
    if (ch >= nch) break;
    cells_chunk<KERNEL, POT>(A, list[ch], sbuf[wib], lane);
  }
}

// Sparse sinks, one per lane: the warp takes 32 consecutive entries of the
// sparse sink list (cell order within a tile of 2048 cells, so that the lanes are
// mostly neighbours; the tiles in any order) and every lane
// walks the stencil of its own cell -- the 27 neighbouring 4x4x4 blocks,
// occupancy & its own stencil mask, the ranges of the occupied cells -- and
// sums its own sources, read through the read-only cache, two at a time with
// the packed f32x2 arithmetic.  No lane evaluates a source outside its
// stencil, and a warp is not bound to one cell block, so sparse regions fill
// whole warps.  The work counter hands out groups of 32 sinks until the
// device-held sparse count is covered.
template <int KERNEL, bool POT>
__global__ void __launch_bounds__(256, 4) near_lane_kernel(
    const uint32_t *__restrict__ nsparse_ptr, uint32_t *__restrict__ work,
    const uint32_t *__restrict__ sparse_list, const uint32_t *__restrict__ cs,
    const unsigned long long *__restrict__ occ, const unsigned long long *__restrict__ stmask,
    Walk walk, const uint32_t *__restrict__ skeys, uint32_t rbegin,
    const float4 *__restrict__ src, int mbits, float soft, const float *__restrict__ box_gm,
    float *__restrict__ ofx, float *__restrict__ ofy, float *__restrict__ ofz,
    float *__restrict__ opot, bool store, unsigned long long *__restrict__ inter) {
  const int lane = threadIdx.x & 31;
  const uint32_t ns = *nsparse_ptr;
  const int M = 1 << mbits;
  const float hc = 1.0f / (float)M;
  const float h2 = soft * soft, hinv = 1.f / soft, hinv3 = hinv * hinv * hinv;
  const f32x2 H2 = f2_pack(h2, h2);
  for (;;) {
    uint32_t ch = 0;
    if (lane == 0) ch = atomicAdd(work, 1u);
    ch = __shfl_sync(0xffffffffu, ch, 0);
    if ((size_t)ch * 32 >= ns) break;
    const uint32_t r = ch * 32 + (uint32_t)lane;
    const bool act = r < ns;
    uint32_t nsrc = 0;
    if (act) {
      const uint32_t i = sparse_list[r];
      const uint32_t key = skeys[i - rbegin];
      const float4 si = src[i];
      const uint32_t p = key & 63u, blk = key >> 6;
      const float GM = __ldg(box_gm + (key >> (3 * mbits)));
      int px, py, pz;
      inblock((int)p, px, py, pz);
      float nx = 0.f, ny = 0.f, nz = 0.f, np = 0.f;
      f32x2 pax = 0ull, pay = 0ull, paz = 0ull, pap = 0ull;
      const unsigned long long *sm = stmask + p * 27;
#pragma unroll 1
      for (int o = 0; o < 27; o++) {
        const unsigned long long m = __ldg(sm + o);
        if (!m) continue;
        const uint32_t nb = walk.add(blk, o);
        unsigned long long word = __ldg(occ + nb) & m;
        const int dX = 4 * (o / 9 - 1) - px, dY = 4 * ((o / 3) % 3 - 1) - py,
                  dZ = 4 * (o % 3 - 1) - pz;
        while (word) {
          const int c = __ffsll((long long)word) - 1;
          word &= word - 1;
          const uint32_t ck = (nb << 6) | (uint32_t)c;
          const uint32_t j0 = __ldg(cs + ck), j1 = __ldg(cs + ck + 1);
          nsrc += j1 - j0;
          int bx, by, bz;
          inblock(c, bx, by, bz);
          // the sink relative to the source cell's centre
          const float xs = si.x - (float)(dX + bx) * hc, ys = si.y - (float)(dY + by) * hc,
                      zs = si.z - (float)(dZ + bz) * hc;
          uint32_t j = j0;
          if constexpr (KERNEL == CT2G_SOFT_PLUMMER) {
            const f32x2 X = f2_pack(xs, xs), Y = f2_pack(ys, ys), Z = f2_pack(zs, zs);
            for (; j + 1 < j1; j += 2) {
              const float4 a = __ldg(src + j), b = __ldg(src + j + 1);
              const f32x2 dx = f2_sub(X, f2_pack(a.x, b.x));
              const f32x2 dy = f2_sub(Y, f2_pack(a.y, b.y));
              const f32x2 dz = f2_sub(Z, f2_pack(a.z, b.z));
              const f32x2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, H2)));
              float r0, r1;
              f2_unpack(r2, r0, r1);
              const f32x2 ri = f2_pack(rsqrtf(r0), rsqrtf(r1));
              const f32x2 g = f2_mul(f2_mul(ri, ri), ri);
              pax = f2_fma(dx, g, pax);
              pay = f2_fma(dy, g, pay);
              paz = f2_fma(dz, g, paz);
              if (POT) pap = f2_sub(pap, ri);
            }
          }
          for (; j < j1; j++) {
            const float4 q = __ldg(src + j);
            ct2g_pair_term<KERNEL, POT>(xs - q.x, ys - q.y, zs - q.z, h2, hinv, hinv3, nx, ny,
                                        nz, np, true);
          }
        }
      }
      if constexpr (KERNEL == CT2G_SOFT_PLUMMER) {
        float a0, a1;
        f2_unpack(pax, a0, a1);
        nx -= a0 + a1;
        f2_unpack(pay, a0, a1);
        ny -= a0 + a1;
        f2_unpack(paz, a0, a1);
        nz -= a0 + a1;
        if (POT) {
          f2_unpack(pap, a0, a1);
          np += a0 + a1;
        }
      }
      // added to the far field already in the force buffers, or stored (the
      // product rounded on its own, as in write_sink)
      const float gx = __fmul_rn(GM, nx), gy = __fmul_rn(GM, ny), gz = __fmul_rn(GM, nz);
      if (store) {
        ofx[i] = gx;
        ofy[i] = gy;
        ofz[i] = gz;
        if (POT) opot[i] = __fmul_rn(GM, np);
      } else {
        ofx[i] += gx;
        ofy[i] += gy;
        ofz[i] += gz;
        if (POT) opot[i] += __fmul_rn(GM, np);
      }
    }
    unsigned long long c = nsrc;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0 && c && inter) atomicAdd(inter, c);
  }
}

template <int K, bool POT>
int launch_near_lanes(ct2g_ctx *ctx, const Walk &walk, cudaStream_t st, float *fx, float *fy,
                      float *fz, float *pot, bool store) {
  auto k = near_lane_kernel<K, POT>;
  int per_sm = 0;
  CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
  const size_t nr = ctx->n - ctx->rung_begin;
  if (ctx->near_blocks_per_sm > 0) per_sm = std::min(per_sm, ctx->near_blocks_per_sm);
  size_t blocks = (size_t)std::max(1, per_sm) * ctx->num_sms;
  blocks = std::max<size_t>(1, std::min(blocks, (nr + 255) / 256));
  uint32_t *c = ctx->d_counts;
  k<<<(unsigned)blocks, 256, 0, st>>>(
      c + 1, c + 11, ctx->sparse_list, ctx->cell_start, ctx->occ, ctx->stmask, walk, ctx->keys,
      (uint32_t)ctx->rung_begin, ctx->src, ctx->mbits, ctx->opt.hsoft, ctx->box_gm, fx, fy, fz,
      pot, store, ctx->d_inter);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

Walk make_walk(int mbits) {
  Walk w{0u, 0u, 0u};
  for (int i = 0; i < mbits - 2; i++) {
    w.mx |= 1u << (3 * i + 2);
    w.my |= 1u << (3 * i + 1);
    w.mz |= 1u << (3 * i);
  }
  return w;
}

NearArgs near_args(ct2g_ctx *ctx, const unsigned long long *stm, int lo2, int hi2, float *fx,
                   float *fy, float *fz, float *pot, bool store) {
  NearArgs A{};
  A.cs = ctx->cell_start;
  A.occ = ctx->occ;
  A.stm = stm;
  A.walk = make_walk(ctx->mbits);
  A.skeys = ctx->keys;
  A.rbegin = (uint32_t)ctx->rung_begin;
  A.src = ctx->src;
  A.mbits = ctx->mbits;
  A.soft = ctx->opt.hsoft;
  A.lo2 = lo2;
  A.hi2 = hi2;
  A.box_gm = ctx->box_gm;
  A.ofx = fx;
  A.ofy = fy;
  A.ofz = fz;
  A.opot = pot;
  A.store = store;
  A.heavy = ctx->keys2;  // binning scratch: as many entries as particles, free by now
  A.heavy_min = heavy_min(ctx->M);
  A.warps = (uint32_t)ctx->num_sms * 32u;
  return A;
}

// Persistent grids: the resident blocks of every SM (or the tuned count), no
// more than one block per sink of the range.  (One block per 256 sinks, the earlier
// limit, left a sparse set's 4096 chunks of 8 sinks on 128 blocks: 49 us
// at 32^3 particles on a 64^3 mesh.)
unsigned near_grid(const ct2g_ctx *ctx, int per_sm, const NearArgs &A) {
  const size_t nr = ctx->n - ctx->rung_begin;
  if (ctx->near_blocks_per_sm > 0) per_sm = std::min(per_sm, ctx->near_blocks_per_sm);
  size_t blocks = std::min((size_t)std::max(1, per_sm) * ctx->num_sms, nr);
  // capped groups: enough blocks for every chunk the range can have (one per
  // sink at most, times the warps that share it); blocks past the device-held
  // chunk count exit at once
  if (A.maxch) {
    const size_t groups = std::max(nr, std::min(8 * nr, (size_t)A.warps));
    blocks = (groups + 8 * (size_t)A.maxch - 1) / (8 * (size_t)A.maxch);
  }
  return (unsigned)std::max<size_t>(1, blocks);
}

// the sparse chunks of A, then the dense and the heavy ones
template <int K, bool POT>
int launch_stream(ct2g_ctx *ctx, const NearArgs &A, cudaStream_t st) {
  int per_sm = 0;
  if (A.nsparse) {
    auto k = near_sparse_kernel<K, POT>;
    CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
    k<<<near_grid(ctx, per_sm, A), 256, 0, st>>>(A);
    CT2G_LAUNCHED(ctx);
  }
  auto k = near_coop_kernel<K, POT>;
  CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
  k<<<near_grid(ctx, per_sm, A), 256, 0, st>>>(A);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

template <int K, bool POT>
int launch_cells(ct2g_ctx *ctx, const NearArgs &A, cudaStream_t st) {
  int per_sm = 0;
  auto k = near_cells_kernel<K, POT>;
  CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
  k<<<near_grid(ctx, per_sm, A), 256, 0, st>>>(A);
  CT2G_LAUNCHED(ctx);
  return CT2G_OK;
}

// the dense chunks (counts[0]) and the sparse sinks: streamed with them as the
// per-block chunks (counts[2]; sparse_path 2), the
// same chunks cell by cell (sparse_path 1), or one sink per lane (sparse_path
// 0, counts[1] of them); work counters counts[8..11]
template <int K, bool POT>
int launch_near(ct2g_ctx *ctx, cudaStream_t st, float *fx, float *fy, float *fz, float *pot,
                bool store) {
  uint32_t *c = ctx->d_counts;
  NearArgs A = near_args(ctx, ctx->stmask, -1, ct2g_radius2(ctx->opt.bwidth), fx, fy, fz, pot, store);
  A.dchunks = ctx->chunks;
  A.schunks = ctx->schunks;
  A.ndense = c;
  A.slist = ctx->sparse_list;
  A.work = c + 8;
  // capped warps only beside the mesh solve (overlap), where they let the
  // mesh kernels' blocks in
  A.maxch = store ? (uint32_t)ctx->near_chunks_per_warp : 0u;
  A.inter = ctx->d_inter;
  const bool stream = ctx->sparse_path == 2;
  if (stream) A.nsparse = c + 2;
  CT2G_TRY((launch_stream<K, POT>(ctx, A, st)));
  if (stream) return CT2G_OK;
  if (ctx->sparse_path == 0)
    return launch_near_lanes<K, POT>(ctx, A.walk, st, fx, fy, fz, pot, store);
  A.nsparse = c + 2;
  A.work = c + 11;
  return launch_cells<K, POT>(ctx, A, st);
}

int near_all(ct2g_ctx *ctx, bool pot, cudaStream_t st, float *fx, float *fy, float *fz,
             float *po, bool store) {
  if (ctx->opt.kernel == CT2G_SOFT_SPHERE)
    return pot ? launch_near<CT2G_SOFT_SPHERE, true>(ctx, st, fx, fy, fz, po, store)
               : launch_near<CT2G_SOFT_SPHERE, false>(ctx, st, fx, fy, fz, po, store);
  return pot ? launch_near<CT2G_SOFT_PLUMMER, true>(ctx, st, fx, fy, fz, po, store)
             : launch_near<CT2G_SOFT_PLUMMER, false>(ctx, st, fx, fy, fz, po, store);
}

// far field + near field, added in that order: f = far + GM * near
__global__ void combine_kernel(size_t b, size_t n, float *__restrict__ fx, float *__restrict__ fy,
                               float *__restrict__ fz, const float *__restrict__ nfx,
                               const float *__restrict__ nfy, const float *__restrict__ nfz,
                               float *__restrict__ po, const float *__restrict__ npo) {
  for (size_t i = b + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    fx[i] += nfx[i];
    fy[i] += nfy[i];
    fz[i] += nfz[i];
    if (po) po[i] += npo[i];
  }
}

}  // namespace

// The widened sums of selected cells: dense-style chunks (<= 32 consecutive
// sinks of one cell, *nd at dch) over the stencil masks stm, and sparse-style
// ones (*ns at sch, their sinks in slist) over the cells lo2 < |o|^2 <= hi2,
// added into the given force buffers; work: four zeroed counters
int ct2g_near_window(ct2g_ctx *ctx, const uint2 *dch, const uint32_t *nd, const uint2 *sch,
                     const uint32_t *ns, const uint32_t *slist, uint32_t *work,
                     const unsigned long long *stm, int lo2, int hi2, bool pot, float *fx,
                     float *fy, float *fz, float *po) {
  NearArgs A = near_args(ctx, stm, lo2, hi2, fx, fy, fz, po, false);
  A.dchunks = dch;
  A.ndense = nd;
  A.schunks = sch;
  A.slist = slist;
  A.work = work;
  const bool stream = ctx->sparse_path == 2, plummer = ctx->opt.kernel != CT2G_SOFT_SPHERE;
  if (stream) A.nsparse = ns;
  if (plummer)
    CT2G_TRY((pot ? launch_stream<CT2G_SOFT_PLUMMER, true>(ctx, A, ctx->stream)
                  : launch_stream<CT2G_SOFT_PLUMMER, false>(ctx, A, ctx->stream)));
  else
    CT2G_TRY((pot ? launch_stream<CT2G_SOFT_SPHERE, true>(ctx, A, ctx->stream)
                  : launch_stream<CT2G_SOFT_SPHERE, false>(ctx, A, ctx->stream)));
  if (stream) return CT2G_OK;
  A.nsparse = ns;
  A.work = work + 3;
  if (plummer)
    return pot ? launch_cells<CT2G_SOFT_PLUMMER, true>(ctx, A, ctx->stream)
               : launch_cells<CT2G_SOFT_PLUMMER, false>(ctx, A, ctx->stream);
  return pot ? launch_cells<CT2G_SOFT_SPHERE, true>(ctx, A, ctx->stream)
             : launch_cells<CT2G_SOFT_SPHERE, false>(ctx, A, ctx->stream);
}

int ct2g_forces(ct2g_ctx *ctx, bool pot) {
  // the far-field pass (the inverse z pass with L2P) has written the range's entries
  CT2G_CUDA(ctx, cudaMemsetAsync(ctx->d_inter, 0, sizeof(unsigned long long), ctx->stream));
  CT2G_CUDA(ctx, cudaMemsetAsync(ctx->d_counts + 8, 0, 4 * sizeof(uint32_t), ctx->stream));
  if (ctx->n == ctx->rung_begin) return CT2G_OK;
  CT2G_TRY(near_all(ctx, pot, ctx->stream, ctx->fx, ctx->fy, ctx->fz, ctx->pot, false));
  return ct2g_learned_apply(ctx, pot);
}

// Far field and near field of the current range.  Serial (ctx->overlap 0):
// the mesh solve writes the far field, then the near field adds to it.
// Overlapped: the near field forks onto stream2 as soon as binning is done
// and stores into its own buffers while the mesh solve runs on the context
// stream (the near kernels are issue-bound, the mesh passes bound by memory
// latency, so the two fill each other's idle cycles); the context stream then
// joins it and adds the two, in the serial order (far + GM near), so both
// forms give the same forces bit for bit.
int ct2g_all_forces(ct2g_ctx *ctx, bool pot) {
  if (!ctx->overlap || ctx->n == ctx->rung_begin) {
    CT2G_TRY(ct2g_far_field(ctx, pot));
    return ct2g_forces(ctx, pot);
  }
  cudaStream_t st = ctx->stream;
  CT2G_CUDA(ctx, cudaMemsetAsync(ctx->d_inter, 0, sizeof(unsigned long long), st));
  CT2G_CUDA(ctx, cudaMemsetAsync(ctx->d_counts + 8, 0, 4 * sizeof(uint32_t), st));
  CT2G_CUDA(ctx, cudaEventRecord(ctx->ev_fork, st));
  CT2G_CUDA(ctx, cudaStreamWaitEvent(ctx->stream2, ctx->ev_fork, 0));
  CT2G_TRY(near_all(ctx, pot, ctx->stream2, ctx->nfx, ctx->nfy, ctx->nfz, ctx->npot, true));
  CT2G_CUDA(ctx, cudaEventRecord(ctx->ev_join, ctx->stream2));
  const int rc = ct2g_far_field(ctx, pot);
  // join before any return, so that stream2 never outlives a recording
  CT2G_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_join, 0));
  CT2G_TRY(rc);
  const size_t b = ctx->rung_begin, nr = ctx->n - b;
  combine_kernel<<<(unsigned)std::min<size_t>((nr + 255) / 256, (size_t)ctx->num_sms * 16), 256, 0,
                   st>>>(b, ctx->n, ctx->fx, ctx->fy, ctx->fz, ctx->nfx, ctx->nfy, ctx->nfz,
                         pot ? ctx->pot : nullptr, ctx->npot);
  CT2G_LAUNCHED(ctx);
  return ct2g_learned_apply(ctx, pot);
}

