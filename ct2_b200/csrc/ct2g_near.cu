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
// issued instruction.  A warp's source batch is staged as pair records --
// (x0, x1, y0, y1) in one 16-byte slot and (z0, z1) after them -- so one
// broadcast load of each feeds two interactions.
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
// Streamed near field.  A chunk is <= 32 sinks, one per lane: sinks of one
// cell (dense), or the sparse cells' sinks of one 4x4x4 block (sparse).  Its
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
// and one shuffle gives its (first particle - first position).  The source's
// offset from the chunk's frame (the sink cell's centre; the block's first cell
// for a sparse chunk) is the difference of the fixed-point positions,
// periodic by itself, rounded once to FP32 and negated, so that the inner loop adds.
//
// What bounds it: 11 packed FP32 instructions and two MUFU operations per two
// interactions (22 and 16 cycles of their pipes per warp and SM sub-partition), so
// 11.6 interactions per clock and SM, 3.4e12 per second, when nothing else
// is issued.  A packed instruction takes two issue slots, so what else a pair
// needs (two shared loads, two MUFU, its share of the staging) counts against
// it: FMA pipe 71%, all issue slots used.  Against one warp per chunk, cells'
// sources in batches of their own halves of blocks (dense), a table of stencil entries
// per lane in shared memory (sparse) and scalar arithmetic (sphere kernel):
// 2.5 M particles in halos 35.2 -> 34.4 ms, 128^3 in Plummer spheres 3.52 ->
// 3.23, 300 k with the sphere kernel and potentials 10.2 -> 7.0 ms, 400 k
// in 48 halos 10.0 -> 6.7 ms.
// ---------------------------------------------------------------------------
struct NearArgs {
  const uint2 *dchunks;     // dense chunks (first particle, sinks), *ndense of them
  const uint32_t *ndense;
  const uint2 *schunks;     // sparse chunks (first sparse_list entry, sinks),
  const uint32_t *soff;     // starting at schunks[*soff] (null: 0), *nsparse of
  const uint32_t *nsparse;  // them (null: none)
  const uint32_t *slist;
  const uint32_t *cs;
  const unsigned long long *occ, *stm;
  Walk walk;
  const uint32_t *skeys;
  uint32_t rbegin;
  const uint32_t *x, *y, *z;
  const float4 *src;        // offsets from the own cell's centre
  int mbits;
  float soft;
  int lo2, hi2;             // sparse: source cells with lo2 < |o|^2 <= hi2 of a lane's own
  const float *box_gm;
  float *ofx, *ofy, *ofz, *opot;
  bool store;               // store into the buffers instead of adding to them
  uint32_t *work;           // [0] chunks taken, [1] heavy chunks, [2] heavy ones taken
  uint32_t *heavy;          // list of the heavy chunks
  uint32_t warps;           // warps the launch may spread few chunks over
  uint32_t maxch;
  unsigned long long *inter;
};

// A chunk whose 27 neighbouring blocks hold more sources than this is left to
// a second launch in which the eight warps of a block share each chunk: one warp
// on its own walks 1000 sources in about 10 us, and clustered sets have
// chunks of 10^5 (2.5 ms on a single warp while the rest of the GPU idled, at
// 400 k particles in 48 halos), while splitting repeats the window walk
// in every warp (about 1000 instructions each, 5% of the work at this size).
constexpr uint32_t kHeavySources = 16384;
constexpr int kStage = 256;  // floats of staging per warp: two batches of pair records
// a coordinate that makes r^2 infinite: an empty slot of the last batch adds 0
constexpr float kFar = 3e19f;

// two interactions of a sink at (X, Y, Z) (both halves equal) with the sources of
// pair record pr (negated coordinates); accumulates d g and 1/r (the caller negates)
template <int KERNEL, bool POT, bool MASKED>
__device__ __forceinline__ void pair_term(const float *sb, int pr, uint32_t bits, f32x2 X, f32x2 Y,
                                          f32x2 Z, f32x2 H2, float h2, float hinv, float hinv3,
                                          f32x2 &ax, f32x2 &ay, f32x2 &az, f32x2 &ap) {
  const float4 a = reinterpret_cast<const float4 *>(sb)[pr];  // x0 x1 y0 y1
  float z0, z1;
  bool on0 = true, on1 = true;
  if (MASKED) {
    const float4 b = reinterpret_cast<const float4 *>(sb + 64)[pr];  // z0 z1 and the cells' bits
    z0 = b.x;
    z1 = b.y;
    on0 = (__float_as_uint(b.z) & bits) != 0u;
    on1 = (__float_as_uint(b.w) & bits) != 0u;
  } else {
    const float2 b = reinterpret_cast<const float2 *>(sb + 64)[pr];
    z0 = b.x;
    z1 = b.y;
  }
  const f32x2 dx = f2_add(X, f2_pack(a.x, a.y));
  const f32x2 dy = f2_add(Y, f2_pack(a.z, a.w));
  const f32x2 dz = f2_add(Z, f2_pack(z0, z1));
  f32x2 g, pp;
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
  ax = f2_fma(dx, g, ax);
  ay = f2_fma(dy, g, ay);
  az = f2_fma(dz, g, az);
  if (POT) ap = f2_add(ap, pp);
}

// the barrier of the S warps (a power of two) that share a chunk
__device__ __forceinline__ void group_sync(int S, int group) {
  if (S > 1) asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(32 * S) : "memory");
}

// One chunk, its windows' sums added in window order.  S warps may share it:
// warp s takes the windows s, s + S, ..., and warp 0 adds each round's S
// sums in order, so the result does not depend on S.  HEAVY: the eight warps take
// every eighth batch of each window instead, and warp 0 adds their eight sums.
// stage: this warp's kStage floats (the group's warps' lie one after
// another).  Without HEAVY a heavy chunk is left alone (false returned).
template <int KERNEL, bool POT, bool SPARSE, bool HEAVY>
__device__ __forceinline__ bool near_chunk(const NearArgs &A, const uint2 cd, int s, int S,
                                           int group, float *stage, int lane) {
  const int sh = 32 - A.mbits;
  const bool act = (uint32_t)lane < cd.y;
  const uint32_t slot = cd.x + (act ? (uint32_t)lane : 0u);
  const uint32_t i = SPARSE ? A.slist[slot] : slot;
  const uint32_t key = A.skeys[i - A.rbegin];
  const uint32_t p = key & 63u, blk = key >> 6;  // blk is the same for the whole chunk
  // in-block positions present in the chunk
  unsigned long long pm = 1ull << p;
  if (SPARSE)
    pm = ((unsigned long long)__reduce_or_sync(0xffffffffu, (uint32_t)(pm >> 32)) << 32) |
         __reduce_or_sync(0xffffffffu, (uint32_t)pm);
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
  if (!HEAVY) {
    const uint32_t w = word ? A.cs[(size_t)(nblk + 1) << 6] - A.cs[(size_t)nblk << 6] : 0u;
    if (__reduce_add_sync(0xffffffffu, w) > kHeavySources) return false;
  }
  // the frame's origin and this lane's sink in it
  const uint32_t fk = (SPARSE ? key & ~63u : key) & ((1u << (3 * A.mbits)) - 1u);
  const uint32_t half = 1u << (sh - 1);
  const uint32_t ox = (ct2g_compact3(fk >> 2) << sh) + half,
                 oy = (ct2g_compact3(fk >> 1) << sh) + half, oz = (ct2g_compact3(fk) << sh) + half;
  const float sc = (float)CT2G_TWO_M32;
  const float sx = (float)(int32_t)(A.x[i] - ox) * sc, sy = (float)(int32_t)(A.y[i] - oy) * sc,
              sz = (float)(int32_t)(A.z[i] - oz) * sc;
  const f32x2 X = f2_pack(sx, sx), Y = f2_pack(sy, sy), Z = f2_pack(sz, sz);
  const float h2 = A.soft * A.soft, hinv = 1.f / A.soft, hinv3 = hinv * hinv * hinv;
  const f32x2 H2 = f2_pack(h2, h2);
  f32x2 ax = 0ull, ay = 0ull, az = 0ull, ap = 0ull;
  float nx = 0.f, ny = 0.f, nz = 0.f, np = 0.f;
  uint32_t nsrc = 0;
  // the packed sums so far, and back to zero
  auto take = [&]() {
    float a0, a1;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    f2_unpack(ax, a0, a1);
    v.x = a0 + a1;
    f2_unpack(ay, a0, a1);
    v.y = a0 + a1;
    f2_unpack(az, a0, a1);
    v.z = a0 + a1;
    if (POT) {
      f2_unpack(ap, a0, a1);
      v.w = a0 + a1;
    }
    ax = ay = az = ap = 0ull;
    return v;
  };
  auto add = [&](const float4 &v) {
    nx += v.x;
    ny += v.y;
    nz += v.z;
    if (POT) np += v.w;
  };
  // the first nw warps' sums into warp 0's totals, in order
  auto share = [&](int nw) {
    const float4 v = take();
    __syncwarp();  // every lane is done with this warp's staging
    if (s > 0) reinterpret_cast<float4 *>(stage)[lane] = v;
    group_sync(S, group);
    if (s == 0) {
      add(v);
      for (int k = 1; k < nw; k++)
        add(reinterpret_cast<const float4 *>(stage + k * kStage)[lane]);
    }
    group_sync(S, group);
  };
  // candidate cells before each neighbouring block's, and in all
  const uint32_t c1 = (uint32_t)__popcll(word);
  uint32_t in1 = c1;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, in1, d);
    if (lane >= d) in1 += t;
  }
  const uint32_t ex1 = in1 - c1, C = __shfl_sync(0xffffffffu, in1, 31);
  const int rec = 4 * (lane >> 1) + (lane & 1);
  const int recz = 64 + (SPARSE ? rec : 2 * (lane >> 1) + (lane & 1));
  const uint32_t bs = HEAVY ? (uint32_t)s : 0u, bS = HEAVY ? 8u : 1u;  // this warp's batches
  for (uint32_t r0 = 0; r0 < C; r0 += HEAVY ? 32u : 32u * (uint32_t)S) {
    const uint32_t w0 = HEAVY ? r0 : r0 + 32u * (uint32_t)s;
    if (w0 < C) {
      const bool valid = w0 + (uint32_t)lane < C;
      // window cell of this lane: the (g - ex1[o])-th candidate cell of block o
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
      const uint32_t excl = incl - c, total = __shfl_sync(0xffffffffu, incl, 31);
      uint32_t bits = 0xffffffffu;
      if (SPARSE) {
        bits = 0u;
        int bx, by, bz;
        inblock(q, bx, by, bz);
        const int cx = 4 * (o / 9 - 1) + bx, cy = 4 * ((o / 3) % 3 - 1) + by, cz = 4 * (o % 3 - 1) + bz;
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
      // source b0 + lane of the stream (its cell's bit in t)
      const uint32_t base = jb - excl;
      uint32_t px = 0, py = 0, pz = 0, t = 0;
      auto fetch = [&](uint32_t b0) {
        const uint32_t g1 = min(b0 + (uint32_t)lane, total - 1);
        const uint32_t before = __ballot_sync(0xffffffffu, valid && excl < b0);
        const uint32_t rel = excl - b0;
        const uint32_t heads = __reduce_or_sync(0xffffffffu, valid && rel < 32u ? 1u << rel : 0u);
        t = __popc(before) + __popc(heads & (0xffffffffu >> (31u - (g1 - b0)))) - 1;
        const uint32_t j = __shfl_sync(0xffffffffu, base, (int)t) + g1;
        px = __ldg(A.x + j);
        py = __ldg(A.y + j);
        pz = __ldg(A.z + j);
      };
      uint32_t b0 = 32u * bs;
      int flip = 0;
      if (b0 < total) fetch(b0);
      __syncwarp();  // the previous window's last batch is read
      for (; b0 < total; b0 += 32u * bS) {
        float *sb = stage + flip;
        flip ^= kStage / 2;
        const bool on = b0 + (uint32_t)lane < total;
        sb[rec] = on ? (float)(int32_t)(ox - px) * sc : kFar;
        sb[rec + 2] = (float)(int32_t)(oy - py) * sc;
        sb[recz] = (float)(int32_t)(oz - pz) * sc;
        if (SPARSE) sb[recz + 2] = __uint_as_float(on ? 1u << t : 0u);
        __syncwarp();
        const uint32_t n = total - b0;
        if (b0 + 32u * bS < total) fetch(b0 + 32u * bS);
        if (n >= 32) {
#pragma unroll 8
          for (int pr = 0; pr < 16; pr++)
            pair_term<KERNEL, POT, SPARSE>(sb, pr, bits, X, Y, Z, H2, h2, hinv, hinv3, ax, ay, az,
                                           ap);
        } else {
          const int np = (int)(n + 1) >> 1;
#pragma unroll 2
          for (int pr = 0; pr < np; pr++)
            pair_term<KERNEL, POT, SPARSE>(sb, pr, bits, X, Y, Z, H2, h2, hinv, hinv3, ax, ay, az,
                                           ap);
        }
      }
    }
    if (!HEAVY) {
      if (S == 1)
        add(take());
      else
        share((int)min((uint32_t)S, (C - r0 + 31u) / 32u));
    }
  }
  if (HEAVY) share(8);
  if (A.inter && (!HEAVY || s == 0)) {
    unsigned long long c;
    if (SPARSE)
      c = __reduce_add_sync(0xffffffffu, act ? nsrc : 0u);
    else
      c = (unsigned long long)nsrc * cd.y;
    if (lane == 0 && c) atomicAdd(A.inter, c);
  }
  if (s > 0) return true;
  // added to the far field (L2P, with GM) already in the force buffers, or
  // stored into the near-field buffers when the two run side by side; the
  // product is rounded on its own (no fused multiply-add into the far
  // field), so that both forms add the same two values
  if (act) {
    const float GM = __ldg(A.box_gm + (key >> (3 * A.mbits)));
    const float gx = __fmul_rn(GM, -nx), gy = __fmul_rn(GM, -ny), gz = __fmul_rn(GM, -nz);
    if (A.store) {
      A.ofx[i] = gx;
      A.ofy[i] = gy;
      A.ofz[i] = gz;
      if (POT) A.opot[i] = __fmul_rn(GM, -np);
    } else {
      A.ofx[i] += gx;
      A.ofy[i] += gy;
      A.ofz[i] += gz;
      if (POT) A.opot[i] += __fmul_rn(GM, -np);
    }
  }
  return true;
}

// The dense chunks and after them the sparse ones, taken from a device
// counter by groups of S warps; blocks are persistent.  S = 1 wherever the chunks
// alone fill the warps the GPU holds (A.warps); fewer chunks are shared by
// 2, 4 or 8 warps each (12^3 particles on a 16^3 mesh are 64 chunks: 48 us
// with one warp each on 7 blocks).  HEAVY: the second launch, eight warps on
// each chunk that the first one listed.  The sums depend neither on S nor on the
// launch shape, and the heavy rule only on a chunk's neighbourhood.
template <int KERNEL, bool POT, bool HEAVY>
__global__ void __launch_bounds__(256, 4) near_stream_kernel(const NearArgs A) {
  __shared__ __align__(16) float stage[8 * kStage];
  __shared__ uint32_t taken_s[2][8];  // by the parity of the turn: one barrier a turn
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t nd = *A.ndense, ns = A.nsparse ? *A.nsparse : 0u;
  const uint2 *sch = A.soff ? A.schunks + *A.soff : A.schunks;
  const uint32_t nch = HEAVY ? A.work[1] : nd + ns;
  int S = 8;
  if (!HEAVY)
    while (S > 1 && (size_t)nch * S > A.warps) S >>= 1;
  const int s = wib & (S - 1), group = wib / S;
  // maxch > 0: a group takes at most maxch chunks and the block then exits,
  // so that blocks of kernels on other streams get the SM in between
  for (uint32_t taken = 0; HEAVY || A.maxch == 0 || taken < A.maxch; taken++) {
    uint32_t ch = 0;
    if (S > 1) {
      if (s == 0 && lane == 0) taken_s[taken & 1][group] = atomicAdd(A.work + (HEAVY ? 2 : 0), 1u);
      group_sync(S, group);
      ch = taken_s[taken & 1][group];
    } else {
      if (lane == 0) ch = atomicAdd(A.work, 1u);
      ch = __shfl_sync(0xffffffffu, ch, 0);
    }
    if (ch >= nch) break;
    if (HEAVY) ch = A.heavy[ch];
    float *st = stage + wib * kStage;
    const bool done =
        ch < nd
            ? near_chunk<KERNEL, POT, false, HEAVY>(A, A.dchunks[ch], s, S, group, st, lane)
            : near_chunk<KERNEL, POT, true, HEAVY>(A, sch[ch - nd], s, S, group, st, lane);
    if (!done && s == 0 && lane == 0) A.heavy[atomicAdd(A.work + 1, 1u)] = ch;
  }
}

// Sparse chunks cell by cell (tuning sparse_path 1, and meshes of 8, where a
// block-sized frame is not smaller than half the box): one warp per chunk; each
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
  if (act) {  // as near_chunk
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
  const uint2 *list = A.soff ? A.schunks + *A.soff : A.schunks;
  for (uint32_t taken = 0; A.maxch == 0 || taken < A.maxch; taken++) {
    uint32_t ch = 0;
    if (lane == 0) ch = atomicAdd(A.work, 1u);
    ch = __shfl_sync(0xffffffffu, ch, 0);
    if (ch >= nch) break;
    cells_chunk<KERNEL, POT>(A, list[ch], sbuf[wib], lane);
  }
}

// Sparse sinks, one per lane: the warp takes 32 consecutive entries of the
// sparse sink list (cell order, so the lanes are neighbours) and every lane
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
      // product rounded on its own, as in near_chunk)
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

NearArgs near_args(ct2g_ctx *ctx, const unsigned long long *stm, float lo2, float hi2, float *fx,
                   float *fy, float *fz, float *pot, bool store) {
  NearArgs A{};
  A.cs = ctx->cell_start;
  A.occ = ctx->occ;
  A.stm = stm;
  A.walk = make_walk(ctx->mbits);
  A.skeys = ctx->keys;
  A.rbegin = (uint32_t)ctx->rung_begin;
  A.x = ctx->x;
  A.y = ctx->y;
  A.z = ctx->z;
  A.src = ctx->src;
  A.mbits = ctx->mbits;
  A.soft = ctx->opt.hsoft;
  // integers d2 with lo2 < d2 <= hi2
  A.lo2 = (int)std::floor(lo2);
  A.hi2 = (int)std::floor(hi2);
  A.box_gm = ctx->box_gm;
  A.ofx = fx;
  A.ofy = fy;
  A.ofz = fz;
  A.opot = pot;
  A.store = store;
  A.heavy = ctx->keys2;  // binning scratch: as many entries as particles, free by now
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

// dense and sparse chunks of A, then the heavy ones among them
template <int K, bool POT>
int launch_stream(ct2g_ctx *ctx, const NearArgs &A, cudaStream_t st) {
  int per_sm = 0;
  auto k = near_stream_kernel<K, POT, false>;
  CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 256, 0));
  k<<<near_grid(ctx, per_sm, A), 256, 0, st>>>(A);
  CT2G_LAUNCHED(ctx);
  auto kh = near_stream_kernel<K, POT, true>;
  CT2G_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kh, 256, 0));
  const size_t nr = ctx->n - ctx->rung_begin;
  if (nr > kHeavySources) {  // fewer particles than a heavy chunk has sources: none
    kh<<<near_grid(ctx, per_sm, A), 256, 0, st>>>(A);
    CT2G_LAUNCHED(ctx);
  }
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

// the streamed sparse form works in a frame of up to 8 cells from its origin,
// which has to be less than half the box
bool stream_sparse(const ct2g_ctx *ctx) { return ctx->sparse_path == 2 && ctx->M >= 16; }

// the dense chunks (counts[0]) and the sparse sinks: streamed with them as the
// per-block chunks stored after the dense ones (counts[2]; sparse_path 2), the
// same chunks cell by cell (sparse_path 1), or one sink per lane (sparse_path
// 0, counts[1] of them); work counters counts[8..11]
template <int K, bool POT>
int launch_near(ct2g_ctx *ctx, cudaStream_t st, float *fx, float *fy, float *fz, float *pot,
                bool store) {
  uint32_t *c = ctx->d_counts;
  NearArgs A = near_args(ctx, ctx->stmask, -1.f, ctx->opt.bwidth * ctx->opt.bwidth, fx, fy, fz, pot,
                         store);
  A.dchunks = A.schunks = ctx->chunks;
  A.ndense = A.soff = c;
  A.slist = ctx->sparse_list;
  A.work = c + 8;
  // capped warps only beside the mesh solve (overlap), where they let the
  // mesh kernels' blocks in
  A.maxch = store ? (uint32_t)ctx->near_chunks_per_warp : 0u;
  A.inter = ctx->d_inter;
  const bool stream = stream_sparse(ctx);
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
                     const unsigned long long *stm, float lo2, float hi2, bool pot, float *fx,
                     float *fy, float *fz, float *po) {
  NearArgs A = near_args(ctx, stm, lo2, hi2, fx, fy, fz, po, false);
  A.dchunks = dch;
  A.ndense = nd;
  A.schunks = sch;
  A.slist = slist;
  A.work = work;
  const bool stream = stream_sparse(ctx), plummer = ctx->opt.kernel != CT2G_SOFT_SPHERE;
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

