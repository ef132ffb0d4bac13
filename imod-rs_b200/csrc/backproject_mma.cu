// backproject_mma.cu -- weighted back-projection of FP32-staged, R-weighted series on the
// 5th-generation tensor cores (tcgen05).
//
// Semantics: apps/tilt/src/main.rs:1002-1090 with sample_row_with_fill 386-406.  The
// sample position of a voxel does not depend on its slice, so one view's samples of
// a block of voxels and slices are a matrix product
//     sample[voxel][slice] = W[voxel][k] * row[k][slice]
// over the window of row elements the block projects onto.  W has two nonzeros per
// row, so it pays only if the window is short: a tile is a hexagon of 126 voxels in
// (x, z) (14 columns, 13 depths: hex_x0 / hex_len; hexagons tile the plane), which
// projects onto at most 16 elements at every tilt angle -- one K = 16 product of M =
// 128 voxels x N = 256 slices per term.  (An 8 x 16 rectangle needs up to 19, so two.)
//
// FP32 from FP16 operands: rows = hi + lo and weights = hi + lo in FP16 (22 significant
// bits), three products hi*lo + lo*hi + hi*hi; each block of 8 rows is staged times a power
// of two that keeps it in FP16's range (oct_exponent), undone on the sums.  The tensor cores
// truncate their FP32 sums, so they form the samples of two views only (their small
// terms first), and the sum over views is the consumer warps': tensor memory -> FP32
// register accumulators, round to nearest.  The result is as close to FP64 as the
// separately rounded f32 interpolation, but not bit for bit the reference's, so series
// without R-weighting, whose result is exactly reproducible, keep bp_fast_kernel (and so
// do the half staging forms, which round every sample: one tensor-memory round trip
// per view instead of per pair measured slower than their packed half arithmetic).
//
// Persistent CTAs (one per SM), warp-specialised, all roles walking the same tiles:
//   warps 0-7   consumers: tensor memory -> registers, epilogue.  128 accumulators
//               per thread: one voxel x 128 slices.
//   warps 8-11  weights: one voxel per thread, its rows of W per view to shared memory; and
//               the sum of the means of the views whose rows the voxel is outside of,
//               which the consumers add to its slices (it is the same in all of them)
//   warp 12     producer: one TMA box per view, the 16-element windows of the tile's
//               8-slice blocks in both planes (layout OCT: [plane][view][block of 8
//               slices][element][8]); any start element, since an element is 16 bytes
//               and the operand layout has no swizzle.  (One cp.async.bulk per block
//               and plane instead: 62 cycles each, 64 a view, measured 4x slower.)
//   warps 13-14 one thread each issues the tcgen05.mma's of every other view into its
//               tensor-memory buffer of 256 columns and commits
// A tile's epilogue overlaps the next tile's first views.  Blocks of 8 slices with values
// that are not finite, or rows far below their scale, take bp_oct_kernel, launched behind it.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>

#include "f32x2.cuh"
#include "pipe.cuh"
#include "tcgen05.cuh"
#include "tg_internal.h"

namespace tg {

namespace {

constexpr int NCONS = 8, NWGT = 4;          // consumer and weight warps
constexpr int NTHR = 16 * 32;               // four warpgroups (one warp idle)
// registers per thread after the split: 256*176 + 128*96 + 128*64 = 512*128 (compiled alone, the
// weight and issuing roles need at most 85 and 56)
constexpr int REG_CONS = 176, REG_WGT = 96, REG_PROD = 64;
constexpr int MAX_N = 256;                  // slices per tile
constexpr int BAND = 12;                    // tiles per band of the tile order
constexpr int HX = 14, HZ = 9, HROWS = 13;  // hexagon: period in x, in z, rows
constexpr int NVOX = 126;

// row r of the hexagon: columns [x0, x0 + len) about its centre
__device__ __forceinline__ int hex_x0(int r) {
  const int m = min(r, HROWS - 1 - r);  // distance from the nearer end: 0..6
  return m >= 4 ? -7 : m == 3 ? -5 : m == 2 ? -4 : m == 1 ? -3 : -1;
}
__device__ __forceinline__ int hex_len(int r) {
  const int m = min(r, HROWS - 1 - r);
  return m >= 4 ? 14 : m == 3 ? 11 : m == 2 ? 8 : m == 1 ? 6 : 3;
}
// voxel of row m of W: (column, depth) about the hexagon's centre
__device__ __forceinline__ int2 hex_voxel(int m) {
  int r = 0;
  while (r < HROWS - 1 && m >= hex_len(r)) m -= hex_len(r++);
  return make_int2(hex_x0(r) + m, r - 6);
}
// convex hull of the hexagon's voxels
__device__ constexpr signed char HULL[12][2] = {{-1, -6}, {1, -6}, {-3, -5}, {5, -3}, {-7, -2}, {6, -2},
                                                {-7, 2},  {6, 2},  {5, 3},   {-3, 5}, {-1, 6},  {1, 6}};

template <int KS> struct Cfg {
  static constexpr int KW = KS * 16;                 // staged window, elements
  static constexpr int A = 128 * KW * 2;             // one block of W
  static constexpr int B = (MAX_N / 8) * KW * 16;    // one plane's window
  static constexpr int VIEW = 2 * A + 2 * B;         // one view's W blocks and windows
  static constexpr int STAGE = 2 * VIEW;             // a ring stage is a pair of views
  static constexpr int TR = NCONS * 16 * 33 * 4;     // statistics transpose
  static constexpr int PART = MAX_N * 4 * 16;        // statistics of the four lane quarters
  static constexpr int FILL = 2 * 128 * 4;           // fill sums of the voxels of two tiles
  static constexpr int NST = KS == 1 ? 4 : 2;
  static constexpr int SMEM = NST * STAGE + TR + PART + FILL;
  static_assert(SMEM <= 226 * 1024 && SMEM > 114 * 1024, "one CTA per SM");
};

// Sample position in the reference's separately rounded order: monotone in dx and in dz,
// so a hull's vertices bound every voxel's position.
__device__ __forceinline__ float position(float dx, float dz, const float4 &g, float cx) {
  return __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(dx, g.x), g.w), __fmul_rn(__fmul_rn(dz, g.y), g.z)), cx);
}

struct Tile { int ox, oz, iy0, n, idx; };  // hexagon centre, first slice, slices, tile of its slice group
__device__ __forceinline__ Tile tile_at(const BpArgs &a, int t) {
  // bands of BAND tiles across, walked down in depth: the tiles in flight together
  // cover a compact region, whose windows overlap in L2
  const int ntxz = a.ntiles_xz, nbx = a.nbx, nbz = ntxz / nbx;
  const int grp = t / ntxz, t2 = t - grp * ntxz;
  const int band = t2 / (BAND * nbz), w = min(BAND, nbx - band * BAND), r = t2 - band * BAND * nbz;
  const int j = r / w, i = band * BAND + r - j * w;
  Tile q;
  q.ox = HX * i + ((j & 1) ? HX / 2 : 0);
  q.oz = HZ * j + 2;
  q.iy0 = grp * a.nper;
  q.n = min(a.nper, ((a.ny - q.iy0) + 15) & ~15);
  q.idx = i + j * nbx;
  return q;
}

// First element of each view's window over the hexagon; lane l of a warp computes
// view v0 + l, the warp reads them back by shuffle.
template <int KW>
__device__ __forceinline__ int window_start(const BpArgs &a, const Tile &q, int v) {
  const float4 g = __ldg(&a.vg[min(v, a.nviews - 1)]);
  const float dx0 = __fsub_rn((float)q.ox, a.ocx), dz0 = __fsub_rn((float)q.oz, a.cz);
  float mn = 3.0e38f, mx = -3.0e38f;
#pragma unroll
  for (int i = 0; i < 12; ++i) {
    const float x = position(dx0 + (float)HULL[i][0], dz0 + (float)HULL[i][1], g, a.cx);
    mn = fminf(mn, x);
    mx = fmaxf(mx, x);
  }
  const int k0 = (int)floorf(mn), last = (int)floorf(mx) + 1;  // a sample takes floor(x) and the next element
  if (last - k0 >= KW && v < a.nviews) atomicOr(a.err, 2);     // the host chooses KW so this never fires
  // voxels of the hexagon outside the volume may project outside the padded row;
  // those inside do not, so the shifted window still holds theirs
  return min(max(k0, -a.padL), a.PW - a.padL - KW);
}

__device__ __forceinline__ uint32_t half_pair(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ float half_val(uint32_t w, int i) {
  return __half2float(__ushort_as_half((uint16_t)(i ? w >> 16 : w & 0xffffu)));
}
// acc += a pair of views' samples of 32 slices
__device__ __forceinline__ void accumulate(float (&acc)[128], int c, const float (&r)[32]) {
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    const float2 s = up2(add2(pk2(acc[32 * c + i], acc[32 * c + i + 1]), pk2(r[i], r[i + 1])));
    acc[32 * c + i] = s.x;
    acc[32 * c + i + 1] = s.y;
  }
}

// The samples of a voxel in 8 slices, and apart from them its fills, summed over the views
// without the tensor cores, each row unscaled by its own exponent
__device__ __forceinline__ void sum_views(const BpArgs &a, float dx, float dz, int blk, float (&s8)[8], float &fill) {
#pragma unroll
  for (int j = 0; j < 8; ++j) s8[j] = 0.0f;
  fill = 0.0f;
  const size_t plane = (size_t)a.nviews * a.rows_alloc * a.PW;
  auto value = [](uint32_t hi, uint32_t lo, int i) {
    const float h = half_val(hi, i);
    return fabsf(h) <= 65504.0f ? h + half_val(lo, i) : h;
  };
#pragma unroll 2
  for (int v = 0; v < a.nviews; ++v) {
    const float x = position(dx, dz, __ldg(&a.vg[v]), a.cx);
    const float tt = __fadd_rd(x, MAGIC);
    const float f = __fsub_rn(x, __fsub_rn(tt, MAGIC));
    int k = (int)(__float_as_uint(tt) - MAGIC_BITS);
    const bool in = (uint32_t)k <= (uint32_t)(a.nx - 2);
    if (!in && k >= 0) ++k;
    if (!in && a.fill) fill = __fadd_rn(fill, __ldg(a.fill + v));
    const uint4 *e = reinterpret_cast<const uint4 *>(a.pairs) + ((size_t)v * a.rows_alloc + blk) * a.PW + (k + a.padL);
    const uint2 exps = __ldg(reinterpret_cast<const uint2 *>(a.exps) + (size_t)v * ((a.ny + 7) / 8) + blk);
    const uint4 u0 = __ldg(e), z0 = __ldg(e + plane), u1 = in ? __ldg(e + 1) : u0, z1 = in ? __ldg(e + 1 + plane) : z0;
    const uint32_t *p0 = &u0.x, *q0 = &z0.x, *p1 = &u1.x, *q1 = &z1.x;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float inv = pow2f(-(int)(signed char)((j < 4 ? exps.x : exps.y) >> (8 * (j & 3))));
      const float v0 = value(p0[j / 2], q0[j / 2], j & 1);
      s8[j] += inv * (in ? v0 * (1.0f - f) + value(p1[j / 2], q1[j / 2], j & 1) * f : v0);
    }
  }
}

template <int N> __device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
// Barrier of all consumer threads, and whether q held in any of them: every thread gets the
// same answer, whatever another role writes to the abort flag meanwhile.
__device__ __forceinline__ bool cons_any(bool q) {
  uint32_t r;
  __syncwarp();
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.or.pred p, 1, %2, q;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)q), "n"(NCONS * 32)
      : "memory");
  return r != 0;
}
// A wait of a whole warp: its lanes agree on the outcome, so that none leaves the loop
// while others go on to the warp-wide instructions behind the wait.
__device__ __forceinline__ bool warp_poll(uint32_t bar, uint32_t parity, volatile int *abort, uint64_t limit) {
  return __all_sync(0xffffffffu, poll_phase(bar, parity, abort, limit));
}

// A wait gave up: the series of this CTA's unfinished tiles report it.
template <class Job> __device__ __noinline__ void abandon(const Job &job, int t0, int ntiles) {
  for (; t0 < ntiles; t0 += gridDim.x) {
    int t = t0;
    atomicOr(job(t).err, 1);
  }
}

// The tiles blockIdx.x, + gridDim.x, ... of the launch's ntiles; job(t) gives a tile's
// series and rewrites t to the tile inside it.
template <int KS, class Job>
__device__ __forceinline__ void mma_body(const Job &job, int ntiles, unsigned char *sm) {
  using C = Cfg<KS>;
  constexpr int KW = C::KW, NST = C::NST;
  __shared__ __align__(8) uint64_t fullb[NST], full[NST], empty[NST], tfull[2], tempty[2], ffull[2], fempty[2], done[2];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ring = smem_u32(sm);
  float *fills = reinterpret_cast<float *>(sm + NST * C::STAGE + C::TR + C::PART);

  if (warp == 13) tmem_alloc(smem_u32(&s_tmem), 512);
  if (tid == 0) {
    for (int b = 0; b < NST; ++b) {
      mbar_init(smem_u32(&fullb[b]), 1);    // the windows
      mbar_init(smem_u32(&full[b]), NWGT);  // the weights, and (through the first weight warp) the windows
      mbar_init(smem_u32(&empty[b]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&tfull[b]), 1);
      mbar_init(smem_u32(&tempty[b]), NCONS);
      mbar_init(smem_u32(&ffull[b]), NWGT);
      mbar_init(smem_u32(&fempty[b]), NCONS);
    }
    for (int e = 0; e < 2; ++e) mbar_init(smem_u32(&done[e]), 1);
    fence_mbar_init();
    s_abort = 0;
  }
  tcgen05_before_sync();
  __syncthreads();
  tcgen05_after_sync();
  const uint32_t tm = s_tmem;

  if (warp < NCONS) {
    // ---------------- consumers ----------------
    reg_inc<REG_CONS>();
    const int2 vox = hex_voxel(min((warp & 3) * 32 + lane, NVOX - 1));
    const bool real = (warp & 3) * 32 + lane < NVOX;
    float *tr = reinterpret_cast<float *>(sm + NST * C::STAGE) + warp * (16 * 33);
    StatPartial *part = reinterpret_cast<StatPartial *>(sm + NST * C::STAGE + C::TR);
    int ph = 0;  // bit e: phase of tensor-memory buffer e
    int fb = 0, fph = 0;  // the tile's buffer of fill sums and its phase
    for (int t0 = blockIdx.x; t0 < ntiles; t0 += gridDim.x) {
      int t = t0;
      const BpArgs &a = job(t);
      const Tile q = tile_at(a, t);
      const int nviews = a.nviews, onx = a.onx, onz = a.onz;
      // this warp's columns: the first or second part of the tile's slices
      const int nh = ((q.n / 2) + 15) & ~15, c0 = warp < 4 ? 0 : nh, cnt = warp < 4 ? nh : q.n - nh;
      const int ox = q.ox + vox.x, oz = q.oz + vox.y;
      const bool ok = real && ox >= 0 && ox < onx && oz >= 0 && oz < onz;
      float acc[128];
#pragma unroll
      for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
      bool go = true;
      const uint64_t limit = a.wait_limit_ns;
      for (int i = 0; 2 * i < nviews; ++i) {
        const int e = i & 1;
        if (!(go = warp_poll(smem_u32(&tfull[e]), (ph >> e) & 1, &s_abort, limit))) break;
        tcgen05_after_sync();
        const uint32_t src = tm + ((uint32_t)(warp & 3) << 21) + e * 256 + c0;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (32 * c < cnt) {
            float r[32];
            tmem_ld32(src + 32 * c, r);
            if (32 * (c + 1) >= cnt) {  // all read: the buffer is free
              tcgen05_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&tempty[e]));
            }
            accumulate(acc, c, r);
          }
        if (cnt == 0 && lane == 0) mbar_arrive(smem_u32(&tempty[e]));
        ph ^= 1 << e;
      }
      go = go && warp_poll(smem_u32(&ffull[fb]), fph, &s_abort, limit);
      const float fill = fills[fb * 128 + (warp & 3) * 32 + lane];
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&fempty[fb]));
      fph ^= fb;
      fb ^= 1;
      if (!go) s_abort = 1;
      // all consumer warps store this tile, or none does: the barriers of the epilogue expect
      // them all.  (Behind this one, the previous tile's statistics have been read.)
      if (cons_any(!go || s_abort)) {
        s_abort = 1;
        if (lane == 0) abandon(job, t0, ntiles);
        break;
      }
      // ---------------- epilogue ----------------
      const size_t sl = (size_t)onz * onx;
      const float inv_n = a.inv_n;
      const int iy = q.iy0 + c0, ny = min(cnt, a.ny - iy);  // slices of this warp inside the volume
      // its blocks of 8 slices that bp_oct_kernel stores
      const int blk = min(iy / 8 + lane, (a.ny - 1) / 8);
      const unsigned skip = __ballot_sync(0xffffffffu, 8 * lane < ny && __ldg(a.flags + blk));
      {  // undo the blocks' staging scales (powers of two)
        const float inv = pow2f(-oct_exponent(__uint_as_float(__ldg(a.range + blk)), a.gain));
#pragma unroll
        for (int b = 0; b < 16; ++b) {
          const float u = __shfl_sync(0xffffffffu, inv, b);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[8 * b + j] = fmaf(acc[8 * b + j], u, fill);
        }
      }
      float *out = a.vol + ((size_t)iy * onz + oz) * onx + ox;
      const int mode = a.mode;
      if (mode == 2) {  // SIRT update vol += relax * v: 8 old values loaded together before their stores
        const float relax = a.relax;
#pragma unroll
        for (int j0 = 0; j0 < 128; j0 += 8) {
          if (j0 >= ny) break;
          const bool put = ok && !((skip >> (j0 / 8)) & 1);
          float old[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) old[j] = (put && j0 + j < ny) ? out[(size_t)j * sl] : 0.0f;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (put && j0 + j < ny)
              out[(size_t)j * sl] = __fadd_rn(old[j], __fmul_rn(relax, __fmul_rn(acc[j0 + j], inv_n)));
          out += 8 * sl;
        }
      } else if (mode == 1) {
#pragma unroll
        for (int j = 0; j < 128; ++j) {
          if (ok && j < ny && !((skip >> (j / 8)) & 1)) *out = __fmul_rn(acc[j], inv_n);
          out += sl;
        }
      } else {
        const float dw = a.dw, os = a.os, oa = a.oa;
        const unsigned okm = __ballot_sync(0xffffffffu, ok);
#pragma unroll
        for (int j0 = 0; j0 < 128; j0 += 16) {
          if (j0 >= cnt) break;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float y = __fadd_rn(__fmul_rn(__fmul_rn(__fmul_rn(acc[j0 + j], inv_n), dw), os), oa);
            if (ok && j0 + j < ny && !((skip >> ((j0 + j) / 8)) & 1)) *out = y;
            out += sl;
            tr[j * 33 + lane] = y;
          }
          // statistics: two lanes fold one slice of this warp's 32 voxels (a transpose through
          // shared memory; shuffling every slice would cost ten times the exchanges)
          __syncwarp();
          float mn = 3.40282347e+38f, mx = -3.40282347e+38f;
          double sum = 0.0;
          const int sj = lane & 15, i0 = lane & 16;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float y = tr[sj * 33 + i0 + i];
            if ((okm >> (i0 + i)) & 1) {
              mn = fminf(mn, y);
              mx = fmaxf(mx, y);
              sum += (double)y;
            }
          }
          mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, 16));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
          sum += __shfl_xor_sync(0xffffffffu, sum, 16);
          if (lane < 16) {
            StatPartial p;
            p.mn = mn;
            p.mx = mx;
            p.sum = sum;
            part[(c0 + j0 + lane) * 4 + (warp & 3)] = p;
          }
          __syncwarp();
        }
        cons_any(false);
        if (tid < q.n && q.iy0 + tid < a.ny && !__ldg(a.flags + (q.iy0 + tid) / 8)) {
          StatPartial p = part[tid * 4];
#pragma unroll
          for (int w = 1; w < 4; ++w) {
            const StatPartial o = part[tid * 4 + w];
            p.mn = fminf(p.mn, o.mn);
            p.mx = fmaxf(p.mx, o.mx);
            p.sum += o.sum;
          }
          a.partial[(size_t)(q.iy0 + tid) * a.ntiles_xz + q.idx] = p;
        }
      }
    }
  } else if (warp < NCONS + NWGT) {
    // ---------------- weights ----------------
    reg_dec<REG_WGT>();
    const int row = tid - NCONS * 32;
    const int2 vox = hex_voxel(min(row, NVOX - 1));
    int b = 0, ph = 1, fb = 0, fph = 1;
    for (int t0 = blockIdx.x; t0 < ntiles && !__any_sync(0xffffffffu, s_abort); t0 += gridDim.x) {
      int t = t0;
      const BpArgs &a = job(t);
      const Tile q = tile_at(a, t);
      const int nviews = a.nviews, nx2 = a.nx - 2;
      const int ox = q.ox + vox.x, oz = q.oz + vox.y;
      const bool ok = row < NVOX && ox >= 0 && ox < a.onx && oz >= 0 && oz < a.onz;
      const float dx = __fsub_rn((float)ox, a.ocx), dz = __fsub_rn((float)oz, a.cz), cx = a.cx;
      const float4 *vg = a.vg;
      const float *means = a.fill;
      float fill = 0.0f;
      const uint64_t limit = a.wait_limit_ns;
      int k0s = 0;
      // a voxel's row of W in view v: p the words at element pair kw and the next in the
      // first block, r in the second
      struct Row { uint32_t p0, p1, r0, r1; int kw; };
      auto row_of = [&](const float4 &g, int k0, int v) -> Row {
        const float x = position(dx, dz, g, cx);
        const float tt = __fadd_rd(x, MAGIC);  // MAGIC + floor(x), exactly
        const float f = __fsub_rn(x, __fsub_rn(tt, MAGIC));
        int k = (int)(__float_as_uint(tt) - MAGIC_BITS);
        // the weights of elements k and k + 1: leading halves, remainders
        const float omf = __fsub_rn(1.0f, f);
        uint32_t w0 = half_pair(omf, f);
        uint32_t w1 = half_pair(__fsub_rn(omf, half_val(w0, 0)), __fsub_rn(f, half_val(w0, 1)));
        if ((uint32_t)k > (uint32_t)nx2) {
          // outside the row: the fill alone, which the padding holds in edge mode (element nx - 1
          // is the last sample, so the right side takes the element after)
          if (means && v < nviews) fill = __fadd_rn(fill, __ldg(means + v));
          w0 = half_pair(1.0f, 0.0f);
          w1 = 0u;
          k += k >= 0 ? 1 : 0;
        }
        const int rel = k - k0;
        const bool odd = rel & 1;
        if (!ok) w0 = w1 = 0u;
        return Row{odd ? w0 << 16 : w0, odd ? w0 >> 16 : 0u, odd ? w1 << 16 : w1, odd ? w1 >> 16 : 0u, rel >> 1};
      };
      auto store_row = [&](const Row &w, uint32_t dst) {
#pragma unroll
        for (int c = 0; c < 2 * KS; ++c) {  // chunks of 8 elements, [chunk][row][8]
          uint32_t u[4], z[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int i = 4 * c + j;
            u[j] = w.kw == i ? w.p0 : w.kw == i - 1 ? w.p1 : 0u;
            z[j] = w.kw == i ? w.r0 : w.kw == i - 1 ? w.r1 : 0u;
          }
          sts128(dst + c * 2048, u[0], u[1], u[2], u[3]);
          sts128(dst + C::A + c * 2048, z[0], z[1], z[2], z[3]);
        }
      };
      float4 g0 = __ldg(vg), g1 = __ldg(vg + min(1, nviews - 1));
      bool go = true;
      for (int v = 0; v < nviews; v += 2) {
        if ((v & 31) == 0) k0s = window_start<KW>(a, q, v + lane);
        const int ka = __shfl_sync(0xffffffffu, k0s, v & 31), kb = __shfl_sync(0xffffffffu, k0s, (v + 1) & 31);
        const Row wa = row_of(g0, ka, v), wb = row_of(g1, kb, v + 1);
        g0 = __ldg(vg + min(v + 2, nviews - 1));
        g1 = __ldg(vg + min(v + 3, nviews - 1));
        const bool two = v + 1 < nviews;
        if (!(go = warp_poll(smem_u32(&empty[b]), ph, &s_abort, limit))) break;
        const uint32_t dst = ring + b * C::STAGE + row * 16;
        store_row(wa, dst);
        if (two) store_row(wb, dst + C::VIEW);
        fence_proxy_async();
        // the first weight warp also waits for the windows, so that the issuing threads wait once
        if (warp == NCONS && !(go = warp_poll(smem_u32(&fullb[b]), ph ^ 1, &s_abort, limit))) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&full[b]));
        if (++b == NST) { b = 0; ph ^= 1; }
      }
      if (go && (go = warp_poll(smem_u32(&fempty[fb]), fph, &s_abort, limit))) {
        fills[fb * 128 + row] = fill;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ffull[fb]));
        fph ^= fb;
        fb ^= 1;
      }
      if (!go) {
        s_abort = 1;
        break;
      }
    }
  } else {
    reg_dec<REG_PROD>();
    if (warp == 12) {
      // ---------------- producer ----------------
      int b = 0, ph = 1, issued = 0, skipped = -1;
      uint64_t limit = 0;
      const void *acquired = nullptr;
      for (int t0 = blockIdx.x; t0 < ntiles && !__any_sync(0xffffffffu, s_abort); t0 += gridDim.x) {
        int t = t0;
        const BpArgs &a = job(t);
        const Tile q = tile_at(a, t);
        const int nviews = a.nviews, padL = a.padL, skip = a.fault_skip_stage;
        const uint32_t bytes = (uint32_t)(2 * (a.nper / 8) * KW * 16);
        const void *map = job.map(a);
        if (Job::MAP_IN_MEMORY && map != acquired) {
          if (lane == 0) tensormap_acquire(map);
          acquired = map;
        }
        const int ra = a.rows_alloc;
        int y = q.iy0 / 8;
        limit = a.wait_limit_ns;
        int k0s = 0;
        bool go = true;
        for (int v = 0; v < nviews; v += 2) {
          if ((v & 31) == 0) k0s = window_start<KW>(a, q, v + lane);
          const int ka = __shfl_sync(0xffffffffu, k0s, v & 31), kb = __shfl_sync(0xffffffffu, k0s, (v + 1) & 31);
          const bool two = v + 1 < nviews;
          if (!(go = warp_poll(smem_u32(&empty[b]), ph, &s_abort, limit))) break;
          if (v / 2 == skip) {  // test hook: no copy, fullb[b] never completes
            skipped = issued++;
          } else {
            if (lane == 0) {
              const uint32_t dst = ring + b * C::STAGE + 2 * C::A, bar = smem_u32(&fullb[b]);
              mbar_expect_tx(bar, two ? 2 * bytes : bytes);
              tma_box3(dst, map, (ka + padL) * 8, y, 0, bar);
              if (two) tma_box3(dst + C::VIEW, map, (kb + padL) * 8, y + ra, 0, bar);
            }
            ++issued;
          }
          y += 2 * ra;
          if (++b == NST) { b = 0; ph ^= 1; }
        }
        if (!go) {
          s_abort = 1;
          break;
        }
      }
      if (lane == 0)  // no copy may land after the CTA exits (another role may give up any time)
        for (int g = max(0, issued - NST); g < issued; ++g)
          if (g != skipped) poll_phase(smem_u32(&fullb[g % NST]), (g / NST) & 1, nullptr, limit);
    } else if (warp <= 14 && lane == 0) {
      // ---------------- tensor cores: one thread per tensor-memory buffer issues alternate
      // pairs of views ----------------
      const int e = warp - 13;
      int b0 = 0, ph0 = 0, tph = 1;  // stage of the tile's first pair; phase of tempty[e]
      uint64_t limit = 0;
      bool go = true;
      auto advance = [](int &st, int &p, int n) {
        st += n;
        while (st >= NST) { st -= NST; p ^= 1; }
      };
      for (int t0 = blockIdx.x; t0 < ntiles && go && !s_abort; t0 += gridDim.x) {
        int t = t0;
        const BpArgs &a = job(t);
        const Tile q = tile_at(a, t);
        const int nviews = a.nviews, npairs = (nviews + 1) / 2;
        limit = a.wait_limit_ns;
        const uint32_t idesc = mma_idesc_f16(128, q.n, /*b_mn_major=*/true);
        const uint32_t plane = (uint32_t)(a.nper / 8) * (KW * 16), d = tm + e * 256;
        int b = b0, ph = ph0;
        advance(b, ph, e);
        for (int i = e; i < npairs; i += 2) {
          const bool two = 2 * i + 1 < nviews;
          if (!poll_phase(smem_u32(&full[b]), ph, &s_abort, limit) ||
              !poll_phase(smem_u32(&tempty[e]), tph, &s_abort, limit)) {
            go = false;
            break;
          }
          tcgen05_after_sync();
          // W: [chunk of 8 elements][row][8]; rows: [slice block][element][8 slices]
          auto product = [&](int view, int wblk, int rblk, bool acc) {
            const uint32_t A = ring + b * C::STAGE + view * C::VIEW + wblk * C::A;
            const uint32_t B = ring + b * C::STAGE + view * C::VIEW + 2 * C::A + rblk * plane;
            const uint64_t da = smem_desc(A, 2048, 128), db = smem_desc(B, 128, KW * 16);
#pragma unroll
            for (int k = 0; k < KS; ++k)
              mma_f16_ss(d, da + k * (4096 >> 4), db + k * (256 >> 4), idesc, acc || k > 0);
          };
          // the small terms of both views first: every product truncates its sum, and these
          // truncate sums that are 2^-11 of a sample
          product(0, 0, 1, false);
          product(0, 1, 0, true);
          if (two) {
            product(1, 0, 1, true);
            product(1, 1, 0, true);
          }
          product(0, 0, 0, true);
          if (two) product(1, 0, 0, true);
          mma_commit(smem_u32(&empty[b]));
          mma_commit(smem_u32(&tfull[e]));
          tph ^= 1;
          advance(b, ph, 2);
        }
        advance(b0, ph0, npairs);
      }
      if (!go) s_abort = 1;
      mma_commit(smem_u32(&done[e]));  // nothing in flight at exit
      poll_phase(smem_u32(&done[e]), 0, nullptr, limit);
    }
  }
  __syncwarp();
  tcgen05_before_sync();
  __syncthreads();
  if (warp == 13) {
    tcgen05_after_sync();
    tmem_dealloc(tm, 512);
  }
}

struct OneJob {  // a launch over one series, its map a kernel parameter
  static constexpr bool MAP_IN_MEMORY = false;
  const BpArgs &a;
  const TensorMap &m;
  __device__ __forceinline__ const BpArgs &operator()(int &) const { return a; }
  __device__ __forceinline__ const void *map(const BpArgs &) const { return &m; }
};
struct ManyJobs {  // tile t belongs to the series j with jobs[j].tile0 <= t < jobs[j+1].tile0
  static constexpr bool MAP_IN_MEMORY = true;
  const BpArgs *jobs;
  int n;
  __device__ __forceinline__ const BpArgs &operator()(int &t) const {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(&jobs[mid].tile0) <= t) lo = mid;
      else hi = mid - 1;
    }
    t -= __ldg(&jobs[lo].tile0);
    return jobs[lo];
  }
  __device__ __forceinline__ const void *map(const BpArgs &a) const { return a.tmap; }
};

template <int KS>
__global__ void __launch_bounds__(NTHR, 1) bp_mma_kernel(const __grid_constant__ BpArgs a, const __grid_constant__ TensorMap map,
                                                         int ntiles) {
  extern __shared__ __align__(128) unsigned char sm[];
  mma_body<KS>(OneJob{a, map}, ntiles, sm);
}
template <int KS>
__global__ void __launch_bounds__(NTHR, 1) bp_mma_batch_kernel(const BpArgs *__restrict__ jobs, int njobs, int ntiles) {
  extern __shared__ __align__(128) unsigned char sm[];
  mma_body<KS>(ManyJobs{jobs, njobs}, ntiles, sm);
}

// The blocks of 8 slices that the tensor-core kernel leaves out: those with rows of a scale of
// their own, and with a value that is not finite, which a product with the zeros of W spreads
// to the voxels of its slice that do not sample it.  The same tiles, one voxel per thread, sample
// by sample.  A kernel of its own, so that the tensor-core kernel's warps
// never wait for such a tile and the rest of a series keeps its speed; with no such block a
// CTA reads one word and ends.
constexpr int OCT_T = 128;
__device__ __forceinline__ void oct_blocks(const BpArgs &a, int ntiles_xz) {
  const int nblk = (a.ny + 7) / 8;
  if (!a.flags[nblk]) return;
  __shared__ StatPartial part[OCT_T / 32][8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int2 vox = hex_voxel(min(tid, NVOX - 1));
  int first = blockIdx.x;  // this CTA's first tile of the next flagged block
  for (int b0 = 0; b0 < nblk; b0 += 32) {
    unsigned todo = __ballot_sync(0xffffffffu, b0 + lane < nblk && a.flags[min(b0 + lane, nblk - 1)]);
    for (; todo; todo &= todo - 1) {
      const int blk = b0 + __ffs(todo) - 1, iy = 8 * blk;
      int t = first;
      for (; t < ntiles_xz; t += gridDim.x) {
        const Tile q = tile_at(a, t);
        const int ox = q.ox + vox.x, oz = q.oz + vox.y;
        const bool ok = tid < NVOX && ox >= 0 && ox < a.onx && oz >= 0 && oz < a.onz;
        const float dx = __fsub_rn((float)min(max(ox, 0), a.onx - 1), a.ocx);
        const float dz = __fsub_rn((float)min(max(oz, 0), a.onz - 1), a.cz);
        float s8[8], fill;
        sum_views(a, dx, dz, blk, s8, fill);
        float *out = a.vol + ((size_t)iy * a.onz + oz) * a.onx + ox;
        const size_t sl = (size_t)a.onz * a.onx;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const bool put = ok && iy + j < a.ny;
          float y = __fmul_rn(__fadd_rn(s8[j], fill), a.inv_n);
          if (a.mode == 2 && put) y = __fadd_rn(out[j * sl], __fmul_rn(a.relax, y));
          if (a.mode == 0) {
            y = __fadd_rn(__fmul_rn(__fmul_rn(y, a.dw), a.os), a.oa);
            float mn = put ? fminf(3.40282347e+38f, y) : 3.40282347e+38f, mx = put ? fmaxf(-3.40282347e+38f, y) : -3.40282347e+38f;
            double sum = put ? (double)y : 0.0;
            for (int o = 16; o > 0; o >>= 1) {
              mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
              mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
              sum += __shfl_xor_sync(0xffffffffu, sum, o);
            }
            if (lane == 0) {
              part[warp][j].mn = mn;
              part[warp][j].mx = mx;
              part[warp][j].sum = sum;
            }
          }
          if (put) out[j * sl] = y;
        }
        if (a.mode == 0) {
          __syncthreads();
          if (tid < 8 && iy + tid < a.ny) {
            StatPartial p = part[0][tid];
            for (int w = 1; w < OCT_T / 32; ++w) {
              p.mn = fminf(p.mn, part[w][tid].mn);
              p.mx = fmaxf(p.mx, part[w][tid].mx);
              p.sum += part[w][tid].sum;
            }
            a.partial[(size_t)(iy + tid) * ntiles_xz + q.idx] = p;
          }
          __syncthreads();
        }
      }
      first = t - ntiles_xz;  // blocks follow each other in one tile sequence over the CTAs
    }
  }
}
__global__ void __launch_bounds__(OCT_T) bp_oct_kernel(const __grid_constant__ BpArgs a) { oct_blocks(a, a.ntiles_xz); }
__global__ void __launch_bounds__(OCT_T) bp_oct_batch_kernel(const BpArgs *__restrict__ jobs, int njobs) {
  for (int j = 0; j < njobs; ++j) oct_blocks(jobs[j], jobs[j].ntiles_xz);
}

int sm_count() {
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}
int grid_for(int ntiles) { return std::max(1, std::min(ntiles, sm_count())); }
int oct_grid(int ntiles) { return std::max(1, std::min(ntiles, 8 * sm_count())); }
template <class K> int set_smem(K kern, int smem) {
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  return e == cudaSuccess ? TG_OK : cuda_fail(e, "cudaFuncSetAttribute(bp_mma)");
}
template <int KS> int launch_t(const BpArgs &a, const TensorMap &map, int ntiles, cudaStream_t st) {
  const int rc = set_smem(bp_mma_kernel<KS>, Cfg<KS>::SMEM);
  if (rc != TG_OK) return rc;
  bp_mma_kernel<KS><<<grid_for(ntiles), NTHR, Cfg<KS>::SMEM, st>>>(a, map, ntiles);
  bp_oct_kernel<<<oct_grid(ntiles), OCT_T, 0, st>>>(a);
  return TG_OK;
}
template <int KS> int launch_batch_t(const BatchLaunch &bl, cudaStream_t st) {
  const int rc = set_smem(bp_mma_batch_kernel<KS>, Cfg<KS>::SMEM);
  if (rc != TG_OK) return rc;
  bp_mma_batch_kernel<KS><<<grid_for(bl.ntiles), NTHR, Cfg<KS>::SMEM, st>>>(bl.jobs, bl.njobs, bl.ntiles);
  bp_oct_batch_kernel<<<oct_grid(bl.ntiles), OCT_T, 0, st>>>(bl.jobs, bl.njobs);
  return TG_OK;
}

}  // namespace

// K steps of 16 elements that a hexagon's window needs, from the view's position slopes:
// its width w spans at most floor(w) + 1 elements, and each sample takes one more (16 up
// to w = 14; every view without z-factor has w <= 13.61).  w <= 30 with |sin * zf| <= 2.
int bp_mma_steps(const std::vector<float4> &vg) {
  static const int hull[6][2] = {{1, 6}, {-1, 6}, {5, 3}, {-3, 5}, {6, 2}, {-7, 2}};
  double width = 0.0;
  for (const float4 &g : vg) {
    const double c = (double)g.x * g.w, s = (double)g.y * g.z;
    double mn = 0.0, mx = 0.0;
    for (const auto &p : hull)
      for (int m = -1; m <= 1; m += 2) {  // the hull is symmetric in z
        const double x = p[0] * c + m * p[1] * s;
        mn = std::min(mn, x);
        mx = std::max(mx, x);
      }
    width = std::max(width, mx - mn);
  }
  return width <= 13.9 ? 1 : 2;
}

// Tile grid of one series: hexagons per slice group, slices per tile balanced over the groups.
long long bp_mma_plan(BpArgs &a) {
  a.nbx = (a.onx - 1 + 7) / HX + 1;
  a.ntiles_xz = bp_mma_ntiles(a.onx, a.onz);
  const int groups = (a.ny + MAX_N - 1) / MAX_N;
  a.nper = (((a.ny + groups - 1) / groups) + 15) & ~15;
  return (long long)a.ntiles_xz * ((a.ny + a.nper - 1) / a.nper);
}

// The TMA map of an OCT buffer: boxes of one view's KS*16-element windows of nper/8 blocks in
// both planes.
int bp_mma_tensor_map(void *pairs, int nviews, int rows_alloc, int PW, int nper, int steps, TensorMap *out) {
  static_assert(sizeof(CUtensorMap) == sizeof(TensorMap) && alignof(CUtensorMap) <= alignof(TensorMap), "tensor map");
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                              const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? reinterpret_cast<Encode>(fn) : nullptr;
  }();
  if (!encode) { set_error("no cuTensorMapEncodeTiled in the driver"); return TG_ERR_CUDA; }
  const cuuint64_t dims[3] = {(cuuint64_t)PW * 8, (cuuint64_t)rows_alloc * nviews, 2};
  const cuuint64_t strides[2] = {(cuuint64_t)PW * 16, (cuuint64_t)PW * 16 * rows_alloc * nviews};
  const cuuint32_t box[3] = {(cuuint32_t)(steps * 128), (cuuint32_t)(nper / 8), 2}, one[3] = {1, 1, 1};
  CUtensorMap m;
  const CUresult e = encode(&m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, pairs, dims, strides, box, one,
                                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (e != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed"); return TG_ERR_CUDA; }
  memcpy(out->bytes, &m, sizeof m);
  return TG_OK;
}

// Whether the tensor-core kernel is the faster one.  A tile takes its views' round trips
// through tensor memory however few its slices (about 560 + n/2 cycles a view, 8000 + 85 n
// a tile, measured at 1.85 GHz on 61 views: 23 us a wave of tiles with 16 slices, 40 us with
// 256), so it needs slices to spread them over and enough tiles for every SM; the fast
// kernel does 3.0e12 to 4.1e12 updates/s whatever the shape.  512 x 200, 61 views: 128 slices
// 0.179 against 0.250 ms, 96 slices 0.172 against 0.192, 64 slices 0.159 against 0.131.
bool bp_mma_pays(int onx, int onz, int ny, int nviews) {
  BpArgs a{};
  a.onx = onx;
  a.onz = onz;
  a.ny = ny;
  const double waves = (double)((bp_mma_plan(a) + 147) / 148);
  const double tile = nviews * (560.0 + 0.5 * a.nper) + 8000.0 + 85.0 * a.nper;
  return waves * tile / 1.85e9 < (double)onx * onz * ny * nviews / 3.6e12;
}

int bp_mma_ntiles(int onx, int onz) { return ((onx - 1 + 7) / HX + 1) * ((onz - 1 + 4) / HZ + 1); }

int launch_bp_mma(const BpArgs &a0, const TensorMap &map, int steps, cudaStream_t st, int *ntiles) {
  BpArgs a = a0;
  const long long n = bp_mma_plan(a);
  if (n >= (1ll << 31) - (1ll << 20)) { set_error("too many tiles"); return TG_ERR_UNSUPPORTED; }
  if (ntiles) *ntiles = a.ntiles_xz;
  return steps == 1 ? launch_t<1>(a, map, (int)n, st) : launch_t<2>(a, map, (int)n, st);
}

int launch_bp_mma_batch(const BatchLaunch &bl, int steps, cudaStream_t st) {
  return steps == 1 ? launch_batch_t<1>(bl, st) : launch_batch_t<2>(bl, st);
}

}  // namespace tg
