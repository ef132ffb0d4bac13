// ctf.cu -- CTF phase flip of a tilt series on the GPU.
//
// Semantics: apps/ctfphaseflip/src/main.rs (the default CPU path) and, for the
// per-strip seam, GpuCtfSession::correct_strip with ctf_correct.wgsl
// (apps/ctfphaseflip/src/gpu.rs:107-262).
//
// Each view is cut into strips perpendicular to the tilt axis (main.rs:443-
// 470).  Per strip: the bounding box of its pixels is transformed by a 2D FFT,
// every frequency whose CTF -- computed in f64 as the reference's CPU path does
// -- is negative is negated, the transform is inverted, and the strip's pixels
// enter per-pixel weighted sums with the reference's triangular weights; the
// sum is divided by the weight (or the input kept where no strip weighs in).
// Strip geometry (centres, bounds, bounding boxes) depends on the image size
// and tilt axis only, so the host works it out once per stack with the
// reference's f64 expressions; the device repeats only the per-pixel membership
// test, in the same f64 operation order (no FMA contraction).
//
// A strip is small -- at most strip_width samples across the tilt axis, 16 with
// the automatic width of a 512-pixel view -- and a stack has thousands of them,
// so the work is batched: one launch per stage over every strip of a chunk of
// views (blockIdx.y is the strip of the chunk), four launches per chunk:
//   rows in     box rows -> FFT -> written transposed
//   columns     FFT, sign flip, inverse FFT in shared memory, transposed back
//   rows out    inverse FFT -> real part, scaled
//   combine     per pixel, the strips that hold it, in strip order
// Each CTA transforms several rows at once, so the transposed stores cover
// whole 32-byte sectors.  A chunk's strips stay in L2 (CTF_CHUNK_BYTES).  Copies
// and kernels share one stream: while a chunk's kernels run, the host only stages
// the next chunk's pageable views.
// 512x512x41 with 16-pixel strips (1312 strips), host to host: 88.7 ms with nine
// launches per strip (11,852 launches, bound by the launching thread and by
// grids of a few blocks), 18.0 ms batched, of which the copies from and to the
// caller's pageable memory take about 12 (about 13 in all with the output pages
// faulted in meanwhile, fault_ahead.h).
//
// Layout in device memory: the stack [nz][ny][nx] f32, corrected in place; two
// buffers of a chunk's strips (sw*sh float2 each); the strip and view tables;
// twiddle tables per transform length; the per-(view, tile) partial statistics
// of volume_ops.  A view whose strips exceed the chunk (wide boxes of a rotated
// tilt axis) is corrected in runs of strips with its weighted sums in memory.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <string>
#include <vector>

#include "fault_ahead.h"
#include "fft.cuh"
#include "tg_internal.h"

namespace tg {

namespace {

constexpr double PI32_D = (double)3.14159265358979323846f;  // `PI as f64` (f32 constant widened)
constexpr int CTF_MAX_N = 12288;                             // transform length: 2n float2 in shared memory
constexpr size_t CTF_CHUNK_BYTES = 32u << 20;                // both buffers of a chunk: a quarter of L2
constexpr size_t CTF_SMEM = 72 * 1024;                       // per CTA: 3 CTAs per SM
constexpr int CTF_ROWS = 16;                                 // most rows per CTA: 128-byte transposed segments

struct CtfPlan {  // one transform length
  FftPlanDev plan;
  const float2 *tw;  // exp(-2 pi i k / n)
};

struct CtfStrip {  // one strip, the same for all views
  double center, lo, hi, dx_a;
  size_t off;  // first sample of its box within a view's strips
  int x0, y0, sw, sh, plan_w, plan_h;
  float scale;
};

struct CtfView {
  double def1, def2, sin_tilt, astig_rad;
  int has_astig;
};

struct CtfArgs {
  float *stack;  // [nz][ny][nx]
  const CtfStrip *strips;
  const CtfView *views;
  const CtfPlan *plans;
  float2 *A, *B;
  size_t view_stride, base;  // samples between views of the chunk; `off` of its first strip
  int nx, ny, z0, s0, ns;    // the chunk: views from z0, strips s0 .. s0 + ns
  double pixel_a, wl, cs_a, amp, w_phase, cuton, plate, tilt_axis_rad, cos_ta, sin_ta;
};

// Row stride in shared memory: odd, so that a column of rows (the transposed
// store) touches different banks.
__host__ __device__ __forceinline__ int ctf_ld(int n) { return n | 1; }

template <int R, bool INV>
__device__ __forceinline__ void rows_pass(const float2 *X, float2 *Y, int n, int rows, int Ns, const float2 *tw) {
  const int nb = n / R, tstride = n / (Ns * R), ld = ctf_ld(n);
  for (int i = threadIdx.x; i < nb * rows; i += blockDim.x) {
    const int row = i / nb, j = i - row * nb, k = j % Ns;
    const float2 *x = X + row * ld;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = x[j + r * nb];
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        float2 w = __ldg(&tw[r * k * tstride]);
        if (INV) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
    }
    bfly<R, INV>(v, tw, n);
    float2 *y = Y + row * ld + (j - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) y[r * Ns] = v[r];
  }
}

// A prime radix above 7: each output sums its R inputs with table twiddles (for
// a prime length, the direct DFT), four rows per twiddle.
template <bool INV>
__device__ __forceinline__ void rows_pass_prime(const float2 *X, float2 *Y, int n, int R, int rows, int Ns,
                                                const float2 *tw) {
  const int nb = n / R, tstride = n / (Ns * R), ld = ctf_ld(n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int q = i / nb, j = i - q * nb, k = j % Ns;
    const int step = (k + q * Ns) * tstride;  // < n
    const int o = (j - k) * R + k + q * Ns;
    for (int r0 = 0; r0 < rows; r0 += 4) {
      const int m = min(4, rows - r0);
      float2 acc[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = make_float2(0.0f, 0.0f);
      int e = 0;  // (r * step) mod n
      for (int r = 0; r < R; ++r) {
        float2 w = __ldg(&tw[e]);
        if (INV) w.y = -w.y;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u < m) acc[u] = cadd(acc[u], cmul(X[(r0 + u) * ld + j + r * nb], w));
        e += step;
        if (e >= n) e -= n;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (u < m) Y[(r0 + u) * ld + o] = acc[u];
    }
  }
}

// Stockham over `rows` rows of length n at A (row stride ctf_ld(n)); B is the
// other buffer.  Returns the one that holds the result, after a barrier.
template <bool INV> __device__ float2 *rows_fft(float2 *A, float2 *B, const CtfPlan *p, int rows) {
  const int n = p->plan.n, nfac = p->plan.nfac;
  const float2 *tw = p->tw;
  int Ns = 1;
  for (int i = 0; i < nfac; ++i) {
    const int R = p->plan.fac[i];
    switch (R) {
      case 4: rows_pass<4, INV>(A, B, n, rows, Ns, tw); break;
      case 2: rows_pass<2, INV>(A, B, n, rows, Ns, tw); break;
      case 3: rows_pass<3, INV>(A, B, n, rows, Ns, tw); break;
      case 5: rows_pass<5, INV>(A, B, n, rows, Ns, tw); break;
      case 7: rows_pass<7, INV>(A, B, n, rows, Ns, tw); break;
      default: rows_pass_prime<INV>(A, B, n, R, rows, Ns, tw); break;
    }
    __syncthreads();
    float2 *t = A; A = B; B = t;
    Ns *= R;
  }
  return A;
}

// Box rows of a strip -> FFT -> B[fx][y] (transposed).
__global__ void __launch_bounds__(256) ctf_rows_in_kernel(CtfArgs a, int rpb) {
  extern __shared__ __align__(16) float2 csm[];
  const int v = blockIdx.y / a.ns;
  const CtfStrip &g = a.strips[a.s0 + blockIdx.y - v * a.ns];
  const int n = g.sw, sh = g.sh, ld = ctf_ld(n);
  const float *view = a.stack + (size_t)(a.z0 + v) * a.nx * a.ny;
  float2 *out = a.B + v * a.view_stride + (g.off - a.base);
  for (int r0 = blockIdx.x * rpb; r0 < sh; r0 += gridDim.x * rpb) {
    const int rows = min(rpb, sh - r0);
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int r = i / n, c = i - r * n;
      csm[r * ld + c] = make_float2(view[(size_t)(g.y0 + r0 + r) * a.nx + g.x0 + c], 0.0f);
    }
    __syncthreads();
    const float2 *R = rows_fft<false>(csm, csm + rpb * ld, a.plans + g.plan_w, rows);
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int c = i / rows, r = i - c * rows;
      out[(size_t)c * sh + r0 + r] = R[r * ld + c];
    }
    __syncthreads();  // both buffers are reused by the next rows
  }
}

// main.rs:553-617: true where the CTF (f64) at (fx, fy) is negative; never below
// the cut-on frequency.
__device__ __forceinline__ bool ctf_negative(const CtfArgs &f, int sw, int sh, int fx, int fy, double base1,
                                             double base2, int has_astig, double astig_rad) {
  const double freq_y = fy <= sh / 2 ? (double)fy : __dsub_rn((double)fy, (double)sh);
  const double freq_x = fx <= sw / 2 ? (double)fx : __dsub_rn((double)fx, (double)sw);
  double rfx = freq_x, rfy = freq_y;
  if (fabs(f.tilt_axis_rad) > 1e-6) {
    rfx = __dadd_rn(__dmul_rn(freq_x, f.cos_ta), __dmul_rn(freq_y, f.sin_ta));
    rfy = __dadd_rn(__dmul_rn(-freq_x, f.sin_ta), __dmul_rn(freq_y, f.cos_ta));
  }
  const double sx = __ddiv_rn(rfx, __dmul_rn((double)sw, f.pixel_a));
  const double sy = __ddiv_rn(rfy, __dmul_rn((double)sh, f.pixel_a));
  const double s2 = __dadd_rn(__dmul_rn(sx, sx), __dmul_rn(sy, sy));
  if (sqrt(s2) < f.cuton) return false;
  double def = base1;
  if (has_astig) {  // effective_defocus, main.rs:213-219
    const double da = __dsub_rn(atan2(sy, sx), astig_rad);
    const double c = cos(da), s = sin(da);
    def = __dadd_rn(__dmul_rn(base1, __dmul_rn(c, c)), __dmul_rn(base2, __dmul_rn(s, s)));
  }
  // chi = PI * lambda * s2 * (def - 0.5 * Cs * lambda^2 * s2), left to right
  const double t = __dmul_rn(__dmul_rn(__dmul_rn(__dmul_rn(0.5, f.cs_a), f.wl), f.wl), s2);
  const double chi = __dmul_rn(__dmul_rn(__dmul_rn(3.14159265358979323846, f.wl), s2), __dsub_rn(def, t));
  const double chi_t = __dadd_rn(chi, f.plate);
  return __dadd_rn(__dmul_rn(-sin(chi_t), f.w_phase), __dmul_rn(cos(chi_t), f.amp)) < 0.0;
}

// Columns fx of a strip's spectrum: FFT along y, flip, inverse FFT -> A[y][fx].
__global__ void __launch_bounds__(256) ctf_columns_kernel(CtfArgs a, int rpb) {
  extern __shared__ __align__(16) float2 csm[];
  const int v = blockIdx.y / a.ns;
  const CtfStrip &g = a.strips[a.s0 + blockIdx.y - v * a.ns];
  const CtfView &w = a.views[a.z0 + v];
  const int n = g.sh, sw = g.sw, ld = ctf_ld(n), has_astig = w.has_astig;
  const double slope = __dmul_rn(g.dx_a, w.sin_tilt), astig_rad = w.astig_rad;
  const double base1 = __dadd_rn(w.def1, slope), base2 = __dadd_rn(w.def2, slope);
  const size_t off = v * a.view_stride + (g.off - a.base);
  for (int c0 = blockIdx.x * rpb; c0 < sw; c0 += gridDim.x * rpb) {
    const int rows = min(rpb, sw - c0);
    const float2 *in = a.B + off + (size_t)c0 * n;
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int r = i / n, k = i - r * n;
      csm[r * ld + k] = in[i];
    }
    __syncthreads();
    float2 *R = rows_fft<false>(csm, csm + rpb * ld, a.plans + g.plan_h, rows);
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int r = i / n, k = i - r * n;
      if (ctf_negative(a, sw, n, c0 + r, k, base1, base2, has_astig, astig_rad)) {
        const float2 x = R[r * ld + k];
        R[r * ld + k] = make_float2(-x.x, -x.y);
      }
    }
    __syncthreads();
    R = rows_fft<true>(R, R == csm ? csm + rpb * ld : csm, a.plans + g.plan_h, rows);
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int y = i / rows, r = i - y * rows;
      a.A[off + (size_t)y * sw + c0 + r] = R[r * ld + y];
    }
    __syncthreads();
  }
}

// Rows of A -> inverse FFT -> real part times 1 / (sw * sh), into B's memory.
__global__ void __launch_bounds__(256) ctf_rows_out_kernel(CtfArgs a, int rpb) {
  extern __shared__ __align__(16) float2 csm[];
  const int v = blockIdx.y / a.ns;
  const CtfStrip &g = a.strips[a.s0 + blockIdx.y - v * a.ns];
  const int n = g.sw, sh = g.sh, ld = ctf_ld(n);
  const size_t off = v * a.view_stride + (g.off - a.base);
  const float scale = g.scale;
  for (int r0 = blockIdx.x * rpb; r0 < sh; r0 += gridDim.x * rpb) {
    const int rows = min(rpb, sh - r0);
    const float2 *in = a.A + off + (size_t)r0 * n;
    float *out = reinterpret_cast<float *>(a.B) + off + (size_t)r0 * n;
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int r = i / n, c = i - r * n;
      csm[r * ld + c] = in[i];
    }
    __syncthreads();
    const float2 *R = rows_fft<true>(csm, csm + rpb * ld, a.plans + g.plan_w, rows);
    for (int i = threadIdx.x; i < rows * n; i += blockDim.x) {
      const int r = i / n, c = i - r * n;
      out[i] = __fmul_rn(R[r * ld + c].x, scale);
    }
    __syncthreads();
  }
}

struct CombineArgs {
  double cxp, cyp, perp_x, perp_y, min_perp, width, half_w;
  float *wsum, *wtot;  // one view's sums where its strips take several chunks, else nullptr
  int first, last;     // the chunk holds the view's first / last strip
  int max_off;         // strips skipped for an empty box shift the index by at most this
};

// main.rs:654-680 per pixel: every strip of the chunk with d in [lo, hi) adds
// val*w and w, in strip order; then the division.  The strips tile the range of
// d up to the rounding of their bounds, so those next to the one that d falls in
// are looked at as well.
__global__ void __launch_bounds__(256) ctf_combine_kernel(CtfArgs a, CombineArgs q) {
  const unsigned npix = (unsigned)a.nx * a.ny, p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npix) return;
  const int v = blockIdx.y, y = (int)(p / a.nx), x = (int)(p - (unsigned)y * a.nx);
  const double d = __dadd_rn(__dmul_rn(__dsub_rn((double)x, q.cxp), q.perp_x),
                             __dmul_rn(__dsub_rn((double)y, q.cyp), q.perp_y));
  const int k = (int)floor((d - q.min_perp) / q.width);
  float ws = 0.0f, wt = 0.0f;
  if (q.wsum && !q.first) {
    ws = q.wsum[p];
    wt = q.wtot[p];
  }
  const float *val = reinterpret_cast<const float *>(a.B) + v * a.view_stride;
  const int s_lo = max(a.s0, k - 1 - q.max_off), s_hi = min(a.s0 + a.ns - 1, k + 1);
  for (int s = s_lo; s <= s_hi; ++s) {
    const CtfStrip &g = a.strips[s];
    if (!(d >= g.lo && d < g.hi)) continue;
    const float dist = (float)fabs(__ddiv_rn(__dsub_rn(d, g.center), q.half_w));
    const float w = fmaxf(__fsub_rn(1.0f, dist), 0.0f);
    ws = __fadd_rn(ws, __fmul_rn(val[g.off - a.base + (size_t)(y - g.y0) * g.sw + (x - g.x0)], w));
    wt = __fadd_rn(wt, w);
  }
  if (q.last) {
    if (wt > 1e-10f) a.stack[(size_t)(a.z0 + v) * npix + p] = __fdiv_rn(ws, wt);
  } else {
    q.wsum[p] = ws;
    q.wtot[p] = wt;
  }
}

// ctf_correct.wgsl in f32 (the shader's operation order; accurate sin/cos/atan2)
__global__ void ctf_strip_f32_kernel(float *re, float *im, tg_ctf_strip_params p) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)p.sw * p.sh) return;
  const uint32_t fx_idx = (uint32_t)(i % p.sw), fy_idx = (uint32_t)(i / p.sw);
  const float sw = (float)p.sw, sh = (float)p.sh;
  float freq_x = fx_idx <= p.sw / 2u ? (float)fx_idx : __fsub_rn((float)fx_idx, sw);
  float freq_y = fy_idx <= p.sh / 2u ? (float)fy_idx : __fsub_rn((float)fy_idx, sh);
  if (fabsf(p.tilt_axis_rad) > 1e-6f) {
    const float ca = cosf(p.tilt_axis_rad), sa = sinf(p.tilt_axis_rad);
    const float rx = __fadd_rn(__fmul_rn(freq_x, ca), __fmul_rn(freq_y, sa));
    const float ry = __fadd_rn(__fmul_rn(-freq_x, sa), __fmul_rn(freq_y, ca));
    freq_x = rx;
    freq_y = ry;
  }
  const float sx = __fdiv_rn(freq_x, __fmul_rn(sw, p.pixel_a));
  const float sy = __fdiv_rn(freq_y, __fmul_rn(sh, p.pixel_a));
  const float s2 = __fadd_rn(__fmul_rn(sx, sx), __fmul_rn(sy, sy));
  if (__fsqrt_rn(s2) < p.cuton_freq) return;
  float def = p.defocus1;
  if (p.has_astigmatism == 1u) {
    const float da = __fsub_rn(atan2f(sy, sx), p.astig_angle_rad);
    const float c = cosf(da), s = sinf(da);
    def = __fadd_rn(__fmul_rn(p.defocus1, __fmul_rn(c, c)), __fmul_rn(p.defocus2, __fmul_rn(s, s)));
  }
  const float wl = p.wavelength;
  const float t = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(0.5f, p.cs_a), wl), wl), s2);
  const float chi = __fmul_rn(__fmul_rn(__fmul_rn(3.14159265358979323846f, wl), s2), __fsub_rn(def, t));
  const float chi_t = __fadd_rn(chi, p.plate_phase_rad);
  const float w = p.amp_contrast;
  const float w_phase = __fsqrt_rn(__fsub_rn(1.0f, __fmul_rn(w, w)));
  const float ctf = __fadd_rn(__fmul_rn(-sinf(chi_t), w_phase), __fmul_rn(cosf(chi_t), w));
  if (ctf < 0.0f) {
    re[i] = -re[i];
    im[i] = -im[i];
  }
}

double electron_wavelength(float kv) {  // main.rs:706-718
  const double v = (double)kv * 1000.0;
  const double m0 = 9.10938e-31, e = 1.60218e-19, c = 2.99792e8, h = 6.62607e-34;
  const double lam = h / sqrt(2.0 * m0 * e * v * (1.0 + e * v / (2.0 * m0 * c * c)));
  return lam * 1e10;
}

struct DevBuf {  // device allocations of one call, freed on every return path
  std::vector<void *> ptrs;
  cudaStream_t st = nullptr;
  ~DevBuf() {
    if (st) cudaStreamSynchronize(st);
    for (void *p : ptrs) cudaFree(p);
    if (st) cudaStreamDestroy(st);
  }
  template <class T> cudaError_t alloc(T **p, size_t bytes) {
    cudaError_t e = cudaMalloc((void **)p, std::max<size_t>(bytes, 16));
    if (e == cudaSuccess) ptrs.push_back(*p);
    return e;
  }
};

// Rows per CTA of a stage whose transforms have at most n samples: as many as
// CTF_SMEM holds, at least one (up to CTF_MAX_N samples, 196 KB).
int ctf_rows_per_block(int n) {
  int r = CTF_ROWS;
  while (r > 1 && (size_t)2 * r * ctf_ld(n) * sizeof(float2) > CTF_SMEM) r /= 2;
  return r;
}

template <class K> void launch_stage(K kernel, const CtfArgs &a, int n, int max_rows, int items, cudaStream_t st) {
  const int rpb = ctf_rows_per_block(n);
  const size_t smem = (size_t)2 * rpb * ctf_ld(n) * sizeof(float2);
  // the same limit from every thread, whatever the length
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * ctf_ld(CTF_MAX_N) * (int)sizeof(float2));
  kernel<<<dim3((max_rows + rpb - 1) / rpb, items), 256, smem, st>>>(a, rpb);
}

}  // namespace

int ctf_strip_width(const tg_ctf_options *o, int nx, const float *view_def, int nviews) {  // main.rs:284-324
  size_t max_w;
  if (o->max_strip_width > 0) {
    max_w = (size_t)o->max_strip_width;
  } else {
    double max_def = 0.0;
    if (view_def) {
      for (int v = 0; v < nviews; ++v)
        max_def = std::max(max_def, (double)std::max(fabsf(view_def[3 * v]), fabsf(view_def[3 * v + 1])) * 10.0);
    } else {
      max_def = (double)fabsf(o->defocus) * 10.0;
    }
    const double wl = electron_wavelength(o->voltage);
    if (max_def > 1.0 && wl > 0.0) {
      const double safe = std::max((double)o->pixel_size / (wl * (max_def / (double)nx)), 16.0);
      max_w = (size_t)safe;
    } else {
      max_w = (size_t)std::max(o->strip_width, 0);
    }
  }
  return (int)std::min((size_t)std::max(o->strip_width, 0), max_w);
}

}  // namespace tg

using namespace tg;

extern "C" {

void tg_ctf_options_default(tg_ctf_options *o) {
  if (!o) return;
  memset(o, 0, sizeof *o);
  o->defocus = -3000.0f;
  o->voltage = 300.0f;
  o->cs = 2.7f;
  o->pixel_size = 1.0f;
  o->strip_width = 256;
  o->tilt_axis_angle = 0.0f;
  o->max_strip_width = 0;
  o->amplitude_contrast = 0.07f;
  o->cuton_freq = 0.0f;
  o->plate_phase = 0.0f;
  o->device = 0;
}

int tg_ctf_strip_width(const tg_ctf_options *o, int32_t nx, const float *view_defocus, int32_t n_view_defocus,
                       int32_t *out) {
  if (!o || !out || nx < 1) return TG_ERR_INVALID_ARG;
  *out = ctf_strip_width(o, nx, view_defocus, view_defocus ? n_view_defocus : 0);
  return TG_OK;
}

int tg_ctf_phaseflip(const tg_ctf_options *o, const float *host_in, int32_t nx, int32_t ny, int32_t nz,
                     const float *angles, int32_t n_angles, const float *view_defocus, int32_t n_view_defocus,
                     float *host_out, tg_stats *stats) {
  if (!o || !host_in || !host_out || nx < 1 || ny < 1 || nz < 1 || (n_angles > 0 && !angles)) {
    set_error("tg_ctf_phaseflip: null pointer or empty stack");
    return TG_ERR_INVALID_ARG;
  }
  const int strip_width = ctf_strip_width(o, nx, view_defocus, view_defocus ? n_view_defocus : 0);
  if (strip_width < 1) { set_error("strip width must be at least 1"); return TG_ERR_INVALID_ARG; }
  // strip geometry (main.rs:436-509), once for the stack
  const double tilt_axis_rad = (double)o->tilt_axis_angle * PI32_D / 180.0;
  const double perp_x = cos(tilt_axis_rad), perp_y = sin(tilt_axis_rad);
  const double cxp = (double)nx / 2.0, cyp = (double)ny / 2.0;
  double min_perp = 1.79769313486231570e+308, max_perp = -1.79769313486231570e+308;
  const double corners[4][2] = {{0.0, 0.0}, {(double)nx, 0.0}, {0.0, (double)ny}, {(double)nx, (double)ny}};
  for (auto &c : corners) {
    const double d = (c[0] - cxp) * perp_x + (c[1] - cyp) * perp_y;
    min_perp = std::min(min_perp, d);
    max_perp = std::max(max_perp, d);
  }
  const double sw_d = (double)strip_width;
  const double n_strips_d = ceil((max_perp - min_perp) / sw_d);
  if (!(n_strips_d >= 0.0 && n_strips_d <= (double)nx + (double)ny + 2.0)) {
    set_error("tilt axis angle must be finite");
    return TG_ERR_INVALID_ARG;
  }
  const int n_strips = (int)n_strips_d;
  struct Box { int x0, x1, y0, y1; };
  std::vector<CtfStrip> strips(n_strips);
  std::vector<Box> box(n_strips, Box{nx, 0, ny, 0});
  for (int k = 0; k < n_strips; ++k) {
    CtfStrip &g = strips[k];
    g.center = min_perp + ((double)k + 0.5) * sw_d;
    g.lo = g.center - sw_d / 2.0;
    g.hi = g.center + sw_d / 2.0;
  }
  // bounding boxes, one walk over the pixels: along a row in the direction in
  // which d grows, the strips' bounds are passed in order
  for (int y = 0; y < ny; ++y) {
    const double ty = ((double)y - cyp) * perp_y;
    for (int i = 0, k = 0; i < nx; ++i) {
      const int x = perp_x >= 0.0 ? i : nx - 1 - i;
      const double d = ((double)x - cxp) * perp_x + ty;
      while (k < n_strips && d >= strips[k].hi) ++k;
      for (int j = k; j < n_strips && d >= strips[j].lo; ++j) {
        Box &b = box[j];
        b.x0 = std::min(b.x0, x);
        b.x1 = std::max(b.x1, x + 1);
        b.y0 = std::min(b.y0, y);
        b.y1 = std::max(b.y1, y + 1);
      }
    }
  }
  size_t view_samples = 0, work = 1;  // samples of all strips of a view, and of the largest
  int max_w = 1, max_h = 1, kept = 0;
  std::map<int, int> lengths;  // transform length -> plan index
  for (int k = 0; k < n_strips; ++k) {
    const Box &b = box[k];
    if (b.x1 <= b.x0 || b.y1 <= b.y0) continue;
    CtfStrip g = strips[k];
    g.x0 = b.x0; g.y0 = b.y0; g.sw = b.x1 - b.x0; g.sh = b.y1 - b.y0;
    if (g.sw > CTF_MAX_N || g.sh > CTF_MAX_N) {
      set_error("strip dimension above " + std::to_string(CTF_MAX_N) + " samples");
      return TG_ERR_UNSUPPORTED;
    }
    g.dx_a = g.center * (double)o->pixel_size;
    g.scale = 1.0f / (float)((size_t)g.sw * g.sh);
    g.off = view_samples;
    g.plan_w = lengths.emplace(g.sw, (int)lengths.size()).first->second;
    g.plan_h = lengths.emplace(g.sh, (int)lengths.size()).first->second;
    view_samples += (size_t)g.sw * g.sh;
    work = std::max(work, (size_t)g.sw * g.sh);
    max_w = std::max(max_w, g.sw);
    max_h = std::max(max_h, g.sh);
    strips[kept++] = g;
  }
  strips.resize(kept);
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { set_error("no CUDA device"); return TG_ERR_NO_DEVICE; }
  if (o->device < 0 || o->device >= ndev) { set_error("bad device ordinal"); return TG_ERR_INVALID_ARG; }
  TG_CUDA(cudaSetDevice(o->device));
  DevBuf mem;
  TG_CUDA(cudaStreamCreateWithFlags(&mem.st, cudaStreamNonBlocking));
  cudaStream_t st = mem.st;
  const size_t npix = (size_t)nx * ny, ntot = npix * nz;
  FaultAhead out_pages(host_out, ntot * 4);
  // Views per chunk, or (0) runs of strips of one view: whole views where they fit.
  const size_t view_bytes = std::max<size_t>(view_samples, 1) * 2 * sizeof(float2);
  int nv = kept > 0 && kept <= 65535 ? (int)std::min<size_t>({CTF_CHUNK_BYTES / view_bytes, (size_t)(65535 / kept), (size_t)nz}) : 0;
  size_t cap = nv ? view_samples * nv : std::max(work, CTF_CHUNK_BYTES / (2 * sizeof(float2)));
  float *d_stack, *d_wsum = nullptr, *d_wtot = nullptr, *d_slice, *d_stats3;
  float2 *d_work;
  StatPartial *d_part;
  CtfStrip *d_strips;
  CtfView *d_views;
  CtfPlan *d_plans;
  cudaError_t e;
  if ((e = mem.alloc(&d_stack, ntot * 4)) || (e = mem.alloc(&d_part, (size_t)nz * 64 * sizeof(StatPartial))) ||
      (e = mem.alloc(&d_slice, (size_t)nz * 12)) || (e = mem.alloc(&d_stats3, 16)) ||
      (e = mem.alloc(&d_strips, (size_t)kept * sizeof(CtfStrip))) ||
      (e = mem.alloc(&d_views, (size_t)nz * sizeof(CtfView))) ||
      (e = mem.alloc(&d_plans, lengths.size() * sizeof(CtfPlan))))
    return cuda_fail(e, "cudaMalloc(ctfphaseflip)");
  e = mem.alloc(&d_work, cap * 2 * sizeof(float2));
  if (e == cudaErrorMemoryAllocation && cap > work) {  // little memory left: strip by strip
    cudaGetLastError();
    nv = 0;
    cap = work;
    e = mem.alloc(&d_work, cap * 2 * sizeof(float2));
  }
  if (e == cudaSuccess && nv == 0)
    if ((e = mem.alloc(&d_wsum, npix * 4)) == cudaSuccess) e = mem.alloc(&d_wtot, npix * 4);
  if (e) return cuda_fail(e, "cudaMalloc(ctfphaseflip)");

  // tables: plans with their twiddles, strips, views
  std::vector<CtfPlan> plans(lengths.size());
  size_t tw_total = 0;
  for (auto &kv : lengths) tw_total += kv.first;
  std::vector<float2> tw(std::max<size_t>(tw_total, 1));
  float2 *d_tw;
  if ((e = mem.alloc(&d_tw, tw.size() * sizeof(float2)))) return cuda_fail(e, "cudaMalloc(twiddles)");
  tw_total = 0;
  for (auto &kv : lengths) {
    const int n = kv.first;
    CtfPlan &p = plans[kv.second];
    int m = n;
    fft_plan(n, &p.plan);  // the factors up to 7; the rest are prime radices
    for (int i = 0; i < p.plan.nfac; ++i) m /= p.plan.fac[i];
    for (int r = 11; m > 1; r += 2)
      for (; m % r == 0; m /= r) p.plan.fac[p.plan.nfac++] = r;
    p.tw = d_tw + tw_total;
    for (int k = 0; k < n; ++k) {
      const double t = -2.0 * M_PI * (double)k / (double)n;
      tw[tw_total + k] = make_float2((float)cos(t), (float)sin(t));
    }
    tw_total += n;
  }
  const double amp = (double)o->amplitude_contrast;
  std::vector<CtfView> views(nz);
  for (int z = 0; z < nz; ++z) {
    const float tilt_deg = z < n_angles ? angles[z] : 0.0f;
    float d1 = o->defocus, d2 = o->defocus, astig = 0.0f;
    if (view_defocus && z < n_view_defocus) {
      d1 = view_defocus[3 * z];
      d2 = view_defocus[3 * z + 1];
      astig = view_defocus[3 * z + 2];
    }
    CtfView &w = views[z];
    w.sin_tilt = sin((double)tilt_deg * PI32_D / 180.0);
    w.def1 = (double)d1 * 10.0;
    w.def2 = (double)d2 * 10.0;
    w.astig_rad = (double)astig * PI32_D / 180.0;
    w.has_astig = fabs(w.def1 - w.def2) > 0.01 ? 1 : 0;
  }
  TG_CUDA(cudaMemcpyAsync(d_tw, tw.data(), tw_total * sizeof(float2), cudaMemcpyHostToDevice, st));
  TG_CUDA(cudaMemcpyAsync(d_plans, plans.data(), plans.size() * sizeof(CtfPlan), cudaMemcpyHostToDevice, st));
  TG_CUDA(cudaMemcpyAsync(d_strips, strips.data(), strips.size() * sizeof(CtfStrip), cudaMemcpyHostToDevice, st));
  TG_CUDA(cudaMemcpyAsync(d_views, views.data(), views.size() * sizeof(CtfView), cudaMemcpyHostToDevice, st));

  CtfArgs f{};
  f.stack = d_stack;
  f.strips = d_strips;
  f.views = d_views;
  f.plans = d_plans;
  f.A = d_work;
  f.B = d_work + cap;
  f.nx = nx;
  f.ny = ny;
  f.pixel_a = (double)o->pixel_size;
  f.wl = electron_wavelength(o->voltage);
  f.cs_a = (double)o->cs * 1e7;
  f.amp = amp;
  f.w_phase = sqrt(1.0 - amp * amp);
  f.cuton = (double)o->cuton_freq;
  f.plate = (double)o->plate_phase * PI32_D / 180.0;
  f.tilt_axis_rad = tilt_axis_rad;
  f.cos_ta = cos(tilt_axis_rad);
  f.sin_ta = sin(tilt_axis_rad);
  CombineArgs q{};
  q.cxp = cxp; q.cyp = cyp; q.perp_x = perp_x; q.perp_y = perp_y;
  q.min_perp = min_perp; q.width = sw_d; q.half_w = sw_d / 2.0;
  q.wsum = d_wsum;
  q.wtot = d_wtot;
  q.max_off = n_strips - kept;
  {
    NvtxRange nv_range("tg.ctfphaseflip");
    const int dz = std::max(nv, 1);
    for (int z = 0; z < nz; z += dz) {
      const int cv = std::min(dz, nz - z);
      f.z0 = z;
      TG_CUDA(cudaMemcpyAsync(d_stack + z * npix, host_in + z * npix, cv * npix * 4, cudaMemcpyHostToDevice, st));
      for (int s = 0, s1; s < kept; s = s1) {
        s1 = nv ? kept : s + 1;
        while (s1 < kept && s1 - s < 65535 &&
               strips[s1].off + (size_t)strips[s1].sw * strips[s1].sh - strips[s].off <= cap)
          ++s1;
        f.s0 = s;
        f.ns = s1 - s;
        f.base = strips[s].off;
        f.view_stride = view_samples;  // one view unless it is a whole number of them
        q.first = s == 0;
        q.last = s1 == kept;
        launch_stage(ctf_rows_in_kernel, f, max_w, max_h, cv * f.ns, st);
        launch_stage(ctf_columns_kernel, f, max_h, max_w, cv * f.ns, st);
        launch_stage(ctf_rows_out_kernel, f, max_w, max_h, cv * f.ns, st);
        ctf_combine_kernel<<<dim3((unsigned)((npix + 255) / 256), cv), 256, 0, st>>>(f, q);
        TG_CUDA(cudaGetLastError());
      }
    }
    // statistics (main.rs:681-693): per-section min, max and f64 sum, folded in order
    int ntiles = 0;
    launch_transform_stats(d_stack, nx, ny, nz, 1.0f, 1.0f, 0.0f, d_part, &ntiles, st);
    launch_stats_reduce(d_part, nz, ntiles, (int)npix, d_slice, d_stats3, st);
    TG_CUDA(cudaGetLastError());
  }
  out_pages.join();
  TG_CUDA(cudaMemcpyAsync(host_out, d_stack, ntot * 4, cudaMemcpyDeviceToHost, st));
  float s3[3];
  TG_CUDA(cudaMemcpyAsync(s3, d_stats3, 12, cudaMemcpyDeviceToHost, st));
  TG_CUDA(cudaStreamSynchronize(st));
  if (stats) {
    stats->amin = s3[0];
    stats->amax = s3[1];
    stats->amean = s3[2];
  }
  return TG_OK;
}

int tg_ctf_correct_strip(float *strip_re, float *strip_im, const tg_ctf_strip_params *p, int32_t device) {
  if (!strip_re || !strip_im || !p || p->sw == 0 || p->sh == 0) return TG_ERR_INVALID_ARG;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { set_error("no CUDA device"); return TG_ERR_NO_DEVICE; }
  if (device < 0 || device >= ndev) { set_error("bad device ordinal"); return TG_ERR_INVALID_ARG; }
  TG_CUDA(cudaSetDevice(device));
  const size_t n = (size_t)p->sw * p->sh;
  DevBuf mem;
  TG_CUDA(cudaStreamCreateWithFlags(&mem.st, cudaStreamNonBlocking));
  float *d_re, *d_im;
  cudaError_t e;
  if ((e = mem.alloc(&d_re, n * 4)) || (e = mem.alloc(&d_im, n * 4))) return cuda_fail(e, "cudaMalloc(strip)");
  TG_CUDA(cudaMemcpyAsync(d_re, strip_re, n * 4, cudaMemcpyHostToDevice, mem.st));
  TG_CUDA(cudaMemcpyAsync(d_im, strip_im, n * 4, cudaMemcpyHostToDevice, mem.st));
  ctf_strip_f32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, mem.st>>>(d_re, d_im, *p);
  TG_CUDA(cudaGetLastError());
  TG_CUDA(cudaMemcpyAsync(strip_re, d_re, n * 4, cudaMemcpyDeviceToHost, mem.st));
  TG_CUDA(cudaMemcpyAsync(strip_im, d_im, n * 4, cudaMemcpyDeviceToHost, mem.st));
  TG_CUDA(cudaStreamSynchronize(mem.st));
  return TG_OK;
}

}  // extern "C"
