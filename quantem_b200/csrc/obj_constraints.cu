// Optional object constraints of the reference's object model and the probe-overlap
// FOV mask they use (object_models.py:273-480, ptychography_base.py:191-216):
//
//  * probe overlap: sum over positions of |probe mode 0|^2 placed at each patch window;
//  * hard constraint with the FOV mask (apply_fov_mask): complex / pure-phase objects
//    amp m exp(i (angle - mean angle) m) m, potentials (V - offset)+ m, the potential's
//    baseline offset taken from the mask's background (fix_potential_baseline);
//  * exp(i V) of a (filtered) potential;
//  * Gaussian blur (gaussian_sigma): zero-padded separable correlation, self-adjoint;
//  * identical slices: every slice replaced by the slice mean;
//  * soft constraints: TV of phase / amplitude / potential along z and in-plane, and the
//    surface-zero terms of the first and last slices, with their gradients.
//
// Every pass is an HBM-bound elementwise or stencil sweep over the (S, Ho, Wo) object;
// reductions go through fixed-order per-block partials, so every result repeats bit for bit.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "line_fft.cuh"
#include "ptycho_b200.h"

int qb_record_error(int code, const char* msg);

namespace {

constexpr int kBlocks = 296;  // 2 x 148 SMs
constexpr int kThreads = 256;

__device__ __forceinline__ double block_sum_d(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
  return t;  // valid in thread 0
}

// fixed-order sum of n partials, broadcast to the whole block
__device__ __forceinline__ double partials_sum(const double* part, int n) {
  __shared__ double red[32];
  __shared__ double bc;
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) v += part[i];
  const double t = block_sum_d(v, red);
  if (threadIdx.x == 0) bc = t;
  __syncthreads();
  return bc;
}

__device__ __forceinline__ int wrapi(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

__device__ __forceinline__ float sgnf(float x) { return (x > 0.f) - (x < 0.f); }

// ------------------------------------------------------------------ probe overlap
__global__ void probe_overlap_kernel(const float* __restrict__ inten, int n, const float* __restrict__ pos, int npos,
                                     int Ho, int Wo, float* __restrict__ out) {
  const int64_t nn = (int64_t)n * n;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nn * npos; t += (int64_t)gridDim.x * blockDim.x) {
    const int b = (int)(t / nn);
    const int k = (int)(t % nn);
    const int i = k / n, j = k % n;
    const int fi = i < (n + 1) / 2 ? i : i - n, fj = j < (n + 1) / 2 ? j : j - n;  // fftfreq index
    const int r = wrapi((int)rintf(pos[2 * b]) + fi, Ho);
    const int c = wrapi((int)rintf(pos[2 * b + 1]) + fj, Wo);
    atomicAdd(out + (int64_t)r * Wo + c, inten[k]);
  }
}

// ------------------------------------------------- hard constraint with the FOV mask
// work layout (doubles): [0, kBlocks) angle partials, [kBlocks, 2 kBlocks) gradient partials
__global__ void angle_partials_kernel(const float2* __restrict__ obj, int64_t n, double* part) {
  __shared__ double red[32];
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 o = obj[i];
    v += (double)atan2f(o.y, o.x);
  }
  const double t = block_sum_d(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// out = A exp(i theta m), A = amp m^2, theta = angle - mean angle (PURE: amp = 1)
template <bool PURE>
__global__ void fov_apply_kernel(const float2* __restrict__ obj, const float* __restrict__ mask, int64_t hw,
                                 float2* __restrict__ out, int64_t n, const double* part) {
  const float mean = (float)(partials_sum(part, kBlocks) / (double)n);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 o = obj[i];
    const float m = mask[i % hw];
    const float amp = PURE ? 1.0f : fminf(fmaxf(hypotf(o.x, o.y), 0.0f), 1.0f);
    const float A = amp * m * m;
    float s, c;
    sincosf((atan2f(o.y, o.x) - mean) * m, &s, &c);
    out[i] = make_float2(A * c, A * s);
  }
}

// g_theta = m A Im(conj(e) G), summed for the mean-phase term
template <bool PURE>
__global__ void fov_vjp_partials_kernel(const float2* __restrict__ obj, const float* __restrict__ mask, int64_t hw,
                                        const float2* __restrict__ g, int64_t n, const double* part_fwd,
                                        double* part) {
  __shared__ double red[32];
  const float mean = (float)(partials_sum(part_fwd, kBlocks) / (double)n);
  double v = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 o = obj[i], gg = g[i];
    const float m = mask[i % hw];
    const float amp = PURE ? 1.0f : fminf(fmaxf(hypotf(o.x, o.y), 0.0f), 1.0f);
    float s, c;
    sincosf((atan2f(o.y, o.x) - mean) * m, &s, &c);
    v += (double)(m * amp * m * m * (gg.y * c - gg.x * s));
  }
  const double t = block_sum_d(v, red);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

template <bool PURE>
__global__ void fov_vjp_apply_kernel(const float2* __restrict__ obj, const float* __restrict__ mask, int64_t hw,
                                     const float2* __restrict__ g, float2* __restrict__ gout, int64_t n,
                                     const double* part_fwd, const double* part_g) {
  const float mean = (float)(partials_sum(part_fwd, kBlocks) / (double)n);
  __syncthreads();
  const float gmean = (float)(partials_sum(part_g, kBlocks) / (double)n);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float2 o = obj[i], gg = g[i];
    const float m = mask[i % hw];
    const float mag = hypotf(o.x, o.y);
    const float amp = PURE ? 1.0f : fminf(fmaxf(mag, 0.0f), 1.0f);
    float s, c;
    sincosf((atan2f(o.y, o.x) - mean) * m, &s, &c);
    const float g_amp = m * m * (gg.x * c + gg.y * s);               // Re(conj(e) G) m^2
    const float g_ph = m * amp * m * m * (gg.y * c - gg.x * s) - gmean;  // mean-removed g_theta
    const float g_mag = (!PURE && mag >= 0.0f && mag <= 1.0f) ? g_amp : 0.0f;
    float2 r = make_float2(0.f, 0.f);
    if (mag != 0.0f) {
      const float inv = 1.0f / mag;
      r.x = g_mag * o.x * inv - g_ph * o.y * inv * inv;
      r.y = g_mag * o.y * inv + g_ph * o.x * inv * inv;
    }
    gout[i] = r;
  }
}

// ------------------------------------------------------------- potential base
// work layout: [0, kB) max of the mask (per block), [kB, 2kB) background sums,
// [2kB, 3kB) background counts, [3kB, 4kB) minima of V
__global__ void mask_max_kernel(const float* __restrict__ mask, int64_t hw, double* part) {
  __shared__ float red[32];
  float m = -INFINITY;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < hw; i += (int64_t)gridDim.x * blockDim.x)
    m = fmaxf(m, mask[i]);
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, red[w]);
    part[blockIdx.x] = (double)fmaxf(m, red[0]);
  }
}

__device__ __forceinline__ float partials_max(const double* part, int n) {
  __shared__ float bc;
  if (threadIdx.x == 0) {
    double m = part[0];
    for (int i = 1; i < n; ++i) m = fmax(m, part[i]);
    bc = (float)m;
  }
  __syncthreads();
  return bc;
}

__global__ void background_stats_kernel(const float* __restrict__ v, const float* __restrict__ mask, int64_t hw,
                                        int64_t n, double* work) {
  __shared__ double red[32];
  __shared__ float redm[32];
  const float mmax = mask ? partials_max(work, kBlocks) : 0.0f;
  double sum = 0.0, cnt = 0.0;
  float mn = INFINITY;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = v[i];
    mn = fminf(mn, x);
    if (mask && mask[i % hw] < 0.5f * mmax) {
      sum += (double)x;
      cnt += 1.0;
    }
  }
  const double ts = block_sum_d(sum, red);
  const double tc = block_sum_d(cnt, red);
  for (int o = 16; o > 0; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  if ((threadIdx.x & 31) == 0) redm[threadIdx.x >> 5] = mn;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mn = fminf(mn, redm[w]);
    work[kBlocks + blockIdx.x] = ts;
    work[2 * kBlocks + blockIdx.x] = tc;
    work[3 * kBlocks + blockIdx.x] = (double)fminf(mn, redm[0]);
  }
}

// offset = factor * (mean of V over the background, or min V without one); 0 when not fixed
__device__ __forceinline__ float potential_offset_bg(const double* work, int fix, float factor) {
  if (!fix) return 0.0f;
  const double s = partials_sum(work + kBlocks, kBlocks);
  __syncthreads();
  const double c = partials_sum(work + 2 * kBlocks, kBlocks);
  __shared__ float bc;
  if (threadIdx.x == 0) {
    double off;
    if (c > 0.0) {
      off = (double)(float)(s / c);
    } else {
      double m = work[3 * kBlocks];
      for (int i = 1; i < kBlocks; ++i) m = fmin(m, work[3 * kBlocks + i]);
      off = m;
    }
    bc = (float)off * factor;
  }
  __syncthreads();
  return bc;
}

__global__ void potential_base_kernel(const float* __restrict__ v, const float* __restrict__ mask, int64_t hw,
                                      float* __restrict__ out, int64_t n, int positivity, int fix, float factor,
                                      const double* work) {
  const float off = potential_offset_bg(work, fix, factor);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float x = v[i] - off;
    if (positivity) x = fmaxf(x, 0.0f);
    out[i] = mask ? x * mask[i % hw] : x;
  }
}

// the offset is detached (as in the reference); the clamp passes where V - offset >= 0
__global__ void potential_base_vjp_kernel(const float* __restrict__ v, const float* __restrict__ mask, int64_t hw,
                                          const float* __restrict__ g, float* __restrict__ gout, int64_t n,
                                          int positivity, int fix, float factor, const double* work) {
  const float off = potential_offset_bg(work, fix, factor);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = v[i] - off;
    const bool pass = !positivity || x >= 0.0f;
    gout[i] = pass ? (mask ? g[i] * mask[i % hw] : g[i]) : 0.0f;
  }
}

// ------------------------------------------------------------------ exp(i V)
__global__ void phase_exp_kernel(const float* __restrict__ v, float2* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float s, c;
    sincosf(v[i], &s, &c);
    out[i] = make_float2(c, s);
  }
}

__global__ void phase_exp_vjp_kernel(const float* __restrict__ v, const float2* __restrict__ g, float* __restrict__ gout,
                                     int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float s, c;
    sincosf(v[i], &s, &c);
    gout[i] = g[i].y * c - g[i].x * s;  // Re(conj(G) i t)
  }
}

// --------------------------------------------------------------- Gaussian blur
// out[s, r, c, k] = sum_t taps[t] in[s, r + t - R, c, k] (AXIS 0) or along c (AXIS 1),
// zero outside; K floats per element (1 real, 2 complex)
template <int AXIS>
__global__ void blur_pass_kernel(const float* __restrict__ in, float* __restrict__ out, int S, int Ho, int Wo, int K,
                                 const float* __restrict__ taps, int ntaps) {
  __shared__ float st[256];
  for (int t = threadIdx.x; t < ntaps; t += blockDim.x) st[t] = taps[t];
  __syncthreads();
  const int R = ntaps / 2;
  const int64_t rowlen = (int64_t)Wo * K;
  const int64_t n = (int64_t)S * Ho * rowlen;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t plane = i / ((int64_t)Ho * rowlen);
    const int64_t rem = i % ((int64_t)Ho * rowlen);
    const int r = (int)(rem / rowlen);
    const int64_t ck = rem % rowlen;
    const int c = (int)(ck / K);
    const int k = (int)(ck % K);
    const float* base = in + plane * Ho * rowlen;
    float acc = 0.f;
    if (AXIS == 0) {
      for (int t = 0; t < ntaps; ++t) {
        const int rr = r + t - R;
        if (rr >= 0 && rr < Ho) acc = fmaf(st[t], base[(int64_t)rr * rowlen + ck], acc);
      }
    } else {
      for (int t = 0; t < ntaps; ++t) {
        const int cc = c + t - R;
        if (cc >= 0 && cc < Wo) acc = fmaf(st[t], base[(int64_t)r * rowlen + (int64_t)cc * K + k], acc);
      }
    }
    out[i] = acc;
  }
}

// Both passes in one: a 32 x 32 tile and its halo of R = ntaps / 2 <= kBlurHalo elements in
// shared memory, along the rows first, then along the columns, with the same sums as the two
// passes.  Bound by the walk over the taps: 31, 39, 58 and 105 us for 3, 7, 15 and 33 taps at 8 x 510 x 516
// complex values, 17 MB each way; the two passes, each output walking its taps through the L1 cache,
// take 60, 81, 122 and 202.  Longer kernels take the two passes, since their tile would be mostly halo, and so do objects of
// fewer than kBlurLeast elements, whose tiles leave SMs idle (complex, 7 and 33 taps, passes against
// tiles: 1 x 100 x 100 5.0 / 7.6 us against 9.4 / 14.7, 1 x 400 x 400 9.6 / 19.6 against 10.1 / 18.7, 1 x 450
// x 450 11.5 / 24.3 against 10.2 / 18.9).
constexpr int64_t kBlurLeast = 200000;
constexpr int kBlurTile = 32, kBlurHalo = 16;
// dynamic shared memory with the longest taps, complex values
constexpr size_t kBlurSmem = sizeof(float) * 2 * (2 * kBlurTile + 2 * kBlurHalo) * (kBlurTile + 2 * kBlurHalo);
template <int K>
__global__ void __launch_bounds__(kThreads) blur_tile_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                             int Ho, int Wo, const float* __restrict__ taps,
                                                             int ntaps) {
  extern __shared__ float bsh[];
  __shared__ float st[2 * kBlurHalo + 1];
  const int R = ntaps / 2, side = kBlurTile + 2 * R, pitch = side * K;
  float *tile = bsh, *mid = bsh + side * pitch;  // side x side, then 32 x side
  for (int t = threadIdx.x; t < ntaps; t += kThreads) st[t] = taps[t];
  const int64_t rowlen = (int64_t)Wo * K;
  const float* src = in + (int64_t)blockIdx.z * Ho * rowlen;
  float* dst = out + (int64_t)blockIdx.z * Ho * rowlen;
  const int r0 = blockIdx.y * kBlurTile, c0 = blockIdx.x * kBlurTile;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = kThreads / 32;
  for (int i = w; i < side; i += nw) {
    const int r = r0 + i - R;
    for (int j = lane; j < pitch; j += 32) {
      const int64_t ck = (int64_t)(c0 - R) * K + j;
      tile[i * pitch + j] = r >= 0 && r < Ho && ck >= 0 && ck < rowlen ? src[r * rowlen + ck] : 0.f;
    }
  }
  __syncthreads();
  // out-of-range elements are 0 in the tile: a sum over all taps adds exact zeros
  for (int i = w; i < kBlurTile; i += nw)
    for (int j = lane; j < pitch; j += 32) {
      float acc = 0.f;
      for (int t = 0; t < ntaps; ++t) acc = fmaf(st[t], tile[(i + t) * pitch + j], acc);
      mid[i * pitch + j] = acc;
    }
  __syncthreads();
  for (int i = w; i < kBlurTile; i += nw) {
    if (r0 + i >= Ho) break;
    for (int j = lane; j < kBlurTile * K; j += 32) {
      const int64_t ck = (int64_t)c0 * K + j;
      if (ck >= rowlen) break;
      float acc = 0.f;
      for (int t = 0; t < ntaps; ++t) acc = fmaf(st[t], mid[i * pitch + j + t * K], acc);
      dst[(r0 + i) * rowlen + ck] = acc;
    }
  }
}

// ------------------------------------------------------------- identical slices
__global__ void slice_mean_kernel(const float* __restrict__ in, float* __restrict__ out, int S, int64_t plane) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < plane; p += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int s = 0; s < S; ++s) acc += (double)in[(int64_t)s * plane + p];
    const float m = (float)(acc / (double)S);
    for (int s = 0; s < S; ++s) out[(int64_t)s * plane + p] = m;
  }
}

// ------------------------------------------------------------ soft constraints
// KIND 0: complex (phase and amplitude terms), 1: pure phase (phase terms), 2: real potential.
// work: [0, kB) loss partials, [kB, 2kB) / [2kB, 3kB) sum |phase| of the first / last slice,
// [3kB, 4kB) / [4kB, 5kB) sum sign(u) of the first / last slice
template <int KIND>
__device__ __forceinline__ void values_at(const float* obj, int64_t i, float& ph, float& amp) {
  if (KIND == 2) {
    ph = obj[i];
    amp = 0.f;
  } else {
    const float2 o = reinterpret_cast<const float2*>(obj)[i];
    ph = atan2f(o.y, o.x);
    amp = hypotf(o.x, o.y);
  }
}

template <int KIND>
__global__ void surface_abs_phase_kernel(const float* __restrict__ obj, int S, int64_t hw, double* work) {
  __shared__ double red[32];
  double a0 = 0.0, a1 = 0.0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < hw; p += (int64_t)gridDim.x * blockDim.x) {
    float ph, amp;
    values_at<KIND>(obj, p, ph, amp);
    a0 += fabsf(ph);
    values_at<KIND>(obj, (int64_t)(S - 1) * hw + p, ph, amp);
    a1 += fabsf(ph);
  }
  const double t0 = block_sum_d(a0, red);
  const double t1 = block_sum_d(a1, red);
  if (threadIdx.x == 0) {
    work[kBlocks + blockIdx.x] = t0;
    work[2 * kBlocks + blockIdx.x] = t1;
  }
}

template <int KIND>
__global__ void surface_sign_kernel(const float* __restrict__ obj, int S, int64_t hw, double* work) {
  __shared__ double red[32];
  const float m0 = (float)(partials_sum(work + kBlocks, kBlocks) / (double)hw);
  __syncthreads();
  const float m1 = (float)(partials_sum(work + 2 * kBlocks, kBlocks) / (double)hw);
  double a0 = 0.0, a1 = 0.0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < hw; p += (int64_t)gridDim.x * blockDim.x) {
    float ph, amp;
    values_at<KIND>(obj, p, ph, amp);
    a0 += sgnf(fabsf(ph) - m0);
    values_at<KIND>(obj, (int64_t)(S - 1) * hw + p, ph, amp);
    a1 += sgnf(fabsf(ph) - m1);
  }
  const double t0 = block_sum_d(a0, red);
  const double t1 = block_sum_d(a1, red);
  if (threadIdx.x == 0) {
    work[3 * kBlocks + blockIdx.x] = t0;
    work[4 * kBlocks + blockIdx.x] = t1;
  }
}

// Weights and surface terms of one launch (object_models.py:398-411): z with wz (3-D arrays, S > 1),
// rows and columns with wxy; each term w mean|diff| divided by the number of weighted dimensions.
struct SoftTerms {
  float c0, c1, c2, wsurf, inv_hw, m0, m1, sg0, sg1;
  bool surf;
};
template <int KIND>
__device__ SoftTerms soft_terms(int S, int Ho, int Wo, float wz, float wxy, float wsurf, const double* work) {
  const int64_t hw = (int64_t)Ho * Wo;
  SoftTerms t = {0.f, 0.f, 0.f, wsurf, 1.0f / (float)hw, 0.f, 0.f, 0.f, 0.f, wsurf > 0.f && S >= 3};
  if (t.surf && KIND != 2) {
    t.m0 = (float)(partials_sum(work + kBlocks, kBlocks) / (double)hw);
    __syncthreads();
    t.m1 = (float)(partials_sum(work + 2 * kBlocks, kBlocks) / (double)hw);
    __syncthreads();
    t.sg0 = (float)(partials_sum(work + 3 * kBlocks, kBlocks) / (double)hw);
    __syncthreads();
    t.sg1 = (float)(partials_sum(work + 4 * kBlocks, kBlocks) / (double)hw);
  }
  const float w0 = S > 1 ? wz : 0.f;
  const int nd = (w0 > 0.f) + 2 * (wxy > 0.f);
  if (nd && w0 > 0.f) t.c0 = w0 / (nd * (float)((int64_t)(S - 1) * hw));
  if (nd && wxy > 0.f) {
    t.c1 = wxy / (nd * (float)((int64_t)S * (Ho - 1) * Wo));
    t.c2 = wxy / (nd * (float)((int64_t)S * Ho * (Wo - 1)));
  }
  return t;
}
// Loss terms (into lacc) and gradient of element i of slice s.  tv(dim) yields each weighted dimension's
// neighbours: per dimension the loss term of the diff to the next element, the gradient from the diffs on
// both sides.
template <int KIND, typename TV>
__device__ __forceinline__ void soft_element(const float* obj, float* grad, int64_t i, int s, int S, const SoftTerms& t,
                                             float2 here, double& lacc, TV tv) {
  constexpr bool amp_terms = KIND == 0;
  const float ph = here.x, amp = here.y;
  float gph = 0.f, gamp = 0.f;
  auto dim = [&](float cw, bool has_lo, auto lo, bool has_hi, auto hi) {
    if (cw == 0.f) return;
    if (has_hi) {
      const float2 q = hi();
      const float d = q.x - ph;
      lacc += (double)(cw * fabsf(d));
      gph -= cw * sgnf(d);
      if (amp_terms) {
        const float da = q.y - amp;
        lacc += (double)(cw * fabsf(da));
        gamp -= cw * sgnf(da);
      }
    }
    if (has_lo) {
      const float2 q = lo();
      gph += cw * sgnf(ph - q.x);
      if (amp_terms) gamp += cw * sgnf(amp - q.y);
    }
  };
  tv(dim);
  if (t.surf && (s == 0 || s == S - 1)) {
    if (KIND == 2) {
      lacc += (double)(t.wsurf * fabsf(ph) * t.inv_hw);
      gph += t.wsurf * sgnf(ph) * t.inv_hw;
    } else {
      const float m = s == 0 ? t.m0 : t.m1, sgm = s == 0 ? t.sg0 : t.sg1;
      const float u = fabsf(ph) - m;
      lacc += (double)(t.wsurf * fabsf(u) * t.inv_hw);
      gph += t.wsurf * (sgnf(u) - sgm) * t.inv_hw * sgnf(ph);
      if (amp_terms) {
        lacc += (double)(t.wsurf * (1.0f - amp) * t.inv_hw);
        gamp -= t.wsurf * t.inv_hw;
      }
    }
  }
  if (KIND == 2) {
    grad[i] = gph;
  } else {
    const float2 o = reinterpret_cast<const float2*>(obj)[i];
    float2 gz = make_float2(0.f, 0.f);
    if (amp != 0.f) {  // G = g_amp z / |z| + i g_phase z / |z|^2 (zero at a zero pixel)
      const float inv = 1.0f / amp;
      gz.x = gamp * o.x * inv - gph * o.y * inv * inv;
      gz.y = gamp * o.y * inv + gph * o.x * inv * inv;
    }
    reinterpret_cast<float2*>(grad)[i] = gz;
  }
}

// One thread per element, the stencil's values read (and for complex objects evaluated, up to seven times)
// where they are needed.
template <int KIND>
__global__ void __launch_bounds__(kThreads) soft_direct_kernel(const float* __restrict__ obj, int S, int Ho, int Wo,
                                                               float wz, float wxy, float wsurf,
                                                               float* __restrict__ grad, double* work) {
  __shared__ double red[32];
  const int64_t hw = (int64_t)Ho * Wo, n = (int64_t)S * hw;
  const SoftTerms t = soft_terms<KIND>(S, Ho, Wo, wz, wxy, wsurf, work);
  double lacc = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int s = (int)(i / hw);
    const int64_t p = i % hw;
    const int r = (int)(p / Wo), c = (int)(p % Wo);
    auto at = [&](int64_t k) {
      return [&obj, k] {
        float ph, amp;
        values_at<KIND>(obj, k, ph, amp);
        return make_float2(ph, amp);
      };
    };
    soft_element<KIND>(obj, grad, i, s, S, t, at(i)(), lacc, [&](auto dim) {
      dim(t.c0, s > 0, at(i - hw), s < S - 1, at(i + hw));
      dim(t.c1, r > 0, at(i - Wo), r < Ho - 1, at(i + Wo));
      dim(t.c2, c > 0, at(i - 1), c < Wo - 1, at(i + 1));
    });
  }
  const double sum = block_sum_d(lacc, red);
  if (threadIdx.x == 0) work[blockIdx.x] = sum;
}

// Complex objects of large planes: a block marches a 32 x 8 tile through `run` slices.  The phase and
// amplitude of the tile and its one-element halo are evaluated once per slice into shared memory (two
// slices alternate), the slice before stays in registers.  Bound by atan2 and hypot (1.33 per element and
// slice against up to 7): 8 x 510 x 516 takes 80 us, 107 element by element.
constexpr int kSoftX = 32, kSoftY = 8;
inline int soft_tiles(int Ho, int Wo) { return ((Wo + kSoftX - 1) / kSoftX) * ((Ho + kSoftY - 1) / kSoftY); }
template <int KIND>
__global__ void __launch_bounds__(kThreads) soft_march_kernel(const float* __restrict__ obj, int S, int Ho, int Wo,
                                                              float wz, float wxy, float wsurf,
                                                              float* __restrict__ grad, double* work, int run) {
  static_assert(kThreads == kSoftX * kSoftY, "one thread per tile element");
  constexpr int PX = kSoftX + 2, PY = kSoftY + 2;
  __shared__ double red[32];
  __shared__ float2 val[2][PY][PX];  // (phase, amplitude)
  const int64_t hw = (int64_t)Ho * Wo;
  const SoftTerms t = soft_terms<KIND>(S, Ho, Wo, wz, wxy, wsurf, work);
  const int tx = threadIdx.x % kSoftX, ty = threadIdx.x / kSoftX;
  const int tiles_x = (Wo + kSoftX - 1) / kSoftX, tiles = tiles_x * ((Ho + kSoftY - 1) / kSoftY);
  const int tasks = tiles * ((S + run - 1) / run);
  double lacc = 0.0;
  for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
    const int tile = task % tiles, s0 = task / tiles * run, s1 = min(S, s0 + run);
    const int rb = tile / tiles_x * kSoftY, cb = tile % tiles_x * kSoftX;
    const int r = rb + ty, c = cb + tx;
    const bool on = r < Ho && c < Wo;
    auto value = [&](int64_t k) {
      float ph, amp;
      values_at<KIND>(obj, k, ph, amp);
      return make_float2(ph, amp);
    };
    auto fill = [&](int s) {
      float2(*v)[PX] = val[s & 1];
      for (int k = threadIdx.x; k < PY * PX; k += kThreads) {
        const int y = k / PX, x = k % PX, rr = rb + y - 1, cc = cb + x - 1;
        if (rr < 0 || rr >= Ho || cc < 0 || cc >= Wo) continue;
        if ((y == 0 || y == PY - 1) && (x == 0 || x == PX - 1)) continue;  // corners are not read
        v[y][x] = value(s * hw + (int64_t)rr * Wo + cc);
      }
    };
    const int64_t own = (int64_t)r * Wo + c;
    __syncthreads();  // the last task's values are read
    fill(s0);
    float2 before = make_float2(0.f, 0.f);
    if (on && s0 > 0) before = value((s0 - 1) * hw + own);
    for (int s = s0; s < s1; ++s) {
      __syncthreads();  // slice s is in place and slice s - 1 no longer read
      if (s + 1 < s1) fill(s + 1);
      const float2(*v)[PX] = val[s & 1];
      const float2 here = v[ty + 1][tx + 1];
      float2 after = here;
      if (s + 1 < s1) {  // the own element of the next slice: this thread may not have filled it
        __syncthreads();
        after = val[(s + 1) & 1][ty + 1][tx + 1];
      } else if (on && s + 1 < S) {
        after = value((s + 1) * hw + own);
      }
      if (on)
        soft_element<KIND>(obj, grad, s * hw + own, s, S, t, here, lacc, [&](auto dim) {
          dim(t.c0, s > 0, [&] { return before; }, s < S - 1, [&] { return after; });
          dim(t.c1, r > 0, [&] { return v[ty][tx + 1]; }, r < Ho - 1, [&] { return v[ty + 2][tx + 1]; });
          dim(t.c2, c > 0, [&] { return v[ty + 1][tx]; }, c < Wo - 1, [&] { return v[ty + 1][tx + 2]; });
        });
      before = here;
    }
  }
  const double sum = block_sum_d(lacc, red);
  if (threadIdx.x == 0) work[blockIdx.x] = sum;
}

__global__ void loss_from_partials_kernel(const double* __restrict__ part, float* __restrict__ out) {
  const double t = partials_sum(part, kBlocks);
  if (threadIdx.x == 0) *out = (float)t;
}

int check(const char* what);
int grid_for(int64_t n);

// Dynamic shared memory that a kernel may be launched with: one bound for all of its calls.  The
// attribute belongs to the device, so a bound of each call's own size could be lowered by another
// host thread before the launch.
template <typename K>
int allow_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess
             ? PTYCHO_OK
             : check("shared memory bound");
}

// ---------------------------------------------------------------- Butterworth filter
// object_models.py:481-520: per slice, mean removed, ifft2(fft2(x) env), mean added back.
// The mean is the DC term, so the filter is ifft2(fft2(x - c) env') + c with env' = env but 1
// at DC, for any constant c; its VJP (P g - mean(P g) + mean(g)) is the same filter.  c is a
// sampled mean (256 values of the slice): it only keeps the transform's rounding relative to
// the variation of x instead of its offset.
//
// Three passes of line transforms of any length (line_fft.cuh): rows forward, columns forward
// + envelope + columns inverse in one pass, rows inverse.  Each pass reads and writes the
// object once (17 MB at 8 x 510 x 516, L2-resident), 55 to 60 us each; bound by the chain of stages: the 27
// of 64 warps wait at the stages' barriers (3.9 cycles per issued instruction in the row passes, 1.7 in the
// columns) and for their shared and twiddle loads (3.9 and 3.6), with 50 to 58 % of the issue slots and
// 32 to 41 % of the load/store data pipe used.  At 8 x 510 x 516 (factors 17 and 43 among the radices) the filter took 3.4 ms as
// four direct n^2 line transforms with transposes, mean and envelope passes in between.
constexpr int kLineThreads = 512;

// c of a slice: the mean of 256 of its values (fixed-order sums, every thread).  Value k lies in
// row k H / 256 and, for sides that a stride would alias with (512 x 512 at hw / 256 is column 0
// alone), in the column that k golden-ratio turns reach: rows and columns both covered evenly, so c
// is within about a sixteenth of the slice's deviation from its mean whatever its structure.
template <bool REAL>
__device__ float2 sampled_mean(const float* in, int H, int W, float2* red) {
  const unsigned k = threadIdx.x;
  float2 v = make_float2(0.f, 0.f);
  if (k < 256) {
    const unsigned i = (k * H >> 8) * W + (((k * 40503 & 0xffff) * W) >> 16);  // sides <= 6144; 40503 / 2^16 = 0.618
    v = REAL ? make_float2(in[i], 0.f) : reinterpret_cast<const float2*>(in)[i];
  }
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  __syncthreads();  // red is free
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float2 t = make_float2(0.f, 0.f);
  for (int w = 0; w < 8; ++w) t = make_float2(t.x + red[w].x, t.y + red[w].y);
  const float inv = 1.0f / 256.0f;
  return make_float2(t.x * inv, t.y * inv);
}

// Rows: a = row transforms of (in - c) (INV = false; c kept in base), or out = inverse row
// transforms of a, plus c (INV = true).
template <bool REAL, bool INV>
__global__ void __launch_bounds__(kLineThreads, 2)
    butter_rows_kernel(const float* __restrict__ in, float2* __restrict__ a, float* __restrict__ out,
                       float2* __restrict__ base, const qb::LinePlan p, int S, int H, int lg, int LP) {
  extern __shared__ float2 sh[];
  __shared__ float2 red[kLineThreads / 32];
  const int n = p.n, L = 1 << lg;
  float2 *x = sh, *y = sh + n * LP, *tw = y + n * LP;
  qb::line_twiddles(tw, n);
  const int per = (H + L - 1) / L;  // line groups per slice
  const int64_t hw = (int64_t)H * n;
  for (int g = blockIdx.x; g < S * per; g += gridDim.x) {
    const int s = g / per, r0 = (g - s * per) * L, nl = min(L, H - r0);
    float2 c;
    if (INV) {
      c = base[s];
    } else {
      c = sampled_mean<REAL>(in + s * hw * (REAL ? 1 : 2), H, n, red);
      if (r0 == 0 && threadIdx.x == 0) base[s] = c;
    }
    const int64_t off = s * hw + (int64_t)r0 * n;
    for (int l = 0; l < L; ++l)
      for (int e = threadIdx.x; e < n; e += kLineThreads) {
        float2 v = make_float2(0.f, 0.f);
        if (l < nl) {
          const int64_t i = off + (int64_t)l * n + e;
          if (INV) {
            v = a[i];
          } else {
            v = REAL ? make_float2(in[i], 0.f) : reinterpret_cast<const float2*>(in)[i];
            v = make_float2(v.x - c.x, v.y - c.y);
          }
        }
        x[e * LP + l] = v;
      }
    __syncthreads();
    const float2* r = qb::line_dft<INV>(x, y, tw, p, lg, LP);
    for (int l = 0; l < nl; ++l)
      for (int e = threadIdx.x; e < n; e += kLineThreads) {
        const int64_t i = off + (int64_t)l * n + e;
        const float2 v = r[e * LP + l];
        if (!INV)
          a[i] = v;
        else if (REAL)
          out[i] = v.x + c.x;
        else
          reinterpret_cast<float2*>(out)[i] = make_float2(v.x + c.x, v.y + c.y);
      }
    __syncthreads();
  }
}

// Columns of the row spectra, in place: forward, times the envelope (1 at DC) and the
// normalisation, inverse.
__global__ void __launch_bounds__(kLineThreads, 2)
    butter_cols_kernel(float2* __restrict__ a, const float* __restrict__ env, const qb::LinePlan p, int S, int W,
                       int lg, int LP) {
  extern __shared__ float2 sh[];
  const int n = p.n, L = 1 << lg;
  float2 *x = sh, *y = sh + n * LP, *tw = y + n * LP;
  qb::line_twiddles(tw, n);
  const int per = (W + L - 1) / L;
  const float scale = (float)(1.0 / ((double)n * (double)W));
  for (int g = blockIdx.x; g < S * per; g += gridDim.x) {
    const int s = g / per, c0 = (g - s * per) * L;
    float2* as = a + (int64_t)s * n * W + c0;
    for (int t = threadIdx.x; t < n << lg; t += kLineThreads) {
      const int l = t & (L - 1), e = t >> lg;
      x[e * LP + l] = c0 + l < W ? as[(int64_t)e * W + l] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    float2* r = qb::line_dft<false>(x, y, tw, p, lg, LP);
    for (int t = threadIdx.x; t < n << lg; t += kLineThreads) {
      const int l = t & (L - 1), e = t >> lg;
      if (c0 + l >= W) continue;
      const float w = (e == 0 && c0 + l == 0 ? 1.0f : env[(int64_t)e * W + c0 + l]) * scale;
      float2& v = r[e * LP + l];
      v = make_float2(v.x * w, v.y * w);
    }
    __syncthreads();
    const float2* o = qb::line_dft<true>(r, r == x ? y : x, tw, p, lg, LP);
    for (int t = threadIdx.x; t < n << lg; t += kLineThreads) {
      const int l = t & (L - 1), e = t >> lg;
      if (c0 + l < W) as[(int64_t)e * W + l] = o[e * LP + l];
    }
    __syncthreads();
  }
}

// out = ifft2(env' fft2(in - c)) + c of S planes H x W; a: S H W complex scratch, base: S
template <bool REAL>
int butterworth(const float* in, float* out, int S, int H, int W, const float* env, float2* a, float2* base,
                cudaStream_t st) {
  const qb::LinePlan pr = qb::line_plan(W), pc = qb::line_plan(H);
  const int lr = qb::line_log2(W), lc = qb::line_log2(H);
  const size_t sr = qb::line_smem(W, lr), sc = qb::line_smem(H, lc);
  if (int rc = allow_smem(butter_rows_kernel<REAL, false>, qb::kLineSmem)) return rc;
  if (int rc = allow_smem(butter_rows_kernel<REAL, true>, qb::kLineSmem)) return rc;
  if (int rc = allow_smem(butter_cols_kernel, qb::kLineSmem)) return rc;
  // two blocks per SM, evened out over the rounds
  auto grid = [](int64_t groups) {
    const int64_t rounds = (groups + kBlocks - 1) / kBlocks;
    return (int)((groups + rounds - 1) / rounds);
  };
  const int gr = grid((int64_t)S * ((H + (1 << lr) - 1) >> lr)), gc = grid((int64_t)S * ((W + (1 << lc) - 1) >> lc));
  butter_rows_kernel<REAL, false><<<gr, kLineThreads, sr, st>>>(in, a, nullptr, base, pr, S, H, lr, qb::line_pitch(lr));
  butter_cols_kernel<<<gc, kLineThreads, sc, st>>>(a, env, pc, S, W, lc, qb::line_pitch(lc));
  butter_rows_kernel<REAL, true><<<gr, kLineThreads, sr, st>>>(nullptr, a, out, base, pr, S, H, lr, qb::line_pitch(lr));
  return check("butterworth");
}

int check(const char* what) {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PTYCHO_OK : qb_record_error(PTYCHO_ERR_CUDA, what);
}

int grid_for(int64_t n) {
  const int64_t g = (n + kThreads - 1) / kThreads;
  return (int)(g < kBlocks ? (g < 1 ? 1 : g) : kBlocks);
}

}  // namespace

extern "C" {

int ptycho_obj_constraint_work_elems(void) { return 5 * kBlocks; }

int ptycho_probe_overlap(const float* intensity, int n, const float* positions, int npos, int Ho, int Wo, float* out,
                         void* stream) {
  if (!intensity || !positions || !out || n < 1 || npos < 0 || Ho < 1 || Wo < 1)
    return qb_record_error(PTYCHO_ERR_INVALID, "probe_overlap: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(out, 0, sizeof(float) * (size_t)Ho * Wo, st) != cudaSuccess)
    return qb_record_error(PTYCHO_ERR_CUDA, "probe_overlap: memset");
  if (npos == 0) return PTYCHO_OK;
  probe_overlap_kernel<<<4 * kBlocks, kThreads, 0, st>>>(intensity, n, positions, npos, Ho, Wo, out);
  return check("probe_overlap_kernel");
}

int ptycho_obj_constrain_fov(const void* obj, const float* mask, int64_t hw, void* out, int64_t count, int pure,
                             double* work, int nwork, void* stream) {
  if (!obj || !mask || !out || !work || count < 1 || hw < 1 || count % hw || nwork < 5 * kBlocks)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_constrain_fov: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float2* o = static_cast<const float2*>(obj);
  angle_partials_kernel<<<kBlocks, kThreads, 0, st>>>(o, count, work);
  if (pure)
    fov_apply_kernel<true><<<kBlocks, kThreads, 0, st>>>(o, mask, hw, static_cast<float2*>(out), count, work);
  else
    fov_apply_kernel<false><<<kBlocks, kThreads, 0, st>>>(o, mask, hw, static_cast<float2*>(out), count, work);
  return check("fov_apply_kernel");
}

int ptycho_obj_constrain_fov_vjp(const void* obj, const float* mask, int64_t hw, const void* grad_c, void* grad_raw,
                                 int64_t count, int pure, double* work, int nwork, void* stream) {
  if (!obj || !mask || !grad_c || !grad_raw || !work || count < 1 || hw < 1 || count % hw || nwork < 5 * kBlocks)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_constrain_fov_vjp: bad arguments");
  if (grad_raw == obj || grad_raw == grad_c)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_constrain_fov_vjp: grad_raw aliases an input");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float2* o = static_cast<const float2*>(obj);
  const float2* g = static_cast<const float2*>(grad_c);
  angle_partials_kernel<<<kBlocks, kThreads, 0, st>>>(o, count, work);
  if (pure) {
    fov_vjp_partials_kernel<true><<<kBlocks, kThreads, 0, st>>>(o, mask, hw, g, count, work, work + kBlocks);
    fov_vjp_apply_kernel<true><<<kBlocks, kThreads, 0, st>>>(o, mask, hw, g, static_cast<float2*>(grad_raw), count,
                                                             work, work + kBlocks);
  } else {
    fov_vjp_partials_kernel<false><<<kBlocks, kThreads, 0, st>>>(o, mask, hw, g, count, work, work + kBlocks);
    fov_vjp_apply_kernel<false><<<kBlocks, kThreads, 0, st>>>(o, mask, hw, g, static_cast<float2*>(grad_raw), count,
                                                              work, work + kBlocks);
  }
  return check("fov_vjp_apply_kernel");
}

int ptycho_obj_potential_base(const float* v, const float* baseline_mask, const float* apply_mask, int64_t hw,
                              float* out, int64_t count, int positivity, int fix_baseline, float factor,
                              double* work, int nwork, void* stream) {
  if (!v || !out || !work || count < 1 || hw < 1 || count % hw || nwork < 5 * kBlocks)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_potential_base: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (fix_baseline) {
    if (baseline_mask) mask_max_kernel<<<kBlocks, kThreads, 0, st>>>(baseline_mask, hw, work);
    background_stats_kernel<<<kBlocks, kThreads, 0, st>>>(v, baseline_mask, hw, count, work);
  }
  potential_base_kernel<<<kBlocks, kThreads, 0, st>>>(v, apply_mask, hw, out, count, positivity, fix_baseline, factor,
                                                      work);
  return check("potential_base_kernel");
}

int ptycho_obj_potential_base_vjp(const float* v, const float* baseline_mask, const float* apply_mask, int64_t hw,
                                  const float* grad_out, float* grad_v, int64_t count, int positivity,
                                  int fix_baseline, float factor, double* work, int nwork, void* stream) {
  if (!v || !grad_out || !grad_v || !work || count < 1 || hw < 1 || count % hw || nwork < 5 * kBlocks)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_potential_base_vjp: bad arguments");
  if (grad_v == v) return qb_record_error(PTYCHO_ERR_INVALID, "obj_potential_base_vjp: grad_v aliases v");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (fix_baseline) {
    if (baseline_mask) mask_max_kernel<<<kBlocks, kThreads, 0, st>>>(baseline_mask, hw, work);
    background_stats_kernel<<<kBlocks, kThreads, 0, st>>>(v, baseline_mask, hw, count, work);
  }
  potential_base_vjp_kernel<<<kBlocks, kThreads, 0, st>>>(v, apply_mask, hw, grad_out, grad_v, count, positivity,
                                                          fix_baseline, factor, work);
  return check("potential_base_vjp_kernel");
}

int ptycho_phase_exp(const float* v, void* out, int64_t count, void* stream) {
  if (!v || !out || count < 0) return qb_record_error(PTYCHO_ERR_INVALID, "phase_exp: bad arguments");
  if (count == 0) return PTYCHO_OK;
  phase_exp_kernel<<<grid_for(count), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(v, static_cast<float2*>(out),
                                                                                        count);
  return check("phase_exp_kernel");
}

int ptycho_phase_exp_vjp(const float* v, const void* grad_t, float* grad_v, int64_t count, void* stream) {
  if (!v || !grad_t || !grad_v || count < 0) return qb_record_error(PTYCHO_ERR_INVALID, "phase_exp_vjp: bad arguments");
  if (grad_v == v) return qb_record_error(PTYCHO_ERR_INVALID, "phase_exp_vjp: grad_v aliases v");
  if (count == 0) return PTYCHO_OK;
  phase_exp_vjp_kernel<<<grid_for(count), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      v, static_cast<const float2*>(grad_t), grad_v, count);
  return check("phase_exp_vjp_kernel");
}

int ptycho_obj_blur(const void* in, void* out, void* tmp, int S, int Ho, int Wo, int is_complex, const float* taps,
                    int ntaps, void* stream) {
  if (!in || !out || !tmp || !taps || S < 1 || Ho < 1 || Wo < 1 || ntaps < 1 || ntaps > 255 || ntaps % 2 == 0)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_blur: bad arguments (odd tap count <= 255)");
  if (tmp == in || tmp == out) return qb_record_error(PTYCHO_ERR_INVALID, "obj_blur: tmp aliases in or out");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int K = is_complex ? 2 : 1;
  if (ntaps / 2 <= kBlurHalo && (int64_t)S * Ho * Wo >= kBlurLeast && S <= 65535 && in != out) {
    const int side = kBlurTile + ntaps - 1;
    const size_t smem = sizeof(float) * (size_t)(side + kBlurTile) * side * K;
    const dim3 grid((Wo + kBlurTile - 1) / kBlurTile, (Ho + kBlurTile - 1) / kBlurTile, S);
    if (grid.y <= 65535) {
      if (is_complex) {
        if (int rc = allow_smem(blur_tile_kernel<2>, kBlurSmem)) return rc;
        blur_tile_kernel<2><<<grid, kThreads, smem, st>>>(static_cast<const float*>(in), static_cast<float*>(out), Ho,
                                                          Wo, taps, ntaps);
      } else {
        blur_tile_kernel<1><<<grid, kThreads, smem, st>>>(static_cast<const float*>(in), static_cast<float*>(out), Ho,
                                                          Wo, taps, ntaps);
      }
      return check("blur_tile_kernel");
    }
  }
  blur_pass_kernel<0><<<4 * kBlocks, kThreads, 0, st>>>(static_cast<const float*>(in), static_cast<float*>(tmp), S, Ho,
                                                        Wo, K, taps, ntaps);
  blur_pass_kernel<1><<<4 * kBlocks, kThreads, 0, st>>>(static_cast<const float*>(tmp), static_cast<float*>(out), S,
                                                        Ho, Wo, K, taps, ntaps);
  return check("blur_pass_kernel");
}

int ptycho_obj_slice_mean(const void* in, void* out, int S, int64_t hw, int is_complex, void* stream) {
  if (!in || !out || S < 1 || hw < 1) return qb_record_error(PTYCHO_ERR_INVALID, "obj_slice_mean: bad arguments");
  const int64_t plane = hw * (is_complex ? 2 : 1);
  slice_mean_kernel<<<grid_for(plane), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float*>(in), static_cast<float*>(out), S, plane);
  return check("slice_mean_kernel");
}

int ptycho_obj_butterworth(const void* in, void* out, int S, int Ho, int Wo, int is_real, const float* env, void* tmp,
                           void* means, void* stream) {
  if (!in || !out || !env || !tmp || !means || S < 1 || Ho < 1 || Wo < 1 || Ho > 6144 || Wo > 6144)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_butterworth: bad arguments (object sides <= 6144)");
  if (tmp == in || tmp == out) return qb_record_error(PTYCHO_ERR_INVALID, "obj_butterworth: tmp aliases in or out");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float2* a = static_cast<float2*>(tmp);
  float2* base = static_cast<float2*>(means);
  const float* x = static_cast<const float*>(in);
  float* o = static_cast<float*>(out);
  return is_real ? butterworth<true>(x, o, S, Ho, Wo, env, a, base, st)
                 : butterworth<false>(x, o, S, Ho, Wo, env, a, base, st);
}

int ptycho_obj_butterworth_vjp(const void* grad_out, void* grad_in, int S, int Ho, int Wo, int is_real,
                               const float* env, void* tmp, void* means, void* stream) {
  if (!grad_out || !grad_in || !env || !tmp || !means || S < 1 || Ho < 1 || Wo < 1 || Ho > 6144 || Wo > 6144)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_butterworth_vjp: bad arguments (object sides <= 6144)");
  if (tmp == grad_out || tmp == grad_in)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_butterworth_vjp: tmp aliases a gradient");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float2* a = static_cast<float2*>(tmp);
  float2* base = static_cast<float2*>(means);
  const float* x = static_cast<const float*>(grad_out);
  float* o = static_cast<float*>(grad_in);
  return is_real ? butterworth<true>(x, o, S, Ho, Wo, env, a, base, st)
                 : butterworth<false>(x, o, S, Ho, Wo, env, a, base, st);
}

}  // extern "C"

namespace {
// Complex objects march where at least three quarters of the tiles' elements exist and the tiles, in runs of
// four slices, fill the blocks; the runs are then as long as leaves four tasks per block.  Measured (march
// against element by element, amplitude and phase): 200 x 128 x 128 115 us against 150 (345 as one run),
// 64 x 200 x 200 100 against 127, 8 x 256 x 256 39 against 44, 1 x 510 x 516 16.5 both, 8 x 128 x 128 (128
// tasks) 30 against 29, 1 x 3000 x 40 (62 % of the tiles) 14.5 against 12.5.  Potentials have nothing to
// evaluate: 8 x 510 x 516 29 us element by element, 39 marching.
template <int KIND>
void soft_launch(const float* o, int S, int Ho, int Wo, float wz, float wxy, float wsurf, float* g, double* work,
                 cudaStream_t st) {
  if constexpr (KIND != 2) {
    const int64_t tiles = soft_tiles(Ho, Wo);
    if ((int64_t)Ho * Wo * 4 >= tiles * kThreads * 3 && tiles * ((S + 3) / 4) >= kBlocks) {
      const int64_t parts = (4 * kBlocks + tiles - 1) / tiles;  // of the slices
      const int run = parts * 4 >= S ? 4 : (int)((S + parts - 1) / parts);
      soft_march_kernel<KIND><<<kBlocks, kThreads, 0, st>>>(o, S, Ho, Wo, wz, wxy, wsurf, g, work, run);
      return;
    }
  }
  soft_direct_kernel<KIND><<<kBlocks, kThreads, 0, st>>>(o, S, Ho, Wo, wz, wxy, wsurf, g, work);
}
}  // namespace

extern "C" {

int ptycho_obj_soft_loss(const void* obj, int S, int Ho, int Wo, int kind, float tv_weight_z, float tv_weight_xy,
                         float surface_zero_weight, double* work, int nwork, float* loss, void* grad, void* stream) {
  if (!obj || !work || !loss || !grad || S < 1 || Ho < 2 || Wo < 2 || kind < 0 || kind > 2 || nwork < 5 * kBlocks)
    return qb_record_error(PTYCHO_ERR_INVALID, "obj_soft_loss: bad arguments");
  if (grad == obj) return qb_record_error(PTYCHO_ERR_INVALID, "obj_soft_loss: grad aliases obj");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const float* o = static_cast<const float*>(obj);
  float* g = static_cast<float*>(grad);
  const int64_t hw = (int64_t)Ho * Wo;
  const bool surf = surface_zero_weight > 0.f && S >= 3;
  if (kind == 0) {
    if (surf) {
      surface_abs_phase_kernel<0><<<kBlocks, kThreads, 0, st>>>(o, S, hw, work);
      surface_sign_kernel<0><<<kBlocks, kThreads, 0, st>>>(o, S, hw, work);
    }
    soft_launch<0>(o, S, Ho, Wo, tv_weight_z, tv_weight_xy, surface_zero_weight, g, work, st);
  } else if (kind == 1) {
    if (surf) {
      surface_abs_phase_kernel<1><<<kBlocks, kThreads, 0, st>>>(o, S, hw, work);
      surface_sign_kernel<1><<<kBlocks, kThreads, 0, st>>>(o, S, hw, work);
    }
    soft_launch<1>(o, S, Ho, Wo, tv_weight_z, tv_weight_xy, surface_zero_weight, g, work, st);
  } else {
    soft_launch<2>(o, S, Ho, Wo, tv_weight_z, tv_weight_xy, surface_zero_weight, g, work, st);
  }
  loss_from_partials_kernel<<<1, kThreads, 0, st>>>(work, loss);
  return check("soft_loss_kernel");
}

}  // extern "C"
