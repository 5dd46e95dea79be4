// Discrete Fourier transforms of any length along lines held in shared memory (sm_100a),
// for the object-sized transforms of the Butterworth filter.
//
// L = 2^lg lines of n complex values are interleaved (element e of line l at e LP + l, LP odd so
// that both the element-contiguous fill and the line-contiguous stages spread over the
// banks) in two buffers.  n is factored into radices: 8, 4, 2, 3, 5 as register butterflies
// (Stockham order, no reordering pass) and any other prime p by its defining sum over
// (p - 1) / 2 pairs: with s_e = x_e + x_{p-e} and d_e = x_e - x_{p-e},
//   X_k, X_{p-k} = x_0 + sum_e s_e cos(2 pi e k / p) -+ i sum_e d_e sin(2 pi e k / p),
// four real products per pair of inputs and pair of outputs, a quarter of the direct sum.
// The largest such prime goes first, where no twiddles are due.  Cost per line: n (sum of
// the primes) / 2 + O(n log n) instead of n^2 complex products.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fft_engine.cuh"

namespace qb {

constexpr int kLineMaxFactors = 16;
struct LinePlan {
  int n;                        // length
  int nf;                       // number of radices
  int radix[kLineMaxFactors];   // in stage order
};

// Radices of n: primes without a butterfly first (largest first), then 5, 3, 2, 4, 8.
inline LinePlan line_plan(int n) {
  LinePlan p;
  p.n = n;
  p.nf = 0;
  int odd[kLineMaxFactors], no = 0, m = n, e2 = 0, e3 = 0, e5 = 0;
  while (m % 2 == 0) m /= 2, ++e2;
  while (m % 3 == 0) m /= 3, ++e3;
  while (m % 5 == 0) m /= 5, ++e5;
  for (int d = 7; m > 1; d += 2) {
    if ((int64_t)d * d > m) d = m;
    while (m % d == 0) m /= d, odd[no++] = d;
  }
  for (int i = no - 1; i >= 0; --i) p.radix[p.nf++] = odd[i];  // found in rising order
  for (int i = 0; i < e5; ++i) p.radix[p.nf++] = 5;
  for (int i = 0; i < e3; ++i) p.radix[p.nf++] = 3;
  for (; e2 >= 3; e2 -= 3) p.radix[p.nf++] = 8;
  if (e2 == 2) p.radix[p.nf++] = 4;
  if (e2 == 1) p.radix[p.nf++] = 2;
  return p;
}

// w_n^k = exp(-2 pi i k / n), k < n, in float64 rounded to float32
__device__ __forceinline__ void line_twiddles(float2* tw, int n) {
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    double s, c;
    sincospi(-2.0 * (double)k / (double)n, &s, &c);
    tw[k] = make_float2((float)c, (float)s);
  }
}

template <bool INV>
__device__ __forceinline__ void dft5(float2 (&v)[5]) {
  const float c1 = 0.30901699437494745f, c2 = -0.8090169943749475f;  // cos(2 pi / 5), cos(4 pi / 5)
  const float s1 = 0.9510565162951535f, s2 = 0.5877852522924731f;    // sin(2 pi / 5), sin(4 pi / 5)
  const float2 a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]), a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
  const float2 p1 = make_float2(fmaf(c2, a2.x, fmaf(c1, a1.x, v[0].x)), fmaf(c2, a2.y, fmaf(c1, a1.y, v[0].y)));
  const float2 p2 = make_float2(fmaf(c1, a2.x, fmaf(c2, a1.x, v[0].x)), fmaf(c1, a2.y, fmaf(c2, a1.y, v[0].y)));
  float2 q1 = make_float2(fmaf(s2, b2.x, s1 * b1.x), fmaf(s2, b2.y, s1 * b1.y));
  float2 q2 = make_float2(fmaf(-s1, b2.x, s2 * b1.x), fmaf(-s1, b2.y, s2 * b1.y));
  if (INV) {
    q1 = make_float2(-q1.x, -q1.y);
    q2 = make_float2(-q2.x, -q2.y);
  }
  v[0] = cadd(v[0], cadd(a1, a2));  // X_k = p - i q, X_{5-k} = p + i q
  v[1] = make_float2(p1.x + q1.y, p1.y - q1.x);
  v[4] = make_float2(p1.x - q1.y, p1.y + q1.x);
  v[2] = make_float2(p2.x + q2.y, p2.y - q2.x);
  v[3] = make_float2(p2.x - q2.y, p2.y + q2.x);
}

// One Stockham stage of radix R: ls = product of the radices before it.
template <int R, bool INV>
__device__ __forceinline__ void line_stage(const float2* x, float2* y, const float2* tw, int n, int ls, int lg, int LP) {
  const int L = 1 << lg;
  const int m = n / R;            // butterflies per line
  const int step = n / (ls * R);  // twiddle step
  for (int t = threadIdx.x; t < m * L; t += blockDim.x) {
    const int l = t & (L - 1), j = t >> lg;
    const int k = j % ls;
    float2 v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      v[q] = x[(j + q * m) * LP + l];
      if (q > 0 && ls > 1) {
        const float2 w = tw[q * k * step];  // q k step < R ls n / (ls R) = n
        v[q] = INV ? cmulc(v[q], w) : cmul(v[q], w);
      }
    }
    if constexpr (R == 3)
      dft3<INV>(v[0], v[1], v[2]);
    else if constexpr (R == 5)
      dft5<INV>(v);
    else
      dft_reg<R, INV>(v);
    float2* o = y + ((j - k) * R + k) * LP + l;
#pragma unroll
    for (int q = 0; q < R; ++q) o[q * ls * LP] = v[q];
  }
}

// A stage of any odd prime p.  RK output pairs per task keep RK + 2 shared loads for 4 RK
// products.
template <bool INV>
__device__ __forceinline__ void line_stage_prime(float2* x, float2* y, const float2* tw, int n, int p, int ls, int lg,
                                                 int LP) {
  constexpr int RK = 4;
  const int L = 1 << lg;
  const int m = n / p, h = (p - 1) / 2, kg = (h + RK - 1) / RK;
  if (ls > 1) {  // twiddles in place
    const int step = n / (ls * p);
    for (int t = threadIdx.x; t < (n - m) * L; t += blockDim.x) {
      const int l = t & (L - 1), e = m + (t >> lg);
      const int q = e / m, k = (e % m) % ls;
      const float2 w = tw[q * k * step];
      float2& v = x[e * LP + l];
      v = INV ? cmulc(v, w) : cmul(v, w);
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < m * kg * L; t += blockDim.x) {
    const int l = t & (L - 1), u = t >> lg, j = u / kg, g = u - j * kg;
    const int k0 = j % ls;
    const float2* xi = x + j * LP + l;
    const int es = m * LP;  // between inputs e and e + 1
    float2 A[RK], Bq[RK], x0 = xi[0], tot = x0;
    int idx[RK], inc[RK];
#pragma unroll
    for (int r = 0; r < RK; ++r) {
      A[r] = x0;
      Bq[r] = make_float2(0.f, 0.f);
      const int k = min(g * RK + r + 1, h);
      inc[r] = idx[r] = k * m;  // exponent e k n / p modulo n
    }
    for (int e = 1; e <= h; ++e) {
      const float2 a = xi[e * es], b = xi[(p - e) * es];
      const float2 s = cadd(a, b), d = csub(a, b);
      tot = cadd(tot, s);
#pragma unroll
      for (int r = 0; r < RK; ++r) {
        const float2 w = tw[idx[r]];  // (cos, -sin)
        A[r] = make_float2(fmaf(s.x, w.x, A[r].x), fmaf(s.y, w.x, A[r].y));
        Bq[r] = make_float2(fmaf(d.x, w.y, Bq[r].x), fmaf(d.y, w.y, Bq[r].y));
        idx[r] += inc[r];
        if (idx[r] >= n) idx[r] -= n;
      }
    }
    float2* o = y + ((j - k0) * p + k0) * LP + l;
    const int os = ls * LP;
    if (g == 0) o[0] = tot;
#pragma unroll
    for (int r = 0; r < RK; ++r) {
      const int k = g * RK + r + 1;
      if (k > h) break;
      const float2 q = INV ? make_float2(-Bq[r].x, -Bq[r].y) : Bq[r];
      o[k * os] = make_float2(A[r].x - q.y, A[r].y + q.x);        // A + i B
      o[(p - k) * os] = make_float2(A[r].x + q.y, A[r].y - q.x);  // A - i B
    }
  }
}

// Unnormalised DFT of the L interleaved lines in x; y is the second buffer.  Returns the
// buffer that holds the result.  Entered and left with the data visible to the whole block.
template <bool INV>
__device__ float2* line_dft(float2* x, float2* y, const float2* tw, const LinePlan& p, int lg, int LP) {
  int ls = 1;
  for (int f = 0; f < p.nf; ++f) {
    const int r = p.radix[f];
    switch (r) {
      case 2: line_stage<2, INV>(x, y, tw, p.n, ls, lg, LP); break;
      case 3: line_stage<3, INV>(x, y, tw, p.n, ls, lg, LP); break;
      case 4: line_stage<4, INV>(x, y, tw, p.n, ls, lg, LP); break;
      case 5: line_stage<5, INV>(x, y, tw, p.n, ls, lg, LP); break;
      case 8: line_stage<8, INV>(x, y, tw, p.n, ls, lg, LP); break;
      default: line_stage_prime<INV>(x, y, tw, p.n, r, ls, lg, LP); break;
    }
    __syncthreads();
    float2* t = x;
    x = y;
    y = t;
    ls *= r;
  }
  return x;
}

// Lines per block (log2, at most 8 lines) for a length: both buffers and the twiddles twice
// per SM, or once where that leaves fewer than four lines.
inline int line_pitch(int lg) { return lg > 0 ? (1 << lg) + 1 : 1; }
inline size_t line_smem(int n, int lg) { return sizeof(float2) * ((size_t)2 * n * line_pitch(lg) + n); }
constexpr size_t kLineSmem = 225 * 1024;  // of one block: the longest line (6144) takes 144 KB
inline int line_log2(int n) {
  for (int lg = 3; lg >= 2; --lg)
    if (line_smem(n, lg) <= 112 * 1024) return lg;
  for (int lg = 3; lg > 0; --lg)
    if (line_smem(n, lg) <= kLineSmem) return lg;
  return 0;
}

}  // namespace qb
