// Register-resident 2-D FFT engine for one N x N complex64 wave per CTA (sm_100a).
//
// A CTA of T threads holds the wave in registers, E = N^2 / T complex values per
// thread.  The 2-D transform is factored into three register stages that each
// consume a subset of the 2*log2(N) index bits, with one shared-memory exchange
// between consecutive stages:
//
//   columns c = cB + B*cA  (N = A*B),   rows r = rD + D*rC  (N = C*D)
//   S1 : A-point DFT over cA            for fixed (r, cB)          -> kA
//   S2 : twiddle w_N^(cB*kA); B-point DFT over cB; C-point DFT over rC;
//        twiddle w_N^(rD*kC)            for fixed (rD, kA)         -> (kB, kC)
//   S3 : D-point DFT over rD            for fixed (kC, column)     -> kD
//
// The forward output of S3 is in natural frequency order: register (g, e) of a
// thread holds X[kC_g + C*e][col].  The inverse runs S3' -> S2' -> S1' with
// conjugate twiddles, so a forward transform, an elementwise multiply in Fourier
// space and an inverse transform need no exchange between S3 and S3'; likewise
// an inverse, a real-space multiply and a forward transform meet in S1 without
// an exchange.  One multislice step (FFT, propagator, IFFT, transmission) costs
// four exchanges.
//
// Exchanges.  The rows rD + D*rC of one residue rD form a class: S1 and S2 of a class
// touch no other class, and one warp owns whole classes (A threads each), so the
// exchange between S1 and S2 stays inside the warp (__syncwarp).  Only S2 <-> S3 crosses
// warps, with each side reading and writing the same elements in place: one
// __syncthreads per transform.  The class's transpose (A x (B C), padded) and its C rows
// of N spectral values share the class's region of the buffer.  Every warp access is two
// wavefronts per 256 bytes, the minimum for 8-byte words.
//
// No unit of the batch kernels is full.  At 128^2 the load/store unit's data pipe is at 59 % of its peak,
// the FP32 pipe at 50 %, the issue slots at 39 %; the 16 warps of an SM wait most for global loads
// (2.2 cycles per issued instruction), then for the FP32 pipe (1.7).  The data pipe being the busiest,
// the factorisation is chosen for the real-space accesses: B = 8 puts 8 consecutive columns x 4 rows in a warp
// access of the object (B = 4: 4 columns x 8 rows took 3.7 L1 wavefronts per gather and
// 4.6 per gradient scatter, B = 8 takes 1.7 and 2.3: 28.5 -> 26.4 ms per 4096-position
// launch).  At 64^2 B = 4 keeps 16 registers per thread, half the code and three CTAs per
// SM (256 threads of 80 registers); B = 8 with 32 registers and four CTAs of 128 threads
// was 5-15 % slower on single-slice and forward-only launches, its code no longer fitting
// the instruction caches (no-instruction stalls 1.4 per issue against 0.3).
//
// At 96^2, A = 8 and two CTAs of 192 threads (168 registers, 48 of them pairs of the wave)
// replaced a 48 x 2 / 24 x 4 factorisation with one CTA of 255 registers, whose six warps left
// the SM idle: 1000 positions of 4 slices and 2 modes 1849 -> 1214 us, forward 737 -> 583 us.
//
// Supported N: 64 (A=16,B=4,C=4,D=16, 256 threads), 96 (A=8,B=12,C=4,D=24, 192 threads of
// 48 registers, mixed radix 3 x 2^k, two CTAs per SM) and 128 (A=16,B=8,C=4,D=32, 512 threads).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace qb {

// ---------------------------------------------------------------------------
// complex helpers
// ---------------------------------------------------------------------------
// Complex arithmetic.  With QB_F32X2_ADD / QB_F32X2_MUL set (per translation unit,
// before this header) it runs on sm_100's packed FP32 pairs, one instruction for the
// real and imaginary parts, with the same roundings as the scalar forms
//   a * b       = (fma(a.x, b.x, -(a.y b.y)), fma(a.x, b.y, a.y b.x))
//   a * conj(b) = (fma(a.x, b.x, a.y b.y),    fma(a.y, b.x, -(a.x b.y)))
// so results are bit-identical either way.  The packed operands live in aligned
// register pairs, which costs registers: packed products pay everywhere but in the 128^2
// kernels with extensions or the analytic update (they pack their additions and the
// middle-stage twiddles).
#ifndef QB_F32X2_ADD
#define QB_F32X2_ADD 0
#endif
#ifndef QB_F32X2_MUL
#define QB_F32X2_MUL 0
#endif
#if QB_F32X2_ADD
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
#else
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
#endif
#if QB_F32X2_MUL
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return __ffma2_rn(make_float2(a.x, a.x), b, __fmul2_rn(make_float2(a.y, a.y), make_float2(-b.y, b.x)));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return __ffma2_rn(a, make_float2(b.x, b.x), __fmul2_rn(make_float2(a.y, -a.x), make_float2(b.y, b.y)));
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
#else
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
#endif
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
// Packed products whatever the switches above say; QB_F32X2_S2 uses them for the
// twiddle multiplies of the 2-D engine's middle stage only (no extra spills in the
// 128^2 batch kernel, unlike packed products everywhere).
__device__ __forceinline__ float2 pcmul(float2 a, float2 b) {
  return __ffma2_rn(make_float2(a.x, a.x), b, __fmul2_rn(make_float2(a.y, a.y), make_float2(-b.y, b.x)));
}
__device__ __forceinline__ float2 pcmulc(float2 a, float2 b) {
  return __ffma2_rn(a, make_float2(b.x, b.x), __fmul2_rn(make_float2(a.y, -a.x), make_float2(b.y, b.y)));
}
#ifndef QB_F32X2_S2
#define QB_F32X2_S2 0
#endif
__device__ __forceinline__ float cabs2(float2 a) { return fmaf(a.x, a.x, a.y * a.y); }

// cos(2*pi*m/64) for m = 0..16 (first quadrant), IEEE double rounded to float.
__device__ __forceinline__ float qcos64(int m) {
  switch (m) {
    case 0: return 1.0f;
    case 1: return 0.99518472667219693f;
    case 2: return 0.98078528040323043f;
    case 3: return 0.95694033573220882f;
    case 4: return 0.92387953251128674f;
    case 5: return 0.88192126434835505f;
    case 6: return 0.83146961230254524f;
    case 7: return 0.77301045336273699f;
    case 8: return 0.70710678118654757f;
    case 9: return 0.63439328416364549f;
    case 10: return 0.55557023301960229f;
    case 11: return 0.47139673682599781f;
    case 12: return 0.38268343236508984f;
    case 13: return 0.29028467725446233f;
    case 14: return 0.19509032201612833f;
    case 15: return 0.09801714032956077f;
    default: return 0.0f;
  }
}

// Multiply by w_64^m (forward: exp(-2 pi i m/64); inverse: conjugate), m a
// compile-time constant after unrolling.  Quarter turns are exact.
template <bool INV>
__device__ __forceinline__ float2 twmul64(float2 a, int m) {
  m &= 63;
  if (m == 0) return a;
  if (m == 16) return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  if (m == 32) return make_float2(-a.x, -a.y);
  if (m == 48) return INV ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
  const int q = m >> 4, r = m & 15;
  float c, s;  // cos/sin(2 pi m / 64)
  if (q == 0) { c = qcos64(r); s = qcos64(16 - r); }
  else if (q == 1) { c = -qcos64(16 - r); s = qcos64(r); }
  else if (q == 2) { c = -qcos64(r); s = -qcos64(16 - r); }
  else { c = qcos64(16 - r); s = -qcos64(r); }
  if (!INV) s = -s;
  return cmul(a, make_float2(c, s));
}

__host__ __device__ constexpr int bitrev(int k, int n) {
  int r = 0;
  for (int i = 1; i < n; i <<= 1) { r = (r << 1) | (k & 1); k >>= 1; }
  return r;
}

// In-register N-point DFT (N <= 64, power of two) on x[OFF + STRIDE*i], natural
// order in and out.  Radix-2 decimation in frequency, then a register rename.
template <int N, bool INV, int STRIDE = 1, int OFF = 0, int LEN>
__device__ __forceinline__ void dft_reg(float2 (&x)[LEN]) {
  if constexpr (N == 1) {
    return;
  } else if constexpr (N == 2) {
    float2 a = x[OFF], b = x[OFF + STRIDE];
    x[OFF] = cadd(a, b);
    x[OFF + STRIDE] = csub(a, b);
  } else {
#pragma unroll
    for (int half = N / 2; half >= 1; half >>= 1) {
#pragma unroll
      for (int blk = 0; blk < N; blk += 2 * half) {
#pragma unroll
        for (int j = 0; j < half; ++j) {
          const int i0 = OFF + STRIDE * (blk + j), i1 = OFF + STRIDE * (blk + j + half);
          float2 a = x[i0], b = x[i1];
          x[i0] = cadd(a, b);
          x[i1] = twmul64<INV>(csub(a, b), j * (64 / (2 * half)));
        }
      }
    }
    float2 y[N];
#pragma unroll
    for (int k = 0; k < N; ++k) y[k] = x[OFF + STRIDE * bitrev(k, N)];
#pragma unroll
    for (int k = 0; k < N; ++k) x[OFF + STRIDE * k] = y[k];
  }
}

// ---------------------------------------------------------------------------
// mixed radix (N = 3 * 2^k) for 96 x 96 windows
// ---------------------------------------------------------------------------
// cos(2*pi*m/96) for m = 0..24 (first quadrant), IEEE double rounded to float.
__device__ __forceinline__ float qcos96(int m) {
  switch (m) {
    case 0: return 1.0f;
    case 1: return 0.9978589232386035f;
    case 2: return 0.9914448613738104f;
    case 3: return 0.9807852804032304f;
    case 4: return 0.9659258262890683f;
    case 5: return 0.9469301294951057f;
    case 6: return 0.9238795325112867f;
    case 7: return 0.8968727415326884f;
    case 8: return 0.8660254037844387f;
    case 9: return 0.8314696123025452f;
    case 10: return 0.7933533402912352f;
    case 11: return 0.7518398074789774f;
    case 12: return 0.7071067811865476f;
    case 13: return 0.6593458151000688f;
    case 14: return 0.6087614290087207f;
    case 15: return 0.5555702330196024f;
    case 16: return 0.5000000000000001f;
    case 17: return 0.44228869021900125f;
    case 18: return 0.38268343236508984f;
    case 19: return 0.3214394653031617f;
    case 20: return 0.25881904510252074f;
    case 21: return 0.19509032201612833f;
    case 22: return 0.1305261922200517f;
    case 23: return 0.06540312923014327f;
    default: return 0.0f;
  }
}
// Multiply by w_96^m (forward exp(-2 pi i m/96), inverse its conjugate); m a
// compile-time constant after unrolling, quarter turns exact.
template <bool INV>
__device__ __forceinline__ float2 twmul96(float2 a, int m) {
  m %= 96;
  if (m < 0) m += 96;
  if (m == 0) return a;
  if (m == 24) return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  if (m == 48) return make_float2(-a.x, -a.y);
  if (m == 72) return INV ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
  const int q = m / 24, r = m % 24;
  float c, s;  // cos / sin(2 pi m / 96)
  if (q == 0) { c = qcos96(r); s = qcos96(24 - r); }
  else if (q == 1) { c = -qcos96(24 - r); s = qcos96(r); }
  else if (q == 2) { c = -qcos96(r); s = -qcos96(24 - r); }
  else { c = qcos96(24 - r); s = -qcos96(r); }
  if (!INV) s = -s;
  return cmul(a, make_float2(c, s));
}
// 3-point DFT in place: (a, b, c) -> (X0, X1, X2), w3 = exp(-+2 pi i / 3).
template <bool INV>
__device__ __forceinline__ void dft3(float2& a, float2& b, float2& c) {
  const float h = 0.8660254037844386f;  // sin(pi / 3)
  const float2 t1 = cadd(b, c);
  const float2 t2 = make_float2(fmaf(-0.5f, t1.x, a.x), fmaf(-0.5f, t1.y, a.y));
  const float2 d = csub(b, c);
  // forward: -i * sin(pi/3) * (b - c); inverse: +i * sin(pi/3) * (b - c)
  const float2 t3 = INV ? make_float2(-h * d.y, h * d.x) : make_float2(h * d.y, -h * d.x);
  a = cadd(a, t1);
  b = cadd(t2, t3);
  c = csub(t2, t3);
}
// In-register N-point DFT for N = 3*M (M a power of two) or a power of two, on
// x[OFF + STRIDE*i], natural order in and out: three M-point DFTs over the
// residues of i mod 3, twiddles w_N^(r*k), M three-point DFTs, register rename.
template <int N, bool INV, int STRIDE = 1, int OFF = 0, int LEN>
__device__ __forceinline__ void dft_reg_n(float2 (&x)[LEN]) {
  if constexpr ((N & (N - 1)) == 0) {
    dft_reg<N, INV, STRIDE, OFF>(x);
  } else {
    static_assert(N % 3 == 0 && ((N / 3) & (N / 3 - 1)) == 0 && 96 % N == 0, "N = 3 * 2^k dividing 96");
    constexpr int M = N / 3;
    dft_reg<M, INV, 3 * STRIDE, OFF>(x);
    dft_reg<M, INV, 3 * STRIDE, OFF + STRIDE>(x);
    dft_reg<M, INV, 3 * STRIDE, OFF + 2 * STRIDE>(x);
#pragma unroll
    for (int k = 1; k < M; ++k) {
      x[OFF + STRIDE * (3 * k + 1)] = twmul96<INV>(x[OFF + STRIDE * (3 * k + 1)], (96 / N) * k);
      x[OFF + STRIDE * (3 * k + 2)] = twmul96<INV>(x[OFF + STRIDE * (3 * k + 2)], (96 / N) * 2 * k);
    }
#pragma unroll
    for (int k = 0; k < M; ++k)
      dft3<INV>(x[OFF + STRIDE * (3 * k)], x[OFF + STRIDE * (3 * k + 1)], x[OFF + STRIDE * (3 * k + 2)]);
    float2 y[N];  // X[k + M j] sits at position 3k + j
#pragma unroll
    for (int k = 0; k < M; ++k)
#pragma unroll
      for (int j = 0; j < 3; ++j) y[k + M * j] = x[OFF + STRIDE * (3 * k + j)];
#pragma unroll
    for (int i = 0; i < N; ++i) x[OFF + STRIDE * i] = y[i];
  }
}

// ---------------------------------------------------------------------------
// 2-D engine
// ---------------------------------------------------------------------------
template <int N> struct FftCfg;
// LB: consecutive columns of a warp's real-space access
template <> struct FftCfg<64> { static constexpr int A = 16, B = 4, C = 4, D = 16, LB = 4, CTAS = 3; };
template <> struct FftCfg<96> { static constexpr int A = 8, B = 12, C = 4, D = 24, LB = 4, CTAS = 2; };
template <> struct FftCfg<128> { static constexpr int A = 16, B = 8, C = 4, D = 32, LB = 8, CTAS = 1; };

template <int N>
struct Fft2 {
  static constexpr int A = FftCfg<N>::A, B = FftCfg<N>::B, C = FftCfg<N>::C, D = FftCfg<N>::D;
  static constexpr int E = B * C;        // complex registers per thread
  static constexpr int T = N * N / E;    // threads per CTA
  static constexpr int CTAS = FftCfg<N>::CTAS;  // resident CTAs per SM of the batch kernels
  static constexpr int G1 = E / A;       // S1 groups per thread
  static constexpr int LB = FftCfg<N>::LB, LR = A / LB;  // columns x rows of a class's lanes in S1
  static constexpr int GB = B / LB;      // S1 column groups
  static constexpr int G3 = E / D;       // S3 groups per thread
  static constexpr int PITCH = N + 1;    // row pitch of a plain N x N tile kept in this buffer
  static constexpr int PP = B * C + 1;   // pitch of a class's A x (B C) transpose
  static constexpr int CS = A * PP;      // class stride: its transpose, or its C rows of N
  static constexpr int SM_FLOAT2 = D * CS;
  static_assert(A * B == N && C * D == N, "bad factorisation");
  static_assert(G3 * D == E && G1 * A == E, "stage sizes must match");
  static_assert(CS >= C * N && SM_FLOAT2 >= N * PITCH, "buffer too small");
  static_assert(D * A == T && 32 % A == 0 && LB * LR == A && GB * LB == B && G1 % GB == 0,
                "a warp owns whole classes");

  // stage coordinates of this thread
  int s1_r0, s1_cB;      // S1: row and column residue of group 0
  int s2_rD, s2_kA;      // S2 (s2_rD: the class this thread works on in S1 and S2)
  int s3_c, s3_kC0;      // S3: column, first kC (group g adds 4*g)
  int pv_w, pv_r;        // class-private transpose: S1 side, S2 side
  int mn_2, mn_3;        // main exchange: S2 side, S3 side

  __device__ __forceinline__ void init(int tid) {
    const int lane = tid & 31, w = tid >> 5;
    const int cl = tid & (A - 1);  // thread within its class (A threads)
    s2_rD = tid / A;
    s2_kA = cl;
    s1_cB = cl % LB;
    s1_r0 = s2_rD + D * (cl / LB);
    constexpr int CW = N / 32;  // warps per 32-column strip
    s3_c = lane + 32 * (w % CW);
    s3_kC0 = w / CW;
    pv_w = s2_rD * CS + (cl / LB) * B + cl % LB;
    pv_r = s2_rD * CS + PP * cl;
    mn_2 = s2_rD * CS + cl;
    mn_3 = s3_kC0 * N + s3_c;
  }
  __device__ __forceinline__ int s3_kC(int g) const { return s3_kC0 + (T / 32 / (N / 32)) * g; }
  // natural (row, col) of S1 register (g, e) = x[g A + e]
  __device__ __forceinline__ int s1_row(int g) const { return s1_r0 + D * LR * (g / GB); }
  __device__ __forceinline__ int s1_col(int g, int e) const { return s1_cB + LB * (g % GB) + B * e; }
  // the class's line of group g, from the line of group 0
  static __device__ __forceinline__ constexpr int line(int g) { return LB * (g % GB) + B * LR * (g / GB); }
  // frequency row of S3 register (g, e)
  __device__ __forceinline__ int s3_row(int g, int e) const { return s3_kC(g) + C * e; }

  // ---- class-private transpose between S1 and S2 (one warp, __syncwarp only) ----
  // element (kA, line l = B rC + cB) of the class at kA PP + l
  __device__ __forceinline__ void write_s1(float2* sm, const float2 (&x)[E]) const {
#pragma unroll
    for (int g = 0; g < G1; ++g)
#pragma unroll
      for (int e = 0; e < A; ++e) sm[pv_w + PP * e + line(g)] = x[g * A + e];
  }
  __device__ __forceinline__ void read_s1(const float2* sm, float2 (&x)[E]) const {
#pragma unroll
    for (int g = 0; g < G1; ++g)
#pragma unroll
      for (int e = 0; e < A; ++e) x[g * A + e] = sm[pv_w + PP * e + line(g)];
  }
  // S2 input layout (cB, rC)
  __device__ __forceinline__ void read_s2_in(const float2* sm, float2 (&x)[E]) const {
#pragma unroll
    for (int cB = 0; cB < B; ++cB)
#pragma unroll
      for (int rC = 0; rC < C; ++rC) x[cB * C + rC] = sm[pv_r + B * rC + cB];
  }
  __device__ __forceinline__ void write_s2_in(float2* sm, const float2 (&x)[E]) const {
#pragma unroll
    for (int cB = 0; cB < B; ++cB)
#pragma unroll
      for (int rC = 0; rC < C; ++rC) sm[pv_r + B * rC + cB] = x[cB * C + rC];
  }
  // ---- main exchange between S2 and S3: element (rD, kC, column) at rD CS + kC N + column ----
  // S2 output layout (kB, kC): column kA + A kB
  __device__ __forceinline__ void write_s2_out(float2* sm, const float2 (&x)[E]) const {
#pragma unroll
    for (int kB = 0; kB < B; ++kB)
#pragma unroll
      for (int kC = 0; kC < C; ++kC) sm[mn_2 + N * kC + A * kB] = x[kB * C + kC];
  }
  __device__ __forceinline__ void read_s2_out(const float2* sm, float2 (&x)[E]) const {
#pragma unroll
    for (int kB = 0; kB < B; ++kB)
#pragma unroll
      for (int kC = 0; kC < C; ++kC) x[kB * C + kC] = sm[mn_2 + N * kC + A * kB];
  }
  __device__ __forceinline__ int s3_slot(int g, int e) const { return mn_3 + CS * e + (T / 32 / (N / 32)) * N * g; }
  // S3 layout (g, e): rD = e, kC = kC_g, column s3_c
  __device__ __forceinline__ void read_s3(const float2* sm, float2 (&x)[E]) const {
#pragma unroll
    for (int g = 0; g < G3; ++g)
#pragma unroll
      for (int e = 0; e < D; ++e) x[g * D + e] = sm[mn_3 + CS * e + (T / 32 / (N / 32)) * N * g];
  }
  __device__ __forceinline__ void write_s3(float2* sm, const float2 (&x)[E]) const {
#pragma unroll
    for (int g = 0; g < G3; ++g)
#pragma unroll
      for (int e = 0; e < D; ++e) sm[mn_3 + CS * e + (T / 32 / (N / 32)) * N * g] = x[g * D + e];
  }

  // ---- register stages ----
  // G transforms of L consecutive registers each
  template <int L, int G, bool INV, int K>
  __device__ __forceinline__ void groups(float2 (&x)[E]) const {
    if constexpr (K < G) {
      dft_reg_n<L, INV, 1, K * L>(x);
      groups<L, G, INV, K + 1>(x);
    }
  }
  template <bool INV>
  __device__ __forceinline__ void s1(float2 (&x)[E]) const {
    groups<A, G1, INV, 0>(x);
  }

  template <bool INV>
  __device__ __forceinline__ void s3(float2 (&x)[E]) const {
    groups<D, G3, INV, 0>(x);
  }

  // S2 twiddles in the order the warps read them: w_N^(cB kA) at (cB - 1) A + kA (a
  // class's lanes on consecutive words), then w_N^(rD kC) at TWC + (kC - 1) D + rD (one word
  // per class).
  static constexpr int TWC = (B - 1) * A;
  static constexpr int TW_FLOAT2 = TWC + (C - 1) * D;
  static __device__ __forceinline__ void fill_twiddles(float2* tw, int tid, int nthreads) {
    for (int k = tid; k < TW_FLOAT2; k += nthreads) {
      const int e = k < TWC ? (k / A + 1) * (k % A) : ((k - TWC) / D + 1) * ((k - TWC) % D);
      double s, c;
      sincospi(-2.0 * (double)e / (double)N, &s, &c);
      tw[k] = make_float2((float)c, (float)s);
    }
  }
  // S2 forward: x holds (cB, rC) on entry, (kB, kC) on exit.
  __device__ __forceinline__ void s2_fwd(float2 (&x)[E], const float2* tw) const {
#pragma unroll
    for (int cB = 1; cB < B; ++cB) {
      const float2 w = tw[(cB - 1) * A + s2_kA];
#pragma unroll
      for (int rC = 0; rC < C; ++rC) x[cB * C + rC] = QB_F32X2_S2 ? pcmul(x[cB * C + rC], w) : cmul(x[cB * C + rC], w);
    }
    s2_core<false>(x);
#pragma unroll
    for (int kC = 1; kC < C; ++kC) {
      const float2 w = tw[TWC + (kC - 1) * D + s2_rD];
#pragma unroll
      for (int kB = 0; kB < B; ++kB) x[kB * C + kC] = QB_F32X2_S2 ? pcmul(x[kB * C + kC], w) : cmul(x[kB * C + kC], w);
    }
  }
  // S2 inverse: (kB, kC) on entry, (cB, rC) on exit.
  __device__ __forceinline__ void s2_inv(float2 (&x)[E], const float2* tw) const {
#pragma unroll
    for (int kC = 1; kC < C; ++kC) {
      const float2 w = tw[TWC + (kC - 1) * D + s2_rD];
#pragma unroll
      for (int kB = 0; kB < B; ++kB) x[kB * C + kC] = QB_F32X2_S2 ? pcmulc(x[kB * C + kC], w) : cmulc(x[kB * C + kC], w);
    }
    s2_core<true>(x);
#pragma unroll
    for (int cB = 1; cB < B; ++cB) {
      const float2 w = tw[(cB - 1) * A + s2_kA];
#pragma unroll
      for (int rC = 0; rC < C; ++rC) x[cB * C + rC] = QB_F32X2_S2 ? pcmulc(x[cB * C + rC], w) : cmulc(x[cB * C + rC], w);
    }
  }
  // B-point DFT along index 0 (stride C) and C-point DFT along index 1 (stride 1).
  template <bool INV>
  __device__ __forceinline__ void s2_core(float2 (&x)[E]) const {
    s2_bdft<INV, 0>(x);
    s2_cdft<INV, 0>(x);
  }
  template <bool INV, int RC>
  __device__ __forceinline__ void s2_bdft(float2 (&x)[E]) const {
    if constexpr (RC < C) {
      dft_reg_n<B, INV, C, RC>(x);
      s2_bdft<INV, RC + 1>(x);
    }
  }
  template <bool INV, int KB>
  __device__ __forceinline__ void s2_cdft(float2 (&x)[E]) const {
    if constexpr (KB < B) {
      dft_reg_n<C, INV, 1, KB * C>(x);
      s2_cdft<INV, KB + 1>(x);
    }
  }

  // ---- whole transforms between layouts ----
  // One CTA barrier each.  Between two barriers either every class is owned by its warp
  // (S2 side: main exchange, private transpose, S1) or every (kC, column) pair by its
  // thread (S3 side reads and writes the same elements), so no barrier is needed before
  // a write.  A caller that leaves the S2 side (after inverse) without forward, or enters
  // it (forward) without inverse, puts a __syncthreads between.
  // Forward: registers in S1 layout -> registers in S3 layout (unnormalised).
  __device__ __forceinline__ void forward(float2 (&x)[E], float2* sm, const float2* tw) const {
    s1<false>(x);
    __syncwarp();  // the warp's reads of the inverse's transpose are complete
    write_s1(sm, x);
    __syncwarp();
    read_s2_in(sm, x);
    s2_fwd(x, tw);
    __syncwarp();
    write_s2_out(sm, x);
    __syncthreads();
    read_s3(sm, x);
    s3<false>(x);
  }
  // Inverse: registers in S3 layout -> registers in S1 layout (unnormalised).
  __device__ __forceinline__ void inverse(float2 (&x)[E], float2* sm, const float2* tw) const {
    s3<true>(x);
    write_s3(sm, x);
    __syncthreads();
    read_s2_out(sm, x);
    s2_inv(x, tw);
    __syncwarp();
    write_s2_in(sm, x);
    __syncwarp();
    read_s1(sm, x);
    s1<true>(x);
  }
};

}  // namespace qb
