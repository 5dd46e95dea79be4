// Batch norm of channels-last FP32 activations, forward and backward, one launch each
// (nn.BatchNorm2d, torch.nn.functional.batch_norm).
//
// A thread-block cluster owns CW channels (a warp: CW channels x 32 / CW rows) and its CTAs
// split the rows: per-channel sums (float over runs of rows, then double), one exchange of the
// partial sums through distributed shared memory, and the elementwise pass over the same rows.
// The backward also sums the bias gradient.  Bound by its cluster barriers at few rows (64 x 512: 12.5
// cycles per issued instruction) and by the latency of its loads at many (16384 x 32: 4.4), the
// layers' 64 KB to 2 MB being L2-resident.  As partial sums, a serial final sum over up
// to 592 partials and separate elementwise and bias-gradient passes, the batch norms of one
// training step of the 5-level network took 229 launches and 1.3 ms.
//
// Many rows take separate launches over all SMs instead (below): a cluster per sector of channels leaves
// most of the device idle then.
//
// The float runs are those of a fixed partition of the rows (BnRows), whatever the cluster: the
// statistics feed BF16 roundings, so they keep their values from one launch shape to the next.
#pragma once
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "cnn_act.cuh"

namespace qb {
namespace bn {

namespace cg = cooperative_groups;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCtas = 8;
constexpr int kMaxCw = 32;

// Float runs: chunk k of rows [k rpc, (k + 1) rpc), run t of it its rows t, t + RP, ...
struct BnRows {
  int R, C, RP, rpc, runs;
  BnRows(int rows, int cols) : R(rows), C(cols) {
    const int tc = cols < 256 ? cols : 256;
    RP = 256 / tc;
    int chunks = (rows + RP * 16 - 1) / (RP * 16);
    if (chunks > 592) chunks = 592;
    rpc = (rows + chunks - 1) / chunks;
    runs = (rows + rpc - 1) / rpc * RP;
  }
};

// Sums of NV doubles per channel over the cluster, every thread of a channel gets them.
template <int NV>
struct Sums {
  double part[kWarps][kMaxCw][NV];
  double slots[kMaxCtas][kMaxCw][NV];
};
template <int NV>
__device__ __forceinline__ void cluster_sums(Sums<NV>& sm, double (&v)[NV], int CW) {
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nc = (int)cl.num_blocks();
#pragma unroll
  for (int i = 0; i < NV; ++i)
    for (int o = 16; o >= CW; o >>= 1) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
  __syncthreads();  // a previous use of part is over
  if (lane < CW)
#pragma unroll
    for (int i = 0; i < NV; ++i) sm.part[w][lane][i] = v[i];
  __syncthreads();
  if ((int)threadIdx.x < CW * nc) {
    const int c = threadIdx.x % CW, dst = threadIdx.x / CW;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      double t = 0.0;
      for (int k = 0; k < kWarps; ++k) t += sm.part[k][c][i];
      cl.map_shared_rank(&sm.slots[0][0][0], dst)[((int)cl.block_rank() * kMaxCw + c) * NV + i] = t;
    }
  }
  cl.sync();
  const int c = lane % CW;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = 0.0;
    for (int k = 0; k < nc; ++k) v[i] += sm.slots[k][c][i];
  }
}

// One float run: v[0] += sum a, v[1] += sum a b over rows r, r + step, ... < r1, in float up to
// 64 rows at a time.  Eight rows are loaded before they are used: a load at a time, the latency of
// its 16 or so rows was most of the kernel.
template <typename L>
__device__ __forceinline__ void run_sums(int r, int r1, int step, double (&v)[2], L load) {
  while (r < r1) {
    float f0 = 0.f, f1 = 0.f;
    for (int i = 0; i < 64 && r < r1; i += 8) {
      float a[8], b[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        a[j] = b[j] = 0.f;
        if (r + j * step < r1) load(r + j * step, a[j], b[j]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (r + j * step < r1) {
          f0 += a[j];
          f1 = fmaf(a[j], b[j], f1);
        }
      r += 8 * step;
    }
    v[0] += f0;
    v[1] += f1;
  }
}

struct Forward {
  const float* x;
  int ldx;
  const float *gamma, *beta;
  float *run_mean, *run_var, *mean, *rstd;
  float momentum, eps;
  int training;
  __nv_bfloat16* y;
  int ldy;
};

__global__ void __launch_bounds__(kThreads) bn_forward_kernel(const Forward p, const BnRows rows, int CW) {
  __shared__ Sums<2> sm;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nc = (int)cl.num_blocks();
  const int rl = 32 / CW;                                     // rows of a warp
  const int slot = ((int)cl.block_rank() * kWarps + w) * rl + lane / CW, nslots = nc * kWarps * rl;
  const int c = (int)(blockIdx.x / nc) * CW + lane % CW;
  const bool on = c < rows.C;
  float m = 0.f, rs = 0.f;
  if (p.training) {
    cl.sync();  // every CTA of the cluster runs before a peer writes its slots
    double v[2] = {0.0, 0.0};
    if (on)
      for (int t = slot; t < rows.runs; t += nslots) {
        const int r0 = t / rows.RP * rows.rpc, r1 = min(rows.R, r0 + rows.rpc);
        run_sums(r0 + t % rows.RP, r1, rows.RP, v,
                 [&](int r, float& a, float& b) { a = b = p.x[(int64_t)r * p.ldx + c]; });
      }
    cluster_sums<2>(sm, v, CW);
    const double mean = v[0] / rows.R;
    double var = v[1] / rows.R - mean * mean;
    if (var < 0.0) var = 0.0;
    m = (float)mean;
    rs = (float)(1.0 / sqrt(var + (double)p.eps));
    if (on && cl.block_rank() == 0 && w == 0 && lane < CW) {
      p.mean[c] = m;
      p.rstd[c] = rs;
      if (p.run_mean) {
        const double unb = rows.R > 1 ? var * rows.R / (rows.R - 1) : var;
        p.run_mean[c] = (float)((1.0 - p.momentum) * p.run_mean[c] + p.momentum * mean);
        p.run_var[c] = (float)((1.0 - p.momentum) * p.run_var[c] + p.momentum * unb);
      }
    }
  } else if (on) {
    m = p.run_mean[c];
    rs = rsqrtf(p.run_var[c] + p.eps);
    if (cl.block_rank() == 0 && w == 0 && lane < CW) {
      p.mean[c] = m;
      p.rstd[c] = rs;
    }
  }
  if (on) {
    const float g = p.gamma[c], b = p.beta[c];
    for (int r = slot; r < rows.R; r += 8 * nslots) {
      float a[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (r + j * nslots < rows.R) a[j] = p.x[(int64_t)(r + j * nslots) * p.ldx + c];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (r + j * nslots < rows.R)
          p.y[(int64_t)(r + j * nslots) * p.ldy + c] = __float2bfloat16_rn((a[j] - m) * rs * g + b);
    }
  }
  if (p.training) cl.sync();  // no CTA leaves while a peer may still write its slots
}

struct Backward {
  const float* dy;
  int lddy;
  const float* x;  // the batch norm's input, after the activation `act`
  int ldx;
  const float *gamma, *mean, *rstd;  // gamma NULL: no batch norm
  int training, act;
  float *dgamma, *dbeta;
  float* dbias;  // optional: sum of dz
  float* dz32;   // optional
  __nv_bfloat16* dz16;
  int ldz;
};

// Up to eight rows r, r + step, ... < end of dz for channel c; returns their sum.
__device__ __forceinline__ float dz_rows(const Backward& p, int r, int step, int end, int c, float m, float rs, float ga,
                                         float sdy, float sdx, float invR) {
  float xv[8], g[8], f = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (r + j * step < end) {
      xv[j] = p.x[(int64_t)(r + j * step) * p.ldx + c];
      g[j] = p.dy[(int64_t)(r + j * step) * p.lddy + c];
    }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (r + j * step < end) {
      if (p.gamma) {
        if (p.training) {
          const float xh = (xv[j] - m) * rs;
          g[j] = ga * rs * (g[j] - sdy * invR - xh * sdx * invR);
        } else {
          g[j] = g[j] * ga * rs;
        }
      }
      if (p.act) g[j] *= act_grad_from_output(p.act, xv[j]);
      const int64_t o = (int64_t)(r + j * step) * p.ldz + c;
      if (p.dz32) p.dz32[o] = g[j];
      if (p.dz16) p.dz16[o] = __float2bfloat16_rn(g[j]);
      f += g[j];
    }
  return f;
}

// dz = act'(x) gamma rstd (dy - s_dy / R - xhat s_dyxhat / R) (training statistics),
// act'(x) dy gamma rstd (running statistics), act'(x) dy (no batch norm).
__global__ void __launch_bounds__(kThreads) bn_backward_kernel(const Backward p, const BnRows rows, int CW) {
  __shared__ Sums<2> sm;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nc = (int)cl.num_blocks();
  const int rl = 32 / CW;
  const int slot = ((int)cl.block_rank() * kWarps + w) * rl + lane / CW, nslots = nc * kWarps * rl;
  const int c = (int)(blockIdx.x / nc) * CW + lane % CW;
  const bool on = c < rows.C, first = cl.block_rank() == 0 && w == 0 && lane < CW;
  float m = 0.f, rs = 0.f, ga = 0.f, sdy = 0.f, sdx = 0.f;
  if (p.gamma || p.dbias) cl.sync();  // every CTA of the cluster runs before a peer writes its slots
  if (p.gamma) {
    if (on) {
      m = p.mean[c];
      rs = p.rstd[c];
      ga = p.gamma[c];
    }
    double v[2] = {0.0, 0.0};
    if (on)
      for (int t = slot; t < rows.runs; t += nslots) {
        const int r0 = t / rows.RP * rows.rpc, r1 = min(rows.R, r0 + rows.rpc);
        run_sums(r0 + t % rows.RP, r1, rows.RP, v, [&](int r, float& a, float& b) {
          a = p.dy[(int64_t)r * p.lddy + c];
          b = (p.x[(int64_t)r * p.ldx + c] - m) * rs;
        });
      }
    cluster_sums<2>(sm, v, CW);
    sdy = (float)v[0];
    sdx = (float)v[1];
    if (on && first) {
      p.dbeta[c] = sdy;
      p.dgamma[c] = sdx;
    }
  }
  const float invR = 1.0f / (float)rows.R;
  double sum[2] = {0.0, 0.0};
  if (on)
    for (int r = slot; r < rows.R; r += 8 * nslots)
      sum[0] += dz_rows(p, r, nslots, rows.R, c, m, rs, ga, sdy, sdx, invR);
  if (p.dbias) {
    if (p.gamma) cl.sync();  // every CTA has read the first sums' slots
    cluster_sums<2>(sm, sum, CW);
    if (on && first) p.dbias[c] = (float)sum[0];
  }
  if (p.gamma || p.dbias) cl.sync();  // no CTA leaves while a peer may still write its slots
}

// ---- many rows: separate launches over all SMs ----
// A cluster's channels are at least one 32-byte sector wide, so C / 8 clusters of 8 CTAs are all that
// the kernels above can put to work: at 32 channels 32 CTAs, whatever the number of rows.  Here blocks
// of 256 threads (a thread: one channel, every RP-th row of a chunk, the same float runs) write partial
// sums, a warp per channel adds them in a fixed order, and an elementwise pass follows.  Bound by the
// latency of the loads of 29 warps per SM, at 31 to 43 % of the DRAM throughput (262144 x 32, cold).
constexpr int kWideThreads = 256;

struct WideRows {
  int c, first, step, end;  // this thread's channel and rows
  bool on;
  __device__ __forceinline__ WideRows(const BnRows& rows) {
    const int tc = rows.C < kWideThreads ? rows.C : kWideThreads;
    const int tx = threadIdx.x % tc, ty = threadIdx.x / tc, r0 = blockIdx.x * rows.rpc;
    c = blockIdx.y * tc + tx;
    on = ty < rows.RP && c < rows.C;
    first = r0 + ty;
    step = rows.RP;
    end = min(rows.R, r0 + rows.rpc);
  }
};
// Sums of v over the threads of a channel, in the first row of threads
template <int NV>
__device__ __forceinline__ void wide_block_sums(double (&v)[NV], const BnRows& rows) {
  __shared__ double red[NV][kWideThreads];
  const int tc = rows.C < kWideThreads ? rows.C : kWideThreads;
#pragma unroll
  for (int i = 0; i < NV; ++i) red[i][threadIdx.x] = v[i];
  __syncthreads();
  if ((int)threadIdx.x < tc)
#pragma unroll
    for (int i = 0; i < NV; ++i)
      for (int k = 1; k < rows.RP; ++k) v[i] += red[i][k * tc + threadIdx.x];
}

// part[(2 chunk + i) C + c]: sums of x and x^2 (forward), of dy and dy xhat (backward)
__global__ void __launch_bounds__(kWideThreads)
    wide_forward_sums_kernel(const Forward p, const BnRows rows, double* __restrict__ part) {
  const WideRows w(rows);
  double v[2] = {0.0, 0.0};
  if (w.on)
    run_sums(w.first, w.end, w.step, v, [&](int r, float& a, float& b) { a = b = p.x[(int64_t)r * p.ldx + w.c]; });
  wide_block_sums<2>(v, rows);
  if (w.on && w.first == (int)blockIdx.x * rows.rpc)
    for (int i = 0; i < 2; ++i) part[((int64_t)blockIdx.x * 2 + i) * rows.C + w.c] = v[i];
}
__global__ void __launch_bounds__(kWideThreads)
    wide_backward_sums_kernel(const Backward p, const BnRows rows, double* __restrict__ part) {
  const WideRows w(rows);
  double v[2] = {0.0, 0.0};
  if (w.on) {
    const float m = p.mean[w.c], rs = p.rstd[w.c];
    run_sums(w.first, w.end, w.step, v, [&](int r, float& a, float& b) {
      a = p.dy[(int64_t)r * p.lddy + w.c];
      b = (p.x[(int64_t)r * p.ldx + w.c] - m) * rs;
    });
  }
  wide_block_sums<2>(v, rows);
  if (w.on && w.first == (int)blockIdx.x * rows.rpc)
    for (int i = 0; i < 2; ++i) part[((int64_t)blockIdx.x * 2 + i) * rows.C + w.c] = v[i];
}
// Sum of value i of every chunk for channel c, one warp
__device__ __forceinline__ double wide_total(const double* part, int chunks, int nv, int i, int C, int c) {
  double t = 0.0;
  for (int k = threadIdx.x & 31; k < chunks; k += 32) t += part[((int64_t)k * nv + i) * C + c];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}
__global__ void __launch_bounds__(kWideThreads)
    wide_forward_stats_kernel(const Forward p, const BnRows rows, int chunks, const double* __restrict__ part) {
  const int c = blockIdx.x * (kWideThreads / 32) + (threadIdx.x >> 5);
  if (c >= rows.C) return;
  const double s0 = wide_total(part, chunks, 2, 0, rows.C, c), s1 = wide_total(part, chunks, 2, 1, rows.C, c);
  if (threadIdx.x & 31) return;
  const double mean = s0 / rows.R;
  double var = s1 / rows.R - mean * mean;
  if (var < 0.0) var = 0.0;
  p.mean[c] = (float)mean;
  p.rstd[c] = (float)(1.0 / sqrt(var + (double)p.eps));
  if (p.run_mean) {
    const double unb = rows.R > 1 ? var * rows.R / (rows.R - 1) : var;
    p.run_mean[c] = (float)((1.0 - p.momentum) * p.run_mean[c] + p.momentum * mean);
    p.run_var[c] = (float)((1.0 - p.momentum) * p.run_var[c] + p.momentum * unb);
  }
}
// out0[c], out1[c] = sums 0 and 1 of nv per chunk (out1 may be NULL)
__global__ void __launch_bounds__(kWideThreads)
    wide_totals_kernel(const double* __restrict__ part, int chunks, int nv, int C, float* out0, float* out1) {
  const int c = blockIdx.x * (kWideThreads / 32) + (threadIdx.x >> 5);
  if (c >= C) return;
  const double s0 = wide_total(part, chunks, nv, 0, C, c), s1 = out1 ? wide_total(part, chunks, nv, 1, C, c) : 0.0;
  if (threadIdx.x & 31) return;
  out0[c] = (float)s0;
  if (out1) out1[c] = (float)s1;
}
__global__ void __launch_bounds__(kWideThreads) wide_forward_kernel(const Forward p, const BnRows rows) {
  const WideRows w(rows);
  if (!w.on) return;
  float m, rs;
  if (p.training) {
    m = p.mean[w.c];
    rs = p.rstd[w.c];
  } else {
    m = p.run_mean[w.c];
    rs = rsqrtf(p.run_var[w.c] + p.eps);
    if (w.first == 0) {
      p.mean[w.c] = m;
      p.rstd[w.c] = rs;
    }
  }
  const float g = p.gamma[w.c], b = p.beta[w.c];
  for (int r = w.first; r < w.end; r += 8 * w.step) {
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (r + j * w.step < w.end) a[j] = p.x[(int64_t)(r + j * w.step) * p.ldx + w.c];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (r + j * w.step < w.end)
        p.y[(int64_t)(r + j * w.step) * p.ldy + w.c] = __float2bfloat16_rn((a[j] - m) * rs * g + b);
  }
}
// dz; part[chunk C + c]: its sums (with dbias)
__global__ void __launch_bounds__(kWideThreads)
    wide_backward_kernel(const Backward p, const BnRows rows, double* __restrict__ part) {
  const WideRows w(rows);
  double sum[1] = {0.0};
  if (w.on) {
    float m = 0.f, rs = 0.f, ga = 0.f, sdy = 0.f, sdx = 0.f;
    if (p.gamma) {
      m = p.mean[w.c];
      rs = p.rstd[w.c];
      ga = p.gamma[w.c];
      sdy = p.dbeta[w.c];
      sdx = p.dgamma[w.c];
    }
    const float invR = 1.0f / (float)rows.R;
    for (int r = w.first; r < w.end; r += 8 * w.step)
      sum[0] += dz_rows(p, r, w.step, w.end, w.c, m, rs, ga, sdy, sdx, invR);
  }
  if (p.dbias) {
    wide_block_sums<1>(sum, rows);
    if (w.on && w.first == (int)blockIdx.x * rows.rpc) part[(int64_t)blockIdx.x * rows.C + w.c] = sum[0];
  }
}

// Channels per warp and CTAs per cluster: narrow tiles for many rows (16384 x 32, forward / backward: 8
// channels 14.6 / 18.7 us a call, 16 channels 16.7 / 29.9, 32 channels 26.9 / 53.5; one CTA instead of
// eight 47.8 / 98.7), few CTAs for few rows, whose barriers cost more than they share out (16 x 1024: one to
// four CTAs of 16 or 32 channels 12.0 / 12.6, eight of 8 channels 20.7 / 25.3).  In between the
// shapes are equal, at the 12 us of a call.
struct Shape {
  int cw, ctas, grid;
  Shape(int R, int C) {
    cw = C <= 64 && R >= 2048 ? 8 : (C <= 256 && R >= 256 ? 16 : 32);
    ctas = R >= 1024 ? 8 : (R >= 256 ? 4 : (R >= 64 ? 2 : 1));
    grid = (C + cw - 1) / cw * ctas;
  }
};
template <typename P>
cudaError_t launch(void (*kernel)(P, BnRows, int), const P& p, int R, int C, cudaStream_t st) {
  const Shape s(R, C);
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)s.grid, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)s.ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, p, BnRows(R, C), s.cw);
}

// Where the launches over all SMs replace the cluster launch: from 32768 rows in the forward with batch
// statistics (three launches; device times at 32 channels: 8192 rows 9.4 us against 7.2, 16384 rows 9.2
// against 9.9, 32768 rows 10.6 against 15.4, 262144 rows 27 against 87; at 128 channels 16384 rows
// 16.6 against 15.2, 32768 rows 21.6 against 25.8), from 16384 rows in the other passes (backward at 32
// channels: 8192 rows 11.7 us against 10.6, 16384 rows 11.9 against 16.6, 262144 rows 43 against 260;
// running statistics, 16384 rows: 3.3 against 5.5).
inline bool wide(int R, bool batch_stats_forward) { return R >= (batch_stats_forward ? 32768 : 16384); }

// Partial sums (doubles) of the wide launches
inline int64_t wide_elems(int R, int C) {
  const BnRows rows(R, C);
  return (int64_t)2 * (rows.runs / rows.RP) * C;
}
inline cudaError_t launch_wide(const Forward& p, int R, int C, double* part, cudaStream_t st) {
  const BnRows rows(R, C);
  const int chunks = rows.runs / rows.RP, tiles = (C + kWideThreads - 1) / kWideThreads;
  const dim3 grid(chunks, tiles);
  if (p.training) {
    wide_forward_sums_kernel<<<grid, kWideThreads, 0, st>>>(p, rows, part);
    wide_forward_stats_kernel<<<(C + 7) / 8, kWideThreads, 0, st>>>(p, rows, chunks, part);
  }
  wide_forward_kernel<<<grid, kWideThreads, 0, st>>>(p, rows);
  return cudaGetLastError();
}
inline cudaError_t launch_wide(const Backward& p, int R, int C, double* part, cudaStream_t st) {
  const BnRows rows(R, C);
  const int chunks = rows.runs / rows.RP, tiles = (C + kWideThreads - 1) / kWideThreads;
  const dim3 grid(chunks, tiles);
  if (p.gamma) {
    wide_backward_sums_kernel<<<grid, kWideThreads, 0, st>>>(p, rows, part);
    wide_totals_kernel<<<(C + 7) / 8, kWideThreads, 0, st>>>(part, chunks, 2, C, p.dbeta, p.dgamma);
  }
  wide_backward_kernel<<<grid, kWideThreads, 0, st>>>(p, rows, part);
  if (p.dbias) wide_totals_kernel<<<(C + 7) / 8, kWideThreads, 0, st>>>(part, chunks, 1, C, p.dbias, nullptr);
  return cudaGetLastError();
}

}  // namespace bn
}  // namespace qb
