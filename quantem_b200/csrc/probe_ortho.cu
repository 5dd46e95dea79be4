// Mixed-state probe orthogonalisation and its gradient (reference:
// ProbePixelated._probe_orthogonalization_constraint, probe_models.py:484-525):
// modified Gram-Schmidt over the P modes with the running vector, each mode
// rescaled to its original norm, modes sorted by descending real-space intensity.
//
// The algorithm is a chain of P (P + 5) / 2 dependent reductions (a projection coefficient per pair of
// modes, three norms per mode, float64) over P modes of N*N elements.  One thread-block cluster
// of 8 CTAs (16 for windows above 128^2 where the device holds such a cluster) splits every
// mode by elements: a thread touches only its own elements, kept in shared memory where
// they fit, and each reduction is one block sum plus one exchange of partial sums through
// distributed shared memory (one cluster barrier).  The gradient replays the steps
// backwards.  Bound by those barriers (about 1 us a step), not by the data (0.5 MB at four
// 128^2 modes).  One CTA walking all elements through L2 took 83 + 169 us (forward +
// gradient) at four 128^2 modes and 541 + 1266 us at six 256^2 modes.
//
// Work buffer (float2 view, caller-owned, reused by the gradient):
//   q    [P * nn]      orthonormal modes (unsorted)
//   gq   [P * nn]      gradient scratch of q
//   meta               c[P*P] (complex, row i: coefficients of mode i), then per mode
//                      n0, nrm, nrm_c as float2 (x = value) and the sort order
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>

#include "ptycho_b200.h"

int qb_record_error(int code, const char* msg);

namespace {

constexpr int kThreads = 512;
constexpr int kMaxCtas = 16;
constexpr int kMaxModes = 16;

int fail(int code, const char* fmt, ...) {
  char buf[400];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  return qb_record_error(code, buf);
}

namespace cg = cooperative_groups;

struct Z {
  double re, im;
};

// Sums over the cluster: block partials by shuffles, then one slot per CTA in every CTA's
// shared memory, added in rank order.  Two slot sets alternate, so one cluster barrier per
// sum is enough: a CTA writes a set again only after the barrier of the sum in between,
// which every CTA reaches after reading that set.
struct ClusterSum {
  double2* red;    // [kThreads / 32]
  double2* slots;  // [2][kMaxCtas]
  int turn;
  __device__ Z operator()(double re, double im) {
    cg::cluster_group cl = cg::this_cluster();
    const int nc = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    if (l == 0) red[w] = make_double2(re, im);
    __syncthreads();
    double2* set = slots + turn * kMaxCtas;
    if (w == 0) {
      double2 v = l < kThreads / 32 ? red[l] : make_double2(0.0, 0.0);
      for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
      }
      if (l < nc) cl.map_shared_rank(set, l)[rank] = v;
    }
    cl.sync();
    Z t = {0.0, 0.0};
    for (int i = 0; i < nc; ++i) {  // fixed order, every thread
      t.re += set[i].x;
      t.im += set[i].y;
    }
    turn ^= 1;
    return t;
  }
};

// Elements [lo, hi) of every mode belong to this CTA, element lo + k of a mode to thread
// k % kThreads.  A mode array lives either in global memory (pitch nn) or in the CTA's
// shared memory (pitch per, from element lo on).
struct Slice {
  int64_t lo;
  int len;  // elements of this CTA
  int per;  // elements per CTA (pitch of the shared arrays)
};
__device__ __forceinline__ Slice my_slice(int64_t nn) {
  cg::cluster_group cl = cg::this_cluster();
  const int nc = (int)cl.num_blocks();
  Slice s;
  s.per = (int)((nn + nc - 1) / nc);
  s.lo = (int64_t)s.per * cl.block_rank();
  const int64_t left = nn - s.lo;
  s.len = left < 0 ? 0 : (left < s.per ? (int)left : s.per);
  return s;
}

__device__ __forceinline__ float2 cmul_(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cconjmul(float2 a, float2 b) {  // conj(a) * b
  return make_float2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

struct Meta {
  float2* c;     // P*P
  float2* norm;  // P: (n0, nrm), P: (nrm_c, 0)
  int* order;    // P
};
__device__ __forceinline__ Meta meta_of(float2* work, int P, int64_t nn) {
  Meta m;
  m.c = work + 2 * (int64_t)P * nn;
  m.norm = m.c + P * P;
  m.order = reinterpret_cast<int*>(m.norm + 2 * P);
  return m;
}

// q_shared: the orthonormal modes are worked on in shared memory (copied to the work buffer
// at the end), else in the work buffer itself.
__global__ void __launch_bounds__(kThreads, 1)
    probe_ortho_kernel(const float2* __restrict__ in, float2* __restrict__ out, int P, int64_t nn, float2* work,
                       int q_shared) {
  extern __shared__ float2 dyn[];
  __shared__ double2 red[kThreads / 32], slots[2 * kMaxCtas];
  __shared__ float inten[kMaxModes], n0s[kMaxModes];
  __shared__ int order[kMaxModes];
  ClusterSum sum{red, slots, 0};
  const Slice sl = my_slice(nn);
  const Meta m = meta_of(work, P, nn);
  const int tid = threadIdx.x;
  const bool lead = tid == 0 && cg::this_cluster().block_rank() == 0;
  float2* q = q_shared ? dyn : work + sl.lo;
  const int64_t qp = q_shared ? sl.per : nn;
  cg::this_cluster().sync();  // every CTA runs before any access to its shared memory
  for (int i = 0; i < P; ++i) {
    const float2* pi = in + (int64_t)i * nn + sl.lo;
    float2* qi = q + i * qp;
    double s = 0.0;
    for (int k = tid; k < sl.len; k += kThreads) {
      const float2 v = pi[k];
      qi[k] = v;  // running vector u, in place
      s += (double)v.x * v.x + (double)v.y * v.y;
    }
    const double n0 = sqrt(sum(s, 0.0).re);
    for (int j = 0; j < i; ++j) {  // c = sum conj(q_j) u ; u -= c q_j
      const float2* qj = q + j * qp;
      double cr = 0.0, ci = 0.0;
      for (int k = tid; k < sl.len; k += kThreads) {
        const float2 t = cconjmul(qj[k], qi[k]);
        cr += t.x;
        ci += t.y;
      }
      const Z c = sum(cr, ci);
      const float2 cf = make_float2((float)c.re, (float)c.im);
      if (lead) m.c[i * P + j] = cf;
      for (int k = tid; k < sl.len; k += kThreads) {
        const float2 t = cmul_(cf, qj[k]);
        qi[k] = make_float2(qi[k].x - t.x, qi[k].y - t.y);
      }
    }
    double s2 = 0.0;
    for (int k = tid; k < sl.len; k += kThreads) s2 += (double)qi[k].x * qi[k].x + (double)qi[k].y * qi[k].y;
    const double nrm = sqrt(sum(s2, 0.0).re);
    const double nrm_c = nrm > 1e-12 ? nrm : 1e-12;
    const float inv = (float)(1.0 / nrm_c);
    double s3 = 0.0;
    for (int k = tid; k < sl.len; k += kThreads) {
      const float2 v = make_float2(qi[k].x * inv, qi[k].y * inv);
      qi[k] = v;
      const float ox = v.x * (float)n0, oy = v.y * (float)n0;
      s3 += (double)ox * ox + (double)oy * oy;
    }
    const double it = sum(s3, 0.0).re;
    if (tid == 0) {
      n0s[i] = (float)n0;
      inten[i] = (float)it;
    }
    if (lead) {
      m.norm[i] = make_float2((float)n0, (float)nrm);
      m.norm[P + i] = make_float2((float)nrm_c, 0.f);
    }
  }
  if (tid == 0) {  // stable descending order of the intensities (the same in every CTA)
    for (int i = 0; i < P; ++i) order[i] = i;
    for (int i = 1; i < P; ++i)
      for (int j = i; j > 0 && inten[order[j]] > inten[order[j - 1]]; --j) {
        const int t = order[j];
        order[j] = order[j - 1];
        order[j - 1] = t;
      }
  }
  __syncthreads();
  if (lead)
    for (int i = 0; i < P; ++i) m.order[i] = order[i];
  for (int r = 0; r < P; ++r) {
    const int i = order[r];
    const float n0 = n0s[i];
    const float2* qi = q + i * qp;
    float2* o = out + (int64_t)r * nn + sl.lo;
    float2* qg = work + (int64_t)i * nn + sl.lo;
    for (int k = tid; k < sl.len; k += kThreads) {
      const float2 v = qi[k];
      o[k] = make_float2(v.x * n0, v.y * n0);
      if (q_shared) qg[k] = v;
    }
  }
  cg::this_cluster().sync();  // no CTA leaves while a peer may still write its slots
}

// Reverse of probe_ortho_kernel (torch convention: the gradient of a real loss
// with respect to z is dL/dRe z + i dL/dIm z).  in_shared: how many of the arrays u (the
// running vector), gq (gradients of the q, P modes) and q (P modes) live in shared memory,
// in this order; the others are used in global memory (u: in grad_in's mode, whose
// gradient is written last).
__global__ void __launch_bounds__(kThreads, 1)
    probe_ortho_vjp_kernel(const float2* __restrict__ in, const float2* __restrict__ grad_sorted,
                           float2* __restrict__ grad_in, int P, int64_t nn, float2* work, int in_shared) {
  extern __shared__ float2 dyn[];
  __shared__ double2 red[kThreads / 32], slots[2 * kMaxCtas];
  __shared__ float fac[kMaxModes];
  ClusterSum sum{red, slots, 0};
  const Slice sl = my_slice(nn);
  const Meta m = meta_of(work, P, nn);
  const int tid = threadIdx.x;
  float2* gq = in_shared >= 2 ? dyn + sl.per : work + (int64_t)P * nn + sl.lo;
  const int64_t gp = in_shared >= 2 ? sl.per : nn;
  const float2* q = in_shared >= 3 ? dyn + (int64_t)(1 + P) * sl.per : work + sl.lo;
  const int64_t qp = in_shared >= 3 ? sl.per : nn;
  if (in_shared >= 3) {
    float2* qs = dyn + (int64_t)(1 + P) * sl.per;
    for (int i = 0; i < P; ++i)
      for (int k = tid; k < sl.len; k += kThreads) qs[(int64_t)i * sl.per + k] = work[(int64_t)i * nn + sl.lo + k];
  }
  cg::this_cluster().sync();  // every CTA runs before any access to its shared memory
  // g_q = g_out n0 ; g_in = in / n0 * Re<q, g_out>
  for (int r = 0; r < P; ++r) {
    const int i = m.order[r];
    const float n0 = m.norm[i].x;
    const float2* go = grad_sorted + (int64_t)r * nn + sl.lo;
    const float2* qi = q + i * qp;
    float2* gqi = gq + i * gp;
    double s = 0.0;
    for (int k = tid; k < sl.len; k += kThreads) {
      const float2 g = go[k];
      gqi[k] = make_float2(g.x * n0, g.y * n0);
      s += (double)qi[k].x * g.x + (double)qi[k].y * g.y;
    }
    const double gn0 = sum(s, 0.0).re;
    if (tid == 0) fac[i] = (float)(n0 > 0.f ? gn0 / (double)n0 : 0.0);
  }
  __syncthreads();
  for (int i = P - 1; i >= 0; --i) {
    const float nrm = m.norm[i].y, nrm_c = m.norm[P + i].x;
    const float2* qi = q + i * qp;
    float2* gqi = gq + i * gp;
    float2* u = in_shared >= 1 ? dyn : grad_in + (int64_t)i * nn + sl.lo;
    // u = q_i nrm_c ; g_u = g_q / nrm_c (+ u / nrm * g_nrm), kept in gqi
    double s = 0.0;
    for (int k = tid; k < sl.len; k += kThreads)
      s += ((double)qi[k].x * gqi[k].x + (double)qi[k].y * gqi[k].y) * nrm_c;  // Re<u, g_q>
    const double sdot = sum(s, 0.0).re;
    const bool live = nrm >= 1e-12f;
    const float gnrm = live ? (float)(-sdot / ((double)nrm_c * nrm_c)) : 0.f;
    const float a = 1.f / nrm_c, bq = live ? gnrm * nrm_c / nrm : 0.f;  // g_u = a g_q + bq q
    for (int k = tid; k < sl.len; k += kThreads) {
      const float2 v = qi[k];
      gqi[k] = make_float2(a * gqi[k].x + bq * v.x, a * gqi[k].y + bq * v.y);
      u[k] = make_float2(v.x * nrm_c, v.y * nrm_c);
    }
    // walk j = i-1 .. 0 with u^(j) = u^(j+1) + c_ij q_j (u^(j) = u_prev of step j)
    for (int j = i - 1; j >= 0; --j) {
      const float2 cij = m.c[i * P + j];
      const float2* qj = q + j * qp;
      float2* gqj = gq + j * gp;
      double gr = 0.0, gim = 0.0;
      for (int k = tid; k < sl.len; k += kThreads) {
        const float2 t = cconjmul(qj[k], gqi[k]);  // conj(q_j) g_u
        gr += t.x;
        gim += t.y;
      }
      const Z gcs = sum(gr, gim);
      const float2 gc = make_float2((float)-gcs.re, (float)-gcs.im);  // g_c = -sum conj(q_j) g_u
      for (int k = tid; k < sl.len; k += kThreads) {
        const float2 v = qj[k];
        const float2 t0 = cmul_(cij, v);
        const float2 up = make_float2(u[k].x + t0.x, u[k].y + t0.y);
        u[k] = up;
        const float2 gu = gqi[k];
        // g_q_j += -conj(c) g_u + conj(g_c) u_prev
        const float2 t1 = cconjmul(cij, gu);
        const float2 t2 = cconjmul(gc, up);
        gqj[k] = make_float2(gqj[k].x - t1.x + t2.x, gqj[k].y - t1.y + t2.y);
        // g_u_prev = g_u + q_j g_c
        const float2 t3 = cmul_(v, gc);
        gqi[k] = make_float2(gu.x + t3.x, gu.y + t3.y);
      }
    }
    const float f = fac[i];
    const float2* pi = in + (int64_t)i * nn + sl.lo;
    float2* gi = grad_in + (int64_t)i * nn + sl.lo;
    for (int k = tid; k < sl.len; k += kThreads)
      gi[k] = make_float2(pi[k].x * f + gqi[k].x, pi[k].y * f + gqi[k].y);
  }
  cg::this_cluster().sync();  // no CTA leaves while a peer may still write its slots
}

constexpr size_t kSmemLimit = 232448 - 2048;  // dynamic shared memory beside the static arrays

template <typename K, typename... A>
cudaError_t launch_cluster(K kernel, int ctas, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// 16 CTAs (a non-portable cluster size) if the device can hold such a cluster with this much
// shared memory, else 8.  The kernel's shared-memory bound is the same in every call: it belongs
// to the device, and host threads that each set their own call's size would lower it between
// another's set and launch.
template <typename K>
bool fits_cluster(K kernel, int ctas, size_t smem) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit) != cudaSuccess ||
      cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (ctas <= 8) return true;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return n >= 1;
}

}  // namespace

extern "C" {

int64_t ptycho_probe_ortho_work_elems(int P, int64_t nn) {
  // q, gq, c, norms (float2 units) + the order (ints, rounded up to float2)
  return 2 * (int64_t)P * nn + (int64_t)P * P + 2 * P + (P + 1) / 2;
}

int ptycho_probe_orthogonalize(const void* probe, void* out, int P, int64_t nn, void* work, int64_t work_elems,
                               void* stream) {
  if (!probe || !out || !work || P < 1 || P > kMaxModes || nn < 1)
    return fail(PTYCHO_ERR_INVALID, "probe_orthogonalize: bad arguments (1 <= P <= %d)", kMaxModes);
  if (work_elems < ptycho_probe_ortho_work_elems(P, nn))
    return fail(PTYCHO_ERR_INVALID, "probe_orthogonalize: work needs %lld complex elements",
                (long long)ptycho_probe_ortho_work_elems(P, nn));
  if (probe == out) return fail(PTYCHO_ERR_INVALID, "probe_orthogonalize: out must not alias the input");
  // Windows above 128^2 have enough elements for 16 CTAs (forward / gradient, 8 against 16: six 256^2 modes
  // 143 / 199 us against 72 / 103); smaller ones are bound by the barriers (four 64^2 modes 26.7 / 26.7
  // against 28.8 / 27.0, four 128^2 modes 30.8 / 33.6 against 32.9 / 32.9; 4 CTAs 36.9 / 51.3)
  cudaError_t e = cudaErrorUnknown;
  for (int ctas = nn > 128 * 128 ? 16 : 8; ctas >= 8; ctas -= 8) {
    const size_t q = sizeof(float2) * (size_t)P * (size_t)((nn + ctas - 1) / ctas);
    const int q_shared = q <= kSmemLimit;
    if (!fits_cluster(probe_ortho_kernel, ctas, q_shared ? q : 0)) continue;
    e = launch_cluster(probe_ortho_kernel, ctas, q_shared ? q : 0, static_cast<cudaStream_t>(stream),
                       static_cast<const float2*>(probe), static_cast<float2*>(out), P, nn, static_cast<float2*>(work),
                       q_shared);
    break;
  }
  return e == cudaSuccess ? PTYCHO_OK : fail(PTYCHO_ERR_CUDA, "probe_ortho_kernel: %s", cudaGetErrorString(e));
}

int ptycho_probe_orthogonalize_vjp(const void* probe, const void* grad_sorted, void* grad_probe, int P, int64_t nn,
                                   void* work, int64_t work_elems, void* stream) {
  if (!probe || !grad_sorted || !grad_probe || !work || P < 1 || P > kMaxModes || nn < 1)
    return fail(PTYCHO_ERR_INVALID, "probe_orthogonalize_vjp: bad arguments (1 <= P <= %d)", kMaxModes);
  if (work_elems < ptycho_probe_ortho_work_elems(P, nn))
    return fail(PTYCHO_ERR_INVALID, "probe_orthogonalize_vjp: work needs %lld complex elements",
                (long long)ptycho_probe_ortho_work_elems(P, nn));
  // the kernel reads probe and grad_sorted while it writes grad_probe (restrict pointers)
  if (grad_probe == probe || grad_probe == grad_sorted || grad_probe == work)
    return fail(PTYCHO_ERR_INVALID, "probe_orthogonalize_vjp: grad_probe must not alias probe, grad_sorted or work");
  cudaError_t e = cudaErrorUnknown;
  for (int ctas = nn > 128 * 128 ? 16 : 8; ctas >= 8; ctas -= 8) {
    const size_t one = sizeof(float2) * (size_t)((nn + ctas - 1) / ctas);
    const int in_shared = one * (1 + 2 * P) <= kSmemLimit ? 3 : (one * (1 + P) <= kSmemLimit ? 2 : one <= kSmemLimit);
    const size_t smem = one * (in_shared == 3 ? 1 + 2 * P : (in_shared == 2 ? 1 + P : in_shared));
    if (!fits_cluster(probe_ortho_vjp_kernel, ctas, smem)) continue;
    e = launch_cluster(probe_ortho_vjp_kernel, ctas, smem, static_cast<cudaStream_t>(stream),
                       static_cast<const float2*>(probe), static_cast<const float2*>(grad_sorted),
                       static_cast<float2*>(grad_probe), P, nn, static_cast<float2*>(work), in_shared);
    break;
  }
  return e == cudaSuccess ? PTYCHO_OK : fail(PTYCHO_ERR_CUDA, "probe_ortho_vjp_kernel: %s", cudaGetErrorString(e));
}

}  // extern "C"
