// Host-side launch helpers shared by the per-size translation units.
#pragma once
#include <cuda_runtime.h>

#include "cluster_kernels.cuh"
#include "ptycho_b200.h"
#include "ptycho_kernels.cuh"

namespace qb {

inline BatchParams to_params(const ptycho_batch_args* a) {
  BatchParams p;
  p.obj = static_cast<const float2*>(a->obj);
  p.probe_hat = static_cast<const float2*>(a->probe_hat);
  p.prop = static_cast<const float2*>(a->prop);
  p.prop_r = static_cast<const float2*>(a->prop_r);
  p.prop_c = static_cast<const float2*>(a->prop_c);
  p.positions = a->positions;
  p.batch_idx = a->batch_idx;
  p.targets = a->targets;
  p.mask = a->mask;
  p.grad_obj = static_cast<float2*>(a->grad_obj);
  p.probe_grad_part = static_cast<float2*>(a->probe_grad_part);
  p.scratch = static_cast<float2*>(a->scratch);
  p.loss_part = a->loss_part;
  p.out_intensity = a->out_intensity;
  p.out_exit = static_cast<float2*>(a->out_exit);
  p.out_waves = static_cast<float2*>(a->out_waves);
  p.status = a->status;
  p.S = a->S;
  p.P = a->P;
  p.B = a->B;
  p.Ho = a->Ho;
  p.Wo = a->Wo;
  p.npos = a->npos;
  p.loss_scale = a->loss_scale;
  p.inv_mean_intensity = a->inv_mean_intensity;
  p.loss_type = a->loss_type;
  p.analytic = a->analytic;
  p.an_norm = a->an_norm;
  p.ckpt = a->recompute_every;
  p.grad_positions = a->grad_positions;
  p.descan = a->descan;
  p.grad_descan = a->grad_descan;
  p.grad_prop = a->grad_prop;
  p.sep_shared = 0;
  p.tile_out = 0;
  return p;
}

// dynamic shared memory of a launch with (tile) or without the intensity tile in it
template <int N>
size_t batch_smem(const ptycho_batch_args* a, bool tile = true) {
  return batch_smem_bytes<N>(tile, a->prop_r != nullptr && sep_in_smem<N>(tile, a->S), a->S);
}
// smallest shared-memory carve-out (percent) that holds the resident CTAs: the rest is L1
template <int N>
int carveout(size_t smem) {
  const size_t pc = Fft2<N>::CTAS * (smem + 2048) * 100 / (228 * 1024) + 1;
  return pc < 100 ? (int)pc : 100;
}
template <int N>
BatchParams batch_params(const ptycho_batch_args* a, bool tile = true, bool tile_out = false) {
  BatchParams p = to_params(a);
  p.tile_out = tile_out;
  p.sep_shared = sep_in_smem<N>(tile, a->S);
  return p;
}

// Dynamic shared memory that a batch kernel may be launched with: one bound for all of its calls,
// whatever the call at hand takes.  The attribute belongs to the device, so a bound of each call's
// own size could be lowered by another host thread before the launch.
template <typename K>
bool allow_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) == cudaSuccess;
}

// the serial kernel with its optional extensions compiled in (descan, position / descan /
// propagator gradients)
inline bool wants_ext(const ptycho_batch_args* a) {
  return a->descan || a->grad_descan || a->grad_prop || a->grad_positions;
}

template <int N, bool ADJ>
int launch_ext(const BatchParams& p, int grid, size_t smem, cudaStream_t st) {
  if (!allow_smem(fused_batch_kernel<N, ADJ, false, true>)) return PTYCHO_ERR_CUDA;
  if (ADJ)
    cudaFuncSetAttribute(fused_batch_kernel<N, ADJ, false, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         carveout<N>(smem));
  fused_batch_kernel<N, ADJ, false, true><<<grid, Fft2<N>::T, smem, st>>>(p);
  return PTYCHO_OK;
}

// Where the forward kernel sums the mode intensities.  One mode: nowhere, it goes straight through the loss.
// Several: a tile in shared memory if it fits beside the separable factors without costing a resident
// CTA, else the output array if there is one.
template <int N>
bool forward_tile(const ptycho_batch_args* a) {
  if (a->P == 1) return false;
  return !a->out_intensity || batch_smem_bytes<N>(true, a->prop_r != nullptr, a->S) <= max_smem<N>(Fft2<N>::CTAS);
}

// One CTA per position, modes in sequence.  The attributes are per device; setting them on
// every launch keeps multi-device processes correct and costs far less than one launch.
// The adjoint kernels take the smallest shared-memory carve-out that fits: the rest of the
// 256 KB is L1.
template <int N>
int launch_plain(const ptycho_batch_args* a, bool adj, cudaStream_t st) {
  const bool tile = !adj && forward_tile<N>(a);
  const BatchParams p = batch_params<N>(a, tile, !adj && !tile);
  const size_t smem = batch_smem<N>(a, tile);
  if (adj) {
    if (!allow_smem(fused_batch_kernel<N, true>)) return PTYCHO_ERR_CUDA;
    cudaFuncSetAttribute(fused_batch_kernel<N, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         carveout<N>(smem));
    fused_batch_kernel<N, true><<<a->grid, Fft2<N>::T, smem, st>>>(p);
  } else {
    if (!allow_smem(fused_batch_kernel<N, false>)) return PTYCHO_ERR_CUDA;
    fused_batch_kernel<N, false><<<a->grid, Fft2<N>::T, smem, st>>>(p);
  }
  return cudaPeekAtLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

// the instances with the analytic update or with extensions
template <int N>
int launch_special(const ptycho_batch_args* a, bool adj, cudaStream_t st) {
  const bool tile = !adj && forward_tile<N>(a);
  const BatchParams p = batch_params<N>(a, tile, !adj && !tile);
  const size_t smem = batch_smem<N>(a, tile);
  if (!a->analytic) {
    const int rc = adj ? launch_ext<N, true>(p, a->grid, smem, st) : launch_ext<N, false>(p, a->grid, smem, st);
    if (rc) return rc;
  } else {
    if (!allow_smem(fused_batch_kernel<N, true, true>)) return PTYCHO_ERR_CUDA;
    cudaFuncSetAttribute(fused_batch_kernel<N, true, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         carveout<N>(smem));
    fused_batch_kernel<N, true, true><<<a->grid, Fft2<N>::T, smem, st>>>(p);
  }
  return cudaPeekAtLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

inline bool wants_special(const ptycho_batch_args* a) { return a->analytic || wants_ext(a); }

template <int N>
int launch_serial(const ptycho_batch_args* a, bool adj, cudaStream_t st) {
  return wants_special(a) ? launch_special<N>(a, adj, st) : launch_plain<N>(a, adj, st);
}

// several datasets in one persistent launch (serial body, adjoint)
template <int N>
int launch_multi(const ptycho_batch_args* sets, int nsets, cudaStream_t st) {
  MultiParams mp;
  mp.nd = nsets;
  mp.begin[0] = 0;
  size_t smem = 0;
  for (int d = 0; d < nsets; ++d) {
    mp.d[d] = batch_params<N>(&sets[d], false);
    mp.begin[d + 1] = mp.begin[d] + sets[d].grid;
    const size_t sd = batch_smem<N>(&sets[d], false);
    if (sd > smem) smem = sd;
  }
  if (!allow_smem(multi_batch_kernel<N, true>)) return PTYCHO_ERR_CUDA;
  cudaFuncSetAttribute(multi_batch_kernel<N, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                       carveout<N>(smem));
  multi_batch_kernel<N, true><<<mp.begin[nsets], Fft2<N>::T, smem, st>>>(mp);
  return cudaPeekAtLastError() == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

template <int N, bool ADJ>
cudaLaunchConfig_t cluster_config(const ptycho_batch_args* a, int grid, cudaStream_t st, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3(Fft2<N>::T, 1, 1);
  cfg.dynamicSmemBytes = batch_smem<N>(a);
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)a->P;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Number of clusters of P CTAs that can be resident at once.
template <int N>
int max_clusters(const ptycho_batch_args* a, bool adj) {
  cudaLaunchAttribute attr[1];
  int n = 0;
  cudaError_t e;
  if (adj) {
    e = allow_smem(cluster_batch_kernel<N, true>) ? cudaSuccess : cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = cluster_config<N, true>(a, a->P, nullptr, attr);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, cluster_batch_kernel<N, true>, &cfg);
  } else {
    e = allow_smem(cluster_batch_kernel<N, false>) ? cudaSuccess : cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = cluster_config<N, false>(a, a->P, nullptr, attr);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, cluster_batch_kernel<N, false>, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return n;
}

template <int N>
int launch_cluster(const ptycho_batch_args* a, bool adj, cudaStream_t st) {
  const BatchParams p = batch_params<N>(a);
  cudaLaunchAttribute attr[1];
  cudaError_t e;
  if (adj) {
    if (!allow_smem(cluster_batch_kernel<N, true>)) return PTYCHO_ERR_CUDA;
    cudaFuncSetAttribute(cluster_batch_kernel<N, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)((batch_smem<N>(a) + 1024) * 100 / (228 * 1024) + 1));
    cudaLaunchConfig_t cfg = cluster_config<N, true>(a, a->grid, st, attr);
    e = cudaLaunchKernelEx(&cfg, cluster_batch_kernel<N, true>, p);
  } else {
    if (!allow_smem(cluster_batch_kernel<N, false>)) return PTYCHO_ERR_CUDA;
    cudaLaunchConfig_t cfg = cluster_config<N, false>(a, a->grid, st, attr);
    e = cudaLaunchKernelEx(&cfg, cluster_batch_kernel<N, false>, p);
  }
  return e == cudaSuccess ? PTYCHO_OK : PTYCHO_ERR_CUDA;
}

}  // namespace qb
