// Serial-mode batch kernels instantiated for a 128 x 128 probe window: the plain forward and
// adjoint kernels.  Complex arithmetic on packed FP32 pairs (fft_engine.cuh): 25.7 -> 24.8 ms
// per 4096-position launch (8 slices, 4 modes) against packed additions and middle-stage
// twiddles only.
#define QB_F32X2_ADD 1
#define QB_F32X2_MUL 1
#include "launch_impl.cuh"

// defined in fused_n128x.cu
int qb_launch_special_128(const ptycho_batch_args* a, bool adj, cudaStream_t st);

int qb_launch_serial_128(const ptycho_batch_args* a, bool adj, cudaStream_t st) {
  return qb::wants_special(a) ? qb_launch_special_128(a, adj, st) : qb::launch_plain<128>(a, adj, st);
}
