// Serial-mode batch kernels for a 128 x 128 probe window with the analytic update or the
// optional extensions.  They sit at 128 registers with more live values than the plain
// kernels: packed products cost them spills (analytic 160 -> 360 bytes, 895 -> 927 us per
// 400 positions), so only additions and the middle-stage twiddles are packed.
#define QB_F32X2_ADD 1
#define QB_F32X2_S2 1
#include "launch_impl.cuh"

int qb_launch_special_128(const ptycho_batch_args* a, bool adj, cudaStream_t st) {
  return qb::launch_special<128>(a, adj, st);
}
