// Learned-initialiser CNN: the tcgen05 BF16 GEMM launcher and the NHWC layer
// kernels around it (im2col with circular padding, transposed-convolution
// gather/scatter, batch-norm statistics and application, ReLU masks, 2x2 max
// pooling, transposes, casts, MSE loss).  Every function here is part of the C
// ABI declared in include/ptycho_b200.h.
//
// Layout: an activation of shape (B, C, H, W) is stored channels-last as a
// row-major matrix with R = B*H*W rows (row r = (b*H + y)*W + x) and a leading
// dimension ld >= C, so a channel slice of a wider buffer (skip concatenation)
// is addressed by a column offset and the wider ld.
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>

#include <mutex>

#include "cnn_bn.cuh"
#include "gemm_tcgen05.cuh"
#include "ptycho_b200.h"

int qb_record_error(int code, const char* msg);

namespace {

using bf16 = __nv_bfloat16;

int fail(int code, const char* fmt, ...) {
  char buf[400];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  return qb_record_error(code, buf);
}
int check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(PTYCHO_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
  return PTYCHO_OK;
}
constexpr int kSms = 148;
bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
int blocks_for(int64_t n, int threads, int cap = 148 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  return static_cast<int>(b < cap ? b : cap);
}

// ---------------------------------------------------------------------------
// GEMM launcher
// ---------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

int encode_fn() {
  std::call_once(g_encode_once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  return g_encode ? PTYCHO_OK : fail(PTYCHO_ERR_CUDA, "gemm: cuTensorMapEncodeTiled is not available");
}

// Row-major bf16 matrix [rows][ld], `cols` used -> 2-D tensor map with a box of 64 columns x
// box_rows and the 128-byte swizzle (K-major: rows x k; MN-major: k x rows, 64 k per box).
int make_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows) {
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(qb::gemm::BK), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? PTYCHO_OK : fail(PTYCHO_ERR_INVALID, "gemm: tensor map encode failed (%d)", (int)r);
}

template <int BN, bool A_MN, bool B_MN, bool DEEP>
int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, int splits, int kb_per, int a_rows,
                const qb::gemm::Epilogue& epi, int* status, cudaStream_t st) {
  using L = qb::gemm::Smem<BN, DEEP>;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(qb::gemm::gemm_bf16_kernel<BN, A_MN, B_MN, DEEP>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
  });
  if (attr != cudaSuccess) return fail(PTYCHO_ERR_CUDA, "gemm: smem attribute: %s", cudaGetErrorString(attr));
  dim3 grid((M + qb::gemm::BM - 1) / qb::gemm::BM, (N + BN - 1) / BN, splits);
  qb::gemm::gemm_bf16_kernel<BN, A_MN, B_MN, DEEP>
      <<<grid, qb::gemm::THREADS, L::BYTES, st>>>(ta, tb, M, N, K, kb_per, a_rows, epi, status);
  return check_launch("gemm_bf16_kernel");
}

// An operand of the product: rows of K values (K-major), or K rows of its values (mn).
struct Operand {
  const void* p;
  int ld;
  bool mn;
};

// Tile width and ring of a product of M x N, `splits` parts of K and a_rows rows of A per tile.
//
// A CTA's time goes with the rows that its copies bring per k-block, a_rows + BN, and the tiles are
// worked off in rounds of one per SM: the width with the fewest rounds x (a_rows + BN), the widest of
// equals.  16384 x 32 x 9216: 58 us as 128 CTAs of 32 columns, 98 as 256 of 16 in two rounds;
// 16 x 1024 x 9216: 29 us at 16 columns, 46 at 128.  In several rounds two CTAs share an SM (widths 32
// and 64 with a ring of four k-blocks), so that one's epilogue runs beside the other's copies: 65536 x
// 32 x 288 takes 19 us, 31 with the deep ring; 20000 x 32 x 288 (157 CTAs) 12.5 against 17.  In one round
// the deep ring is the faster: 18944 x 32 x 2304 (148 CTAs) 17 us against 19.  16 columns only in one
// round: 262144 x 16 x 144 took 66 us with them, 40 with 32 columns.
// A column's products and sums do not depend on the tile width.  MN-major B tiles are copied in boxes of
// 64 columns.
struct Tile {
  int bn;
  int64_t ctas;
  bool deep;
};
Tile tile_of(int M, int N, int splits, int a_rows, bool b_mn) {
  const int64_t tiles_m = (M + qb::gemm::BM - 1) / qb::gemm::BM * (int64_t)splits;
  const int least = b_mn ? 64 : 16;
  int widest = N <= 32 ? 32 : (N <= 64 ? 64 : 128);
  if (widest < least) widest = least;
  Tile t{0, 0, true};
  int64_t best = 0;
  for (int w = widest; w >= least; w /= 2) {
    const int64_t n = tiles_m * ((N + w - 1) / w), cost = (n + kSms - 1) / kSms * (a_rows + w);
    if (w == 16 && n > kSms) break;
    if (t.bn == 0 || cost < best) t = {w, n, true}, best = cost;
  }
  t.deep = b_mn || t.bn == 16 || t.bn == 128 || t.ctas <= kSms;
  return t;
}
int rows_of_a(int M, bool a_mn) { return a_mn || M >= qb::gemm::BM ? qb::gemm::BM : (M + 7) / 8 * 8; }

int gemm_run(const Operand& A, const Operand& B, void* C, int ldc, int M, int N, int K, const float* bias, int flags,
             int splits, int* status, cudaStream_t st) {
  using namespace qb::gemm;
  if (!A.p || !B.p || !C || M < 1 || N < 1 || K < 1 || A.ld < (A.mn ? M : K) || B.ld < (B.mn ? N : K) || ldc < N)
    return fail(PTYCHO_ERR_INVALID, "gemm: bad sizes (M=%d N=%d K=%d lda=%d ldb=%d ldc=%d)", M, N, K, A.ld, B.ld, ldc);
  if ((A.ld & 7) || (B.ld & 7) || !al16(A.p) || !al16(B.p))
    return fail(PTYCHO_ERR_INVALID, "gemm: A/B must be 16-byte aligned with leading dimensions a multiple of 8");
  if (flags & ~(EPI_BF16 | EPI_RELU | EPI_ATOMIC | EPI_ACT_MASK))
    return fail(PTYCHO_ERR_INVALID, "gemm: unknown flags %d", flags);
  int act = (flags & EPI_ACT_MASK) >> EPI_ACT_SHIFT;
  if (act >= qb::ACT_COUNT || ((flags & EPI_RELU) && act && act != qb::ACT_RELU))
    return fail(PTYCHO_ERR_INVALID, "gemm: bad activation in flags %d", flags);
  if (flags & EPI_RELU) act = qb::ACT_RELU;
  const int nkb = (K + BK - 1) / BK;
  if (splits < 1) splits = 1;
  if (splits > nkb) splits = nkb;
  const bool accumulate = (flags & EPI_ATOMIC) != 0;  // add into C as it is
  if (splits > 1) flags |= EPI_ATOMIC;
  if ((flags & EPI_ATOMIC) && ((flags & EPI_BF16) || act))
    return fail(PTYCHO_ERR_INVALID, "gemm: split-K / atomic output needs FP32 output without an activation");
  if (int rc = encode_fn()) return rc;
  const int kb_per = (nkb + splits - 1) / splits;
  splits = (nkb + kb_per - 1) / kb_per;  // every split gets >= 1 k-block
  const int a_rows = rows_of_a(M, A.mn);
  const Tile t = tile_of(M, N, splits, a_rows, B.mn);
  const int BN = t.bn;
  CUtensorMap ta, tb;
  if (int rc = A.mn ? make_map(&ta, A.p, K, M, A.ld, BK) : make_map(&ta, A.p, M, K, A.ld, a_rows)) return rc;
  if (int rc = B.mn ? make_map(&tb, B.p, K, N, B.ld, BK) : make_map(&tb, B.p, N, K, B.ld, BN)) return rc;
  if (!accumulate && splits > 1) {
    if (cudaMemset2DAsync(C, (size_t)ldc * 4, 0, (size_t)N * 4, (size_t)M, st) != cudaSuccess)
      return check_launch("gemm: clear split-K output");
  }
  const Epilogue epi{C, bias, ldc, flags, act};
#define QB_GEMM(bn, a, b, deep) \
  return launch_gemm<bn, a, b, deep>(ta, tb, M, N, K, splits, kb_per, a_rows, epi, status, st)
  if (A.mn && B.mn) {
    if (BN == 64) QB_GEMM(64, true, true, true);
    QB_GEMM(128, true, true, true);
  }
  if (B.mn) {
    if (BN == 64) QB_GEMM(64, false, true, true);
    QB_GEMM(128, false, true, true);
  }
  if (A.mn) return fail(PTYCHO_ERR_UNSUPPORTED, "gemm: an MN-major A goes with an MN-major B");
  if (!t.deep) {
    if (BN == 32) QB_GEMM(32, false, false, false);
    QB_GEMM(64, false, false, false);
  }
  switch (BN) {
    case 16: QB_GEMM(16, false, false, true);
    case 32: QB_GEMM(32, false, false, true);
    case 64: QB_GEMM(64, false, false, true);
    default: QB_GEMM(128, false, false, true);
  }
#undef QB_GEMM
}

// ---------------------------------------------------------------------------
// layer kernels
// ---------------------------------------------------------------------------
__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// col[r][(ky*3 + kx)*C + c] = x[b, (y+ky-1) mod H, (x+kx-1) mod W, c]; 8 channels per thread.
__global__ void im2col3x3_kernel(const bf16* __restrict__ x, int B, int H, int W, int C, int ldx,
                                 bf16* __restrict__ col, int ldcol) {
  const int c8 = C >> 3;
  const int64_t total = (int64_t)B * H * W * 9 * c8;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int cv = (int)(i % c8);
    int64_t t = i / c8;
    const int tap = (int)(t % 9);
    const int64_t r = t / 9;
    const int xx = (int)(r % W), yy = (int)((r / W) % H), b = (int)(r / ((int64_t)W * H));
    const int sy = wrap(yy + tap / 3 - 1, H), sx = wrap(xx + tap % 3 - 1, W);
    const uint4 v = *reinterpret_cast<const uint4*>(x + ((int64_t)(b * H + sy) * W + sx) * ldx + cv * 8);
    *reinterpret_cast<uint4*>(col + r * ldcol + tap * C + cv * 8) = v;
  }
}

// dx[b, y, x, c] (+)= sum_tap dcol[(b, (y-ky+1) mod H, (x-kx+1) mod W)][tap*C + c]; 4 channels per thread.
__global__ void col2im3x3_kernel(const float* __restrict__ dcol, int ldcol, int B, int H, int W, int C,
                                 float* __restrict__ dx, int ldx, int accumulate) {
  const int c4 = C >> 2;
  const int64_t total = (int64_t)B * H * W * c4;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int cv = (int)(i % c4);
    const int64_t r = i / c4;
    const int xx = (int)(r % W), yy = (int)((r / W) % H), b = (int)(r / ((int64_t)W * H));
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const int sy = wrap(yy - tap / 3 + 1, H), sx = wrap(xx - tap % 3 + 1, W);
      const float4 v =
          *reinterpret_cast<const float4*>(dcol + ((int64_t)(b * H + sy) * W + sx) * ldcol + tap * C + cv * 4);
      acc.x += v.x;
      acc.y += v.y;
      acc.z += v.z;
      acc.w += v.w;
    }
    float4* o = reinterpret_cast<float4*>(dx + r * ldx + cv * 4);
    if (accumulate) {
      const float4 p = *o;
      acc.x += p.x;
      acc.y += p.y;
      acc.z += p.z;
      acc.w += p.w;
    }
    *o = acc;
  }
}

// Transposed convolution 3x3, stride 2, padding 1, output padding 1 (zero padded):
// out[b, oy, ox, co] = bias[co] + sum over taps with oy = 2 iy - 1 + ky, ox = 2 ix - 1 + kx
// of colT[(b, iy, ix)][(ky*3 + kx)*Co + co].  Output (B, 2H, 2W, Co) in bf16.
__global__ void convT_gather_kernel(const float* __restrict__ colT, int ldcol, int B, int H, int W, int Co,
                                    const float* __restrict__ bias, bf16* __restrict__ out, int ldo) {
  const int H2 = 2 * H, W2 = 2 * W;
  const int64_t total = (int64_t)B * H2 * W2 * Co;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int co = (int)(i % Co);
    const int64_t r = i / Co;
    const int ox = (int)(r % W2), oy = (int)((r / W2) % H2), b = (int)(r / ((int64_t)W2 * H2));
    float acc = bias ? bias[co] : 0.0f;
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      const int ty = oy + 1 - ky;
      if (ty < 0 || (ty & 1)) continue;
      const int iy = ty >> 1;
      if (iy >= H) continue;
#pragma unroll
      for (int kx = 0; kx < 3; ++kx) {
        const int tx = ox + 1 - kx;
        if (tx < 0 || (tx & 1)) continue;
        const int ix = tx >> 1;
        if (ix >= W) continue;
        acc += colT[((int64_t)(b * H + iy) * W + ix) * ldcol + (ky * 3 + kx) * Co + co];
      }
    }
    out[r * ldo + co] = __float2bfloat16_rn(acc);
  }
}

// Backward of the transposed convolution's scatter:
// dcol[(b, iy, ix)][(ky*3+kx)*Co + co] = dout[b, 2iy-1+ky, 2ix-1+kx, co] (0 outside), bf16.
__global__ void convT_im2col_kernel(const float* __restrict__ dout, int ldo, int B, int H, int W, int Co,
                                    bf16* __restrict__ dcol, int ldcol) {
  const int H2 = 2 * H, W2 = 2 * W;
  const int64_t total = (int64_t)B * H * W * 9 * Co;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int co = (int)(i % Co);
    int64_t t = i / Co;
    const int tap = (int)(t % 9);
    const int64_t r = t / 9;
    const int ix = (int)(r % W), iy = (int)((r / W) % H), b = (int)(r / ((int64_t)W * H));
    const int oy = 2 * iy - 1 + tap / 3, ox = 2 * ix - 1 + tap % 3;
    float v = 0.0f;
    if (oy >= 0 && oy < H2 && ox >= 0 && ox < W2) v = dout[((int64_t)(b * H2 + oy) * W2 + ox) * ldo + co];
    dcol[r * ldcol + tap * Co + co] = __float2bfloat16_rn(v);
  }
}

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<bf16>(bf16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ bf16 from_f<bf16>(float v) { return __float2bfloat16_rn(v); }

// out[z][c][r] = in[z][r][c] (32 x 32 tiles through shared memory), batched over z.
template <typename Ti, typename To>
__global__ void transpose_kernel(const Ti* __restrict__ in, int R, int C, int ldi, int64_t zsi, To* __restrict__ out,
                                 int ldo, int64_t zso) {
  __shared__ float tile[32][33];
  in += blockIdx.z * zsi;
  out += blockIdx.z * zso;
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int r = r0 + j, c = c0 + threadIdx.x;
    tile[j][threadIdx.x] = (r < R && c < C) ? to_f<Ti>(in[(int64_t)r * ldi + c]) : 0.0f;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int c = c0 + j, r = r0 + threadIdx.x;
    if (c < C && r < R) out[(int64_t)c * ldo + r] = from_f<To>(tile[threadIdx.x][j]);
  }
}

// Deterministic column sums over the rows of an FP32 matrix, in two passes: per-chunk
// partials (double) then a fixed-order sum per column.
constexpr int kColThreads = 256;
__global__ void colsum_partial_kernel(const float* __restrict__ a, int lda, int R, int C, int rows_per_chunk,
                                      double* __restrict__ part) {
  __shared__ double red0[kColThreads];
  const int TC = C < kColThreads ? C : kColThreads;
  const int RP = kColThreads / TC;
  const int tx = threadIdx.x % TC, ty = threadIdx.x / TC;
  const int c = blockIdx.y * TC + tx;
  const int r0 = blockIdx.x * rows_per_chunk, r1 = min(R, r0 + rows_per_chunk);
  double s0 = 0.0;
  if (ty < RP && c < C) {
    float f0 = 0.f;
    int cnt = 0;
    for (int r = r0 + ty; r < r1; r += RP) {
      f0 += a[(int64_t)r * lda + c];
      if (++cnt == 64) {  // flush to double every 64 rows
        s0 += f0;
        f0 = 0.f;
        cnt = 0;
      }
    }
    s0 += f0;
  }
  red0[threadIdx.x] = s0;
  __syncthreads();
  if (ty == 0 && c < C) {
    for (int k = 1; k < RP; ++k) s0 += red0[k * TC + tx];
    part[(int64_t)blockIdx.x * C + c] = s0;
  }
}

__global__ void colsum_final_kernel(const double* __restrict__ part, int nchunks, int C, float* out, int accumulate) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  double s0 = 0.0;
  for (int k = 0; k < nchunks; ++k) s0 += part[(int64_t)k * C + c];
  out[c] = accumulate ? out[c] + (float)s0 : (float)s0;
}

// y = bf16(x) (layers without batch norm)
__global__ void to_bf16_kernel(const float* __restrict__ x, int ldx, int R, int C, bf16* __restrict__ y, int ldy) {
  const int64_t total = (int64_t)R * C;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const int64_t r = i / C;
    y[r * ldy + c] = __float2bfloat16_rn(x[r * ldx + c]);
  }
}

// 2x2 max pool, stride 2 (H, W even); argmax code (dy*2 + dx) of the first maximum in
// row-major window order, as torch's max_pool2d picks it.
__global__ void maxpool2_kernel(const bf16* __restrict__ in, int ldi, int B, int H, int W, int C,
                                bf16* __restrict__ out, int ldo, uint8_t* __restrict__ arg) {
  const int Ho = H / 2, Wo = W / 2;
  const int64_t total = (int64_t)B * Ho * Wo * C;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const int64_t r = i / C;
    const int ox = (int)(r % Wo), oy = (int)((r / Wo) % Ho), b = (int)(r / ((int64_t)Wo * Ho));
    float best = -INFINITY;
    int code = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int y = 2 * oy + (k >> 1), x = 2 * ox + (k & 1);
      const float v = __bfloat162float(in[((int64_t)(b * H + y) * W + x) * ldi + c]);
      if (k == 0 || v > best) {
        best = v;
        code = k;
      }
    }
    out[r * ldo + c] = __float2bfloat16_rn(best);
    arg[r * C + c] = (uint8_t)code;
  }
}

// din[b, y, x, c] (+)= dout[b, y/2, x/2, c] if (y, x) held the window maximum, else 0.
__global__ void maxpool2_backward_kernel(const float* __restrict__ dout, int lddo, const uint8_t* __restrict__ arg,
                                         int B, int H, int W, int C, float* __restrict__ din, int lddi,
                                         int accumulate) {
  const int Wo = W / 2, Ho = H / 2;
  const int64_t total = (int64_t)B * H * W * C;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const int64_t r = i / C;
    const int x = (int)(r % W), y = (int)((r / W) % H), b = (int)(r / ((int64_t)W * H));
    const int64_t ro = (int64_t)(b * Ho + y / 2) * Wo + x / 2;
    const float g = (arg[ro * C + c] == (uint8_t)(((y & 1) << 1) | (x & 1))) ? dout[ro * lddo + c] : 0.0f;
    float* o = din + r * lddi + c;
    *o = accumulate ? *o + g : g;
  }
}

__global__ void cast_bf16_kernel(const float* __restrict__ in, bf16* __restrict__ out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16_rn(in[i]);
}

// Mean squared error over n values: partial sums of (p - t)^2 per block (double) and
// dp = 2 (p - t) / n in FP32 and BF16.
__global__ void mse_kernel(const float* __restrict__ p, const float* __restrict__ t, int64_t n,
                           double* __restrict__ part, float* __restrict__ dp32, bf16* __restrict__ dp16) {
  __shared__ double red[256];
  double s = 0.0;
  const float sc = 2.0f / (float)n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float d = p[i] - t[i];
    s += (double)d * d;
    if (dp32) dp32[i] = sc * d;
    if (dp16) dp16[i] = __float2bfloat16_rn(sc * d);
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}
__global__ void mse_final_kernel(const double* part, int nparts, int64_t n, float* loss) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < nparts; ++i) s += part[i];
    *loss = (float)(s / (double)n);
  }
}

// Network input features from diffraction data: per scan position p and bin (u, v)
// of a bin x bin block, f = sqrt(norm * sum of the block's intensities) (amplitudes
// are squared first), then (f - mean[u*nb + v]) * scale, written as BF16 row p.
__global__ void bin_features_kernel(const float* __restrict__ pat, int npos, int n, int bin, int amplitudes,
                                    float norm, const float* __restrict__ mean, float scale, bf16* __restrict__ out,
                                    int ldo) {
  const int nb = n / bin;
  const int64_t total = (int64_t)npos * nb * nb;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % (nb * nb));
    const int64_t p = i / (nb * nb);
    const int u = c / nb, v = c % nb;
    const float* src = pat + p * n * n + (int64_t)(u * bin) * n + v * bin;
    float s = 0.0f;
    for (int a = 0; a < bin; ++a)
      for (int b = 0; b < bin; ++b) {
        const float x = src[a * n + b];
        s += amplitudes ? x * x : x;
      }
    float f = sqrtf(fmaxf(s * norm, 0.0f));
    if (mean) f -= mean[c];
    out[p * ldo + c] = __float2bfloat16_rn(f * scale);
  }
}

constexpr int kMseBlocks = 296;

int work_check(int C, int64_t work_elems) {
  if (work_elems < 2 * (int64_t)C)
    return fail(PTYCHO_ERR_INVALID, "cnn: reduction workspace too small (%lld doubles for C=%d)",
                (long long)work_elems, C);
  return PTYCHO_OK;
}

int colsum(const float* a, int lda, int R, int C, double* work, int64_t work_elems, float* out, int accumulate,
           cudaStream_t st) {
  if (int rc = work_check(C, work_elems)) return rc;
  const int TC = C < kColThreads ? C : kColThreads;
  const int RP = kColThreads / TC;
  int chunks = (R + RP * 16 - 1) / (RP * 16);
  if (chunks > 592) chunks = 592;
  if ((int64_t)chunks * 2 * C > work_elems) chunks = (int)(work_elems / (2 * (int64_t)C));
  const int rpc = (R + chunks - 1) / chunks;
  chunks = (R + rpc - 1) / rpc;
  dim3 grid(chunks, (C + TC - 1) / TC);
  colsum_partial_kernel<<<grid, kColThreads, 0, st>>>(a, lda, R, C, rpc, work);
  if (int rc = check_launch("colsum_partial_kernel")) return rc;
  colsum_final_kernel<<<(C + 127) / 128, 128, 0, st>>>(work, chunks, C, out, accumulate);
  return check_launch("colsum_final_kernel");
}

int bn_check(const qb::bn::Forward& f, int R, int C) {
  if (!f.x || !f.y || R < 1 || C < 1 || f.ldx < C || f.ldy < C)
    return fail(PTYCHO_ERR_INVALID, "bn_forward: bad arguments");
  if (f.gamma && (!f.beta || !f.mean || !f.rstd || (f.run_mean && !f.run_var) || (!f.training && !f.run_mean)))
    return fail(PTYCHO_ERR_INVALID, "bn_forward: missing statistics buffers");
  return PTYCHO_OK;
}
int bn_check(const qb::bn::Backward& b, int R, int C) {
  if (!b.dy || !b.x || R < 1 || C < 1 || b.lddy < C || b.ldx < C || b.ldz < C || (!b.dz32 && !b.dz16) || b.act < 0 ||
      b.act >= qb::ACT_COUNT)
    return fail(PTYCHO_ERR_INVALID, "bn_backward: bad arguments");
  if (b.gamma && (!b.mean || !b.rstd || !b.dgamma || !b.dbeta))
    return fail(PTYCHO_ERR_INVALID, "bn_backward: missing buffers");
  return PTYCHO_OK;
}
// work: scratch for the partial sums of many rows (may be NULL or too small: the cluster launch runs)
bool bn_wide(int R, int C, bool forward, bool sums, const double* work, int64_t work_elems) {
  return qb::bn::wide(R, forward && sums) && (!sums || (work && (reinterpret_cast<uintptr_t>(work) & 7) == 0 &&
                                          work_elems >= qb::bn::wide_elems(R, C)));
}
int bn_forward(const qb::bn::Forward& f, int R, int C, double* work, int64_t work_elems, cudaStream_t st) {
  if (int rc = bn_check(f, R, C)) return rc;
  if (!f.gamma) {
    to_bf16_kernel<<<blocks_for((int64_t)R * C, 256), 256, 0, st>>>(f.x, f.ldx, R, C, f.y, f.ldy);
    return check_launch("to_bf16_kernel");
  }
  const cudaError_t e = bn_wide(R, C, true, f.training, work, work_elems)
                            ? qb::bn::launch_wide(f, R, C, work, st)
                            : qb::bn::launch(qb::bn::bn_forward_kernel, f, R, C, st);
  return e == cudaSuccess ? PTYCHO_OK : fail(PTYCHO_ERR_CUDA, "bn_forward_kernel: %s", cudaGetErrorString(e));
}
int bn_backward(const qb::bn::Backward& b, int R, int C, double* work, int64_t work_elems, cudaStream_t st) {
  if (int rc = bn_check(b, R, C)) return rc;
  const cudaError_t e = bn_wide(R, C, false, b.gamma || b.dbias, work, work_elems)
                            ? qb::bn::launch_wide(b, R, C, work, st)
                            : qb::bn::launch(qb::bn::bn_backward_kernel, b, R, C, st);
  return e == cudaSuccess ? PTYCHO_OK : fail(PTYCHO_ERR_CUDA, "bn_backward_kernel: %s", cudaGetErrorString(e));
}

}  // namespace

// Dropout (nn.Dropout, blocks.py:134-135): x *= keep / (1 - p) with keep = u >= p, u a
// uniform draw per element from a counter-based hash of (seed, row * C + column) -- the
// SplitMix64 finaliser (Steele, Lea and Flood, 2014) -- so the backward regenerates the
// forward's mask from the same seed instead of storing it.
__device__ __forceinline__ float dropout_uniform(uint64_t seed, uint64_t i) {
  uint64_t z = seed + (i + 1) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (float)(z >> 40) * (1.0f / 16777216.0f);  // 24 random bits in [0, 1)
}

template <typename T>
__global__ void dropout_kernel(T* __restrict__ x, int R, int C, int ld, float p, float scale, uint64_t seed) {
  const int64_t total = (int64_t)R * C;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / C;
    const int c = (int)(i % C);
    const bool keep = dropout_uniform(seed, (uint64_t)i) >= p;
    T* e = x + r * ld + c;
    if constexpr (sizeof(T) == 4) {
      *e = keep ? *e * scale : 0.0f;
    } else {
      *e = keep ? __float2bfloat16_rn(__bfloat162float(*e) * scale) : __float2bfloat16_rn(0.0f);
    }
  }
}

// ===========================================================================
// C ABI
// ===========================================================================
extern "C" {

int ptycho_gemm_bf16(const void* A, int lda, const void* B, int ldb, void* C, int ldc, int M, int N, int K,
                     const float* bias, int flags, int splits, int* status, void* stream) {
  return gemm_run({A, lda, false}, {B, ldb, false}, C, ldc, M, N, K, bias, flags, splits, status,
                  static_cast<cudaStream_t>(stream));
}

int ptycho_gemm_plan(int M, int N, int K, int splits, int a_mn, int b_mn, int* tile_n, int64_t* ctas, int* ctas_per_sm) {
  if (M < 1 || N < 1 || K < 1 || (a_mn && !b_mn)) return fail(PTYCHO_ERR_INVALID, "gemm_plan: bad arguments");
  const int nkb = (K + qb::gemm::BK - 1) / qb::gemm::BK;
  splits = splits < 1 ? 1 : (splits > nkb ? nkb : splits);
  const int kb_per = (nkb + splits - 1) / splits;
  const Tile t = tile_of(M, N, (nkb + kb_per - 1) / kb_per, rows_of_a(M, a_mn != 0), b_mn != 0);
  if (tile_n) *tile_n = t.bn;
  if (ctas) *ctas = t.ctas;
  if (ctas_per_sm) *ctas_per_sm = t.deep ? 1 : 2;
  return PTYCHO_OK;
}

int ptycho_gemm_bf16_mn(const void* A, int lda, int a_mn, const void* B, int ldb, void* C, int ldc, int M, int N,
                        int K, int flags, int splits, int* status, void* stream) {
  return gemm_run({A, lda, a_mn != 0}, {B, ldb, true}, C, ldc, M, N, K, nullptr, flags, splits, status,
                  static_cast<cudaStream_t>(stream));
}

int ptycho_cnn_im2col3x3(const void* x, int B, int H, int W, int C, int ldx, void* col, int ldcol, void* stream) {
  if (!x || !col || B < 1 || H < 1 || W < 1 || C < 8 || (C & 7) || (ldx & 7) || (ldcol & 7) || ldx < C ||
      ldcol < 9 * C || !al16(x) || !al16(col))
    return fail(PTYCHO_ERR_INVALID, "im2col3x3: bad arguments (C and leading dims multiples of 8, 16-byte aligned)");
  const int64_t n = (int64_t)B * H * W * 9 * (C / 8);
  im2col3x3_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const bf16*>(x), B, H, W, C, ldx, static_cast<bf16*>(col), ldcol);
  return check_launch("im2col3x3_kernel");
}

int ptycho_cnn_col2im3x3(const float* dcol, int ldcol, int B, int H, int W, int C, float* dx, int ldx, int accumulate,
                         void* stream) {
  if (!dcol || !dx || B < 1 || H < 1 || W < 1 || C < 4 || (C & 3) || (ldcol & 3) || (ldx & 3) || ldcol < 9 * C ||
      ldx < C || !al16(dcol) || !al16(dx))
    return fail(PTYCHO_ERR_INVALID, "col2im3x3: bad arguments (C and leading dims multiples of 4, 16-byte aligned)");
  const int64_t n = (int64_t)B * H * W * (C / 4);
  col2im3x3_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(dcol, ldcol, B, H, W, C, dx, ldx,
                                                                                       accumulate);
  return check_launch("col2im3x3_kernel");
}

int ptycho_cnn_convT_gather(const float* colT, int ldcol, int B, int H, int W, int Co, const float* bias, void* out,
                            int ldo, void* stream) {
  if (!colT || !out || B < 1 || H < 1 || W < 1 || Co < 1 || ldcol < 9 * Co || ldo < Co)
    return fail(PTYCHO_ERR_INVALID, "convT_gather: bad arguments");
  const int64_t n = (int64_t)B * 4 * H * W * Co;
  convT_gather_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      colT, ldcol, B, H, W, Co, bias, static_cast<bf16*>(out), ldo);
  return check_launch("convT_gather_kernel");
}

int ptycho_cnn_convT_im2col(const float* dout, int ldo, int B, int H, int W, int Co, void* dcol, int ldcol,
                            void* stream) {
  if (!dout || !dcol || B < 1 || H < 1 || W < 1 || Co < 1 || ldo < Co || ldcol < 9 * Co)
    return fail(PTYCHO_ERR_INVALID, "convT_im2col: bad arguments");
  const int64_t n = (int64_t)B * H * W * 9 * Co;
  convT_im2col_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      dout, ldo, B, H, W, Co, static_cast<bf16*>(dcol), ldcol);
  return check_launch("convT_im2col_kernel");
}

// dtypes: 0 = FP32, 1 = BF16.
int ptycho_cnn_transpose(const void* in, int in_dtype, int R, int C, int ldi, int64_t batch_stride_in, void* out,
                         int out_dtype, int ldo, int64_t batch_stride_out, int batch, void* stream) {
  if (!in || !out || R < 1 || C < 1 || ldi < C || ldo < R || batch < 1 || batch > 65535 || in_dtype < 0 ||
      in_dtype > 1 || out_dtype < 0 || out_dtype > 1)
    return fail(PTYCHO_ERR_INVALID, "transpose: bad arguments");
  dim3 grid((C + 31) / 32, (R + 31) / 32, batch), block(32, 8);
  if ((C + 31) / 32 > 2147483647 || (R + 31) / 32 > 65535) return fail(PTYCHO_ERR_INVALID, "transpose: too many rows");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (in_dtype == 0 && out_dtype == 1)
    transpose_kernel<float, bf16><<<grid, block, 0, st>>>(static_cast<const float*>(in), R, C, ldi, batch_stride_in,
                                                          static_cast<bf16*>(out), ldo, batch_stride_out);
  else if (in_dtype == 1 && out_dtype == 1)
    transpose_kernel<bf16, bf16><<<grid, block, 0, st>>>(static_cast<const bf16*>(in), R, C, ldi, batch_stride_in,
                                                         static_cast<bf16*>(out), ldo, batch_stride_out);
  else if (in_dtype == 0 && out_dtype == 0)
    transpose_kernel<float, float><<<grid, block, 0, st>>>(static_cast<const float*>(in), R, C, ldi, batch_stride_in,
                                                           static_cast<float*>(out), ldo, batch_stride_out);
  else
    transpose_kernel<bf16, float><<<grid, block, 0, st>>>(static_cast<const bf16*>(in), R, C, ldi, batch_stride_in,
                                                          static_cast<float*>(out), ldo, batch_stride_out);
  return check_launch("transpose_kernel");
}

int ptycho_cnn_bn_forward(const float* x, int ldx, int R, int C, const float* gamma, const float* beta,
                          float* run_mean, float* run_var, float momentum, float eps, int training, float* mean,
                          float* rstd, double* work, int64_t work_elems, void* out, int ldo, void* stream) {
  const qb::bn::Forward f{x, ldx, gamma, beta, run_mean, run_var, mean, rstd, momentum, eps, training,
                          static_cast<bf16*>(out), ldo};
  if (int rc = bn_check(f, R, C)) return rc;
  if (gamma && training)
    if (int rc = work_check(C, work_elems)) return rc;
  return bn_forward(f, R, C, work, work_elems, static_cast<cudaStream_t>(stream));
}

int ptycho_cnn_bn_backward(const float* dy, int lddy, const float* x, int ldx, int R, int C, const float* gamma,
                           const float* mean, const float* rstd, int training, int act, float* dgamma, float* dbeta,
                           double* work, int64_t work_elems, float* dz32, void* dz16, int ldz, void* stream) {
  const qb::bn::Backward b{dy, lddy, x, ldx, gamma, mean, rstd, training, act, dgamma, dbeta, nullptr, dz32,
                           static_cast<bf16*>(dz16), ldz};
  if (int rc = bn_check(b, R, C)) return rc;
  if (gamma)
    if (int rc = work_check(C, work_elems)) return rc;
  return bn_backward(b, R, C, work, work_elems, static_cast<cudaStream_t>(stream));
}

int ptycho_cnn_colsum(const float* a, int lda, int R, int C, float* out, int accumulate, double* work,
                      int64_t work_elems, void* stream) {
  if (!a || !out || R < 1 || C < 1 || lda < C) return fail(PTYCHO_ERR_INVALID, "colsum: bad arguments");
  return colsum(a, lda, R, C, work, work_elems, out, accumulate, static_cast<cudaStream_t>(stream));
}

int ptycho_cnn_maxpool2(const void* in, int ldi, int B, int H, int W, int C, void* out, int ldo, void* argmax,
                        void* stream) {
  if (!in || !out || !argmax || B < 1 || H < 2 || W < 2 || (H & 1) || (W & 1) || C < 1 || ldi < C || ldo < C)
    return fail(PTYCHO_ERR_INVALID, "maxpool2: bad arguments (H, W even)");
  const int64_t n = (int64_t)B * (H / 2) * (W / 2) * C;
  maxpool2_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const bf16*>(in), ldi, B, H, W, C, static_cast<bf16*>(out), ldo, static_cast<uint8_t*>(argmax));
  return check_launch("maxpool2_kernel");
}

int ptycho_cnn_maxpool2_backward(const float* dout, int lddo, const void* argmax, int B, int H, int W, int C,
                                 float* din, int lddi, int accumulate, void* stream) {
  if (!dout || !argmax || !din || B < 1 || H < 2 || W < 2 || (H & 1) || (W & 1) || C < 1 || lddo < C || lddi < C)
    return fail(PTYCHO_ERR_INVALID, "maxpool2_backward: bad arguments");
  const int64_t n = (int64_t)B * H * W * C;
  maxpool2_backward_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      dout, lddo, static_cast<const uint8_t*>(argmax), B, H, W, C, din, lddi, accumulate);
  return check_launch("maxpool2_backward_kernel");
}

int ptycho_cnn_cast_bf16(const float* in, void* out, int64_t n, void* stream) {
  if (!in || !out || n < 0) return fail(PTYCHO_ERR_INVALID, "cast_bf16: bad arguments");
  if (n == 0) return PTYCHO_OK;
  cast_bf16_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(in, static_cast<bf16*>(out), n);
  return check_launch("cast_bf16_kernel");
}

int ptycho_cnn_mse(const float* pred, const float* target, int64_t n, float* loss, float* dpred32, void* dpred16,
                   double* work, int64_t work_elems, void* stream) {
  if (!pred || !target || !loss || n < 1 || !work || work_elems < kMseBlocks)
    return fail(PTYCHO_ERR_INVALID, "mse: bad arguments (workspace >= %d doubles)", kMseBlocks);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  mse_kernel<<<kMseBlocks, 256, 0, st>>>(pred, target, n, work, dpred32, static_cast<bf16*>(dpred16));
  if (int rc = check_launch("mse_kernel")) return rc;
  mse_final_kernel<<<1, 32, 0, st>>>(work, kMseBlocks, n, loss);
  return check_launch("mse_final_kernel");
}

int ptycho_cnn_bin_features(const float* patterns, int npos, int n, int bin, int amplitudes, float norm,
                            const float* mean, float scale, void* out, int ldo, void* stream) {
  if (!patterns || !out || npos < 1 || n < 1 || bin < 1 || n % bin || ldo < (n / bin) * (n / bin))
    return fail(PTYCHO_ERR_INVALID, "bin_features: bad arguments (n divisible by bin, ldo >= (n/bin)^2)");
  const int64_t total = (int64_t)npos * (n / bin) * (n / bin);
  bin_features_kernel<<<blocks_for(total, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      patterns, npos, n, bin, amplitudes, norm, mean, scale, static_cast<bf16*>(out), ldo);
  return check_launch("bin_features_kernel");
}

int ptycho_cnn_dropout(void* x, int dtype, int R, int C, int ld, float p, uint64_t seed, void* stream) {
  if (!x || R < 1 || C < 1 || ld < C || !(p >= 0.0f && p <= 1.0f) || (dtype != 0 && dtype != 1))
    return fail(PTYCHO_ERR_INVALID, "dropout: bad arguments");
  const float scale = p < 1.0f ? 1.0f / (1.0f - p) : 0.0f;  // p = 1 drops everything
  const int g = blocks_for((int64_t)R * C, 256);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == 0)
    dropout_kernel<float><<<g, 256, 0, st>>>(static_cast<float*>(x), R, C, ld, p, scale, seed);
  else
    dropout_kernel<bf16><<<g, 256, 0, st>>>(static_cast<bf16*>(x), R, C, ld, p, scale, seed);
  return check_launch("dropout_kernel");
}

}  // extern "C"

namespace {
// Arguments of a whole-layer call, all of them checked before its first launch: rows of
// B H W `up` pixels (a patch matrix of more than 2^30 rows fits no device), channel counts and
// leading dimensions that the copies of 16 bytes can take, and the pointers that are not optional.
constexpr int64_t kMaxRows = 1 << 30;
int layer_check(const char* what, int B, int H, int W, int up, int c, int co) {
  if (B < 1 || H < 1 || W < 1 || c < 8 || (c & 7) || co < 1 || c > (1 << 27) || co > (1 << 27) ||
      (int64_t)B * H > kMaxRows || (int64_t)B * H * W > kMaxRows / up)
    return fail(PTYCHO_ERR_INVALID, "%s: bad sizes (B=%d H=%d W=%d, channels %d -> %d)", what, B, H, W, c, co);
  return PTYCHO_OK;
}
// the pointers of an operand that is copied 16 bytes at a time, and its leading dimension (0: packed)
bool operand(const void* p, int ld = 0, int cols = 0) { return p && al16(p) && !(ld & 7) && ld >= cols; }
int bad_args(const char* what) { return fail(PTYCHO_ERR_INVALID, "%s: bad arguments", what); }
}  // namespace

extern "C" {

int ptycho_cnn_conv_forward(const void* x, int ldx, int B, int H, int W, int C, const void* w, int co,
                            const float* bias, int act, const float* gamma, const float* beta, float* run_mean,
                            float* run_var, float momentum, float eps, int training, float* mean, float* rstd,
                            void* col, float* r, void* out, int ldo, void* stream) {
  if (int rc = layer_check("conv_forward", B, H, W, 1, C, co)) return rc;
  const int R = B * H * W;
  const qb::bn::Forward f{r, co, gamma, beta, run_mean, run_var, mean, rstd, momentum, eps, training,
                          static_cast<bf16*>(out), ldo};
  if (!operand(x, ldx, C) || !operand(w) || !operand(col) || !r || act < 0 || act >= qb::ACT_COUNT)
    return bad_args("conv_forward");
  if (out)
    if (int rc = bn_check(f, R, co)) return rc;
  if (int rc = ptycho_cnn_im2col3x3(x, B, H, W, C, ldx, col, 9 * C, stream)) return rc;
  if (int rc = ptycho_gemm_bf16(col, 9 * C, w, 9 * C, r, co, R, co, 9 * C, bias, act << 8, 1, nullptr, stream))
    return rc;
  if (!out) return PTYCHO_OK;
  // the patches are used up: their memory takes the partial sums
  return bn_forward(f, R, co, static_cast<double*>(col), (int64_t)R * 9 * C / 4, static_cast<cudaStream_t>(stream));
}

namespace {
// Weight gradient dw (M x N, zero on entry) = A^T B over K rows, split over K to about two CTAs
// per SM with at least four k-blocks each.  One split stores its result: adding the 38 MB of a
// 1024 x 9216 gradient atomically took 94 us.
int wgrad(const void* A, int lda, const void* B, int ldb, float* dw, int M, int N, int K, cudaStream_t st) {
  const int bn = N <= 32 ? 32 : (N <= 64 ? 64 : 128);
  const int tiles = ((M + 127) / 128) * ((N + bn - 1) / bn), nkb = (K + 63) / 64;
  int s = 2 * 148 / (tiles > 0 ? tiles : 1);
  if (s > nkb / 4) s = nkb / 4;
  return gemm_run({A, lda, true}, {B, ldb, true}, dw, N, M, N, K, nullptr, s > 1 ? PTYCHO_GEMM_ATOMIC : 0, s, nullptr,
                  st);
}
}  // namespace

int ptycho_cnn_conv_backward(const float* dy, int lddy, const void* x, int ldx, int B, int H, int W, int C,
                             const void* w, const float* r, int co, const float* gamma, const float* mean,
                             const float* rstd, int training, int act, float* dw, float* db, float* dgamma,
                             float* dbeta, void* dz, int ldz, void* col, float* dcol, float* dx, int lddx,
                             int dx_accumulate, void* stream) {
  if (int rc = layer_check("conv_backward", B, H, W, 1, C, co)) return rc;
  const int R = B * H * W, K9 = 9 * C;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (!operand(x, ldx, C) || !operand(dz, ldz, co) || !operand(col) || !dw ||
      (dx && (!operand(w) || !operand(dcol) || !al16(dx) || (lddx & 3) || lddx < C)))
    return bad_args("conv_backward");
  if (int rc = bn_backward({dy, lddy, r, co, gamma, mean, rstd, training, act, dgamma, dbeta, db, nullptr,
                            static_cast<bf16*>(dz), ldz},
                           R, co, static_cast<double*>(col), (int64_t)R * K9 / 4, st))
    return rc;
  // weight gradient dz^T col
  if (int rc = ptycho_cnn_im2col3x3(x, B, H, W, C, ldx, col, K9, stream)) return rc;
  if (int rc = wgrad(dz, ldz, col, K9, dw, co, K9, R, st)) return rc;
  if (!dx) return PTYCHO_OK;
  // input gradient: dz w, folded over the taps
  if (int rc = gemm_run({dz, ldz, false}, {w, K9, true}, dcol, K9, R, K9, co, nullptr, 0, 1, nullptr, st)) return rc;
  return ptycho_cnn_col2im3x3(dcol, K9, B, H, W, C, dx, lddx, dx_accumulate, stream);
}

int ptycho_cnn_up_forward(const void* y, int ldy, int B, int H, int W, int ci, int co, const void* wt, const float* bt,
                          const void* w1, const float* b1, const float* gamma, const float* beta, float* run_mean,
                          float* run_var, float momentum, float eps, int training, float* mean, float* rstd,
                          float* colT, void* t, float* r, void* out, int ldo, void* stream) {
  if (int rc = layer_check("up_forward", B, H, W, 4, ci, co)) return rc;
  const int Rin = B * H * W, R = 4 * Rin;
  const qb::bn::Forward f{r, co, gamma, beta, run_mean, run_var, mean, rstd, momentum, eps, training,
                          static_cast<bf16*>(out), ldo};
  if (!operand(y, ldy, ci) || !operand(wt) || !operand(w1) || !operand(t) || !colT) return bad_args("up_forward");
  if (int rc = bn_check(f, R, co)) return rc;
  if (int rc = ptycho_gemm_bf16(y, ldy, wt, ci, colT, 9 * ci, Rin, 9 * ci, ci, nullptr, 0, 1, nullptr, stream))
    return rc;
  if (int rc = ptycho_cnn_convT_gather(colT, 9 * ci, B, H, W, ci, bt, t, ci, stream)) return rc;
  if (int rc = ptycho_gemm_bf16(t, ci, w1, ci, r, co, R, co, ci, b1, 0, 1, nullptr, stream)) return rc;
  // the transposed convolution's products are used up
  return bn_forward(f, R, co, reinterpret_cast<double*>(colT), (int64_t)Rin * 9 * ci / 2,
                    static_cast<cudaStream_t>(stream));
}

int ptycho_cnn_up_backward(const float* dup, int lddup, const void* y, int ldy, const void* t, const float* r, int B,
                           int H, int W, int ci, int co, const void* wt, const void* w1, const float* gamma,
                           const float* mean, const float* rstd, int training, float* dwt, float* dbt, float* dw1,
                           float* db1, float* dgamma, float* dbeta, void* dz, int ldz, float* dt, void* dcolT,
                           double* work, int64_t work_elems, float* dy, void* stream) {
  if (int rc = layer_check("up_backward", B, H, W, 4, ci, co)) return rc;
  const int Rin = B * H * W, R = 4 * Rin, C9 = 9 * ci;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (!operand(y, ldy, ci) || !operand(t) || !operand(wt) || !operand(w1) || !operand(dz, ldz, co) || !operand(dcolT) ||
      !dt || !dwt || !dbt || !dw1 || !dy || !work)
    return bad_args("up_backward");
  if (int rc = work_check(ci, work_elems)) return rc;
  if (int rc = bn_backward({dup, lddup, r, co, gamma, mean, rstd, training, 0, dgamma, dbeta, db1, nullptr,
                            static_cast<bf16*>(dz), ldz},
                           R, co, work, work_elems, st))
    return rc;
  // 1x1 convolution: dw1 = dz^T t, dt = dz w1
  if (int rc = wgrad(dz, ldz, t, ci, dw1, co, ci, R, st)) return rc;
  if (int rc = gemm_run({dz, ldz, false}, {w1, ci, true}, dt, ci, R, ci, co, nullptr, 0, 1, nullptr, st)) return rc;
  // transposed convolution: bias, weight and input gradients
  if (int rc = colsum(dt, ci, R, ci, work, work_elems, dbt, 0, st)) return rc;
  if (int rc = ptycho_cnn_convT_im2col(dt, ci, B, H, W, ci, dcolT, C9, stream)) return rc;
  if (int rc = wgrad(dcolT, C9, y, ldy, dwt, C9, ci, Rin, st)) return rc;
  return gemm_run({dcolT, C9, false}, {wt, ci, true}, dy, ci, Rin, ci, C9, nullptr, 0, 1, nullptr, st);
}

}  // extern "C"
