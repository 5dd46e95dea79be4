// 256 x 256 complex 2-D FFT staged across a cluster of 4 CTAs (sm_100a).
//
// A 256^2 complex64 wave (512 KB) does not fit one SM, so four CTAs of a
// thread-block cluster hold a quarter each (512 threads x 32 registers).
//
//   Layout A (real space / row slab): CTA q holds rows r = 64q + line,
//     thread (line = tid/8, tl = tid%8) holds columns c = tl + 8e, e = 0..31.
//   Layout B (spectrum / column slab): CTA q holds spectral columns
//     kc = 64q + line; after the column transform thread (line, g = tl) holds
//     kr = 4g + a + 32kB in register a*8 + kB.
//
// Each 256-point 1-D transform is local to a CTA: a 32-point register DFT over
// e, the twiddle w256^(tl*k1), a shared-memory exchange inside the line, and
// four 8-point register DFTs (k = k1 + 32*k2, natural order).  Between the row
// and column transforms the slabs are redistributed across the cluster: every
// thread stores its values straight into the owning CTA's shared memory
// (distributed shared memory), bracketed by cluster barriers.  A 2-D FFT thus
// costs two local exchanges and one cluster exchange.
//
// A line's eight threads sit in one warp, and the four lines of a warp own one region of
// the buffer in all three layouts (line-local exchange, column slab, row slab), so the
// local exchanges need __syncwarp only; the CTA-wide and cluster-wide ordering is the two
// cluster barriers of the slab exchange.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "fft_engine.cuh"

namespace qb {

namespace cg = cooperative_groups;

struct Fft256C {
  static constexpr int N = 256;
  static constexpr int T = 512;
  static constexpr int E = 32;
  static constexpr int LINES = 64;
  static constexpr int GS = 1056;           // region of a warp's four lines
  static constexpr int SM_FLOAT2 = 16 * GS;
  // twiddle table: tw[t*33 + k1] = w256^(t*k1), t < 8, k1 < 32 (row padding 33 keeps the
  // eight t rows on distinct banks)
  static constexpr int TW_FLOAT2 = 8 * 33;
  static __device__ __forceinline__ void fill_twiddles(float2* tw, int tid, int nthreads) {
    for (int k = tid; k < 8 * 32; k += nthreads) {
      const int t = k >> 5, k1 = k & 31;
      double s, c;
      sincospi(-2.0 * (double)(t * k1) / 256.0, &s, &c);
      tw[t * 33 + k1] = make_float2((float)c, (float)s);
    }
  }

  int q;     // cluster rank (0..3)
  int line;  // tid / 8
  int tl;    // tid % 8

  __device__ __forceinline__ void init(int tid, int rank) {
    q = rank;
    line = tid >> 3;
    tl = tid & 7;
  }
  // Buffer layouts (float2 index), G = line / 4 the warp, i = line % 4.  Every address is a
  // per-thread base plus a compile-time offset, and every local access takes two wavefronts.
  //   line-local exchange, element (k1, t):      G GS + 264 i + 33*(k1/4) + 8*(k1%4) + t
  //   column slab, element (kc = line, r):       G GS + 260 i + r
  //   row slab spectrum, element (r = line, kc): G GS + 256 i + 4*(kc/4) + pos
  // A remote store of a warp writes 4 consecutive elements to each of 8 lines; the slabs keep
  // those four in one 32-byte sector (8 sectors per store; padded layouts that were only
  // bank-conflict-free took 13: 13.9 -> 13.0 ms per 64 positions of 16 slices and 6 modes).
  // In the row slab the four elements of a sector are rotated by pos = (kc + 2 (kc / 16 % 2) +
  // line % 2) % 4 so that the reads, at stride 4, still spread over the banks.
  static constexpr int LP = 264, BP = 260, AP = 256;
  __device__ __forceinline__ int local_base() const { return (line >> 2) * GS + (line & 3) * LP; }
  __device__ __forceinline__ int col_base() const { return (line >> 2) * GS + (line & 3) * BP; }
  __device__ __forceinline__ int row_base() const { return (line >> 2) * GS + (line & 3) * AP; }

  // coordinates
  __device__ __forceinline__ int a_row() const { return 64 * q + line; }     // layout A row
  __device__ __forceinline__ int a_col(int e) const { return tl + 8 * e; }   // layout A column
  __device__ __forceinline__ int b_kc() const { return 64 * q + line; }      // layout B spectral column
  __device__ __forceinline__ int b_kr(int i) const { return 4 * tl + (i >> 3) + 32 * (i & 7); }  // register i = a*8+kB

  // four 8-point DFTs on registers a*8 .. a*8+7 (compile-time offsets keep x in registers)
  template <bool INV, int A>
  __device__ __forceinline__ void dft8_groups(float2 (&x)[E]) const {
    if constexpr (A < 4) {
      dft_reg<8, INV, 1, A * 8>(x);
      dft8_groups<INV, A + 1>(x);
    }
  }

  // Split cluster barrier: the first barrier of a cluster exchange only has to
  // order every CTA's last reads of its own buffer before the peers' remote
  // stores, so each thread arrives right after those reads and waits just before
  // its own remote stores; the register work in between hides the barrier.
  // (A CTA fence and a relaxed arrive instead of the release: 14.2 against 13.0 ms per 64
  // positions of 16 slices and 6 modes.)
  static __device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  static __device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }

  // ---- 256-point transform along the line: x[e] = element tl + 8e in, natural
  //      frequency k = 4*tl + a + 32*kB in register a*8 + kB out ----
  // ARRIVE: arrive on the cluster barrier after the last read of the buffer
  template <bool INV, bool ARRIVE = false>
  __device__ __forceinline__ void line_fwd(float2 (&x)[E], float2* sm, const float2* tw) const {
    dft_reg<32, INV>(x);
    {
      const float2* twr = tw + 33 * tl;
#pragma unroll
      for (int k1 = 1; k1 < 32; ++k1) x[k1] = INV ? cmulc(x[k1], twr[k1]) : cmul(x[k1], twr[k1]);
    }
    __syncwarp();  // the warp's reads of its region are complete
    {
      float2* w = sm + local_base() + tl;  // + offset of (k1, 0)
#pragma unroll
      for (int k1 = 0; k1 < 32; ++k1) w[33 * (k1 >> 2) + 8 * (k1 & 3)] = x[k1];
    }
    __syncwarp();
    {
      const float2* r = sm + local_base() + 33 * tl;  // group g = tl: k1 = 4g + a
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int t = 0; t < 8; ++t) x[a * 8 + t] = r[8 * a + t];
    }
    if (ARRIVE) cluster_arrive();
    dft8_groups<INV, 0>(x);
  }
  // inverse direction of line_fwd's data flow: frequency distribution in,
  // element tl + 8e out (INV selects the conjugate transform)
  template <bool INV, bool ARRIVE = false>
  __device__ __forceinline__ void line_bwd(float2 (&x)[E], float2* sm, const float2* tw) const {
    dft8_groups<INV, 0>(x);
    __syncwarp();  // the warp's reads of its region are complete
    {
      float2* w = sm + local_base() + 33 * tl;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int t = 0; t < 8; ++t) w[8 * a + t] = x[a * 8 + t];
    }
    __syncwarp();
    {
      const float2* r = sm + local_base() + tl;
#pragma unroll
      for (int k1 = 0; k1 < 32; ++k1) x[k1] = r[33 * (k1 >> 2) + 8 * (k1 & 3)];
    }
    if (ARRIVE) cluster_arrive();
    {
      const float2* twr = tw + 33 * tl;
#pragma unroll
      for (int k1 = 1; k1 < 32; ++k1) x[k1] = INV ? cmulc(x[k1], twr[k1]) : cmul(x[k1], twr[k1]);
    }
    dft_reg<32, INV>(x);
  }

  // ---- cluster exchanges ----
  // 32-bit shared::cluster address of `local` in the CTA of cluster rank `rank`
  static __device__ __forceinline__ uint32_t peer_addr(const void* local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r)
                 : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return r;
  }
  static __device__ __forceinline__ void st_peer(uint32_t addr, float2 v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
  }
  // A (row spectrum, register a*8+kB holds kc = 4tl + a + 32kB of row a_row())
  //   -> B (column slab, register e holds r = tl + 8e of spectral column b_kc())
  // (the caller arrived on the cluster barrier after its last read of sm)
  __device__ __forceinline__ void a_to_b(float2 (&x)[E], float2* sm, cg::cluster_group& cl) const {
    cluster_wait();  // every CTA of the cluster is done reading its buffer
    // spectral column 4 tl + a + 32 x: warp region tl + 8 x, line a
    const float2* mine = sm + GS * tl + 64 * q + line;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const uint32_t dst = peer_addr(mine, (uint32_t)d);
#pragma unroll
      for (int xb = 0; xb < 2; ++xb)
#pragma unroll
        for (int a = 0; a < 4; ++a) st_peer(dst + 8u * (uint32_t)(BP * a + 8 * GS * xb), x[a * 8 + 2 * d + xb]);
    }
    cl.sync();
    const float2* r = sm + col_base() + tl;
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = r[8 * e];
  }
  // B (column slab, register e holds r = tl + 8e of spectral column b_kc())
  //   -> A (row spectrum distribution of row a_row())
  __device__ __forceinline__ void b_to_a(float2 (&x)[E], float2* sm, cg::cluster_group& cl) const {
    cluster_wait();  // arrived after the caller's last read of sm
    // row tl + 8 j: warp region tl / 4 + 2 j, line tl % 4; kc = 64 q + line
    const int pos = ((line & 3) + 2 * ((line >> 4) & 1) + (tl & 1)) & 3;
    const float2* mine = sm + GS * (tl >> 2) + AP * (tl & 3) + 64 * q + (line & ~3) + pos;
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const uint32_t dst = peer_addr(mine, (uint32_t)d);
#pragma unroll
      for (int j = 0; j < 8; ++j) st_peer(dst + 8u * (uint32_t)(2 * GS * j), x[8 * d + j]);
    }
    cl.sync();
    // kc = 4 tl + a + 32 kB
    const float2* r = sm + row_base() + 4 * tl;
    const int rot = 2 * (tl >> 2) + (line & 1);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const float2* ra = r + ((a + rot) & 3);
#pragma unroll
      for (int kB = 0; kB < 8; ++kB) x[a * 8 + kB] = ra[32 * kB];
    }
  }

  // ---- whole 2-D transforms (unnormalised) ----
  // layout A real space -> layout B spectrum
  __device__ __forceinline__ void forward(float2 (&x)[E], float2* sm, const float2* tw, cg::cluster_group& cl) const {
    line_fwd<false, true>(x, sm, tw);
    a_to_b(x, sm, cl);
    line_fwd<false>(x, sm, tw);
  }
  // layout B spectrum -> layout A real space
  __device__ __forceinline__ void inverse(float2 (&x)[E], float2* sm, const float2* tw, cg::cluster_group& cl) const {
    line_bwd<true, true>(x, sm, tw);
    b_to_a(x, sm, cl);
    line_bwd<true>(x, sm, tw);
  }
};

}  // namespace qb
