// FP64-accuracy SP2 squarings on the tcgen05 integer tensor cores (kind::i8).
//
// An SP2 iterate X is symmetric with its spectrum in [0, 1] (to the interval's margins), so
// every element lies in [-1, 1]. It is held, besides its fp64 copy, as eight int8 digit
// planes in fixed point, x = 2^-6 (a_0 + 2^-7 (a_1 + ... + 2^-7 a_7)) + r with |r| <= 2^-56;
// the split is exact in fp64 (each step scales by a power of two and subtracts the nearest
// integer) and every digit lies in [-64, 64]. The product is then
//   X X = 2^-12 sum_g 2^-7g G_g,   G_g = sum_{i + j = g} A_i A_j^T   (g = 0 .. 7),
// each G_g an exact int32 sum of int8 products (|G_g| <= 8 * 4096 * n), the terms with
// i + j > 7 (below 2^-56 per product element) dropped: the Ozaki-scheme emulation of an fp64
// product with fixed-point splits. The error of one squaring is ~1e-17 n in the largest
// element, about that of an fp64 GEMM.
//
// Bound: one int8 MMA of N = 64 reads 4 KB of A and 2 KB of B from shared memory in the 32 clk the
// tensor core needs, 192 of the 128 B/clk the shared memory gives, so eight 64-column accumulators
// in one pass (k_sp2_step_i8) cannot pass 2/3 of the int8 rate. Where the lower tiles fill the
// GPU, pairs of CTAs work on 256 x 128 tiles instead (k_sp2_step_i8_pair): each holds 128 rows of A
// and half of B's columns, which the pair's MMAs (cta_group::2, M = 256, N = 128) read together, 6
// KB per 64 clk and CTA, 96 B/clk. Eight accumulators of 128 columns would need 1,024 TMEM columns,
// so the digit pairs are taken in two passes over K: i + j = 4 .. 7 (26 pairs, all planes), then
// 0 .. 3 (10 pairs, planes 0 .. 3 only), the Horner sum held in registers in between: 12 planes x
// 192 rows per 128 x 128 outputs through L2 against 16 x 192 for two 128 x 64 tiles.
//
// The digit planes lie in global memory as the operand tiles want them in shared memory: per 128
// rows and 32 columns two blocks of 128 rows x 128 bytes, planes 0 .. 3 and 4 .. 7 side by side,
// 16-byte chunks in the 128-byte swizzle, so that a stage is a few untiled copies of consecutive
// memory and an MMA picks its plane by the start address alone.
//
// A producer lane feeds the stages by bulk copies (no multicast), an MMA lane issues, the epilogue
// warps combine the accumulators in fp64 (Horner over g) into a staging tile, release TMEM for the
// next tile and apply the fused SP2 step while its MMAs run: X_{k+1} = X_k^2 or 2 X_k - X_k^2 by
// the step's decision, written in fp64 with its mirror (coalesced), and each 128 x 64 tile's share
// of tr X_{k+1} and |X_{k+1}|_F^2 for the next decision (in one order in both kernels: the same
// bits). Measured: the MMAs alone run at 67 clk (N = 128) against 56 (N = 64); a step with its
// split takes 161 us in pairs and 208 us in single CTAs at 2,004 orbitals. A separate elementwise kernel then splits X_{k+1} into its digit planes (integer
// arithmetic, every SM busy). Every mbarrier wait has a time limit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "common.cuh"
#include "kernels.hpp"
#include "tcgen05.cuh"

namespace pm7 {
namespace {
using namespace tc;

constexpr int kDigits = 8;               // int8 planes per element
constexpr int IM = 128, IN = 64;         // tile rows, columns
constexpr int KB = 32;                   // K columns per block of digits and per MMA
constexpr int kTmemCols = 512;           // all of TMEM: 8 accumulators of 64 columns or 4 of 128
constexpr int kHalf = 64 * 128;          // bytes of 64 rows x 4 planes x 32 columns
// A stage: A planes 0-3 and 4-7 (128 rows each), B planes 0-3 and 4-7 (64 rows each); the pair
// kernel's second pass holds planes 0-3 of two K blocks in the same places.
constexpr int kA1 = 2 * kHalf, kB0 = 4 * kHalf, I_STAGE = 6 * kHalf;
// A kernel's ring of ST stages and its staging tile of 128 rows x W columns.
template <int ST, int W>
struct I8Shape {
  static constexpr int STAGES = ST, WIDTH = W, LDT = W + 1;
  static constexpr int SMEM = ST * I_STAGE + IM * LDT * 8 + 128 + (3 * ST + 3) * 8 + 16 + 1024;
  static_assert(SMEM <= 227 * 1024, "one CTA per SM within the shared-memory limit");
};
using OneShape = I8Shape<3, 64>;   // one pass: the 64 columns of a tile at once
using PairShape = I8Shape<3, 32>;  // two passes, beside the next tile's stages
// The pair's last tile of a CTA has the ring to itself: all 128 columns at once, so that the sums'
// chains run side by side (four rounds of them, 8,000 clk each, were 17 of 165 us at n = 2,004).
struct LastShape {
  static constexpr int WIDTH = 128, LDT = 129;
  static_assert(IM * LDT * 8 <= PairShape::STAGES * I_STAGE, "the staging tile fits the ring");
};

// Shared-memory matrix descriptor: K-major operand, 128-byte rows in the 128-byte swizzle (8-row
// groups 1,024 bytes apart), version 1; `addr` is a block's base (1,024-byte aligned) plus the
// plane's 32 bytes.
__device__ __forceinline__ uint64_t desc_128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);           // start address
  d |= (uint64_t)1 << 16;                          // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset
  d |= (uint64_t)1 << 46;                          // version
  d |= (uint64_t)2 << 61;                          // SWIZZLE_128B
  return d;
}

// Instruction descriptor, kind::i8: s32 accumulate, signed 8-bit A and B, both K-major.
constexpr uint32_t idesc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

template <int CG>  // CTAs that share the MMA
__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t accumulate) {
  if (CG == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc_i8(IM, IN)), "r"(accumulate));
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(idesc_i8(2 * IM, 2 * IN)), "r"(accumulate));
}

// `bytes` consecutive bytes into shared memory, counted on the barrier (16-byte aligned, no tensor
// map: the blocks lie in memory as the stage wants them. Every SM reading, these untiled copies
// bring 49 B/clk per SM from L2 with three 48 KB stages in flight).
__device__ __forceinline__ void load_block(uint32_t dst, const int8_t *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Arrives on the barrier of both CTAs of the pair once the MMAs issued so far have completed.
__device__ __forceinline__ void pair_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}

// Offset of the digit block of 128-row block rb, K block kt, plane group g (group 1 follows 0).
constexpr int kBlock = 128 * 128;
__host__ __device__ __forceinline__ size_t block_at(int rb, int kt, int g, int kts) {
  return (((size_t)rb * kts + kt) * 2 + g) * kBlock;
}

// The digits of x (see the file header) by integer arithmetic: x rounded to a multiple of
// 2^-55 (a 64-bit fixed-point integer, exact scaling), then balanced base-128 digits from the
// lowest (each in [-64, 63], the remainder divided exactly by 128), the first digit what is
// left (|a_0| <= 127 for |x| < 1.98). False, with zero digits, beyond that range or for a
// non-finite x.
__device__ __forceinline__ bool split_digits(double x, int8_t (&a)[kDigits]) {
  if (!(fabs(x) < 1.98)) {
#pragma unroll
    for (int p = 0; p < kDigits; ++p) a[p] = 0;
    return false;
  }
  long long v = __double2ll_rn(x * 36028797018963968.0);  // x 2^55
#pragma unroll
  for (int p = kDigits - 1; p >= 1; --p) {
    const long long d = ((v + 64) & 127) - 64;
    a[p] = (int8_t)d;
    v = (v - d) >> 7;
  }
  a[0] = (int8_t)v;
  return true;
}

// Lower tiles of 128 x 64: row block r holds column blocks 0 .. min(2r + 1, tn - 1).
__host__ __device__ __forceinline__ int i8_tile_count(int n) {
  const int tm = (n + IM - 1) / IM, tn = (n + IN - 1) / IN;
  int t = 0;
  for (int r = 0; r < tm; ++r) t += 2 * r + 2 < tn ? 2 * r + 2 : tn;
  return t;
}
__device__ __forceinline__ int i8_tile_index(int bm, int bn, int n) {
  const int tn = (n + IN - 1) / IN;
  int t = bn;
  for (int r = 0; r < bm; ++r) t += 2 * r + 2 < tn ? 2 * r + 2 : tn;
  return t;
}
__device__ __forceinline__ void i8_tile(int t, int n, int &bm, int &bn) {
  const int tn = (n + IN - 1) / IN;
  int r = 0;
  for (;;) {
    const int c = 2 * r + 2 < tn ? 2 * r + 2 : tn;
    if (t < c) break;
    t -= c;
    ++r;
  }
  bm = r;
  bn = t;
}

// The fused step of W columns (from n0) of a 128-row tile whose X_k^2 stands in the staging tile T,
// by NT epilogue threads (barrier 1): the lower-triangle elements updated and written with their
// mirror; their trace and |.|_F^2, summed per column and row half in ascending rows and over 32
// columns by a shuffle tree, to red: 64-column tile b, its 32-column group g, row half h at
// red[8 b + 2 (g + 2 h)] (b counted from the 128-column boundary for W = 128, else 0). INNER: all
// of it lies below the diagonal and inside the matrix.
template <class Shape, int NT, bool INNER>
__device__ __forceinline__ void finish_columns(double *T, int tid, int m0, int n0, int n, bool square,
                                               const double *__restrict__ x_in, double *__restrict__ x_out,
                                               double *red) {
  constexpr int W = Shape::WIDTH, LDT = Shape::LDT;
  constexpr int RS = NT / W;  // rows per pass
  const int c = tid % W, gc = n0 + c;
#pragma unroll 1
  for (int i0 = tid / W; i0 < IM; i0 += 16 * RS) {
    double xo[16];
    const double *px = x_in + (size_t)(m0 + i0) * n + gc;
#pragma unroll
    for (int v = 0; v < 16; ++v) {
      const int gr = m0 + i0 + v * RS;
      xo[v] = !square && (INNER || (gr < n && gc < n && gr >= gc)) ? __ldg(px + (size_t)(v * RS) * n) : 0.0;
    }
    double *po = x_out + (size_t)(m0 + i0) * n + gc, *pt = T + i0 * LDT + c;
#pragma unroll
    for (int v = 0; v < 16; ++v) {
      const int gr = m0 + i0 + v * RS;
      if (INNER || (gr < n && gc < n && gr >= gc)) {
        const double y = pt[v * RS * LDT], x = square ? y : 2.0 * xo[v] - y;
        pt[v * RS * LDT] = x;
        po[(size_t)(v * RS) * n] = x;
      }
    }
  }
  asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
  if (tid < 2 * W) {
    double tr = 0.0, fro = 0.0;
    const int h = tid / W;
    const double *pt = T + h * (IM / 2) * LDT + c;
    const int gr0 = m0 + h * (IM / 2);
#pragma unroll 1
    for (int i0 = 0; i0 < IM / 2; i0 += 16) {
      double x[16];
#pragma unroll
      for (int v = 0; v < 16; ++v) x[v] = pt[(i0 + v) * LDT];
#pragma unroll
      for (int v = 0; v < 16; ++v) {
        if (INNER) {
          fro = __fma_rn(2.0 * x[v], x[v], fro);
        } else {  // weights 2, 1 (diagonal) and 0 (not this tile's): no branches
          const int gr = gr0 + i0 + v;
          const double xv = gr < n && gc < n && gr >= gc ? x[v] : 0.0;
          if (gr == gc) tr += xv;
          fro = __fma_rn(gr == gc ? xv : 2.0 * xv, xv, fro);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      tr += __shfl_down_sync(0xffffffffu, tr, o);
      fro += __shfl_down_sync(0xffffffffu, fro, o);
    }
    if ((tid & 31) == 0) {
      const int g = (c >> 5) & 1, at = 8 * (c / IN) + 2 * ((W < IN ? (gc & (IN - 1)) >> 5 : g) + 2 * h);
      red[at] = tr;
      red[at + 1] = fro;
    }
  }
  constexpr int MG = 2 * W == NT ? NT / 128 : 1;  // groups of 128 threads that mirror (the sums' threads too, or the others)
  if (tid >= NT - MG * 128) {
    // the mirror (the columns as rows), thread = column of it
    const int mt = (tid - (NT - MG * 128)) & 127, mc = m0 + mt, q0 = (tid - (NT - MG * 128)) / 128 * (W / MG);
    double *po = x_out + (size_t)(n0 + q0) * n + mc;
    const double *pt = T + mt * LDT + q0;
#pragma unroll 8
    for (int q = 0; q < W / MG; ++q)
      if (INNER || (n0 + q0 + q < n && mc < n && mc > n0 + q0 + q)) po[(size_t)q * n] = pt[q];
  }
  asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");  // sums written, staging reads done
}
template <class Shape, int NT>
__device__ __forceinline__ void finish(double *T, int tid, int m0, int n0, int n, bool square,
                                       const double *__restrict__ x_in, double *__restrict__ x_out, double *red) {
  if (m0 >= n0 + Shape::WIDTH && m0 + IM <= n)
    finish_columns<Shape, NT, true>(T, tid, m0, n0, n, square, x_in, x_out, red);
  else
    finish_columns<Shape, NT, false>(T, tid, m0, n0, n, square, x_in, x_out, red);
}
// A 128 x 64 tile's partials from its four sums (one thread).
__device__ __forceinline__ void write_parts(double *__restrict__ parts, int t, const double *red) {
  parts[2 * t] = (red[0] + red[2]) + (red[4] + red[6]);
  parts[2 * t + 1] = (red[1] + red[3]) + (red[5] + red[7]);
}

template <class Shape>
struct I8Smem {
  unsigned char *stage;
  double *T, *red;
  uint64_t *full, *empty, *peer, *tmem_full, *tmem_empty, *drained;
  uint32_t *tmem_slot;
  volatile int *abort_flag;
  int *fills;  // stages handed to the copies (the producer's last word)
  __device__ explicit I8Smem(unsigned char *raw) {
    stage = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    T = reinterpret_cast<double *>(stage + Shape::STAGES * I_STAGE);
    red = T + IM * Shape::LDT;
    full = reinterpret_cast<uint64_t *>(red + 16);
    empty = full + Shape::STAGES;
    peer = empty + Shape::STAGES;
    tmem_full = peer + Shape::STAGES;
    tmem_empty = tmem_full + 1;
    drained = tmem_empty + 1;
    tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    fills = reinterpret_cast<int *>(tmem_slot + 2);
  }
};

// Persistent fused SP2 steps (see the file header) into x_out (fp64; its digit planes follow from
// k_sp2_digits), one pass per 128 x 64 tile: one CTA per SM walks the tiles with specialised warps:
// warp 4 lane 0 feeds the ring (running ahead into the next tile), warp 5 lane 0 issues the
// MMAs and owns the TMEM allocation, warps 0-3 (TMEM lane quarters 0-3) are the epilogue. The step
// does nothing once an earlier step has stopped the purification.
__global__ void __launch_bounds__(192, 1) k_sp2_step_i8(const int8_t *__restrict__ dig, int n,
                                                        const double *__restrict__ x_in, double *__restrict__ x_out,
                                                        double *__restrict__ state, int step,
                                                        double *__restrict__ parts, int *__restrict__ error,
                                                        int withhold) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if (!sp2_active(state, step)) return;  // the whole CTA, before any barrier or TMEM set-up
  const int tiles = i8_tile_count(n);
  const bool square = state[kSp2Square] != 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) state[kSp2Parts] = (double)tiles;
  constexpr int ISTAGES = OneShape::STAGES, LDT = OneShape::LDT;
  const I8Smem<OneShape> S(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kts = (n + KB - 1) / KB;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ISTAGES; ++s) {
      mbar_init(&S.full[s], 1);
      mbar_init(&S.empty[s], 1);
    }
    mbar_init(S.tmem_full, 1);
    mbar_init(S.tmem_empty, 4);  // one arrival per epilogue warp
    mbar_init(S.drained, 1);
    *S.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(S.tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *S.tmem_slot;

  if (warp == 4) {
    if (lane == 0) {  // producer: the ring over all of this CTA's tiles
      int g = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        int bm, bn;
        i8_tile(t, n, bm, bn);
        for (int kt = 0; kt < kts; ++kt, ++g) {
          const int s = g % ISTAGES;
          if (g >= ISTAGES && !mbar_wait(&S.empty[s], (uint32_t)((g / ISTAGES - 1) & 1), S.abort_flag)) {
            ok = false;
            break;
          }
          const uint32_t st = smem_u32(S.stage + s * I_STAGE);
          const int8_t *b = dig + block_at(bn >> 1, kt, 0, kts) + kHalf * (bn & 1);
          mbar_expect_tx(&S.full[s], I_STAGE);
          if (g >= withhold) continue;  // failure drill: the stage never fills, every wait runs out
          load_block(st, dig + block_at(bm, kt, 0, kts), 2 * kBlock, &S.full[s]);
          load_block(st + kB0, b, kHalf, &S.full[s]);
          load_block(st + kB0 + kHalf, b + kBlock, kHalf, &S.full[s]);
        }
      }
      *S.fills = g;
    }
  } else if (warp == 5) {
    if (lane == 0) {  // MMA issuer: digit pairs (i, j), i + j <= 7, into accumulator i + j
      int g = 0, u = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++u) {
        // the epilogue has drained the previous tile's accumulators
        if (u > 0 && !mbar_wait(S.tmem_empty, (uint32_t)((u - 1) & 1), S.abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        for (int kt = 0; kt < kts; ++kt, ++g) {
          const int s = g % ISTAGES;
          if (!mbar_wait(&S.full[s], (uint32_t)((g / ISTAGES) & 1), S.abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t st = smem_u32(S.stage + s * I_STAGE);
          // plane offsets go into the descriptors' start-address field (16-byte units; the stages
          // lie below 256 KB, so the 14-bit field does not carry)
          const uint64_t da = desc_128(st), db = desc_128(st + kB0);
#pragma unroll
          for (int i = 0; i < kDigits; ++i) {
            const uint64_t a = da + (uint64_t)(((i >> 2) * kA1 + (i & 3) * KB) >> 4);
#pragma unroll
            for (int j = 0; j + i < kDigits; ++j)
              mma_i8<1>(tmem + (uint32_t)((i + j) * IN), a, db + (uint64_t)(((j >> 2) * kHalf + (j & 3) * KB) >> 4),
                        (kt > 0 || i > 0) ? 1u : 0u);
          }
          mma_commit(&S.empty[s]);  // the stage is free once these MMAs have read it
        }
        if (ok) mma_commit(S.tmem_full);  // the tile's accumulators are final once its MMAs completed
      }
      if (!ok) *S.abort_flag = 1;
    }
  } else {
    // epilogue, warps 0-3: warp w reads TMEM lanes 32 w .. 32 w + 31 = tile rows
    int u = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++u) {
      int bm, bn;
      i8_tile(t, n, bm, bn);
      const bool ok = mbar_wait(S.tmem_full, (uint32_t)(u & 1), S.abort_flag);
      asm volatile("bar.sync 1, 128;" ::: "memory");  // every epilogue thread has its verdict
      if (!ok || *S.abort_flag) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      // accumulators -> X_k^2 tile in fp64 (Horner over g), thread = tile row
#pragma unroll 1
      for (int h = 0; h < IN / 32; ++h) {
        double acc[32];
        uint32_t r[32];
        tmem_ld32(tmem, warp, (kDigits - 1) * IN + 32 * h, r);
#pragma unroll
        for (int q = 0; q < 32; ++q) acc[q] = (double)(int)r[q];
#pragma unroll 1
        for (int g = kDigits - 2; g >= 0; --g) {
          tmem_ld32(tmem, warp, g * IN + 32 * h, r);
#pragma unroll
          for (int q = 0; q < 32; ++q) acc[q] = (double)(int)r[q] + acc[q] * 0.0078125;  // 2^-7
        }
#pragma unroll
        for (int q = 0; q < 32; ++q) S.T[(warp * 32 + lane) * LDT + 32 * h + q] = acc[q] * 0.000244140625;  // 2^-12
      }
      // TMEM is free for the next tile's MMAs
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(S.tmem_empty)) : "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the staging tile is complete
      finish<OneShape, 128>(S.T, threadIdx.x, bm * IM, bn * IN, n, square, x_in, x_out, S.red);
      if (threadIdx.x == 0) write_parts(parts, t, S.red);
    }
  }
  if (threadIdx.x == 0 && *S.abort_flag) atomicExch(error, 1);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (*S.abort_flag) {
    if (warp == 4 && lane == 0) drain_ring(S.full, *S.fills, ISTAGES);
    if (warp == 5 && lane == 0) {
      mma_commit(S.drained);
      mbar_drain(S.drained, 0u);
    }
    __syncthreads();
  }
  if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// Tiles of 256 x 128 that hold lower-triangle elements: row block r holds column blocks
// 0 .. min(2 r + 1, tn - 1).
__host__ __device__ __forceinline__ int pair_tile_count(int n) {
  const int tm = (n + 2 * IM - 1) / (2 * IM), tn = (n + 2 * IN - 1) / (2 * IN);
  int t = 0;
  for (int r = 0; r < tm; ++r) t += 2 * r + 2 < tn ? 2 * r + 2 : tn;
  return t;
}
__device__ __forceinline__ void pair_tile(int t, int n, int &r, int &c) {
  const int tn = (n + 2 * IN - 1) / (2 * IN);
  r = 0;
  for (;;) {
    const int k = 2 * r + 2 < tn ? 2 * r + 2 : tn;
    if (t < k) break;
    t -= k;
    ++r;
  }
  c = t;
}

// mbar_wait on a barrier that the pair's other CTA arrives on: acquires at cluster scope.
__device__ __forceinline__ bool pair_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag) {
  const uint32_t addr = smem_u32(bar);
  unsigned long long t0 = 0;
  for (uint32_t it = 0; it < (1u << 30); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 15) == 15) {
      if (*abort_flag) return false;
      const unsigned long long t = global_ns();
      if (it == 15) t0 = t;
      else if (t - t0 > kWaitNs) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// Arrives on the leader's copy of a barrier.
__device__ __forceinline__ void arrive_leader(uint64_t *bar) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(bar)));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(a) : "memory");
}

// The same steps by CTA pairs on 256 x 128 tiles, two passes over K (see the file header). In each
// CTA warps 0-7 are the epilogue (warp w: TMEM lanes 32 (w & 3) .., columns 64 (w >> 2) ..), warp 8
// lane 0 the producer of this CTA's share of the stages, warp 9 owns the TMEM allocation; warp 9
// lane 0 of the leader (rank 0) issues the pair's MMAs. Barriers: full (own copies), empty and
// tmem_full (the commits arrive on both CTAs) in each CTA; peer (the other CTA's stage is full) and
// tmem_empty in the leader.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1)
    k_sp2_step_i8_pair(const int8_t *__restrict__ dig, int n, const double *__restrict__ x_in,
                       double *__restrict__ x_out, double *__restrict__ state, int step, double *__restrict__ parts,
                       int *__restrict__ error, int withhold) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  if (!sp2_active(state, step)) return;  // the whole cluster, before any barrier or TMEM set-up
  const int tiles = pair_tile_count(n);
  const bool square = state[kSp2Square] != 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) state[kSp2Parts] = (double)i8_tile_count(n);
  constexpr int ISTAGES = PairShape::STAGES, LDT = PairShape::LDT, W = PairShape::WIDTH;
  const I8Smem<PairShape> S(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kts = (n + KB - 1) / KB, stages2 = (kts + 1) / 2;  // K blocks; stages of the second pass
  const int rank = blockIdx.x & 1, first = blockIdx.x >> 1, stride = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ISTAGES; ++s) {
      mbar_init(&S.full[s], 1);
      mbar_init(&S.empty[s], 1);
      mbar_init(&S.peer[s], 1);
    }
    mbar_init(S.tmem_full, 1);
    mbar_init(S.tmem_empty, 16);  // one arrival per epilogue warp of both CTAs
    mbar_init(S.drained, 1);
    *S.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(S.tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *S.tmem_slot;

  if (warp == 8) {
    if (lane == 0) {  // producer: this CTA's 128 rows of A and 64 rows of B, counted on its own barriers
      int g = 0;
      bool ok = true;
      for (int t = first; t < tiles && ok; t += stride) {
        int tr, tc;
        pair_tile(t, n, tr, tc);
        const int rb = 2 * tr + rank;
        for (int q = 0; q < kts + stages2; ++q, ++g) {
          const int s = g % ISTAGES;
          if (g >= ISTAGES && !mbar_wait(&S.empty[s], (uint32_t)((g / ISTAGES - 1) & 1), S.abort_flag)) {
            ok = false;
            break;
          }
          const uint32_t st = smem_u32(S.stage + s * I_STAGE);
          const int8_t *a, *b;
          bool two = true;  // the second half of the stage: planes 4-7, or the next K block
          size_t next;
          if (q < kts) {
            a = dig + block_at(rb, q, 0, kts);
            b = dig + block_at(tc, q, 0, kts) + kHalf * rank;
            next = kBlock;
          } else {
            const int kt = 2 * (q - kts);
            a = dig + block_at(rb, kt, 0, kts);
            b = dig + block_at(tc, kt, 0, kts) + kHalf * rank;
            next = 2 * kBlock;
            two = kt + 1 < kts;
          }
          mbar_expect_tx(&S.full[s], two ? I_STAGE : I_STAGE / 2);
          if (g >= withhold) continue;  // (see k_sp2_step_i8)
          load_block(st, a, kBlock, &S.full[s]);
          load_block(st + kB0, b, kHalf, &S.full[s]);
          if (two) {
            load_block(st + kA1, a + next, kBlock, &S.full[s]);
            load_block(st + kB0 + kHalf, b + next, kHalf, &S.full[s]);
          }
        }
      }
      *S.fills = g;
    }
  } else if (warp == 9) {
    if (lane == 0 && rank == 1) {  // tells the leader of each stage that this CTA has filled
      int g = 0;
      bool ok = true;
      for (int t = first; t < tiles && ok; t += stride)
        for (int q = 0; q < kts + stages2; ++q, ++g) {
          const int s = g % ISTAGES;
          ok = mbar_wait(&S.full[s], (uint32_t)((g / ISTAGES) & 1), S.abort_flag);
          if (!ok) break;
          arrive_leader(&S.peer[s]);
        }
    } else if (lane == 0) {  // MMA issuer of the pair
      int g = 0, u = 0;            // stages, passes
      bool ok = true;
      for (int t = first; t < tiles && ok; t += stride) {
        for (int pass = 0; pass < 2 && ok; ++pass, ++u) {
          // the epilogues have drained the previous pass's accumulators
          if (u > 0 && !pair_wait(S.tmem_empty, (uint32_t)((u - 1) & 1), S.abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const int stages = pass == 0 ? kts : stages2;
          for (int q = 0; q < stages; ++q, ++g) {
            const int s = g % ISTAGES;
            if (!mbar_wait(&S.full[s], (uint32_t)((g / ISTAGES) & 1), S.abort_flag) ||
                !pair_wait(&S.peer[s], (uint32_t)((g / ISTAGES) & 1), S.abort_flag)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t st = smem_u32(S.stage + s * I_STAGE);
            const uint64_t da = desc_128(st), db = desc_128(st + kB0);
            if (pass == 0) {  // pairs i + j = 4 .. 7 into accumulator i + j - 4
#pragma unroll
              for (int i = 0; i < kDigits; ++i) {
                const uint64_t a = da + (uint64_t)(((i >> 2) * kA1 + (i & 3) * KB) >> 4);
#pragma unroll
                for (int j = (i < 4 ? 4 - i : 0); j + i < kDigits; ++j)
                  mma_i8<2>(tmem + (uint32_t)((i + j - 4) * 2 * IN), a,
                            db + (uint64_t)(((j >> 2) * kHalf + (j & 3) * KB) >> 4), (q > 0 || i > 0) ? 1u : 0u);
              }
            } else {  // pairs i + j = 0 .. 3 of one or two K blocks
              const int halves = 2 * q + 1 < kts ? 2 : 1;
              for (int h = 0; h < halves; ++h)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const uint64_t a = da + (uint64_t)((h * kA1 + i * KB) >> 4);
#pragma unroll
                  for (int j = 0; j + i < 4; ++j)
                    mma_i8<2>(tmem + (uint32_t)((i + j) * 2 * IN), a, db + (uint64_t)((h * kHalf + j * KB) >> 4),
                              (q > 0 || h > 0 || i > 0) ? 1u : 0u);
                }
            }
            pair_commit(&S.empty[s]);  // the stage is free in both CTAs once these MMAs have read it
          }
          if (ok) pair_commit(S.tmem_full);
        }
      }
      if (!ok) *S.abort_flag = 1;
    }
  } else {
    const int tid = threadIdx.x, half = warp >> 2, quarter = warp & 3;
    int u = 0;
    bool ok = true;
    for (int t = first; t < tiles && ok; t += stride) {
      int tr, tc;
      pair_tile(t, n, tr, tc);
      const int bm = 2 * tr + rank;
      if (!square && bm * IM + tid / 2 < n) {  // this tile of X_k towards L2 while its products run: half a row per thread
        const double *px = x_in + (size_t)(bm * IM + tid / 2) * n + tc * 2 * IN + (tid & 1) * IN;
#pragma unroll
        for (int q = 0; q < IN; q += 16)
          if (tc * 2 * IN + (tid & 1) * IN + q < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(px + q));
      }
      double acc[64];
#pragma unroll
      for (int pass = 0; pass < 2; ++pass, ++u) {
        ok = mbar_wait(S.tmem_full, (uint32_t)(u & 1), S.abort_flag);
        asm volatile("bar.sync 1, 256;" ::: "memory");  // every epilogue thread has its verdict
        if (!ok || *S.abort_flag) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        // Horner over g = 7 .. 4, then 3 .. 0, thread = tile row
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t r[32];
#pragma unroll 1
          for (int g = 3; g >= 0; --g) {
            tmem_ld32(tmem, quarter, g * 2 * IN + half * IN + 32 * h, r);
            if (pass == 0 && g == 3) {
#pragma unroll
              for (int q = 0; q < 32; ++q) acc[32 * h + q] = (double)(int)r[q];
            } else {
#pragma unroll
              for (int q = 0; q < 32; ++q) acc[32 * h + q] = (double)(int)r[q] + acc[32 * h + q] * 0.0078125;  // 2^-7
            }
          }
        }
        // TMEM is free for the next pass
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) arrive_leader(S.tmem_empty);
      }
      if (!ok) break;
      if (tc > bm || bm * IM >= n) continue;  // above the diagonal or past the edge
      const int t0 = i8_tile_index(bm, 2 * tc, n);
      if (t + stride >= tiles) {  // the CTA's last tile: staged whole in the ring, which nothing uses any more
        double *T = reinterpret_cast<double *>(S.stage);
#pragma unroll
        for (int q = 0; q < 64; ++q)
          T[(quarter * 32 + lane) * LastShape::LDT + half * IN + q] = acc[q] * 0.000244140625;  // 2^-12
        asm volatile("bar.sync 1, 256;" ::: "memory");  // the staging tile is complete
        finish<LastShape, 256>(T, tid, bm * IM, 2 * tc * IN, n, square, x_in, x_out, S.red);
        if (tid == 0) {
          write_parts(parts, t0, S.red);
          if ((2 * tc + 1) * IN < n) write_parts(parts, t0 + 1, S.red + 8);
        }
        continue;
      }
      // W columns after W columns through the staging tile
#pragma unroll
      for (int hc = 0; hc < 4; ++hc) {
        if ((2 * tc + (hc >> 1)) * IN >= n) continue;
        if (half == (hc >> 1)) {
#pragma unroll
          for (int q = 0; q < W; ++q)
            S.T[(quarter * 32 + lane) * LDT + q] = acc[(hc & 1) * W + q] * 0.000244140625;  // 2^-12
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");  // the staging tile is complete
        finish<PairShape, 256>(S.T, tid, bm * IM, 2 * tc * IN + hc * W, n, square, x_in, x_out, S.red);
        if ((hc & 1) && tid == 0) write_parts(parts, t0 + (hc >> 1), S.red);
      }
    }
  }
  if (threadIdx.x == 0 && *S.abort_flag) atomicExch(error, 1);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (*S.abort_flag) {
    if (warp == 8 && lane == 0) drain_ring(S.full, *S.fills, ISTAGES);
    if (warp == 9 && lane == 0 && rank == 0) {  // (the leader alone issues MMAs)
      // (on this CTA's barrier alone: an arrival on its way to the other might find it gone)
      asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(S.drained))
                   : "memory");
      mbar_drain(S.drained, 0u);
    }
    __syncthreads();
  }
  // the pair leaves together: neither CTA's barriers, shared memory or TMEM are in use any more
  asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
  if (warp == 9) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// The digit planes (layout: see the file header) of an n x n fp64 matrix: the start iterate, and
// the output of each step (skipped, like the step, once the purification has stopped; step < 0:
// always). A CTA takes 64 rows x 32 columns: coalesced loads into shared memory, then a thread
// splits eight columns of one row and stores each plane's eight digits (four threads fill a
// plane's 32-byte sector). Elements past the edge get zero digits.
__global__ void __launch_bounds__(256) k_sp2_digits(int n, const double *__restrict__ X, int8_t *__restrict__ dig,
                                                    const double *__restrict__ state, int step,
                                                    int *__restrict__ error) {
  if (step >= 0 && !sp2_active(state, step)) return;
  __shared__ double s[64][KB + 1];
  const int kt = blockIdx.x, row0 = blockIdx.y * 64, kts = gridDim.x;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int r = (threadIdx.x >> 5) + 8 * q, c = threadIdx.x & 31;
    s[r][c] = row0 + r < n && kt * KB + c < n ? X[(size_t)(row0 + r) * n + kt * KB + c] : 0.0;
  }
  __syncthreads();
  const int r = threadIdx.x >> 2, q = threadIdx.x & 3, row = row0 + r;
  uint32_t word[kDigits][2];
#pragma unroll
  for (int p = 0; p < kDigits; ++p) word[p][0] = word[p][1] = 0u;
  bool good = true;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    int8_t a[kDigits];
    good = split_digits(s[r][8 * q + e], a) && good;
#pragma unroll
    for (int p = 0; p < kDigits; ++p) word[p][e >> 2] |= (uint32_t)(uint8_t)a[p] << (8 * (e & 3));
  }
#pragma unroll
  for (int p = 0; p < kDigits; ++p) {
    const size_t at = block_at(row >> 7, kt, p >> 2, kts) + (row & 127) * 128 +
                      (size_t)((((p & 3) * 2 + (q >> 1)) ^ (row & 7)) * 16 + (q & 1) * 8);
    *reinterpret_cast<uint2 *>(dig + at) = make_uint2(word[p][0], word[p][1]);
  }
  if (!good) atomicExch(error, 2);
}

}  // namespace

// The SMs of the current device, and the CTA pairs it holds at once.
struct I8Limits {
  int sms = 0, pairs = 0;
};
static I8Limits i8_limits() {
  static std::mutex mu;
  static I8Limits lim[64];
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  I8Limits &L = lim[dev & 63];
  if (L.sms == 0) {
    cudaFuncSetAttribute(k_sp2_step_i8, cudaFuncAttributeMaxDynamicSharedMemorySize, OneShape::SMEM);
    cudaFuncSetAttribute(k_sp2_step_i8_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, PairShape::SMEM);
    int s = 0, pairs = 0;
    if (cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) s = 148;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(s / 2 * 2);
    cfg.blockDim = dim3(320);
    cfg.dynamicSmemBytes = PairShape::SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&pairs, k_sp2_step_i8_pair, &cfg) != cudaSuccess || pairs < 1) pairs = s / 2;
    L.pairs = pairs;
    L.sms = s;
  }
  return L;
}

size_t sp2_i8_digit_bytes(int n) {
  return block_at(2 * ((n + 255) / 256), 0, 0, (n + KB - 1) / KB);
}
int sp2_i8_tiles(int n) { return i8_tile_count(n); }

void launch_sp2_digits(cudaStream_t st, int n, const double *X, int8_t *dig, const double *state, int step,
                       int *error) {
  k_sp2_digits<<<dim3((n + KB - 1) / KB, (n + 63) / 64), 256, 0, st>>>(n, X, dig, state, step, error);
  note_launch();
}

// CTA pairs where the 128 x 64 tiles would take more than one wave (from 1,409 orbitals up on 148
// SMs): a step with its digit split 161 against 208 us at 2,004 orbitals, 2.96 against 3.95 ms at
// 6,000. While one wave holds them the single CTAs are faster: they share a product among twice as
// many SMs (89 against 113 us at 1,400, 71 against 90 at 1,000).
void launch_sp2_step_i8(cudaStream_t st, int n, const int8_t *dig, const double *x_in, double *x_out, int8_t *dig_out,
                        double *state, double *parts, int step, int *error, int withhold) {
  const I8Limits L = i8_limits();
  if (i8_tile_count(n) > L.sms)
    k_sp2_step_i8_pair<<<2 * std::min(L.pairs, pair_tile_count(n)), 320, PairShape::SMEM, st>>>(dig, n, x_in, x_out, state, step,
                                                                                       parts, error, withhold);
  else
    k_sp2_step_i8<<<std::min(L.sms, i8_tile_count(n)), 192, OneShape::SMEM, st>>>(dig, n, x_in, x_out, state, step, parts, error,
                                                                               withhold);
  note_launch();
  launch_sp2_digits(st, n, x_out, dig_out, state, step, error);
}

}  // namespace pm7
