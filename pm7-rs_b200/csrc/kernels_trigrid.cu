// Householder tridiagonalisation of one symmetric matrix by the whole GPU, for eigenvalues alone.
//
// Bound: n dependent reflectors, each a matrix-vector product with the trailing matrix and two
// exchanges between its owners; at n ~ 2,000 the products are 2/3 n^3 flop (0.2 ms of the chip's
// FP64 rate), so the time is n times the latency of a column. The matrix is therefore kept on the
// chip for the whole reduction: rows are dealt cyclically to the CTAs of a cooperative launch, and a
// thread holds its columns (c = thread + 512 k) of 4 rows (up to 512 columns) or 7 in registers, up to 8
// more, the ones that finish first, in shared memory. Nothing is blocked: the rank-2 update of a column is applied to the
// resident rows in the same pass that multiplies them with the next reflector, so a column needs ONE
// grid barrier: each CTA publishes its rows' products p = A v and the owner of the next row that row,
// not yet updated by the current reflector; after the barrier every CTA forms w, applies the update
// to that row itself and derives the next reflector from it.
//
// Every sum is taken in a fixed order that depends on the matrix order alone, and a row's update is the
// same operations wherever the row lies, so the values are the same bits on every grid.
//
// Measured (CUDA events): 0.39 ms at 121 orbitals, 0.65 at 204, 0.99 at 310, 2.4 at 666 and 11.1 at 2,004
// (cuSOLVER dsyevd, values included, 7.4 and 25.7 at the last two): 3.2 to 5.5 us a column, of which the
// barrier is ~1 and the loads behind it ~0.5. The levels of one matrix as a call with its copies, against
// the cluster kernel: 0.80 / 2.2 ms at 204, 1.07 / 2.8 at 270, 2.2 / 6.1 at 512, 3.8 / 10.1 at 666.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "kernels.hpp"

namespace pm7 {
namespace {

constexpr int QT = 512, QW = QT / 32;
constexpr unsigned long long kWaitLimit = 1000000000ull;  // a grid barrier gives up after 1 s

// Arrival and bounded wait of all CTAs (cooperative launch); as grid_sync of kernels_sp2.cu.
__device__ __forceinline__ bool tri_sync(unsigned *count, unsigned &epoch, int *error) {
  __syncthreads();
  ++epoch;
  int bad = 0;
  if (threadIdx.x == 0) {
    const unsigned target = epoch * gridDim.x;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    unsigned long long t0 = 0;
    for (unsigned it = 0;; ++it) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      if (v >= target) break;
      if ((it & 255) == 255) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (it == 255) t0 = t;
        if (t - t0 > kWaitLimit || *(volatile int *)error != 0) {
          atomicExch(error, 1);
          bad = 1;
          break;
        }
      }
    }
  }
  return __syncthreads_or(bad) == 0;
}

// Sum over the CTA in every thread; one barrier, the caller alternates `red` (QW doubles).
__device__ __forceinline__ double cta_sum(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s[QW];
#pragma unroll
  for (int w = 0; w < QW; ++w) s[w] = red[w];
#pragma unroll
  for (int o = QW / 2; o > 0; o >>= 1)
#pragma unroll
    for (int w = 0; w < o; ++w) s[w] += s[w + o];
  return s[0];
}

// Sums of eight values over the warp by halving: lane l ends with value ((l & 16) ? 4 : 0) +
// ((l & 8) ? 2 : 0) + ((l & 4) ? 1 : 0).
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int h = 4; h > 0; h >>= 1) {
    const int o = 4 * h;
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const double give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// An element after the rank-2 update: y - (v_i w_c + w_i v_c). (As two FMAs on y it takes an operation
// less, but rounds at the element's size twice: the levels' error at 666 orbitals 6.5e-15 -> 1.1e-14 rms.)
__device__ __forceinline__ double rank2(double y, double vi, double wi, double vc, double wc) {
  return __dsub_rn(y, __fma_rn(vi, wc, __dmul_rn(wi, vc)));
}

// KC columns per thread; RR rows per CTA in registers (the last ones) and rs in shared memory (the
// first), rs <= 8. pub: 4 n doubles (two sets of p and next row).
template <int KC, int RR>
__global__ void __launch_bounds__(QT, 1) k_tridiag_grid(EigvalsTask T, int rs, double *pub,
                                                        unsigned *count, int *error) {
  extern __shared__ __align__(16) double tg_smem[];
  __shared__ double sums[2][QW], rows_red[2][QW][8], scal[4];
  const int n = T.n, G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double *vs = tg_smem, *ws = vs + n, *sA = ws + n;  // the last reflector and its w, the shared rows
  // scaled by a power of two to a largest element in [1, 2)
  unsigned epoch = 0;
  double big = 0.0;
  for (int i = b; i < n; i += G)
    for (int c = tid; c < n; c += QT) big = fmax(big, fabs(T.src[(size_t)i * T.ld + c]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (lane == 0) sums[0][warp] = big;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < QW; ++w) big = fmax(big, sums[0][w]);
    __stcg(pub + b, big);
  }
  if (!tri_sync(count, epoch, error)) return;
  big = 0.0;
  for (int q = lane; q < G; q += 32) big = fmax(big, __ldcg(pub + q));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (!tri_sync(count, epoch, error)) return;  // (pub is used again)
  const double sc = tri_scale(big);
  if (b == 0 && tid == 0) T.part[3] = 1.0 / sc;
  double a[RR][KC];
#pragma unroll
  for (int r = 0; r < RR; ++r)
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int i = b + G * (rs + r), c = tid + QT * k;
      a[r][k] = i < n && c < n ? T.src[(size_t)i * T.ld + c] * sc : 0.0;
    }
  for (int r = 0; r < rs; ++r)
    for (int c = tid; c < n; c += QT) {
      const int i = b + G * r;
      sA[(size_t)r * n + c] = i < n ? T.src[(size_t)i * T.ld + c] * sc : 0.0;
    }
  double x[KC], v[KC], vp[KC], wp[KC];
#pragma unroll
  for (int k = 0; k < KC; ++k) {
    const int c = tid + QT * k;
    x[k] = c < n ? T.src[c] * sc : 0.0;  // row 0
    v[k] = vp[k] = wp[k] = 0.0;
    if (c < n) vs[c] = ws[c] = 0.0;
  }
  if (tid == 0) {
    if (b == 0) T.d[0] = x[0];
  }
  for (int j = 0; j < n - 1; ++j) {
    // the reflector of column j from its updated row x (columns > j)
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = tid + QT * k;
      if (c == j + 1) scal[0] = x[k];
      if (c > j + 1 && c < n) s += x[k] * x[k];
    }
    const double sigma = cta_sum(s, sums[0]), alpha = scal[0];
    double tau = 0.0, beta = alpha, scale = 0.0;
    if (sigma > 0.0) {
      beta = sqrt(alpha * alpha + sigma);
      if (alpha > 0.0) beta = -beta;
      tau = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
    }
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = tid + QT * k;
      v[k] = c > j + 1 && c < n ? x[k] * scale : c == j + 1 ? 1.0 : 0.0;
    }
    if (b == 0 && tid == 0) T.e[j] = beta;
    // own rows > j: the previous reflector's update, and their products with this one
    const int par = j & 1, next_b = (j + 1) % G, next_r = (j + 1) / G;
    double *gp = pub + (size_t)par * 2 * n, *grow = gp + n;
    const int r0 = j < b ? 0 : (j - b) / G + 1;  // first own row > j
    double part[2][8];
#pragma unroll
    for (int q = 0; q < 8; ++q) part[0][q] = part[1][q] = 0.0;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      if (r < rs && r >= r0) {
        const double vi = vs[b + G * r], wi = ws[b + G * r];
        double *row = sA + (size_t)r * n;
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < KC; ++k) {
          const int c = tid + QT * k;
          if (c > j && c < n) {
            const double y = rank2(row[c], vi, wi, vp[k], wp[k]);
            row[c] = y;
            acc = __fma_rn(y, v[k], acc);
            if (b == next_b && r == next_r) __stcg(grow + c, y);
          }
        }
        part[0][r] = acc;
      }
    }
#pragma unroll
    for (int r = 0; r < RR; ++r) {
      const int lr = rs + r, i = b + G * lr;
      if (lr >= r0 && i < n) {
        const double vi = vs[i], wi = ws[i];
        double acc = 0.0;
#pragma unroll
        for (int k = 0; k < KC; ++k) {
          a[r][k] = rank2(a[r][k], vi, wi, vp[k], wp[k]);
          acc = __fma_rn(a[r][k], v[k], acc);
        }
        part[1][r] = acc;
        if (b == next_b && lr == next_r)
#pragma unroll
          for (int k = 0; k < KC; ++k) {
            const int c = tid + QT * k;
            if (c > j && c < n) __stcg(grow + c, a[r][k]);
          }
      }
    }
    const int slot = ((lane & 16) ? 4 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 1 : 0);
    if (rs > 0) {
      const double t = warp_sum8(part[0], lane);
      if ((lane & 3) == 0) rows_red[0][warp][slot] = t;
    }
    {
      const double t = warp_sum8(part[1], lane);
      if ((lane & 3) == 0) rows_red[1][warp][slot] = t;
    }
    __syncthreads();
    if (tid < 256) {
      const int set = tid >> 7, row = (tid >> 4) & 7, w = tid & 15;
      double t = rows_red[set][w][row];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      const int lr = set == 0 ? row : rs + row, i = b + G * lr;
      if (w == 0 && lr >= r0 && i < n && (set == 0 ? row < rs : row < RR)) __stcg(gp + i, t);
    }
    if (!tri_sync(count, epoch, error)) return;
    // w = tau p - (tau^2 / 2) (p . v) v; row j + 1 after this reflector
    double p[KC], y[KC];
    s = 0.0;
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = tid + QT * k;
      p[k] = y[k] = 0.0;
      if (c > j && c < n) {
        p[k] = __ldcg(gp + c);
        y[k] = __ldcg(grow + c);
      }
    }
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      if (tid + QT * k == j + 1) scal[1] = p[k];
      s += p[k] * v[k];
    }
    const double pv = cta_sum(s, sums[1]);
    const double half = 0.5 * tau * tau * pv, w1 = tau * scal[1] - half;
#pragma unroll
    for (int k = 0; k < KC; ++k) {
      const int c = tid + QT * k;
      const double w = tau * p[k] - half * v[k];
      x[k] = y[k] - w - w1 * v[k];
      vp[k] = v[k];
      wp[k] = w;
      if (c > j && c < n) {
        vs[c] = v[k];
        ws[c] = w;
      }
      if (c == j + 1 && b == 0) T.d[j + 1] = x[k];
    }
  }
  // Gershgorin interval, pivot floor and squared off-diagonal for the Sturm counts
  __threadfence();
  __syncthreads();
  if (b == 0) {
    double lo = 1e300, hi = -1e300, emax = 0.0;
    for (int i = tid; i < n; i += QT) {
      const double el = i > 0 ? fabs(__ldcg(T.e + i - 1)) : 0.0, er = i < n - 1 ? fabs(__ldcg(T.e + i)) : 0.0;
      const double di = __ldcg(T.d + i);
      lo = fmin(lo, di - el - er);
      hi = fmax(hi, di + el + er);
      emax = fmax(emax, er * er);
      if (i < n - 1) T.vec[i] = er * er;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    }
    if (lane == 0) {
      rows_red[0][warp][0] = lo;
      rows_red[0][warp][1] = hi;
      rows_red[0][warp][2] = emax;
    }
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < QW; ++w) {
        lo = fmin(lo, rows_red[0][w][0]);
        hi = fmax(hi, rows_red[0][w][1]);
        emax = fmax(emax, rows_red[0][w][2]);
      }
      const double tnorm = fmax(fabs(lo), fabs(hi));
      const double pivmin = 2.2250738585072014e-308 * fmax(1.0, emax) * 16.0;
      const double pad = 2.1 * n * 2.220446049250313e-16 * tnorm + 4.0 * pivmin;
      T.part[0] = lo - pad;
      T.part[1] = hi + pad;
      T.part[2] = pivmin;
    }
  }
}

constexpr int kGridSmem = 224 * 1024;
struct GridShape {
  const void *fn;
  int rr, ctas, rs;
};

int tri_sms() {
  static std::mutex mu;
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  int &s = sms[dev & 63];
  if (s == 0) {
    for (const void *fn : {(const void *)k_tridiag_grid<1, 4>, (const void *)k_tridiag_grid<2, 7>,
                           (const void *)k_tridiag_grid<3, 7>, (const void *)k_tridiag_grid<4, 7>})
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kGridSmem);
    if (cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) s = 148;
  }
  return s;
}

// Columns per thread by the order; as many CTAs as leave no more rows each than the registers hold,
// at most one per SM, the rest of the rows in shared memory.
GridShape grid_shape(int n, int ctas) {
  const int sms = tri_sms(), kc = (n + QT - 1) / QT;
  GridShape g{};
  g.rr = kc == 1 ? 4 : 7;
  g.fn = kc == 1   ? (const void *)k_tridiag_grid<1, 4>
         : kc == 2 ? (const void *)k_tridiag_grid<2, 7>
         : kc == 3 ? (const void *)k_tridiag_grid<3, 7>
                   : (const void *)k_tridiag_grid<4, 7>;
  g.ctas = ctas > 0 ? ctas : std::min(sms, (n + g.rr - 1) / g.rr);
  g.rs = std::max(0, (n + g.ctas - 1) / g.ctas - g.rr);
  return g;
}

}  // namespace

bool tridiag_grid_supported(int n, int ctas) {
  if (n < 2 || n > kTriGridMax || ctas < 0 || ctas > std::min(n, tri_sms())) return false;
  const GridShape g = grid_shape(n, ctas);
  return g.rs <= 8 && (size_t)(2 + g.rs) * n * 8 <= (size_t)kGridSmem;
}

cudaError_t launch_tridiag_grid(cudaStream_t st, EigvalsTask t, int *error, int ctas) {
  const GridShape g = grid_shape(t.n, ctas);
  double *pub = t.V;  // the blocked kernel's panel space
  unsigned *count = reinterpret_cast<unsigned *>(t.part + 4);
  cudaError_t err = cudaMemsetAsync(count, 0, sizeof(unsigned), st);
  int rs = g.rs;
  void *args[] = {&t, &rs, &pub, &count, &error};
  if (err == cudaSuccess)
    err = cudaLaunchCooperativeKernel(g.fn, dim3(g.ctas), dim3(QT), args, (size_t)(2 + rs) * t.n * 8, st);
  note_launch();
  if (err != cudaSuccess) cudaGetLastError();  // the status is returned; no later check is to find it again
  return err;
}

}  // namespace pm7
