// A whole fp64 SP2 purification in one cooperative launch: spectral bounds (Gershgorin and
// Lanczos), the start iterate, every squaring with its update, decision and stopping rule, and
// the density, with grid barriers in between.
//
// Bound: below ~768 orbitals a purification is a chain of ~20 dependent squarings whose
// arithmetic is small (n = 270: 1e7 FMA, 0.7 us of the chip's FP64 tensor rate), so what counts
// is the latency of a link. As separate launches a link cost a decision kernel and a squaring of
// 64-wide tiles on a few SMs, and the 34 launches of the Lanczos bounds 173 us per purification.
// Here a link is a grid barrier and one or two tiles of 32 x 32 per CTA (n = 200 already gives 28
// of them). A dependent chain of DMMA steps runs at the tensor sub-core's full rate (64 clk per
// m16n8k8, measured), so K is not split: eight product warps hold one 16 x 8 accumulation chain
// each (two per sub-core: one alone cannot hide its fragment loads, 100 clk per step), and every
// element is the same chain over k as in the other FP64 products. Four loader warps stream the
// panels through a cp.async ring; four more sum the step's decision meanwhile and then finish the
// tiles (update, mirror, traces), beside the next tile's products.
//
// Every sum is taken in an order that depends on the matrix order alone (elements, rows, blocks
// of 64), never on the grid, so the result has the same bits on every grid; products and sums
// whose rounding decides a branch are written out, so that no contraction changes them.
//
// Measured (one purification of ~16 steps, CUDA events around it in a solve): n = 121 0.18 ms (two spins
// 36 -> 14 ms a solve), n = 204 0.73 -> 0.20, n = 310 0.26, n = 666 1.36 -> 0.50 ms; a step 24 -> 5.3 us
// at n = 121, 54 -> 20 us at n = 666 (11 us of it DMMA issue), the Lanczos bounds 173 -> 70 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "autotune.hpp"
#include "common.cuh"
#include "kernels.hpp"
#include "tcgen05.cuh"

namespace pm7 {
namespace {

constexpr int GT = 512;                        // threads of a purification CTA: 8 product, 4 finishing, 4 loader warps
constexpr int TS = 32;                         // tile edge, and K rows of a stage
constexpr int STAGES = 6;
constexpr int LA = TS + 4;                     // row stride of a panel in a stage, padded against bank conflicts
constexpr int STAGE = 2 * TS * LA;             // doubles
constexpr int LT = 34;                         // row stride of a finished tile
constexpr int kTile = TS * LT;
constexpr int kSmem = (STAGES * STAGE + 2 * kTile) * 8;
constexpr int kBoundsThreads = 1024;           // of a CTA that only finds the bounds
constexpr int kNormBlocks = 296;               // partial sums of the start iterate's norms
constexpr int kMaxCtas = 512;
constexpr unsigned long long kGridWaitNs = 1000000000ull;  // a grid barrier gives up after 1 s

struct Sp2GridArgs {
  int n, ld;              // order, padded row length of the iterates (multiple of 32)
  const double *F;        // n x n
  double *x0, *x1;        // ping-pong iterates, ld x ld
  double *P;              // w * the projector, n x n
  double w, n_occ;
  Sp2Rule rule;
  double slack;           // sp2_sum_slack(n)
  int lanczos;            // 1: Lanczos-narrowed bounds, 0: Gershgorin, 2: take bounds as given
  double *bounds;         // the interval used (in and out)
  double *state;          // Sp2State of the last step
  double *ws;             // sp2_grid_doubles(n), zero before the first launch
  unsigned *count;        // barrier arrivals, zero at launch
  int *error;             // 1: a barrier wait expired
};

// Workspace (doubles): per-CTA Gershgorin pairs | two mat-vec results | norm partials |
// two sets of (per 64 x 64 lower block and row: |.|^2 of its two 32-column spans, as
// [row][span][block]; the diagonal).
__host__ __device__ __forceinline__ int blocks64(int n) {
  const int t = (n + 63) / 64;
  return t * (t + 1) / 2;
}
struct WsLayout {
  size_t w, norms, rows, diag, set, total;
  __host__ __device__ explicit WsLayout(int n) {
    w = 2 * kMaxCtas;
    norms = w + 2 * (size_t)((n + 1) & ~1);
    rows = norms + 2 * kNormBlocks;
    set = (size_t)128 * blocks64(n) + 64 * (size_t)((n + 63) / 64);
    diag = (size_t)128 * blocks64(n);
    total = rows + 2 * set;
  }
};

// All CTAs of a cooperative launch (what they wrote before is visible after, to loads that go to
// L2: the release covers the CTA's writes ordered before it by the block barrier); epoch e waits
// for e * gridDim.x arrivals. False, in every thread of the CTA, once a wait has expired anywhere
// (the caller returns).
__device__ __forceinline__ bool grid_sync(unsigned *count, unsigned &epoch, int *error) {
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
        if (t - t0 > kGridWaitNs || *(volatile int *)error != 0) {
          atomicExch(error, 1);
          bad = 1;
          break;
        }
      }
    }
  }
  return __syncthreads_or(bad) == 0;
}

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void dmma(double *d, const double *a, const double *b) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};\n"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// Index t of a lower triangle: row r, column t - r (r + 1) / 2.
__device__ __forceinline__ void triangle_of(int t, int &r, int &c) {
  r = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while ((r + 1) * (r + 2) / 2 <= t) ++r;
  while (r * (r + 1) / 2 > t) --r;
  c = t - r * (r + 1) / 2;
}
__device__ __forceinline__ double warp_down(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Sum over i < n, every thread gets it: 1,024 strided partials (s = f(i, s)), a shuffle tree per
// 32 of them, the tree results in ascending order. T threads. One barrier;
// the caller alternates `red` (32 doubles).
template <int T, class Fn>
__device__ __forceinline__ double sum1024(int n, double *red, Fn f) {
    for (int v = threadIdx.x; v < min(1024, (n + 31) & ~31); v += T) {
    double s = 0.0;
    for (int i = v; i < n; i += 1024) s = f(i, s);
    s = warp_down(s);
    if ((threadIdx.x & 31) == 0) red[v >> 5] = s;
  }
  __syncthreads();
  const int warps = min(32, (n + 31) / 32);  // the others are zero
  double s = 0.0;
  for (int w = 0; w < warps; ++w) s += red[w];
  return s;
}

__device__ int sturm_count(const double *a, const double *b, double x) {
  int c = 0;
  double q = a[0] - x;
  if (q == 0.0) q = -1.0e-300;
  c += q < 0.0;
  for (int i = 1; i < kLzSteps; ++i) {
    q = a[i] - x - b[i] * b[i] / q;
    if (q == 0.0) q = -1.0e-300;
    c += q < 0.0;
  }
  return c;
}

// One warp: the eigenvalue of the Lanczos tridiagonal at which the Sturm count reaches `target`,
// by 32-point multisection (12 rounds shrink the interval by 33^12).
__device__ double lanczos_extreme(const double *a, const double *b, double lo, double hi, int target, int lane) {
  for (int it = 0; it < 12; ++it) {
    const double x = lo + (hi - lo) * (double)(lane + 1) / 33.0;
    const unsigned hit = __ballot_sync(0xffffffffu, sturm_count(a, b, x) >= target);
    const double xl = __shfl_sync(0xffffffffu, x, hit ? __ffs(hit) - 1 : 31);
    if (hit) {
      const int f = __ffs(hit) - 1;
      const double xp = __shfl_sync(0xffffffffu, x, f > 0 ? f - 1 : 0);
      hi = xl;
      if (f > 0) lo = xp;
    } else {
      lo = xl;
    }
  }
  return hi;
}

constexpr int kRowsKept = 8, kColsKept = 3;  // F rows a 256-thread group keeps in registers (n <= 768)

// The interval [lo, hi] that holds F's spectrum, the same in every CTA: Gershgorin widened by
// 1e-3 of its range, and with lanczos the Ritz interval of kLzSteps steps (2% and 4% of the
// range beyond its ends) inside it. Rows are dealt to groups of 256 threads; KEEP: a group keeps
// its rows of F in registers through the Lanczos steps where they fit. v: 3 n doubles of shared
// memory. False: a barrier expired.
template <int T, bool KEEP>
__device__ bool spectral_bounds(const Sp2GridArgs &A, double *v, unsigned &epoch, double &lo_out, double &hi_out) {
  constexpr int G = T / 256;
  const int n = A.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = threadIdx.x >> 8, gt = threadIdx.x & 255, gwarp = gt >> 5;
  const int row0 = blockIdx.x * G + group, rstep = gridDim.x * G;
  __shared__ double alpha[kLzSteps], beta[kLzSteps + 1], ends[4], rr[2][32], mm[2][T / 32];
  __shared__ double dots[G][kRowsKept][8];
  const WsLayout L(n);
  double *gpart = A.ws, *wbuf = A.ws + L.w;
  const bool lz = A.lanczos == 1 && n >= 2 * kLzSteps;
  const bool keep = KEEP && n <= 256 * kColsKept && n <= rstep * kRowsKept;
  double f[KEEP ? kRowsKept : 1][KEEP ? kColsKept : 1];
  if (KEEP && keep) {
#pragma unroll
    for (int i = 0; i < kRowsKept; ++i)
#pragma unroll
      for (int u = 0; u < kColsKept; ++u) {
        const int row = row0 + i * rstep, k = gt + 256 * u;
        f[KEEP ? i : 0][KEEP ? u : 0] = row < n && k < n ? A.F[(size_t)row * n + k] : 0.0;
      }
  }
  double lo = 1.0e300, hi = -1.0e300;
  for (int row = blockIdx.x * (T / 32) + warp; row < n; row += gridDim.x * (T / 32)) {
    const double *fi = A.F + (size_t)row * n;
    double off = 0.0;
    for (int j = lane; j < n; j += 32)
      if (j != row) off += fabs(fi[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
    lo = fmin(lo, fi[row] - off);
    hi = fmax(hi, fi[row] + off);
  }
  if (lane == 0) {
    mm[0][warp] = lo;
    mm[1][warp] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < T / 32; ++w) {
      lo = fmin(lo, mm[0][w]);
      hi = fmax(hi, mm[1][w]);
    }
    __stcg(reinterpret_cast<double2 *>(gpart) + blockIdx.x, make_double2(lo, hi));
  }
  double *vc = v, *vp = v + n, *sw = v + 2 * n;
  if (lz) {
    // v_0: a fixed, dense, normalised start vector
    for (int i = threadIdx.x; i < n; i += T) {
      vc[i] = 1.0 + 0.5 * sin(0.7 * i);
      vp[i] = 0.0;
    }
    __syncthreads();
    const double s0 = sum1024<T>(n, rr[0], [&](int i, double s) { return __fma_rn(vc[i], vc[i], s); });
    const double inv0 = 1.0 / sqrt(s0);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += T) vc[i] *= inv0;
    if (threadIdx.x == 0) beta[0] = 0.0;
    __syncthreads();
    double bj = 0.0;
    for (int j = 0; j < kLzSteps; ++j) {
      // w = F v_j: per row, 256 strided partials, a shuffle tree per 32, a tree over the 8
      double *wj = wbuf + (size_t)(j & 1) * n;
      for (int rb = 0; row0 - group + rb * rstep < n; rb += kRowsKept) {
#pragma unroll
        for (int i = 0; i < kRowsKept; ++i) {
          const int row = row0 + (rb + i) * rstep;
          if (row >= n) break;
          double acc = 0.0;
          if (KEEP && keep) {
            double x[8] = {};
#pragma unroll
            for (int u = 0; u < kColsKept; ++u)
              x[u] = gt + 256 * u < n ? __dmul_rn(f[KEEP ? i : 0][KEEP ? u : 0], vc[gt + 256 * u]) : 0.0;
            acc += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
          } else {
            const double *fi = A.F + (size_t)row * n;
            for (int base = gt; base < n; base += 2048) {
              double x[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                const int k = base + 256 * u;
                x[u] = k < n ? __dmul_rn(fi[k], vc[k]) : 0.0;
              }
              acc += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
            }
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          if (lane == 0) dots[group][i][gwarp] = acc;
        }
        bar_sync(1 + group, 256);
        if (gt < kRowsKept && row0 + (rb + gt) * rstep < n) {
          const double *d = dots[group][gt];
          __stcg(wj + row0 + (rb + gt) * rstep, ((d[0] + d[1]) + (d[2] + d[3])) + ((d[4] + d[5]) + (d[6] + d[7])));
        }
        bar_sync(1 + group, 256);
      }
      if (!grid_sync(A.count, epoch, A.error)) return false;
      // every CTA advances the recurrence itself: alpha = w.v, w -= alpha v + beta v_prev, v_next = w / |w|
      for (int i = threadIdx.x; i < n; i += T) sw[i] = __ldcg(wj + i);
      __syncthreads();
      const double a = sum1024<T>(n, rr[0], [&](int i, double s) { return __dadd_rn(s, __dmul_rn(sw[i], vc[i])); });
      for (int i = threadIdx.x; i < n; i += T)
        sw[i] = __fma_rn(-bj, vp[i], __fma_rn(-a, vc[i], sw[i]));  // (v_{-1} = 0)
      __syncthreads();
      const double s2 = sum1024<T>(n, rr[1], [&](int i, double s) { return __fma_rn(sw[i], sw[i], s); });
      bj = sqrt(s2);
      if (threadIdx.x == 0) {
        alpha[j] = a;
        beta[j + 1] = bj;
      }
      const double inv = bj > 1.0e-280 ? 1.0 / bj : 0.0;  // an invariant subspace: v stops
      for (int i = threadIdx.x; i < n; i += T) vp[i] = sw[i] * inv;  // the next vector replaces v_prev
      double *x = vp;
      vp = vc;
      vc = x;
      __syncthreads();
    }
  } else if (!grid_sync(A.count, epoch, A.error)) {
    return false;
  }
  if (warp == 0) {
    double a = 1.0e300, b = -1.0e300;
    for (int i = lane; i < (int)gridDim.x; i += 32) {
      const double2 p = __ldcg(reinterpret_cast<const double2 *>(gpart) + i);
      a = fmin(a, p.x);
      b = fmax(b, p.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
      b = fmax(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if (lane == 0) {
      // widened so that no level starts on 0 or 1 (fixed points of both SP2 maps)
      const double pad = 1.0e-3 * (b - a) + 1.0e-6;
      ends[0] = a - pad;
      ends[1] = b + pad;
    }
  }
  if (lz && (warp == 1 || warp == 2)) {
    double g_lo = 1.0e300, g_hi = -1.0e300;
    for (int i = 0; i < kLzSteps; ++i) {
      const double r = (i > 0 ? fabs(beta[i]) : 0.0) + (i + 1 < kLzSteps ? fabs(beta[i + 1]) : 0.0);
      g_lo = fmin(g_lo, alpha[i] - r);
      g_hi = fmax(g_hi, alpha[i] + r);
    }
    // smallest: count(x) >= 1; largest: count(x) >= kLzSteps
    const double e = lanczos_extreme(alpha, beta, g_lo, g_hi, warp == 1 ? 1 : kLzSteps, lane);
    if (lane == 0) ends[1 + warp] = e;
  }
  __syncthreads();
  lo_out = ends[0];
  hi_out = ends[1];
  if (lz) {
    const double tmin = ends[2], tmax = ends[3], R = tmax - tmin;
    if (R > 0.0 && isfinite(R)) {  // else the Gershgorin interval
      const double elo = fmax(tmin - 0.02 * R, lo_out), ehi = fmin(tmax + 0.04 * R, hi_out);
      const double pad = 1.0e-3 * (ehi - elo) + 1.0e-6;
      lo_out = fmax(elo - pad, lo_out);
      hi_out = fmin(ehi + pad, hi_out);
    }
  }
  return true;
}

__global__ void __launch_bounds__(kBoundsThreads) k_sp2_bounds(Sp2GridArgs A) {
  extern __shared__ __align__(16) double sp2_smem[];
  unsigned epoch = 0;
  double lo, hi;
  if (!spectral_bounds<kBoundsThreads, false>(A, sp2_smem, epoch, lo, hi)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.bounds[0] = lo;
    A.bounds[1] = hi;
  }
}

// Both sums over the 8 virtual warps whose tree results are in wpart, in order; the finishing
// warps call this together (bar 1), before and after.
__device__ __forceinline__ void join_traces(double (&wpart)[2][8], double &a, double &b) {
  bar_sync(1, 128);
  a = b = 0.0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    a += wpart[0][w];
    b += wpart[1][w];
  }
  bar_sync(1, 128);
}

// The traces in their defining order: partials per 64 x 64 block (its rows' span sums in
// ascending order), 256 strided sums of them, a shuffle tree per 32, the 8 results in order; for
// the first step the start iterate's norm partials in place of the blocks.
__device__ __noinline__ void exact_traces(const double *pin, const double *norms, const WsLayout &L, int nb, int step,
                                          int at, int lane, double (&wpart)[2][8], double &a, double &b) {
  for (int half = 0; half < 2; ++half) {
    const int vt = at + 128 * half;
    double da = 0.0, db = 0.0;
    if (step == 0) {
      for (int i = vt; i < kNormBlocks; i += 256) {
        const double2 p = __ldcg(reinterpret_cast<const double2 *>(norms) + i);
        da += p.x;
        db += p.y;
      }
    } else {
      for (int k = vt; k < nb; k += 256) {
        int R, C;
        triangle_of(k, R, C);
        double sa = 0.0, sb = 0.0;
        const double *p = pin + k;
#pragma unroll 32
        for (int r = 0; r < 64; ++r) sb += __ldcg(p + (size_t)(2 * r) * nb) + __ldcg(p + (size_t)(2 * r + 1) * nb);
        if (R == C) {
          const double *d = pin + L.diag + 64 * R;
#pragma unroll 32
          for (int r = 0; r < 64; ++r) sa += __ldcg(d + r);
        }
        da += sa;
        db += sb;
      }
    }
    da = warp_down(da);
    db = warp_down(db);
    if (lane == 0) {
      wpart[0][(at >> 5) + 4 * half] = da;
      wpart[1][(at >> 5) + 4 * half] = db;
    }
  }
  join_traces(wpart, a, b);
}

// Sum of m values by 128 threads, 16 loads of each in flight.
__device__ __forceinline__ double quick_sum(const double *p, int m, int at) {
  double s = 0.0;
  for (int base = at; base < m; base += 16 * 128) {
    double x[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) x[q] = base + 128 * q < m ? __ldcg(p + base + 128 * q) : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < o; ++q) x[q] += x[q + o];
    s += x[0];
  }
  return s;
}

// The same sums in the order the loads come in.
__device__ __forceinline__ void quick_traces(const double *pin, const double *norms, const WsLayout &L, int nb, int n,
                                             int step, int at, int lane, double (&wpart)[2][8], double &a, double &b) {
  double da = 0.0, db = 0.0;
  if (step == 0) {
    for (int i = at; i < kNormBlocks; i += 128) {
      const double2 p = __ldcg(reinterpret_cast<const double2 *>(norms) + i);
      da += p.x;
      db += p.y;
    }
  } else {
    da = quick_sum(pin + L.diag, n, at);
    db = quick_sum(pin, 128 * nb, at);
  }
  da = warp_down(da);
  db = warp_down(db);
  if (lane == 0) {
    wpart[0][at >> 5] = da;
    wpart[1][at >> 5] = db;
    wpart[0][4 + (at >> 5)] = wpart[1][4 + (at >> 5)] = 0.0;
  }
  join_traces(wpart, a, b);
}

// Named barriers of the purification: 1 finishing warps, 2 + b tile buffer b is full, 4 + b tile
// buffer b is free (spectral_bounds uses 1 and 2 before).
__global__ void __launch_bounds__(GT) k_sp2_purify(Sp2GridArgs A) {
  extern __shared__ __align__(16) double sp2_smem[];
  __shared__ double wpart[2][8];
  __shared__ int verdict;
  __shared__ uint64_t full[STAGES], empty[STAGES];
  __shared__ int late;  // a pipeline wait expired
  const int n = A.n, ld = A.ld, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned epoch = 0;
  double lo, hi;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(&full[s], 128);
      tc::mbar_init(&empty[s], 8);
    }
    late = 0;
  }
  if (A.lanczos == 2) {
    lo = A.bounds[0];
    hi = A.bounds[1];
  } else if (!spectral_bounds<GT, true>(A, sp2_smem, epoch, lo, hi)) {
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.bounds[0] = lo;
    A.bounds[1] = hi;
  }
  const WsLayout L(n);
  double *norms = A.ws + L.norms;
  const int nb = blocks64(n);

  // X = (hi I - F) / (hi - lo): spectrum in [0, 1], occupied levels near 1; zero padding
  const double inv = 1.0 / (hi - lo);
  for (int i = blockIdx.x * (GT / 32) + warp; i < ld; i += gridDim.x * (GT / 32))
    for (int j = lane; j < ld; j += 32)
      __stcg(A.x0 + (size_t)i * ld + j,
             i < n && j < n ? ((i == j ? hi : 0.0) - A.F[(size_t)i * n + j]) * inv : 0.0);
  // its trace and |X|_F^2 (= tr X^2: X is symmetric) as kNormBlocks partials of 256 strided sums
  // (shuffle trees per 32, the 8 results in order)
  for (int vb = blockIdx.x; vb < kNormBlocks; vb += gridDim.x) {
    const size_t len = (size_t)n * n;
    double tr = 0.0, sq = 0.0;
    if (threadIdx.x < 256)
      for (size_t e = (size_t)vb * 256 + threadIdx.x; e < len; e += (size_t)kNormBlocks * 256) {
        const size_t i = e / n, j = e - i * n;
        const double v = ((i == j ? hi : 0.0) - A.F[e]) * inv;
        sq = __fma_rn(v, v, sq);
        if (i == j) tr += v;
      }
    tr = warp_down(tr);
    sq = warp_down(sq);
    __syncthreads();
    if (lane == 0 && warp < 8) {
      wpart[0][warp] = tr;
      wpart[1][warp] = sq;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      tr = sq = 0.0;
      for (int w = 0; w < 8; ++w) {
        tr += wpart[0][w];
        sq += wpart[1][w];
      }
      __stcg(reinterpret_cast<double2 *>(norms) + vb, make_double2(tr, sq));
    }
  }
  if (!grid_sync(A.count, epoch, A.error)) return;

  const int tb = ld / TS, tiles = tb * (tb + 1) / 2, slabs = tb;
  const int mine = (int)blockIdx.x < tiles ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  double *T = sp2_smem + STAGES * STAGE;
  double ring[3] = {0.0, 0.0, 0.0};
  unsigned it = 0;  // slabs through the ring so far (product and loader warps)
  for (int step = 0;; ++step) {
    const double *X = step % 2 == 0 ? A.x0 : A.x1;
    double *Y = step % 2 == 0 ? A.x1 : A.x0;
    if (warp >= 12) {
      // loaders: the two panels' 32-row slabs, 16 bytes per copy; X through L2, other CTAs wrote it
      const int tid = threadIdx.x - 384, row = tid >> 4, col = (tid & 15) * 2;
      const unsigned dst = tc::smem_u32(sp2_smem + row * LA + col);
      for (int u = 0; u < mine; ++u) {
        int bm, bn;
        triangle_of(blockIdx.x + u * gridDim.x, bm, bn);
        const double *sa = X + (size_t)row * ld + bm * TS + col, *sb = X + (size_t)row * ld + bn * TS + col;
        for (int k = 0; k < slabs; ++k, ++it) {
          const unsigned s = it % STAGES;
          if (it >= STAGES) tc::mbar_wait(&empty[s], (it / STAGES - 1) & 1, &late);
          const unsigned d = dst + s * STAGE * 8;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + q * 8 * LA * 8),
                         "l"(sa + (size_t)q * 8 * ld)
                         : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + (TS + q * 8) * LA * 8),
                         "l"(sb + (size_t)q * 8 * ld)
                         : "memory");
          }
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(&full[s])) : "memory");
          sa += (size_t)TS * ld;
          sb += (size_t)TS * ld;
        }
      }
    } else if (warp < 8) {
      // products X^T X (X is symmetric: column m of the left factor is a row): warp tile 16 x 8,
      // fragments as the PTX ISA lays out .f64 m16n8k8
      const int g = lane >> 2, t4 = lane & 3, wm = (warp >> 2) * 16, wn = (warp & 3) * 8;
      const double *fa = sp2_smem + t4 * LA + wm + g, *fb = sp2_smem + (TS + t4) * LA + wn + g;
      for (int u = 0; u < mine; ++u) {
        double acc[4] = {};
        for (int k = 0; k < slabs; ++k, ++it) {
          const unsigned s = it % STAGES;
          tc::mbar_wait(&full[s], (it / STAGES) & 1, &late);
          const double *pa = fa + s * STAGE, *pb = fb + s * STAGE;
#pragma unroll
          for (int kk = 0; kk < TS; kk += 8) {
            const double a[4] = {pa[kk * LA], pa[kk * LA + 8], pa[(kk + 4) * LA], pa[(kk + 4) * LA + 8]};
            const double b[2] = {pb[kk * LA], pb[(kk + 4) * LA]};
            dmma(acc, a, b);
          }
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(&empty[s])) : "memory");
        }
        double *tile = T + (u & 1) * kTile;
        if (u >= 2) bar_sync(4 + (u & 1), 384);  // its previous tile has been finished
        double *p = tile + (wm + g) * LT + wn + 2 * t4;
        *reinterpret_cast<double2 *>(p) = make_double2(acc[0], acc[1]);
        *reinterpret_cast<double2 *>(p + 8 * LT) = make_double2(acc[2], acc[3]);
        bar_arrive(2 + (u & 1), 384);
      }
    } else {
      const int at = threadIdx.x - 256;
      const double *pin = A.ws + L.rows + (size_t)(step & 1) * L.set;
      double *pout = A.ws + L.rows + (size_t)((step + 1) & 1) * L.set;
      // The iterate's traces tr X and tr X^2 = |X|_F^2, the branch (square when it brings the trace
      // closer to n_occ) and the stopping rule of sp2_control, the same in every CTA. The sums are
      // defined in one order (exact_traces), whose long chains of additions cost more than a small
      // step; a quick sum differs from them by less than `off` (A.slack: see sp2_sum_slack), so it
      // decides whenever no comparison is that close.
      double trx, trx2;
      quick_traces(pin, norms, L, nb, n, step, at, lane, wpart, trx, trx2);
      double e = trx - trx2;
      const double off = A.slack * (fabs(trx) + trx2) + 1.0e-15;
      const double d1 = fabs(trx2 - A.n_occ), d2 = fabs(2.0 * trx - trx2 - A.n_occ);
      if (!(fabs(e) > 1.0e-7 + 4.0 * off && fabs(d1 - d2) > 8.0 * off) || fabs(fabs(e) - A.rule.tol_floor) < 4.0 * off ||
          fabs(fabs(e) - A.rule.tol_done) < 4.0 * off || (step >= 2 && fabs(fabs(e) - fabs(ring[1])) < 8.0 * off)) {
        exact_traces(pin, norms, L, nb, step, at, lane, wpart, trx, trx2);
        e = trx - trx2;
      }
      const bool square = fabs(trx2 - A.n_occ) < fabs(2.0 * trx - trx2 - A.n_occ);
      const double prev2 = step >= 2 ? ring[1] : 0.0;
      ring[1] = ring[0];
      ring[0] = e;
      bool stop = false, ok = false;
      if (!isfinite(e)) stop = true;
      else if (fabs(e) <= A.rule.tol_done) stop = ok = true;
      else if (step >= 2 && fabs(e) < A.rule.tol_floor && fabs(e) >= fabs(prev2)) stop = ok = true;
      else if (step + 1 >= A.rule.max_steps) stop = true;
      if (at == 0) {
        verdict = stop;
        if (stop && blockIdx.x == 0) {
          A.state[kSp2TrX] = trx;
          A.state[kSp2TrX2] = trx2;
          A.state[kSp2Square] = square ? 1.0 : 0.0;
          A.state[kSp2Err] = e;
          A.state[kSp2Stop] = (double)step;
          A.state[kSp2Ok] = ok ? 1.0 : 0.0;
        }
      }
      // finish the tiles: four threads per row, the two columns 8 j + 2 t of each
      const int r = at >> 2, t = at & 3;
      for (int u = 0; u < mine; ++u) {
        int bm, bn;
        triangle_of(blockIdx.x + u * gridDim.x, bm, bn);
        const int m0 = bm * TS, n0 = bn * TS;
        const bool diag = bm == bn;  // only elements with row >= column count
        double2 own[4] = {};
        if (!square)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            own[j] = __ldcg(reinterpret_cast<const double2 *>(X + (size_t)(m0 + r) * ld + n0 + 8 * j + 2 * t));
        double *tile = T + (u & 1) * kTile;
        bar_sync(2 + (u & 1), 384);
        double rsq = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          double2 *tp = reinterpret_cast<double2 *>(tile + r * LT + 8 * j + 2 * t);
          const double2 x2 = *tp;
          double y[2] = {x2.x, x2.y};
          const double xo[2] = {own[j].x, own[j].y};
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int c = 8 * j + 2 * t + q;
            if (!square) y[q] = 2.0 * xo[q] - y[q];
            if (diag && r < c) continue;
            if (diag && r == c) {
              rsq = __dadd_rn(rsq, __dmul_rn(y[q], y[q]));
              if (!stop) __stcg(pout + L.diag + m0 + r, y[q]);
            } else {
              rsq = __dadd_rn(rsq, 2.0 * __dmul_rn(y[q], y[q]));
            }
          }
          *tp = make_double2(y[0], y[1]);
          if (!diag && !stop)
            __stcg(reinterpret_cast<double2 *>(Y + (size_t)(m0 + r) * ld + n0 + 8 * j + 2 * t), make_double2(y[0], y[1]));
        }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) rsq += __shfl_xor_sync(0xffffffffu, rsq, o);
        if (t == 0 && !stop) {
          const int R = bm >> 1, C = bn >> 1;
          __stcg(pout + (size_t)(2 * ((m0 & 63) + r) + (bn & 1)) * nb + R * (R + 1) / 2 + C, rsq);
        }
        bar_sync(1, 128);  // the tile's final values are in shared memory
        if (stop) {
          // the density: w times the last iterate, both triangles from the lower one
          for (int c = t; c < TS; c += 4) {
            const double v = diag && c > r ? tile[c * LT + r] : tile[r * LT + c];
            if (m0 + r < n && n0 + c < n) A.P[(size_t)(m0 + r) * n + n0 + c] = A.w * v;
            if (!diag && n0 + r < n && m0 + c < n) A.P[(size_t)(n0 + r) * n + m0 + c] = A.w * tile[c * LT + r];
          }
        } else {
          // the mirror, thread = row n0 + r; a diagonal tile whole, from its lower triangle
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int c = 8 * j + 2 * t;
            const double a = diag && c <= r ? tile[r * LT + c] : tile[c * LT + r];
            const double b = diag && c + 1 <= r ? tile[r * LT + c + 1] : tile[(c + 1) * LT + r];
            __stcg(reinterpret_cast<double2 *>(Y + (size_t)(n0 + r) * ld + m0 + c), make_double2(a, b));
          }
        }
        if (u + 2 < mine) bar_arrive(4 + (u & 1), 384);
      }
    }
    __syncthreads();
    if (late) {
      if (warp >= 12) asm volatile("cp.async.wait_all;" ::: "memory");  // no copy outlives the CTA
      if (threadIdx.x == 0) atomicExch(A.error, 1);
      return;
    }
    if (verdict) return;
    if (!grid_sync(A.count, epoch, A.error)) return;
  }
}

// The SMs of the current device; the kernels' shared memory is opted in once per device.
int grid_sms() {
  static std::mutex mu;
  static int sms[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  int &s = sms[dev & 63];
  if (s == 0) {
    cudaFuncSetAttribute(k_sp2_purify, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    cudaFuncSetAttribute(k_sp2_bounds, cudaFuncAttributeMaxDynamicSharedMemorySize, 3 * kSp2BoundsMax * 8);
    if (cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) s = 148;
  }
  return std::min(s, kMaxCtas);
}

cudaError_t grid_launch(cudaStream_t st, const void *fn, int ctas, int threads, size_t smem, Sp2GridArgs &A) {
  cudaError_t err = cudaMemsetAsync(A.count, 0, sizeof(unsigned), st);
  void *args[] = {&A};
  if (err == cudaSuccess) err = cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(threads), args, smem, st);
  note_launch();
  if (err != cudaSuccess) cudaGetLastError();  // the status is returned; no later check is to find it again
  return err;
}

}  // namespace

// What the quick sum and the defining sum of the same non-negative terms may differ by, relative to the
// sum: a rounding (2^-53) per addition in the longest chain of each. Quick: 128 nb / 2,048 in a row, a tree
// over 16, a warp, eight warps; defined: a row's two spans, 64 rows, nb / 256 blocks, a warp, eight
// warps. 1e-13 covers 900 of them, up to 9,900 orbitals; beyond that the chains decide.
double sp2_sum_slack(int n) {
  const int nb = blocks64(n), quick = (128 * nb + 2047) / 2048 + 4 + 5 + 8, defined = 1 + 64 + (nb + 255) / 256 + 5 + 8;
  return std::max(1.0e-13, (quick + defined + 1) * 1.1102230246251565e-16);
}

int sp2_grid_ld(int n) { return (n + TS - 1) / TS * TS; }
size_t sp2_grid_doubles(int n) { return WsLayout(n).total; }

cudaError_t launch_sp2_bounds(cudaStream_t st, int n, const double *F, bool lanczos, double *ws, double *bounds,
                              unsigned *count, int *error) {
  const int sms = grid_sms();
  Sp2GridArgs A{};
  A.n = n;
  A.F = F;
  A.lanczos = lanczos ? 1 : 0;
  A.bounds = bounds;
  A.ws = ws;
  A.count = count;
  A.error = error;
  const int rows = kBoundsThreads / 256;  // at a time per CTA
  return grid_launch(st, (const void *)k_sp2_bounds, std::min(sms, (n + rows - 1) / rows), kBoundsThreads,
                     3 * (size_t)n * 8, A);
}

// The grid of a purification: a CTA per SM at most, no more than there are tiles or (so that a
// CTA keeps its rows of F in registers through the Lanczos steps) row sets; or, the tuner's other
// variant, the fewest CTAs that take the tiles in as many waves, whose barriers are cheaper. While one
// wave takes all tiles the two are the same number and nothing is timed: a timing runs three extra
// purifications (0.45 to 0.6 ms) in the first call of a size bucket.
cudaError_t launch_sp2_purify(cudaStream_t st, int n, const double *F, int lanczos, double n_occ, double w,
                              Sp2Rule rule, double *x0, double *x1, double *P, double *ws, double *bounds,
                              double *state, unsigned *count, int *error) {
  const int sms = grid_sms();
  Sp2GridArgs A{};
  A.n = n;
  A.ld = sp2_grid_ld(n);
  A.F = F;
  A.x0 = x0;
  A.x1 = x1;
  A.P = P;
  A.w = w;
  A.n_occ = n_occ;
  A.rule = rule;
  A.slack = sp2_sum_slack(n);
  A.lanczos = lanczos;
  A.bounds = bounds;
  A.state = state;
  A.ws = ws;
  A.count = count;
  A.error = error;
  if (lanczos == 1 && 3 * (size_t)n * 8 > kSmem) {  // the Lanczos vectors need the other kernel's shared memory
    const cudaError_t err = launch_sp2_bounds(st, n, F, true, ws, bounds, count, error);
    if (err != cudaSuccess) return err;
    A.lanczos = 2;
  }
  const int tb = A.ld / TS, tiles = tb * (tb + 1) / 2, waves = (tiles + sms - 1) / sms;
  const int rows = (n + 2 * kRowsKept - 1) / (2 * kRowsKept);
  const int most = std::min(sms, std::max(tiles, rows));
  const int even = std::min(sms, std::max((tiles + waves - 1) / waves, rows));
  const int bucket = ((n + 255) / 256) * 256;
  // the verdict is "not settled" until a kernel that ran says otherwise
  const cudaError_t err = cudaMemsetAsync(state + kSp2Ok, 0, sizeof(double), st);
  if (err != cudaSuccess) return err;
  auto launch = [&](int v) { return grid_launch(st, (const void *)k_sp2_purify, v == 0 ? most : even, GT, kSmem, A); };
  const int bt = bucket / TS;
  const bool alike = bt * (bt + 1) / 2 <= sms;  // one wave for every order of the bucket
  if (!alike && most == even) return launch(0);
  return autotune_checked(st, "sp2_square|n" + std::to_string(bucket), 2, launch, nullptr, alike);
}

}  // namespace pm7
