// Cyclic Jacobi eigensolver in shared memory, one thread block per symmetric matrix of
// order n <= kJacobiMax, eigenvectors and eigenvalues. Used wherever a matrix that small is
// diagonalised on the SCF path: the plain SCF of a small molecule, the batch's small
// molecules and the divide-and-conquer subsystems; it replaces, for those orders,
// `symmetric_eigen` (pm7-rs src/linalg.rs:231-278, faer's self_adjoint_eigen).
//
// A Fock matrix changes little from one SCF iteration to the next, so the previous
// iteration's eigenvectors W nearly diagonalise it: with `warm` the kernel forms W F W^T and
// runs parallel cyclic Jacobi sweeps on that, which converges in a few sweeps, and accumulates
// the rotations into W; cold, it starts from the identity. The indices are paired off in twos,
// the twos meet by round robin (n/4 disjoint sets of four indices a round) and a set's four cross
// pairs are annihilated in two steps by the small-angle rotation (Golub & Van Loan, sym.schur2);
// the pairs inside the twos come first in a sweep. Sweeps
// stop when the off-diagonal part falls below 1e-15 of the diagonal (Frobenius norms), or
// after kJacSweeps; the job's info word then says whether it converged. Eigenvalues are
// sorted ascending (ties by index) and the eigenvectors written as rows of the np x np slot
// (zero padding; padding eigenvalues `pad`).
#include <cuda_runtime.h>

#include <cmath>

#include "engine_internal.hpp"
#include "kernels.hpp"

namespace pm7 {
namespace {

__device__ __forceinline__ double jac_warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block sum in a fixed order (warps, then warp 0 over the warp sums); result in thread 0.
__device__ double block_sum(double v, double *sh) {
  v = jac_warp_sum(v);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (w == 0) {
    t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    t = jac_warp_sum(t);
  }
  __syncthreads();
  return t;
}

constexpr int kJacSweeps = 24;
constexpr int kJacSets = kJacobiMax / 4;
static_assert(kJacobiMax % 4 == 0 && kJacSets <= 32, "a lane of the first warp per set of four indices");
static_assert(kJacSets * (kJacSets - 1) / 2 <= kJacobiThreads, "a thread per pair of sets");
static_assert(kJacSets * ((kJacobiMax + 7) / 8) <= kJacobiThreads, "a thread per 4 x 8 elements of a product");

// What bounds a round is shared memory (a rotation does four operations on every two elements it
// loads and stores) and the chain that finds the angles. Two steps of a set go over the matrix
// together, so an element is moved once for both; only the tiles on and below the diagonal are kept;
// the angles of the next round are worked out by one warp while the others rotate W. Order 112:
// 6,000 clocks a rotation step with both triangles, an angle phase of its own and an index division
// per element.
//
// Doubles of the matrix of order n4, as tiles or as rows of n4 + 1 (a multiple of two).
__host__ __device__ constexpr size_t jac_matrix(int n4) {
  const size_t blocks = n4 / 2, tiles = 4 * blocks * (blocks | 1), rows = (size_t)n4 * (n4 + 1);
  return tiles > rows ? tiles : rows;
}

// The matrix in 2 x 2 tiles (I, J), I >= J: row a of a tile is one double2 of plane a. An odd number
// of tiles a row keeps lanes that walk I or J free of bank conflicts.
struct JacTiles {
  double2 *t;
  int stride, plane;
  __device__ JacTiles(double *mem, int blocks) : t((double2 *)mem), stride(blocks | 1), plane(blocks * (blocks | 1)) {}
  __device__ double get(int i, int j) const {  // i >= j
    const double2 v = t[(i & 1) * plane + (i >> 1) * stride + (j >> 1)];
    return j & 1 ? v.y : v.x;
  }
  // v[a][b] = element (2 I + a, 2 J + b), from the tile or from its mirror image
  __device__ void load(int I, int J, double &v00, double &v01, double &v10, double &v11) const {
    const int k = max(I, J) * stride + min(I, J);
    const double2 x = t[k], y = t[plane + k];
    const bool low = I >= J;
    v00 = x.x, v11 = y.y;
    v01 = low ? x.y : y.x;
    v10 = low ? y.x : x.y;
  }
  __device__ void store(int I, int J, double v00, double v01, double v10, double v11) const {
    const int k = max(I, J) * stride + min(I, J);
    const bool low = I >= J;
    t[k] = make_double2(v00, low ? v01 : v10);
    t[plane + k] = make_double2(low ? v10 : v01, v11);
  }
};

// The twos of set k in round r of `rounds` (the fixed two 0 meets two r + 1).
__device__ __forceinline__ void jac_set(int k, int r, int rounds, int &I, int &J) {
  int a = r + k, b = r - k;
  if (a >= rounds) a -= rounds;
  if (b < 0) b += rounds;
  I = k == 0 ? 0 : a + 1;
  J = k == 0 ? r + 1 : b + 1;
}

// The small-angle rotation that annihilates apq: with h = sqrt(d^2 + 4 apq^2), cos 2x = |d| / h and
// sin 2x = 2 |apq| / h. (An element below 1e-145 stays.)
__device__ __forceinline__ double2 jac_angle(double app, double aqq, double apq) {
  const double d = aqq - app, h2 = d * d + 4.0 * apq * apq;
  if (apq == 0.0 || h2 < 1.0e-290) return make_double2(1.0, 0.0);
  const double r = rsqrt(h2), c2 = 0.5 + 0.5 * fabs(d) * r, rc = rsqrt(c2);
  const double s = apq * r * rc;
  return make_double2(c2 * rc, d < 0.0 ? -s : s);
}
__device__ __forceinline__ void jac_turn(double2 q, double &x, double &y) {
  const double u = x;
  x = q.x * u - q.y * y;
  y = q.y * u + q.x * y;
}
// A set's steps: (0,2)(1,3), then (0,3)(1,2); first of all in a sweep (0,1)(2,3).
template <class Turn>
__device__ __forceinline__ void jac_steps(bool first, Turn turn) {
  if (first) turn(4, 0, 1), turn(5, 2, 3);
  turn(0, 0, 2), turn(1, 1, 3);
  turn(2, 0, 3), turn(3, 1, 2);
}

// Set k's rotations of round r into q, and the set's own 4 x 4 block.
__device__ void jac_angles(const JacTiles &A, int k, int r, int rounds, double2 *q) {
  int I, J;
  jac_set(k, r, rounds, I, J);
  double a[4][4];
  A.load(I, I, a[0][0], a[0][1], a[1][0], a[1][1]);
  A.load(J, J, a[2][2], a[2][3], a[3][2], a[3][3]);
  A.load(I, J, a[0][2], a[0][3], a[1][2], a[1][3]);
  a[0][1] = a[1][0], a[2][3] = a[3][2];
  a[2][0] = a[0][2], a[3][0] = a[0][3], a[2][1] = a[1][2], a[3][1] = a[1][3];
  auto step = [&](int n, int p1, int q1, int p2, int q2) {
    const double2 u = jac_angle(a[p1][p1], a[q1][q1], a[p1][q1]), w = jac_angle(a[p2][p2], a[q2][q2], a[p2][q2]);
    q[n] = u, q[n + 1] = w;
#pragma unroll
    for (int i = 0; i < 4; ++i) jac_turn(u, a[i][p1], a[i][q1]), jac_turn(w, a[i][p2], a[i][q2]);
#pragma unroll
    for (int i = 0; i < 4; ++i) jac_turn(u, a[p1][i], a[q1][i]), jac_turn(w, a[p2][i], a[q2][i]);
    if (u.y != 0.0) a[p1][q1] = a[q1][p1] = 0.0;
    if (w.y != 0.0) a[p2][q2] = a[q2][p2] = 0.0;
  };
  if (r == 0) step(4, 0, 1, 2, 3);
  step(0, 0, 2, 1, 3);
  step(2, 0, 3, 1, 2);
  A.store(I, I, a[0][0], a[1][0], a[1][0], a[1][1]);
  A.store(J, J, a[2][2], a[3][2], a[3][2], a[3][3]);
  A.store(I, J, a[0][2], a[0][3], a[1][2], a[1][3]);
}

// The 4 x 4 block of sets k1 (rows) and k2 (columns).
__device__ void jac_cross(const JacTiles &A, int k1, int k2, int r, int rounds, const double2 *q1, const double2 *q2) {
  int I1, J1, I2, J2;
  jac_set(k1, r, rounds, I1, J1);
  jac_set(k2, r, rounds, I2, J2);
  double a[4][4];
  A.load(I1, I2, a[0][0], a[0][1], a[1][0], a[1][1]);
  A.load(I1, J2, a[0][2], a[0][3], a[1][2], a[1][3]);
  A.load(J1, I2, a[2][0], a[2][1], a[3][0], a[3][1]);
  A.load(J1, J2, a[2][2], a[2][3], a[3][2], a[3][3]);
  jac_steps(r == 0, [&](int n, int p, int q) {
    const double2 u = q2[n];
#pragma unroll
    for (int i = 0; i < 4; ++i) jac_turn(u, a[i][p], a[i][q]);
  });
  jac_steps(r == 0, [&](int n, int p, int q) {
    const double2 u = q1[n];
#pragma unroll
    for (int i = 0; i < 4; ++i) jac_turn(u, a[p][i], a[q][i]);
  });
  A.store(I1, I2, a[0][0], a[0][1], a[1][0], a[1][1]);
  A.store(I1, J2, a[0][2], a[0][3], a[1][2], a[1][3]);
  A.store(J1, I2, a[2][0], a[2][1], a[3][0], a[3][1]);
  A.store(J1, J2, a[2][2], a[2][3], a[3][2], a[3][3]);
}

// Thread's 4 x 8 elements of a product of order n4 from shared memory, sums in index order: out(i, j)
// = sum_l x(i, l) y(l, j). Lanes take neighbouring rows.
template <class X, class Y, class Out>
__device__ __forceinline__ void jac_product(int n4, X x, Y y, Out out) {
  const int rows = n4 / 4, cols = (n4 + 7) / 8;
  if ((int)threadIdx.x >= rows * cols) return;
  const int i0 = threadIdx.x % rows, j0 = threadIdx.x / rows;
  double s[4][8] = {};
  int jc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) jc[j] = min(j0 + j * cols, n4 - 1);
  for (int l = 0; l < n4; ++l) {
    double xv[4], yv[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) xv[i] = x(i0 + i * rows, l);
#pragma unroll
    for (int j = 0; j < 8; ++j) yv[j] = y(l, jc[j]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) s[i][j] = __fma_rn(xv[i], yv[j], s[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j0 + j * cols < n4) out(i0 + i * rows, j0 + j * cols, s[i][j]);
}

__global__ void __launch_bounds__(kJacobiThreads) k_jacobi(const JacobiJob *__restrict__ jobs, int warm, double pad) {
  extern __shared__ double2 jsm[];
  __shared__ double2 qs[2][kJacSets][6];
  __shared__ double red[32];
  __shared__ int rk[kJacobiMax], inv[kJacobiMax];
  __shared__ int done;
  const JacobiJob jb = jobs[blockIdx.x];
  const int n = jb.n, np = jb.np;
  if (n <= 0 || n > kJacobiMax) return;
  // padded by rows of zeros to whole sets, at least two twos
  const int n4 = (n + 3) / 4 * 4, ld = n4 + 1, blocks = n4 / 2, sets = n4 / 4, rounds = blocks - 1;
  double *M = (double *)jsm, *W = M + jac_matrix(n4);
  const JacTiles A(M, blocks);
  const int tid = threadIdx.x, nt = blockDim.x, warp = tid >> 5, lane = tid & 31;
  for (int i = warp; i < n4; i += nt / 32)
    for (int k = lane; k < n4; k += 32) {
      const bool in = i < n && k < n;
      W[i * ld + k] = warm ? (in ? jb.basis[(size_t)i * np + k] : 0.0) : (i == k ? 1.0 : 0.0);
      if (warm) M[i * ld + k] = in ? jb.slot[(size_t)i * np + k] : 0.0;
    }
  __syncthreads();
  if (warm) {
    // T = F W^T by way of the slot, then W T into the slot
    auto to_slot = [&](int i, int j, double v) {
      if (i < n && j < n) jb.slot[(size_t)i * np + j] = v;
    };
    jac_product(n4, [&](int i, int l) { return M[i * ld + l]; }, [&](int l, int j) { return W[j * ld + l]; }, to_slot);
    __syncthreads();
    for (int i = warp; i < n; i += nt / 32)
      for (int k = lane; k < n; k += 32) M[i * ld + k] = jb.slot[(size_t)i * np + k];
    __syncthreads();
    jac_product(n4, [&](int i, int l) { return W[i * ld + l]; }, [&](int l, int j) { return M[l * ld + j]; }, to_slot);
    __syncthreads();
  }
  for (int I = warp; I < blocks; I += nt / 32)
    for (int J = lane; J <= I; J += 32) {  // symmetric part
      double v[2][2];
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const int i = 2 * I + a, j = 2 * J + b;
          v[a][b] = i < n && j < n ? 0.5 * (jb.slot[(size_t)i * np + j] + jb.slot[(size_t)j * np + i]) : 0.0;
        }
      A.store(I, J, v[0][0], v[0][1], v[1][0], v[1][1]);
    }
  __syncthreads();
  // squares of the elements off and on the diagonal, in thread 0
  auto norms = [&](double &off, double &dia) {
    off = dia = 0.0;
    for (int i = warp; i < n; i += nt / 32)
      for (int j = lane; j <= i; j += 32) {
        const double v = A.get(i, j);
        if (i == j) dia += v * v;
        else off += 2.0 * v * v;
      }
    off = block_sum(off, red);
    dia = block_sum(dia, red);
  };
  int k1 = 0, k2 = 0;  // this thread's pair of sets, k1 > k2 (k1 = 0: none)
  if (tid < sets * (sets - 1) / 2) {
    k1 = 1;
    while ((k1 + 1) * k1 / 2 <= tid) ++k1;
    k2 = tid - k1 * (k1 - 1) / 2;
  }
  for (int sweep = 0; sweep < kJacSweeps; ++sweep) {
    double off, dia;
    norms(off, dia);
    if (tid == 0) done = !(off > 1.0e-30 * dia);
    __syncthreads();
    if (done) break;
    if (tid < sets) jac_angles(A, tid, 0, rounds, qs[0][tid]);
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
      const double2(*q)[6] = qs[r & 1];
      if (k1 > 0) jac_cross(A, k1, k2, r, rounds, q[k1], q[k2]);
      __syncthreads();
      if (warp == 0) {
        if (lane < sets && r + 1 < rounds) jac_angles(A, lane, r + 1, rounds, qs[(r + 1) & 1][lane]);
      } else {
        for (int k = warp - 1; k < sets; k += nt / 32 - 1) {  // W <- J^T W
          int I, J;
          jac_set(k, r, rounds, I, J);
          double *w0 = W + 2 * I * ld, *w1 = w0 + ld, *w2 = W + 2 * J * ld, *w3 = w2 + ld;
          for (int j = lane; j < n; j += 32) {
            double w[4] = {w0[j], w1[j], w2[j], w3[j]};
            jac_steps(r == 0, [&](int m, int x, int y) { jac_turn(q[k][m], w[x], w[y]); });
            w0[j] = w[0], w1[j] = w[1], w2[j] = w[2], w3[j] = w[3];
          }
        }
      }
      __syncthreads();
    }
  }
  {
    // convergence and finiteness of what is handed on
    double off, dia;
    norms(off, dia);
    if (tid == 0) *jb.info = !(isfinite(off) && isfinite(dia)) ? 2 : (off > 1.0e-24 * dia ? 1 : 0);
  }
  for (int i = tid; i < n; i += nt) {  // a total order (NaN last), so the ranks are a permutation
    const double vi = A.get(i, i), v = vi == vi ? vi : INFINITY;
    int r = 0;
    for (int j = 0; j < n; ++j) {
      const double uj = A.get(j, j), u = uj == uj ? uj : INFINITY;
      r += (u < v) || (u == v && j < i);
    }
    rk[i] = r;
  }
  __syncthreads();
  for (int i = tid; i < n; i += nt) {
    inv[rk[i]] = i;
    jb.eps[rk[i]] = A.get(i, i);
  }
  for (int i = n + tid; i < np; i += nt) jb.eps[i] = pad;
  __syncthreads();
  for (int e = tid; e < np * np; e += nt) {
    const int r = e / np, k = e % np;
    const double v = (r < n && k < n) ? W[inv[r] * ld + k] : 0.0;
    jb.slot[e] = v;
    jb.basis[e] = v;
  }
}

}  // namespace

size_t jacobi_smem(int n) {
  const int n4 = (n + 3) / 4 * 4;
  return sizeof(double) * (jac_matrix(n4) + (size_t)n4 * (n4 + 1));
}

void prepare_jacobi_eigen(int max_n) {
  CUDA_OK(cudaFuncSetAttribute(k_jacobi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jacobi_smem(max_n)));
}

void launch_jacobi_eigen(cudaStream_t st, const JacobiJob *jobs, int count, int max_n, int warm, double pad) {
  if (count <= 0) return;
  k_jacobi<<<(unsigned)count, kJacobiThreads, jacobi_smem(max_n), st>>>(jobs, warm, pad);
  note_launch();
}

}  // namespace pm7
