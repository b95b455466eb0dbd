// gm_deflation_pairs: the k smallest eigenpairs of a symmetric matrix on the
// GPU, for the deflation vectors of the f(A)b engine.
//
// The reference computes them on the host with MATLAB's eigs(K, M, k, 'sm')
// (process_nonuniform.m:38-40, 106-110): shift-invert Arnoldi, which needs a
// sparse factorisation.  On the GPU the method is Chebyshev-filtered subspace
// iteration (Y. Zhou, Y. Saad, M. L. Tiago, J. R. Chelikowsky, "Self-consistent-
// field calculations using Chebyshev-filtered subspace iteration", J. Comput.
// Phys. 219 (2006), with the scaled three-term filter of their Algorithm 4.1)
// over a block of 32 vectors, all in FP64:
//
//   X <- C_deg(A) X        Chebyshev polynomial of degree deg on the unwanted
//                          interval [a, b] (a = the block's largest Ritz value,
//                          b = Gershgorin bound of A), scaled so that the
//                          block's lowest Ritz value a0 stays O(1)
//   X <- X R^{-1}          CholQR, twice (G = X^T X = R^T R)
//   H = X^T A X, H = W diag(theta) W^T  (Rayleigh-Ritz; cyclic Jacobi in one warp)
//   X <- X W, residuals ||A x_j - theta_j x_j|| / |theta_j| for the k wanted
//
// until every wanted relative residual is below tol.  The degree is chosen
// per iteration so that the filter amplifies a0 over a by at most 1e4 (a
// bounded condition number for CholQR) and is capped by max_degree.
//
// Layout: block vectors [n][32] row-major (one row of the block is 256
// contiguous bytes): the SpMM gathers X[c][0..31] as one coalesced 256-byte row
// per stored entry, two columns per lane of half a warp, and every
// 32 x 32 product (Gram matrices, X W) is a per-row multiply with the small
// matrix in shared memory.  The matrix is CSR (int64 row pointer, int32
// column indices, FP64 values).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/gpumatfun.h"
#include "fab_common.cuh"

namespace gm {
void set_global_error(const char* msg);  // engine.cu: the text gm_last_error(NULL) returns
}  // namespace gm

namespace {

constexpr int P = 32;            // block width: one column per lane
constexpr double kCondCap = 1e4;  // largest amplification of a0 over a per filter
constexpr double kFFUntil = 1e-7; // float-float filter while the wanted residuals are above this

int eig_fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  gm::set_global_error(buf);
  return code;
}

// Y_out = c1 (A X) + c2 X + c3 Y_prev: half a warp per row, two neighbouring
// columns per lane, so that a gathered row of X is one 256-byte access of 16
// lanes and its index, value and address are formed once for two columns.
// A row has few stored entries, so the kernel waits on the dependent chain
// of memory accesses (row pointer, then column indices and values, then the
// gathered rows of X); two rows per warp put twice the chains in flight.  The
// next row's pointers are loaded while the current row is processed, and the
// epilogue's X and Y_prev rows are loaded before the gathers.  Entries are
// taken kChebU at a time, their gathers all in flight before the products.
// Against one row per warp and one column per lane, on a 60k-node disk with
// k = 20 (4,133 float-float and 869 FP64 steps of 32 columns): 214 -> 142 ms
// for the whole iteration, 65 ms of it from k_jacobi; four entries at a time
// 142, eight 139.
constexpr int kChebU = 8;

// Thousands of these kernels follow one another, each a few microseconds: they
// are launched with programmatic stream serialization, so that a kernel's
// blocks start while the last one drains, read their row pointers (the matrix
// does not change) and wait here for the vectors.
__device__ __forceinline__ void dependents_may_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__global__ void k_cheb(long long n, const long long* __restrict__ rp, const int* __restrict__ ci,
                       const double* __restrict__ va, const double* X, const double* Yp, double* Yo, double c1,
                       double c2, double c3) {
  const int hl = threadIdx.x & 15;
  const double2* X2 = reinterpret_cast<const double2*>(X) + hl;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 4;
  long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  dependents_may_launch();
  long long b = r < n ? rp[r] : 0, e = r < n ? rp[r + 1] : 0;
  wait_for_previous();
  for (; r < n; r += nw) {
    const long long rn = r + nw;
    const long long bn = rn < n ? rp[rn] : 0, en = rn < n ? rp[rn + 1] : 0;
    const double2 z = make_double2(0.0, 0.0);
    const double2 xo = c2 != 0.0 ? X2[r * (P / 2)] : z;
    const double2 yo = c3 != 0.0 ? reinterpret_cast<const double2*>(Yp)[r * (P / 2) + hl] : z;
    double2 acc = z;
    const int* cp = ci + b;
    const double* vp = va + b;
    for (int t = (int)(e - b); t > 0; t -= kChebU, cp += kChebU, vp += kChebU) {
      double av[kChebU];
      double2 xv[kChebU];
#pragma unroll
      for (int q = 0; q < kChebU; ++q) {
        av[q] = 0.0;
        xv[q] = z;
        if (q < t) {
          av[q] = __ldg(vp + q);
          xv[q] = X2[(long long)__ldg(cp + q) * (P / 2)];
        }
      }
#pragma unroll
      for (int q = 0; q < kChebU; ++q) {
        acc.x = fma(av[q], xv[q].x, acc.x);
        acc.y = fma(av[q], xv[q].y, acc.y);
      }
    }
    reinterpret_cast<double2*>(Yo)[r * (P / 2) + hl] =
        make_double2(fma(c3, yo.x, fma(c2, xo.x, c1 * acc.x)), fma(c3, yo.y, fma(c2, xo.y, c1 * acc.y)));
    b = bn;
    e = en;
  }
}

// The same three-term step in float-float arithmetic on the FP32 pipe
// (about 48 significant bits): values split as hi + lo floats, block vectors
// as (hi, lo) pairs.  Each product is hi*hi exactly (two_prod) plus the two
// cross terms; the row sum keeps its hi part by two_sum and collects every
// rounding error in lo, renormalised once per row.  About 12 FP32
// instructions per product instead of one FP64 FMA on GB300's narrow FP64
// pipe.  Memory access order as in k_cheb.
__device__ __forceinline__ void cheb_ff_acc(float& hi, float& lo, float2 a, float xh, float xl) {
  const gm::ff p = gm::two_prod(a.x, xh);
  const float cross = fmaf(a.x, xl, a.y * xh);
  const gm::ff s2 = gm::two_sum(hi, p.hi);
  hi = s2.hi;
  lo += s2.lo + (p.lo + cross);
}
__device__ __forceinline__ gm::ff cheb_ff_out(float hi, float lo, float xh, float xl, float yh, float yl, float2 c1,
                                              float2 c2, float2 c3) {
  using gm::ff;
  ff y = gm::ff_mul(gm::fast_two_sum(hi, lo), ff{c1.x, c1.y});
  if (c2.x != 0.f) y = gm::ff_add(y, gm::ff_mul(ff{xh, xl}, ff{c2.x, c2.y}));
  if (c3.x != 0.f) y = gm::ff_add(y, gm::ff_mul(ff{yh, yl}, ff{c3.x, c3.y}));
  return y;
}
__global__ void k_cheb_ff(long long n, const long long* __restrict__ rp, const int* __restrict__ ci,
                          const float* __restrict__ vhi, const float* __restrict__ vlo, const float2* X,
                          const float2* Yp, float2* Yo, float2 c1, float2 c2, float2 c3) {
  const int hl = threadIdx.x & 15;
  const float4* X4 = reinterpret_cast<const float4*>(X) + hl;   // (hi, lo) of two columns
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 4;
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
  long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  dependents_may_launch();
  long long b = r < n ? rp[r] : 0, e = r < n ? rp[r + 1] : 0;
  wait_for_previous();
  for (; r < n; r += nw) {
    const long long rn = r + nw;
    const long long bn = rn < n ? rp[rn] : 0, en = rn < n ? rp[rn + 1] : 0;
    const float4 xo = c2.x != 0.f ? X4[r * (P / 2)] : z;
    const float4 yo = c3.x != 0.f ? reinterpret_cast<const float4*>(Yp)[r * (P / 2) + hl] : z;
    float h0 = 0.f, l0 = 0.f, h1 = 0.f, l1 = 0.f;
    const int* cp = ci + b;
    const float* hp = vhi + b;
    const float* lp = vlo + b;
    for (int t = (int)(e - b); t > 0; t -= kChebU, cp += kChebU, hp += kChebU, lp += kChebU) {
      float2 av[kChebU];
      float4 xv[kChebU];
#pragma unroll
      for (int q = 0; q < kChebU; ++q) {
        av[q] = make_float2(0.f, 0.f);
        xv[q] = z;
        if (q < t) {
          av[q] = make_float2(__ldg(hp + q), __ldg(lp + q));
          xv[q] = X4[(long long)__ldg(cp + q) * (P / 2)];
        }
      }
#pragma unroll
      for (int q = 0; q < kChebU; ++q) {
        cheb_ff_acc(h0, l0, av[q], xv[q].x, xv[q].y);
        cheb_ff_acc(h1, l1, av[q], xv[q].z, xv[q].w);
      }
    }
    const gm::ff a = cheb_ff_out(h0, l0, xo.x, xo.y, yo.x, yo.y, c1, c2, c3);
    const gm::ff c = cheb_ff_out(h1, l1, xo.z, xo.w, yo.z, yo.w, c1, c2, c3);
    reinterpret_cast<float4*>(Yo)[r * (P / 2) + hl] = make_float4(a.hi, a.lo, c.hi, c.lo);
    b = bn;
    e = en;
  }
}

// FP64 block <-> float-float block (hi = fl32(x), lo = fl32(x - hi))
__global__ void k_d2ff(long long count, const double* __restrict__ x, float2* __restrict__ y) {
  const long long nt = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += nt) {
    const float h = (float)x[t];
    y[t] = make_float2(h, (float)(x[t] - (double)h));
  }
}
__global__ void k_ff2d(long long count, const float2* __restrict__ x, double* __restrict__ y) {
  const long long nt = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += nt)
    y[t] = (double)x[t].x + (double)x[t].y;
}

// partial[blk][i * 32 + j] = sum over the block's rows of Y[r][i] Z[r][j]
// (1024 threads: thread (i, j); tiles of 32 rows staged in shared memory).
__global__ void __launch_bounds__(1024) k_gram(long long n, long long rows_per_block, const double* __restrict__ Y,
                                               const double* __restrict__ Z, double* __restrict__ partial) {
  __shared__ double sy[32][P + 1];
  __shared__ double sz[32][P + 1];
  const int t = threadIdx.x, i = t >> 5, j = t & 31;
  const long long r0 = (long long)blockIdx.x * rows_per_block;
  const long long r1 = r0 + rows_per_block < n ? r0 + rows_per_block : n;
  double acc = 0.0;
  for (long long rt = r0; rt < r1; rt += 32) {
    const long long r = rt + i;
    sy[i][j] = r < r1 ? Y[r * P + j] : 0.0;
    sz[i][j] = r < r1 ? Z[r * P + j] : 0.0;
    __syncthreads();
#pragma unroll 8
    for (int q = 0; q < 32; ++q) acc = fma(sy[q][i], sz[q][j], acc);
    __syncthreads();
  }
  partial[(long long)blockIdx.x * (P * P) + t] = acc;
}

// out[t] = sum over the G blocks of partial[b][t], in block order
// (deterministic); 16 loads ahead of the additions, a serial chain of 64 cycles
// each (32 -> 10 us for 304 blocks).
__global__ void k_gram_sum(const double* __restrict__ partial, int G, double* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P * P) return;
  double s = 0.0;
  int b = 0;
  for (; b + 16 <= G; b += 16) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = partial[(long long)(b + u) * (P * P) + t];
#pragma unroll
    for (int u = 0; u < 16; ++u) s += v[u];
  }
  for (; b < G; ++b) s += partial[(long long)b * (P * P) + t];
  out[t] = s;
}

// Out[r][j] = sum_i Y[r][i] M[i][j] (M 32 x 32 row-major; Out may not alias Y).
__global__ void k_rowmul(long long n, const double* __restrict__ Y, const double* __restrict__ M,
                         double* __restrict__ Out) {
  __shared__ double sm[P * P];
  for (int t = threadIdx.x; t < P * P; t += blockDim.x) sm[t] = M[t];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long r = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
    const double y = Y[r * P + lane];
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < P; ++i) acc = fma(__shfl_sync(0xffffffffu, y, i), sm[i * P + lane], acc);
    Out[r * P + lane] = acc;
  }
}

// R[r][j] = AX[r][j] - theta[j] X[r][j]
__global__ void k_resid(long long n, const double* __restrict__ AX, const double* __restrict__ X,
                        const double* __restrict__ theta, double* __restrict__ Rr) {
  const long long nt = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n * P; t += nt)
    Rr[t] = AX[t] - theta[t & (P - 1)] * X[t];
}

// Seeded start block: splitmix64 of (seed, index) mapped to [-1, 1).
__global__ void k_random(long long n, unsigned long long seed, double* __restrict__ X) {
  const long long nt = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n * P; t += nt) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(t + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    X[t] = (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
  }
}

// Q[j][r] (column-major n x k) = X[r][j]
__global__ void k_take_cols(long long n, int k, const double* __restrict__ X, double* __restrict__ Q) {
  const long long nt = (long long)gridDim.x * blockDim.x;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n * k; t += nt) {
    const long long j = t / n, r = t - j * n;
    Q[t] = X[r * P + j];
  }
}

// One warp: G = L L^T (Cholesky, L lower), then M = L^{-T} (so that X M has
// orthonormal columns).  status[0] = 1 when G is not numerically positive
// definite (a pivot at or below 1e-14 of the largest diagonal entry).
__global__ void k_chol_inv(const double* __restrict__ Gin, double* __restrict__ M, int* __restrict__ status) {
  __shared__ double L[P][P + 1];
  __shared__ double Li[P][P + 1];
  __shared__ int bad;
  const int lane = threadIdx.x;
  for (int i = 0; i < P; ++i) L[i][lane] = Gin[i * P + lane];
  if (lane == 0) bad = 0;
  __syncwarp();
  double dmax = 0.0;
  for (int i = 0; i < P; ++i) dmax = fmax(dmax, L[i][i]);
  for (int k = 0; k < P; ++k) {
    if (lane == 0) {
      const double d = L[k][k];
      if (!(d > 1e-14 * dmax)) bad = 1;
      L[k][k] = sqrt(fmax(d, 1e-300));
    }
    __syncwarp();
    if (lane > k) L[lane][k] /= L[k][k];
    __syncwarp();
    for (int j = k + 1; j < P; ++j)
      if (lane >= j) L[lane][j] -= L[lane][k] * L[j][k];
    __syncwarp();
  }
  // column `lane` of L^{-1} by forward substitution
  for (int i = 0; i < P; ++i) {
    double s = i == lane ? 1.0 : 0.0;
    for (int t = 0; t < i; ++t) s -= L[i][t] * Li[t][lane];
    Li[i][lane] = i >= lane ? s / L[i][i] : 0.0;
    __syncwarp();
  }
  // M[i][j] = (L^{-1})[j][i]
  for (int i = 0; i < P; ++i) M[i * P + lane] = Li[lane][i];
  if (lane == 0) status[0] = bad;
}

// Eigendecomposition of the symmetric 32 x 32 H by cyclic Jacobi rotations
// (G. H. Golub, C. F. Van Loan, Matrix Computations, 4th ed., Algorithms 8.5.2
// and 8.5.3), FP64.  theta ascending, W[i][j] = component i of eigenvector j.
// The rotations of a sweep in cyclic order by rows, (0, 1), (0, 2), ..,
// (30, 31), depend on each other only through a shared index, and the pairs
// with p + q = t share none while every earlier rotation that touches p or q
// has a smaller sum: a sweep is 61 steps of up to 16 rotations, the same
// rotations up to rounding.  One block; warp i and lane j hold H(i, j) and
// V(j, i), and every update is by rows through shared memory: H <- J^T H,
// then J^T of its transpose, and the columns of V as rows.  A warp whose index
// has no partner in the step skips its arithmetic (half of them on average).
// What bounds it is FP64 issue: about 1,500 cycles for a step's angles and
// 1,850 for its updates, where V's run while warp 0 forms the next angles.
// (One warp, one rotation at a time: 6.6 ms a call.)
__global__ void __launch_bounds__(1024) k_jacobi(const double* __restrict__ Hin, double* __restrict__ theta,
                                                 double* __restrict__ W) {
  __shared__ double H[P][P + 1];
  __shared__ double T[P][P + 1];
  __shared__ double Vs[P][P + 1];
  __shared__ double cc[2][P], ss[2][P];   // by step parity: x_i <- cc x_i + ss x_partner
  __shared__ double red[2][P];
  const int lane = threadIdx.x & 31, i = threadIdx.x >> 5;
  const unsigned full = 0xffffffffu;
  auto partner = [](int t, int k) { return t - k >= 0 && t - k < P ? t - k : k; };
  double h = 0.5 * (Hin[i * P + lane] + Hin[lane * P + i]);
  double v = i == lane ? 1.0 : 0.0;
  H[i][lane] = h;
  Vs[i][lane] = v;
  __syncthreads();
  for (int sweep = 0; sweep < 30; ++sweep) {
    const double h2 = h * h;
    const double off = gm::warp_sum(i == lane ? 0.0 : h2), tot = gm::warp_sum(h2);
    if (lane == 0) {
      red[0][i] = off;
      red[1][i] = tot;
    }
    __syncthreads();
    if (gm::warp_sum(red[0][lane]) <= 1e-30 * gm::warp_sum(red[1][lane])) break;   // the same in every warp
    const int last = 2 * P - 3;
    for (int t = 1; t <= last + 1; ++t) {
      const int cur = t & 1, old = cur ^ 1;
      // angles of step t by warp 0; V of step t - 1 by the others, then by warp 0
      if (i == 0 && t <= last) {
        const int pj = partner(t, lane);
        double c = 1.0, s = 0.0;
        if (pj > lane) {
          const double apq = H[lane][pj];
          if (apq != 0.0) {
            const double tau = (H[pj][pj] - H[lane][lane]) / (2.0 * apq);
            const double r = sqrt(1.0 + tau * tau);
            const double tn = tau >= 0.0 ? 1.0 / (tau + r) : -1.0 / (-tau + r);
            c = rsqrt(1.0 + tn * tn);
            s = tn * c;
          }
        }
        const double co = __shfl_sync(full, c, pj), so = __shfl_sync(full, s, pj);
        cc[cur][lane] = pj < lane ? co : c;
        ss[cur][lane] = pj < lane ? so : -s;
      }
      const int qi = partner(t - 1, i);
      if (t > 1 && qi != i) v = cc[old][i] * v + ss[old][i] * Vs[qi][lane];
      __syncthreads();
      if (t > 1 && qi != i) Vs[i][lane] = v;
      if (t > last) break;
      const int pi = partner(t, i);
      const double ci = cc[cur][i], si = ss[cur][i];
      if (pi != i) h = ci * h + si * H[pi][lane];
      T[i][lane] = h;
      __syncthreads();
      h = T[lane][i];
      if (pi != i) {
        h = ci * h + si * T[lane][pi];
        if (lane == pi && si != 0.0) h = 0.0;
      }
      H[i][lane] = h;
      __syncthreads();
    }
  }
  // ascending order: rank of each diagonal entry, by the bits as integers, an
  // order that NaN is part of (the ranks are a permutation whatever H holds)
  __syncthreads();
  auto key = [](double x) {
    const long long b = __double_as_longlong(x == 0.0 ? 0.0 : x);
    return b < 0 ? b ^ 0x7fffffffffffffffll : b;
  };
  const double mine = H[lane][lane];
  const long long km = key(mine);
  int rank = 0;
  for (int j = 0; j < P; ++j) {
    const long long kj = key(H[j][j]);
    rank += kj < km || (kj == km && j < lane);
  }
  if (i == 0) theta[rank] = mine;
  rank = __shfl_sync(full, rank, i);
  W[lane * P + rank] = v;
}

struct Solver {
  long long n = 0, nnz = 0;
  int nsm = 0, G = 0;
  long long rows_per_block = 0;
  long long* rp = nullptr;
  int* ci = nullptr;
  double* va = nullptr;
  float* vhi = nullptr;     // float-float split of the values (float-float filter)
  float* vlo = nullptr;
  unsigned grid64 = 0, grid_ff = 0;   // resident 256-thread blocks of k_cheb / k_cheb_ff
  double* buf[6] = {};      // block vectors [n][32]
  double* part = nullptr;   // Gram partials [G][1024]
  double* small = nullptr;  // [0] G/H 1024, [1024] M/W 1024, [2048] theta 32
  int* status = nullptr;
  long long spmm = 0, spmm_ff = 0;
  std::string err;

  ~Solver() {
    cudaFree(rp);
    cudaFree(ci);
    cudaFree(va);
    cudaFree(vhi);
    cudaFree(vlo);
    for (double* b : buf) cudaFree(b);
    cudaFree(part);
    cudaFree(small);
    cudaFree(status);
  }

  unsigned grid_rows() const { return (unsigned)std::max(1, nsm * 8); }   // 256-thread blocks, a warp per row

  // 256-thread blocks, overlapping the tail of the kernel before (see k_cheb)
  template <class... Args>
  static cudaError_t launch_overlapped(void (*kernel)(Args...), unsigned grid, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
  }

  cudaError_t spmm_axpby(const double* X, const double* Yp, double* Yo, double c1, double c2, double c3) {
    ++spmm;
    return launch_overlapped(k_cheb, grid64, n, (const long long*)rp, (const int*)ci, (const double*)va, X, Yp, Yo, c1,
                             c2, c3);
  }

  static float2 to_ff(double v) {
    const float h = (float)v;
    return make_float2(h, (float)(v - (double)h));
  }

  cudaError_t spmm_axpby_ff(const float2* X, const float2* Yp, float2* Yo, double c1, double c2, double c3) {
    ++spmm;
    ++spmm_ff;
    return launch_overlapped(k_cheb_ff, grid_ff, n, (const long long*)rp, (const int*)ci, (const float*)vhi,
                             (const float*)vlo, X, Yp, Yo, to_ff(c1), to_ff(c2), to_ff(c3));
  }

  // small[0..1024) = Y^T Z
  cudaError_t gram(const double* Y, const double* Z) {
    k_gram<<<G, 1024>>>(n, rows_per_block, Y, Z, part);
    k_gram_sum<<<P, P>>>(part, G, small);
    return cudaGetLastError();
  }

  // X <- X R^{-1} twice (CholQR2) through tmp; returns 1 when G was not
  // positive definite, negative on a CUDA error
  int cholqr2(double* X, double* tmp) {
    for (int pass = 0; pass < 2; ++pass) {
      if (gram(X, X) != cudaSuccess) return -1;
      k_chol_inv<<<1, 32>>>(small, small + P * P, status);
      int bad = 0;
      if (cudaMemcpy(&bad, status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
      if (bad) return 1;
      k_rowmul<<<grid_rows(), 256>>>(n, X, small + P * P, tmp);
      if (cudaMemcpy(X, tmp, (size_t)n * P * sizeof(double), cudaMemcpyDeviceToDevice) != cudaSuccess) return -1;
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
  }
};

}  // namespace

extern "C" int gm_deflation_pairs(int64_t n, const int64_t* rowptr, const int32_t* col, const double* val, int k,
                                  double tol, int max_degree, int max_iter, uint64_t seed, double* lambda, double* Q,
                                  double* stats) {
  // a negative max_degree selects the FP64 filter throughout (|max_degree| is the cap)
  const bool use_ff_arg = max_degree >= 0;
  max_degree = max_degree < 0 ? -max_degree : max_degree;
  gm::set_global_error("");
  if (n < 2 * P) return eig_fail(GM_ERR_ARG, "deflation_pairs: n must be at least %d", 2 * P);
  if (k < 1 || k > P - 8) return eig_fail(GM_ERR_ARG, "deflation_pairs: k must be in [1, %d]", P - 8);
  if (!rowptr || !col || !val || !lambda || !Q) return eig_fail(GM_ERR_ARG, "deflation_pairs: null pointer");
  if (!(tol > 0.0) || max_degree < 4 || max_iter < 1)
    return eig_fail(GM_ERR_ARG, "deflation_pairs: need tol > 0, max_degree >= 4, max_iter >= 1");
  // Host copy of the row pointer (host or device memory): nnz and the
  // Gershgorin bound need it.
  std::vector<int64_t> hrp(n + 1);
  cudaError_t st = cudaMemcpy(hrp.data(), rowptr, sizeof(int64_t) * (n + 1), cudaMemcpyDefault);
  if (st != cudaSuccess) return eig_fail(GM_ERR_CUDA, "deflation_pairs: row pointer copy: %s", cudaGetErrorString(st));
  if (hrp[0] != 0) return eig_fail(GM_ERR_ARG, "deflation_pairs: rowptr[0] must be 0");
  for (long long i = 0; i < n; ++i)
    if (hrp[i + 1] < hrp[i]) return eig_fail(GM_ERR_ARG, "deflation_pairs: rowptr must be non-decreasing");
  const long long nnz = hrp[n];
  std::vector<int32_t> hci(nnz);
  std::vector<double> hva(nnz);
  if ((st = cudaMemcpy(hci.data(), col, sizeof(int32_t) * nnz, cudaMemcpyDefault)) != cudaSuccess ||
      (st = cudaMemcpy(hva.data(), val, sizeof(double) * nnz, cudaMemcpyDefault)) != cudaSuccess)
    return eig_fail(GM_ERR_CUDA, "deflation_pairs: matrix copy: %s", cudaGetErrorString(st));
  double b = 0.0, vmin = HUGE_VAL;
  for (long long i = 0; i < n; ++i) {
    double s = 0.0;
    for (long long t = hrp[i]; t < hrp[i + 1]; ++t) {
      if (hci[t] < 0 || hci[t] >= n) return eig_fail(GM_ERR_ARG, "deflation_pairs: column index out of range");
      if (!std::isfinite(hva[t])) return eig_fail(GM_ERR_ARG, "deflation_pairs: non-finite matrix value");
      s += std::fabs(hva[t]);
      if (hva[t] != 0.0) vmin = std::min(vmin, std::fabs(hva[t]));
    }
    b = std::max(b, s);
  }
  if (!(b > 0.0)) return eig_fail(GM_ERR_ARG, "deflation_pairs: zero matrix");

  Solver S;
  S.n = n;
  S.nnz = nnz;
  int dev = 0;
  if ((st = cudaGetDevice(&dev)) != cudaSuccess ||
      (st = cudaDeviceGetAttribute(&S.nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
    return eig_fail(GM_ERR_CUDA, "deflation_pairs: %s", cudaGetErrorString(st));
  S.G = std::max(1, std::min<int>(2 * S.nsm, (int)((n + 31) / 32)));
  S.rows_per_block = (n + S.G - 1) / S.G;
  auto alloc = [&](void** p, size_t bytes) { return cudaMalloc(p, std::max<size_t>(bytes, 8)); };
  const size_t vbytes = (size_t)n * P * sizeof(double);
  bool ok = alloc((void**)&S.rp, sizeof(long long) * (n + 1)) == cudaSuccess &&
            alloc((void**)&S.ci, sizeof(int) * nnz) == cudaSuccess &&
            alloc((void**)&S.va, sizeof(double) * nnz) == cudaSuccess &&
            alloc((void**)&S.part, sizeof(double) * (size_t)S.G * P * P) == cudaSuccess &&
            alloc((void**)&S.small, sizeof(double) * (2 * P * P + P)) == cudaSuccess &&
            alloc((void**)&S.status, sizeof(int)) == cudaSuccess;
  for (int i = 0; i < 6 && ok; ++i) ok = alloc((void**)&S.buf[i], vbytes) == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    return eig_fail(GM_ERR_OOM, "deflation_pairs: device allocation of %.1f GB failed", (6.0 * vbytes + 12.0 * nnz) / 1e9);
  }
  {
    std::vector<float> hi(nnz), lo(nnz);
    for (long long t = 0; t < nnz; ++t) {
      hi[t] = (float)hva[t];
      lo[t] = (float)(hva[t] - (double)hi[t]);
    }
    if (alloc((void**)&S.vhi, sizeof(float) * nnz) != cudaSuccess || alloc((void**)&S.vlo, sizeof(float) * nnz) != cudaSuccess) {
      cudaGetLastError();
      return eig_fail(GM_ERR_OOM, "deflation_pairs: device allocation failed");
    }
    if ((st = cudaMemcpy(S.vhi, hi.data(), sizeof(float) * nnz, cudaMemcpyHostToDevice)) != cudaSuccess ||
        (st = cudaMemcpy(S.vlo, lo.data(), sizeof(float) * nnz, cudaMemcpyHostToDevice)) != cudaSuccess)
      return eig_fail(GM_ERR_CUDA, "deflation_pairs: upload: %s", cudaGetErrorString(st));
  }
  {
    // grids of resident blocks only (grid-stride loops over the rows)
    int nb64 = 0, nbff = 0;
    if ((st = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb64, k_cheb, 256, 0)) != cudaSuccess ||
        (st = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nbff, k_cheb_ff, 256, 0)) != cudaSuccess)
      return eig_fail(GM_ERR_CUDA, "deflation_pairs: occupancy: %s", cudaGetErrorString(st));
    S.grid64 = (unsigned)std::max(1, nb64 * S.nsm);
    S.grid_ff = (unsigned)std::max(1, nbff * S.nsm);
  }
  if ((st = cudaMemcpy(S.rp, hrp.data(), sizeof(long long) * (n + 1), cudaMemcpyHostToDevice)) != cudaSuccess ||
      (st = cudaMemcpy(S.ci, hci.data(), sizeof(int) * nnz, cudaMemcpyHostToDevice)) != cudaSuccess ||
      (st = cudaMemcpy(S.va, hva.data(), sizeof(double) * nnz, cudaMemcpyHostToDevice)) != cudaSuccess)
    return eig_fail(GM_ERR_CUDA, "deflation_pairs: upload: %s", cudaGetErrorString(st));

  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  cudaEventRecord(t0);
  double* X = S.buf[0];   // current block (orthonormal after each iteration)
  double* AX = S.buf[1];
  double* Y = S.buf[2];   // filter ping-pong
  double* Yp = S.buf[3];
  double* Yn = S.buf[4];
  double* T = S.buf[5];   // scratch
  const unsigned ge = (unsigned)std::max(1, S.nsm * 8);
  // float-float filter only where the values and the filter's intermediates
  // stay well inside FP32's exponent range
  bool use_ff = use_ff_arg && b < 1e30 && vmin > 1e-30;
  double theta[P] = {};
  double res[P] = {};
  int iters = 0, rc = GM_OK;
  double a = 0.0, maxres = 0.0;

  // Rayleigh-Ritz of the orthonormal block Y: X = Y W, AX = (A Y) W, theta,
  // and the wanted relative residuals
  auto rayleigh_ritz = [&](double* Yb) -> int {
    if (S.spmm_axpby(Yb, nullptr, T, 1.0, 0.0, 0.0) != cudaSuccess) return -1;
    if (S.gram(Yb, T) != cudaSuccess) return -1;
    k_jacobi<<<1, 1024>>>(S.small, S.small + 2 * P * P, S.small + P * P);
    k_rowmul<<<S.grid_rows(), 256>>>(n, Yb, S.small + P * P, X);
    k_rowmul<<<S.grid_rows(), 256>>>(n, T, S.small + P * P, AX);
    k_resid<<<ge, 256>>>(n, AX, X, S.small + 2 * P * P, T);
    if (cudaMemcpy(theta, S.small + 2 * P * P, sizeof(theta), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (S.gram(T, T) != cudaSuccess) return -1;
    std::vector<double> g(P * P);
    if (cudaMemcpy(g.data(), S.small, sizeof(double) * P * P, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    maxres = 0.0;
    for (int j = 0; j < P; ++j) {
      res[j] = std::sqrt(std::max(g[j * P + j], 0.0)) / std::max(std::fabs(theta[j]), 1e-300);
      if (j < k) maxres = std::max(maxres, res[j]);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
  };

  k_random<<<ge, 256>>>(n, seed, Y);
  int q = S.cholqr2(Y, T);
  if (q == 0) q = rayleigh_ritz(Y);
  if (q != 0) rc = q < 0 ? eig_fail(GM_ERR_CUDA, "deflation_pairs: %s", cudaGetErrorString(cudaGetLastError()))
                         : eig_fail(GM_ERR_BREAKDOWN, "deflation_pairs: the start block is rank deficient");
  for (; rc == GM_OK && iters < max_iter && !(maxres <= tol); ++iters) {
    a = theta[P - 1];
    const double a0 = theta[0];
    if (!(a < b) || !(a0 < a)) {
      rc = eig_fail(GM_ERR_BREAKDOWN, "deflation_pairs: Ritz values [%g, %g] outside the filter bound %g", a0, a, b);
      break;
    }
    const double e = 0.5 * (b - a), c = 0.5 * (b + a);
    const double rate = std::acosh((c - a0) / e);
    const int deg = (int)std::min<double>(max_degree, std::max(4.0, std::ceil(std::log(kCondCap) / rate)));
    // scaled Chebyshev filter (Zhou, Saad, Tiago, Chelikowsky, Algorithm 4.1).
    // While the wanted residuals are far above kFFUntil it runs in float-float
    // (about 48 bits, on the FP32 pipe); its rounding floors the reachable
    // residual near 1e-7 on an operator with kappa ~ 1e7, so the last
    // iterations, and every Rayleigh-Ritz step, are FP64.
    double sig = e / (a0 - c);
    const double tau = 2.0 / sig;
    const bool ff_now = use_ff && maxres > kFFUntil;
    double* Yf = nullptr;   // the filtered block, FP64
    if (ff_now) {
      float2* pf = reinterpret_cast<float2*>(S.buf[3]);
      float2* yf = reinterpret_cast<float2*>(S.buf[2]);
      float2* nf = reinterpret_cast<float2*>(S.buf[4]);
      k_d2ff<<<ge, 256>>>(n * P, X, pf);
      if (S.spmm_axpby_ff(pf, nullptr, yf, sig / e, -c * sig / e, 0.0) != cudaSuccess) rc = GM_ERR_CUDA;
      for (int i = 2; i <= deg && rc == GM_OK; ++i) {
        const double sig2 = 1.0 / (tau - sig);
        if (S.spmm_axpby_ff(yf, pf, nf, 2.0 * sig2 / e, -2.0 * c * sig2 / e, -sig * sig2) != cudaSuccess)
          rc = GM_ERR_CUDA;
        float2* old = pf;
        pf = yf;
        yf = nf;
        nf = old;
        sig = sig2;
      }
      Yf = yf == reinterpret_cast<float2*>(S.buf[2]) ? S.buf[3] : S.buf[2];
      k_ff2d<<<ge, 256>>>(n * P, yf, Yf);
    } else {
      if (S.spmm_axpby(X, nullptr, Y, sig / e, -c * sig / e, 0.0) != cudaSuccess) rc = GM_ERR_CUDA;
      double* prev = X;
      for (int i = 2; i <= deg && rc == GM_OK; ++i) {
        const double sig2 = 1.0 / (tau - sig);
        if (S.spmm_axpby(Y, prev, Yn, 2.0 * sig2 / e, -2.0 * c * sig2 / e, -sig * sig2) != cudaSuccess)
          rc = GM_ERR_CUDA;
        // rotate: prev <- Y, Y <- Yn (X is kept untouched after the first step)
        double* old = prev == X ? Yp : prev;
        prev = Y;
        Y = Yn;
        Yn = old;
        sig = sig2;
      }
      Yf = Y;
    }
    if (rc != GM_OK) {
      rc = eig_fail(GM_ERR_CUDA, "deflation_pairs: filter launch: %s", cudaGetErrorString(cudaGetLastError()));
      break;
    }
    const double res_before = maxres;
    q = S.cholqr2(Yf, T);
    if (q == 0) q = rayleigh_ritz(Yf);
    // a float-float iteration that no longer halves the residual has met its floor
    if (q == 0 && ff_now && maxres < 1e-3 && maxres > 0.5 * res_before) use_ff = false;
    if (q != 0) {
      rc = q < 0 ? eig_fail(GM_ERR_CUDA, "deflation_pairs: %s", cudaGetErrorString(cudaGetLastError()))
                 : eig_fail(GM_ERR_BREAKDOWN, "deflation_pairs: filtered block rank deficient (degree %d)", deg);
      break;
    }
    // buffers: X and AX hold the new block; Y, Yp, Yn are free again
    Yp = S.buf[3];
    Y = S.buf[2];
    Yn = S.buf[4];
  }
  cudaEventRecord(t1);
  cudaEventSynchronize(t1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, t0, t1);
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  if (rc == GM_OK) {
    k_take_cols<<<ge, 256>>>(n, k, X, T);
    if ((st = cudaMemcpy(Q, T, sizeof(double) * (size_t)n * k, cudaMemcpyDefault)) != cudaSuccess)
      return eig_fail(GM_ERR_CUDA, "deflation_pairs: output copy: %s", cudaGetErrorString(st));
    if ((st = cudaMemcpy(lambda, theta, sizeof(double) * k, cudaMemcpyDefault)) != cudaSuccess)
      return eig_fail(GM_ERR_CUDA, "deflation_pairs: output copy: %s", cudaGetErrorString(st));
    if (!(maxres <= tol))
      rc = eig_fail(GM_ERR_NOCONV, "deflation_pairs: %d iterations reached relative residual %.3e > tol %.3e", iters,
                    maxres, tol);
  }
  if (stats) {
    stats[0] = iters;
    stats[1] = (double)S.spmm;
    stats[2] = ms * 1e-3;
    stats[3] = maxres;
    stats[4] = b;
    stats[5] = a;
    stats[6] = theta[P - 1];
    stats[7] = (double)nnz;
    stats[8] = (double)S.spmm_ff;
  }
  return rc;
}
