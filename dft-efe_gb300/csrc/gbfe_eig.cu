// gbfe_eig.cu -- dense symmetric eigen-decomposition of the projected m x m
// matrices above the host's range: FP32 decomposition, refined to FP64.
//
// cuSOLVER's FP64 syevd of a 256 x 256 matrix takes 7.6 ms on GB300: its
// tridiagonal reduction is a chain of short FP64 kernels.  The FP32 one takes
// 2.1 ms.  Its eigenvectors X are brought to FP64 accuracy by the iteration of
// Ogita & Aishima ("Iterative refinement for symmetric eigenvalue decomposition",
// Japan J. Indust. Appl. Math. 35, 2018; II, 36, 2019, for clusters): with
//   S = X^T A X,  R = I - X^T X,  lambda_i = S_ii / (X^T X)_ii,
//   E_ij = R_ij / 2 + (S_ij + (lambda_i + lambda_j) R_ij / 2) / (lambda_j - lambda_i)
// X <- X + X E converges quadratically, from 1e-7 |A| / gap to below rounding in
// two or three rounds of four products that use all SMs' FP64 pipes.  Eigenvalues
// that the FP32 result does not separate (chains of neighbours closer than delta,
// see k_eig_clusters) get R_ij / 2 only, and their own small block is diagonalised
// by Jacobi rotations, one thread block per cluster.  The second term is
// antisymmetric and, outside the clusters, at most |rounding of S| / delta, so the
// result is orthogonal to rounding whatever the gaps are.  Accepted when the last
// corrections are below 1e-8 (what they leave is their square); else, and with a
// cluster above 64, the caller runs the FP64 syevd on the untouched matrix.
#include "gbfe_internal.cuh"

#include <algorithm>
#include <cmath>

using namespace gbfe;

namespace {

constexpr uint32_t TD = 16;  // output tile of a product: 256 tiles at m = 256, all SMs busy
constexpr uint32_t TK = 32;
constexpr uint32_t CLUSTER_MAX = 64;

// stat words (bits of non-negative doubles, which order as integers)
enum { ST_CORR = 0, ST_NUM = 1, ST_BIG = 2, ST_AMAX = 3 };

__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// Largest |v| of the block into *out; NaN counts as the largest of all.
__device__ __forceinline__ void block_max_bits(unsigned long long b, unsigned long long *out) {
  __shared__ unsigned long long sh[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, b, o);
    b = w > b ? w : b;
  }
  if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t k = 1; k < blockDim.x / 32; ++k) b = sh[k] > b ? sh[k] : b;
    if (b > *out) atomicMax(out, b);
  }
  __syncthreads();
}

// C(i, j) = sum_k op(P)(i, k) Q(k, j) (+ D(i, j)), n x n column-major, op(P) = P^T
// (PT) or P.  An output per thread; blockIdx.z picks the operand and
// result; sym: only tiles on and above the diagonal, mirrored (S and X^T X come out
// exactly symmetric, which keeps the correction's second term antisymmetric).
// Bound by the FP64 pipe (n^3 multiply-adds at two lanes per SM and clock, 29 us at
// 256 x 256): 16 x 16 tiles because larger ones leave SMs idle there, one output per
// thread with the next 32 rows loaded ahead so that eight warps cover the latencies
// (35 us; 64 threads with 2 x 2 outputs 55).
struct ProdArgs {
  const double *P, *Q[2], *D;
  double *C[2];
  uint32_t n;
  int sym;
};
template <bool PT>
__global__ void __launch_bounds__(256) k_eig_product(const ProdArgs a) {
  __shared__ double Ps[TD][TK + 1], Qs[TD][TK + 1];
  const uint32_t n = a.n, nt = (n + TD - 1) / TD;
  uint32_t ti = blockIdx.x % nt, tj = blockIdx.x / nt;
  if (a.sym) {
    uint32_t t = blockIdx.x;
    tj = 0;
    while (t > tj) t -= ++tj;
    ti = t;
  }
  const double *P = a.P, *Q = a.Q[blockIdx.z];
  const uint32_t i0 = ti * TD, j0 = tj * TD;
  const uint32_t tx = threadIdx.x % TD, ty = threadIdx.x / TD;
  double acc = 0.0, pv[2], qv[2];
  auto load = [&](uint32_t k0) {
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const uint32_t t = threadIdx.x + u * 256;
      const uint32_t c = t / TK, k = t % TK;
      qv[u] = k0 + k < n && j0 + c < n ? Q[(uint64_t)(j0 + c) * n + k0 + k] : 0.0;
      if (PT) {
        pv[u] = k0 + k < n && i0 + c < n ? P[(uint64_t)(i0 + c) * n + k0 + k] : 0.0;
      } else {
        const uint32_t cc = t % TD, kk = t / TD;
        pv[u] = k0 + kk < n && i0 + cc < n ? P[(uint64_t)(k0 + kk) * n + i0 + cc] : 0.0;
      }
    }
  };
  load(0);
  for (uint32_t k0 = 0; k0 < n; k0 += TK) {
#pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
      const uint32_t t = threadIdx.x + u * 256;
      Qs[t / TK][t % TK] = qv[u];
      if (PT)
        Ps[t / TK][t % TK] = pv[u];
      else
        Ps[t % TD][t / TD] = pv[u];
    }
    __syncthreads();
    if (k0 + TK < n) load(k0 + TK);
#pragma unroll
    for (uint32_t k = 0; k < TK; ++k) acc = fma(Ps[tx][k], Qs[ty][k], acc);
    __syncthreads();
  }
  const uint32_t i = i0 + tx, j = j0 + ty;
  if (i >= n || j >= n || (a.sym && i > j)) return;
  double *C = a.C[blockIdx.z];
  const uint64_t ij = i + (uint64_t)j * n;
  const double v = a.D ? a.D[ij] + acc : acc;
  C[ij] = v;
  if (a.sym) C[j + (uint64_t)i * n] = v;
}

// the full matrix of the lower triangle, and its largest entry
__global__ void __launch_bounds__(256) k_eig_load(const double *__restrict__ A, uint32_t n, double *__restrict__ F,
                                                  unsigned long long *__restrict__ stat) {
  unsigned long long b = 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < (uint64_t)n * n;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t j = (uint32_t)(t / n), i = (uint32_t)(t % n);
    const double v = i >= j ? A[t] : A[j + (uint64_t)i * n];
    F[t] = v;
    const unsigned long long w = abs_bits(v);
    b = w > b ? w : b;
  }
  block_max_bits(b, stat + ST_AMAX);
}

// FP32 copy, scaled by a power of two to entries of at most 1 (the vectors do not
// change, and no size overflows); zeros where an entry is not finite (the caller
// sees that in ST_AMAX and takes the FP64 routine, as it did before)
__global__ void k_eig_to_f32(const double *__restrict__ F, uint32_t n, float *__restrict__ f,
                             const unsigned long long *__restrict__ stat) {
  const double amax = __longlong_as_double((long long)stat[ST_AMAX]);
  const bool ok = amax > 0.0 && amax <= 1.7976931348623157e308;
  const int ex = ok ? ilogb(amax) + 1 : 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < (uint64_t)n * n;
       t += (uint64_t)gridDim.x * blockDim.x)
    f[t] = ok ? (float)scalbn(F[t], -ex) : 0.0f;
}

__global__ void k_eig_to_f64(const float *__restrict__ f, uint32_t n, double *__restrict__ X) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < (uint64_t)n * n;
       t += (uint64_t)gridDim.x * blockDim.x)
    X[t] = (double)f[t];
}

// lambda (from S and G = X^T X; G == nullptr: lam as it is) and the ascending
// order of its entries: order[rank] = index, ties by index.  One block.
__global__ void __launch_bounds__(1024) k_eig_order(const double *__restrict__ S, const double *__restrict__ G,
                                                    uint32_t n, double *lam, uint32_t *order, double *sorted) {
  extern __shared__ double eig_lam[];
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double l = G ? S[i + (uint64_t)i * n] / G[i + (uint64_t)i * n] : lam[i];
    if (G) lam[i] = l;
    eig_lam[i] = l;
    order[i] = i;  // (a NaN shares its rank with others: no entry is left unset)
  }
  __syncthreads();
  // keys that order as the doubles do: integer compares (an FP64 one takes 64 clocks
  // of its pipe per warp: 40 us of them at 256)
  auto key = [](double v) {
    const long long b = __double_as_longlong(v + 0.0);
    return b ^ ((b >> 63) & 0x7fffffffffffffffll);
  };
  long long *keys = reinterpret_cast<long long *>(eig_lam);
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) keys[i] = key(eig_lam[i]);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double l = lam[i];
    const long long mine = keys[i];
    uint32_t r = 0;
#pragma unroll 8
    for (uint32_t j = 0; j < n; ++j) {
      const long long o = keys[j];
      r += o < mine || (o == mine && j < i);
    }
    order[r] = i;
    if (sorted) sorted[r] = l;
  }
}

// largest |S_ij + (lambda_i + lambda_j) R_ij / 2|, i != j
__global__ void __launch_bounds__(256) k_eig_num(const double *__restrict__ S, const double *__restrict__ G,
                                                 const double *__restrict__ lam, uint32_t n,
                                                 unsigned long long *__restrict__ stat) {
  unsigned long long b = 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < (uint64_t)n * n;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t j = (uint32_t)(t / n), i = (uint32_t)(t % n);
    if (i < j) {
      const unsigned long long w = abs_bits(fma(-0.5 * (lam[i] + lam[j]), G[t], S[t]));
      b = w > b ? w : b;
    }
  }
  block_max_bits(b, stat + ST_NUM);
}

// Clusters of the ordered eigenvalues: chains of neighbours at most delta apart,
// cid[i] = position of the chain's first member, size[first] = members.
// delta = max(2 sqrt(n) max|num|, 4e-7 max|A|): the first keeps every correction
// outside the clusters below 1 / (2 sqrt(n)), so that a round converges; the second
// keeps the rounding of S over the gap below 1e-8 (FP32's own resolution).
__global__ void __launch_bounds__(1024) k_eig_clusters(const double *__restrict__ lam,
                                                       const uint32_t *__restrict__ order, uint32_t n,
                                                       unsigned long long *__restrict__ stat,
                                                       uint32_t *__restrict__ cid, uint32_t *__restrict__ size) {
  const double num = __longlong_as_double((long long)stat[ST_NUM]);
  const double amax = __longlong_as_double((long long)stat[ST_AMAX]);
  const double delta = fmax(2.0 * sqrt((double)n) * num, 4e-7 * amax);
  __shared__ uint32_t big;
  if (threadIdx.x == 0) big = 0;
  __syncthreads();
  for (uint32_t r = threadIdx.x; r < n; r += blockDim.x) {
    uint32_t k = r;  // first member: walk down while the neighbour is close (a cluster too large stops the walk)
    while (k > 0 && r - k <= CLUSTER_MAX && lam[order[k]] - lam[order[k - 1]] <= delta) --k;
    uint32_t e = r + 1;
    while (e < n && e - r <= CLUSTER_MAX && lam[order[e]] - lam[order[e - 1]] <= delta) ++e;
    cid[order[r]] = k;
    if (r == k) size[r] = e - r;
    else size[r] = 0;
    if (e - k > CLUSTER_MAX) big = 1;
  }
  __syncthreads();
  if (threadIdx.x == 0 && big) stat[ST_BIG] = 1;
}

// the corrections E; the largest into stat
__global__ void __launch_bounds__(256) k_eig_correct(const double *__restrict__ S, const double *__restrict__ G,
                                                     const double *__restrict__ lam,
                                                     const uint32_t *__restrict__ cid, uint32_t n,
                                                     double *__restrict__ E, unsigned long long *__restrict__ stat) {
  unsigned long long b = 0;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < (uint64_t)n * n;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t j = (uint32_t)(t / n), i = (uint32_t)(t % n);
    const double r = (i == j ? 1.0 : 0.0) - G[t];
    double e = 0.5 * r;
    if (cid[i] != cid[j]) e += fma(0.5 * (lam[i] + lam[j]), r, S[t]) / (lam[j] - lam[i]);
    E[t] = e;
    const unsigned long long w = abs_bits(e);
    b = w > b ? w : b;
  }
  block_max_bits(b, stat + ST_CORR);
}

// One block per cluster (blocks of other positions leave at once): eigenvectors U
// of its block of S + (lambda_i + lambda_j) R / 2 by cyclic Jacobi (round-robin
// pairs, eight threads each), then X's columns times U and the eigenvalues.
constexpr uint32_t JL = CLUSTER_MAX + 1;
constexpr size_t JAC_SMEM = 2 * CLUSTER_MAX * JL * sizeof(double);
__global__ void __launch_bounds__(256) k_eig_rotate(const double *__restrict__ S, const double *__restrict__ G,
                                                    double *__restrict__ lam, const uint32_t *__restrict__ order,
                                                    const uint32_t *__restrict__ size, uint32_t n,
                                                    const unsigned long long *__restrict__ stat,
                                                    double *__restrict__ X) {
  extern __shared__ double jac_smem[];
  double *M = jac_smem, *U = M + CLUSTER_MAX * JL;
  __shared__ double cs[CLUSTER_MAX / 2][2];
  __shared__ uint32_t col[CLUSTER_MAX];
  __shared__ int rotated;
  const uint32_t k = size[blockIdx.x];
  if (k < 2 || k > CLUSTER_MAX || stat[ST_BIG] != 0) return;
  const double floor_v = 1.1102230246251565e-16 * __longlong_as_double((long long)stat[ST_AMAX]);
  for (uint32_t t = threadIdx.x; t < k; t += 256) col[t] = order[blockIdx.x + t];
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < k * k; t += 256) {
    const uint32_t i = t % k, j = t / k, a = col[i], b = col[j];
    const uint64_t ab = a + (uint64_t)b * n;
    M[i * JL + j] = i == j ? lam[a] : fma(-0.5 * (lam[a] + lam[b]), G[ab], S[ab]);
    U[i * JL + j] = i == j ? 1.0 : 0.0;
  }
  const uint32_t kk = k + (k & 1), half = kk / 2;  // an odd cluster sits one out in each round
  const uint32_t pr = threadIdx.x / 8, lane = threadIdx.x % 8;
  for (int sweep = 0; sweep < 16; ++sweep) {
    __syncthreads();
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (uint32_t rd = 0; rd + 1 < kk; ++rd) {
      uint32_t p = 0, q = 0;
      bool on = pr < half;
      if (on) {
        // circle method: member kk-1 stays, the others turn
        p = pr == 0 ? kk - 1 : (rd + pr) % (kk - 1);
        q = (rd + kk - 1 - pr) % (kk - 1);
        on = p < k && q < k;
      }
      if (on && lane == 0) {
        const double v = M[p * JL + q];
        double c = 1.0, s = 0.0;
        if (fabs(v) > floor_v) {
          const double th = (M[q * JL + q] - M[p * JL + p]) / (2.0 * v);
          const double t = copysign(1.0, th) / (fabs(th) + sqrt(fma(th, th, 1.0)));
          c = 1.0 / sqrt(fma(t, t, 1.0));
          s = t * c;
          rotated = 1;
        }
        cs[pr][0] = c;
        cs[pr][1] = s;
      }
      __syncthreads();
      const double c = on ? cs[pr][0] : 1.0, s = on ? cs[pr][1] : 0.0;
      const bool turn = on && s != 0.0;
      if (turn)
        for (uint32_t i = lane; i < k; i += 8) {
          const double mp = M[i * JL + p], mq = M[i * JL + q];
          M[i * JL + p] = c * mp - s * mq;
          M[i * JL + q] = s * mp + c * mq;
          const double up = U[i * JL + p], uq = U[i * JL + q];
          U[i * JL + p] = c * up - s * uq;
          U[i * JL + q] = s * up + c * uq;
        }
      __syncthreads();
      if (turn)
        for (uint32_t i = lane; i < k; i += 8) {
          const double mp = M[p * JL + i], mq = M[q * JL + i];
          M[p * JL + i] = c * mp - s * mq;
          M[q * JL + i] = s * mp + c * mq;
        }
      __syncthreads();
    }
    if (!rotated) break;  // (read after the round's last barrier, written again after two more)
  }
  __syncthreads();
  for (uint32_t t = threadIdx.x; t < k; t += 256) lam[col[t]] = M[t * JL + t];
  __syncthreads();
  // U <- U + U (I - U^T U) / 2: the rotations' roundings add up to several 1e-15 in a
  // cluster of 40, this takes them out of U's orthogonality again
  for (uint32_t t = threadIdx.x; t < k * k; t += 256) {
    const uint32_t i = t % k, j = t / k;
    double v = 0.0;
    for (uint32_t l = 0; l < k; ++l) v = fma(U[l * JL + i], U[l * JL + j], v);
    M[i * JL + j] = 0.5 * ((i == j ? 1.0 : 0.0) - v);
  }
  __syncthreads();
  double un[CLUSTER_MAX * CLUSTER_MAX / 256];
#pragma unroll
  for (int u = 0; u < (int)(CLUSTER_MAX * CLUSTER_MAX / 256); ++u) {
    const uint32_t t = threadIdx.x + u * 256, i = t % k, j = t / k;
    un[u] = 0.0;
    if (t < k * k) {
      for (uint32_t l = 0; l < k; ++l) un[u] = fma(U[i * JL + l], M[l * JL + j], un[u]);
      un[u] += U[i * JL + j];
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < (int)(CLUSTER_MAX * CLUSTER_MAX / 256); ++u) {
    const uint32_t t = threadIdx.x + u * 256;
    if (t < k * k) U[t % k * JL + t / k] = un[u];
  }
  __syncthreads();
  // X(:, col) U, 64 rows at a time through M's space
  for (uint32_t r0 = 0; r0 < n; r0 += CLUSTER_MAX) {
    const uint32_t rows = min(CLUSTER_MAX, n - r0);
    for (uint32_t t = threadIdx.x; t < rows * k; t += 256) {
      const uint32_t i = t % rows, j = t / rows;
      M[i * JL + j] = X[(uint64_t)col[j] * n + r0 + i];
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < rows * k; t += 256) {
      const uint32_t i = t % rows, j = t / rows;
      double v = 0.0;
      for (uint32_t l = 0; l < k; ++l) v = fma(M[i * JL + l], U[l * JL + j], v);
      X[(uint64_t)col[j] * n + r0 + i] = v;
    }
    __syncthreads();
  }
}

// columns of X in ascending order of their eigenvalues
__global__ void k_eig_columns(const double *__restrict__ X, uint32_t n, const uint32_t *__restrict__ order,
                              double *__restrict__ out) {
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < (uint64_t)n * n;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t j = (uint32_t)(t / n), i = (uint32_t)(t % n);
    out[t] = X[i + (uint64_t)order[j] * n];
  }
}

}  // namespace

namespace gbfe {

// Eigenvectors (columns, into dA) and ascending eigenvalues of the symmetric n x n
// device matrix dA (lower triangle read).  Returns false, dA untouched, where the
// refinement does not reach FP64 accuracy.
bool refined_sym_eig(gbfe_ctx *ctx, int n_, double *dA, double *eig_h) {
  const uint32_t n = (uint32_t)n_;
  const size_t nn = (size_t)n * n;
  cudaStream_t st = ctx->stream;
  ctx->eig_ws.ensure(eig_ws_size(n));
  ctx->eig_f32.ensure(nn + n);
  ctx->eig_idx.ensure(3 * (size_t)n);
  double *A = ctx->eig_ws.p, *AX = A + nn, *S = AX + nn, *G = S + nn, *E = G + nn, *X = E + nn, *Xn = X + nn,
         *lam = Xn + nn, *sorted = lam + n;
  unsigned long long *stat = reinterpret_cast<unsigned long long *>(sorted + n);
  float *f = ctx->eig_f32.p, *fw = f + nn;
  uint32_t *order = ctx->eig_idx.p, *cid = order + n, *size = cid + n;
  const unsigned g = (unsigned)std::min<uint64_t>((nn + 255) / 256, (uint64_t)ctx->sm_count * 4);
  GBFE_CUDA(cudaMemsetAsync(stat, 0, 4 * sizeof(*stat), st));
  k_eig_load<<<g, 256, 0, st>>>(dA, n, A, stat);
  k_eig_to_f32<<<g, 256, 0, st>>>(A, n, f, stat);
  check_launch(ctx, "eig_load");
  int lwork = 0;
  GBFE_CUSOLVER(cusolverDnSsyevd_bufferSize(ctx->cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n_, f, n_,
                                            fw, &lwork));
  ctx->lwork.ensure((size_t)std::max(lwork, 1) / 2 + 1);  // floats in a buffer of doubles
  ctx->info.ensure(1);
  GBFE_CUSOLVER(cusolverDnSsyevd(ctx->cusolver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n_, f, n_, fw,
                                 reinterpret_cast<float *>(ctx->lwork.p), lwork, ctx->info.p));
  k_eig_to_f64<<<g, 256, 0, st>>>(f, n, X);
  check_launch(ctx, "eig_start");
  count_launch(ctx, 4);
  const uint32_t nt = (n + TD - 1) / TD;
  GBFE_CUDA(cudaFuncSetAttribute(k_eig_rotate, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)JAC_SMEM));
  for (int it = 0; it < 5; ++it) {
    GBFE_CUDA(cudaMemsetAsync(stat, 0, 3 * sizeof(*stat), st));
    k_eig_product<true><<<nt * nt, 256, 0, st>>>(ProdArgs{A, {X, nullptr}, nullptr, {AX, nullptr}, n, 0});
    k_eig_product<true><<<dim3(nt * (nt + 1) / 2, 1, 2), 256, 0, st>>>(ProdArgs{X, {AX, X}, nullptr, {S, G}, n, 1});
    k_eig_order<<<1, 1024, n * sizeof(double), st>>>(S, G, n, lam, order, nullptr);
    k_eig_num<<<g, 256, 0, st>>>(S, G, lam, n, stat);
    k_eig_clusters<<<1, 1024, 0, st>>>(lam, order, n, stat, cid, size);
    k_eig_correct<<<g, 256, 0, st>>>(S, G, lam, cid, n, E, stat);
    k_eig_product<false><<<nt * nt, 256, 0, st>>>(ProdArgs{X, {E, nullptr}, X, {Xn, nullptr}, n, 0});
    k_eig_rotate<<<n, 256, JAC_SMEM, st>>>(S, G, lam, order, size, n, stat, Xn);
    check_launch(ctx, "eig_refine");
    count_launch(ctx, 8);
    std::swap(X, Xn);
    double h[4];
    GBFE_CUDA(cudaMemcpyAsync(h, stat, sizeof(h), cudaMemcpyDeviceToHost, st));
    GBFE_CUDA(cudaStreamSynchronize(st));
    if (!(h[ST_AMAX] > 0.0) || h[ST_BIG] != 0.0 || !(h[ST_CORR] < 0.5)) return false;
    if (h[ST_CORR] > 1e-8) continue;
    k_eig_order<<<1, 1024, n * sizeof(double), st>>>(nullptr, nullptr, n, lam, order, sorted);
    k_eig_columns<<<g, 256, 0, st>>>(X, n, order, dA);
    check_launch(ctx, "eig_columns");
    count_launch(ctx, 2);
    GBFE_CUDA(cudaMemcpyAsync(eig_h, sorted, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    GBFE_CUDA(cudaStreamSynchronize(st));
    return true;
  }
  return false;
}

}  // namespace gbfe
