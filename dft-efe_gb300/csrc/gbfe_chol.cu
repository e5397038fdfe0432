// gbfe_chol.cu -- Cholesky factor of the m x m projected overlap and the triangular
// solves with it, above the host's range of m.
//
// At m = 256 the library's potrf takes 0.77 ms and each triangular solve 0.29 ms: one
// or a few SMs' FP64 pipes (two multiply-adds a clock each) do the work.  Here the
// factor goes by 32-column panels, a launch for the panel (each block factors the
// 32 x 32 diagonal block for itself, the rows below are spread over the chip) and
// one for the rest of the matrix (16 x 16 tiles); a solve is one launch with two
// right-hand sides per block, so that all SMs share them: 0.27 and 0.09 ms.
#include "gbfe_internal.cuh"

#include <algorithm>

using namespace gbfe;

namespace {

constexpr uint32_t CB = 32;  // panel width

// Columns k0 .. k0 + 31 of the factor of the column-major A (lower triangle).  256
// threads; block b solves rows k0 + 32 + 32 b ...  The diagonal block goes to diag
// (the other blocks may still read it in A) and is put into A by k_chol_rest; the
// last panel writes it itself.  Bound by its chain: 32 x (rsqrt, scale, one
// barrier each, up to four multiply-adds a warp), about 10 us.
__global__ void __launch_bounds__(256) k_chol_panel(double *__restrict__ A, uint32_t n, uint32_t k0,
                                                    double *__restrict__ diag, int *__restrict__ info) {
  pdl_enter();
  __shared__ double D[CB][CB + 1];
  __shared__ double rd[CB];
  const uint32_t nb = min(CB, n - k0), lane = threadIdx.x % 32, w = threadIdx.x / 32;
  for (uint32_t t = threadIdx.x; t < CB * CB; t += 256) {
    const uint32_t i = t % CB, j = t / CB;
    D[i][j] = i < nb && j <= i ? __ldcg(A + (uint64_t)(k0 + j) * n + k0 + i) : (i == j ? 1.0 : 0.0);
  }
  for (uint32_t j = 0; j < CB; ++j) {
    __syncthreads();
    if (w == 0) {
      const double d = D[j][j];
      if (!(d > 0.0) && lane == 0 && blockIdx.x == 0 && *info == 0) *info = (int)(k0 + j + 1);
      const double rs = rsqrt(d);
      __syncwarp();
      if (lane == j) {
        D[j][j] = d * rs;
        rd[j] = rs;
      } else if (lane > j) {
        D[lane][j] *= rs;
      }
    }
    __syncthreads();
    for (uint32_t k = j + 1 + w; k < CB; k += 8)
      if (lane >= k) D[lane][k] = fma(-D[lane][j], D[k][j], D[lane][k]);
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (uint32_t t = threadIdx.x; t < CB * CB; t += 256) {
      const uint32_t i = t % CB, j = t / CB;
      if (i >= nb || j > i) continue;
      if (n > k0 + CB) {
        diag[t] = D[i][j];
      } else {
        A[(uint64_t)(k0 + j) * n + k0 + i] = D[i][j];
        A[(uint64_t)(k0 + i) * n + k0 + j] = D[i][j];
      }
    }
  // rows below: eight lanes a row, four columns each
  const uint32_t r = k0 + CB + blockIdx.x * 32 + threadIdx.x / 8, l8 = threadIdx.x % 8;
  const bool in = r < n;  // (nb == 32 where rows are left)
  double a[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = in ? __ldcg(A + (uint64_t)(k0 + q * 8 + l8) * n + r) : 0.0;
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const int j = q * 8 + l;
      const double x = __shfl_sync(0xffffffffu, a[q], l, 8) * rd[j];
      if ((int)l8 == l) a[q] = x;
#pragma unroll
      for (int p = q; p < 4; ++p) {
        const int c = p * 8 + (int)l8;
        if (c > j) a[p] = fma(-x, D[c][j], a[p]);
      }
    }
  if (in)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t c = k0 + q * 8 + l8;
      A[(uint64_t)c * n + r] = a[q];
      A[(uint64_t)r * n + c] = a[q];  // L^T, for the solves with it
    }
}

// A(i, j) -= sum_k L(i, k) L(j, k) over the panel, i >= j >= k0 + 32: one 16 x 16
// tile per block, one entry per thread.
__global__ void __launch_bounds__(256) k_chol_rest(double *__restrict__ A, uint32_t n, uint32_t k0,
                                                   const double *__restrict__ diag) {
  pdl_enter();
  __shared__ double P[16][CB + 1], Q[16][CB + 1];
  uint32_t t = blockIdx.x, ti = 0;
  while (t > ti) t -= ++ti;  // tile (ti, t), t <= ti
  const uint32_t i0 = k0 + CB + ti * 16, j0 = k0 + CB + t * 16;
  for (uint32_t u = threadIdx.x; u < 16 * CB; u += 256) {
    const uint32_t i = u % 16, k = u / 16;
    P[i][k] = i0 + i < n ? __ldcg(A + (uint64_t)(k0 + k) * n + i0 + i) : 0.0;
    Q[i][k] = j0 + i < n ? __ldcg(A + (uint64_t)(k0 + k) * n + j0 + i) : 0.0;
  }
  if (blockIdx.x == 0)
    for (uint32_t u = threadIdx.x; u < CB * CB; u += 256) {
      const uint32_t i = u % CB, j = u / CB;
      if (j > i) continue;
      A[(uint64_t)(k0 + j) * n + k0 + i] = diag[u];
      A[(uint64_t)(k0 + i) * n + k0 + j] = diag[u];
    }
  __syncthreads();
  const uint32_t i = i0 + threadIdx.x % 16, j = j0 + threadIdx.x / 16;
  if (i >= n || j >= n || i < j) return;
  double s = 0.0;
#pragma unroll
  for (uint32_t k = 0; k < CB; ++k) s = fma(P[threadIdx.x % 16][k], Q[threadIdx.x / 16][k], s);
  double *a = A + (uint64_t)j * n + i;
  *a = __ldcg(a) - s;
}

// X = L^-1 B, or L^-T B with UP, for two columns of B per block; L holds the factor
// below and its transpose above the diagonal.  X may be B; TR stores X^T (to another
// array).  By 32-row blocks: a warp per column solves with the diagonal block, then
// all threads take the solved rows out of the others.  At 256 x 256 half of the time
// is the chain of the first (shuffle, division by a two-word reciprocal,
// multiply-add, subtraction).
constexpr uint32_t TC = 2;
template <bool UP, bool TR>
__global__ void __launch_bounds__(256) k_tri_solve(const double *__restrict__ L, uint32_t n, const double *B,
                                                   double *X) {
  pdl_enter();
  extern __shared__ double tri_x[];  // TC x n
  __shared__ double D[CB][CB + 1], rd[2][CB];
  const uint32_t c0 = blockIdx.x * TC, nc = min(TC, n - c0);
  for (uint32_t t = threadIdx.x; t < TC * n; t += 256)
    tri_x[t] = t < nc * n ? __ldcg(B + (uint64_t)c0 * n + t) : 0.0;
  const uint32_t blocks = (n + CB - 1) / CB, lane = threadIdx.x % 32, w = threadIdx.x / 32;
  for (uint32_t s = 0; s < blocks; ++s) {
    const uint32_t k0 = (UP ? blocks - 1 - s : s) * CB, nb = min(CB, n - k0);
    // D[i][j]: entry (row i, column j) of the block of L or L^T
    for (uint32_t t = threadIdx.x; t < CB * CB; t += 256) {
      const uint32_t i = t % CB, j = t / CB;
      D[i][j] = i < nb && j < nb && (UP ? i <= j : i >= j) ? __ldcg(L + (uint64_t)(k0 + j) * n + k0 + i) : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < CB) {
      // 1 / d in two words: v / d = fma(v, hi, v lo) rounds once (with one word the
      // error of its rounding is the same for all columns, and the residual twice
      // the library's)
      const double d = threadIdx.x < nb ? D[threadIdx.x][threadIdx.x] : 1.0, hi = 1.0 / d;
      rd[0][threadIdx.x] = hi;
      rd[1][threadIdx.x] = fma(-hi, d, 1.0) * hi;
    }
    __syncthreads();
    if (w < TC) {
      const double v = lane < nb ? tri_x[w * n + k0 + lane] : 0.0;
      double acc = 0.0, x = 0.0;  // (a sum of its own: its roundings are smaller than v's)
#pragma unroll 8
      for (uint32_t q = 0; q < CB; ++q) {
        const uint32_t j = UP ? CB - 1 - q : q;
        const double vj = __shfl_sync(0xffffffffu, v - acc, j), y = fma(vj, rd[0][j], vj * rd[1][j]);
        if (lane == j) x = y;
        acc = fma(D[lane][j], y, acc);  // (zeros for the rows that are solved)
      }
      if (lane < nb) tri_x[w * n + k0 + lane] = x;
    }
    __syncthreads();
    const uint32_t lo = UP ? 0 : k0 + nb, hi = UP ? k0 : n;
    for (uint32_t r = lo + threadIdx.x; r < hi; r += 256) {
      double a0 = 0.0, a1 = 0.0;
#pragma unroll 8
      for (uint32_t j = 0; j < nb; ++j) {
        const double l = __ldcg(L + (uint64_t)(k0 + j) * n + r);
        a0 = fma(l, tri_x[k0 + j], a0);
        a1 = fma(l, tri_x[n + k0 + j], a1);
      }
      tri_x[r] -= a0;
      tri_x[n + r] -= a1;
    }
    __syncthreads();
  }
  for (uint32_t t = threadIdx.x; t < nc * n; t += 256) {
    const uint32_t c = t / n, r = t % n;
    X[TR ? (uint64_t)r * n + c0 + c : (uint64_t)(c0 + c) * n + r] = tri_x[t];
  }
}

template <bool UP, bool TR>
void tri_solve(gbfe_ctx *ctx, const double *L, uint32_t n, const double *B, double *X) {
  pdl_launch(ctx, k_tri_solve<UP, TR>, (n + TC - 1) / TC, 256, TC * n * sizeof(double), ctx->stream, L, n, B, X);
  check_launch(ctx, "tri_solve");
}

}  // namespace

namespace gbfe {

// A = L L^T in place (L below the diagonal, L^T above); info_d: 0, or the order of
// the first leading minor that is not positive.
void device_cholesky(gbfe_ctx *ctx, uint32_t n, double *A, int *info_d) {
  ctx->eig_ws.ensure(eig_ws_size(n));
  double *diag = ctx->eig_ws.p;
  GBFE_CUDA(cudaMemsetAsync(info_d, 0, sizeof(int), ctx->stream));
  for (uint32_t k0 = 0; k0 < n; k0 += CB) {
    const uint32_t rest = n - std::min(n, k0 + CB);
    pdl_launch(ctx, k_chol_panel, std::max(1u, (rest + 31) / 32), 256, 0, ctx->stream, A, n, k0, diag, info_d);
    check_launch(ctx, "chol_panel");
    if (!rest) break;
    const uint32_t nt = (rest + 15) / 16;
    pdl_launch(ctx, k_chol_rest, nt * (nt + 1) / 2, 256, 0, ctx->stream, A, n, k0, (const double *)diag);
    check_launch(ctx, "chol_rest");
  }
}

// S <- L^-1 S L^-T for a symmetric S (the full matrix given and returned)
void device_sandwich(gbfe_ctx *ctx, uint32_t n, const double *L, double *S) {
  ctx->eig_ws.ensure(eig_ws_size(n));
  double *W = ctx->eig_ws.p;
  tri_solve<false, true>(ctx, L, n, S, W);  // W = (L^-1 S)^T = S L^-T
  tri_solve<false, false>(ctx, L, n, W, S);
}

// V <- L^-T V
void device_trsm_lower_t(gbfe_ctx *ctx, uint32_t n, const double *L, double *V) {
  tri_solve<true, false>(ctx, L, n, V, V);
}

}  // namespace gbfe
