// gbfe_pcg.cu -- batched Jacobi-preconditioned CG over independent Poisson
// instances stored as one block-diagonal system.
//
// Each instance i owns the dof range [off_i, off_{i+1}) of the concatenated
// vectors; the operator is the block-diagonal union of the instances' cell
// operators (one cell launch serves all of them).  Every scalar of
// CGLinearSolver::solve (linearAlgebra/CGLinearSolver.t.cpp:68-313) -- the
// dots z.r and p.w, alpha, beta, the residual norm and the convergence /
// divergence tests -- is kept per instance on the device, so an iteration is
// a fixed sequence of kernels with no host round trip.  That sequence is
// captured once into a CUDA graph and replayed; the host reads the count of
// still-active instances every `chunk` iterations.
//
// A converged (or diverged) instance is frozen: no kernel touches its vectors
// again (nor works on its cells), so its x stays the iterate at which it
// converged -- the xConverged of the reference.
// Reductions run over fixed chunks of dofs per instance in a fixed summation
// order, so results are bitwise reproducible.
//
// An iteration is four launches: the cell product (on the tensor cores where
// the cells share matrices, gbfe_shared.cu), the assembly with p.w, the x / r
// update with z = D^-1 r and both dots, and the p update with the convergence
// tests.  Each kernel sums the partials it needs itself.
#include "gbfe_internal.cuh"

#include <algorithm>
#include <cmath>

using namespace gbfe;

namespace {

constexpr unsigned kThreads = 256;
constexpr uint64_t kInstChunks = 128, kMaxChunk = 4096;

// The dofs of every instance in chunks of a multiple of kThreads; instance i owns
// chunks [first[i], first[i + 1]), a block each.  The length depends on the
// instance alone, so its sums, and its results, are those of a solve of its own
// whatever else is in the batch: 128 chunks, unless they are longer than 4,096 dofs
// (alone, most SMs have one; in a batch a block's start and sums, 45 FP64 warp
// instructions at 64 clocks, stay below its work, six for 32 dofs).  Blocks take the
// chunks in descending length, so that all SMs get the same share of long and short
// ones.  24 instances of 2.66 M dofs: 55.2 ms, in the order of the instances 59.2;
// 64 chunks 54.6, but 389 k dofs alone 49.0 -> 57.2 us an iteration.
struct Chunk {
  uint64_t begin;
  uint32_t len, inst, index;
};
struct Chunks {
  const Chunk *chunk;
  const uint32_t *first;
};
uint64_t chunk_size(uint64_t len) {
  const uint64_t per = (len + kInstChunks - 1) / kInstChunks;
  return std::min<uint64_t>(kMaxChunk, (per + kThreads - 1) / kThreads * kThreads);
}

// per-instance state; what one block writes while others read the old value
// (zr and the running flag) exists twice, and alternate iterations swap the two
struct PcgState {
  const double *zr;
  const int *active;
  double *zr_new;
  int *active_new;
  double *bnorm, *rnorm;
  int *status;
  uint32_t *iters, *iter;
  double *part[3];  // partial sums per chunk: p.w (or b.b at the start), z.r, r.r
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sums of a and b over the block in a fixed order into *pa and *pb (b only when
// pb is given): a warp per sum adds the threads' values 32 apart, then shuffles
// (one warp's adds instead of every warp's: the FP64 pipe takes 64 clocks each)
template <unsigned NT = kThreads>
__device__ __forceinline__ void block_sums(double a, double b, double *pa, double *pb) {
  __shared__ double sh[2][NT];
  sh[0][threadIdx.x] = a;
  if (pb) sh[1][threadIdx.x] = b;
  __syncthreads();
  const unsigned w = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (w == 0 || (w == 1 && pb)) {
    double v = sh[w][lane];
#pragma unroll
    for (unsigned k = 1; k < NT / 32; ++k) v += sh[w][lane + 32 * k];
    v = warp_sum(v);
    if (lane == 0) *(w ? pb : pa) = v;
  }
}

// sum of instance i's partials, by one warp (valid in its lanes): every block
// that needs it forms it again (at most a few hundred values from L2, the same
// order in every block) instead of a launch between two kernels of the iteration
__device__ __forceinline__ double inst_sum(const double *part, const Chunks &ch, uint32_t i) {
  double v = 0.0;
  for (uint32_t c = ch.first[i] + threadIdx.x % 32; c < ch.first[i + 1]; c += 32) v += part[c];
  return warp_sum(v);
}
// a value of warp 0 for the whole block
__device__ __forceinline__ double from_warp0(double v) {
  __shared__ double sh;
  if (threadIdx.x == 0) sh = v;
  __syncthreads();
  return sh;
}

// partials of x.y, and of u.v when u is given (NT: the threads of the kernel that forms
// the same sum elsewhere, so that the order is the same)
template <unsigned NT = kThreads>
__global__ void __launch_bounds__(NT) k_chunk_dots(const Chunks ch, const double *__restrict__ x,
                                                   const double *__restrict__ y, double *__restrict__ pxy,
                                                   const double *__restrict__ u, const double *__restrict__ v,
                                                   double *__restrict__ puv) {
  pdl_enter();
  const Chunk ck = ch.chunk[blockIdx.x];
  const uint64_t b = ck.begin, e = b + ck.len;
  double s = 0.0, q = 0.0;
  for (uint64_t t = b + threadIdx.x; t < e; t += NT) {
    s += x[t] * y[t];
    if (u) q += u[t] * v[t];
  }
  block_sums<NT>(s, q, pxy + ck.index, u ? puv + ck.index : nullptr);
}

// w = assembled cell-wise product (Dirichlet rows zero) and the partials of
// p.w: bound by the latency of its indirect reads (slot list and cell rows, 93
// MB at 2.66 M dofs), so it wants threads rather than loads per thread: 2,048
// threads on an SM at 32 registers, two dofs each per pass, take 28.7 us; three
// dofs the same, 1,024 threads with four dofs 38, 1,536 37.  (The x / r update
// is bound by its FP64 operations: 512 threads per block make it 31.5 us
// instead of 28.5.)
constexpr unsigned kAsmThreads = 512;
__global__ void __launch_bounds__(kAsmThreads, 2048 / kAsmThreads) k_assemble_dot(const Chunks ch, const int *__restrict__ active,
                                                           const double *__restrict__ Yc,
                                                           const uint32_t *__restrict__ slot_ptr,
                                                           const uint32_t *__restrict__ slot,
                                                           const uint8_t *__restrict__ is_row,
                                                           const double *__restrict__ p, double *__restrict__ w,
                                                           double *__restrict__ ppw) {
  pdl_enter();
  const Chunk ck = ch.chunk[blockIdx.x];
  if (!active[ck.inst]) return;
  const uint64_t b = ck.begin, e = b + ck.len;
  double s = 0.0;
  // two dofs per pass: their slot ranges, then the slots (in order; the first
  // one starts the sum), so the indirect loads of both are in flight
  for (uint64_t t0 = b + threadIdx.x; t0 < e; t0 += 2 * kAsmThreads) {
    uint32_t q[2], qe[2];
    double acc[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint64_t t = t0 + k * kAsmThreads;
      const bool on = t < e && !(is_row && is_row[t]);
      q[k] = on ? slot_ptr[t] : 0u;
      qe[k] = on ? slot_ptr[t + 1] : 0u;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) acc[k] = q[k] < qe[k] ? Yc[slot[q[k]]] : 0.0;
#pragma unroll
    for (int k = 0; k < 2; ++k)
      for (uint32_t j = q[k] + 1; j < qe[k]; ++j) acc[k] += Yc[slot[j]];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint64_t t = t0 + k * kAsmThreads;
      if (t < e) {
        w[t] = acc[k];
        s += p[t] * acc[k];
      }
    }
  }
  block_sums<kAsmThreads>(s, 0.0, ppw + ck.index, nullptr);
}

// alpha = zr / p.w;  x += alpha p;  r -= alpha w  (add(ones, x, alpha, p, x)
// etc.), and with a Jacobi preconditioner (d given) z = d o r on the fly and
// the partials of z.r and r.r
__global__ void __launch_bounds__(kThreads) k_update_xr(const Chunks ch, const PcgState s,
                                                        const double *__restrict__ p, const double *__restrict__ w,
                                                        const double *__restrict__ d, double *__restrict__ x,
                                                        double *__restrict__ r) {
  pdl_enter();
  const Chunk ck = ch.chunk[blockIdx.x];
  const uint32_t i = ck.inst;
  if (!s.active[i]) return;
  const double a = from_warp0(threadIdx.x < 32 ? s.zr[i] / inst_sum(s.part[0], ch, i) : 0.0);
  const uint64_t b = ck.begin, e = b + ck.len;
  double zr = 0.0, rr = 0.0;
#pragma unroll 4
  for (uint64_t t = b + threadIdx.x; t < e; t += kThreads) {
    double rt = r[t];
    if (a != 0.0) {
      x[t] = x[t] + a * p[t];
      rt = rt + (-a) * w[t];
      r[t] = rt;
    }
    if (d) {
      zr += (d[t] * rt) * rt;
      rr += rt * rt;
    }
  }
  if (d) block_sums(zr, rr, s.part[1] + ck.index, s.part[2] + ck.index);
}

// beta = zr_new / zr;  p = z + beta p  (z = d o r, or the vector z) with the
// Dirichlet rows of the next product's input zeroed; the first block of an
// instance also runs the convergence / divergence tests of the iteration.
// start: iteration 0 (p = z, every instance running)
__global__ void __launch_bounds__(kThreads) k_update_p(const Chunks ch, const PcgState s, bool start,
                                                       double abs_tol, double rel_tol, double div_tol,
                                                       uint32_t max_iter, const double *__restrict__ d,
                                                       const double *__restrict__ r, const double *__restrict__ z,
                                                       const uint8_t *__restrict__ is_row, double *__restrict__ p) {
  pdl_enter();
  const Chunk ck = ch.chunk[blockIdx.x];
  const uint32_t i = ck.inst;
  const bool head = ch.first[i] == ck.index;
  const bool act = start || s.active[i];
  if (!act) {
    if (head && threadIdx.x == 0) s.active_new[i] = 0;
    return;
  }
  const double zrn = from_warp0(threadIdx.x < 32 ? inst_sum(s.part[1], ch, i) : 0.0);
  const double beta = start ? 0.0 : zrn / s.zr[i];
  const uint64_t b = ck.begin, e = b + ck.len;
#pragma unroll 4
  for (uint64_t t = b + threadIdx.x; t < e; t += kThreads) {
    const double zt = d ? d[t] * r[t] : z[t];
    const double pt = start ? zt : zt + beta * p[t];
    p[t] = (is_row && is_row[t]) ? 0.0 : pt;
  }
  if (!head || threadIdx.x >= 32) return;
  const double rn = sqrt(inst_sum(s.part[2], ch, i));
  const double bn = start ? sqrt(inst_sum(s.part[0], ch, i)) : 0.0;
  if (threadIdx.x != 0) return;
  if (start) {
    s.bnorm[i] = bn;
    s.status[i] = GBFE_ERR_NOT_CONVERGED;
    s.iters[i] = 0;
    s.iter[i] = 0;
  }
  const uint32_t it = s.iter[i];
  s.iter[i] = it + 1;
  s.zr_new[i] = zrn;
  s.rnorm[i] = rn;
  int on = 1;
  const double tol = fmax(abs_tol, s.bnorm[i] * rel_tol);
  if (rn < tol) {
    on = 0;
    s.status[i] = GBFE_OK;
    s.iters[i] = it;
  } else if (rn > div_tol) {
    on = 0;
    s.status[i] = GBFE_ERR_DIVERGED;
    s.iters[i] = it;
  } else if (it >= max_iter) {
    on = 0;
    s.status[i] = GBFE_ERR_NOT_CONVERGED;
    s.iters[i] = it + 1;
  }
  s.active_new[i] = on;
}

// r = b - w (iteration 0)
__global__ void k_residual0(double *__restrict__ r, const double *__restrict__ b, const double *__restrict__ w,
                            uint64_t N) {
  pdl_enter();
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < N; t += (uint64_t)gridDim.x * blockDim.x)
    r[t] = 1.0 * b[t] + (-1.0) * w[t];
}

__global__ void k_count_active(const int *__restrict__ active, uint32_t n, int *__restrict__ out) {
  __shared__ int sh[256];
  int c = 0;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) c += active[i];
  sh[threadIdx.x] = c;
  __syncthreads();
  for (unsigned w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

}  // namespace

extern "C" int gbfe_pcg_solve_batched(const gbfe_op *A, const gbfe_op *PC, const gbfe_mv *b, gbfe_mv *x,
                                      uint32_t n_inst, const uint64_t *inst_dof_off, uint32_t max_iter,
                                      double abs_tol, double rel_tol, double div_tol, uint32_t iters_chunk,
                                      uint32_t *iters_out, int *status_out, double *rnorm_out) {
  if (!A || !PC || !b || !x || !inst_dof_off || n_inst == 0) return GBFE_ERR_ARG;
  gbfe_ctx *ctx = x->mesh->ctx;
  return gbfe_guard(ctx, [&] {
    TempScope temps(ctx);
    gbfe_mesh *me = x->mesh;
    GBFE_REQUIRE(b->mesh == me && A->mesh == me && PC->mesh == me, "pcg_batched: operands on different meshes");
    GBFE_REQUIRE(b->m == 1 && x->m == 1 && b->dtype == GBFE_F64 && x->dtype == GBFE_F64,
                 "pcg_batched: b and x are FP64 single vectors over all instances");
    GBFE_REQUIRE(inst_dof_off[0] == 0 && inst_dof_off[n_inst] == me->n_dofs,
                 "pcg_batched: instance offsets must cover [0, n_dofs)");
    for (uint32_t i = 0; i < n_inst; ++i)
      GBFE_REQUIRE(inst_dof_off[i + 1] > inst_dof_off[i], "pcg_batched: empty or unsorted instance range");
    const uint64_t N = me->n_dofs;
    const Restore<int> no_profiling(ctx->profiling, 0);  // event brackets cannot be captured into the graph
    // chunk table
    std::vector<Chunk> h_chunk;
    std::vector<uint32_t> h_first(n_inst + 1);
    for (uint32_t i = 0; i < n_inst; ++i) {
      h_first[i] = (uint32_t)h_chunk.size();
      const uint64_t end = inst_dof_off[i + 1], per = chunk_size(end - inst_dof_off[i]);
      for (uint64_t t = inst_dof_off[i]; t < end; t += per)
        h_chunk.push_back(Chunk{t, (uint32_t)std::min(per, end - t), i, (uint32_t)h_chunk.size()});
    }
    const uint32_t n_chunks = h_first[n_inst] = (uint32_t)h_chunk.size();
    std::stable_sort(h_chunk.begin(), h_chunk.end(), [](const Chunk &x, const Chunk &y) { return x.len > y.len; });
    DBuf<Chunk> d_chunk;
    DBuf<uint32_t> d_first, cnt;
    d_chunk.upload(h_chunk.data(), h_chunk.size(), ctx->stream);
    d_first.upload(h_first.data(), h_first.size(), ctx->stream);
    const Chunks ch{d_chunk.p, d_first.p};
    DBuf<double> sc, part;
    sc.alloc((size_t)4 * n_inst);
    part.alloc((size_t)3 * n_chunks);
    DBuf<int> flags;
    flags.alloc((size_t)3 * n_inst + 1);
    cnt.alloc((size_t)2 * n_inst);
    PcgState s{};
    double *const zr_buf[2] = {sc.p, sc.p + n_inst};
    int *const act_buf[2] = {flags.p, flags.p + n_inst};
    s.bnorm = sc.p + 2 * n_inst;
    s.rnorm = sc.p + 3 * n_inst;
    s.status = flags.p + 2 * n_inst;
    int *d_active_count = flags.p + 3 * n_inst;
    s.iters = cnt.p;
    s.iter = cnt.p + n_inst;
    for (int k = 0; k < 3; ++k) s.part[k] = part.p + (size_t)k * n_chunks;
    // state buffers of an iteration that reads buffer k and writes the other
    auto turn = [&](int k) {
      s.zr = zr_buf[k];
      s.active = act_buf[k];
      s.zr_new = zr_buf[k ^ 1];
      s.active_new = act_buf[k ^ 1];
    };
    gbfe_mv r, z, p, w;
    for (gbfe_mv *v : {&r, &z, &p, &w}) {
      v->mesh = me;
      v->m = 1;
      v->dtype = GBFE_F64;
      v->d.alloc(N);
      GBFE_CUDA(cudaMemsetAsync(v->d.p, 0, N * 8, ctx->stream));
    }
    const unsigned gN = (unsigned)std::min<uint64_t>((N + 255) / 256, (uint64_t)ctx->sm_count * 16);
    // Cell operators without a nonlocal part: the product (on the tensor cores for
    // the instances whose cells share matrices), then, with homogeneous Dirichlet
    // rows only (what a Poisson batch is), one kernel for the assembly and p.w, else
    // two with the same sums.  Anything else goes through the general apply.
    const bool cells = A->kind == OP_CELL && !A->nl;
    const bool fused = cells && (!A->cons || A->cons->pure_dirichlet);
    const uint8_t *is_row = fused && A->cons ? A->cons->is_row.p : nullptr;
    SharedInst shared_inst;
    const gbfe_shared *shared = cells ? shared_plan(A, n_inst, inst_dof_off, shared_inst) : nullptr;
    const double *jac = PC->kind == OP_JACOBI ? PC->diag.p : nullptr;
    if (cells) A->cellbuf.ensure((size_t)me->total_cell_dofs);
    // iteration 0 (outside the graph; the general apply also sizes its scratch).  The
    // product that the iterations use takes 0.1 ms here, the FP64 one 1.2.
    if (shared) {
      constraints_p2c(ctx, A->cons, x);
      cell_apply_shared(A, *shared, x->d.p, A->cellbuf.p, nullptr, shared_inst);
      assemble_cells(me, A->cons, GBFE_F64, A->cellbuf.p, &w, nullptr, nullptr);
    } else {
      apply_op(A, x, &w);
    }
    pdl_launch(ctx, k_residual0, gN, 256, 0, ctx->stream, r.d.p, b->d.p, w.d.p, N);
    apply_op(PC, &r, &z);
    pdl_launch(ctx, k_chunk_dots<kThreads>, n_chunks, kThreads, 0, ctx->stream, ch, b->d.p, b->d.p, s.part[0],
               nullptr, nullptr, nullptr);
    pdl_launch(ctx, k_chunk_dots<kThreads>, n_chunks, kThreads, 0, ctx->stream, ch, z.d.p, r.d.p, s.part[1], r.d.p,
               r.d.p, s.part[2]);
    turn(1);
    pdl_launch(ctx, k_update_p, n_chunks, kThreads, 0, ctx->stream, ch, s, true, abs_tol, rel_tol, div_tol, max_iter,
               nullptr, r.d.p, z.d.p, is_row, p.d.p);
    check_launch(ctx, "pcg_start");
    count_launch(ctx, 3);
    // one CG iteration, captured
    auto iteration = [&](int k) {
      turn(k);
      if (fused || shared) {
        if (!fused) constraints_p2c(ctx, A->cons, &p);
        if (shared)
          cell_apply_shared(A, *shared, p.d.p, A->cellbuf.p, s.active, shared_inst);
        else
          cell_product_f64(A, &p, A->cellbuf.p);
      }
      if (fused) {
        pdl_launch(ctx, k_assemble_dot, n_chunks, kAsmThreads, 0, ctx->stream, ch, s.active, A->cellbuf.p,
                   me->slot_ptr.p, me->slot.p, is_row, p.d.p, w.d.p, s.part[0]);
      } else {
        if (shared)
          assemble_cells(me, A->cons, GBFE_F64, A->cellbuf.p, &w, nullptr, nullptr);
        else
          apply_op(A, &p, &w);
        pdl_launch(ctx, k_chunk_dots<kAsmThreads>, n_chunks, kAsmThreads, 0, ctx->stream, ch, p.d.p, w.d.p, s.part[0],
                   nullptr, nullptr, nullptr);
      }
      pdl_launch(ctx, k_update_xr, n_chunks, kThreads, 0, ctx->stream, ch, s, p.d.p, w.d.p, jac, x->d.p, r.d.p);
      if (!jac) {
        apply_op(PC, &r, &z);
        pdl_launch(ctx, k_chunk_dots<kThreads>, n_chunks, kThreads, 0, ctx->stream, ch, z.d.p, r.d.p, s.part[1], r.d.p, r.d.p,
                   s.part[2]);
        count_launch(ctx);
      }
      pdl_launch(ctx, k_update_p, n_chunks, kThreads, 0, ctx->stream, ch, s, false, abs_tol, rel_tol, div_tol,
                 max_iter, jac, r.d.p, z.d.p, is_row, p.d.p);
      check_launch(ctx, "pcg_iteration");
      count_launch(ctx, 2);
    };
    // iterations per replay: the requested polling interval, rounded up to even
    // (the state alternates between two buffers)
    const uint32_t chunk = (std::max<uint32_t>(1, iters_chunk) + 1) / 2 * 2;
    struct Graph {
      cudaGraph_t graph = nullptr;
      cudaGraphExec_t exec = nullptr;
      ~Graph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
      }
    } g;
    uint64_t per_replay = 0;
    {
      const Restore<uint64_t> not_launched(ctx->launches, ctx->launches);
      const uint64_t before = ctx->launches;
      CaptureScope capture(ctx->stream, ctx->capturing);
      GBFE_CUDA(capture.begin());
      for (uint32_t k = 0; k < chunk; ++k) iteration(k & 1);
      GBFE_CUDA(capture.end(&g.graph));
      per_replay = ctx->launches - before;
    }
    GBFE_CUDA(cudaGraphInstantiate(&g.exec, g.graph, 0));
    int active = 1;
    uint32_t done_iters = 0;
    while (true) {
      k_count_active<<<1, 256, 0, ctx->stream>>>(act_buf[0], n_inst, d_active_count);
      count_launch(ctx);
      GBFE_CUDA(cudaMemcpyAsync(&active, d_active_count, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      GBFE_CUDA(cudaStreamSynchronize(ctx->stream));
      if (active == 0 || done_iters > max_iter) break;
      if (ctx->cancel && ctx->cancel->load()) throw Error(GBFE_ERR_CANCELLED, "cancelled");
      GBFE_CUDA(cudaGraphLaunch(g.exec, ctx->stream));
      ctx->launches += per_replay;
      done_iters += chunk;
    }
    std::vector<double> rn(n_inst);
    GBFE_CUDA(cudaMemcpyAsync(rn.data(), s.rnorm, n_inst * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (iters_out) GBFE_CUDA(cudaMemcpyAsync(iters_out, s.iters, n_inst * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (status_out) GBFE_CUDA(cudaMemcpyAsync(status_out, s.status, n_inst * 4, cudaMemcpyDeviceToHost, ctx->stream));
    GBFE_CUDA(cudaStreamSynchronize(ctx->stream));
    if (rnorm_out) std::copy(rn.begin(), rn.end(), rnorm_out);
  });
}
