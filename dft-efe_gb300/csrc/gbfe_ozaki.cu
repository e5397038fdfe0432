// gbfe_ozaki.cu -- FP64-accurate cell product on the BF16 tensor cores
// (the splitting scheme of Ozaki, Ogita, Oishi & Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication", Numer. Algorithms 59, 2012).
//
// GB300 runs FP64 FMA at ~1.25 TFLOP/s, so the FP64 cell product of the plain
// path is bound by the FP64 pipe.  Here each operand is cut into seven
// balanced base-256 digit slices (gbfe_oz.cuh), which BF16 represents exactly:
//     A_op[j][k] = 2^(ea_j+1) sum_s a_s[j][k] 2^-8s     (per-row exponent ea_j)
//     X[i][v]    = 2^(ex_v+1) sum_t x_t[i][v] 2^-8t     (per-vector exponent ex_v)
// with a rounding error below 2^-56 of the row / vector maximum.  For every
// level g = s + t (2..8) the tensor cores accumulate
//     L_g[j][v] = sum_{s+t=g} sum_k a_s[j][k] x_t[k][v]
// in FP32 TMEM accumulators of 64 vectors, one per level and a second one for level
// 6: every sum of levels 2 to 6 is exact for cells of up to 256 dofs (gbfe_oz.cuh has
// the bound of levels 7 and 8).  The epilogue adds the levels, rounds once to FP64
// and applies 2^(ea_j + ex_v - 62).  The 28 digit-pair products of a K step are
// issued as 11 MMAs (N up to 256) over stacked slices.
//
// Data movement follows the persistent split-BF16 kernel: A slices are
// pre-laid-out in HBM (per cell, per K chunk of 32, 7 slices in the canonical
// K-major core-matrix layout) and land by bulk TMA copies; X rows are gathered
// by two groups of eight warps that cut each FP64 value into digits with integer
// instructions and also run the epilogue; one thread issues tcgen05.mma, one
// thread the bulk copies.
// Cells with more than 128 dofs are processed as two 128-row work items.
//
// An item of 216-dof cells takes about 30 k clocks: 7 K chunks at 2.5 k (1.86 k of
// MMAs, which keep shared memory busy: their small-N products read A again and
// again) and 8 k of epilogue, in which the MMAs wait for TMEM.  Measured on the
// way, 1,000 cells of 216 dofs, 256 vectors, product alone: 1,202 us with 8 slices
// of base 128, eight warps and two shared stages; 954 with 7 slices of base 256
// and ids loaded a chunk ahead; 924 with 16 warps; 854 with three B stages, filled
// before the epilogue of the item before; 805 with barriers asked before the abort
// flag.  (512 cells, ncu: 413 us so, 430 with the second accumulator of level 6 and
// every block copying the A slices for itself.)
#include "gbfe_internal.cuh"
#include "gbfe_oz.cuh"
#include "gbfe_tc_ptx.cuh"

#include <algorithm>

using namespace gbfe;
using namespace gbfe::tc;

namespace {

constexpr int OZ_S = oz::S7;   // slices per operand
constexpr int OZ_N = 64;       // vectors per work item
// Accumulators of 64 TMEM columns each: levels 2 .. 8, and one more of level 6 for A
// slice 5.  Over K <= 256 a product of two slices stays within 2^22, so levels up to 6
// (four products at most in each accumulator) are exact in FP32.
constexpr int OZ_ACC = 8, OZ_ACC_L6B = 7;
constexpr int OZ_AST = 2, OZ_BST = 3;          // ring stages of A and of B chunks
constexpr int OZ_GROUPS = 2;                   // groups of 8 gather warps, taking the chunks in turn
constexpr int OZ_GW = 8 * OZ_GROUPS;           // gather / epilogue warps
constexpr uint32_t OZ_ECOLS = OZ_N / (OZ_GW / 4);  // epilogue columns per warp
constexpr int OZ_EPI_COLS = 4;                 // of them at a time
constexpr int OZ_EPI_DOUBLES = 32 * OZ_EPI_COLS;
constexpr int OZ_TMA_WARP = OZ_GW, OZ_MMA_WARP = OZ_GW + 1;
constexpr int OZ_THREADS = (OZ_GW + 2) * 32;
constexpr uint32_t OZ_A_PART = 128 * KC * 2;  // one slice of a 128-row A chunk (bytes)
constexpr uint32_t OZ_B_PART = OZ_N * KC * 2;  // one slice of a B chunk
constexpr uint32_t OZ_A_STAGE = OZ_S * OZ_A_PART, OZ_B_STAGE = OZ_S * OZ_B_PART;
constexpr uint32_t OZ_RINGS = OZ_AST * OZ_A_STAGE + OZ_BST * OZ_B_STAGE;
constexpr uint32_t OZ_EPI = OZ_GW * OZ_EPI_DOUBLES * 8;  // epilogue staging, one tile per warp
constexpr uint32_t OZ_SMEM = OZ_RINGS + OZ_EPI + 1024 + 512;
static_assert(OZ_SMEM <= 227 * 1024, "sliced cell product: shared memory");

__device__ __forceinline__ int oz_exponent(double vmax) { return oz::exponent_of(vmax); }

// A_op = A_c^T slices: per (cell, chunk) [slice][MT8 x KC] canonical tiles,
// and per-row exponents (one per cell dof).
__global__ void k_build_oz_mats(const double *__restrict__ mats, const uint64_t *__restrict__ mat_off,
                                const uint32_t *__restrict__ cell_off, const uint64_t *__restrict__ a_off,
                                uint32_t n_cells, __nv_bfloat16 *__restrict__ out, int *__restrict__ row_exp) {
  const uint32_t c = blockIdx.x;
  if (c >= n_cells) return;
  const uint32_t off = cell_off[c], nd = cell_off[c + 1] - off;
  const uint32_t mt8 = (nd + 7) / 8 * 8, nk = (nd + KC - 1) / KC;
  const double *A = mats + mat_off[c];
  for (uint32_t j = threadIdx.x; j < nd; j += blockDim.x) {
    double mx = 0.0;
    for (uint32_t k = 0; k < nd; ++k) mx = fmax(mx, fabs(A[k + (uint64_t)nd * j]));
    row_exp[off + j] = oz_exponent(mx);
  }
  __syncthreads();
  __nv_bfloat16 *dst = out + a_off[c];
  const uint32_t per_slice = mt8 * KC;
  for (uint32_t idx = threadIdx.x; idx < nk * per_slice; idx += blockDim.x) {
    const uint32_t kc = idx / per_slice, rem = idx - kc * per_slice;
    const uint32_t r = rem / KC, kk = rem - r * KC;
    const uint32_t k = kc * KC + kk;
    const uint64_t u = oz::biased7(r < nd && k < nd ? A[k + (uint64_t)nd * r] : 0.0, r < nd ? row_exp[off + r] : 0);
    const uint32_t pos = (r / 8) * (KC / 8) * 64 + (kk / 8) * 64 + (r % 8) * 8 + (kk % 8);
    __nv_bfloat16 *base = dst + (uint64_t)kc * OZ_S * per_slice;
#pragma unroll
    for (int s = 0; s < OZ_S; ++s) base[(uint64_t)s * per_slice + pos] = __float2bfloat16_rn(oz::digit7(u, s + 1));
  }
}

// per-vector exponent of the largest |X[i][v]| (two-stage max of the exponent
// bits, integer instructions; max is order-free)
__global__ void k_colmax_partial(const double *__restrict__ X, uint64_t rows, uint32_t m, int *__restrict__ part) {
  pdl_enter();
  oz::colmax_partial_block(X, X, 1, m, rows, part);
}

__global__ void k_colmax_final(const int *__restrict__ part, uint32_t nb, uint32_t m, int *__restrict__ ex) {
  pdl_enter();
  oz::colmax_final_block(part, nb, m, ex);
}

struct OzArgs {
  const double *X;
  uint32_t m;
  const uint32_t *ids;
  const uint32_t *cell_off;
  const uint32_t *cells;  // cells of this launch
  uint32_t ncells;
  uint32_t mts;           // 128-row items per cell in this launch (1 or 2)
  uint32_t vt;            // vector tiles per cell
  const uint64_t *a_off;
  const __nv_bfloat16 *Aoz;
  const int *row_exp;
  const int *x_exp;
  double *Yc;
  uint32_t tmem_cols;
  int *status;
};

__global__ void __launch_bounds__(OZ_THREADS, 1) k_cell_apply_oz(const OzArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t *bring = smem + OZ_AST * OZ_A_STAGE;
  double *epi_scratch = (double *)(smem + OZ_RINGS);
  uint64_t *bars = (uint64_t *)(smem + OZ_RINGS + OZ_EPI);
  uint64_t *full_a = bars, *empty_a = full_a + OZ_AST;
  uint64_t *full_b = empty_a + OZ_AST, *empty_b = full_b + OZ_BST;
  uint64_t *tfull = empty_b + OZ_BST;
  uint64_t *tempty = tfull + 1;
  uint64_t *spare = tempty + 1;  // drain_mmas before TMEM is freed
  uint32_t *tmem_slot = (uint32_t *)(spare + 1);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const uint32_t m = a.m;
  const uint32_t per_cell = a.mts * a.vt;
  const uint32_t n_items = a.ncells * per_cell;
  const uint32_t first = blockIdx.x, step = gridDim.x;

  if (tid == 0) {
    for (int s = 0; s < OZ_AST; ++s) {
      mbar_init(&full_a[s], 1);
      mbar_init(&empty_a[s], 1);
    }
    for (int s = 0; s < OZ_BST; ++s) {
      mbar_init(&full_b[s], 8);
      mbar_init(&empty_b[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, OZ_GW);
    mbar_init(spare, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == OZ_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(a.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();  // (after the allocation, see pdl_trigger)
  if (warp != OZ_TMA_WARP) pdl_wait();  // (the A slices are complete: built under a stream synchronisation)

  auto wait = [&](uint64_t *bar, uint32_t parity, int code) -> bool {
    if (mbar_test(bar, parity)) return true;
    if (*abort_flag) return false;
    if (mbar_wait(bar, parity, a.status, code)) return true;
    *abort_flag = 1;
    return false;
  };
  auto decode = [&](uint32_t it, uint32_t &c, uint32_t &mt, uint32_t &v0) {
    c = a.cells[it / per_cell];
    const uint32_t rem = it % per_cell;
    mt = rem / a.vt;
    v0 = rem % a.vt * OZ_N;
  };

  if (warp == OZ_TMA_WARP) {
    // ---------------- TMA producer: the slice tiles of each chunk
    if (lane == 0) {
      uint32_t q = 0;
      // the vector tiles of a cell read its slices at about the same time, then they go
      // (evict-first with several tiles: 1,010 us, plain policy 1,008, as good)
      const uint64_t pol = l2_evict_first_policy();
      for (uint32_t it = first; it < n_items && !*abort_flag; it += step) {
        uint32_t c, mt, v0;
        decode(it, c, mt, v0);
        const uint32_t nd = a.cell_off[c + 1] - a.cell_off[c];
        const uint32_t mt8 = (nd + 7) / 8 * 8, nk = (nd + KC - 1) / KC;
        const uint32_t rows = min(128u, mt8 - 128 * mt);
        const __nv_bfloat16 *Acell = a.Aoz + a.a_off[c];
        for (uint32_t kc = 0; kc < nk; ++kc, ++q) {
          const uint32_t s = q % OZ_AST;
          if (q >= OZ_AST && !wait(&empty_a[s], ((q / OZ_AST) - 1) & 1, 21)) break;
          uint8_t *Ast = smem + s * OZ_A_STAGE;
          const uint32_t bytes = rows * KC * 2;
          mbar_arrive_expect_tx(&full_a[s], OZ_S * bytes);
          for (int sl = 0; sl < OZ_S; ++sl) {
            const __nv_bfloat16 *src = Acell + ((uint64_t)kc * OZ_S + sl) * mt8 * KC + (uint64_t)mt * 128 * KC;
            bulk_g2s_stream(Ast + sl * OZ_A_PART, src, bytes, &full_a[s], pol);
          }
        }
      }
      drain_copies(full_a, q, OZ_AST);
    }
    __syncwarp();
  } else if (warp == OZ_MMA_WARP) {
    // ---------------- MMA issuer: 28 products per K step into the level accumulators
    if (lane == 0) {
      uint32_t q = 0, li = 0;
      for (uint32_t it = first; it < n_items && !*abort_flag; it += step, ++li) {
        uint32_t c, mt, v0;
        decode(it, c, mt, v0);
        const uint32_t nd = a.cell_off[c + 1] - a.cell_off[c];
        const uint32_t nk = (nd + KC - 1) / KC;
        if (li >= 1 && !wait(tempty, (li - 1) & 1, 22)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        bool ok = true;
        for (uint32_t kc = 0; kc < nk; ++kc, ++q) {
          const uint32_t sa = q % OZ_AST, sb = q % OZ_BST;
          if (!mbar_test2(&full_a[sa], (q / OZ_AST) & 1, &full_b[sb], (q / OZ_BST) & 1) &&
              (!wait(&full_a[sa], (q / OZ_AST) & 1, 23) || !wait(&full_b[sb], (q / OZ_BST) & 1, 24))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t abase = smem_u32(smem + sa * OZ_A_STAGE);
          const uint32_t bbase = smem_u32(bring + sb * OZ_B_STAGE);
          for (uint32_t ks = 0; ks < KC / 16; ++ks) {
            // slice sl of A against the stacked B slices t0..t1 (one descriptor, N = 64
            // (t1 - t0 + 1)) into the contiguous levels sl+t0 .. sl+t1: 11 MMAs per K step;
            // the two sl = 1 MMAs and slice 5's one into its own accumulator start them all
            // (slice 5 in one MMA with all of level 6 in one accumulator: 1,008 us of
            // the 1,035 of an apply of 1,000 cells of 216 dofs, 256 vectors, and with all
            // digits at their limit results off by up to seven units of their last place)
            const uint32_t more = (kc | ks) == 0 ? 0u : 1u;
            auto run = [&](int sl, int t0, int t1, int acc, uint32_t add) {
              umma(tmem + acc * OZ_N, smem_desc(abase + (sl - 1) * OZ_A_PART + ks * 2 * LBO),
                   smem_desc(bbase + (t0 - 1) * OZ_B_PART + ks * 2 * LBO), instr_desc(128, OZ_N * (t1 - t0 + 1)), add);
            };
#pragma unroll
            for (int sl = 1; sl <= OZ_S; ++sl) {
              const int tl = OZ_S + 1 - sl;  // last slice of X
              if (sl == 5) {
                run(5, 1, 1, OZ_ACC_L6B, more);
                run(5, 2, tl, 5, 1);
                continue;
              }
#pragma unroll
              for (int t0 = 1; t0 <= tl; t0 += 4) run(sl, t0, t0 + 3 < tl ? t0 + 3 : tl, sl + t0 - 2, sl == 1 ? more : 1u);
            }
          }
          umma_commit(&empty_b[sb]);
          umma_commit(&empty_a[sa]);
        }
        if (!ok) break;
        umma_commit(tfull);
      }
      drain_mmas(spare);
    }
    __syncwarp();
  } else {
    // ---------------- gather warps: X rows -> digit slices; epilogue
    // (KC/8) K blocks x (OZ_N/32) vector groups = 8 warps per chunk; warp w always
    // gathers K block w % 4 of vector group (w / 4) % 2, and the OZ_GROUPS groups
    // of 8 warps take the chunks in turn.  The rows of a group's next chunk (of
    // this item or of a later one, across the epilogue) are loaded before the
    // current chunk's digits are cut, through ids loaded a chunk earlier still.
    const uint32_t kb = warp % 4, v = (warp / 4 % 2) * 32 + lane, grp = warp / 8;
    uint32_t c_it = first, c_kc = 0, c_nk = 0, c_off = 0, c_nd = 0, c_v = 0;  // cursor of the id loads
    auto cursor_item = [&]() {
      if (c_it >= n_items) return;
      uint32_t c, mt, v0;
      decode(c_it, c, mt, v0);
      c_off = a.cell_off[c];
      c_nd = a.cell_off[c + 1] - c_off;
      c_nk = (c_nd + KC - 1) / KC;
      c_v = v0 + v;
    };
    auto cursor_step = [&](uint32_t n) {
      while (n-- && c_it < n_items)
        if (++c_kc == c_nk) {
          c_kc = 0;
          c_it += step;
          cursor_item();
        }
    };
    uint32_t id[8], idv = 0;
    auto load_ids = [&]() {
      const bool on = c_it < n_items && c_v < m;
      idv = c_v;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const uint32_t k = c_kc * KC + kb * 8 + kk;
        id[kk] = on && k < c_nd ? a.ids[c_off + k] : 0xffffffffu;
      }
    };
    auto load_x = [&](double(&x)[8]) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        x[kk] = id[kk] != 0xffffffffu ? __ldg(a.X + (uint64_t)id[kk] * m + idv) : 0.0;
    };
    // epilogue of item number li (single TMEM buffer): warp w reads TMEM lanes of
    // quadrant w % 4 and OZ_ECOLS columns from OZ_ECOLS (w / 4), OZ_EPI_COLS at a
    // time, staged through its scratch tile into row segments
    auto epilogue = [&](uint32_t li, uint32_t it) -> bool {
      uint32_t c, mt, v0;
      decode(it, c, mt, v0);
      const uint32_t off = a.cell_off[c], nd = a.cell_off[c + 1] - off;
      const uint32_t quad = warp % 4, col0 = warp / 4 * OZ_ECOLS;
      const uint32_t row = mt * 128 + quad * 32 + lane;
      const int er = row < nd ? a.row_exp[off + row] : 0;
      const uint32_t ve = v0 + col0 + lane;
      const int xe = lane < OZ_ECOLS && ve < m ? a.x_exp[ve] : 0;  // lane l: exponent of column col0 + l
      if (!__all_sync(0xffffffffu, wait(tfull, li & 1, 26))) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      double *scr = epi_scratch + warp * OZ_EPI_DOUBLES;
#pragma unroll 1
      for (uint32_t cg = 0; cg < OZ_ECOLS; cg += OZ_EPI_COLS) {
        oz::CarrySum t[OZ_EPI_COLS];
        const uint32_t ta = tmem + ((quad * 32) << 16) + col0 + cg;
        // (four accumulators at a time: all eight at once spill)
        uint32_t L[4][OZ_EPI_COLS];
        auto load = [&](int a0, int a1, int a2, int a3) {
          oz::tmem_issue(ta + a0 * OZ_N, L[0]);
          oz::tmem_issue(ta + a1 * OZ_N, L[1]);
          oz::tmem_issue(ta + a2 * OZ_N, L[2]);
          oz::tmem_issue(ta + a3 * OZ_N, L[3]);
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int j = 0; j < OZ_EPI_COLS; ++j) tmem_landed(L[g][j]);
        };
        load(6, 5, 4, OZ_ACC_L6B);
        oz::carry_levels<6>(t, L[0]);
        oz::carry_levels<5>(t, L[1]);
        oz::carry_level4_parts(t, L[2], L[3]);
        load(3, 2, 1, 0);
        oz::carry_levels<3>(t, L[0]);
        oz::carry_levels<2>(t, L[1]);
        oz::carry_levels<1>(t, L[2]);
        double y[OZ_EPI_COLS];
        int sc[OZ_EPI_COLS];
        bool plain = true;
#pragma unroll
        for (int j = 0; j < OZ_EPI_COLS; ++j) {
          y[j] = oz::carry_finish(t[j], __uint_as_float(L[3][j]));
          sc[j] = er + __shfl_sync(0xffffffffu, xe, cg + j) - 62;
          const int e = (__double2hiint(y[j]) >> 20) & 0x7ff;
          plain = plain && (e == 0 || (e + sc[j] > 0 && e + sc[j] < 0x7ff));
        }
#pragma unroll
        for (int j = 0; j < OZ_EPI_COLS; ++j) {
          double r = y[j];
          if (!plain)
            r = oz::ldexp_outlined(r, sc[j]);
          else if ((__double2hiint(r) & 0x7ff00000) != 0)  // the exponent moves, zero stays
            r = __hiloint2double(__double2hiint(r) + (sc[j] << 20), __double2loint(r));
          scr[lane * OZ_EPI_COLS + (j ^ (lane & (OZ_EPI_COLS - 1)))] = r;
        }
        __syncwarp();
        const uint32_t j = lane % OZ_EPI_COLS, vc = v0 + col0 + cg + j;
#pragma unroll
        for (uint32_t i = 0; i < OZ_EPI_COLS; ++i) {
          const uint32_t r = (32 / OZ_EPI_COLS) * i + lane / OZ_EPI_COLS, orow = mt * 128 + quad * 32 + r;
          if (orow < nd && vc < m)
            a.Yc[(uint64_t)(off + orow) * m + vc] = scr[r * OZ_EPI_COLS + (j ^ (r & (OZ_EPI_COLS - 1)))];
        }
        __syncwarp();
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty);
      return true;
    };
    uint32_t q = 0, li = 0, prev_it = 0;
    bool ok = true;
    double xcur[8], xnxt[8];
    cursor_item();
    cursor_step(grp);
    load_ids();
    load_x(xcur);
    cursor_step(OZ_GROUPS);
    load_ids();
    for (uint32_t it = first; it < n_items && ok; it += step, ++li) {
      uint32_t c, mt, v0;
      decode(it, c, mt, v0);
      const uint32_t nd = a.cell_off[c + 1] - a.cell_off[c];
      const uint32_t nk = (nd + KC - 1) / KC;
      const int ex = (v0 + v) < m ? a.x_exp[v0 + v] : 0;
      // the previous item's epilogue runs once this item's first chunks fill the
      // B ring: the next MMAs start the moment TMEM is free.  (A later chunk could
      // not be cut before it: its stage waits for MMAs that wait for the epilogue.)
      const uint32_t lag = min((uint32_t)OZ_BST, nk) - 1;
      for (uint32_t kc = 0; kc < nk && ok; ++kc, ++q) {
        if (q % OZ_GROUPS == grp) {
          const uint32_t s = q % OZ_BST;
          load_x(xnxt);
          cursor_step(OZ_GROUPS);
          load_ids();
          uint32_t packed[OZ_S][4];
#pragma unroll
          for (int kk = 0; kk < 8; kk += 2) {
            uint32_t pp[OZ_S];
            oz::digits7_pair_bf16(xcur[kk], xcur[kk + 1], ex, pp);
#pragma unroll
            for (int sl = 0; sl < OZ_S; ++sl) packed[sl][kk / 2] = pp[sl];
          }
          if (q >= OZ_BST) {
            ok = __all_sync(0xffffffffu, wait(&empty_b[s], ((q / OZ_BST) - 1) & 1, 25));
            if (!ok) break;
          }
          uint8_t *Bst = bring + s * OZ_B_STAGE + (v / 8) * SBO + kb * LBO + (v % 8) * 16;
#pragma unroll
          for (int sl = 0; sl < OZ_S; ++sl)
            *(uint4 *)(Bst + sl * OZ_B_PART) = make_uint4(packed[sl][0], packed[sl][1], packed[sl][2], packed[sl][3]);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) mbar_arrive(&full_b[s]);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) xcur[kk] = xnxt[kk];
        }
        if (kc == lag && li >= 1) ok = epilogue(li - 1, prev_it);
      }
      prev_it = it;
    }
    if (ok && li >= 1) epilogue(li - 1, prev_it);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == OZ_MMA_WARP) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols) : "memory");
  }
}

}  // namespace

namespace gbfe {

bool oz_supported(const gbfe_mesh *me) { return me->nd_max <= 256; }

void build_oz_mats(gbfe_op *op) {
  gbfe_mesh *me = op->mesh;
  gbfe_ctx *ctx = me->ctx;
  std::vector<uint64_t> aoff(me->n_cells + 1, 0);
  for (uint32_t c = 0; c < me->n_cells; ++c) {
    const uint64_t nd = me->h_nd[c];
    const uint64_t mt8 = (nd + 7) / 8 * 8, nk = (nd + KC - 1) / KC;
    aoff[c + 1] = aoff[c] + nk * OZ_S * mt8 * KC;
  }
  op->oz_aoff.upload(aoff.data(), aoff.size(), ctx->stream);
  op->oz_mats.alloc(aoff.back());
  op->oz_row_exp.alloc(me->total_cell_dofs);
  k_build_oz_mats<<<me->n_cells, 128, 0, ctx->stream>>>(op->mats.p, op_mat_off(op), me->cell_off.p, op->oz_aoff.p,
                                                        me->n_cells, op->oz_mats.p, op->oz_row_exp.p);
  check_launch(ctx, "build_oz_mats");
}

// Yc (FP64 cell-wise buffer) = FP64-accurate sliced tensor-core products
// per-column exponents of X into op's buffer (context stream)
const int *oz_column_exponents(const gbfe_op *op, const gbfe_mv *X) {
  gbfe_mesh *me = op->mesh;
  gbfe_ctx *ctx = me->ctx;
  const uint32_t m = X->m;
  const uint64_t rows = me->n_dofs;
  const unsigned nb = (unsigned)std::min<uint64_t>(8 * (uint64_t)ctx->sm_count, std::max<uint64_t>(1, rows));
  ctx->oz_ipart.ensure((size_t)nb * m);
  op->oz_xexp.ensure(m);
  pdl_launch(ctx, k_colmax_partial, nb, oz::COLMAX_THREADS, 0, ctx->stream, X->d.p, rows, m, ctx->oz_ipart.p);
  pdl_launch(ctx, k_colmax_final, (m + 31) / 32, oz::COLMAX_FINAL_THREADS, 0, ctx->stream, ctx->oz_ipart.p, nb, m,
             op->oz_xexp.p);
  count_launch(ctx, 2);
  return op->oz_xexp.p;
}

void cell_apply_oz(const gbfe_op *op, const gbfe_mv *X, double *Yc, const int *xexp, cudaStream_t stream) {
  gbfe_mesh *me = op->mesh;
  gbfe_ctx *ctx = me->ctx;
  const uint32_t m = X->m;
  if (!stream) stream = ctx->stream;
  if (!xexp) xexp = oz_column_exponents(op, X);
  const uint32_t vt = (m + OZ_N - 1) / OZ_N;
  const uint32_t smem = OZ_SMEM;
  static PerDeviceOnce attr_once;
  attr_once.run(ctx->device, [&] {
    GBFE_CUDA(cudaFuncSetAttribute(k_cell_apply_oz, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  });
  for (uint32_t mts = 1; mts <= 2; ++mts) {
    uint32_t b0 = UINT32_MAX, b1 = 0;
    for (uint32_t b = 0; b < me->bin_nd.size(); ++b)
      if ((me->bin_nd[b] + 127) / 128 == mts) {
        b0 = std::min(b0, b);
        b1 = b + 1;
      }
    if (b0 == UINT32_MAX) continue;
    const uint32_t cbeg = me->bin_begin[b0], ncell = me->bin_begin[b1] - cbeg;
    const uint32_t items = ncell * mts * vt;
    const uint32_t grid = std::min<uint32_t>(items, (uint32_t)ctx->sm_count);
    OzArgs args{X->d.p, m, me->ids.p, me->cell_off.p, me->bin_cells.p + cbeg, ncell, mts, vt, op->oz_aoff.p,
                op->oz_mats.p, op->oz_row_exp.p, xexp, Yc, 512, ctx->status.p};
    const double frac = (double)ncell / me->n_cells;
    ProfScope prof(ctx, "cell_apply_f64_oz", 2.0 * m * (double)me->total_mat * frac,
                   8.0 * (2.0 * (double)me->n_dofs * m + (double)me->total_mat) * frac);
    pdl_launch(ctx, k_cell_apply_oz, grid, OZ_THREADS, smem, stream, args);
    check_launch(ctx, "cell_apply_oz");
  }
}

}  // namespace gbfe
