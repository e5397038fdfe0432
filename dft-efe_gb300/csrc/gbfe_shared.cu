// gbfe_shared.cu -- FP64 cell product of ONE vector for operators whose cells
// share stored matrices (gbfe_cellmat_upload_indexed), the product inside a
// batched CG iteration.
//
// Cells that share a matrix turn their matrix-vector products into one
// contraction Y[j][c] = sum_k A(k, j) X[ids_c[k]] with the CELL as the column
// index, so the tensor cores can run it although there is one vector only.
// On the FP64 pipe (1.25 TFLOP/s on GB300) the product of 48,180 cells of 64
// and 125 dofs (1.15 GFLOP) takes 1,077 us of a 1.22 ms CG iteration, here 63 us
// on average over a solve (items of finished instances are skipped).
//
// Operands are cut into eight balanced base-256 digits (bf16 holds integers up
// to 256 exactly) of a 62-bit fixed-point number, per matrix row and per CELL:
//     a = 2^(ea+2) sum_s a_s 2^-8s,   x = 2^(ex+2) sum_t x_t 2^-8t,
// |first digit| <= 64, |others| <= 128.  The 36 digit products with s + t <= 9
// accumulate in eight FP32 level accumulators (s + t = 2 .. 9).  A level holds
// two products <= 2^13 and up to six <= 2^14 per row, so over K <= 128 rows
// every partial sum is an integer below 2^24: exact.  What is dropped (s + t >=
// 10) stays below 2^-59 of max|a| max|x| per row.  The epilogue adds the levels
// exactly and rounds ONCE to FP64 (an FMA chain rounds K times): measured
// against 80-bit sums over cells of 1 to 128 dofs the error is 3 to 7 times
// below the FMA product's, relative to sum |a||x| and to max|a| max|x|.
//
// Work item = up to 64 cells of one matrix (all its rows: at most 128).  Eight
// warps gather the item's X values into registers, find each cell's exponent
// and cut the digits chunk by chunk; the A digit tiles (shared by every item of
// the matrix: L2 hits) land by bulk copies; one thread issues the MMAs; eight
// warps run the epilogue while the next item's digits are cut.  TMEM lane =
// output row, so a warp's stores of one cell are 256 contiguous bytes.  An item
// takes 17 k clocks in the MMAs (waiting for 64 KB of A digits per 32 rows, 2 us
// after issue) and 17 - 25 k in the epilogue with four warps, which share the TMEM
// and so follow one another; the digit cut hides behind them.  A single epilogue
// warp per scheduler waits for its own chains (issue 21 %, ncu): two make the
// kernel 78 -> 63 us, although 96 registers a thread spill 52 bytes.
// Non-finite values: where a cell's X values or a matrix row hold an infinity or
// NaN, the results are summed from the operands as the FMA product does.
#include "gbfe_internal.cuh"
#include "gbfe_oz.cuh"
#include "gbfe_tc_ptx.cuh"

#include <algorithm>
#include <unordered_map>

using namespace gbfe;
using namespace gbfe::tc;

namespace {

constexpr int SS = 8;    // slices per operand
constexpr int SN = 64;   // cells per work item (8 levels x 64 = 512 TMEM columns)
constexpr int SST = 2;   // ring stages
constexpr int SGW = 8;   // gather warps
constexpr int S_TMA = SGW, S_MMA = SGW + 1;
constexpr int SEW = 8;   // epilogue warps, two per TMEM lane quadrant
constexpr int S_THREADS = (SGW + 2 + SEW) * 32;
constexpr int S_EXPBUF = 4;  // column exponents of the items in flight
constexpr int S_KCHUNKS = 4;  // K chunks a thread holds in registers: cells of up to 128 dofs
constexpr uint32_t S_ND_MAX = S_KCHUNKS * KC;
constexpr uint32_t S_A_PART = 128 * KC * 2, S_B_PART = SN * KC * 2;
constexpr uint32_t S_STAGE = SS * (S_A_PART + S_B_PART);
constexpr uint32_t S_SMEM = SST * S_STAGE + S_EXPBUF * 4 * SN * 4 + 1024 + 512;
static_assert(S_SMEM <= 227 * 1024, "shared-matrix product: shared memory");
constexpr int EXP_NONFINITE = 100000;  // a column / row holding an infinity or NaN

// exponent of |v| as oz::exp_bits, with non-finite values above every finite one
__device__ __forceinline__ int exp_or_nonfinite(double v) {
  const int E = (int)(((uint64_t)__double_as_longlong(v) >> 52) & 0x7ff);
  return E == 0 ? oz::EXP_NONE : E == 0x7ff ? EXP_NONFINITE : E - 1022;
}

// trunc(v 2^(62-e)) + 0x8080...: byte b of the sum is digit + 128, most
// significant byte first (|v| < 2^e, so the left shift of the 53-bit mantissa
// is at most 9)
__device__ __forceinline__ uint64_t biased_digits(double v, int e) {
  const uint64_t bits = (uint64_t)__double_as_longlong(v);
  const int ex = (int)((bits >> 52) & 0x7ff);
  const int r = e + 1022 - ex;
  const uint64_t m62 = ((bits & ((1ull << 52) - 1)) | (1ull << 52)) << 9;
  uint64_t fx = (ex == 0 || r > 63 || r < 0) ? 0 : m62 >> r;
  if (bits >> 63) fx = 0 - fx;
  return fx + 0x8080808080808080ull;
}

// sum_g L[g] 256^(6-g) (levels 2 .. 9 = L[0 .. 7]), rounded once to FP64, the
// part of the last level below half a unit of the level before dropped (integer
// sums and two FP64 adds took 344 clocks per warp, this takes 270)
__device__ __forceinline__ double levels_to_double(float (&L)[8]) {
  L[6] += fmaf(L[7], 0.00390625f, oz::CARRY_MAGIC) - oz::CARRY_MAGIC;
  oz::CarrySum t;
  oz::carry_level<6>(t, L[6]);
  oz::carry_level<5>(t, L[5]);
  oz::carry_level<4>(t, L[4]);
  oz::carry_level<3>(t, L[3]);
  oz::carry_level<2>(t, L[2]);
  oz::carry_level<1>(t, L[1]);
  return oz::carry_finish(t, L[0]);
}

// one entry of the product from its operands
__device__ __noinline__ double row_product(const double *A, const double *X, const uint32_t *ids, uint32_t nd) {
  double v = 0.0;
  for (uint32_t k = 0; k < nd; ++k) v = fma(A[k], X[ids[k * SN]], v);
  return v;
}

// digit of byte b (0 least significant) as a float in [-128, 127]
__device__ __forceinline__ float digit_float(uint32_t word, int byte) {
  const uint32_t sel = 0x7650u | (uint32_t)byte;  // {word.byte, 0, 0, 0x4B}
  return __uint_as_float(__byte_perm(word, 0x4B000000u, sel)) - 8388736.0f;  // 2^23 + 128
}

// the 8 slices of two consecutive K values as bf16 pairs (low half = first)
__device__ __forceinline__ void digit_pairs(double v0, double v1, int e, uint32_t (&p)[SS]) {
  const uint64_t u0 = biased_digits(v0, e), u1 = biased_digits(v1, e);
#pragma unroll
  for (int s = 0; s < SS; ++s) {
    const int b = 7 - s;  // byte index of slice s
    const uint32_t w0 = (uint32_t)(b >= 4 ? u0 >> 32 : u0), w1 = (uint32_t)(b >= 4 ? u1 >> 32 : u1);
    p[s] = __byte_perm(__float_as_uint(digit_float(w0, b & 3)), __float_as_uint(digit_float(w1, b & 3)), 0x7632);
  }
}

// digit tiles of the distinct matrices: per (matrix, K chunk) [slice][MT8 x KC]
// canonical K-major tiles of A_op[j][k] = A(k, j), and a row exponent per j
__global__ void k_build_shared(const double *__restrict__ mats, const uint64_t *__restrict__ moff,
                               const uint32_t *__restrict__ mnd, const uint64_t *__restrict__ aoff,
                               const uint32_t *__restrict__ roff, __nv_bfloat16 *__restrict__ out,
                               int *__restrict__ row_exp) {
  const uint32_t u = blockIdx.x, nd = mnd[u];
  const uint32_t mt8 = (nd + 7) / 8 * 8, nk = (nd + KC - 1) / KC;
  const double *A = mats + moff[u];
  int *re = row_exp + roff[u];
  for (uint32_t j = threadIdx.x; j < nd; j += blockDim.x) {
    int mx = oz::EXP_NONE;
    for (uint32_t k = 0; k < nd; ++k) mx = max(mx, exp_or_nonfinite(A[k + (uint64_t)nd * j]));
    re[j] = mx;
  }
  __syncthreads();
  const uint32_t per_slice = mt8 * KC;
  for (uint32_t idx = blockIdx.y * blockDim.x + threadIdx.x; idx < nk * per_slice; idx += blockDim.x * gridDim.y) {
    const uint32_t kc = idx / per_slice, rem = idx - kc * per_slice;
    const uint32_t r = rem / KC, kk = rem - r * KC, k = kc * KC + kk;
    uint64_t d = 0x8080808080808080ull;
    if (r < nd && k < nd) d = biased_digits(A[k + (uint64_t)nd * r], re[r]);
    const uint32_t pos = (r / 8) * (KC / 8) * 64 + (kk / 8) * 64 + (r % 8) * 8 + (kk % 8);
    __nv_bfloat16 *base = out + aoff[u] + (uint64_t)kc * SS * per_slice;
#pragma unroll
    for (int s = 0; s < SS; ++s)
      base[(uint64_t)s * per_slice + pos] = __int2bfloat16_rn((int)((d >> (8 * (7 - s))) & 255u) - 128);
  }
}

// ids of an item's cells with the cell index fastest ([k][SN]): the gather's
// id loads of a warp are then 128 contiguous bytes
__global__ void k_shared_ids(const gbfe_shared_item *__restrict__ items, const uint32_t *__restrict__ start,
                             const uint32_t *__restrict__ ids, uint32_t *__restrict__ out) {
  const gbfe_shared_item it = items[blockIdx.x];
  for (uint32_t t = threadIdx.x; t < it.nd * SN; t += blockDim.x) {
    const uint32_t v = t / it.nd, k = t - v * it.nd;
    out[it.ids_off + (uint64_t)k * SN + v] = v < it.n ? ids[start[it.first + v] + k] : 0u;
  }
}

struct SharedArgs {
  const double *X;
  const gbfe_shared_item *items;
  uint32_t n_items;
  const uint32_t *start, *idsT;  // first cell-wise row of each cell (item order); ids, cell-fastest
  const __nv_bfloat16 *dig;
  const int *row_exp;
  const double *mats;
  double *Yc;
  const int *active;         // per instance; nullptr: every item runs
  const uint32_t *item_inst;  // first and last instance of each item
  int *status;
};

__global__ void __launch_bounds__(S_THREADS, 1) k_cell_apply_shared(const SharedArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  int *cexp_buf = (int *)(smem + SST * S_STAGE);  // [S_EXPBUF][4][SN] partial column exponents
  uint64_t *bars = (uint64_t *)(cexp_buf + S_EXPBUF * 4 * SN);
  uint64_t *full_a = bars, *full_b = bars + SST, *empty = bars + 2 * SST;
  uint64_t *tfull = bars + 3 * SST, *tempty = tfull + 1, *cfull = tempty + 1, *erdy = cfull + 1;
  uint64_t *spare = erdy + 1;  // drain_mmas before TMEM is freed
  uint32_t *tmem_slot = (uint32_t *)(spare + 1);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const uint32_t tid = threadIdx.x, warp = tid / 32, lane = tid % 32;

  if (tid == 0) {
    for (int s = 0; s < SST; ++s) {
      mbar_init(&full_a[s], 1);
      mbar_init(&full_b[s], SGW);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, SEW);
    mbar_init(cfull, SGW);
    mbar_init(erdy, 1);
    mbar_init(spare, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == S_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_trigger();  // (after the allocation, see pdl_trigger)
  pdl_wait();
  auto wait = [&](uint64_t *bar, uint32_t parity, int code) -> bool {
    if (mbar_test(bar, parity)) return true;
    if (*abort_flag) return false;
    if (mbar_wait(bar, parity, a.status, code)) return true;
    *abort_flag = 1;
    return false;
  };
  // next item of this CTA at or after `it` with a running instance; every role
  // takes the same decision (`active` does not change during the launch)
  auto next = [&](uint32_t it) -> uint32_t {
    if (!a.active) return it;
    for (; it < a.n_items; it += gridDim.x) {
      const uint32_t i1 = a.item_inst[2 * it + 1];
      for (uint32_t i = a.item_inst[2 * it]; i <= i1; ++i)
        if (a.active[i]) return it;
    }
    return it;
  };

  if (warp == S_TMA) {
    if (lane == 0) {
      uint32_t q = 0;
      for (uint32_t it = next(blockIdx.x); it < a.n_items && !*abort_flag; it = next(it + gridDim.x)) {
        const gbfe_shared_item I = a.items[it];
        const uint32_t mt8 = (I.nd + 7) / 8 * 8, nk = (I.nd + KC - 1) / KC;
        for (uint32_t kc = 0; kc < nk; ++kc, ++q) {
          const uint32_t s = q % SST;
          if (q >= SST && !wait(&empty[s], ((q / SST) - 1) & 1, 61)) break;
          uint8_t *At = smem + s * S_STAGE;
          const uint32_t bytes = mt8 * KC * 2;
          mbar_arrive_expect_tx(&full_a[s], SS * bytes);
          for (int sl = 0; sl < SS; ++sl)
            bulk_g2s(At + sl * S_A_PART, a.dig + I.a_off + ((uint64_t)kc * SS + sl) * mt8 * KC, bytes, &full_a[s]);
        }
      }
      drain_copies(full_a, q, SST);
    }
    __syncwarp();
  } else if (warp == S_MMA) {
    if (lane == 0) {
      uint32_t q = 0, li = 0;
      for (uint32_t it = next(blockIdx.x); it < a.n_items && !*abort_flag; it = next(it + gridDim.x), ++li) {
        const uint32_t nk = (a.items[it].nd + KC - 1) / KC;
        if (li >= 1 && !wait(tempty, (li - 1) & 1, 62)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        bool ok = true;
        for (uint32_t kc = 0; kc < nk; ++kc, ++q) {
          const uint32_t s = q % SST;
          if (!mbar_test2(&full_a[s], (q / SST) & 1, &full_b[s], (q / SST) & 1) &&
              (!wait(&full_a[s], (q / SST) & 1, 63) || !wait(&full_b[s], (q / SST) & 1, 64))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t abase = smem_u32(smem + s * S_STAGE), bbase = abase + SS * S_A_PART;
          for (uint32_t ks = 0; ks < KC / 16; ++ks) {
            // slice sl of A against up to four stacked B slices (see k_cell_apply_oz)
#pragma unroll
            for (int sl = 1; sl <= SS; ++sl) {
#pragma unroll
              for (int t0 = 1; t0 <= SS + 1 - sl; t0 += 4) {
                const int t1 = t0 + 3 < SS + 1 - sl ? t0 + 3 : SS + 1 - sl;
                umma(tmem + (sl + t0 - 2) * SN, smem_desc(abase + (sl - 1) * S_A_PART + ks * 2 * LBO),
                     smem_desc(bbase + (t0 - 1) * S_B_PART + ks * 2 * LBO), instr_desc(128, SN * (t1 - t0 + 1)),
                     ((kc | ks) == 0 && sl == 1) ? 0u : 1u);
              }
            }
          }
          umma_commit(&empty[s]);
        }
        if (!ok) break;
        // the gather's exponents, seen through full_b, handed on to the epilogue
        mbar_arrive(erdy);
        umma_commit(tfull);
      }
      drain_mmas(spare);
    }
    __syncwarp();
  } else if (warp < SGW) {
    // gather: thread = (cell v of the item, K block kb of every chunk).  The
    // values of the whole item sit in registers; once a chunk's digits are cut
    // its registers take the next item's values, whose ids were loaded a chunk
    // earlier, so both latencies pass behind the cutting.
    const uint32_t kb = warp % 4, v = (warp / 4) * 32 + lane;
    double x[S_KCHUNKS][8];
    uint32_t idn[8];
    auto load_ids = [&](const gbfe_shared_item &I, int kc) {
      const uint32_t *id = a.idsT + I.ids_off + v;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const uint32_t k = kc * KC + kb * 8 + kk;
        idn[kk] = (v < I.n && k < I.nd) ? __ldg(id + (uint64_t)k * SN) : 0xffffffffu;
      }
    };
    auto load_x = [&](double(&xc)[8]) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) xc[kk] = idn[kk] != 0xffffffffu ? __ldg(a.X + idn[kk]) : 0.0;
    };
    uint32_t q = 0, li = 0;
    bool ok = true;
    uint32_t it = next(blockIdx.x);
    gbfe_shared_item I{};
    if (it < a.n_items) {
      I = a.items[it];
#pragma unroll
      for (int kc = 0; kc < S_KCHUNKS; ++kc) {
        load_ids(I, kc);
        load_x(x[kc]);
      }
    }
    while (it < a.n_items && ok) {
      const uint32_t nk = (I.nd + KC - 1) / KC;
      int mx = oz::EXP_NONE;
#pragma unroll
      for (int kc = 0; kc < S_KCHUNKS; ++kc)
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) mx = max(mx, exp_or_nonfinite(x[kc][kk]));
      // the buffer's last reader is the epilogue of item li - 4: the ring waits
      // below let this warp reach item li only after the MMAs of item li - 3
      // finished, and those started after that epilogue
      int *cexp = cexp_buf + (li % S_EXPBUF) * 4 * SN;
      cexp[kb * SN + v] = mx;
      __syncwarp();
      if (lane == 0) mbar_arrive(cfull);
      const uint32_t nit = next(it + gridDim.x);
      gbfe_shared_item J{};  // nd = n = 0 past the last item: zeros are loaded
      if (nit < a.n_items) J = a.items[nit];
      load_ids(J, 0);
      ok = __all_sync(0xffffffffu, wait(cfull, li & 1, 67));
      if (!ok) break;
      const int ex = oz::exp_or_zero(max(max(cexp[v], cexp[SN + v]), max(cexp[2 * SN + v], cexp[3 * SN + v])));
#pragma unroll
      for (int kc = 0; kc < S_KCHUNKS; ++kc) {
        if ((uint32_t)kc < nk && ok) {
          const uint32_t s = q % SST;
          uint32_t packed[SS][4];
#pragma unroll
          for (int kk = 0; kk < 8; kk += 2) {
            uint32_t pp[SS];
            digit_pairs(x[kc][kk], x[kc][kk + 1], ex, pp);
#pragma unroll
            for (int sl = 0; sl < SS; ++sl) packed[sl][kk / 2] = pp[sl];
          }
          if (q >= SST) ok = __all_sync(0xffffffffu, wait(&empty[s], ((q / SST) - 1) & 1, 65));
          if (ok) {
            uint8_t *Bst = smem + s * S_STAGE + SS * S_A_PART + (v / 8) * SBO + kb * LBO + (v % 8) * 16;
#pragma unroll
            for (int sl = 0; sl < SS; ++sl)
              *(uint4 *)(Bst + sl * S_B_PART) = make_uint4(packed[sl][0], packed[sl][1], packed[sl][2], packed[sl][3]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_b[s]);
            ++q;
          }
        }
        load_x(x[kc]);
        if (kc + 1 < S_KCHUNKS) load_ids(J, kc + 1);
      }
      it = nit;
      I = J;
      ++li;
    }
  } else {
    // epilogue: the two warps of a quadrant turn alternate groups of eight columns of
    // the item's levels into FP64 rows
    const uint32_t quad = warp % 4, row = quad * 32 + lane, half = (warp - SGW - 2) / 4;
    uint32_t li = 0;
    bool ok = true;
    for (uint32_t it = next(blockIdx.x); it < a.n_items && ok; it = next(it + gridDim.x), ++li) {
      const gbfe_shared_item I = a.items[it];
      const int er = row < I.nd ? oz::exp_or_zero(a.row_exp[I.row_off + row]) : 0;
      // lane l holds the first row and the exponent of cells l and l + 32
      uint32_t st[2];
      int ecs[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) st[h] = h * 32 + lane < I.n ? a.start[I.first + h * 32 + lane] : 0u;
      ok = __all_sync(0xffffffffu, wait(erdy, li & 1, 68)) && __all_sync(0xffffffffu, wait(tfull, li & 1, 66));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int *cexp = cexp_buf + (li % S_EXPBUF) * 4 * SN + lane;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        ecs[h] = oz::exp_or_zero(
            max(max(cexp[h * 32], cexp[h * 32 + SN]), max(cexp[h * 32 + 2 * SN], cexp[h * 32 + 3 * SN])));
      if (quad * 32 < I.nd) {  // a quadrant past the cell's rows has nothing to store
#pragma unroll 1
        for (uint32_t col = half * 8; col < I.n; col += SEW / 4 * 8) {
          const uint32_t ta = tmem + ((quad * 32) << 16) + col;
          uint32_t t[8][8];
#pragma unroll
          for (int g = 0; g < 8; ++g) tmem_ld8_issue(ta + g * SN, t[g]);
          tmem_wait_ld();
          // (no branch between the columns: eight independent chains hide the
          // FP64 adds' 64-clock issue and their latency)
          double y[8];
          int sc[8];
          bool plain = true;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float L[8];
#pragma unroll
            for (int g = 0; g < 8; ++g) {
              tmem_landed(t[g][j]);
              L[g] = __uint_as_float(t[g][j]);
            }
            y[j] = levels_to_double(L);
            const int ec = __shfl_sync(0xffffffffu, col < 32 ? ecs[0] : ecs[1], (col + j) % 32);
            sc[j] = er + ec - 60;
            const int e = (__double2hiint(y[j]) >> 20) & 0x7ff;
            plain = plain && (e == 0 ? sc[j] < EXP_NONFINITE / 2 : e + sc[j] > 0 && e + sc[j] < 0x7ff);
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t out0 = __shfl_sync(0xffffffffu, col < 32 ? st[0] : st[1], (col + j) % 32);
            double v = y[j];
            if (plain)  // exact: the exponent moves, zero stays
              v = (__double2hiint(v) & 0x7ff00000) == 0
                      ? v
                      : __hiloint2double(__double2hiint(v) + (sc[j] << 20), __double2loint(v));
            else if (sc[j] < EXP_NONFINITE / 2)  // the result leaves the normal range
              v = oz::ldexp_outlined(v, sc[j]);
            else if (row < I.nd && col + j < I.n)
              v = row_product(a.mats + I.m_off + (uint64_t)row * I.nd, a.X, a.idsT + I.ids_off + col + j, I.nd);
            if (row < I.nd && col + j < I.n) a.Yc[(uint64_t)out0 + row] = v;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == S_MMA) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

}  // namespace

namespace gbfe {

// Cells of the instances that take this product.  An instance is judged by its own
// cells, so that its results do not depend on what else is in the batch (a cell's
// results depend on neither the item nor the columns beside it):
//   * its cells have at most 128 dofs (their X values fit a thread's registers);
//   * their matrices, expanded, have at least SHARED_MIN entries: a line between what
//     a small instance costs alone and in a batch.  Alone, us an iteration, FMA kernel /
//     items: 1.4 M entries 24.5 / 33.7, 2.1 M 25.8 / 33.5, 3.4 M 30.7 / 36.6, 5.4 M 35.6 /
//     36.8; beside larger instances, which run the items anyway, a batch of 24 (6^3 to
//     18^3 cells) takes 53.3, 55.2, 58 ms with the line at 0.8, 2 and 4 M;
//   * items of its cells alone would be at least a quarter full (a matrix named by
//     fewer than 16 cells leaves most of an item's columns empty).
constexpr uint64_t SHARED_MIN = 2000000;
static std::vector<uint8_t> shared_cells(const gbfe_op *op, uint32_t n_inst, const std::vector<uint32_t> &cell_inst) {
  const gbfe_mesh *me = op->mesh;
  const std::vector<uint64_t> &moff = op->h_mat_off_own;
  std::vector<uint64_t> entries(n_inst, 0), slots(n_inst, 0), cells(n_inst, 0);
  std::vector<uint8_t> small(n_inst, 1), out(me->n_cells);
  std::unordered_map<uint64_t, uint32_t> last;  // (matrix, instance) -> cells of the item that is being filled
  uint64_t key0 = 0;
  uint32_t *fill = nullptr;  // (neighbouring cells mostly share both)
  for (uint32_t c = 0; c < me->n_cells; ++c) {
    const uint32_t i = cell_inst[c], nd = me->h_nd[c];
    entries[i] += (uint64_t)nd * nd;
    ++cells[i];
    small[i] &= nd <= S_ND_MAX;
    const uint64_t key = moff[c] * n_inst + i;
    if (!fill || key != key0) fill = &last[key];
    key0 = key;
    if (*fill == 0) slots[i] += SN;
    *fill = (*fill + 1) % SN;
  }
  for (uint32_t c = 0; c < me->n_cells; ++c) {
    const uint32_t i = cell_inst[c];
    out[c] = small[i] && entries[i] >= SHARED_MIN && slots[i] <= 4 * cells[i];
  }
  return out;
}

// digit tiles and work items for the cells flagged in `in`, the list of the others
static std::unique_ptr<gbfe_shared> build_shared_plan(const gbfe_op *op, std::vector<uint8_t> in) {
  gbfe_mesh *me = op->mesh;
  gbfe_ctx *ctx = me->ctx;
  auto plan = std::make_unique<gbfe_shared>();
  // cells by matrix (equal offsets = one matrix), largest matrices first so
  // that the short items fill the last wave
  std::vector<uint32_t> &cells = plan->h_cells;
  for (uint32_t c = 0; c < me->n_cells; ++c) (in[c] ? cells : plan->h_rest).push_back(c);
  const std::vector<uint64_t> &moff = op->h_mat_off_own;
  std::sort(cells.begin(), cells.end(), [&](uint32_t x, uint32_t y) {
    return std::make_tuple(~me->h_nd[x], moff[x], x) < std::make_tuple(~me->h_nd[y], moff[y], y);
  });
  std::vector<gbfe_shared_item> &items = plan->h_items;
  std::vector<uint64_t> mo, ao;
  std::vector<uint32_t> mnd, ro;
  uint64_t a_len = 0, ids_len = 0;
  uint32_t r_len = 0;
  const uint32_t n = (uint32_t)cells.size();
  for (uint32_t i = 0; i < n;) {
    const uint64_t off = moff[cells[i]];
    const uint32_t nd = me->h_nd[cells[i]];
    mo.push_back(off);
    mnd.push_back(nd);
    ao.push_back(a_len);
    ro.push_back(r_len);
    uint32_t e = i;
    while (e < n && moff[cells[e]] == off && me->h_nd[cells[e]] == nd) ++e;
    for (; i < e; i += SN) {
      items.push_back(gbfe_shared_item{ids_len, a_len, off, i, std::min<uint32_t>(SN, e - i), nd, r_len});
      ids_len += (uint64_t)nd * SN;
    }
    i = e;
    a_len += (uint64_t)((nd + KC - 1) / KC) * SS * ((nd + 7) / 8 * 8) * KC;
    r_len += nd;
  }
  GBFE_CUDA(cudaFuncSetAttribute(k_cell_apply_shared, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S_SMEM));
  plan->items.upload(items.data(), items.size(), ctx->stream);
  std::vector<uint32_t> start(n);
  for (uint32_t i = 0; i < n; ++i) start[i] = me->h_cell_off[cells[i]];
  plan->start.upload(start.data(), n, ctx->stream);
  if (!plan->h_rest.empty()) plan->rest.upload(plan->h_rest.data(), plan->h_rest.size(), ctx->stream);
  plan->dig.alloc(a_len);
  plan->row_exp.alloc(r_len);
  plan->ids.alloc(ids_len);
  DBuf<uint64_t> d_mo, d_ao;
  DBuf<uint32_t> d_nd, d_ro;
  d_mo.upload(mo.data(), mo.size(), ctx->stream);
  d_ao.upload(ao.data(), ao.size(), ctx->stream);
  d_nd.upload(mnd.data(), mnd.size(), ctx->stream);
  d_ro.upload(ro.data(), ro.size(), ctx->stream);
  k_build_shared<<<(unsigned)mo.size(), 256, 0, ctx->stream>>>(op->mats.p, d_mo.p, d_nd.p, d_ao.p, d_ro.p,
                                                               plan->dig.p, plan->row_exp.p);
  check_launch(ctx, "build_shared");
  k_shared_ids<<<(unsigned)items.size(), 256, 0, ctx->stream>>>(plan->items.p, plan->start.p, me->ids.p, plan->ids.p);
  check_launch(ctx, "shared_ids");
  GBFE_CUDA(cudaStreamSynchronize(ctx->stream));  // the host tables above go away
  plan->in_items = std::move(in);
  return plan;
}

// Plan of the one-vector product for a batch of instances (an instance's cells have
// their dofs in [inst_dof_off[i], inst_dof_off[i + 1])), and the instances of its items
// and of the cells beside them; nullptr: no instance takes it.  The plan stays on the
// operator and is laid out again when a call selects other cells.
const gbfe_shared *shared_plan(const gbfe_op *op, uint32_t n_inst, const uint64_t *inst_dof_off, SharedInst &inst) {
  gbfe_mesh *me = op->mesh;
  gbfe_ctx *ctx = me->ctx;
  if (op->kind != OP_CELL || op->h_mat_off_own.empty() || me->nd_min > S_ND_MAX || me->total_mat < SHARED_MIN)
    return nullptr;
  std::vector<uint32_t> cell_inst(me->n_cells);
  uint32_t i = 0;
  for (uint32_t c = 0; c < me->n_cells; ++c) {
    const uint64_t d = me->h_first[c];
    if (d < inst_dof_off[i] || d >= inst_dof_off[i + 1])
      i = (uint32_t)(std::upper_bound(inst_dof_off, inst_dof_off + n_inst + 1, d) - inst_dof_off) - 1;
    cell_inst[c] = i;
  }
  std::vector<uint8_t> in = shared_cells(op, n_inst, cell_inst);
  const size_t rest = std::count(in.begin(), in.end(), 0);
  // the cells beside the items take the FMA kernel for lists of cells; where that is not
  // the product they have alone (very large cells, sliced FP64 products), all of them do
  if (rest == in.size() || (rest && (me->nd_max > F64_LIST_ND_MAX || (ctx->fp64_tc && op->oz_aoff.p)))) return nullptr;
  if (!op->shared || op->shared->in_items != in) {
    op->shared.reset();
    op->shared = build_shared_plan(op, std::move(in));
  }
  const gbfe_shared &P = *op->shared;
  std::vector<uint32_t> h(2 * P.h_items.size());
  for (size_t t = 0; t < P.h_items.size(); ++t) {
    const gbfe_shared_item &I = P.h_items[t];
    uint32_t lo = UINT32_MAX, hi = 0;
    for (uint32_t v = 0; v < I.n; ++v) {
      const uint32_t k = cell_inst[P.h_cells[I.first + v]];
      lo = std::min(lo, k);
      hi = std::max(hi, k);
    }
    h[2 * t] = lo;
    h[2 * t + 1] = hi;
  }
  std::vector<uint32_t> r(rest);
  for (size_t t = 0; t < rest; ++t) r[t] = cell_inst[P.h_rest[t]];
  inst.item.upload(h.data(), h.size(), ctx->stream);
  if (rest) inst.rest.upload(r.data(), rest, ctx->stream);
  GBFE_CUDA(cudaStreamSynchronize(ctx->stream));  // (h and r go away)
  return op->shared.get();
}

// Yc (cell-wise) = A_c x_c for one FP64 vector, the items and then the cells beside
// them; with `active` (per instance) the items whose instances are all done, and the
// cells of such instances, are skipped and their rows of Yc keep what they held
void cell_apply_shared(const gbfe_op *op, const gbfe_shared &P, const double *x, double *Yc, const int *active,
                       const SharedInst &inst) {
  gbfe_ctx *ctx = op->mesh->ctx;
  const uint32_t n = (uint32_t)P.h_items.size();
  SharedArgs args{x,           P.items.p,  n,  P.start.p, P.ids.p,     P.dig.p,
                  P.row_exp.p, op->mats.p, Yc, active,    inst.item.p, ctx->status.p};
  pdl_launch(ctx, k_cell_apply_shared, std::min<uint32_t>(n, (uint32_t)ctx->sm_count), S_THREADS, S_SMEM, ctx->stream,
             args);
  check_launch(ctx, "cell_apply_shared");
  // (on a stream beside the items': batch of 24 instances 59.8 ms, here 59.2)
  if (!P.h_rest.empty())
    cell_apply_f64_list(op, x, Yc, P.rest.p, (uint32_t)P.h_rest.size(), active, inst.rest.p);
}

}  // namespace gbfe
