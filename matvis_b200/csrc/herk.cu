// A7: V = conj(Z) Z^T on the 5th-generation tensor cores (tcgen05 + TMEM),
// upper-triangle tiles only, in split precision.
//
// Reference: gpu/matprod.py:31-36 / gpu/_cublas.py:7-65 (one full c/zgemm with
// OP_C, OP_N per time and chunk), cpu/matprod.py:11-32 (z.conj().dot(z.T)),
// core/matprod.py:103-115 (sum over source chunks).
//
// Formulation.  For rows m, n of Z (row = ant * nfeed + feed):
//   Re V[m, n] = sum_k Zr[m,k] Zr[n,k] + Zi[m,k] Zi[n,k]
//   Im V[m, n] = sum_k Zr[m,k] Zi[n,k] - Zi[m,k] Zr[n,k]
// A 128 x 128 complex tile (I, J), I <= J, lives in one 128 x 256 FP32 TMEM
// block D (columns 0..127 real, 128..255 imaginary) filled by three UMMAs per
// k-step and split-term product (pa, pb), issued in this order:
//   D[:,   0:128] += Zi_I^pa . Zi_J^pb^T                  (N = 128)
//   D[:, 128:256] += Zi_I^pa . (-Zr_J^pb)^T               (N = 128, negate-B bit)
//   D[:,   0:256] += Zr_I^pa . [Zr_J^pb ; Zi_J^pb]^T     (N = 256)
// (with the N = 256 product first the whole-slice error measured 3.6e-7
// against 3.0e-7 at the same speed).  A diagonal tile (I = J) drops the
// Zr_I . Zi_I^T half of the last UMMA (N = 128, real half only): its
// imaginary half then holds W = -sum Zi^pa Zr^pb^T, and since the split-term
// products are symmetric under pa <-> pb, Im V = W - W^T, which the reduction
// forms from the partial tile's two triangles.  Three of the four real
// 128 x 128 products on 6 of the 21 tiles of a 700-row panel: 7 % fewer
// tensor-core cycles per slice.
// Where the caller states the live rows and at most 96 (64) of the last block's 128
// are, that block's tiles have 96 (64) columns: less to read, multiply and store, the
// same sums in the same order (700 x 196,608, eight panels: job 10.96 -> 10.72 ms, of
// which lower power is part; 90 rows of one block: 1,095 -> 1,088 us; 74: 287 -> 285).
//
// Accuracy.  The tensor core rounds its FP32 accumulator toward zero at every
// UMMA, so a long in-TMEM sum drifts by about one ulp per instruction (3e-5
// relative after 2,048 columns).  Each group of KD k-steps (32-byte column
// blocks; KD = 2 by default, one stage) is therefore accumulated into a FRESH
// TMEM block, products in ascending order of magnitude -- BF16_6 {11, 02, 20, 01,
// 10, 00}, BF16_3 / TF32_3 / F16_3 {01, 10, 00}, each product over all the
// block's k-steps before the next -- so only the final hi x hi UMMAs round at
// full magnitude, and the block is drained by the epilogue warps into FP32
// registers with round-to-nearest adds.  (Issuing the cross terms of both
// k-steps of a stage before its hi x hi products, instead of k-step by k-step,
// measured 3.6e-7 against 5.0e-7 on a whole config-2 slice and a 4 % shorter
// product.)  One
// k-slice (k_chunk columns) of register sums is one partial tile; slices are
// summed in float-float (TwoSum, ~2^-44) and rounded to FP64 by herk_reduce_*.
//
// Schedule.  Work unit u = (panel g, k-slice s, tile t), t fastest so the CTAs
// that run together read the same Z columns (L2 reuse).  A launch covers ngroup
// panels of one shape (the frequencies of a time step, zstride bytes apart)
// that share the column count; with ngroup = 1 it is one product.
// Persistent CTAs (one per SM, 192 KB of shared memory) take units in index
// order from a counter in the workspace (0 at each launch), after a
// first one of their own index, so a CTA that drew cheaper diagonal tiles takes more units: with
// static round-robin the CTAs' loads differed by up to a tile's work (one
// panel of 700 rows: 0.92-0.96 of the mean).  Each unit's sums do not depend
// on which CTA computes it.  Warp roles (576 threads):
//   warp 0 lane 0 : producer; fetches the CTA's next unit index and hands it
//                   to the other roles through a 4-entry shared-memory ring
//                   (full / empty mbarriers); one 1-D bulk copy per operand
//                   per stage: the panel stores each (k-block, row block) as
//                   the stage's shared-memory image (all 2P split/component
//                   planes of 128 rows x 64 bytes, 64-byte swizzled; two
//                   k-steps), so an operand is one contiguous 2P x 8 KB run.  A bulk copy of it
//                   completes in about half the time of the same bytes as tiled
//                   TMA boxes of 64-byte rows, and the three stages in flight no
//                   longer leave the MMA waiting;
//   warp 1        : TMEM owner (512 columns = two k-step blocks); one lane issues
//                   the UMMAs and tcgen05.commit's the stage / block barriers;
//   warps 2..17   : epilogue; warp w drains TMEM lane quadrant (w % 4), column
//                   quarter (w - 2) / 4 (64 of the 256 columns), 64 FP32
//                   register sums per thread, and at the end of a unit stores
//                   them coalesced to the workspace [u][256 columns][128 rows].
// K_valid is cut into equal k-slices (multiples of 64 columns, at most k_chunk)
// whose number is chosen on the device, from the device-side source count, to
// fill whole waves of SMs (plan_splits).
// Every mbarrier wait is bounded by wall time (wait_ns, 4 s unless
// mvb_set_wait_limit_ns changed it); on expiry the CTA records MVB_DEV_TIMEOUT
// in the status word, stops issuing work, drains the copies and MMAs it issued
// (each drain wait bounded by kDrainLimitNs), frees TMEM and returns.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace mvb {

constexpr int kEpiWarps = 16;
constexpr int kPlanExtra = 31;  // extra k-slices the split planner may add to fill the SMs (one per lane)
constexpr int kHerkThreads = 64 + 32 * kEpiWarps;
constexpr uint64_t kWaitLimitNs = 4000000000ull;   // 4 s: the default limit of a pipeline wait
constexpr uint64_t kDrainLimitNs = 200000000ull;   // 0.2 s
constexpr int kPlaneBytes = 128 * 64;              // one 128-row x 64-byte plane tile (two k-steps)
constexpr int kSmemBudget = 192 * 1024;
constexpr int kUnitRing = 4;       // unit indices the producer may fetch ahead of the MMA and epilogue
constexpr size_t kCounterBytes = 256;  // the launch's unit counter, in the last 16 bytes of the workspace

template <int MODE>
struct HerkCfg {
  static constexpr int P = MODE == MVB_GEMM_BF16_6 ? 3 : 2;
  static constexpr int ES = MODE == MVB_GEMM_TF32_3 ? 4 : 2;
  static constexpr int KSTEP = 32 / ES;  // elements per 32-byte k-step (= UMMA K)
  static constexpr int KB = 64 / ES;     // elements per 64-byte k-block: one stage, two k-steps
  static_assert(KB * ES == kKBlockBytes, "one stage is one k-block of the panel");
  static constexpr int OPER_BYTES = 2 * P * kPlaneBytes;
  static constexpr int STAGE_BYTES = 2 * OPER_BYTES;
  static constexpr int STAGES = kSmemBudget / STAGE_BYTES;
  static_assert(STAGES >= 2, "a drained block of four k-steps holds two stages");
  static constexpr int NPROD = P == 3 ? 6 : 3;
  // UMMA operand format: 0 = F16, 1 = BF16, 2 = TF32
  static constexpr uint32_t FMT = MODE == MVB_GEMM_TF32_3 ? 2u : (MODE == MVB_GEMM_F16_3 ? 0u : 1u);
  static constexpr uint32_t ID256 = umma_idesc(FMT, 256, 0);
  static constexpr uint32_t ID128 = umma_idesc(FMT, 128, 0);
  static constexpr uint32_t ID128N = umma_idesc(FMT, 128, 1);
};

// Split-term products (pa, pb), ascending magnitude 2^-8(pa + pb).
// Tables packed one nibble per product: 6 products pa = 1,0,2,0,1,0 and
// pb = 1,2,0,1,0,0; 3 products pa = 0,1,0 and pb = 1,0,0.
__device__ __forceinline__ void product_terms(int nprod, int q, uint32_t &pa, uint32_t &pb) {
  const uint32_t ta = nprod == 6 ? 0x010201u : 0x010u;
  const uint32_t tb = nprod == 6 ? 0x001021u : 0x001u;
  pa = (ta >> (4 * q)) & 0xFu;
  pb = (tb >> (4 * q)) & 0xFu;
}

// Splits K_valid into nsplit equal slices of kc columns (a multiple of 64, at
// most kmax), choosing nsplit in [ceil(K/kmax), +kPlanExtra] so that
// n_tiles * nsplit work units fill whole waves of nsm SMs as evenly as possible
// (a candidate replaces the best so far only when 1e-3 more efficient, so ties
// keep fewer slices; the scan stops at the first candidate of 64 columns).
// Each lane of a warp evaluates one candidate, and the scan jumps from one
// improvement to the next with a ballot, so every warp reaches the same plan in
// one candidate's arithmetic and a few votes; every lane of the warp must call it.
// Every count fits 32 bits (check_herk_shape).  Used identically by the product
// and its reductions.
__device__ __forceinline__ void plan_splits(int64_t kvalid, int n_tiles, int kmax, int nsm, int &nsplit, int64_t &kc) {
  if (kvalid <= 0) {  // kvalid is uniform over the grid
    nsplit = 0;
    kc = kmax;
    return;
  }
  const uint32_t kv = (uint32_t)kvalid, lane = threadIdx.x & 31;
  const uint32_t n = (kv + (uint32_t)kmax - 1) / (uint32_t)kmax + lane;
  const uint32_t c = ((kv + n - 1) / n + 63) / 64 * 64;
  const uint32_t ne = (kv + c - 1) / c;
  const uint32_t units = (uint32_t)n_tiles * ne;
  const uint32_t waves = (units + (uint32_t)nsm - 1) / (uint32_t)nsm;
  const double eff = (double)units / ((double)waves * (double)nsm);
  const unsigned stop = __ballot_sync(0xffffffffu, c <= 64);
  const unsigned allowed = stop ? 0xffffffffu >> (32 - __ffs(stop)) : 0xffffffffu;  // up to the first stop, inclusive
  int win = 0;
  double best = __shfl_sync(0xffffffffu, eff, 0);
  while (true) {
    const unsigned better = __ballot_sync(0xffffffffu, eff > best + 1e-3) & allowed & (0xfffffffeu << win);
    if (!better) break;
    win = __ffs(better) - 1;
    best = __shfl_sync(0xffffffffu, eff, win);
  }
  nsplit = (int)__shfl_sync(0xffffffffu, ne, win);
  kc = (int64_t)__shfl_sync(0xffffffffu, c, win);
}

// Valid K columns: (source count) x (columns per source), clamped to the panel.
__device__ __forceinline__ int64_t valid_k(const int32_t *n_dev, int64_t n_host, int kmul, int64_t Kcap) {
  int64_t n = n_dev ? (int64_t)__ldcg(n_dev) : n_host;
  n = n < 0 ? 0 : n;
  return min(n * kmul, Kcap);
}

__device__ __forceinline__ void decode_tile(int t, int T, int &I, int &J) {
  int i = 0;
  while (t >= T - i) {
    t -= T - i;
    ++i;
  }
  I = i;
  J = i + t;
}

template <int MODE>
__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if constexpr (MODE == MVB_GEMM_TF32_3)
    umma_tf32(d, a, b, idesc, acc);
  else
    umma_bf16(d, a, b, idesc, acc);
}

// One k-step of one split product into the block at d: the two products of the Zi
// rows first, so that the block's real and imaginary halves each start from Zi
// terms, then the Zr rows'.  A full off-diagonal tile takes Zr against [Zr; Zi] as
// one N = 256 instruction, a diagonal one only its real half (see the file's head).
// NC < 128: a tile of the last block column, NC columns live; off the diagonal
// Zr takes two instructions (the live rows of the two planes are not adjacent).  An
// instruction of N columns takes max(N / 2, 32 + N / 4) cycles (the operands' 4 KB +
// 32 N bytes at 128 bytes a cycle): 192 and 224 a k-step at 64 and 96 columns instead
// of 256.
template <int MODE, int NC>
__device__ __forceinline__ void umma_kstep(uint32_t d, uint64_t a_re, uint64_t a_im, uint64_t b_re, uint64_t b_im,
                                           uint32_t id_re, bool diag, uint32_t acc) {
  using C = HerkCfg<MODE>;
  if constexpr (NC == 128) {
    umma<MODE>(d, a_im, b_im, C::ID128, acc);
    umma<MODE>(d + 128, a_im, b_re, C::ID128N, acc);
    umma<MODE>(d, a_re, b_re, id_re, 1u);
  } else {
    constexpr uint32_t id = umma_idesc(C::FMT, NC, 0), id_neg = umma_idesc(C::FMT, NC, 1);
    umma<MODE>(d, a_im, b_im, id, acc);
    umma<MODE>(d + 128, a_im, b_re, id_neg, acc);
    umma<MODE>(d, a_re, b_re, id, 1u);
    if (!diag) umma<MODE>(d + 128, a_re, b_im, id, 1u);
  }
}

// A launch's work units come either from one panel shape repeated ngroup
// times (the frequencies of a job's time step), or from a table of panels of
// different shapes (the panel groups of several jobs, mvb_herk_batch).  A table
// entry is one panel: its k-slice plan fills waves for plan_tiles tiles and its
// partial tiles sit at index in its group's workspace, so that each group's
// sums equal those of its own grouped launch.
constexpr int kMaxBatchPanels = 32;
struct HerkPanel {
  const uint8_t *panel;
  const int32_t *n_dev;
  float *partials;  // the group's workspace
  int32_t *status;
  int64_t n_host, Kcap;
  int T, kmul, k_chunk, plan_tiles, index;
};
struct HerkTable {
  HerkPanel p[kMaxBatchPanels];
  int n;
};
struct NoTable {};  // a launch of one repeated shape does not carry the table's 2.6 KB of parameters

// KD: k-steps accumulated in one TMEM block before it is drained (1, 2 or 4).
// TABLE: the units come from the table (a batch) instead of one repeated shape.
// TAIL > 0: the last block is narrow, its first TAIL rows.
template <int MODE, int KD, bool TABLE, int TAIL>
__global__ void __launch_bounds__(kHerkThreads, 1)
    herk_kernel(const uint8_t *__restrict__ zpanels, int64_t zstride, int ngroup, int T, int n_tiles,
                const int32_t *__restrict__ n_dev, int64_t n_host, int kmul, int64_t Kcap, int k_chunk, int nsm,
                float *__restrict__ partials, int32_t *__restrict__ status, int *__restrict__ unit_next,
                uint64_t wait_ns, const __grid_constant__ std::conditional_t<TABLE, HerkTable, NoTable> table) {
  using C = HerkCfg<MODE>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[C::STAGES];
  __shared__ __align__(8) uint64_t empty_bar[C::STAGES];
  __shared__ __align__(8) uint64_t dfull_bar[2];
  __shared__ __align__(8) uint64_t dempty_bar[2];
  __shared__ __align__(8) uint64_t drain_bar;
  __shared__ __align__(8) uint64_t ufull_bar[kUnitRing];   // a unit index is in unit_q
  __shared__ __align__(8) uint64_t uempty_bar[kUnitRing];  // every role has read it
  __shared__ int unit_q[kUnitRing];
  __shared__ uint32_t tmem_base_sh;
  __shared__ volatile int abort_flag;

  __shared__ int s_first[kMaxBatchPanels + 1];  // a table's first unit per panel
  __shared__ int s_nsplit[kMaxBatchPanels];
  __shared__ int64_t s_kc[kMaxBatchPanels], s_kvalid[kMaxBatchPanels];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr bool tabled = TABLE;
  // barriers and tensor memory, while the kernel before this one may still run
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&dfull_bar[b], 1);
      mbar_init(&dempty_bar[b], kEpiWarps);
    }
    mbar_init(&drain_bar, 1);
    for (int i = 0; i < kUnitRing; ++i) {
      mbar_init(&ufull_bar[i], 1);
      mbar_init(&uempty_bar[i], 1 + kEpiWarps);
    }
    abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_sh, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base_sh;
  pdl_wait();

  int64_t kvalid = 0, kc = 0;
  int per_panel = 0, n_units;
  if constexpr (tabled) {
    if (warp == 0) {  // every lane plans (plan_splits is warp-wide); lane 0 records
      int acc = 0;
      for (int q = 0; q < table.n; ++q) {
        const HerkPanel &e = table.p[q];
        const int64_t kv = valid_k(e.n_dev, e.n_host, e.kmul, e.Kcap);
        int ns;
        int64_t kcq;
        plan_splits(kv, e.plan_tiles, e.k_chunk, nsm, ns, kcq);
        if (lane == 0) {
          s_first[q] = acc;
          s_nsplit[q] = ns;
          s_kc[q] = kcq;
          s_kvalid[q] = kv;
        }
        acc += ns * (e.T * (e.T + 1) / 2);
      }
      if (lane == 0) s_first[table.n] = acc;
    }
    __syncthreads();
    n_units = s_first[table.n];
  } else {
    kvalid = valid_k(n_dev, n_host, kmul, Kcap);
    int nsplit;
    plan_splits(kvalid, n_tiles * ngroup, k_chunk, nsm, nsplit, kc);
    per_panel = n_tiles * nsplit;
    n_units = per_panel * ngroup;
  }
  if ((int)blockIdx.x >= n_units) {  // uniform over the CTA
    if (warp == 1) tmem_dealloc(tbase, 512);
    return;
  }

  // Where unit u is: its panel and block count, tile, the tile's columns (TAIL in
  // a narrow last block, else 128), its k range and its partial tile.
  auto place = [&](int u, const uint8_t *&zpanel, float *&partial, int &Tu, int &I, int &J, int &nc, int64_t &k0,
                   int64_t &klen) {
    if constexpr (tabled) {
      int q = 0;
      while (q + 1 < table.n && s_first[q + 1] <= u) ++q;
      const HerkPanel &e = table.p[q];
      const int nt = e.T * (e.T + 1) / 2;
      const int r = u - s_first[q];
      Tu = e.T;
      decode_tile(r % nt, e.T, I, J);
      zpanel = e.panel;
      partial = e.partials + ((size_t)e.index * s_nsplit[q] * nt + r) * (256 * 128);
      k0 = (int64_t)(r / nt) * s_kc[q];
      klen = min(s_kc[q], s_kvalid[q] - k0);
    } else {
      const int r = u % per_panel;
      Tu = T;
      decode_tile(r % n_tiles, T, I, J);
      zpanel = zpanels + (int64_t)(u / per_panel) * zstride;
      partial = partials + (size_t)u * (256 * 128);
      k0 = (int64_t)(r / n_tiles) * kc;
      klen = min(kc, kvalid - k0);
    }
    nc = TAIL > 0 && J == Tu - 1 ? TAIL : 128;
  };
  // a bounded wait ran out: every status word of the launch learns it
  auto flag_timeout = [&]() {
    if (status) atomicOr(status, MVB_DEV_TIMEOUT);
    if constexpr (tabled)
      for (int q = 0; q < table.n; ++q)
        if (table.p[q].status) atomicOr(table.p[q].status, MVB_DEV_TIMEOUT);
  };

  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  uint64_t issued = 0;            // producer: stages issued
  bool lead = warp == 1 && lane == 0;  // the thread that issues the UMMAs
  if (warp == 0 && lane == 0) {
    // ---------------- bulk-copy producer ----------------
    uint32_t st = 0, ph = 0;
    for (uint32_t uk = 0; !abort_flag; ++uk) {
      // the CTA's next unit from the launch's counter, handed to the other roles
      const int us = uk % kUnitRing;
      if (!mbar_wait(&uempty_bar[us], ((uk / kUnitRing) & 1u) ^ 1u, wait_ns)) {
        flag_timeout();
        abort_flag = 1;
        break;
      }
      // (the first is its own index: no atomic before the first load)
      const int u = uk == 0 ? (int)blockIdx.x : min(atomicAdd(unit_next, 1) + (int)gridDim.x, n_units);
      unit_q[us] = u;
      mbar_arrive(&ufull_bar[us]);
      if (u >= n_units) break;
      const uint8_t *zpanel;
      float *partial;
      int Tu, I, J, nc;
      int64_t k0, klen;
      place(u, zpanel, partial, Tu, I, J, nc, k0, klen);
      const int nkb = (int)((klen + C::KB - 1) / C::KB);
      const bool diag = I == J;
      const uint32_t b_bytes = TAIL ? 2 * C::P * 64u * (uint32_t)nc : C::OPER_BYTES;  // block J's rows of every plane
      const uint32_t bytes = diag ? b_bytes : C::OPER_BYTES + b_bytes;
      for (int kbi = 0; kbi < nkb; ++kbi) {
        if (!mbar_wait(&empty_bar[st], ph ^ 1, wait_ns)) {
          flag_timeout();
          abort_flag = 1;
          break;
        }
        mbar_arrive_expect_tx(&full_bar[st], bytes);
        uint8_t *a = smem + (size_t)st * C::STAGE_BYTES;
        // k-block index: k0 is a multiple of 64 elements, a k-block 64 bytes;
        // operand (kb, R) starts at ((kb T + R) 2P) planes of 8 KB
        const int64_t kb = (k0 + (int64_t)kbi * C::KB) / C::KB;
        if constexpr (TAIL > 0) {
          if (!diag) bulk_load(a, zpanel + (kb * Tu + I) * (int64_t)C::OPER_BYTES, C::OPER_BYTES, &full_bar[st]);
          uint8_t *b = diag ? a : a + C::OPER_BYTES;
          const uint8_t *zb = zpanel + (kb * Tu + J) * (int64_t)C::OPER_BYTES;
          if (nc == 128)
            bulk_load(b, zb, C::OPER_BYTES, &full_bar[st]);
          else
            for (int pl = 0; pl < 2 * C::P; ++pl)
              bulk_load(b + pl * kPlaneBytes, zb + pl * kPlaneBytes, 64u * (uint32_t)nc, &full_bar[st]);
        } else {
          bulk_load(a, zpanel + (kb * Tu + I) * (int64_t)C::OPER_BYTES, C::OPER_BYTES, &full_bar[st]);
          if (!diag)
            bulk_load(a + C::OPER_BYTES, zpanel + (kb * Tu + J) * (int64_t)C::OPER_BYTES, C::OPER_BYTES, &full_bar[st]);
        }
        ++issued;
        if (++st == C::STAGES) {
          st = 0;
          ph ^= 1;
        }
      }
    }
  } else if (KD == 2 && warp == 1) {
    // ---------------- UMMA issuer, KD = 2: one fresh TMEM block per stage ----------------
    // The warp stays converged and an elected lane issues, so that descriptors and
    // loop state live in uniform registers; and the barriers of the NEXT block (its
    // stage filled, its TMEM block drained, at a unit's end the next unit) are waited
    // on between the last UMMAs of this one.  A single lane that waited between blocks
    // left the tensor pipe idle for 470 of 1,900 cycles per block: the pipe's queue
    // holds only the last few UMMAs, and the barrier checks, commits and descriptor
    // arithmetic took longer than those run.  Tensor pipe busy, 700 rows, fp16x3, by
    // clock64: 66 % that way, 79 % with both waits before the last k-step, 84-86 %
    // with the waits apart (tf32x3 66, 83, 89 %).  Under the power cap the clock gives
    // part of it back: 8 slices of K = 49,152 run at the sustained cuBLAS rate (1.40
    // PFLOP/s executed), K = 196,608 10.46 -> 9.71 ms, tf32x3 x 3 1.89 -> 1.66 ms; 128
    // two-feed antennas, K = 30,000 43.1 -> 35.4 us, 90 of one feed x 8 42.6 -> 34.7.
    // Within a block, products in ascending magnitude across both k-steps -- every
    // cross term, then the hi x hi products -- so that the block's large partial sum
    // exists only for its last instructions (the accumulator is truncated toward
    // zero at each).
    lead = elect_one();
    uint32_t st = 0, ph = 0, buf = 0, dph = 0, uk = 0;
    int nks = 0;
    bool diag = false, ok = true;
    bool narrow_unit = false;  // the unit's tile has TAIL columns
    auto wait_all = [&](uint64_t *bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, wait_ns)) != 0;
    };
    // the next unit's k-step count and tile kind; false when there is none (or a wait ran out)
    auto next_unit = [&]() {
      const int us = uk % kUnitRing;
      if (__any_sync(0xffffffffu, abort_flag)) return false;
      if (!wait_all(&ufull_bar[us], (uk / kUnitRing) & 1u)) {
        ok = false;
        return false;
      }
      const int u = __shfl_sync(0xffffffffu, unit_q[us], 0);
      if (lane == 0) mbar_arrive(&uempty_bar[us]);
      ++uk;
      if (u >= n_units) return false;
      const uint8_t *zpanel;
      float *partial;
      int Tu, I, J, nc;
      int64_t k0, klen;
      place(u, zpanel, partial, Tu, I, J, nc, k0, klen);
      nks = __shfl_sync(0xffffffffu, (int)((klen + C::KSTEP - 1) / C::KSTEP), 0);
      diag = __shfl_sync(0xffffffffu, I == J ? 1 : 0, 0) != 0;
      if constexpr (TAIL > 0) narrow_unit = __shfl_sync(0xffffffffu, nc, 0) < 128;
      return true;
    };
    bool have = next_unit();
    int ks = 0;
    if (have) ok = wait_all(&dempty_bar[0], 1u) && wait_all(&full_bar[0], 0u);
    // the blocks of consecutive units of one kind of tile
    auto issue_blocks = [&](auto narrow) {
      constexpr bool NARROW = decltype(narrow)::value;
      constexpr int NC = NARROW ? TAIL : 128;
      while (have && ok && (!TAIL || narrow_unit == NARROW)) {
        tc_fence_after();
        const int nk = min(2, nks - ks);
        const uint32_t d = tbase + buf * 256;
        const uint64_t a0 = umma_desc_sw64(smem_u32(smem) + st * C::STAGE_BYTES);
        const uint64_t b0 = diag ? a0 : a0 + (C::OPER_BYTES >> 4);
        const uint32_t id_re = diag ? C::ID128 : C::ID256;
        const bool dg = NARROW && diag;  // (next_unit changes it)
        const uint32_t st2 = st + 1 == C::STAGES ? 0 : st + 1, ph2 = st2 == 0 ? ph ^ 1u : ph;
        const uint32_t dph2 = dph ^ (1u << buf);
#pragma unroll
        for (int q = 0; q < C::NPROD; ++q) {
          uint32_t pa, pb;
          product_terms(C::NPROD, q, pa, pb);
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            // the next block, while the pipe still has the products before the last one
            // queued; the two waits apart, each covered by the UMMAs around it
            if (NARROW ? (q == C::NPROD - 2 && kk == 1) : (q == C::NPROD - 1 && kk == 0)) {
              ks += 2;
              if (ks >= nks) {
                have = next_unit();
                ks = 0;
              }
              if (have) ok = wait_all(&full_bar[st2], ph2);
            } else if (q == C::NPROD - 1 && kk == (NARROW ? 0 : 1) && have && ok) {
              ok = wait_all(&dempty_bar[buf ^ 1u], ((dph2 >> (buf ^ 1u)) & 1u) ^ 1u);
            }
            if (lead && kk < nk) {
              const uint64_t a_re = a0 + ((2 * pa * kPlaneBytes + kk * 32) >> 4);
              const uint64_t a_im = a0 + (((2 * pa + 1) * kPlaneBytes + kk * 32) >> 4);
              const uint64_t b_re = b0 + ((2 * pb * kPlaneBytes + kk * 32) >> 4);
              const uint64_t b_im = b0 + (((2 * pb + 1) * kPlaneBytes + kk * 32) >> 4);
              umma_kstep<MODE, NC>(d, a_re, a_im, b_re, b_im, id_re, dg, (q > 0 || kk > 0) ? 1u : 0u);
            }
            __syncwarp();
          }
        }
        if (lead) {
          tc_commit(&empty_bar[st]);  // the stage is consumed
          tc_commit(&dfull_bar[buf]);  // the block is complete
        }
        __syncwarp();
        st = st2;
        ph = ph2;
        dph = dph2;
        buf ^= 1u;
      }
    };
    if constexpr (TAIL > 0) {
      while (have && ok) {
        if (narrow_unit)
          issue_blocks(std::true_type{});
        else
          issue_blocks(std::false_type{});
      }
    } else {
      issue_blocks(std::false_type{});
    }
    if (!ok) {
      if (lane == 0) flag_timeout();
      abort_flag = 1;
    }
  } else if (KD != 2 && warp == 1 && lane == 0) {
    // ---------------- UMMA issuer, KD = 1 or 4: one thread, a wait before each block ----------------
    uint32_t st = 0, ph = 0, buf = 0, dph = 0;
    for (uint32_t uk = 0; !abort_flag; ++uk) {
      const int us = uk % kUnitRing;
      if (!mbar_wait(&ufull_bar[us], (uk / kUnitRing) & 1u, wait_ns)) {
        flag_timeout();
        abort_flag = 1;
        break;
      }
      const int u = unit_q[us];
      mbar_arrive(&uempty_bar[us]);
      if (u >= n_units) break;
      const uint8_t *zpanel;
      float *partial;
      int Tu, I, J, nc;
      int64_t k0, klen;
      place(u, zpanel, partial, Tu, I, J, nc, k0, klen);
      const int nks = (int)((klen + C::KSTEP - 1) / C::KSTEP);
      const bool diag = I == J;
      bool ok = true;
      if constexpr (KD == 4) {
        // a TMEM block is KD / 2 whole stages (two k-steps each): products
        // ordered by magnitude across the block's k-steps -- every cross term,
        // then the hi x hi products -- so that the block's large partial sum
        // exists only for its last instructions (the accumulator is truncated
        // toward zero at each)
        constexpr int SPB = KD / 2;
        for (int ks = 0; ks < nks; ks += KD) {
          const int nk = min(KD, nks - ks);
          const int nst = (nk + 1) / 2;
          uint32_t slot[SPB];
          if (!mbar_wait(&dempty_bar[buf], ((dph >> buf) & 1u) ^ 1u, wait_ns)) ok = false;
#pragma unroll
          for (int j = 0; j < SPB; ++j) {
            if (j >= nst || !ok) break;
            if (!mbar_wait(&full_bar[st], ph, wait_ns)) {
              ok = false;
              break;
            }
            slot[j] = st;
            if (++st == C::STAGES) {
              st = 0;
              ph ^= 1;
            }
          }
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tbase + buf * 256;
#pragma unroll
          for (int q = 0; q < C::NPROD; ++q) {
            uint32_t pa, pb;
            product_terms(C::NPROD, q, pa, pb);
#pragma unroll
            for (int kk = 0; kk < KD; ++kk) {
              if (kk >= nk) break;
              const uint32_t a_base =
                  smem_u32(smem + (size_t)slot[kk >> 1] * C::STAGE_BYTES) + (uint32_t)(kk & 1) * 32;
              const uint32_t b_base = diag ? a_base : a_base + C::OPER_BYTES;
              const uint64_t a_re = umma_desc_sw64(a_base + (2 * pa) * kPlaneBytes);
              const uint64_t a_im = umma_desc_sw64(a_base + (2 * pa + 1) * kPlaneBytes);
              const uint64_t b_re = umma_desc_sw64(b_base + (2 * pb) * kPlaneBytes);
              const uint64_t b_im = umma_desc_sw64(b_base + (2 * pb + 1) * kPlaneBytes);
              umma_kstep<MODE, 128>(d, a_re, a_im, b_re, b_im, diag ? C::ID128 : C::ID256, diag,
                                       (q > 0 || kk > 0) ? 1u : 0u);
            }
          }
#pragma unroll
          for (int j = 0; j < SPB; ++j)
            if (j < nst) tc_commit(&empty_bar[slot[j]]);  // the block's stages are consumed
          tc_commit(&dfull_bar[buf]);                      // the block is complete
          dph ^= 1u << buf;
          buf ^= 1u;
        }
      } else {
      // k-steps in order; a TMEM block holds KD of them, a stage (one 64-byte
      // k-block) two: the block and stage boundaries are independent
      for (int ks = 0; ks < nks; ++ks) {
        if (ks % KD == 0) {  // a fresh TMEM block
          if (!mbar_wait(&dempty_bar[buf], ((dph >> buf) & 1u) ^ 1u, wait_ns)) {
            ok = false;
            break;
          }
          tc_fence_after();
        }
        if ((ks & 1) == 0) {  // a new stage
          if (!mbar_wait(&full_bar[st], ph, wait_ns)) {
            ok = false;
            break;
          }
          tc_fence_after();
        }
        const uint32_t d = tbase + buf * 256;
        const uint32_t koff = (uint32_t)(ks & 1) * 32;  // the k-step's 32 bytes within the 64-byte rows
        const uint32_t a_base = smem_u32(smem + (size_t)st * C::STAGE_BYTES) + koff;
        const uint32_t b_base = diag ? a_base : a_base + C::OPER_BYTES;
#pragma unroll
        for (int q = 0; q < C::NPROD; ++q) {
          uint32_t pa, pb;
          product_terms(C::NPROD, q, pa, pb);
          const uint64_t a_re = umma_desc_sw64(a_base + (2 * pa) * kPlaneBytes);
          const uint64_t a_im = umma_desc_sw64(a_base + (2 * pa + 1) * kPlaneBytes);
          const uint64_t b_re = umma_desc_sw64(b_base + (2 * pb) * kPlaneBytes);
          const uint64_t b_im = umma_desc_sw64(b_base + (2 * pb + 1) * kPlaneBytes);
          umma_kstep<MODE, 128>(d, a_re, a_im, b_re, b_im, diag ? C::ID128 : C::ID256, diag,
                                   (ks % KD != 0 || q > 0) ? 1u : 0u);
        }
        if ((ks & 1) == 1 || ks == nks - 1) {  // the stage is consumed
          tc_commit(&empty_bar[st]);
          if (++st == C::STAGES) {
            st = 0;
            ph ^= 1;
          }
        }
        if (ks % KD == KD - 1 || ks == nks - 1) {  // the block is complete
          tc_commit(&dfull_bar[buf]);
          dph ^= 1u << buf;
          buf ^= 1u;
        }
      }
      }
      if (!ok) {
        flag_timeout();
        abort_flag = 1;
        break;
      }
    }
  } else if (warp >= 2) {
    // ---------------- epilogue: drain every k-step block into FP32 registers ----------------
    const int quad = warp & 3;
    const int quarter = (warp - 2) >> 2;  // columns [64 quarter, 64 quarter + 64)
    const int row = quad * 32 + lane;
    uint32_t buf = 0, dph = 0;
    float acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.f;
    for (uint32_t uk = 0; !abort_flag; ++uk) {
      const int us = uk % kUnitRing;
      // every lane waits; the vote keeps the warp converged
      if (!__all_sync(0xffffffffu, mbar_wait(&ufull_bar[us], (uk / kUnitRing) & 1u, wait_ns))) {
        if (lane == 0) flag_timeout();
        abort_flag = 1;
        break;
      }
      const int u = unit_q[us];
      __syncwarp();
      if (lane == 0) mbar_arrive(&uempty_bar[us]);
      if (u >= n_units) break;
      const uint8_t *zpanel;
      float *partial;
      int Tu, I, J, nc;
      int64_t k0, klen;
      place(u, zpanel, partial, Tu, I, J, nc, k0, klen);
      const int nks = (int)((klen + C::KSTEP - 1) / C::KSTEP);
      // live columns of this warp's quarter; none of a quadrant of padding rows (which
      // only the last diagonal tile has: its rows are its columns)
      const int mine = !TAIL ? 64 : I == J && quad * 32 >= nc ? 0 : max(0, nc - (quarter & 1) * 64);
      const bool live = !TAIL || I != J || row < nc;
      bool ok = true;
      for (int g0 = 0; g0 < nks; g0 += KD) {
        // every lane waits; the vote keeps the warp converged for tcgen05.ld
        ok = __all_sync(0xffffffffu, mbar_wait(&dfull_bar[buf], (dph >> buf) & 1u, wait_ns));
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tbase + ((uint32_t)(quad * 32) << 16) + buf * 256 + quarter * 64;
        constexpr int W = KD == 2 ? 8 : 16;  // columns per load: 16 spill beside the KD = 2 issuer
#pragma unroll
        for (int c = 0; c < 64 / W; ++c) {
          if (TAIL && c * W >= mine) break;
          uint32_t v[W];
          tmem_ld<W>(taddr + c * W, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < W; ++j) acc[c * W + j] += __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&dempty_bar[buf]);
        dph ^= 1u << buf;
        buf ^= 1u;
      }
      if (!ok) {
        if (lane == 0) flag_timeout();
        abort_flag = 1;
        break;
      }
      float *dst = partial + (size_t)quarter * 64 * 128;
#pragma unroll
      for (int j = 0; j < 64; ++j) {
        if (live && j < mine) dst[j * 128 + row] = acc[j];
        acc[j] = 0.f;
      }
    }
  }

  // Takes effect with the first thread that gets here, the producer's, while the CTA's
  // last stages are still multiplied and stored: a dependent may be scheduled from then
  // on, and reads nothing of this launch before its pdl_wait().
  pdl_trigger();
  __syncthreads();
  if (abort_flag) {
    if (warp == 0 && lane == 0) {
      // wait for the copies still in flight (the last STAGES issued)
      const uint64_t first = issued > (uint64_t)C::STAGES ? issued - C::STAGES : 0;
      for (uint64_t i = first; i < issued; ++i)
        mbar_wait(&full_bar[i % C::STAGES], (uint32_t)((i / C::STAGES) & 1), kDrainLimitNs);
    }
    if (lead) {
      tc_commit(&drain_bar);
      mbar_wait(&drain_bar, 0, kDrainLimitNs);
    }
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tbase, 512);
  }
}

// ---------------------------------------------------------------------------
// FP64 reduction of the partial tiles into the reference output layout
// out[pair, p, q] = V[ant_i * F + q, ant_j * F + p].
// ---------------------------------------------------------------------------
constexpr int kRedBlocks = 16;    // 32 x 32 blocks of a 128 x 128 tile, one CTA each
constexpr int kRedThreads = 256;  // threads over one block: four rows of one column each
constexpr int kRedPairThreads = 64;  // pair lists: small CTAs, so that a short list spreads over the SMs

__device__ __forceinline__ int tile_index(int I, int J, int T) { return I * T - (I * (I - 1)) / 2 + (J - I); }

template <typename OT>
__device__ __forceinline__ void store_out(void *out, int64_t idx, double re, double im, int accumulate) {
  OT *o = static_cast<OT *>(out) + idx;
  if (accumulate) {
    o->x += re;
    o->y += im;
  } else {
    o->x = re;
    o->y = im;
  }
}

// Float-float accumulator: Knuth's TwoSum keeps the exact rounding error of each
// FP32 addition in a second FP32 word (about 2^-44 relative), on the FP32 pipe;
// the per-element float -> double conversions it replaces ran on the
// conversion unit and bounded the reduction's rate.
struct FF {
  float hi = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float s = __fadd_rn(hi, v);
    const float bb = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(v, bb));
    hi = s;
    lo = __fadd_rn(lo, err);
  }
  __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Adds the slices of NP runs of four rows (a float4 each, sstride float4 apart
// per slice) to their float-float sums in slice order, U slices' loads in flight
// at a time.
template <int NP, int U>
__device__ __forceinline__ void sum_slices(const float4 *const (&p)[NP], int nsplit, size_t sstride,
                                           FF (&acc)[NP][4]) {
  for (int s = 0; s < nsplit; s += U) {
    float4 v[U][NP];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s + u < nsplit) {
#pragma unroll
        for (int k = 0; k < NP; ++k) v[u][k] = __ldcg(p[k] + (s + u) * sstride);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (s + u < nsplit) {
#pragma unroll
        for (int k = 0; k < NP; ++k) {
          acc[k][0].add(v[u][k].x);
          acc[k][1].add(v[u][k].y);
          acc[k][2].add(v[u][k].z);
          acc[k][3].add(v[u][k].w);
        }
      }
  }
}

// One CTA per 32 x 32 block of an upper tile; a thread sums four rows of one
// column.  A diagonal tile's imaginary half is W - W^T of its partial sums (the
// product leaves W there): its CTA also sums the mirrored block of W and the two
// are transposed through shared memory once, after the sums.  Blocks of padding
// rows are not read.
// What bounds it: the slices' bytes where there are many tiles, the chain of
// loads of one thread where there are few (the plan then cuts many slices).  Both
// want loads in flight and no barrier between them: 15 or 16 independent 16-byte
// loads a thread.  Measured against CTAs of 8 columns x 128 rows, whose diagonal
// tiles transposed every second slice through shared memory (two barriers each):
// 8 panels of 700 rows, K = 196,608: 302 -> 251 us (4.2 TB/s of partial tiles); one
// 43.5 -> 28.0; 8 panels of 90 rows, K = 11,180: 12.2 -> 8.6; one of 122 rows,
// K = 20,000, slices of 576: 23.2 -> 13.4.  Four groups of threads sharing a block's
// slices (1,024-thread CTAs) were slower: 10.8 us on the 90 rows, 14.2 on the 122.
// F is a template parameter (no runtime integer division in the index
// arithmetic).  blockIdx.y is the panel of a grouped product; its output is
// out_stride bytes further.
template <typename OT, int F>
__global__ void __launch_bounds__(kRedThreads, 2)
    herk_reduce_all_kernel(const float *__restrict__ part, int ngroup, int T, int n_tiles,
                           const int32_t *__restrict__ n_dev, int64_t n_host, int kmul, int64_t Kcap, int k_chunk,
                           int nsm, int A, void *__restrict__ out_base, int64_t out_stride, double vscale,
                           const float *__restrict__ zscale, int accumulate, int *__restrict__ unit_next) {
  __shared__ FF turn_sm[32][33];
  pdl_wait();
  pdl_trigger();
  if (unit_next && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *unit_next = 0;  // for the next product
  const int t = blockIdx.x / kRedBlocks, rb = blockIdx.x % 4, cb = blockIdx.x / 4 % 4;
  int I, J;
  decode_tile(t, T, I, J);
  const int M = A * F;
  if (I * 128 + rb * 32 >= M || J * 128 + cb * 32 >= M) return;  // padding (uniform over the CTA)
  const int64_t kvalid = valid_k(n_dev, n_host, kmul, Kcap);
  int nsplit;
  int64_t kc;
  plan_splits(kvalid, n_tiles * ngroup, k_chunk, nsm, nsplit, kc);
  if (zscale) vscale = 1.0 / ((double)*zscale * (double)*zscale);
  void *out = static_cast<uint8_t *>(out_base) + (int64_t)blockIdx.y * out_stride;
  part += (size_t)blockIdx.y * nsplit * n_tiles * (256 * 128);
  const int cc = threadIdx.x >> 3, rr = 4 * (threadIdx.x & 7);  // column and first row within the block
  const int c = cb * 32 + cc, r0 = rb * 32 + rr;
  const float *tile = part + (size_t)t * (256 * 128);
  const size_t sstride = (size_t)n_tiles * (256 * 128) / 4;  // in float4
  const bool diag = I == J;
  const float4 *pre = reinterpret_cast<const float4 *>(tile + c * 128 + r0);
  const float4 *pim = reinterpret_cast<const float4 *>(tile + (128 + c) * 128 + r0);
  FF acc[3][4];
  if (diag && rb != cb) {
    // the mirrored block: its column rb * 32 + cc, rows cb * 32 + rr ..
    const float4 *const p[3] = {
        pre, pim, reinterpret_cast<const float4 *>(tile + (128 + rb * 32 + cc) * 128 + cb * 32 + rr)};
    sum_slices<3, 5>(p, nsplit, sstride, acc);
  } else {
    const float4 *const p[2] = {pre, pim};
    FF(&acc2)[2][4] = reinterpret_cast<FF(&)[2][4]>(acc);
    sum_slices<2, 8>(p, nsplit, sstride, acc2);
  }
  if (diag) {
    // element (row r, column c) subtracts W(c, r): column r, row c of the mirrored block
#pragma unroll
    for (int j = 0; j < 4; ++j) turn_sm[cc][rr + j] = rb != cb ? acc[2][j] : acc[1][j];
    __syncthreads();
  }
  const int n = J * 128 + c;
  if (n >= M) return;
  const int64_t AF2 = (int64_t)A * F * F;
  const int jj = n / F, pp = n % F;  // F is 1 or 2: shifts and masks
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int m = I * 128 + r0 + k;
    if (m >= M) break;
    // an autocorrelation of one feed (m == n) is real, as conj(z) z is in the reference
    const double wi = diag ? acc[1][k].value() - turn_sm[rr + k][cc].value() : acc[1][k].value();
    const double re = acc[0][k].value() * vscale, im = m == n ? 0.0 : wi * vscale;
    const int i = m / F, q = m % F;
    // direct: rows m -> (i, q), columns n -> (j, p); out[(i*A + j)*F*F + p*F + q]
    store_out<OT>(out, i * AF2 + (int64_t)jj * F * F + pp * F + q, re, im, accumulate);
    // mirror: V[n, m] = conj(V[m, n]) for the off-diagonal tiles (a diagonal tile
    // holds both triangles and is written directly)
    if (!diag) store_out<OT>(out, jj * AF2 + (int64_t)i * F * F + q * F + pp, re, -im, accumulate);
  }
}

// Explicit pair list: one thread per (pair, p, q).  Its loads are scattered, a line
// each, so the lines an SM can look up bound a short list on few CTAs: 64 threads each
// (64 one-feed antennas, 2,000 pairs, K = 64,000: 11.9 us, 21.7 with 256, and 19.5 with
// 256 and one slice in flight instead of eight).
// A pair naming an antenna outside [0, A) reads nothing and gets NaN.
// blockIdx.y is the panel of a grouped product.
template <typename OT>
__global__ void herk_reduce_pairs_kernel(const float *__restrict__ part, int ngroup, int T, int n_tiles,
                                         const int32_t *__restrict__ n_dev, int64_t n_host, int kmul, int64_t Kcap,
                                         int k_chunk, int nsm, int A, int F, const int32_t *__restrict__ pairs,
                                         int64_t npairs, void *__restrict__ out_base, int64_t out_stride,
                                         double vscale, const float *__restrict__ zscale, int accumulate,
                                         int *__restrict__ unit_next) {
  const int64_t total = npairs * F * F;
  pdl_wait();
  pdl_trigger();
  if (unit_next && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *unit_next = 0;  // for the next product
  const int64_t kvalid = valid_k(n_dev, n_host, kmul, Kcap);
  int nsplit;
  int64_t kc;
  plan_splits(kvalid, n_tiles * ngroup, k_chunk, nsm, nsplit, kc);
  if (zscale) vscale = 1.0 / ((double)*zscale * (double)*zscale);
  void *out = static_cast<uint8_t *>(out_base) + (int64_t)blockIdx.y * out_stride;
  part += (size_t)blockIdx.y * nsplit * n_tiles * (256 * 128);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pr = e / (F * F);
    const int p = (int)((e / F) % F), q = (int)(e % F);
    const int ai = pairs[2 * pr], aj = pairs[2 * pr + 1];
    if (ai < 0 || ai >= A || aj < 0 || aj >= A) {
      store_out<OT>(out, e, __longlong_as_double(0x7ff8000000000000ll), 0.0, 0);
      continue;
    }
    int m = ai * F + q, n = aj * F + p;
    bool conj = false;
    if (m / 128 > n / 128) {
      const int tmp = m;
      m = n;
      n = tmp;
      conj = true;
    }
    const int t = tile_index(m / 128, n / 128, T);
    const int r = m % 128, c = n % 128;
    const bool diag = m / 128 == n / 128;  // imaginary half W - W^T (see herk_reduce_all_kernel)
    FF re, im, imt;
    const float *p0 = part + (size_t)t * (256 * 128);
    const size_t sstride = (size_t)n_tiles * (256 * 128);
    constexpr int U = 8;  // slices in flight: the chain of scattered loads bounds a thread
    for (int s = 0; s < nsplit; s += U) {
      float vr[U], vi[U], vt[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (s + u < nsplit) {
          const float *ps = p0 + (s + u) * sstride;
          vr[u] = __ldcg(ps + c * 128 + r);
          vi[u] = __ldcg(ps + (128 + c) * 128 + r);
          if (diag) vt[u] = __ldcg(ps + (128 + r) * 128 + c);
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (s + u < nsplit) {
          re.add(vr[u]);
          im.add(vi[u]);
          if (diag) imt.add(vt[u]);
        }
    }
    const double wi = diag ? im.value() - imt.value() : im.value();
    const double vi = m == n ? 0.0 : (conj ? -wi : wi) * vscale;  // one-feed autos are real
    store_out<OT>(out, e, re.value() * vscale, vi, accumulate);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Raises a kernel's dynamic shared-memory limit once per (device, slot); the
// attribute is not touched again, in particular not during graph capture.
int set_smem_once(const void *fn, int bytes, int slot) {
  static bool done[64][64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || slot < 0 || slot >= 64)
    return fail(MVB_ERR_CUDA, "set_smem_once: bad device");
  if (done[dev][slot]) return MVB_OK;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return fail(MVB_ERR_CUDA, "smem attribute: %s", cudaGetErrorString(e));
  done[dev][slot] = true;
  return MVB_OK;
}

// Wall-time limit of the product's pipeline waits, process-wide (see
// mvb_set_wait_limit_ns); read at each launch.
static std::atomic<uint64_t> g_wait_limit_ns{kWaitLimitNs};
uint64_t wait_limit_ns() { return g_wait_limit_ns.load(std::memory_order_relaxed); }

// table.n > 0: the units come from the table (z, ngroup, shape and status arguments unused).
template <int MODE, int KD>
static int launch_herk(const void *z, int64_t zstride, int ngroup, int64_t Mpad, int rows, int64_t Kcap,
                       const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, float *partials, int32_t *status,
                       int *unit_next, bool clear_counter, cudaStream_t s, const HerkTable &table) {
  using C = HerkCfg<MODE>;
  const int T = (int)(Mpad / 128);
  const int n_tiles = T * (T + 1) / 2;
  const int nsm = num_sms();
  int64_t max_units = (int64_t)ngroup * n_tiles * (ceil_div(Kcap, k_chunk) + kPlanExtra);
  if (table.n > 0) {
    max_units = 0;
    for (int q = 0; q < table.n; ++q) {
      const HerkPanel &e = table.p[q];
      max_units += (int64_t)(e.T * (e.T + 1) / 2) * (ceil_div(e.Kcap, e.k_chunk) + kPlanExtra);
    }
  }
  const int grid = (int)std::min<int64_t>(max_units, nsm);
  const size_t smem = (size_t)C::STAGES * C::STAGE_BYTES + 1024;
  // The last block of one repeated shape as its live rows rounded up to 64 or 96, under
  // the default drain.  The forms' waits and drains are the more expensive ones for full
  // tiles, so a shape without a narrow block keeps the plain form (384 rows: 1.5 % more
  // cycles in the narrow one).
  constexpr int kTail64 = KD == 2 ? 64 : 0, kTail96 = KD == 2 ? 96 : 0;
  const int last = (int)(rows - (Mpad - 128));
  const int tail = KD != 2 || table.n > 0 || last > 96 ? 0 : last > 64 ? 96 : 64;
  // slots 16 + 3 * MODE + {0, 1, 2} for KD = {1, 2, 4}, 15 more for the table forms; 50 + MODE and 55 + MODE for
  // the narrow ones
  const int slot = tail == 96   ? 55 + MODE
                   : tail == 64 ? 50 + MODE
                                : 16 + 3 * MODE + (KD == 4 ? 2 : KD - 1) + (table.n > 0 ? 15 : 0);
  const void *fn = table.n > 0  ? reinterpret_cast<const void *>(herk_kernel<MODE, KD, true, 0>)
                   : tail == 96 ? reinterpret_cast<const void *>(herk_kernel<MODE, KD, false, kTail96>)
                   : tail == 64 ? reinterpret_cast<const void *>(herk_kernel<MODE, KD, false, kTail64>)
                                : reinterpret_cast<const void *>(herk_kernel<MODE, KD, false, 0>);
  int rc = set_smem_once(fn, (int)smem, slot);
  if (rc) return rc;
  if (grid <= 0) return MVB_OK;
  const uint64_t wait_ns = wait_limit_ns();
  if (clear_counter) {  // the CTAs take units from this counter
    cudaError_t e = cudaMemsetAsync(unit_next, 0, sizeof(int), s);
    if (e != cudaSuccess) return fail(MVB_ERR_CUDA, "herk unit counter: %s", cudaGetErrorString(e));
  }
  auto launch = [&](auto kernel, auto units) {
    return launch_chained("herk_kernel", kernel, grid, kHerkThreads, smem, s, static_cast<const uint8_t *>(z), zstride,
                          ngroup, T, n_tiles, n_dev, n_host, kmul, Kcap, k_chunk, nsm, partials, status, unit_next,
                          wait_ns, units);
  };
  if (table.n > 0) return launch(herk_kernel<MODE, KD, true, 0>, table);
  if (tail == 96) return launch(herk_kernel<MODE, KD, false, kTail96>, NoTable{});
  if (tail == 64) return launch(herk_kernel<MODE, KD, false, kTail64>, NoTable{});
  return launch(herk_kernel<MODE, KD, false, 0>, NoTable{});
}

// Argument checks shared by the product and its reductions (the slice plan
// the reductions recompute is the product's only if these hold).
static int check_herk_shape(const char *who, int ngroup, int64_t Mpad, int64_t Kcap, const int32_t *n_dev,
                            int64_t n_host, int kmul, int k_chunk) {
  if (ngroup <= 0 || Mpad <= 0 || Mpad % 128 || Kcap <= 0 || Kcap % kKAlign || k_chunk <= 0 || k_chunk % kKAlign ||
      n_host < 0 || kmul <= 0)
    return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  if (!n_dev && n_host * kmul > Kcap) return fail(MVB_ERR_ARG, "%s: n * kmul exceeds Kcap", who);
  if (Kcap > INT32_MAX || Mpad > 65536) return fail(MVB_ERR_ARG, "%s: panel too large", who);
  const int64_t T = Mpad / 128;
  if ((int64_t)ngroup * (T * (T + 1) / 2) * (ceil_div(Kcap, k_chunk) + kPlanExtra) > INT32_MAX)
    return fail(MVB_ERR_ARG, "%s: too many work units", who);
  return MVB_OK;
}

// The checks of one product (a group of ngroup panels of one shape).
static int check_herk_group(const char *who, const void *z, int64_t zstride, int ngroup, int mode, int64_t Mpad,
                            int64_t Kcap, const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, const void *ws,
                            size_t ws_bytes, const int32_t *status) {
  if (!z || !ws || !status) return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  int rc = check_herk_shape(who, ngroup, Mpad, Kcap, n_dev, n_host, kmul, k_chunk);
  if (rc) return rc;
  if (reinterpret_cast<uintptr_t>(z) % 16 || zstride % 16) return fail(MVB_ERR_ARG, "%s: panel not 16-byte aligned", who);
  if (ngroup > 1 && (size_t)zstride < mvb_zpanel_bytes(mode, Mpad, Kcap))
    return fail(MVB_ERR_ARG, "%s: panels overlap (stride below mvb_zpanel_bytes)", who);
  if (ws_bytes / (size_t)ngroup < mvb_herk_ws_bytes(Mpad, Kcap, k_chunk))
    return fail(MVB_ERR_ARG, "%s: workspace too small", who);
  if (reinterpret_cast<uintptr_t>(ws) % 16) return fail(MVB_ERR_ARG, "%s: ws must be 16-byte aligned", who);
  return MVB_OK;
}

// Past every partial tile: each group's share of ws_bytes holds kCounterBytes spare.
static int *unit_counter(void *ws, size_t ws_bytes) {
  return reinterpret_cast<int *>(static_cast<uint8_t *>(ws) + ((ws_bytes - 16) & ~size_t(15)));
}

static int herk_impl(const char *who, const void *z, int64_t zstride, int ngroup, int mode, int64_t Mpad, int64_t Kcap,
                     const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int drain_ksteps, void *ws,
                     size_t ws_bytes, int32_t *status, void *stream, const HerkTable &table = HerkTable{},
                     bool clear_counter = true, int64_t live_rows = 0) {
  const int rows = (int)(live_rows ? live_rows : Mpad);
  if (table.n == 0) {
    if (rows > Mpad || rows <= Mpad - 128) return fail(MVB_ERR_ARG, "%s: rows do not end in the last block", who);
    int rc = check_herk_group(who, z, zstride, ngroup, mode, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, ws, ws_bytes,
                              status);
    if (rc) return rc;
  }
  if (drain_ksteps < 0 || drain_ksteps > 4 || drain_ksteps == 3)
    return fail(MVB_ERR_ARG, "%s: drain_ksteps must be 0, 1, 2 or 4", who);
  // default: a block per stage (two k-steps), the fastest interval in every mode
  const int kd = drain_ksteps ? drain_ksteps : 2;
  cudaStream_t s = as_stream(stream);
  float *part = static_cast<float *>(ws);
  int *next = unit_counter(ws, ws_bytes);
#define MVB_HERK(M)                                                                                          \
  return kd == 1   ? launch_herk<M, 1>(z, zstride, ngroup, Mpad, rows, Kcap, n_dev, n_host, kmul, k_chunk, part, status, \
                                       next, clear_counter, s, table)                                                       \
         : kd == 2 ? launch_herk<M, 2>(z, zstride, ngroup, Mpad, rows, Kcap, n_dev, n_host, kmul, k_chunk, part, status, \
                                       next, clear_counter, s, table)                                                       \
                   : launch_herk<M, 4>(z, zstride, ngroup, Mpad, rows, Kcap, n_dev, n_host, kmul, k_chunk, part, status, \
                                       next, clear_counter, s, table)
  switch (mode) {
    case MVB_GEMM_BF16_3: MVB_HERK(MVB_GEMM_BF16_3);
    case MVB_GEMM_BF16_6: MVB_HERK(MVB_GEMM_BF16_6);
    case MVB_GEMM_TF32_3: MVB_HERK(MVB_GEMM_TF32_3);
    case MVB_GEMM_F16_3: MVB_HERK(MVB_GEMM_F16_3);
    default: return fail(MVB_ERR_ARG, "%s: unknown mode %d", who, mode);
  }
#undef MVB_HERK
}

static int reduce_impl(const char *who, const void *ws, size_t ws_bytes, int ngroup, int64_t Mpad, int64_t Kcap,
                       const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int nant, int nfeed,
                       const int32_t *pairs, int64_t npairs, void *out, int64_t out_stride, int out_c128,
                       double vscale, const float *zscale, int accumulate, void *stream, int *unit_next = nullptr) {
  // the checks of mvb_herk: the slice plan recomputed here is then the product's
  if (!ws || !out || nant <= 0 || (nfeed != 1 && nfeed != 2) || (int64_t)nant * nfeed > Mpad || (pairs && npairs < 0))
    return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  int rc = check_herk_shape(who, ngroup, Mpad, Kcap, n_dev, n_host, kmul, k_chunk);
  if (rc) return rc;
  if (ws_bytes / (size_t)ngroup < mvb_herk_ws_bytes(Mpad, Kcap, k_chunk))
    return fail(MVB_ERR_ARG, "%s: workspace smaller than the product's (mvb_herk_ws_bytes)", who);
  if (reinterpret_cast<uintptr_t>(ws) % 16) return fail(MVB_ERR_ARG, "%s: ws must be 16-byte aligned", who);
  const int64_t per_out = (pairs ? npairs : (int64_t)nant * nant) * nfeed * nfeed * (out_c128 ? 16 : 8);
  if (ngroup > 1 && out_stride < per_out) return fail(MVB_ERR_ARG, "%s: outputs overlap (out_stride too small)", who);
  if (ngroup > 65535) return fail(MVB_ERR_ARG, "%s: at most 65535 panels per launch", who);
  const int T = (int)(Mpad / 128);
  const int n_tiles = T * (T + 1) / 2;
  const int nsm = num_sms();
  const float *part = static_cast<const float *>(ws);
  cudaStream_t s = as_stream(stream);
  if (!pairs) {
    const dim3 grid((unsigned)(n_tiles * kRedBlocks), (unsigned)ngroup);
#define MVB_RED(OT, FF_)                                                                                           \
  return launch_chained(who, herk_reduce_all_kernel<OT, FF_>, grid, kRedThreads, 0, s, part, ngroup, T, n_tiles,   \
                        n_dev, n_host, kmul, Kcap, k_chunk, nsm, nant, out, out_stride, vscale, zscale, accumulate, \
                        unit_next)
    if (out_c128) {
      if (nfeed == 2) MVB_RED(double2, 2); else MVB_RED(double2, 1);
    } else {
      if (nfeed == 2) MVB_RED(float2, 2); else MVB_RED(float2, 1);
    }
#undef MVB_RED
  } else {
    if (npairs == 0) return MVB_OK;
    const int64_t total = npairs * nfeed * nfeed;
    const dim3 grid((unsigned)std::min<int64_t>(ceil_div(total, kRedPairThreads), (int64_t)nsm * 32), (unsigned)ngroup);
    const auto kernel = out_c128 ? herk_reduce_pairs_kernel<double2> : herk_reduce_pairs_kernel<float2>;
    return launch_chained(who, kernel, grid, kRedPairThreads, 0, s, part, ngroup, T, n_tiles, n_dev, n_host, kmul, Kcap, k_chunk,
                          nsm, nant, nfeed, pairs, npairs, out, out_stride, vscale, zscale, accumulate, unit_next);
  }
}

int herk_grouped_chained(const void *z, size_t z_stride, int ngroup, int mode, int64_t Mpad, int64_t rows,
                         int64_t Kcap, const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int drain_ksteps,
                         void *ws, size_t ws_bytes, int32_t *status, void *stream) {
  return herk_impl("mvb_herk_grouped", z, (int64_t)z_stride, ngroup, mode, Mpad, Kcap, n_dev, n_host, kmul, k_chunk,
                   drain_ksteps, ws, ws_bytes, status, stream, HerkTable{}, false, rows);
}

int herk_reduce_grouped_chained(void *ws, size_t ws_bytes, int ngroup, int64_t Mpad, int64_t Kcap,
                                const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int nant, int nfeed,
                                const int32_t *pairs, int64_t npairs, void *out, size_t out_stride, int out_c128,
                                double vscale, int accumulate, void *stream) {
  return reduce_impl("mvb_herk_reduce_grouped", ws, ws_bytes, ngroup, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, nant,
                     nfeed, pairs, npairs, out, (int64_t)out_stride, out_c128, vscale, nullptr, accumulate, stream,
                     unit_counter(ws, ws_bytes));
}

int clear_unit_counter(void *ws, size_t ws_bytes, void *stream) {
  cudaError_t e = cudaMemsetAsync(unit_counter(ws, ws_bytes), 0, sizeof(int), as_stream(stream));
  return e == cudaSuccess ? MVB_OK : fail(MVB_ERR_CUDA, "herk unit counter: %s", cudaGetErrorString(e));
}

}  // namespace mvb

using namespace mvb;

extern "C" uint64_t mvb_set_wait_limit_ns(uint64_t limit_ns) {
  return g_wait_limit_ns.exchange(limit_ns ? limit_ns : kWaitLimitNs);
}

extern "C" size_t mvb_herk_ws_bytes(int64_t Mpad, int64_t Kcap, int k_chunk) {
  if (Mpad <= 0 || Kcap <= 0 || k_chunk <= 0) return 0;
  const int64_t T = Mpad / 128;
  return (size_t)(T * (T + 1) / 2) * (size_t)(ceil_div(Kcap, k_chunk) + kPlanExtra) * 256 * 128 * sizeof(float) +
         kCounterBytes;
}

extern "C" int mvb_herk(const void *z, int mode, int64_t Mpad, int64_t Kcap, const int32_t *n_dev, int64_t n_host,
                        int kmul, int k_chunk, int drain_ksteps, void *ws, size_t ws_bytes, int32_t *status,
                        void *stream) {
  return herk_impl("mvb_herk", z, 0, 1, mode, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, drain_ksteps, ws, ws_bytes,
                   status, stream);
}

extern "C" int mvb_herk_grouped(const void *z, size_t z_stride, int ngroup, int mode, int64_t Mpad, int64_t Kcap,
                                const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int drain_ksteps,
                                void *ws, size_t ws_bytes, int32_t *status, void *stream) {
  if (z_stride > (size_t)INT64_MAX) return fail(MVB_ERR_ARG, "mvb_herk_grouped: bad arguments");
  return herk_impl("mvb_herk_grouped", z, (int64_t)z_stride, ngroup, mode, Mpad, Kcap, n_dev, n_host, kmul, k_chunk,
                   drain_ksteps, ws, ws_bytes, status, stream);
}

extern "C" int mvb_herk_grouped_rows(const void *z, size_t z_stride, int ngroup, int mode, int64_t Mpad, int64_t rows,
                                     int64_t Kcap, const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk,
                                     int drain_ksteps, void *ws, size_t ws_bytes, int32_t *status, void *stream) {
  const char *who = "mvb_herk_grouped_rows";
  if (z_stride > (size_t)INT64_MAX || rows <= 0) return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  return herk_impl(who, z, (int64_t)z_stride, ngroup, mode, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, drain_ksteps, ws,
                   ws_bytes, status, stream, HerkTable{}, true, rows);
}

extern "C" int mvb_herk_batch(const mvb_herk_group *groups, int ngroups, int mode, int drain_ksteps, void *stream) {
  if (!groups || ngroups <= 0) return fail(MVB_ERR_ARG, "mvb_herk_batch: bad arguments");
  HerkTable table{};
  for (int g = 0; g < ngroups; ++g) {
    const mvb_herk_group &e = groups[g];
    if (e.z_stride > (size_t)INT64_MAX) return fail(MVB_ERR_ARG, "mvb_herk_batch: bad arguments");
    int rc = check_herk_group("mvb_herk_batch", e.z, (int64_t)e.z_stride, e.ngroup, mode, e.Mpad, e.Kcap, e.n_dev,
                              e.n_host, e.kmul, e.k_chunk, e.ws, e.ws_bytes, e.status);
    if (rc) return rc;
    if (table.n + e.ngroup > kMaxBatchPanels)
      return fail(MVB_ERR_ARG, "mvb_herk_batch: more than %d panels in one launch", kMaxBatchPanels);
    const int T = (int)(e.Mpad / 128);
    for (int j = 0; j < e.ngroup; ++j) {
      HerkPanel &p = table.p[table.n++];
      p.panel = static_cast<const uint8_t *>(e.z) + (int64_t)j * (int64_t)e.z_stride;
      p.n_dev = e.n_dev;
      p.partials = static_cast<float *>(e.ws);
      p.status = e.status;
      p.n_host = e.n_host;
      p.Kcap = e.Kcap;
      p.T = T;
      p.kmul = e.kmul;
      p.k_chunk = e.k_chunk;
      p.plan_tiles = e.ngroup * (T * (T + 1) / 2);
      p.index = j;
    }
  }
  const mvb_herk_group &e0 = groups[0];
  return herk_impl("mvb_herk_batch", e0.z, 0, 1, mode, e0.Mpad, e0.Kcap, e0.n_dev, e0.n_host, e0.kmul, e0.k_chunk,
                   drain_ksteps, e0.ws, e0.ws_bytes, nullptr, stream, table);
}

extern "C" int mvb_herk_reduce(const void *ws, size_t ws_bytes, int64_t Mpad, int64_t Kcap, const int32_t *n_dev,
                               int64_t n_host, int kmul, int k_chunk, int nant, int nfeed, const int32_t *pairs,
                               int64_t npairs, void *out, int out_c128, double vscale, int accumulate, void *stream) {
  return reduce_impl("mvb_herk_reduce", ws, ws_bytes, 1, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, nant, nfeed, pairs,
                     npairs, out, 0, out_c128, vscale, nullptr, accumulate, stream);
}

extern "C" int mvb_herk_reduce_scaled(const void *ws, size_t ws_bytes, int64_t Mpad, int64_t Kcap,
                                      const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int nant, int nfeed,
                                      const int32_t *pairs, int64_t npairs, void *out, int out_c128,
                                      const float *zscale, int accumulate, void *stream) {
  if (!zscale) return fail(MVB_ERR_ARG, "mvb_herk_reduce_scaled: bad arguments");
  return reduce_impl("mvb_herk_reduce_scaled", ws, ws_bytes, 1, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, nant, nfeed,
                     pairs, npairs, out, 0, out_c128, 1.0, zscale, accumulate, stream);
}

extern "C" int mvb_herk_reduce_grouped(const void *ws, size_t ws_bytes, int ngroup, int64_t Mpad, int64_t Kcap,
                                       const int32_t *n_dev, int64_t n_host, int kmul, int k_chunk, int nant,
                                       int nfeed, const int32_t *pairs, int64_t npairs, void *out, size_t out_stride,
                                       int out_c128, double vscale, int accumulate, void *stream) {
  if (out_stride > (size_t)INT64_MAX) return fail(MVB_ERR_ARG, "mvb_herk_reduce_grouped: bad arguments");
  return reduce_impl("mvb_herk_reduce_grouped", ws, ws_bytes, ngroup, Mpad, Kcap, n_dev, n_host, kmul, k_chunk, nant,
                     nfeed, pairs, npairs, out, (int64_t)out_stride, out_c128, vscale, nullptr, accumulate, stream);
}

// ---------------------------------------------------------------------------
// Sum of per-chunk visibilities (MatProd.sum_chunks, core/matprod.py:103-115):
// out[i] = sum_c vis[c][i] in chunk order, accumulated in FP64.
// ---------------------------------------------------------------------------
namespace mvb {
template <typename T>
__global__ void chunk_sum_kernel(const T *__restrict__ vis, int64_t nchunks, int64_t n, T *__restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double re = 0.0, im = 0.0;
    for (int64_t c = 0; c < nchunks; ++c) {
      const T v = vis[c * n + i];
      re += (double)v.x;
      im += (double)v.y;
    }
    out[i].x = re;
    out[i].y = im;
  }
}
}  // namespace mvb

extern "C" int mvb_chunk_sum(const void *vis, int64_t nchunks, int64_t n, int c128, void *out, void *stream) {
  if (nchunks < 1 || n < 0 || (n > 0 && (!vis || !out))) return fail(MVB_ERR_ARG, "mvb_chunk_sum: bad arguments");
  if (n == 0) return MVB_OK;
  const int64_t blocks = std::min<int64_t>(ceil_div(n, 256), (int64_t)num_sms() * 8);
  if (c128)
    chunk_sum_kernel<double2><<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(static_cast<const double2 *>(vis),
                                                                               nchunks, n, static_cast<double2 *>(out));
  else
    chunk_sum_kernel<float2><<<(unsigned)blocks, 256, 0, as_stream(stream)>>>(static_cast<const float2 *>(vis),
                                                                              nchunks, n, static_cast<float2 *>(out));
  return check_launch("chunk_sum_kernel");
}
