// Expert FFN for prefill-sized segments on the 5th-generation tensor cores, with the weight operand
// in TENSOR MEMORY; tiles of up to 160 token rows, longer segments are shared out over several.
//
// Formulation (operands swapped so that the ragged token count lands on the MMA's N, which has a
// granularity of 16, and the always-full feature axis on its M = 128):
//     D[feature, token] = W[feature, :] . X[token, :]^T          per expert segment
// It replaces the reference's dequant-to-half + wmma kernels nvfp4_matmul / nvfp4_gate_up
// (crates/colibri-backend/cuda/backend_cuda.cu:1355-1430) and its separate silu_mul launch
// (backend_cuda.cu:3785-3787).
// * A operand: two loading warps copy the packed NVFP4 or FP8 bytes from HBM into a shared-memory
//   ring of k-tiles (cp.async, 3 to 9 slots of 18 or 32 KB); 16 producer warps read them (one thread
//   = one weight row = one TMEM lane), convert them to f16 in registers and write 64 k per stage
//   into a ring of 32-column TMEM slots with tcgen05.st.  A stage holds two weight tiles (gate + up
//   of the same 128 features, or two adjacent 128-feature tiles of down); the ring is three stages
//   deep beside 160-column accumulators, six beside 64-column ones.
// * B operand: up to 160 token rows x 64 k of f16 activations per stage, copied by TMA as ONE box
//   (cp.async.bulk.tensor, 128-byte swizzle, no multicast; one tensor map per box height) into a
//   6-deep shared-memory ring and shared by both weight tiles of the stage.
// * tcgen05.mma kind::f16 with A from tensor memory and B through a shared-memory descriptor, two
//   accumulators of 160 columns fed by one issuing warp, two stages per barrier wait; the epilogue
//   forms act(g, u) or writes the two down tiles.
// Why: with both operands in shared memory an MMA of 128 x 128 x 16 fetches 8 KB per 64 cycles,
// the whole shared-memory bandwidth of an SM, before a single decoded weight is stored there; a kernel
// of that form with tiles of 256 tokens was kept for long segments until this one passed it (16384
// tokens with skewed experts, H 6144, I 2048: 6092 + 3241 us against 4990 + 2570).  Here shared memory
// carries the token tiles (16-20 KB written + twice that read per stage) and the packed weights (9 or
// 16 KB each way).
// TMEM budget: 2 x 160 accumulator columns + 6 x 32 weight columns = 512, which is why this
// kernel takes tiles of at most 160 tokens (a layer with 128 rows per expert on average has
// nearly all of its segments under that); wider segments are cut into several work items.
// Layers with short segments run a second instantiation with 2 x 64 + 12 x 32 columns.
//
// What bounds it, measured with clock stamps.  An MMA takes N / 2 cycles from 16 tokens up when it is
// issued back to back; the wait for a stage costs the issuing warp about 190 cycles on top, which long
// tiles hide.  With one branch on the lane index per thread of issue, a wait and a commit per stage and
// accumulator, a stage took 830 cycles whatever its tokens (256 of MMA at 64); with weights loaded into
// the producers' registers it stayed there, and with bulk copies in place of cp.async at 728 (the copy
// engine).  Then the producers' instructions: 2700 per k-tile,
// 1100 of them conversions; slot and phase are counters and a wait is a test and a vote since.  Gate+up and down, before and now: 709 tokens
// on H 7168, I 2048, 256 experts 1461 + 771 us -> 1035 + 535 (4.2 GB of weights: 650 + 325 at the copy
// rate); 4096 tokens 2153 + 1170 -> 1900 + 1000 (1320 + 660 at the tensor rate); FP8, 512 tokens, H 2048,
// I 768, 128 experts 130 + 77 -> 92 + 56; NVFP4, 1024 tokens on the same sizes 123 + 71 -> 99 + 56.
//
// Roles are warp-specialised and synchronise through mbarriers only; the kernel is persistent.
// Every barrier wait is bounded: on a time-out the CTA raises a status word, stops issuing work,
// waits for its own copies and frees its TMEM before returning.
#include <type_traits>

#include "tc_common.cuh"

namespace colib {

// TMEM budget (512 columns): two accumulators of ACC columns (= the most token rows of a tile) and a
// weight ring of 64 columns per stage (gate + up, or two down tiles, of 64 k).  ACC = 160 leaves 3
// stages; ACC = 64, for layers whose segments are short, leaves 6: the hand-over of a weight
// stage (fill -> store wait -> barrier -> MMA -> commit -> barrier) is a latency chain of a few
// thousand cycles, so the stage rate of a tile with few tokens grows with the depth of this ring.
template <int ACC>
struct TtBudget {
  static constexpr int A_STAGES = (512 - 2 * ACC) / 64;
  static constexpr int A_COL0 = 2 * ACC;
  static_assert(ACC % 32 == 0 && A_STAGES >= 3 && A_COL0 + A_STAGES * 64 <= 512, "TMEM budget");
  // shared-memory ring of token tiles (ACC rows x 64 k of f16 per stage); its depth is also the
  // number of stage barriers (a ring twice as deep was measured and changed nothing)
  static constexpr int B_BYTES = ACC * TC_BK * 2;
  static constexpr int B_STAGES = 6;
  static constexpr int NBARS = 2 * B_STAGES + 2 + 2 * 9;  // stages, accumulators, at most 9 weight slots
  static_assert(B_STAGES == 6 && (A_STAGES == 3 || A_STAGES == 6) && B_BYTES % 1024 == 0, "a stage barrier serves both rings");
};
// The token tile of a stage arrives as ONE box of N rows: the copy engine of an SM takes about 64
// cycles per box plus 4 per 128-byte row (measured: 21 B/clk with 32-row boxes, 31 B/clk with
// 160-row ones, on 8 SMs as on 148), and at 21 B/clk the 20 KB tile of a 160-token stage takes
// longer than the stage's MMAs.  One tensor map per box height (16, 32, ... rows).
template <int ACC>
struct TtMaps {
  CUtensorMap m[ACC / TC_BOXN];
};
constexpr int TT_PROD_WARPS = 16;
constexpr int TT_LOAD_WARP0 = 2 + TC_EPI_WARPS + TT_PROD_WARPS;      // the two warps that copy weight slabs
constexpr int TT_LOAD_THREADS = 64;
constexpr int TT_THREADS = 32 * TT_LOAD_WARP0 + TT_LOAD_THREADS;     // 768

// The MMAs of one 64-k stage into both accumulators and the commit that releases the stage's
// operands, as one instruction sequence: four k steps of 16 (8 TMEM columns of f16 weights, 32
// bytes = 2 descriptor units of tokens per step); the second tile's weights are 32 columns on.
__device__ __forceinline__ void tt_issue_stage(uint32_t acc0, uint32_t acc1, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate_first, uint32_t bar) {
#pragma unroll
  for (int k4 = 0; k4 < TC_BK / 16; ++k4) {
    umma_f16_ts(acc0, a_tmem + 8 * k4, bdesc + 2 * k4, idesc, k4 ? 1u : accumulate_first);
    umma_f16_ts(acc1, a_tmem + 32 + 8 * k4, bdesc + 2 * k4, idesc, k4 ? 1u : accumulate_first);
  }
  umma_commit(bar);
}
// 32 consecutive columns of this thread's lane
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,"
      "%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// One FP8 word -> two f16x2 (also: four ue4m3 block scales)
__device__ __forceinline__ void tt_cvt_e4m3x4(uint32_t w, uint32_t &p0, uint32_t &p1) {
  asm("{ .reg .b16 h0, h1;\n"
      "  mov.b32 {h0, h1}, %2;\n"
      "  cvt.rn.f16x2.e4m3x2 %0, h0;\n"
      "  cvt.rn.f16x2.e4m3x2 %1, h1; }\n"
      : "=r"(p0), "=r"(p1)
      : "r"(w));
}
// The 64 weights (32 packed bytes) and 4 block-scale bytes of one row for one 64-k stage.
struct TtPacked {
  uint4 q0, q1;
  uint32_t sc;
};
// `codes` = address of the row's chunk 0 (chunks are permuted by XOR, so chunk j is at codes ^ 16 j),
// `scales` = address of its scale bytes; `half` = which 64 of the k-tile's 128 k.
__device__ __forceinline__ TtPacked tt_read_packed(uint32_t codes, uint32_t scales, int half) {
  TtPacked r;
  const uint32_t a = codes ^ (uint32_t)(half << 5);
  r.q0 = lds128(a);
  r.q1 = lds128(a ^ 16u);
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r.sc) : "r"(scales + half * 4) : "memory");
  return r;
}
// Convert one stage of one row: one conversion and one multiply per pair of weights (the multiply takes
// either half of the scale pair as its operand, so the scales need no spreading).
__device__ __forceinline__ void tt_convert(const TtPacked &pk, uint32_t (&r)[32]) {
  const uint32_t w[8] = {pk.q0.x, pk.q0.y, pk.q0.z, pk.q0.w, pk.q1.x, pk.q1.y, pk.q1.z, pk.q1.w};
  uint32_t s01, s23;
  tt_cvt_e4m3x4(pk.sc, s01, s23);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const __half2 pair = *reinterpret_cast<const __half2 *>(j < 4 ? &s01 : &s23);
    const __half2 m = (j & 2) ? __high2half2(pair) : __low2half2(pair);
    uint4 o;
    asm("{ .reg .b8 b0, b1, b2, b3;\n"
        "  mov.b32 {b0, b1, b2, b3}, %4;\n"
        "  cvt.rn.f16x2.e2m1x2 %0, b0;\n"
        "  cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        "  cvt.rn.f16x2.e2m1x2 %2, b2;\n"
        "  cvt.rn.f16x2.e2m1x2 %3, b3; }\n"
        : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
        : "r"(w[j]));
    const uint32_t v[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const __half2 z = __hmul2_rn(*reinterpret_cast<const __half2 *>(&v[q]), m);
      r[4 * j + q] = *reinterpret_cast<const uint32_t *>(&z);
    }
  }
}

// FP8 (e4m3 codes, one byte per weight): the 64 codes of one row for one 64-k stage and the
// multiplier of the stage.  A weight is code x scale[row block][k-tile] (convert.rs:731-741, f32);
// the accumulator runs over all of K inside tensor memory, so the scale cannot be applied per
// k-tile to partial sums as the decode kernel does.  Instead each 128-row tile is
// normalised by the largest scale of its row block: the stage's codes are multiplied by
// TT_FP8_HEADROOM x scale / max scale (an f16 in (0, 16], one rounding of 2^-11 relative per weight)
// and the epilogue multiplies the finished sum by max scale / TT_FP8_HEADROOM in f32.  The
// headroom keeps products of small codes with small relative scales out of the f16 subnormals.
// Per-row scales (linear.rs:93-109) need no multiplier: the epilogue thread owns one row.
constexpr float TT_FP8_HEADROOM = 16.0f;
struct TtPacked8 {
  uint4 q[4];
  uint32_t mult;  // f16 multiplier in both halves
};
__device__ __forceinline__ uint32_t tt_f16x2_both(float v) {
  const __half2 h = __float2half2_rn(v);
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ TtPacked8 tt_read_packed8(uint32_t codes, int half, uint32_t mult) {
  TtPacked8 r;
#pragma unroll
  for (int j = 0; j < 4; ++j) r.q[j] = lds128(codes ^ (uint32_t)((half << 6) | (j << 4)));
  r.mult = mult;
  return r;
}
template <int FMT>
__device__ __forceinline__ void tt_convert8(const TtPacked8 &pk, uint32_t (&r)[32]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 v = pk.q[j];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      tt_cvt_e4m3x4(w[i], r[8 * j + 2 * i], r[8 * j + 2 * i + 1]);
      if (FMT == COLI_FMT_FP8_B128) {
        r[8 * j + 2 * i] = tc_hmul2(r[8 * j + 2 * i], pk.mult);
        r[8 * j + 2 * i + 1] = tc_hmul2(r[8 * j + 2 * i + 1], pk.mult);
      }
    }
  }
}
// Largest scale of one row block over all k-tiles; a warp's lanes share the block and the loads.
__device__ __forceinline__ float tt_block_scale_max(const float *srow, int KT, int lane) {
  float m = 0.0f;
  for (int kt = lane; kt < KT; kt += 32) m = fmaxf(m, __ldg(srow + kt));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// Shared memory: the ring of token tiles, then a ring of packed weight slabs -- both tiles of a stage,
// one k-tile of 128 k (two stages) per slot -- that two warps fill with 16-byte cp.async copies, far
// ahead of the producer warps.  A slab is one contiguous run of bytes in HBM.  (Bulk copies were
// measured too: the copy engine that brings the token tiles then moves 17 KB per stage of 64 tokens
// at about 23 bytes per clock and is what the kernel waits for.)
template <int FMT, int ACC>
struct TtWeightRing {
  static constexpr int SLAB = FMT == COLI_FMT_NVFP4 ? TC_BM * (64 + 8) : TC_BM * 128;
  static constexpr int SLOT = 2 * SLAB;
  static constexpr int SLOTS = FMT == COLI_FMT_NVFP4 ? (ACC <= 64 ? 9 : 5) : (ACC <= 64 ? 5 : 3);
  static constexpr int BYTES = SLOT * SLOTS;
};

// Whole-warp wait: the common case, a phase that has completed, costs a test and a vote.  (Kept inline:
// with the rest behind a call the producers' registers no longer fit and 160-row tiles lost 8 %.)
__device__ __forceinline__ bool tt_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, int code) {
  return __all_sync(0xffffffffu, mbar_test_wait(bar, parity)) ||
         __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, code));
}

// GATED: the two weight tiles of a stage are gate and up of the same 128 features, result
// h = act(g, u).  Otherwise: two adjacent 128-feature tiles of the down projection, result y.
template <bool GATED, int FMT, int ACC>
__global__ void __launch_bounds__(TT_THREADS, 1) k_ffn_tct(const __grid_constant__ TtMaps<ACC> maps, TcParams p) {
  constexpr int TT_A_STAGES = TtBudget<ACC>::A_STAGES, TT_A_COL0 = TtBudget<ACC>::A_COL0, TT_ACC_COLS = ACC;
  constexpr int TT_B_STAGES = TtBudget<ACC>::B_STAGES, TT_B_BYTES = TtBudget<ACC>::B_BYTES, TT_NBARS = TtBudget<ACC>::NBARS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  using Ring = TtWeightRing<FMT, ACC>;
  const uint32_t wring = smem_u32(smem + TT_B_STAGES * TT_B_BYTES);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + TT_B_STAGES * TT_B_BYTES + Ring::BYTES);
  // filled[s], s even: both operands of stages s and s + 1 (a k-tile), 8 producer warps + the TMA
  // thread's expect_tx arrival; the issuing warp pays one wait for the two.  drained[s]: the commit
  // behind stage s.  The tensor-memory ring is shallower, so a producer about to fill stage `it`
  // waits for drained of stage it - TT_A_STAGES.
  const uint32_t full_s = smem_u32(bars), empty_s = smem_u32(bars + TT_B_STAGES);
  const uint32_t acc_full = smem_u32(bars + TT_NBARS - 2), acc_empty = smem_u32(bars + TT_NBARS - 1);
  // weight slots: filled by the copies of the loading warps, read by the eight producer warps of their k-tile
  const uint32_t wfull = smem_u32(bars + 2 * TT_B_STAGES), wempty = smem_u32(bars + 2 * TT_B_STAGES + Ring::SLOTS);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + TT_NBARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = GATED ? p.H : p.I, Oout = GATED ? p.I : p.H;
  const int Op = (Oout + 15) & ~15;
  const int KB = ((K + 127) >> 7) * 2;      // 64-wide k blocks, covering the zero-padded k tiles
  const int FT = GATED ? TC_BM : 2 * TC_BM;  // output features per tile
  const int n_ftiles = (Oout + FT - 1) / FT;

  if (threadIdx.x == 0) {
    for (int s = 0; s < TT_B_STAGES; ++s) {
      mbar_init(full_s + 8 * s, 9);
      mbar_init(empty_s + 8 * s, 1);
    }
    for (int s = 0; s < Ring::SLOTS; ++s) {
      mbar_init(wfull + 8 * s, TT_LOAD_THREADS);
      mbar_init(wempty + 8 * s, TT_PROD_WARPS / 2);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, TC_EPI_WARPS);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  coli_grid_dependency_sync();  // (the set-up above overlaps the predecessor's end)
  const int n_work = *p.n_items * n_ftiles;

  if (warp == 0) {
    // ---------------- TMA: token tiles ----------------
    if (lane == 0) {
      uint32_t it = 0;
      bool alive = true;
      for (int w = blockIdx.x; w < n_work && alive; w += gridDim.x) {
        const int item = w / n_ftiles;
        const int row0 = p.item_row0[item], nrows = p.item_nrows[item];
        const int N = (nrows + TC_BOXN - 1) / TC_BOXN * TC_BOXN;
        const CUtensorMap *tmap = &maps.m[N / TC_BOXN - 1];  // the map whose box is N rows
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const uint32_t s = it % TT_B_STAGES, ph = (it / TT_B_STAGES) & 1u;
          if (!mbar_wait(empty_s + 8 * s, ph ^ 1u, abort_flag, p.status, TC_ERR_TMA_WAIT)) {
            alive = false;
            break;
          }
          const uint32_t dst = smem_u32(smem + s * TT_B_BYTES);
          const uint32_t full = full_s + 8 * (s & ~1u);  // (both rings of stages and k are even)
          if (!(kb & 1)) mbar_expect_tx(full, (uint32_t)N * TC_BK * 4);
          tma_load_2d(dst, tmap, kb * TC_BK, row0, full);
        }
      }
      if (!alive) {
        // copies already issued still land in this CTA's shared memory: give them time before exit
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
      }
    }
  } else if (warp >= TT_LOAD_WARP0) {
    // ---------------- packed weight slabs: HBM -> shared memory ----------------
    const int tid = (int)threadIdx.x - TT_LOAD_WARP0 * 32;
    constexpr int QB = FMT == COLI_FMT_NVFP4 ? 64 : 128;        // code bytes of a row
    constexpr int SB = FMT == COLI_FMT_NVFP4 ? 8 : 0;           // scale bytes of a row
    constexpr int QI = TC_BM * QB / 16 / TT_LOAD_THREADS;       // chunks per thread: the codes of one tile
    constexpr int SI = TC_BM * SB / 16 / TT_LOAD_THREADS;       // ... and its scales
    static_assert(2 * (QI + SI) * TT_LOAD_THREADS * 16 == Ring::SLOT, "slab split");
    uint32_t slot = 0, ph = 0;
    bool alive = true;
    for (int w = blockIdx.x; w < n_work && alive; w += gridDim.x) {
      const int item = w / n_ftiles, ft = w % n_ftiles;
      const int seg = p.item_seg[item];
      const int ex = p.seg_expert ? p.seg_expert[seg] : seg;
      const WeightRef wt[2] = {GATED ? p.gate[ex] : p.down[ex], GATED ? p.up[ex] : p.down[ex]};
      // this thread's first chunk of each tile's codes and scales; the next k-tile is Op rows on
      const uint8_t *qsrc[2], *ssrc[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const size_t row0 = (size_t)ft * FT + (GATED ? 0 : m * TC_BM);
        qsrc[m] = wt[m].q + row0 * QB + tid * 16;
        ssrc[m] = wt[m].s + row0 * SB + tid * 16;
      }
      const bool whole = ft * FT + FT <= Op;
      // ... and how many it has of them: rows past the end of the matrix have none
      int qn[2], sn[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int n = max(0, min(TC_BM, Op - (ft * FT + (GATED ? 0 : m * TC_BM))));
        qn[m] = (n * QB - tid * 16 + TT_LOAD_THREADS * 16 - 1) / (TT_LOAD_THREADS * 16);
        sn[m] = tid * 16 < n * SB ? SI : 0;
      }
      for (int kt = 0; kt < (KB >> 1); ++kt) {
        if (!tt_wait(wempty + 8 * slot, ph ^ 1u, abort_flag, p.status, TC_ERR_TMA_WAIT)) {
          alive = false;
          break;
        }
        const uint32_t dst = wring + slot * Ring::SLOT + tid * 16;
        if (whole) {
#pragma unroll
          for (int m = 0; m < 2; ++m) {
#pragma unroll
            for (int i = 0; i < QI; ++i)
              cp_async16(dst + m * Ring::SLAB + i * TT_LOAD_THREADS * 16, qsrc[m] + i * TT_LOAD_THREADS * 16);
#pragma unroll
            for (int i = 0; i < SI; ++i)
              cp_async16(dst + m * Ring::SLAB + TC_BM * QB + i * TT_LOAD_THREADS * 16, ssrc[m] + i * TT_LOAD_THREADS * 16);
          }
        } else {
          // Rows past the end keep what the slot held before: a feature is a row of the accumulator of its
          // own, and no feature past the end is stored.  A loop with an address, a bound and a zero fill per
          // chunk made such a tile take twice the time of a whole one, and a layer of few tiles waits for it:
          // kernels of a group of 11 experts, H 3960, I 792, 178 rows, per-row FP8 118 -> 49 us, NVFP4 82 ->
          // 45 (I 768: 45 and 44); 17 experts, H 5808, I 608, 862 rows 170 -> 86 and 125 -> 84.
#pragma unroll
          for (int m = 0; m < 2; ++m) {
#pragma unroll
            for (int i = 0; i < QI; ++i)
              if (i < qn[m]) cp_async16(dst + m * Ring::SLAB + i * TT_LOAD_THREADS * 16, qsrc[m] + i * TT_LOAD_THREADS * 16);
#pragma unroll
            for (int i = 0; i < SI; ++i)
              if (i < sn[m])
                cp_async16(dst + m * Ring::SLAB + TC_BM * QB + i * TT_LOAD_THREADS * 16, ssrc[m] + i * TT_LOAD_THREADS * 16);
          }
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          qsrc[m] += (size_t)Op * QB;
          ssrc[m] += (size_t)Op * SB;
        }
        // arrives when this thread's copies up to here have landed
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(wfull + 8 * slot) : "memory");
        if (++slot == Ring::SLOTS) {
          slot = 0;
          ph ^= 1u;
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // nothing is in flight when this thread leaves
  } else if (warp == 1) {
    // ---------------- MMA issue ----------------
    // The whole warp walks the loop and one elected lane issues, and every operand is a value the
    // compiler knows to be the same in all lanes (constants, loop counters, warp reductions): an MMA
    // takes its descriptors and addresses from uniform registers, and moving them there one by one
    // under a branch on the lane index cost as much of this instruction stream as the MMAs themselves.
    // Measured alone, with a barrier wait and a commit per stage: 317 cycles for the eight MMAs of 32
    // tokens, 373 for 64, 640 (the tensor pipe's N / 2 each) for 160, the wait being about 190 of them
    // that only the longer MMAs hide; two warps with an accumulator each take 435, 435 and 640.
    const uint32_t tmem_u = __reduce_max_sync(0xffffffffu, tmem_base);
    const uint64_t bdesc_ring = umma_smem_desc(smem_u32(smem));  // token-tile stage 0; stages are TT_B_BYTES apart
    const uint32_t a_ring = tmem_u + TT_A_COL0;
    uint32_t tix = 0;
    bool alive = true;
    // ring positions as counters: no division or modulo per stage
    uint32_t sb = 0, phb = 0;
    for (int w = blockIdx.x; w < n_work && alive; w += gridDim.x, ++tix) {
      const int item = w / n_ftiles;
      const int nrows = __reduce_max_sync(0xffffffffu, p.item_nrows[item]);
      const int N = (nrows + TC_BOXN - 1) / TC_BOXN * TC_BOXN;
      const uint32_t idesc = umma_idesc(N);
      alive = tt_wait(acc_empty, (tix & 1u) ^ 1u, abort_flag, p.status, TC_ERR_MMA_WAIT);
      if (!alive) break;
      tc_fence_after();
      for (int kb = 0; kb < KB; kb += 2) {
        alive = tt_wait(full_s + 8 * sb, phb, abort_flag, p.status, TC_ERR_MMA_WAIT);
        if (!alive) break;
        tc_fence_after();
        if (elect_one()) {
          // one copy of the code per ring position: every address is then a constant offset
          auto issue = [&](auto pos) {
            constexpr uint32_t b = 2 * decltype(pos)::value, a0 = b % TT_A_STAGES, a1 = (b + 1) % TT_A_STAGES;
            tt_issue_stage(tmem_u, tmem_u + TT_ACC_COLS, a_ring + a0 * 64, bdesc_ring + (uint64_t)(b * (TT_B_BYTES >> 4)), idesc,
                           kb ? 1u : 0u, empty_s + 8 * b);
            tt_issue_stage(tmem_u, tmem_u + TT_ACC_COLS, a_ring + a1 * 64, bdesc_ring + (uint64_t)((b + 1) * (TT_B_BYTES >> 4)), idesc,
                           1u, empty_s + 8 * (b + 1));
          };
          if (sb == 0)
            issue(std::integral_constant<uint32_t, 0>());
          else if (sb == 2)
            issue(std::integral_constant<uint32_t, 1>());
          else
            issue(std::integral_constant<uint32_t, 2>());
        }
        __syncwarp();
        if ((sb += 2) == TT_B_STAGES) {
          sb = 0;
          phb ^= 1u;
        }
      }
      if (alive && elect_one()) umma_commit(acc_full);
      __syncwarp();
    }
  } else if (warp < 2 + TC_EPI_WARPS) {
    // ---------------- epilogue: TMEM -> registers -> global ----------------
    const int lg = warp & 3;  // TMEM lane group this warp may read
    uint32_t tix = 0;
    for (int w = blockIdx.x; w < n_work; w += gridDim.x, ++tix) {
      const int item = w / n_ftiles, ft = w % n_ftiles;
      const int seg = p.item_seg[item], row0 = p.item_row0[item], nrows = p.item_nrows[item];
      const int ex = p.seg_expert ? p.seg_expert[seg] : seg;
      const int N = (nrows + TC_BOXN - 1) / TC_BOXN * TC_BOXN;
      const int f = ft * FT + lg * 32 + lane;  // accumulator 0; accumulator 1 is feature f + 128 of down
      const WeightRef w0 = GATED ? p.gate[ex] : p.down[ex], w1 = GATED ? p.up[ex] : p.down[ex];
      float s0 = w0.g, s1 = w1.g;
      if (FMT == COLI_FMT_FP8_B128) {
        // undo the per-tile normalisation of the producers (both tiles of a stage are 128-row aligned)
        const int KT = KB >> 1;
        const int rb0 = (ft * FT) >> 7, rb1 = GATED ? rb0 : rb0 + 1, nrb = (Oout + 127) >> 7;
        s0 = tt_block_scale_max(reinterpret_cast<const float *>(w0.s) + (size_t)rb0 * KT, KT, lane) * (1.0f / TT_FP8_HEADROOM);
        s1 = rb1 < nrb ? tt_block_scale_max(reinterpret_cast<const float *>(w1.s) + (size_t)rb1 * KT, KT, lane) * (1.0f / TT_FP8_HEADROOM) : 0.0f;
      } else if (FMT == COLI_FMT_E4M3_ROW) {
        const int f1 = GATED ? f : f + TC_BM;
        s0 = f < Oout ? __ldg(reinterpret_cast<const float *>(w0.s) + f) : 0.0f;
        s1 = f1 < Oout ? __ldg(reinterpret_cast<const float *>(w1.s) + f1) : 0.0f;
      }
      bool ok = true;
      if (lane == 0) ok = mbar_wait(acc_full, tix & 1u, abort_flag, p.status, TC_ERR_EPI_WAIT);
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
      if (!ok) break;
      tc_fence_after();
      const uint32_t tbase = tmem_base + ((uint32_t)(lg * 32) << 16);
      for (int c0 = 0; c0 < N; c0 += 16) {
        uint32_t g[16], u[16];
        tmem_ld16(tbase + c0, g);
        tmem_ld16(tbase + TT_ACC_COLS + c0, u);
        tmem_ld_wait();
        // all 16 columns are computed first, branch-free, so that their dependent chains (scale,
        // exponential, reciprocal, two roundings) overlap; a branch per column would run them one
        // after the other.  Columns beyond the item's rows hold other rows' sums and are not stored.
        const int fq = f & ~3;  // first feature of this lane's quad
        const int cols_valid = nrows - c0;
        if (GATED) {
          uint32_t pk[8];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            pk[j] = tc_pack_f16x2_via_bf16(coli_act_fast(__uint_as_float(g[2 * j]) * s0, __uint_as_float(u[2 * j]) * s1, p.act),
                                           coli_act_fast(__uint_as_float(g[2 * j + 1]) * s0, __uint_as_float(u[2 * j + 1]) * s1, p.act));
          tc_store_cols16(pk, p.h + (size_t)(row0 + c0) * Oout + fq, (size_t)Oout, cols_valid, fq < Oout, lane);
        } else {
          uint32_t pk0[8], pk1[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            pk0[j] = tc_pack_bf16x2(__uint_as_float(g[2 * j]) * s0, __uint_as_float(g[2 * j + 1]) * s0);
            pk1[j] = tc_pack_bf16x2(__uint_as_float(u[2 * j]) * s1, __uint_as_float(u[2 * j + 1]) * s1);
          }
          __nv_bfloat16 *yq = p.y + (size_t)(row0 + c0) * Oout + fq;
          tc_store_cols16(pk0, yq, (size_t)Oout, cols_valid, fq < Oout, lane);
          tc_store_cols16(pk1, yq + TC_BM, (size_t)Oout, cols_valid, fq + TC_BM < Oout, lane);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
    }
  } else {
    // ---------------- weight producers: shared memory -> registers -> f16 -> tensor memory ----------------
    // four groups of four warps (128 lanes = 128 weight rows each): group g converts weight tile
    // (g & 1) of the k-tiles whose running index has parity (g >> 1), two stages each
    const int grp = (warp - 2 - TC_EPI_WARPS) >> 2;
    const int mtx = grp & 1, par = grp >> 1;
    const int quarter = warp & 3;  // TMEM lane quarter this warp may write
    const int row = quarter * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + TT_A_COL0 + mtx * 32;
    const int KT = KB >> 1;
    const uint32_t code_off = FMT == COLI_FMT_NVFP4 ? row * 64 + coli_fp4_chunk(row, 0) * 16 : row * 128 + coli_fp8_chunk(row, 0) * 16;
    int ahead = par;   // k-tiles from the start of the tile to this group's next one
    uint32_t wslot = par, wph = 0;
    // stage barrier of the group's next stage (0, 2 or 4 of 6) and the phase of that round
    uint32_t sb = 2 * par, ph = 0;
    bool alive = true;
    for (int w = blockIdx.x; w < n_work && alive; w += gridDim.x) {
      const float *srow = nullptr;
      float norm = 0.0f, scale = 0.0f;
      int kt = ahead;
      if constexpr (FMT == COLI_FMT_FP8_B128) {
        const int item = w / n_ftiles, ft = w % n_ftiles, seg = p.item_seg[item];
        const int ex = p.seg_expert ? p.seg_expert[seg] : seg;
        const WeightRef wr = GATED ? (mtx ? p.up[ex] : p.gate[ex]) : p.down[ex];
        // (a second tile past the end has no scale row, and none of it is stored)
        const int rb = min(GATED ? ft : 2 * ft + mtx, (Oout - 1) >> 7);
        srow = reinterpret_cast<const float *>(wr.s) + (size_t)rb * KT;
        // a row block whose scales are all zero (an all-zero or padded weight block: the encoder
        // writes scale = amax / 448 = 0) decodes to zeros, as code x 0 does in convert.rs:731-741
        const float mx = tt_block_scale_max(srow, KT, lane);
        norm = mx > 0.0f ? TT_FP8_HEADROOM / mx : 0.0f;
        scale = kt < KT ? __ldg(srow + kt) : 0.0f;
      }
      for (; kt < KT; kt += 2) {
        if (!tt_wait(wfull + 8 * wslot, wph, abort_flag, p.status, TC_ERR_PROD_WAIT)) {
          alive = false;
          break;
        }
        const uint32_t slab = wring + wslot * Ring::SLOT + mtx * Ring::SLAB;
        const uint32_t codes = slab + code_off;
        const uint32_t mult = FMT == COLI_FMT_FP8_B128 ? tt_f16x2_both(scale * norm) : 0x3c003c00u /* 1.0 */;
        if (FMT == COLI_FMT_FP8_B128 && kt + 2 < KT) scale = __ldg(srow + kt + 2);
#pragma unroll
        for (uint32_t half = 0; half < 2; ++half) {
          // The conversion runs BEFORE the wait for the tensor-memory slot, so that only the store stands
          // between the slot's release and the barrier that hands it to the issuing warp.
          uint32_t r[32];
          if constexpr (FMT == COLI_FMT_NVFP4)
            tt_convert(tt_read_packed(codes, slab + TC_BM * 64 + row * 8, half), r);
          else
            tt_convert8<FMT>(tt_read_packed8(codes, half, mult), r);
          if (half == 1) {  // the slab has been read
            __syncwarp();
            if (lane == 0) mbar_arrive(wempty + 8 * wslot);
          }
          // The slot was last read by the stage TT_A_STAGES earlier: the same barrier one round ago with six
          // slots, the one three on (of this round for the later three) with three.  A wait for the round
          // before the first returns at once.
          const uint32_t st = sb + half;
          const uint32_t eb = TT_A_STAGES == 6 ? st : (st >= 3 ? st - 3 : st + 3);
          const uint32_t ep = TT_A_STAGES == 6 || st < 3 ? ph ^ 1u : ph;
          if (!tt_wait(empty_s + 8 * eb, ep, abort_flag, p.status, TC_ERR_PROD_WAIT)) {
            alive = false;
            break;
          }
          tc_fence_after();
          tmem_st32(taddr + (TT_A_STAGES == 6 ? st : (st >= 3 ? st - 3 : st)) * 64, r);
        }
        if (!alive) break;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full_s + 8 * sb);
        if ((wslot += 2) >= (uint32_t)Ring::SLOTS) {
          wslot -= Ring::SLOTS;
          wph ^= 1u;
        }
        if ((sb += 4) >= (uint32_t)TT_B_STAGES) {
          sb -= TT_B_STAGES;
          ph ^= 1u;
        }
      }
      ahead = kt - KT;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

template <bool GATED, int FMT, int ACC>
static int launch_tct(const TcParams &p, const void *rows_base, int rows_cap, int sm_count, cudaStream_t st) {
  const size_t smem = (size_t)TtBudget<ACC>::B_STAGES * TtBudget<ACC>::B_BYTES + TtWeightRing<FMT, ACC>::BYTES + 1024 /*align*/ + 8 * TtBudget<ACC>::NBARS + 16 + 64;
  static ColiPerDeviceOnce attr_once;
  if (!coli_set_smem_limit(attr_once, k_ffn_tct<GATED, FMT, ACC>, smem, "tcgen05 kernel shared-memory attribute")) return 0;
  TtMaps<ACC> maps;
  for (int j = 0; j < ACC / TC_BOXN; ++j)
    if (!make_rows_map(&maps.m[j], rows_base, rows_cap, GATED ? p.H : p.I, (j + 1) * TC_BOXN)) return 0;
  const int FT = GATED ? TC_BM : 2 * TC_BM;
  const int n_ftiles = ((GATED ? p.I : p.H) + FT - 1) / FT;
  const long max_work = (long)p.max_items * n_ftiles;
  const int grid = (int)(max_work < sm_count ? max_work : sm_count);
  if (grid <= 0) return 1;
  coli_count_launch(1);
  return coli_cuda_check(launch_dependent(k_ffn_tct<GATED, FMT, ACC>, dim3(grid), dim3(TT_THREADS), smem, st, maps, p), "tcgen05 expert ffn launch") ? 1 : 0;
}
template <bool GATED, int FMT>
static int launch_tct_acc(const TcParams &p, const void *rows_base, int rows_cap, int sm_count, cudaStream_t st) {
  if (p.tile_tokens == TCT_SHORT_TOKENS) return launch_tct<GATED, FMT, TCT_SHORT_TOKENS>(p, rows_base, rows_cap, sm_count, st);
  if (p.tile_tokens == TCT_MAX_TOKENS) return launch_tct<GATED, FMT, TCT_MAX_TOKENS>(p, rows_base, rows_cap, sm_count, st);
  coli_set_error("tcgen05 expert ffn: the work list must be cut with %d or %d rows per item, not %d", TCT_SHORT_TOKENS, TCT_MAX_TOKENS,
                 p.tile_tokens);
  return 0;
}
template <bool GATED>
static int launch_tct_fmt(const TcParams &p, const void *rows_base, int rows_cap, int sm_count, cudaStream_t st) {
  switch (p.fmt) {
    case COLI_FMT_NVFP4:
      return launch_tct_acc<GATED, COLI_FMT_NVFP4>(p, rows_base, rows_cap, sm_count, st);
    case COLI_FMT_FP8_B128:
      return launch_tct_acc<GATED, COLI_FMT_FP8_B128>(p, rows_base, rows_cap, sm_count, st);
    case COLI_FMT_E4M3_ROW:
      return launch_tct_acc<GATED, COLI_FMT_E4M3_ROW>(p, rows_base, rows_cap, sm_count, st);
  }
  coli_set_error("tcgen05 expert ffn: unsupported weight format %d", p.fmt);
  return 0;
}

int launch_gate_up_tct(const TcParams &p, const void *x_rows, int rows_cap, int sm_count, cudaStream_t st) {
  return launch_tct_fmt<true>(p, x_rows, rows_cap, sm_count, st);
}
int launch_down_tct(const TcParams &p, int rows_cap, int sm_count, cudaStream_t st) {
  return launch_tct_fmt<false>(p, p.h, rows_cap, sm_count, st);
}

}  // namespace colib
