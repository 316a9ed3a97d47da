// Routing: router GEMM with a strictly k-ascending f32 sum per logit, score + top-k
// (softmax / sigmoid+bias / group-limited), and the permutation of (token, kk) pairs into
// expert-contiguous row segments.
//
// Bit-exactness contract.  The CPU restatement of crates/colibri-engine/src/moe.rs:1047-1132
// sums each logit sequentially over k in f32 (linear.rs:199-220), scores with exp, sums the
// softmax denominator sequentially over e, and picks k experts by a strict `>` scan from e = 0.
// Every one of those steps is reproduced here operation for operation:
//   * x and the router weights are bf16, so each product is exact in f32 and one fused
//     multiply-add per k equals the reference's multiply-then-add; each logit is owned by ONE
//     thread that walks k = 0..H-1 in order (no split-K, no tensor cores);
//   * exp / sigmoid come from coli_math.h, compiled identically for host and device;
//   * adds, subs, divides that the compiler could contract or reorder are spelled with the
//     CF_* round-to-nearest intrinsics;
//   * the arg-max of each round is the largest value with the lowest index, which is what the
//     ascending strict-`>` scan returns; a round with no candidate above -inf returns 0.
#include <cmath>

#include "internal.cuh"

namespace colib {

// The counts that the top-k behind a router launch adds to (RouteParams::expert_rows) are cleared by that launch.
__device__ __forceinline__ void clear_expert_rows(const RouteParams &p) {
  if (p.expert_rows && blockIdx.x + blockIdx.y == 0)
    for (int e = threadIdx.x; e < p.E; e += blockDim.x) p.expert_rows[e] = 0;
}

// ---------------------------------------------------------------------------------------------
// Router GEMM, general shape.  Block = 16x16 threads, thread tile TM x TN, k-chunk 32 staged in
// shared memory as f32 (transposed so the inner loop reads broadcast / consecutive words).
// ---------------------------------------------------------------------------------------------
template <int TM, int TN>
__global__ void __launch_bounds__(256) k_router_gemm(RouteParams p) {
  coli_grid_dependency_sync();
  clear_expert_rows(p);
  constexpr int BM = 16 * TM, BN = 16 * TN, BK = 32;
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

  for (int k0 = 0; k0 < p.H; k0 += BK) {
    // stage x[m0..m0+BM, k0..k0+32) and w[n0..n0+BN, k0..k0+32), zero beyond the edges
    for (int idx = threadIdx.x; idx < BM * BK; idx += 256) {
      const int r = idx / BK, c = idx % BK;
      const int m = m0 + r, k = k0 + c;
      float v = 0.0f;
      if (m < p.T && k < p.H) v = __bfloat162float(p.x[(size_t)m * p.H + k]);
      xs[c][r] = v;
    }
    for (int idx = threadIdx.x; idx < BN * BK; idx += 256) {
      const int r = idx / BK, c = idx % BK;
      const int n = n0 + r, k = k0 + c;
      float v = 0.0f;
      if (n < p.E && k < p.H) v = __bfloat162float(p.router_w[(size_t)n * p.H + k]);
      ws[c][r] = v;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = xs[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = __fmaf_rn(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int m = m0 + ty * TM + i, n = n0 + tx * TN + j;
      if (m < p.T && n < p.E) {
        float v = acc[i][j];
        if (p.logit_bias) v = __fadd_rn(v, p.logit_bias[n]);
        p.logits[(size_t)m * p.E + n] = v;
      }
    }
}

// Two independent f32 FMAs in one instruction (sm_100): c.x = fma(a.x, b, c.x), c.y = fma(a.y, b, c.y),
// each rounded as a scalar fmaf, so an output's k-ascending chain is unchanged.  Fed from shared memory,
// an 8 x 8 register tile reaches 110 FMAs per clock and SM with it and 94 without (two warps per
// scheduler; 87 and 75 with one).
__device__ __forceinline__ void coli_ffma2(float2 &c, const float2 a, const float b) {
  unsigned long long cc, aa, bb;
  asm("mov.b64 %0, {%1, %2};" : "=l"(cc) : "f"(c.x), "f"(c.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(aa) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %1};" : "=l"(bb) : "f"(b));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(aa), "l"(bb));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c.x), "=f"(c.y) : "l"(cc));
}

// Router GEMM of the large batches (H % 8 == 0): every thread owns TM x TN outputs, each one k-ascending
// fmaf chain, two tokens per FMA instruction; a warp covers 4 TM tokens x 8 TN experts, a CTA WM x WN
// warps.  Operands are staged as f32, k-major, two buffers of 32 k, with 16-byte loads one block ahead;
// a warp's lanes take consecutive rows, so the transposed stores fall into different banks.  CW warps of
// their own do the staging, or (CW = 0) the computing warps between blocks: with one computing warp per
// scheduler, the 8 x 8 tile, staging in between costs 10 % (443 against 403 us with the top-k, 4096
// tokens x 256 experts x 7168), with the 16 x 8 tile and three CTAs per SM the extra warps cost 4 %.
// Bound by FMA issue and the operand reads between them: 16384 x 384 x 6144 1894 -> 1617 us, 103 FMAs
// per clock and SM of the SM's 128 while its last CTAs keep it full.
template <int TM_, int TN_, int WM_, int WN_, int CW_>
struct RouterPairTile {
  static constexpr int TM = TM_, TN = TN_, WM = WM_, WN = WN_, CW = CW_, BK = 32;
  static constexpr int BM = 4 * TM * WM, BN = 8 * TN * WN, ROWS = BM + BN;
  static constexpr int COMPUTE = 32 * WM * WN, NT = COMPUTE + 32 * CW, STAGING = CW ? 32 * CW : COMPUTE;
  static constexpr int LD = ROWS + 4;              // floats per k: tokens, then experts, then padding
  static constexpr int CPT = ROWS * (BK / 8) / STAGING;  // 16-byte chunks a thread stages per block
  static constexpr size_t SMEM = (size_t)2 * BK * LD * 4;
  static_assert(ROWS * (BK / 8) % STAGING == 0 && ROWS % 32 == 0 && TM % 4 == 0 && TN % 4 == 0, "tile shape");
};
template <class C>
__global__ void __launch_bounds__(C::NT) k_router_pair(RouteParams p) {
  coli_grid_dependency_sync();
  clear_expert_rows(p);
  constexpr int TM = C::TM, TN = C::TN, BK = C::BK, LD = C::LD, BM = C::BM;
  extern __shared__ __align__(16) float rsm[];
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * C::BN;
  const int nkb = (p.H + BK - 1) / BK;
  // staging: by the warps behind the computing ones, or by all
  const int tid = C::CW ? (int)threadIdx.x - C::COMPUTE : (int)threadIdx.x;
  uint4 v[C::CPT];
  auto fetch = [&](int kb) {
#pragma unroll
    for (int i = 0; i < C::CPT; ++i) {
      const int idx = i * C::STAGING + tid, r = idx % C::ROWS, k = kb * BK + idx / C::ROWS * 8;
      const int row = r < BM ? m0 + r : n0 + r - BM;
      v[i] = make_uint4(0, 0, 0, 0);
      if (row < (r < BM ? p.T : p.E) && k < p.H)
        v[i] = *reinterpret_cast<const uint4 *>((r < BM ? p.x : p.router_w) + (size_t)row * p.H + k);
    }
  };
  auto stage = [&](int kb) {
    float *dst = rsm + (kb & 1) * (BK * LD);
#pragma unroll
    for (int i = 0; i < C::CPT; ++i) {
      const int idx = i * C::STAGING + tid, r = idx % C::ROWS, k = idx / C::ROWS * 8;
      const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        dst[(k + 2 * j) * LD + r] = __uint_as_float(u[j] << 16);
        dst[(k + 2 * j + 1) * LD + r] = __uint_as_float(u[j] & 0xffff0000u);
      }
    }
  };
  if (C::CW && threadIdx.x >= C::COMPUTE) {  // block kb + 1 is stored while block kb is multiplied
    fetch(0);
    stage(0);
    if (nkb > 1) fetch(1);
    for (int kb = 0; kb < nkb; ++kb) {
      __syncthreads();
      if (kb + 1 < nkb) {
        stage(kb + 1);  // that buffer was last read one barrier ago
        if (kb + 2 < nkb) fetch(kb + 2);
      }
    }
    return;
  }
  // ---------------- computing warps ----------------
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = (warp / C::WN) * 4 * TM + (lane >> 3) * TM;         // this thread's first token of the tile
  const int nt = (warp % C::WN) * 8 * TN + (lane & 7) * 4;           // and first expert; the others 32 q + j on
  if (!C::CW) {
    fetch(0);
    stage(0);
    if (nkb > 1) fetch(1);
  }
  float2 acc[TM / 2][TN];  // .x = token 2 i, .y = token 2 i + 1
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
  for (int kb = 0; kb < nkb; ++kb) {
    __syncthreads();  // block kb is staged
    const float *buf = rsm + (kb & 1) * (BK * LD);
#pragma unroll 4
    for (int kk = 0; kk < BK; ++kk) {
      float4 a[TM / 4], b[TN / 4];
#pragma unroll
      for (int q = 0; q < TM / 4; ++q) a[q] = *reinterpret_cast<const float4 *>(buf + kk * LD + mt + 4 * q);
#pragma unroll
      for (int q = 0; q < TN / 4; ++q) b[q] = *reinterpret_cast<const float4 *>(buf + kk * LD + BM + nt + 32 * q);
#pragma unroll
      for (int i = 0; i < TM / 2; ++i) {
        const float2 ai = (i & 1) ? make_float2(a[i >> 1].z, a[i >> 1].w) : make_float2(a[i >> 1].x, a[i >> 1].y);
#pragma unroll
        for (int j = 0; j < TN; ++j) coli_ffma2(acc[i][j], ai, (&b[j >> 2].x)[j & 3]);
      }
    }
    if (!C::CW && kb + 1 < nkb) {
      stage(kb + 1);  // fetched while this block was multiplied; that buffer was last read one barrier ago
      if (kb + 2 < nkb) fetch(kb + 2);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int m = m0 + mt + i, n = n0 + nt + (j >> 2) * 32 + (j & 3);
      if (m < p.T && n < p.E) {
        float o = (i & 1) ? acc[i >> 1][j].y : acc[i >> 1][j].x;
        if (p.logit_bias) o = __fadd_rn(o, p.logit_bias[n]);
        p.logits[(size_t)m * p.E + n] = o;
      }
    }
}

// Router GEMM for the batches below those of the kernel above (H % 8 == 0): every thread owns
// TM x TN outputs, each one k-ascending fmaf chain; a warp covers 4 TM tokens x 8 TN experts, a CTA
// WM x WN warps.  Token and expert rows travel as bf16, in k-blocks of BK through a ring of STAGES
// cp.async stages, so the loads of the next stages are in flight while one is multiplied; rows are
// padded by 16 bytes, which puts eight consecutive rows of a quarter-warp's 128-bit loads into
// different banks.
// What bounds it: the chain of H dependent FMAs (4.3 cycles each, measured) with few outputs per SM,
// the issue slots otherwise: for 8 k a thread issues 8 TM TN FMAs, 8 (TM + TN) operations that widen
// bf16 to f32 (at half the FMA rate) and TM + TN shared loads.  A small tile spreads few outputs over
// all SMs, a large one spends fewer slots per FMA: pick_router_tile weighs the two.
// Measured with the top-k behind it, against a kernel of 16 to 128 tokens x 64 experts per CTA: 48 tokens x
// 128 experts x 2048 64 -> 15 us, 24 x 256 x 7168 202 -> 33, 512 x 128 x 2048 65 -> 25, 709 x 256 x 7168
// 320 -> 135, 2048 x 256 x 7168 320 -> 264.  (The top-k's own mending is 5 to 12 us of each.)  Staging the
// operands as f32 by warps of their own was built and is slower from 200 tokens on (shared-memory reads).
template <int TM_, int TN_, int WM_, int WN_, int BK_, int STAGES_>
struct RouterTile {
  static constexpr int TM = TM_, TN = TN_, WM = WM_, WN = WN_, BK = BK_, STAGES = STAGES_;
  static constexpr int BM = 4 * TM * WM, BN = 8 * TN * WN, NT = 32 * WM * WN;
  static constexpr int RS = BK * 2 + 16;  // row stride in bytes: an odd multiple of 16
  static constexpr int CH = BK / 8;       // 16-byte chunks of a row
  static constexpr int STAGE_BYTES = (BM + BN) * RS;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES;
  static_assert((RS / 16) % 2 == 1 && (BM + BN) * CH % NT == 0, "row padding / staging split");
};
template <class C>
__global__ void __launch_bounds__(C::NT) k_router_chain(RouteParams p) {
  coli_grid_dependency_sync();
  clear_expert_rows(p);
  constexpr int TM = C::TM, TN = C::TN, RS = C::RS, CH = C::CH, BM = C::BM, BN = C::BN;
  constexpr bool SMALL = TM * TN <= 8;  // the next chunk's operands are loaded ahead of this one's FMAs
  constexpr bool PAIRED = TM % 2 == 0;  // two tokens per FMA instruction (3 to 6 % at every tile that can)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t smem = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int xrow = (warp / C::WN) * 4 * TM + (lane >> 3), wrow = (warp % C::WN) * 8 * TN + (lane & 7);
  const int nkb = (p.H + C::BK - 1) / C::BK;

  auto fetch = [&](int kb) {  // rows of k-block kb; beyond T, E or H they are zeros
    const uint32_t dst = smem + (uint32_t)(kb % C::STAGES) * C::STAGE_BYTES;
#pragma unroll
    for (int i = 0; i < (BM + BN) * CH / C::NT; ++i) {
      const int idx = i * C::NT + (int)threadIdx.x;
      const int r = idx / CH, c = idx % CH, k = kb * C::BK + c * 8;
      const int row = r < BM ? m0 + r : n0 + r - BM;
      const bool valid = row < (r < BM ? p.T : p.E) && k < p.H;
      const __nv_bfloat16 *src = r < BM ? p.x : p.router_w;
      cp_async16(dst + (uint32_t)(r * RS + c * 16), valid ? src + (size_t)row * p.H + k : src, valid);
    }
  };
#pragma unroll
  for (int s = 0; s < C::STAGES - 1; ++s) {
    if (s < nkb) fetch(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
  float2 acc2[(TM + 1) / 2][TN];
#pragma unroll
  for (int i = 0; i < (TM + 1) / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc2[i][j] = make_float2(0.0f, 0.0f);

  for (int kb = 0; kb < nkb; ++kb) {
    asm volatile("cp.async.wait_group %0;" ::"n"(C::STAGES - 2) : "memory");
    __syncthreads();  // block kb has arrived for every thread, and its predecessor's slot is free
    if (kb + C::STAGES - 1 < nkb) fetch(kb + C::STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const uint32_t xs = smem + (uint32_t)(kb % C::STAGES) * C::STAGE_BYTES + (uint32_t)(xrow * RS);
    const uint32_t ws = smem + (uint32_t)(kb % C::STAGES) * C::STAGE_BYTES + (uint32_t)((BM + wrow) * RS);
    uint4 xv[TM], wv[TN];
    auto load = [&](uint4 (&xv)[TM], uint4 (&wv)[TN], int c) {
#pragma unroll
      for (int i = 0; i < TM; ++i) xv[i] = lds128(xs + (uint32_t)(i * 4 * RS + c * 16));
#pragma unroll
      for (int j = 0; j < TN; ++j) wv[j] = lds128(ws + (uint32_t)(j * 8 * RS + c * 16));
    };
    // element q of a chunk: the low or the high half of word q / 2
    auto widen = [](const uint4 &v, int q) {
      const uint32_t w = (&v.x)[q >> 1];
      return __uint_as_float((q & 1) ? w & 0xffff0000u : w << 16);
    };
#pragma unroll(SMALL ? CH : 1)
    for (int c = 0; c < CH; ++c) {
      if (c == 0 || !SMALL) load(xv, wv, c);
      uint4 xc[TM], wc[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) xc[i] = xv[i];
#pragma unroll
      for (int j = 0; j < TN; ++j) wc[j] = wv[j];
      if (SMALL && c + 1 < CH) load(xv, wv, c + 1);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float a[TM], b[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = widen(xc[i], q);
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = widen(wc[j], q);
        if constexpr (PAIRED) {
#pragma unroll
          for (int i = 0; i < TM; i += 2)
#pragma unroll
            for (int j = 0; j < TN; ++j) coli_ffma2(acc2[i / 2][j], make_float2(a[i], a[i + 1]), b[j]);
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = __fmaf_rn(a[i], b[j], acc[i][j]);
        }
      }
    }
  }
  if constexpr (PAIRED) {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = (i & 1) ? acc2[i / 2][j].y : acc2[i / 2][j].x;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int m = m0 + xrow + 4 * i, n = n0 + wrow + 8 * j;
      if (m < p.T && n < p.E) {
        float v = acc[i][j];
        if (p.logit_bias) v = __fadd_rn(v, p.logit_bias[n]);
        p.logits[(size_t)m * p.E + n] = v;
      }
    }
}

// The logits of a decode-sized CTA: one chain per thread of two computing warps, 8 tokens x 8 experts,
// operands staged as f32.  CW staging warps copy 16-byte chunks of the bf16 rows through a ring of
// cp.async stages, widen them and store them into one of two f32 buffers of 256 k, while the computing
// warps read the other three 128-bit loads ahead of the FMAs that use them.  Rows are padded by 16 bytes
// (banks).  A k takes 5.4 cycles (an FMA's latency is 4.3): a barrier costs the chain about 115, which is why
// a block is 256 k long (128: 6.0; 512: 5.3, but its first block is late); loads further ahead or more staging
// warps change nothing.
struct RouterTiny {
  static constexpr int ROWS = 16, BK = 256, LD = BK + 4, CH = BK / 8, STAGES = 4;
  static constexpr int F32_BYTES = ROWS * LD * 4, RING_BYTES = ROWS * BK * 2;
  static constexpr size_t SMEM = (size_t)2 * F32_BYTES + (size_t)STAGES * RING_BYTES;
};
// The first 2 + CW warps of a CTA call this; logits of tokens m0.. and experts n0.. are written.  EARLY: the kernel may
// still be waiting for its predecessor; the router weights, which are older, are requested first, and the staging warps
// wait before they touch the tokens (the others get everything from them).
template <int CW, bool EARLY>
__device__ __forceinline__ void router_tiny_block(const RouteParams &p, unsigned char *smem_raw, int m0, int n0) {
  using C = RouterTiny;
  constexpr int LD = C::LD, CH = C::CH, BK = C::BK, CPT = (C::ROWS * CH + 32 * CW - 1) / (32 * CW);
  float *const buf = reinterpret_cast<float *>(smem_raw);  // [2][ROWS][LD]: 8 tokens, then 8 experts
  const int nkb = (p.H + BK - 1) / BK;
  auto block_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(64 + 32 * CW) : "memory"); };
  if (threadIdx.x >= 64) {
    const int tid = (int)threadIdx.x - 64;
    unsigned char *const ring = smem_raw + 2 * C::F32_BYTES;
    auto fetch = [&](int kb, bool tokens, bool experts) {  // rows of k-block kb; beyond T, E or H they are zeros
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        const int idx = i * 32 * CW + tid, r = idx / CH, k = kb * BK + idx % CH * 8;
        if (idx >= C::ROWS * CH) break;
        if (!(r < 8 ? tokens : experts)) continue;
        const int row = r < 8 ? m0 + r : n0 + r - 8;
        const __nv_bfloat16 *base = r < 8 ? p.x : p.router_w;
        const bool valid = row < (r < 8 ? p.T : p.E) && k < p.H;
        cp_async16((uint32_t)__cvta_generic_to_shared(ring + (kb % C::STAGES) * C::RING_BYTES + idx * 16),
                   valid ? base + (size_t)row * p.H + k : base, valid);
      }
    };
    // a thread reads back only the chunks it copied itself, so its own wait suffices
    auto convert = [&](int kb) {
      asm volatile("cp.async.wait_group %0;" ::"n"(C::STAGES - 1) : "memory");
#pragma unroll
      for (int i = 0; i < CPT; ++i) {
        const int idx = i * 32 * CW + tid;
        if (idx >= C::ROWS * CH) break;
        const uint4 v = *reinterpret_cast<const uint4 *>(ring + (kb % C::STAGES) * C::RING_BYTES + idx * 16);
        float *dst = buf + (kb & 1) * (C::ROWS * LD) + idx / CH * LD + idx % CH * 8;
        const uint32_t hi = 0xffff0000u;
        reinterpret_cast<uint4 *>(dst)[0] = make_uint4(v.x << 16, v.x & hi, v.y << 16, v.y & hi);
        reinterpret_cast<uint4 *>(dst)[1] = make_uint4(v.z << 16, v.z & hi, v.w << 16, v.w & hi);
      }
      if (kb + C::STAGES < nkb) fetch(kb + C::STAGES, true, true);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (EARLY) {
#pragma unroll 1
      for (int s = 0; s < C::STAGES && s < nkb; ++s) fetch(s, false, true);
      coli_grid_wait();
    }
#pragma unroll 1
    for (int s = 0; s < C::STAGES; ++s) {
      if (s < nkb) fetch(s, true, !EARLY);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    convert(0);
    for (int kb = 0; kb < nkb; ++kb) {
      block_barrier();
      if (kb + 1 < nkb) convert(kb + 1);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return;
  }
  const int xrow = (int)threadIdx.x >> 3, wrow = (int)threadIdx.x & 7;
  float acc = 0.0f;
  for (int kb = 0; kb < nkb; ++kb) {
    block_barrier();  // block kb is staged, and nobody reads its predecessor any more
    const float4 *xs = reinterpret_cast<const float4 *>(buf + (kb & 1) * (C::ROWS * LD) + xrow * LD);
    const float4 *ws = reinterpret_cast<const float4 *>(buf + (kb & 1) * (C::ROWS * LD) + (8 + wrow) * LD);
    constexpr int D = 4;  // 128-bit operands in flight or in use
    float4 a[D], b[D];
#pragma unroll
    for (int i = 0; i < D - 1; ++i) {
      a[i] = xs[i];
      b[i] = ws[i];
    }
#pragma unroll
    for (int i = 0; i < BK / 4; ++i) {
      if (i + D - 1 < BK / 4) {
        a[(i + D - 1) % D] = xs[i + D - 1];
        b[(i + D - 1) % D] = ws[i + D - 1];
      }
      acc = __fmaf_rn(a[i % D].x, b[i % D].x, acc);
      acc = __fmaf_rn(a[i % D].y, b[i % D].y, acc);
      acc = __fmaf_rn(a[i % D].z, b[i % D].z, acc);
      acc = __fmaf_rn(a[i % D].w, b[i % D].w, acc);
    }
  }
  const int m = m0 + xrow, n = n0 + wrow;
  if (m < p.T && n < p.E) {
    if (p.logit_bias) acc = __fadd_rn(acc, p.logit_bias[n]);
    p.logits[(size_t)m * p.E + n] = acc;
  }
}
// ---------------------------------------------------------------------------------------------
// Score + top-k: one warp per token.  Expert e lives in lane e % 32, slot e / 32, scores and keys in
// registers; SLOTS >= E / 32 (<= 16) is a template parameter so that every pass over them unrolls into
// independent operations.  What bounds it is the length of one token's dependent chain, whatever the batch
// (clock stamps on a warm SM, 128 experts softmax top-8 / 256 experts sigmoid in 8 groups, cycles):
//   load + maximum 420, exp 940, ordered sum 560, divide 330, keys 260, selection and weights ...
// k rounds of two warp reductions and a rescan of the winning lane's slots cost 250 cycles each (2000 / 2500
// for k = 8), and a group's two best by one lane per group 2750; both are counting steps now (below).
// ---------------------------------------------------------------------------------------------
constexpr int kMaxSlots = 16;  // E <= 512
// Shared memory of one warp: the row of scores (16-byte aligned), and a list of 32 candidates.
struct TopkCand {
  uint32_t key;
  int id;
  float sc;
  uint32_t pad;
};
__host__ __device__ static constexpr int topk_row_floats(int E) { return ((E + 3) & ~3) + 32 * (int)(sizeof(TopkCand) / 4); }

// order-preserving integer key of a candidate (a value strictly above -inf; NaN is none), 0 otherwise
__device__ __forceinline__ uint32_t topk_key(float c) {
  if (!(c > __uint_as_float(0xff800000u))) return 0u;
  const uint32_t bits = __float_as_uint(__fadd_rn(c, 0.0f));  // -0 and +0 tie like the float compare
  return (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
}
__device__ __forceinline__ float topk_key_value(uint32_t key) {
  return key == 0u ? __uint_as_float(0xff800000u) : __uint_as_float((key & 0x80000000u) ? key & 0x7fffffffu : ~key);
}

// The k best of a warp's keys (largest key, then lowest expert id; key 0 = not a candidate) as list entries
// 0..k-1 of `cand`, in order; fewer candidates leave expert 0 behind them, which is what the reference's scan
// returns.  The k-th largest of the lanes' best keys bounds the k-th largest of all from below, so only keys
// from it upwards can be chosen: a little over k of them as a rule, and each finds its place by counting.
// More than 32 of them (many equal keys) take the rounds.
template <int SLOTS>
__device__ __forceinline__ void topk_select(const uint32_t (&key)[SLOTS], const float (&sc)[SLOTS], int k, TopkCand *cand, int lane) {
  uint32_t bkey = 0u;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) bkey = max(bkey, key[s]);
  uint32_t *best = reinterpret_cast<uint32_t *>(cand);
  best[lane] = bkey;
  __syncwarp();
  int above = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint4 q = *reinterpret_cast<const uint4 *>(best + 4 * j);
    above += (q.x > bkey) + (q.y > bkey) + (q.z > bkey) + (q.w > bkey);
  }
  const uint32_t bound = max(1u, __reduce_min_sync(0xffffffffu, above < k ? bkey : 0xffffffffu));
  uint32_t holders[SLOTS];
  int n = 0;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    holders[s] = __ballot_sync(0xffffffffu, key[s] >= bound);
    n += __popc(holders[s]);
  }
  const float sc0 = __shfl_sync(0xffffffffu, sc[0], 0);  // (also: every lane has read `best`)
  if (n <= 32) {
    int at = 0;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      if (key[s] >= bound) {
        TopkCand c = {key[s], s * 32 + lane, sc[s], 0u};
        *reinterpret_cast<uint4 *>(cand + at + __popc(holders[s] & ((1u << lane) - 1u))) = *reinterpret_cast<const uint4 *>(&c);
      }
      at += __popc(holders[s]);
    }
    __syncwarp();
    const uint4 raw = *reinterpret_cast<const uint4 *>(cand + lane);
    const TopkCand mine = *reinterpret_cast<const TopkCand *>(&raw);
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {  // a slot's candidates precede the next slot's and lanes ascend: j < lane is the lower id
      const uint32_t other = cand[j].key;
      rank += other > mine.key || (other == mine.key && j < lane);
    }
    __syncwarp();
    if (lane < n && rank < k) *reinterpret_cast<uint4 *>(cand + rank) = raw;
    if (lane >= n && lane < k) cand[lane] = TopkCand{0u, 0, sc0, 0u};
    __syncwarp();
    return;
  }
  uint32_t left[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) left[s] = key[s];
  TopkCand mine = {0u, 0, sc0, 0u};  // lane kk keeps place kk
  for (int kk = 0; kk < k; ++kk) {
    uint32_t bk = 0u, bs = 0u;
    float bsc = 0.0f;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)  // ascending e within the lane: strict > keeps the lowest index
      if (left[s] > bk) {
        bk = left[s];
        bs = (uint32_t)s;
        bsc = sc[s];
      }
    const uint32_t top = __reduce_max_sync(0xffffffffu, bk);
    if (top == 0u) break;
    const uint32_t win = __reduce_min_sync(0xffffffffu, bk == top ? bs * 32 + lane : 0xffffffffu);
    const float wsc = __shfl_sync(0xffffffffu, bsc, win & 31);
    if (lane == kk) mine = {top, (int)win, wsc, 0u};
    if (lane == (int)(win & 31)) {
#pragma unroll
      for (int s = 0; s < SLOTS; ++s)
        if (s == (int)bs) left[s] = 0u;
    }
  }
  if (lane < k) cand[lane] = mine;
  __syncwarp();
}

// One warp scores token t and selects its experts; `row` is topk_row_floats(E) floats of shared
// memory, 16-byte aligned and private to the warp.  The experts' ids also go to ids_out[0..k) when given.
template <int SLOTS>
__device__ __forceinline__ void route_topk_slots(const RouteParams &p, int t, float *row, int lane, int *ids_out) {
  const int E = p.E, k = min(p.k, p.E);
  const float *z = p.logits + (size_t)t * E;
  const float NEG_INF = __uint_as_float(0xff800000u);
  TopkCand *cand = reinterpret_cast<TopkCand *>(row + ((E + 3) & ~3));
  const bool biased = p.score != COLI_SCORE_SOFTMAX;

  float sc[SLOTS];  // score of each of this lane's experts
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) sc[s] = lane + 32 * s < E ? __ldcg(z + lane + 32 * s) : NEG_INF;
  float bias[SLOTS];  // requested beside the logits
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) bias[s] = (biased && p.select_bias && lane + 32 * s < E) ? p.select_bias[lane + 32 * s] : 0.0f;
  if (p.score == COLI_SCORE_SOFTMAX) {
    float mx = NEG_INF;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) mx = fmaxf(mx, sc[s]);  // max is order-independent
    mx = topk_key_value(__reduce_max_sync(0xffffffffu, topk_key(mx)));
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) {
      sc[s] = coli_expf(__fsub_rn(sc[s], mx));
      if (lane + 32 * s < E) row[lane + 32 * s] = sc[s];
    }
    __syncwarp();
    float tot = 0.0f;  // sequential over e, every lane redundantly (moe.rs:1068); the next 16 are read ahead
    int e = 0;
    float4 v[4];
    if (E >= 16) {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4 *>(row + 4 * i);
    }
    for (; e + 16 <= E; e += 16) {
      float4 u[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) u[i] = v[i];
      if (e + 32 <= E) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4 *>(row + e + 16 + 4 * i);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) tot = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(tot, u[i].x), u[i].y), u[i].z), u[i].w);
    }
    for (; e < E; ++e) tot = __fadd_rn(tot, row[e]);
    if (tot > 0.0f) {
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) sc[s] = __fdiv_rn(sc[s], tot);
    }
  } else {
#pragma unroll
    for (int s = 0; s < SLOTS; ++s) sc[s] = coli_sigmoidf(sc[s]);
  }

  // selection scores as keys
  uint32_t key[SLOTS];
  float ch[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    ch[s] = biased ? __fadd_rn(sc[s], bias[s]) : sc[s];
    key[s] = lane + 32 * s < E ? topk_key(ch[s]) : 0u;
  }

  // group-limited selection (n_group <= 32): a group's score is the sum of its two largest, found by as many
  // lanes as fit (four for 8 groups); the best topk_group groups are those with fewer than topk_group above
  if (p.n_group > 1) {
    const int G = p.n_group, gs = E / G, kg = min(p.topk_group, G);
    __syncwarp();  // the sum above has read the row
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
      if (lane + 32 * s < E) row[lane + 32 * s] = ch[s];
    __syncwarp();
    int per = 1;  // lanes of a group: a power of two
    while (2 * per * G <= 32) per *= 2;
    const int g = lane / per;
    float m1 = NEG_INF, m2 = NEG_INF;
    if (g < G)
#pragma unroll 4
      for (int i = lane % per; i < gs; i += per) {
        const float c = row[g * gs + i];
        m2 = c > m1 ? m1 : (c > m2 ? c : m2);
        m1 = c > m1 ? c : m1;
      }
    for (int o = 1; o < per; o <<= 1) {
      const float o1 = __shfl_xor_sync(0xffffffffu, m1, o), o2 = __shfl_xor_sync(0xffffffffu, m2, o);
      m2 = fmaxf(fminf(m1, o1), fmaxf(m2, o2));
      m1 = fmaxf(m1, o1);
    }
    const uint32_t gkey = g < G && lane % per == 0 ? topk_key(__fadd_rn(m1, m2)) : 0u;
    uint32_t *gk = reinterpret_cast<uint32_t *>(cand);
    if (lane % per == 0 && g < G) gk[g] = gkey;
    __syncwarp();
    int above = 0;
    for (int j = 0; j < G; ++j) above += gk[j] > gkey || (gk[j] == gkey && j < g);
    const uint32_t kept = __ballot_sync(0xffffffffu, gkey != 0u && above < kg);  // the first lanes of kept groups
    uint32_t gmask = __popc(__ballot_sync(0xffffffffu, gkey != 0u)) < kg ? 1u : 0u;  // no candidate: group 0
    for (int j = 0; j < G; ++j) gmask |= ((kept >> (j * per)) & 1u) << j;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
      if (lane + 32 * s < E && !((gmask >> ((lane + 32 * s) / gs)) & 1u)) key[s] = 0u;
    __syncwarp();
  }

  topk_select<SLOTS>(key, sc, k, cand, lane);
  if (lane < k) {
    float w = cand[lane].sc;
    if (p.norm_topk) {
      float smv = 0.0f;
#pragma unroll 8
      for (int kk = 0; kk < k; ++kk) smv = __fadd_rn(smv, cand[kk].sc);
      smv = __fadd_rn(smv, 1e-20f);
      w = __fdiv_rn(w, smv);
    }
    const int id = cand[lane].id;
    if (p.topk_idx) {
      p.topk_idx[(size_t)t * k + lane] = id;
      p.topk_w[(size_t)t * k + lane] = __fmul_rn(w, p.routed_scale);
      if (p.expert_rows) p.local_rank[(size_t)t * k + lane] = atomicAdd(p.expert_rows + id, 1);
    }
    if (ids_out) ids_out[lane] = id;
  }
  __syncwarp();  // the row may be reused for the warp's next token
}
__device__ __forceinline__ void route_topk_token(const RouteParams &p, int t, float *row, int lane, int *ids_out = nullptr) {
  if (p.E <= 128)
    route_topk_slots<4>(p, t, row, lane, ids_out);
  else if (p.E <= 256)
    route_topk_slots<8>(p, t, row, lane, ids_out);
  else
    route_topk_slots<kMaxSlots>(p, t, row, lane, ids_out);
}

// The same chains for batches above 8 tokens whose 8 x 8 tiles have an SM each.
__global__ void __launch_bounds__(192) k_router_staged(RouteParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  coli_grid_dependency_sync();
  clear_expert_rows(p);
  router_tiny_block<4, false>(p, smem_raw, (int)blockIdx.x * 8, (int)blockIdx.y * 8);
}

__global__ void __launch_bounds__(128) k_route_topk(RouteParams p) {
  coli_grid_dependency_sync();
  extern __shared__ __align__(16) float sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x * 4 + warp;
  if (t >= p.T) return;
  route_topk_token(p, t, sm + (size_t)warp * topk_row_floats(p.E), lane);
}

// The tiles of k_router_chain.
//                              TM TN WM WN  BK  stages
using RouterTile8x8 = RouterTile<1, 1, 2, 1, 128, 8>;
using RouterTile16x32 = RouterTile<2, 2, 2, 2, 64, 8>;
using RouterTile64x64 = RouterTile<8, 4, 2, 2, 64, 6>;
// ... and of k_router_pair:             TM TN WM WN CW
using RouterTile128x64 = RouterPairTile<8, 8, 4, 1, 2>;
using RouterTile128x128 = RouterPairTile<16, 8, 2, 2, 0>;
// A kernel that starts before its predecessor has ended packs its CTAs onto the SMs that are free by then (router of 4096
// tokens 445 -> 1183 us; top-k of 512 tokens 6500 cycles a token where one alone takes 3500).  With shared memory for no
// more CTAs on an SM than an even spread puts there it can start early all the same: `need` raised to that, or
// `need` itself where an SM gets more than four.
constexpr int kSmSharedBytes = 228 * 1024, kSpreadMost = 4;
static int ctas_per_sm(long ctas) { return (int)((ctas + COLI_SMS - 1) / COLI_SMS); }
static size_t spread_smem(long ctas, size_t need) {
  const int per_sm = ctas_per_sm(ctas);
  const size_t alone = (size_t)kSmSharedBytes / (per_sm + 1);
  return per_sm <= kSpreadMost && need < alone ? alone : need;
}
// Launches a router GEMM: early if its CTAs stay spread and the caller gains by it (us a call: 333 tokens, H 1024, 32 experts
// 44.4 -> 41.6; 512 tokens, H 2048, 128 experts 179.6 -> 173.9; 1024 389.0 -> 387.6).
template <class K>
static bool launch_router_kernel(K kernel, ColiPerDeviceOnce &attr_once, dim3 grid, int threads, size_t need, const RouteParams &p, cudaStream_t st,
                                 bool early = true) {
  const long ctas = (long)grid.x * grid.y;
  const size_t smem = spread_smem(ctas, need), most = (size_t)kSmSharedBytes / 2;
  if (!coli_set_smem_limit(attr_once, kernel, need > most ? need : most, "router shared-memory attribute")) return false;
  if (early && ctas_per_sm(ctas) <= kSpreadMost) return coli_cuda_check(launch_dependent(kernel, grid, dim3(threads), smem, st, p), "router launch");
  kernel<<<grid, threads, smem, st>>>(p);
  return true;
}
template <class C>
static bool launch_router_chain(const RouteParams &p, cudaStream_t st) {
  static ColiPerDeviceOnce attr_once;
  return launch_router_kernel(k_router_chain<C>, attr_once, dim3((p.T + C::BM - 1) / C::BM, (p.E + C::BN - 1) / C::BN), C::NT, C::SMEM, p, st);
}
template <class C>
static bool launch_router_pair(const RouteParams &p, cudaStream_t st) {
  static ColiPerDeviceOnce attr_once;
  // (never early: thousands of tokens follow a combine of as many rows, whose last CTAs its own then wait beside; us a call,
  // ordinary / early: 3000 tokens, H 3072, 256 experts 689 / 706; 8192, H 2048, 256 1008 / 1028; 7026, H 1920, 177 572 / 598;
  // 16384, H 2048, 384 10470 / 10700; 4096, H 7168, 256 3750 / 3750)
  return launch_router_kernel(k_router_pair<C>, attr_once, dim3((p.T + C::BM - 1) / C::BM, (p.E + C::BN - 1) / C::BN), C::NT, C::SMEM, p, st, false);
}
// The tile of a batch: 0 = 8 x 8, 1 = 16 x 32, 2 = 64 x 64, 3 = 128 x 64, 4 = 128 x 128 tokens x experts.
// The time of one k is a function of n, the CTAs of the fullest SM; the figures are nanoseconds measured
// on B200 between 21 and 16384 tokens (5.3 and 10 are the chain's latency, with its loads and
// conversions, when an SM has little else).
static int pick_router_tile(int T, int E) {
  auto n = [&](int bm, int bn) { return (float)(((long)((T + bm - 1) / bm) * ((E + bn - 1) / bn) + COLI_SMS - 1) / COLI_SMS); };
  const float ns[5] = {n(8, 8) <= 1.0f ? 2.8f : fmaxf(5.3f, 1.6f * n(8, 8)), fmaxf(10.0f, 3.0f + 5.6f * n(16, 32)), 3.0f + 33.0f * n(64, 64),
                       5.0f + 46.5f * n(128, 64), 8.0f + 81.0f * n(128, 128)};
  int best = 0;
  for (int i = 1; i < 5; ++i)
    if (ns[i] < ns[best]) best = i;
  return best;
}

// 8 x 8 tiles with an SM to themselves take the staged kernel: 2.8 ns a k against 5.3 of the chain kernel, which holds
// its rows as bf16 and widens them between the FMAs (launches of 21 tokens x 128 experts x 2048 9 us, 24 x 256 x 7168 24).
// Two of its CTAs on an SM would be no faster than the chain kernel's.
static long router_tiles_8x8(int T, int E) { return (long)((T + 7) / 8) * ((E + 7) / 8); }
static bool launch_router_staged(const RouteParams &p, cudaStream_t st) {
  static ColiPerDeviceOnce attr_once;
  // (early behind the norm of a layer step, 48 tokens 101.6 -> 100.4 us; not behind another call, 21 tokens 92.8 -> 94.0)
  return launch_router_kernel(k_router_staged, attr_once, dim3((p.T + 7) / 8, (p.E + 7) / 8), 192, RouterTiny::SMEM, p, st, p.in_call);
}

static int launch_router_logits(const RouteParams &p, cudaStream_t st) {
  if (p.E > 32 * kMaxSlots) {
    coli_set_error("router: E=%d exceeds the supported maximum of %d", p.E, 32 * kMaxSlots);
    return 0;
  }
  if (p.k > 32 || p.n_group > 32 || (p.n_group > 1 && p.E % p.n_group != 0)) {
    coli_set_error("router: unsupported k=%d / n_group=%d for E=%d", p.k, p.n_group, p.E);
    return 0;
  }
  if (p.n_group > 1 && p.k > min(p.topk_group, p.n_group) * (p.E / p.n_group)) {
    coli_set_error("router: k=%d exceeds the experts of the %d groups a token may use", p.k, p.topk_group);
    return 0;
  }
  // the batched kernels copy 16-byte chunks of rows; anything else takes the element-wise kernel
  const bool rows16 = p.H % 8 == 0 && ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.router_w)) & 15) == 0;
  if (rows16) {
    bool ok = false;
    switch (pick_router_tile(p.T, p.E)) {
      case 0: ok = router_tiles_8x8(p.T, p.E) <= COLI_SMS ? launch_router_staged(p, st) : launch_router_chain<RouterTile8x8>(p, st); break;
      case 1: ok = launch_router_chain<RouterTile16x32>(p, st); break;
      case 2: ok = launch_router_chain<RouterTile64x64>(p, st); break;
      case 3: ok = launch_router_pair<RouterTile128x64>(p, st); break;
      case 4: ok = launch_router_pair<RouterTile128x128>(p, st); break;
    }
    if (!ok) return 0;
  } else if ((long)((p.T + 31) / 32) * ((p.E + 31) / 32) >= 96) {
    k_router_gemm<2, 2><<<dim3((p.E + 31) / 32, (p.T + 31) / 32), 256, 0, st>>>(p);
  } else {
    k_router_gemm<1, 1><<<dim3((p.E + 15) / 16, (p.T + 15) / 16), 256, 0, st>>>(p);
  }
  coli_count_launch(1);
  return coli_cuda_check(cudaGetLastError(), "router launch") ? 1 : 0;
}

int launch_router(const RouteParams &p, cudaStream_t st) {
  if (p.T <= 0) return 1;
  if (!launch_router_logits(p, st)) return 0;
  const int ctas = (p.T + 3) / 4;
  const size_t sm = spread_smem(ctas, (size_t)4 * topk_row_floats(p.E) * sizeof(float));
  static ColiPerDeviceOnce attr_once;
  if (!coli_set_smem_limit(attr_once, k_route_topk, kSmSharedBytes / 2, "top-k shared-memory attribute")) return 0;
  coli_count_launch(1);
  return coli_cuda_check(launch_dependent(k_route_topk, dim3((p.T + 3) / 4), dim3(128), sm, st, p), "top-k launch") ? 1 : 0;
}

// ---------------------------------------------------------------------------------------------
// Permutation into expert-contiguous segments.  Stable: rows of one expert keep ascending
// token order (moe.rs:1373-1387), positions are a pure function of the routing.
//   1. k_seg_count : one CTA per chunk of 32 tokens; the rank of a pair among the chunk's pairs of
//                    its expert is the number of earlier pairs with the same id, counted by a
//                    thread per pair.  (A token's experts are distinct except in the degenerate
//                    case the reference's scan also has -- a row of NaN logits selects expert 0 k
//                    times -- and pairs of one token rank by kk, so every pair gets a row of its
//                    own.)  An id outside [0, E) gets no row (slot -1).
//   2. k_seg_scan  : per expert an exclusive running sum over chunks; exclusive scan over the
//                    segment order; builds the work list (segments cut into row_per_item runs).
//   3. k_permute   : row position = segment offset + chunk prefix + rank; copies the token row.
// ---------------------------------------------------------------------------------------------
// Number of entries of ids[0..i) equal to ids[i]; ids in shared memory, 16-byte aligned.  A walk in
// order over tokens by one warp, the alternative, costs a few hundred cycles per token.
__device__ __forceinline__ int rank_before(const int *ids, int i) {
  const int v = ids[i];
  int n = 0, j = 0;
#pragma unroll 4
  for (; j + 4 <= i; j += 4) {
    const int4 q = *reinterpret_cast<const int4 *>(ids + j);
    n += (q.x == v) + (q.y == v) + (q.z == v) + (q.w == v);
  }
  for (; j < i; ++j) n += ids[j] == v;
  return n;
}
__global__ void __launch_bounds__(256) k_seg_count(PermuteParams p, int nchunk) {
  coli_grid_dependency_sync();
  extern __shared__ __align__(16) int cnt_sm[];  // 32 k ids of the chunk, then E counters
  int *ids = cnt_sm, *cnt = cnt_sm + 32 * p.k;
  const int chunk = blockIdx.x;
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) cnt[e] = 0;
  const int T = p.virt ? p.virt->total : p.T;
  if (chunk * 32 >= T) return;
  const int t0 = chunk * 32, npairs = (min(T, t0 + 32) - t0) * p.k;
  for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
    const int t = t0 + i / p.k;
    ids[i] = p.topk_idx[(size_t)(p.virt ? coli_virt_row(p.virt, t) : t) * p.k + i % p.k];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
    const int e = ids[i];
    if (e < 0 || e >= p.E) continue;
    p.local_rank[(size_t)t0 * p.k + i] = rank_before(ids, i);
    atomicAdd(cnt + e, 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) p.chunk_cnt[(size_t)chunk * p.E + e] = cnt[e];
}

// Rows per item of a segment of n rows cut into items of at most rpi: items of the tcgen05 kernel
// (rpi >= 64) take equal shares, because a tile of few rows still decodes all of its weights -- 170 rows
// as 96 + 74 and not 160 + 10; the number of items is the same.
__device__ __forceinline__ int work_item_rows(int n, int rpi) {
  if (rpi < 64 || n <= rpi) return rpi;
  const int items = (n + rpi - 1) / rpi;
  return ((n + items - 1) / items + TCT_ROW_GRAIN - 1) / TCT_ROW_GRAIN * TCT_ROW_GRAIN;
}
// Segment offsets and the work list from per-segment row counts in shared memory, by the whole
// CTA: a shuffle scan per warp and a pass over the warps' sums (row offsets and item bases at once),
// then one thread per segment writes that segment's items.  off and ibase hold nseg + 1 entries.
// A serial walk by one thread costs ~60 ns per segment, more than the decode GEMV of a layer
// with a few hundred experts.
__device__ __forceinline__ void build_work_list(const PermuteParams &p, const int *cnt, int nseg, int max_items, int *off,
                                                int *ibase) {
  const int rpi = p.rows_per_item;
  __shared__ int2 warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  int2 run = make_int2(0, 0);  // rows and items of the segments before `base`
  for (int base = 0; base < nseg; base += (int)blockDim.x) {
    const int s = base + (int)threadIdx.x;
    const int n = s < nseg ? cnt[s] : 0;
    const int ni = (n + rpi - 1) / rpi;
    int a = n, b = ni;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) {
        a += ua;
        b += ub;
      }
    }
    if (lane == 31) warp_sum[warp] = make_int2(a, b);
    __syncthreads();
    int2 before = run;
    for (int w = 0; w < nwarp; ++w) {
      const int2 v = warp_sum[w];
      if (w < warp) before.x += v.x, before.y += v.y;
      run.x += v.x, run.y += v.y;
    }
    if (s < nseg) {
      off[s] = before.x + a - n;
      ibase[s] = before.y + b - ni;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    off[nseg] = run.x;
    ibase[nseg] = run.y;
    *p.n_items = min(run.y, max_items);
  }
  __syncthreads();
  for (int s = threadIdx.x; s < nseg; s += blockDim.x) {
    const int n = cnt[s], r0 = off[s];
    const int share = work_item_rows(n, rpi);
    int it = ibase[s];
    for (int r = 0; r < n; r += share, ++it) {
      if (it < max_items) {
        p.item_seg[it] = s;
        p.item_row0[it] = r0 + r;
        p.item_nrows[it] = min(share, n - r);
      }
    }
  }
  __syncthreads();
}

__global__ void __launch_bounds__(1024) k_seg_scan(PermuteParams p, int nchunk, int max_items) {
  coli_grid_dependency_sync();
  __shared__ int seg_cnt[1024 + 1];
  __shared__ int seg_off[1024 + 2];
  __shared__ int seg_ibase[1024 + 2];
  const int E = p.E;
  if (p.virt) nchunk = min(nchunk, (p.virt->total + 31) / 32);
  const int nrt = p.nseg_routed;  // routed segments: E, or the experts resident on this rank
  const int nseg = nrt + (p.has_shared ? 1 : 0);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const int pos = p.expert_slot ? p.expert_slot[e] : e;
    if (pos < 0) continue;  // expert lives on another rank: its pairs get no row here
    int run = 0;
    for (int c0 = 0; c0 < nchunk; c0 += 8) {  // loads of a group are independent of its stores
      int v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (c0 + j < nchunk) ? p.chunk_cnt[(size_t)(c0 + j) * E + e] : 0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (c0 + j < nchunk) {
          p.chunk_cnt[(size_t)(c0 + j) * E + e] = run;
          run += v[j];
        }
    }
    seg_cnt[pos] = run;
  }
  if (threadIdx.x == 0 && p.has_shared) seg_cnt[nrt] = p.virt ? p.virt->total : p.T;
  __syncthreads();
  if (p.rows_cap != 0x7fffffff) {  // a batch that does not fit the row buffers is not run at all (and reported)
    __shared__ int too_many;
    if (threadIdx.x == 0) {
      long total = 0;
      for (int s = 0; s < nseg; ++s) total += seg_cnt[s];
      too_many = total > (long)p.rows_cap ? 1 : 0;
      if (too_many && p.overflow) atomicExch(p.overflow, 1);
    }
    __syncthreads();
    if (too_many)
      for (int s = threadIdx.x; s < nseg; s += blockDim.x) seg_cnt[s] = 0;
    __syncthreads();
  }
  build_work_list(p, seg_cnt, nseg, max_items, seg_off, seg_ibase);
  for (int s = threadIdx.x; s <= nseg; s += blockDim.x) p.seg_off[s] = seg_off[s];
  if (p.seg_count)
    for (int s = threadIdx.x; s < nrt; s += blockDim.x) p.seg_count[s] = seg_cnt[s];
}

__global__ void __launch_bounds__(256) k_permute(PermuteParams p) {
  coli_grid_dependency_sync();
  // one warp per (t, kk) row; rows T*k .. T*k+T-1 are the shared expert's identity rows
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int T = p.virt ? p.virt->total : p.T;
  const int nrouted = T * p.k;
  const int total = nrouted + (p.has_shared ? T : 0);
  if (warp >= total) return;
  int t, pos;
  int trow;  // row of the token in x / topk_idx
  if (warp < nrouted) {
    t = warp / p.k;
    trow = p.virt ? coli_virt_row(p.virt, t) : t;
    const int e = p.topk_idx[(size_t)trow * p.k + (warp - t * p.k)];
    const int s = (e < 0 || e >= p.E) ? -1 : (p.expert_slot ? p.expert_slot[e] : e);
    if (s < 0) {  // not resident here (or not an expert id): no row, the combine skips negative slots
      if (lane == 0) p.slot[warp] = -1;
      return;
    }
    pos = p.seg_off[s] + p.chunk_cnt[(size_t)(t >> 5) * p.E + e] + p.local_rank[warp];
    if (pos >= p.rows_cap) {  // more rows than the buffers hold: drop the pair and report it
      if (lane == 0) {
        p.slot[warp] = -1;
        if (p.overflow) atomicExch(p.overflow, 1);
      }
      return;
    }
    if (lane == 0) p.slot[warp] = pos;
  } else {
    t = warp - nrouted;
    trow = t;
    pos = p.seg_off[p.nseg_routed] + t;
  }
  if (lane == 0) p.row_token[pos] = t;
  const int vec = p.H / 8;
  const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)trow * p.H);
  uint4 *dst = reinterpret_cast<uint4 *>(p.xg + (size_t)pos * p.H);
  int c = lane;
  for (; c + 96 < vec; c += 128) {  // four loads in flight per lane
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = src[c + 32 * u];
#pragma unroll
    for (int u = 0; u < 4; ++u) dst[c + 32 * u] = coli_bf16x8_to_f16x8(v[u]);
  }
  for (; c < vec; c += 32) dst[c] = coli_bf16x8_to_f16x8(src[c]);
}

// The same for the gather of at most 1024 pairs and 128 KB of rows: count, scan, work list, row positions and rows by ONE
// CTA instead of three launches.  Same stable order: positions ascend with the token inside an expert.
struct PermuteSmallSmem {
  __align__(16) int idx[1024];
  int cnt[1024 + 1];
  int off[1024 + 2];
  int rank[1024];
  int ibase[1024 + 2];
};
__global__ void __launch_bounds__(1024) k_permute_small(PermuteParams p, int max_items) {
  coli_grid_wait();
  __shared__ PermuteSmallSmem sm;
  int *cnt = sm.cnt, *off = sm.off, *rank_sm = sm.rank, *idx_sm = sm.idx;
  const int E = p.E, nseg = p.nseg_routed, npairs = p.T * p.k;
  for (int e = threadIdx.x; e <= E; e += blockDim.x) cnt[e] = 0;
  // segment of every pair, fetched with independent loads before the ordered walk below
  for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
    const int e = p.topk_idx[i];
    idx_sm[i] = (e < 0 || e >= E) ? -1 : (p.expert_slot ? p.expert_slot[e] : e);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
    const int s = idx_sm[i];
    if (s < 0) continue;
    rank_sm[i] = rank_before(idx_sm, i);
    atomicAdd(cnt + s, 1);
  }
  __syncthreads();
  build_work_list(p, cnt, nseg, max_items, off, sm.ibase);
  for (int s = threadIdx.x; s <= nseg; s += blockDim.x) p.seg_off[s] = off[s];
  if (p.seg_count)
    for (int s = threadIdx.x; s < nseg; s += blockDim.x) p.seg_count[s] = cnt[s];
  for (int i = threadIdx.x; i < npairs; i += blockDim.x) {
    const int s = idx_sm[i];
    const int pos = s < 0 ? -1 : off[s] + rank_sm[i];
    p.slot[i] = pos;
    if (s >= 0) p.row_token[pos] = i / p.k;
  }
  const int vec = p.H / 8;
  for (int r = threadIdx.x >> 5; r < npairs; r += blockDim.x >> 5) {  // one warp per row
    const int s = idx_sm[r];
    if (s < 0) continue;
    const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)(r / p.k) * p.H);
    uint4 *dst = reinterpret_cast<uint4 *>(p.xg + (size_t)(off[s] + rank_sm[r]) * p.H);
    for (int c = threadIdx.x & 31; c < vec; c += 32) dst[c] = coli_bf16x8_to_f16x8(src[c]);
  }
}

// The same for at most 256 pairs in a block that wants no counts per segment: a thread per pair finds its row --
// the pairs of lower segments and the earlier ones of its own -- by comparing with every other pair, and the
// item that a row opens by the rows that open one before it (a bit per row).  Two barriers and no scan over
// the segments.  Called by `threads` threads of a CTA, numbered i, that meet at barrier `bar`.
// `seg` holds the pairs' segments (below 0: no row), padded to a multiple of 4 entries with INT_MAX, and `opens`
// eight zeros; both are visible to those threads.  A dry run writes nothing.
constexpr int kPairwiseMax = 256;
struct PermutePairsSmem {
  __align__(16) int seg[kPairwiseMax];
  int pos[kPairwiseMax];
  uint32_t opens[kPairwiseMax / 32];
};
__device__ __forceinline__ void permute_pairs(const PermuteParams &p, int max_items, PermutePairsSmem &sm, int i, int threads, int bar, bool dry) {
  const int n = p.T * p.k, rpi = p.rows_per_item;
  int s = -1, below = 0, before = 0, equal = 0, share = 1;
  if (i < n) s = sm.seg[i];
  if (s >= 0) {
    for (int j = 0; j < n; j += 4) {
      const int4 q = *reinterpret_cast<const int4 *>(sm.seg + j);
      below += ((unsigned)q.x < (unsigned)s) + ((unsigned)q.y < (unsigned)s) + ((unsigned)q.z < (unsigned)s) + ((unsigned)q.w < (unsigned)s);
      equal += (q.x == s) + (q.y == s) + (q.z == s) + (q.w == s);
      before += (q.x == s && j < i) + (q.y == s && j + 1 < i) + (q.z == s && j + 2 < i) + (q.w == s && j + 3 < i);
    }
    share = work_item_rows(equal, rpi);
  }
  const int pos = below + before;
  const bool opens = s >= 0 && before % share == 0;
  if (i < n && !dry) {
    sm.pos[i] = s >= 0 ? pos : -1;
    p.slot[i] = s >= 0 ? pos : -1;
    if (s >= 0) p.row_token[pos] = i / p.k;
  }
  if (opens) atomicOr(&sm.opens[pos >> 5], 1u << (pos & 31));
  int rows;  // the shared expert's rows follow them
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %3, 0;\nbarrier.cta.red.popc.aligned.u32 %0, %1, %2, p;\n}"
               : "=r"(rows)
               : "r"(bar), "r"(threads), "r"(s >= 0 ? 1 : 0)
               : "memory");
  int items = 0, item = 0;
#pragma unroll
  for (int w = 0; w < kPairwiseMax / 32; ++w) {
    const uint32_t bits = sm.opens[w];
    if (w < (pos >> 5)) item += __popc(bits);
    if (w == (pos >> 5)) item += __popc(bits & ((1u << (pos & 31)) - 1u));
    items += __popc(bits);
  }
  if (opens && item < max_items && !dry) {
    p.item_seg[item] = s;
    p.item_row0[item] = pos;
    p.item_nrows[item] = min(share, equal - before);
  }
  if (p.has_shared) {
    const int sshare = work_item_rows(p.T, rpi), nsh = (p.T + sshare - 1) / sshare;
    if (i < nsh && items + i < max_items && !dry) {
      p.item_seg[items + i] = p.nseg_routed;
      p.item_row0[items + i] = rows + i * sshare;
      p.item_nrows[items + i] = min(sshare, p.T - i * sshare);
    }
    if (i < p.T && !dry) p.row_token[rows + i] = i;
    items += nsh;
  }
  if (i == 0 && !dry) *p.n_items = min(items, max_items);
  if (p.xg && !dry) {  // gather rows: one warp per row
    const int total = n + (p.has_shared ? p.T : 0);
    const int vec = p.H / 8;
    for (int r = i >> 5; r < total; r += threads >> 5) {
      const int t = r < n ? r / p.k : r - n, to = r < n ? sm.pos[r] : rows + t;
      if (to < 0) continue;
      const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)t * p.H);
      uint4 *dst = reinterpret_cast<uint4 *>(p.xg + (size_t)to * p.H);
      for (int c = i & 31; c < vec; c += 32) dst[c] = coli_bf16x8_to_f16x8(src[c]);
    }
  }
}
// a pair's segment: below 0 for an id that is no expert or lives on another rank
__device__ __forceinline__ int pair_segment(const PermuteParams &p, int id) {
  return (id < 0 || id >= p.E) ? -1 : (p.expert_slot ? p.expert_slot[id] : id);
}

// Decode front end (T <= 8): router logits, top-k and the permutation in ONE launch.  Every CTA
// computes the logits of 8 experts (and converts its slice of the tokens to f16); the CTA
// that finishes last -- found with an atomic ticket, nobody waits for anybody -- scores the
// tokens and builds the segments.  `ticket` must be zero at launch and is left zero.
// The kernel is latency from end to end, and its CTAs must not share an SM: started early, while the
// previous call's last kernels still hold most SMs, two or three packed onto each free one and the chains
// took 14.6 cycles per k instead of 6 (8 tokens, 128 experts x 2048: 30 000 of the kernel's 44 000 cycles).
// kFrontSmem is therefore, with what is static, more than half of an SM's shared memory.  (Beside a CTA of the decode expert
// kernel, which holds the SM until its tasks are done, the front does not fit: at 213 registers a thread the register file is too
// small.  Compiled to 96 to 127, by launch bounds or with a kernel for each number of score slots, it does, and no
// call is shorter by it: 8 tokens 54.9 us a call against 55.1 to 55.6, 1 token 25.2 against 25.2 to 25.5.)  The last CTA runs top-k and permutation once per
// call, with instructions that the streamed weights have pushed out of every cache: two warps that have nothing else to
// do run the same code beside the chains, on router weights for logits, and write nothing (8 tokens, the weights of
// three layers in turn: top-k 2.4 us, permutation 4.6 -> 1.8; the front 15.9 -> 14.4 us).  They and the first router
// weights do not wait for the predecessor: a call of 8 tokens 54.9 -> 53.0 us, of 1 token 25.1 -> 24.3.
constexpr int kFrontStaging = 4, kFrontDry = 64;  // staging warps; threads of the dry run
constexpr size_t kFrontSmem = 112 * 1024;
static_assert(RouterTiny::SMEM <= kFrontSmem && (size_t)9 * topk_row_floats(32 * kMaxSlots) * sizeof(float) <= kFrontSmem - RouterTiny::SMEM,
              "the top-k rows of eight warps and of the dry run lie behind the staging area");
__global__ void __launch_bounds__(256) k_decode_front(RouteParams rp, PermuteParams pp, int max_items, unsigned int *ticket) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ PermutePairsSmem psm;
  __shared__ int ids[kPairwiseMax];
  __shared__ int is_last;
  coli_grid_trigger();  // (each role waits where it first needs the predecessor)
  constexpr int first_dry = 256 - kFrontDry;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *rows = reinterpret_cast<float *>(smem_raw + RouterTiny::SMEM);
  RouteParams tp = rp;
  int first = 0, last = 0;  // the tokens that this warp scores
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {  // both passes run one copy of the code
    const bool dry = pass == 0;
    if (dry) {
      if ((int)threadIdx.x < first_dry) {
        router_tiny_block<kFrontStaging, true>(rp, smem_raw, 0, (int)blockIdx.x * 8);
        continue;
      }
      // beside long chains there is time, and ahead of the wait other kernels run (us a call of 8 tokens, I 512, 128 experts, behind
      // the wait / ahead of it: H 2048 46.4 / 46.05, 3072 57.4 / 57.2, 4096 72.6 / 73.1, 7168 107.6 / 108.3)
      if (rp.H >= 4096) coli_grid_wait();
      tp.logits = const_cast<float *>(reinterpret_cast<const float *>(rp.router_w));  // E * H bf16 hold E floats (H >= 8)
      tp.topk_idx = nullptr;
      last = warp == 7 ? 1 : 0;
    } else {
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();  // this CTA's logits are visible device-wide before its ticket is
        is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1) ? 1 : 0;
        __threadfence();
      }
      __syncthreads();
      if (!is_last) return;
      tp.logits = rp.logits;
      tp.topk_idx = rp.topk_idx;
      first = warp;
      last = rp.T;
    }
    const int i = (int)threadIdx.x - (dry ? first_dry : 0), threads = dry ? kFrontDry : 256, bar = dry ? 2 : 0;
    for (int t = first; t < last; t += 8)
      route_topk_token(tp, t, rows + (size_t)(dry ? 8 : warp) * topk_row_floats(rp.E), lane, ids + t * rp.k);
    if (i < kPairwiseMax / 32) psm.opens[i] = 0u;
    asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(bar), "r"(threads) : "memory");  // the routing is read back below
    for (int j = i; j < kPairwiseMax; j += threads) psm.seg[j] = j < (dry ? rp.k : rp.T * rp.k) ? pair_segment(pp, ids[j]) : 0x7fffffff;
    asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(bar), "r"(threads) : "memory");
    permute_pairs(pp, max_items, psm, i, threads, bar, dry);
    if (dry) {
      coli_grid_wait();
      if (pp.x16) {  // this CTA's share of the f16 copy
        const int n = rp.T * (rp.H / 8);
        const int per = (n + (int)gridDim.x - 1) / (int)gridDim.x;
        const int lo = (int)blockIdx.x * per, hi = min(n, lo + per);
        const uint4 *src = reinterpret_cast<const uint4 *>(rp.x);
        uint4 *dst = reinterpret_cast<uint4 *>(pp.x16);
        for (int i = lo + (int)threadIdx.x - first_dry; i < hi; i += kFrontDry) dst[i] = coli_bf16x8_to_f16x8(src[i]);
      }
    }
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// Rows of a batch whose top-k has counted them (RouteParams::expert_rows): every pair knows its rank among its
// expert's, so what is left is a sum over the segments, which each CTA makes for itself, and the rows.  CTA 0 builds the
// work list while the others write: a warp per (t, kk) row, rows T*k .. T*k+T-1 are the shared expert's, and when
// a token-order f16 copy of x is wanted, a warp more for each 1024 elements of it.
// Against launches for counts per 32 tokens, one CTA's scan over them and the rows (up to 1024 pairs: one CTA for all
// of it), us a call: 333 tokens, H 1024, 32 experts 50.3 -> 44.1; 512 tokens, H 2048, 128 experts 186.9 -> 177.2; 21 tokens
// 96.7 -> 92.7; 48 tokens 111.8 -> 101.8 (these two with the router above).  The whole permutation by the last CTA of the top-k
// was built too: its code, cold and run once, took 10 us more than these launches.
__global__ void __launch_bounds__(256) k_place_rows(PermuteParams p, int max_items) {
  __shared__ int cnt[32 * kMaxSlots + 1], off[32 * kMaxSlots + 2], ibase[32 * kMaxSlots + 2];
  coli_grid_dependency_sync();
  const int nrt = p.nseg_routed, nseg = nrt + (p.has_shared ? 1 : 0), nrouted = p.T * p.k;
  const int warp = (((int)blockIdx.x - 1) * (int)blockDim.x + (int)threadIdx.x) >> 5, lane = threadIdx.x & 31;
  // what this warp's row needs of the routing is requested beside the counts
  int e = -1, rank = 0;
  if (blockIdx.x > 0 && warp < nrouted) {
    e = p.topk_idx[warp];
    rank = p.local_rank[warp];
  }
  for (int i = threadIdx.x; i < p.E; i += blockDim.x) {
    const int s = pair_segment(p, i);
    if (s >= 0) cnt[s] = p.expert_rows[i];
  }
  if (threadIdx.x == 0 && p.has_shared) cnt[nrt] = p.T;
  __syncthreads();
  if (blockIdx.x == 0) {
    build_work_list(p, cnt, nseg, max_items, off, ibase);
    return;
  }
  const int total = nrouted + (p.has_shared ? p.T : 0);
  const int seg = warp < nrouted ? pair_segment(p, e) : nrt;
  int first = 0;  // rows of the segments before this warp's
  if (warp < total)
    for (int i = lane; i < seg; i += 32) first += cnt[i];
  first = __reduce_add_sync(0xffffffffu, first);
  if (warp >= total) {
    if (p.x16) {
      const int n = p.T * (p.H / 8), base = (warp - total) * 128 + lane;
      const uint4 *src = reinterpret_cast<const uint4 *>(p.x);
      uint4 *dst = reinterpret_cast<uint4 *>(p.x16), v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = base + 32 * u < n ? src[base + 32 * u] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (base + 32 * u < n) dst[base + 32 * u] = coli_bf16x8_to_f16x8(v[u]);
    }
    return;
  }
  const int t = warp < nrouted ? warp / p.k : warp - nrouted;
  const int pos = first + (warp < nrouted ? rank : t);
  if (lane == 0) {
    if (warp < nrouted) p.slot[warp] = seg < 0 ? -1 : pos;
    if (seg >= 0) p.row_token[pos] = t;
  }
  if (!p.xg || seg < 0) return;
  const int vec = p.H / 8;
  const uint4 *src = reinterpret_cast<const uint4 *>(p.x + (size_t)t * p.H);
  uint4 *dst = reinterpret_cast<uint4 *>(p.xg + (size_t)pos * p.H);
  int c = lane;
  for (; c + 96 < vec; c += 128) {  // four loads in flight per lane
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = src[c + 32 * u];
#pragma unroll
    for (int u = 0; u < 4; ++u) dst[c + 32 * u] = coli_bf16x8_to_f16x8(v[u]);
  }
  for (; c < vec; c += 32) dst[c] = coli_bf16x8_to_f16x8(src[c]);
}

static int permute_max_items(const PermuteParams &p) {
  return max_work_items(p.T * p.k + (p.has_shared ? p.T : 0), p.nseg_routed + (p.has_shared ? 1 : 0), p.rows_per_item);
}

int launch_decode_front(const RouteParams &rp, const PermuteParams &pp, unsigned int *ticket, cudaStream_t st) {
  if (!(rp.T >= 1 && rp.T <= 8 && rp.H % 8 == 0 && rp.E <= 32 * kMaxSlots && rp.k <= 32 && rp.k <= rp.E &&
        rp.n_group <= 32 && (rp.n_group <= 1 || rp.E % rp.n_group == 0) && pp.seg_count == nullptr && ticket != nullptr))
    return -1;  // not applicable: the caller runs the separate stages
  static_assert(8 * 32 <= kPairwiseMax, "a thread per pair");
  static ColiPerDeviceOnce attr_once;
  if (!coli_set_smem_limit(attr_once, k_decode_front, kFrontSmem, "decode front shared-memory attribute")) return 0;
  coli_count_launch(1);
  return coli_cuda_check(launch_dependent(k_decode_front, dim3((rp.E + 7) / 8), dim3(256), kFrontSmem, st, rp, pp, permute_max_items(pp), ticket),
                         "decode front launch")
             ? 1
             : 0;
}

// Whether a batch's rows are counted by its top-k and placed in one launch (us a call, three launches / one: 100 tokens, H 1024,
// 32 experts 42.3 / 36.3; 100 tokens, H 2048, I 768, 16 experts 62.0 / 54.8; 80 tokens, H 7168, I 512, 32 experts 115.0 / 108.5).
// Above 65536 pairs the atomic counts of a popular expert queue up.
bool place_rows_ok(const PermuteParams &p) {
  return !p.virt && !p.seg_count && p.rows_cap == 0x7fffffff && p.E <= 32 * kMaxSlots && (long)p.T * p.k <= 65536;
}
int launch_place_rows(const PermuteParams &p, cudaStream_t st) {
  const int warps = p.T * p.k + (p.has_shared ? p.T : 0) + (p.x16 ? (int)(((size_t)p.T * (p.H / 8) + 127) / 128) : 0);
  coli_count_launch(1);
  return coli_cuda_check(launch_dependent(k_place_rows, dim3(1 + (warps + 7) / 8), dim3(256), 0, st, p, permute_max_items(p)), "row placement launch") ? 1 : 0;
}

int launch_permute(const PermuteParams &p, cudaStream_t st) {
  if (p.T <= 0) return 1;
  if (p.E > 1024) {
    coli_set_error("permute: E=%d exceeds 1024", p.E);
    return 0;
  }
  if (!p.xg) {
    coli_set_error("permute: no buffer for the gathered rows");
    return 0;
  }
  const int nchunk = (p.T + 31) / 32;
  const int max_items = permute_max_items(p);
  // one CTA gathers 128 KB of rows in time, a megabyte far too slowly
  if (!p.virt && !p.has_shared && p.T * p.k <= 1024 && (size_t)p.T * (p.k + 1) * p.H * 2 <= 128 * 1024) {
    coli_count_launch(1);
    return coli_cuda_check(launch_dependent(k_permute_small, dim3(1), dim3(1024), 0, st, p, max_items), "permute launch") ? 1 : 0;
  }
  const int total = p.T * p.k + (p.has_shared ? p.T : 0);
  coli_count_launch(3);
  return coli_cuda_check(launch_dependent(k_seg_count, dim3(nchunk), dim3(256), (size_t)(32 * p.k + p.E) * sizeof(int), st, p, nchunk), "permute launch") &&
                 coli_cuda_check(launch_dependent(k_seg_scan, dim3(1), dim3(1024), 0, st, p, nchunk, max_items), "permute launch") &&
                 coli_cuda_check(launch_dependent(k_permute, dim3((total + 7) / 8), dim3(256), 0, st, p), "permute launch")
             ? 1
             : 0;
}

// The same for rows that are already expert-contiguous: counts on the device, any number of segments,
// one CTA.  (One thread walking the segments took 12 us for 24 of them.)
__global__ void __launch_bounds__(1024) k_items_from_counts(const int32_t *seg_count, int nseg, int rows_per_item, int32_t *seg_off,
                                                            int32_t *item_seg, int32_t *item_row0, int32_t *item_nrows, int32_t *n_items) {
  __shared__ int2 warp_sum[32];
  coli_grid_dependency_sync();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5, rpi = rows_per_item;
  int2 run = make_int2(0, 0);  // rows and items of the segments before `base`
  for (int base = 0; base < nseg; base += (int)blockDim.x) {
    const int s = base + (int)threadIdx.x;
    const int n = s < nseg ? seg_count[s] : 0;
    const int ni = (n + rpi - 1) / rpi;
    int a = n, b = ni;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int ua = __shfl_up_sync(0xffffffffu, a, o), ub = __shfl_up_sync(0xffffffffu, b, o);
      if (lane >= o) {
        a += ua;
        b += ub;
      }
    }
    if (lane == 31) warp_sum[warp] = make_int2(a, b);
    __syncthreads();
    int2 before = run;
    for (int w = 0; w < nwarp; ++w) {
      const int2 v = warp_sum[w];
      if (w < warp) before.x += v.x, before.y += v.y;
      run.x += v.x, run.y += v.y;
    }
    if (s < nseg) {
      const int row0 = before.x + a - n, share = work_item_rows(n, rpi);
      int it = before.y + b - ni;
      seg_off[s] = row0;
      for (int r = 0; r < n; r += share, ++it) {
        item_seg[it] = s;
        item_row0[it] = row0 + r;
        item_nrows[it] = min(share, n - r);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    seg_off[nseg] = run.x;
    *n_items = run.y;
  }
}

int launch_items_from_counts(const int32_t *seg_count, int nseg, int rows_per_item, int32_t *seg_off,
                             int32_t *item_seg, int32_t *item_row0, int32_t *item_nrows, int32_t *n_items,
                             cudaStream_t st) {
  const int threads = nseg >= 1024 ? 1024 : (nseg + 31) / 32 * 32;
  coli_count_launch(1);
  return coli_cuda_check(launch_dependent(k_items_from_counts, dim3(1), dim3(threads > 0 ? threads : 32), 0, st, seg_count, nseg, rows_per_item,
                                          seg_off, item_seg, item_row0, item_nrows, n_items),
                         "work list launch")
             ? 1
             : 0;
}

}  // namespace colib

extern "C" int coli_b200_router_tile(int T, int E) { return T < 1 || E < 1 ? -1 : colib::pick_router_tile(T, E); }

// ---------------------------------------------------------------------------------------------
// Routing without any allocation.
//
// The router needs a [T,E] f32 logits buffer between its GEMM and its top-k kernel.  Every
// other entry point takes that buffer from a handle's cudaMalloc'ed workspace.  This one is for
// callers that must not allocate at all: a serving process that handed every free byte of HBM
// to its weight and KV pools at start-up (a later cudaMalloc there fails, or trips the host's
// memory ledger), and decode loops that cannot afford the device-wide synchronisation a
// cudaMalloc/cudaFree implies.  The logits live in a fixed array that is part of the library
// image, so each GPU that loads the library carries it (512 KiB) until the process exits.
//
// `g_route_scratch` below is a device symbol.  In host code the name is only a stand-in for
// it, not a device address, so the address handed to the kernels is looked up once per device
// with cudaGetSymbolAddress while that device is current.
// ---------------------------------------------------------------------------------------------
static __device__ __align__(256) float g_route_scratch[COLI_ROUTE_NOALLOC_MAX_LOGITS];

// Device address of the array per device ordinal, null until the first call on that device has
// looked it up.  Several host threads may make that first call at once: the address is published
// with release/acquire ordering, and two threads that both look it up store the same value.
static float *g_route_scratch_addr[COLI_CUDA_MAX_DEVICES];

extern "C" int coli_b200_route_noalloc(const void *x_dev, const void *router_w_dev, const float *select_bias_dev,
                                       const float *logit_bias_dev, int T, int H, int E, int k, int score,
                                       int norm_topk, float routed_scale, int n_group, int topk_group,
                                       int32_t *topk_idx_dev, float *topk_w_dev, void *stream) {
  if (!x_dev || !router_w_dev || !topk_idx_dev || !topk_w_dev || T < 0 || H < 1 || E < 1 || k < 1 || k > E) {
    coli_set_error("route_noalloc: null pointer or bad shape (T=%d H=%d E=%d k=%d)", T, H, E, k);
    return 0;
  }
  if ((long long)T * E > (long long)COLI_ROUTE_NOALLOC_MAX_LOGITS) {
    coli_set_error("route_noalloc: T*E = %lld exceeds the built-in scratch of %d logits; use a ColiMoe handle for larger batches",
                   (long long)T * E, COLI_ROUTE_NOALLOC_MAX_LOGITS);
    return 0;
  }
  if (score != COLI_SCORE_SOFTMAX && score != COLI_SCORE_SIGMOID) {
    coli_set_error("route_noalloc: unknown score function %d", score);
    return 0;
  }
  int dev = -1;
  if (!coli_cuda_check(cudaGetDevice(&dev), "route_noalloc: cudaGetDevice")) return 0;
  if (dev < 0 || dev >= COLI_CUDA_MAX_DEVICES) {
    coli_set_error("route_noalloc: device ordinal %d out of range", dev);
    return 0;
  }
  float *scratch = __atomic_load_n(&g_route_scratch_addr[dev], __ATOMIC_ACQUIRE);
  if (!scratch) {
    // set-up, once per device, with that device current: resolve the symbol to its device address
    float *ptr = nullptr;
    if (!coli_cuda_check(cudaGetSymbolAddress((void **)&ptr, g_route_scratch), "route_noalloc: cudaGetSymbolAddress")) return 0;
    if (!ptr) {
      coli_set_error("route_noalloc: scratch symbol resolved to a null address");
      return 0;
    }
    __atomic_store_n(&g_route_scratch_addr[dev], ptr, __ATOMIC_RELEASE);
    scratch = ptr;
  }
  if (T == 0) return 1;
  if (H % 8 == 0 && ((reinterpret_cast<uintptr_t>(x_dev) | reinterpret_cast<uintptr_t>(router_w_dev)) & 15)) {
    coli_set_error("route_noalloc: x_dev and router_w_dev must be 16-byte aligned (the router reads them with 128-bit loads)");
    return 0;
  }
  colib::RouteParams p;
  p.T = T;
  p.H = H;
  p.E = E;
  p.k = k;
  p.score = score;
  p.norm_topk = norm_topk;
  p.routed_scale = routed_scale;
  p.n_group = n_group < 1 ? 1 : n_group;
  p.topk_group = topk_group < 1 ? 1 : topk_group;
  p.x = (const __nv_bfloat16 *)x_dev;
  p.router_w = (const __nv_bfloat16 *)router_w_dev;
  p.select_bias = select_bias_dev;
  p.logit_bias = logit_bias_dev;
  p.logits = scratch;  // every logit of [T,E] is written before it is read: nothing to clear
  p.topk_idx = topk_idx_dev;
  p.topk_w = topk_w_dev;
  return colib::launch_router(p, (cudaStream_t)stream);
}

