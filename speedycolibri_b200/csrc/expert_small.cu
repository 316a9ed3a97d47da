// Expert FFN for decode-sized segments: a weight-streaming dequant-GEMV/GEMM in which every
// weight byte is read from HBM exactly once per work item with 128-bit loads, converted to
// f16 in registers (one hardware cvt per pair of FP4 or FP8 codes, one half2 multiply by the
// block scale for NVFP4), and contracted against eight token rows at a time with warp-level f16 MMA
// (m16n8k16, f32 accumulate).  The path is HBM-bound: the MMA only takes the multiply-adds
// off the CUDA cores so that the decode arithmetic (about one operation per FP4 weight) is
// all the SM has to issue per byte streamed.
//
// It replaces the reference's per-expert launch trios nvfp4_gemv / nvfp4_wsmm / fp8a16_gemv
// (crates/colibri-backend/cuda/backend_cuda.cu:707-1110,1436-1510,468-496, dispatched from
// 4738-4783) with two launches for ALL experts of a layer: gate+up with SiLU*mul fused
// (the reference runs `silu_mul` as a separate launch, backend_cuda.cu:3785-3787), then down.
//
// Numerics (W4A16 as in crates/colibri-engine/src/linear.rs:110-133): activations are the bf16
// values held in f16 (exact in [2^-14, 65504]), a decoded weight E2M1*ue4m3 has at most 6
// significant bits and is exact in f16, so
// each product is exact and only the f32 summation order differs from the CPU sum.  The
// per-tensor scale is applied once per output, as the reference does.  The intermediate
// h = silu(g)*u is rounded to bf16 (then held in f16) before the down projection.
//
// Two kernels: k_ffn_stream for items of at most eight rows (every decode call), and k_ffn_mm for the host calls
// that hand over up to 32 rows of one matrix.
//
// Work decomposition of k_ffn_mm: grid = (row tiles of 16 outputs, work items); an item is at most 8*NB
// consecutive rows of one expert segment.  The W warps of a CTA split the K axis (k-tile kt
// goes to warp kt % W) where there are few tasks, and reduce through shared memory.
#include "internal.cuh"

namespace colib {

__device__ __forceinline__ void mma_f16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ldg_nc_v4(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// Two bytes of a NVFP4 word (each byte = two consecutive k, low nibble first) -> two f16x2.
// HI selects bytes 2,3 of the word, otherwise bytes 0,1.
template <bool HI>
__device__ __forceinline__ void cvt_e2m1x4(uint32_t w, uint32_t &p0, uint32_t &p1) {
  if (HI)
    asm("{ .reg .b8 b0, b1, b2, b3;\n"
        "  mov.b32 {b0, b1, b2, b3}, %2;\n"
        "  cvt.rn.f16x2.e2m1x2 %0, b2;\n"
        "  cvt.rn.f16x2.e2m1x2 %1, b3; }\n"
        : "=r"(p0), "=r"(p1)
        : "r"(w));
  else
    asm("{ .reg .b8 b0, b1, b2, b3;\n"
        "  mov.b32 {b0, b1, b2, b3}, %2;\n"
        "  cvt.rn.f16x2.e2m1x2 %0, b0;\n"
        "  cvt.rn.f16x2.e2m1x2 %1, b1; }\n"
        : "=r"(p0), "=r"(p1)
        : "r"(w));
}
// One FP8 word (four consecutive k) -> two f16x2; also used for a pair of ue4m3 block scales.
__device__ __forceinline__ void cvt_e4m3x4(uint32_t w, uint32_t &p0, uint32_t &p1) {
  asm("{ .reg .b16 h0, h1;\n"
      "  mov.b32 {h0, h1}, %2;\n"
      "  cvt.rn.f16x2.e4m3x2 %0, h0;\n"
      "  cvt.rn.f16x2.e4m3x2 %1, h1; }\n"
      : "=r"(p0), "=r"(p1)
      : "r"(w));
}

template <int FMT>
struct AFrag {
  // raw bytes of rows g and g+8 of one 16-row tile for one k-tile, as loaded by this lane
  uint4 lo[FMT == COLI_FMT_NVFP4 ? 1 : 2], hi[FMT == COLI_FMT_NVFP4 ? 1 : 2];
  uint32_t sc;  // NVFP4: two scale bytes of row g (low 16 bits) and of row g+8 (high 16 bits)
};

template <int FMT>
__device__ __forceinline__ void load_a(AFrag<FMT> &f, const WeightRef &w, int Op, int r0, int kt, int lane) {
  if (FMT == COLI_FMT_NVFP4) {
    const uint8_t *slab = w.q + ((size_t)kt * Op + r0) * 64;
    // chunk t of rows g and g + 8 (r0 is a multiple of 16, so both are permuted alike)
    const int off = (lane >> 2) * 64 + coli_fp4_chunk(lane >> 2, lane & 3) * 16;
    f.lo[0] = ldg_nc_v4(slab + off);
    f.hi[0] = ldg_nc_v4(slab + 512 + off);
    const uint8_t *ss = w.s + ((size_t)kt * Op + r0) * 8;
    const uint32_t s0 = *reinterpret_cast<const uint16_t *>(ss + lane * 2);
    const uint32_t s1 = *reinterpret_cast<const uint16_t *>(ss + 64 + lane * 2);
    f.sc = s0 | (s1 << 16);
  } else {
    const uint8_t *slab = w.q + ((size_t)kt * Op + r0) * 128;
    const int g = lane >> 2, off0 = g * 128 + coli_fp8_chunk(g, 2 * (lane & 3)) * 16, off1 = off0 ^ 16;
    f.lo[0] = ldg_nc_v4(slab + off0);
    f.lo[1] = ldg_nc_v4(slab + off1);
    f.hi[0] = ldg_nc_v4(slab + 1024 + off0);
    f.hi[1] = ldg_nc_v4(slab + 1024 + off1);
    f.sc = 0;
  }
}

// Per k-tile: the lane's four block scales (rows g and g+8, two 16-k blocks each) as f16; the multiply takes
// either half of a pair as its operand.
struct AScale {
  __half2 lo, hi;
};
template <int FMT>
__device__ __forceinline__ AScale decode_scales(const AFrag<FMT> &f) {
  AScale r = {};
  if (FMT == COLI_FMT_NVFP4) {
    uint32_t sl, sh;
    cvt_e4m3x4(f.sc, sl, sh);  // (s_blk0, s_blk1) of row g; of row g+8
    r.lo = *reinterpret_cast<const __half2 *>(&sl);
    r.hi = *reinterpret_cast<const __half2 *>(&sh);
  }
  return r;
}
__device__ __forceinline__ uint32_t scaled_by(uint32_t v, __half2 pair, bool high) {
  const __half2 z = __hmul2_rn(*reinterpret_cast<const __half2 *>(&v), high ? __high2half2(pair) : __low2half2(pair));
  return *reinterpret_cast<const uint32_t *>(&z);
}

// Decode the fragment of MMA step m (0..7) of a k-tile: a[0],a[2] = row g pairs, a[1],a[3] = row g+8.
template <int FMT>
__device__ __forceinline__ void decode_a(const AFrag<FMT> &f, const AScale &sc, int m, uint32_t (&a)[4]) {
  if (FMT == COLI_FMT_NVFP4) {
    const uint32_t wl = (&f.lo[0].x)[m >> 1], wh = (&f.hi[0].x)[m >> 1];
    uint32_t l0, l1, h0, h1;
    if (m & 1) {
      cvt_e2m1x4<true>(wl, l0, l1);
      cvt_e2m1x4<true>(wh, h0, h1);
    } else {
      cvt_e2m1x4<false>(wl, l0, l1);
      cvt_e2m1x4<false>(wh, h0, h1);
    }
    a[0] = scaled_by(l0, sc.lo, m >= 4);
    a[2] = scaled_by(l1, sc.lo, m >= 4);
    a[1] = scaled_by(h0, sc.hi, m >= 4);
    a[3] = scaled_by(h1, sc.hi, m >= 4);
  } else {
    const uint32_t wl = (&f.lo[m >> 2].x)[m & 3], wh = (&f.hi[m >> 2].x)[m & 3];
    cvt_e4m3x4(wl, a[0], a[2]);
    cvt_e4m3x4(wh, a[1], a[3]);
  }
}

// One matrix over items of 9 to 32 rows: the f32 matmul and ReLU^2 calls on host buffers.
// SPLITK: grid = (row tiles, work items); the W warps of a CTA share one 16-row tile and split
// the k-tiles (few work items).  Otherwise the grid is one-dimensional and sized to what is resident at
// once; every warp walks (item, row tile) tasks with a stride, owns its tile over all of K and needs no
// cross-warp reduction.
template <int FMT, int NB, bool SPLITK>
__global__ void __launch_bounds__(SPLITK ? 256 : 64, SPLITK                  ? 1
                                                      : FMT == COLI_FMT_NVFP4 ? (NB == 2 ? 8 : 4)
                                                                              : (NB == 2 ? 5 : 4))
    k_ffn_mm(FfnParams p) {
  // weight ring depth (k-tiles) and token-fragment ring depth (quarter k-tiles)
  constexpr int D = 2;
  constexpr int R = NB <= 2 ? 4 : 2;
  constexpr int PF = R - 1;
  extern __shared__ __align__(16) float red[];  // [W][NB*4][32]
  coli_grid_dependency_sync();
  const int n_items = *p.n_items;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int K = p.I, Oout = p.H;  // contraction length, output features
  const int Kp = (K + 127) & ~127, KT = Kp >> 7, Op = (Oout + 15) & ~15;
  const int row_tiles = Op >> 4;

  // Tasks are (item, row tile) pairs, one per warp and round (per CTA when K is split).  The entry of a
  // task is requested a task ahead, the first one beside the item count.
  const int n_warps = (int)gridDim.x * W;
  const int n_tasks = n_items * row_tiles;
  struct ItemInfo {
    int seg, row0, nrows;
  };
  auto item_of = [&](int task) {  // the lists hold max_items entries, of which n_items are in use
    ItemInfo r = {0, 0, 0};
    const int item = task / row_tiles;
    if (item < p.max_items) r = {p.item_seg[item], p.item_row0[item], p.item_nrows[item]};
    return r;
  };
  // the first task's entry is requested beside the item count, not after it
  ItemInfo next = item_of(SPLITK ? (int)blockIdx.y * row_tiles + (int)blockIdx.x : (int)blockIdx.x * W + warp);
  for (int done = 0; done < n_tasks; done += n_warps) {
    const int task = SPLITK ? (int)blockIdx.y * row_tiles + (int)blockIdx.x : done + (int)blockIdx.x * W + warp;
    if (task >= n_tasks) break;
    const int r0 = (task % row_tiles) * 16;
    const int seg = next.seg, row0 = next.row0, nrows = next.nrows;
    if (!SPLITK) next = item_of(task + n_warps);
    const int ex = p.seg_expert ? p.seg_expert[seg] : seg;
    const WeightRef w0 = p.down[ex];

    // source row of token column g of each 8-token block (nullptr = column beyond the item)
    const __half *xrow[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      const int r = 8 * j + g;
      xrow[j] = r < nrows ? p.h + (size_t)(row0 + r) * K : nullptr;
    }

    float acc[NB][4];
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[j][c] = 0.0f;

    const int kstep = SPLITK ? W : 1;
    const int kt_first = SPLITK ? warp : 0;

    // token fragments: lane (g,t) reads x[token g][kt*128 + 32t + 8c .. +7] (16 bytes, two MMA
    // steps) for quarter c of k-tile kt
    auto load_x = [&](uint4 (&dst)[NB], int kt, int c) {
      const int k0 = kt * 128 + t * 32 + c * 8;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        dst[j] = make_uint4(0, 0, 0, 0);
        if (xrow[j] != nullptr && kt < KT && k0 + 8 <= K) dst[j] = *reinterpret_cast<const uint4 *>(xrow[j] + k0);
      }
    };

    // Register rings, both unrolled so that every slot is a fixed set of registers (rotating
    // slots with copies would make each iteration wait for the youngest load): packed weight
    // fragments D k-tiles deep, token fragments R quarter-k-tiles deep.
    AFrag<FMT> ring[D];
    uint4 xq[R][NB];
#pragma unroll
    for (int j = 0; j < D - 1; ++j) {
      const int ktl = kt_first + j * kstep;
      if (ktl < KT) load_a<FMT>(ring[j], w0, Op, r0, ktl, lane);
    }
#pragma unroll
    for (int f = 0; f < PF; ++f) load_x(xq[f % R], kt_first + (f / 4) * kstep, f % 4);

    for (int kt0 = kt_first; kt0 < KT; kt0 += D * kstep) {
#pragma unroll
      for (int slot = 0; slot < D; ++slot) {
        const int kt = kt0 + slot * kstep;
        if (kt >= KT) break;
        const int ktn = kt + (D - 1) * kstep;
        if (ktn < KT) load_a<FMT>(ring[(slot + D - 1) % D], w0, Op, r0, ktn, lane);
        const AScale asc = decode_scales<FMT>(ring[slot]);
        float part[NB][4];
        if (FMT == COLI_FMT_FP8_B128) {
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) part[j][c] = 0.0f;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int f = slot * 4 + c;  // position in the unrolled body; 4*D is a multiple of R
          load_x(xq[(f + PF) % R], kt + ((c + PF) / 4) * kstep, (c + PF) % 4);
          const uint4(&xb)[NB] = xq[f % R];
#pragma unroll
          for (int mm = 0; mm < 2; ++mm) {
            const int m = 2 * c + mm;
            uint32_t a[4];
            decode_a<FMT>(ring[slot], asc, m, a);
#pragma unroll
            for (int j = 0; j < NB; ++j) {
              const uint32_t b0 = mm ? xb[j].z : xb[j].x, b1 = mm ? xb[j].w : xb[j].y;
              mma_f16_16816(FMT == COLI_FMT_FP8_B128 ? part[j] : acc[j], a, b0, b1);
            }
          }
        }
        if (FMT == COLI_FMT_FP8_B128) {
          // one f32 scale per (128-row block, k-tile): convert.rs:731-741
          const float s = reinterpret_cast<const float *>(w0.s)[(size_t)(r0 >> 7) * KT + kt];
#pragma unroll
          for (int j = 0; j < NB; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[j][c] = fmaf(s, part[j][c], acc[j][c]);
        }
      }
    }

    // epilogue of one 8-token block given its reduced accumulators
    auto emit = [&](int j, const float(&v)[4]) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int orow = r0 + g + ((c & 2) ? 8 : 0);  // output feature
        const int col = 8 * j + 2 * t + (c & 1);      // token within the item
        if (orow >= Oout || col >= nrows) continue;
        const float s0 = FMT == COLI_FMT_NVFP4 ? w0.g : FMT == COLI_FMT_E4M3_ROW ? reinterpret_cast<const float *>(w0.s)[orow] : 1.0f;
        const size_t row = (size_t)(row0 + col);
        if (p.relu2_out) {
          const float r = fmaxf(v[c] * s0, 0.0f);
          p.relu2_out[row * p.H + orow] = coli_f32_to_f16_via_bf16(r * r);
        } else {
          p.y32[row * p.H + orow] = v[c] * s0;
        }
      }
    };

    if (!SPLITK) {
#pragma unroll
      for (int j = 0; j < NB; ++j) emit(j, acc[j]);
      continue;
    }

    // cross-warp (split-K) reduction; every warp of the CTA is on the same task
    constexpr int NV = NB * 4;
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) red[((size_t)warp * NV + j * 4 + c) * 32 + lane] = acc[j][c];
    __syncthreads();

    for (int j = warp; j < NB; j += W) {
      float v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float s = 0.0f;
        for (int w = 0; w < W; ++w) s += red[((size_t)w * NV + j * 4 + c) * 32 + lane];
        v[c] = s;
      }
      emit(j, v);
    }
    break;  // the CTA's only task
  }
}


// ---- items of at most eight rows: the decode kernel -----------------------------------------------------
// A warp's task is a pair of weight slabs of 16 R rows over all of K -- gate and up of the same features, or two
// adjacent slabs of down -- and its packed k-tiles come through a shared-memory ring of its own, filled by cp.async
// STAGES - 1 k-tiles ahead, across the ends of tasks: no barrier between warps, and the loads never drain.
// Two CTAs of eight or nine warps fill an SM; of every CTA as many warps work as make the rounds of tasks come out even.
// Calls with few tasks split the K of each among 2, 4 or 8 warps of a CTA, so that a single token still loads on every SM.
// An output's products are added in one order, k ascending, or where K is split in as many sums as split_of_k says: by the
// shapes of the call alone, whatever the routing and wherever in the work list a row lies.  (With only the tasks of the last round split,
// by how many there turned out to be, the launches were shorter -- 8 tokens 52.8 us a call against 54.9, 24 tokens 76.2 against
// 81.5 -- and a row's bits changed with its place and with the other tokens' routing.)
// Tasks of the down projection are known before its input is: launched behind the gate/up launch of this
// kernel (which lets it start only when the work list is complete), its warps fill their rings first.
//
// What bounds it: instruction issue (0.57 of the slots; with the weight loads taken out the launches take 0.87 of
// their time, with the token loads out 0.95, with the MMAs out 0.92), and on a large layer the power limit: packed
// weights read at 7 TB/s and nothing else already hold this GPU at 1000 W and 1.44 GHz, so every instruction left out
// comes back as clock.  Per 2304 bytes of weights it executes 210 warp instructions with 32-row slabs and 249 with
// 16-row ones, 144 of them conversions, scale multiplies and MMAs; a kernel with the weights in a register ring
// two k-tiles deep took 257, had half of a warp's time behind its loads, and needed a second wave of CTAs for a
// single token.  Calls, with that kernel and with this one (us): H 2048, I 768, 128 experts 1 token 35.0 -> 24.8, 8 tokens
// 58.7 -> 54.9, 24 tokens 90.8 -> 81.5, 48 tokens 117 -> 99.5; FP8, 21 tokens 99.6 -> 94.5; 24 tokens on H 7168, I 2048, 256 experts
// 769 -> 630.  Nine warps for eight: one round instead of two at 8 tokens, 57.4 -> 54.9.  A lone warp needs half a microsecond a
// k-tile, so a round that few warps work on is long; its two slabs in two warps were no faster (61.3 -> 64.0).
// Built and no better: six ring stages instead of five, one CTA of 16 warps, ring slots of two k-tiles (more instructions).
template <int FMT, int R, int SETS>  // SETS: 0, or of a split K how many of its sums a warp makes
struct StreamTile {
  static constexpr int WARPS = FMT == COLI_FMT_NVFP4 && R == 1 && SETS == 0 ? 9 : 8, CTAS = 2;
  static constexpr int QB = FMT == COLI_FMT_NVFP4 ? 64 : 128;  // code bytes of a row and k-tile
  static constexpr int SB = FMT == COLI_FMT_NVFP4 ? 8 : 0;     // scale bytes
  static constexpr int Q = 16 * R * QB;                        // codes of one slab and k-tile
  static constexpr int SLOT = 2 * 16 * R * (QB + SB);          // both slabs' codes, then their scales
  static constexpr int STAGES = FMT == COLI_FMT_NVFP4 && R == 1 ? 5 : 3;
  static constexpr int UNITS = 8 / R;                          // tasks a warp's loads may be ahead, and more
  static constexpr int SUMS = SETS * 2 * R * 4 * 32;           // floats of a warp's sums of a split task
  static_assert(UNITS > STAGES, "task queue");
};
struct __align__(16) StreamUnit {  // what the multiplying side of a warp needs of a task
  int row0, nrows, r0, pad;
  const float *sc0, *sc1;          // FP8: scales of the two slabs' matrices
  float g0, g1;
  int tok[8];                      // source row of each token column (columns past nrows repeat the last)
};
template <int FMT, int R, int SETS>
constexpr size_t stream_smem() {
  using C = StreamTile<FMT, R, SETS>;
  return (size_t)C::WARPS * (C::STAGES * C::SLOT + C::UNITS * sizeof(StreamUnit) + C::SUMS * sizeof(float));
}
template <int FMT, bool GATED, int R, int SETS>
__global__ void __launch_bounds__(R == 1 && SETS == 0 ? 288 : 256, 2) k_ffn_stream(FfnParams p, int items_known, int ks) {
  using C = StreamTile<FMT, R, SETS>;
  constexpr int QB = C::QB, SB = C::SB, STAGES = C::STAGES, ROWS = GATED ? 16 * R : 32 * R;
  constexpr bool FP4 = FMT == COLI_FMT_NVFP4, SPLIT = SETS > 0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);  // (known to be the same in all lanes)
  const int K = GATED ? p.H : p.I, Oout = GATED ? p.I : p.H;
  const int KT = (K + 127) >> 7, Op = (Oout + 15) & ~15;
  const int tiles = (Op + ROWS - 1) / ROWS;  // tasks of an item
  const __half *src = GATED ? p.x : p.h;
  unsigned char *ring = smem_raw + warp * (STAGES * C::SLOT);
  const uint32_t ring_u = (uint32_t)__cvta_generic_to_shared(ring), ring_end = ring_u + STAGES * C::SLOT;
  StreamUnit *queue = reinterpret_cast<StreamUnit *>(smem_raw + C::WARPS * STAGES * C::SLOT) + warp * C::UNITS;

  if (!items_known) coli_grid_wait();
  if (GATED) coli_grid_trigger();  // behind the wait: the successor may read the work list at once
  const int n_tasks = __ldcg(p.n_items) * tiles;
  // Tasks of a round: one for `step` warps of a CTA (SPLIT: the ks that share its K; otherwise one), with as many warps of
  // every CTA at work as make the rounds come out even.
  const int step = SPLIT ? ks : 1, piece = SPLIT ? warp % step : 0;
  const int grid = (int)gridDim.x, rounds = (n_tasks + grid * C::WARPS - 1) / (grid * C::WARPS);
  const int busy = SPLIT || rounds == 0 ? C::WARPS : (n_tasks + grid * rounds - 1) / (grid * rounds);
  const int round = grid * busy / step;
  const int full = n_tasks / round, rest = n_tasks - full * round;
  const int spread = (warp / step) * grid + (int)blockIdx.x;  // the last round: over the CTAs
  const int n_units = warp < busy ? full + (spread < rest ? 1 : 0) : 0;

  // ---- loading side ----
  struct Item {
    int seg, row0, nrows, tile;
  };
  const int dq = round / tiles, dr = round - dq * tiles;  // from one round's task to the next's
  int fi, ft;
  {
    const int first = SPLIT ? spread : (int)blockIdx.x * busy + warp;
    fi = first / tiles;
    ft = first - fi * tiles;
  }
  auto fetch_item = [&](int v) {  // called for v = 0, 1, 2, ...
    Item it = {0, 0, 1, 0};
    if (v < n_units) {
      if (v == full) {
        const int task = full * round + spread;
        fi = task / tiles;
        ft = task - fi * tiles;
      }
      it = {__ldcg(p.item_seg + fi), __ldcg(p.item_row0 + fi), __ldcg(p.item_nrows + fi), ft};
      fi += dq;
      ft += dr;
      if (ft >= tiles) {
        ft -= tiles;
        ++fi;
      }
    }
    return it;
  };
  const uint8_t *rq0 = nullptr, *rq1 = nullptr, *rs0 = nullptr, *rs1 = nullptr;  // the next unit's matrices
  float rg0 = 0.0f, rg1 = 0.0f;
  int rtok = 0;
  auto fetch_ref = [&](int v, const Item &it) {
    if (v >= n_units) return;
    const int ex = p.seg_expert ? p.seg_expert[it.seg] : it.seg;
    const WeightRef *a = (GATED ? p.gate : p.down) + ex;
    rq0 = a->q, rs0 = a->s, rg0 = a->g;
    if (GATED) {
      const WeightRef *b = p.up + ex;
      rq1 = b->q, rs1 = b->s, rg1 = b->g;
    } else {
      rq1 = rq0, rs1 = rs0, rg1 = rg0;
    }
    const int row = it.row0 + min(g, it.nrows - 1);
    rtok = GATED && p.row_token ? __ldcg(p.row_token + row) : row;
  };
  int lv = 0, left = 0;  // unit and k-tiles that the loads are at
  const uint8_t *q0 = nullptr, *q1 = nullptr, *sp = nullptr;
  size_t qstep = 0, sstep = 0;
  Item it_next = fetch_item(0), it_after = fetch_item(1);
  fetch_ref(0, it_next);
  auto enter_unit = [&]() {  // unit lv: its matrices have been fetched; the next one's follow
    const int r0 = it_next.tile * ROWS;
    // (a missing second slab, R = 1 only: the first one again, and nothing of it is stored)
    const int r1 = GATED ? r0 : (r0 + 16 * R < Op ? r0 + 16 * R : r0);
    const size_t krow = (size_t)piece * Op;
    q0 = rq0 + (krow + r0) * QB + lane * 16;
    q1 = rq1 + (krow + r1) * QB + lane * 16;
    if (FP4) sp = (lane < 8 * R ? rs0 + (krow + r0) * SB : rs1 + (krow + r1) * SB) + (lane & (8 * R - 1)) * 16;
    qstep = (size_t)step * Op * QB;
    sstep = (size_t)step * Op * SB;
    left = (KT - piece + step - 1) / step;
    StreamUnit &u = queue[lv % C::UNITS];
    if (lane == 0) {
      u.row0 = it_next.row0;
      u.nrows = it_next.nrows;
      u.r0 = r0;
      u.sc0 = reinterpret_cast<const float *>(rs0);
      u.sc1 = reinterpret_cast<const float *>(rs1);
      u.g0 = rg0;
      u.g1 = rg1;
    }
    if (t == 0) u.tok[g] = rtok;
    it_next = it_after;
    fetch_ref(lv + 1, it_next);
    it_after = fetch_item(lv + 2);
  };
  uint32_t fill = ring_u;  // the slot that is filled next
  auto issue = [&]() {
    if (left > 0) {
      const uint32_t d = fill + lane * 16;
#pragma unroll
      for (int i = 0; i < C::Q / 512; ++i) {
        cp_async16(d + i * 512, q0 + i * 512);
        cp_async16(d + C::Q + i * 512, q1 + i * 512);
      }
      if (FP4 && lane < 16 * R) cp_async16(d + 2 * C::Q, sp);
      q0 += qstep;
      q1 += qstep;
      if (FP4) sp += sstep;
      fill += C::SLOT;
      if (fill == ring_end) fill = ring_u;
      if (--left == 0 && ++lv < n_units) enter_unit();
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (n_units > 0) enter_unit();
#pragma unroll 1
  for (int i = 0; i < STAGES - 1; ++i) issue();
  if (items_known) coli_grid_wait();  // the input rows
  if (!GATED) coli_grid_trigger();
  __syncwarp();

  // ---- multiplying side ----
  // token fragments: lane (g, t) reads x[token g][kt*128 + 32t + 8c .. +7] (16 bytes, two MMA steps), a k-tile ahead
  const __half *xp = src;  // this lane's fragments of the k-tile loaded last
  bool column = false;
  const bool ragged = (K & 127) != 0;
  auto load_x = [&](uint4 (&x)[4], int kt) {
    if (!ragged || kt + 1 < KT) {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (column) x[c] = *reinterpret_cast<const uint4 *>(xp + 8 * c);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        x[c] = make_uint4(0, 0, 0, 0);
        if (column && kt * 128 + t * 32 + 8 * c + 8 <= K) x[c] = *reinterpret_cast<const uint4 *>(xp + 8 * c);
      }
    }
  };
  // A lane whose column is no row of the item keeps zeros: multiplied by copies of a row instead, the empty
  // columns drew power, and on a large layer the launch runs against the power limit.
  uint4 xa[4], xb[4];
  auto enter_x = [&](uint4 (&x)[4], int v) {
    const StreamUnit &e = queue[v % C::UNITS];
    column = g < e.nrows;
    xp = src + (size_t)e.tok[g] * K + piece * 128 + t * 32;
#pragma unroll
    for (int c = 0; c < 4; ++c) x[c] = make_uint4(0, 0, 0, 0);
    load_x(x, piece);
  };
  if (n_units > 0) enter_x(xa, 0);
  constexpr int NT = 2 * R;  // tile j: rows 16 (j % R) of slab j / R
  float acc[SETS > 1 ? 2 : 1][NT][4];
  // where this lane reads its codes: chunk t (FP8: 2t) of row g
  const uint32_t code_off = FP4 ? g * 64 + coli_fp4_chunk(g, t) * 16 : g * 128 + coli_fp8_chunk(g, 2 * t) * 16;
  uint32_t base = ring_u;  // the slot in use
  int row0 = 0, nrows = 0, r0 = 0;
  const StreamUnit *u = queue;

  // element c of the sums of slab 0 and slab 1 at row tile r
  auto emit = [&](int c, int r, float v0, float v1) {
    const int col = 2 * t + (c & 1), o0 = r0 + 16 * r + g + ((c & 2) ? 8 : 0), o1 = GATED ? o0 : o0 + 16 * R;
    if (col >= nrows) return;
    float s0 = 1.0f, s1 = 1.0f;
    if (FP4) {
      s0 = u->g0;
      s1 = u->g1;
    } else if (FMT == COLI_FMT_E4M3_ROW) {
      s0 = o0 < Oout ? u->sc0[o0] : 0.0f;
      s1 = o1 < Oout ? u->sc1[o1] : 0.0f;
    }
    const size_t row = (size_t)(row0 + col);
    if constexpr (GATED) {
      if (o0 < Oout) p.h[row * p.I + o0] = coli_f32_to_f16_via_bf16(coli_act_fast(v0 * s0, v1 * s1, p.act));
    } else {
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int o = m ? o1 : o0;
        const float v = m ? v1 * s1 : v0 * s0;
        if (o >= Oout) continue;
        if (p.relu2_out) {
          const float f = fmaxf(v, 0.0f);
          p.relu2_out[row * p.H + o] = coli_f32_to_f16_via_bf16(f * f);
        } else if (p.y32) {
          p.y32[row * p.H + o] = v;
        } else {
          p.y[row * p.H + o] = __float2bfloat16_rn(v);
        }
      }
    }
  };

  // one k-tile, added to `acc`: its token fragments are in x; `more`: the task goes on at k-tile `next`, whose fragments go
  // to xnext, otherwise those of the next task's first k-tile do
  auto k_tile = [&](float (&acc)[NT][4], const uint4 (&x)[4], uint4 (&xnext)[4], int v, int kt, bool more, int next) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncwarp();  // this k-tile has arrived for every lane, and the slot before it has been read by all
    issue();
    if (more) {
      xp += (next - kt) * 128;
      load_x(xnext, next);
    } else if (v + 1 < n_units) {
      enter_x(xnext, v + 1);
    }
    float kscale[2] = {1.0f, 1.0f};
    if (FMT == COLI_FMT_FP8_B128) {  // one f32 scale per (128-row block, k-tile): convert.rs:731-741
      const int rb = (r0 >> 7) * KT + kt;
      kscale[0] = __ldg(u->sc0 + rb);
      kscale[1] = GATED ? __ldg(u->sc1 + rb) : kscale[0];  // (both down slabs are in one block of 128 rows)
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      AFrag<FMT> f[2];
      AScale asc[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const uint32_t q = base + m * C::Q + r * 16 * QB;
        if constexpr (FP4) {
          const uint32_t sc = base + 2 * C::Q + (m * R + r) * 128 + lane * 2;
          f[m].lo[0] = lds128(q + code_off);
          f[m].hi[0] = lds128(q + 512 + code_off);
          uint16_t a, b;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(a) : "r"(sc) : "memory");
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(b) : "r"(sc + 64) : "memory");
          f[m].sc = (uint32_t)a | ((uint32_t)b << 16);
        } else {
          f[m].lo[0] = lds128(q + code_off);
          f[m].lo[1] = lds128(q + (code_off ^ 16));
          f[m].hi[0] = lds128(q + 1024 + code_off);
          f[m].hi[1] = lds128(q + 1024 + (code_off ^ 16));
          f[m].sc = 0;
        }
        asc[m] = decode_scales<FMT>(f[m]);
      }
      float part[2][4];
      if (FMT == COLI_FMT_FP8_B128) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int c = 0; c < 4; ++c) part[m][c] = 0.0f;
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const uint4 &xv = x[s >> 1];
        const uint32_t b0 = (s & 1) ? xv.z : xv.x, b1 = (s & 1) ? xv.w : xv.y;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint32_t a[4];
          decode_a<FMT>(f[m], asc[m], s, a);
          mma_f16_16816(FMT == COLI_FMT_FP8_B128 ? part[m] : acc[m * R + r], a, b0, b1);
        }
      }
      if (FMT == COLI_FMT_FP8_B128) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[m * R + r][c] = fmaf(kscale[m], part[m][c], acc[m * R + r][c]);
      }
    }
    base += C::SLOT;
    if (base == ring_end) base = ring_u;
  };

  float *const sums = reinterpret_cast<float *>(smem_raw + C::WARPS * (STAGES * C::SLOT + C::UNITS * sizeof(StreamUnit)));  // SPLIT
  for (int v = 0; v < n_units; ++v) {
    u = queue + v % C::UNITS;
    row0 = u->row0;
    nrows = u->nrows;
    r0 = u->r0;
#pragma unroll
    for (int i = 0; i < (SETS > 1 ? 2 : 1); ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.0f;
    if (!column) {
#pragma unroll
      for (int c = 0; c < 4; ++c) xb[c] = make_uint4(0, 0, 0, 0);
    }
    int kt = piece;
#pragma unroll 1
    for (; kt + step < KT; kt += 2 * step) {  // two buffers of fragments in turn: no copies between them
      k_tile(acc[0], xa, xb, v, kt, true, kt + step);
      k_tile(acc[SETS > 1 ? 1 : 0], xb, xa, v, kt + step, kt + 2 * step < KT, kt + 2 * step);
    }
    if (kt < KT) {
      k_tile(acc[0], xa, xb, v, kt, false, 0);
#pragma unroll
      for (int c = 0; c < 4; ++c) xa[c] = xb[c];
    }
    if constexpr (SPLIT) {  // the task's sums, in the order of the k-tiles they start with
      auto group_barrier = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / step), "r"(32 * step) : "memory"); };
#pragma unroll
      for (int i = 0; i < SETS; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c) sums[warp * C::SUMS + ((i * NT + j) * 4 + c) * 32 + lane] = acc[i][j][c];
      group_barrier();
      for (int e = piece; e < 4 * R; e += step) {  // element e % 4 of row tile e / 4
        float v0 = 0.0f, v1 = 0.0f;
        for (int i = 0; i < SETS; ++i)
          for (int w = 0; w < step; ++w) {
            const float *part = sums + (warp - piece + w) * C::SUMS + (i * NT * 4 + e) * 32 + lane;
            v0 += part[0];
            v1 += part[4 * R * 32];
          }
        emit(e & 3, e >> 2, v0, v1);
      }
      if (v + 1 < n_units) group_barrier();  // before the next task's sums
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) emit(c, r, acc[0][r][c], acc[0][R + r][c]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Warps that share a task, each with every ks-th k-tile, where there are too few (item, 16 rows) tasks to fill the SMs
// with one warp each.  A pure function of the shapes, and the same for every task of a launch: the order in which
// an output's products are added depends on neither the routing, the item's place in the list nor the other rows.
static int split_of_k(int items_expected, int O, int K) {
  const int KT = (K + 127) / 128;
  if ((long)(items_expected > 0 ? items_expected : 1) * ((O + 15) / 16) >= 12L * COLI_SMS) return 1;
  return KT >= 8 ? 8 : KT >= 4 ? 4 : KT >= 2 ? 2 : 1;
}
template <int FMT, int R, int SETS>
static int launch_stream(const FfnParams &p, bool gated, bool items_known, int ks, cudaStream_t st) {
  using C = StreamTile<FMT, R, SETS>;
  constexpr size_t smem = stream_smem<FMT, R, SETS>();
  static ColiPerDeviceOnce once[2];
  if (!(gated ? coli_set_smem_limit(once[0], k_ffn_stream<FMT, true, R, SETS>, smem, "expert ffn shared-memory attribute")
              : coli_set_smem_limit(once[1], k_ffn_stream<FMT, false, R, SETS>, smem, "expert ffn shared-memory attribute")))
    return 0;
  const dim3 grid(C::CTAS * COLI_SMS);
  const cudaError_t e = gated ? launch_dependent(k_ffn_stream<FMT, true, R, SETS>, grid, dim3(32 * C::WARPS), smem, st, p, 0, ks)
                              : launch_dependent(k_ffn_stream<FMT, false, R, SETS>, grid, dim3(32 * C::WARPS), smem, st, p, items_known ? 1 : 0, ks);
  coli_count_launch(1);
  return coli_cuda_check(e, "expert ffn launch") ? 1 : 0;
}
// Slabs of 16 or of 32 rows (NVFP4; of FP8's k-tiles, twice as long, two CTAs of 32-row rings do not fit an SM): the
// instructions around a k-tile are then spent on twice the weights (210 a 2304 bytes against 249), but there are half as many
// tasks, and with fewer than six of eight warps at work an SM waits for its loads.  Weighed as rounds x warps at work x
// instructions, with the tasks that independent, even routing gives.  Us a call, 16 / 32 rows, H 2048, I 768, 128 experts
// (gate+up): 4 tokens 41.8 / 46.3, 8 tokens 55.5 / 55.5, 12 tokens 67.4 / 64.3, 16 tokens 73.3 / 70.0, 24 tokens (one round of 32 rows and a
// little) 79.1 / 82.8, 48 tokens 104.4 / 99.1; H 7168, I 2048, 256 experts, 8 tokens 318 / 301, 24 tokens 713 / 630.
template <int FMT>
static int launch_stream_rows(const FfnParams &p, bool gated, bool items_known, cudaStream_t st) {
  const int O = gated ? p.I : p.H, K = gated ? p.H : p.I, KT = (K + 127) / 128, rows = gated ? 16 : 32, ctas = 2 * COLI_SMS;
  const long tasks = (long)p.items_likely * ((O + rows - 1) / rows);
  const int ks = split_of_k(p.items_expected, O, K);
  if (ks > 1) {
    // a sum a warp, or (NVFP4: FP8 leaves no room) two, which takes half as many warps: whichever has fewer k-tiles in a row,
    // the end of a task counted as two (us a call, 8 warps a task with one sum / 4 with two: H 2048, I 768, 2 tokens 35.1 / 33.8, 3 tokens 40.2 / 38.4)
    auto in_a_row = [&](int step) { return (tasks * step + ctas * 8 - 1) / (ctas * 8) * ((KT + step - 1) / step + 2); };
    if (FMT == COLI_FMT_NVFP4 && in_a_row(ks / 2) <= in_a_row(ks)) return launch_stream<FMT, 1, FMT == COLI_FMT_NVFP4 ? 2 : 1>(p, gated, items_known, ks / 2, st);
    return launch_stream<FMT, 1, 1>(p, gated, items_known, ks, st);
  }
  if constexpr (FMT == COLI_FMT_NVFP4) {
    auto cost = [&](long n, int warps, int least, int instructions) {
      const long rounds = (n + ctas * warps - 1) / (ctas * warps), busy = rounds ? (n + ctas * rounds - 1) / (ctas * rounds) : 0;
      return rounds * (busy > least ? busy : least) * instructions;
    };
    if (O % (2 * rows) == 0 && cost(tasks / 2, StreamTile<FMT, 2, 0>::WARPS, 6, 2 * 210) < cost(tasks, StreamTile<FMT, 1, 0>::WARPS, 1, 249))
      return launch_stream<FMT, 2, 0>(p, gated, items_known, 1, st);
  }
  return launch_stream<FMT, 1, 0>(p, gated, items_known, 1, st);
}
// ---- one token: down and combine ---------------------------------------------------------------------
// A CTA makes 16 features of the result: a warp for each of the token's rows (its k experts and the shared one), all
// of K through a ring of its own, then the weighted sum of k_combine -- the same terms, rounded the same way -- out of
// shared memory.  The result rows never leave the SM, and a launch and its wait are gone from a chain of four.
// The rings are filled before the input is there, as those of the kernel above.
// Two kernels / this one, us a call: H 2048, I 768, 128 experts 25.9 / 24.7, FP8 28.3 / 27.5; H 1024, I 512 18.8 / 17.4, I 768 20.8 / 19.6.
// Not from more features than SMs x 16 on (H 7168, I 2048, 256 experts 80.7 / 84.4), nor from eight k-tiles on, where one warp's
// chain is as long as that of eight warps that share the K: I 1024 20.8 / 21.5 (H 1024), 24.5 / 24.5 (1536), 27.6 / 27.6 (2048), 30.9 /
// 30.3 (2304); I 1408 32.8 / 34.6 (2048); I 2048 25.4 / 31.8 (1024), 37.0 / 40.8 (2048).
constexpr int kOneRows = 17, kOneStages = 6, kOneTiles = 7;
template <int FMT>
constexpr size_t one_smem(int rows) {  // a warp's ring, its row of the result, its sums
  return (size_t)rows * (kOneStages * 16 * (FMT == COLI_FMT_NVFP4 ? 72 : 128) + (16 + 4 * 16) * sizeof(float));
}
// CHAIN: all of K is one sum.  Otherwise k-tile kt adds into sum kt % ks and the sums are added in order, as the ks warps of a
// split task do it; two k-tiles, of different sums, are multiplied side by side.
template <int FMT, bool CHAIN>
__global__ void __launch_bounds__(32 * kOneRows) k_down_combine_one(FfnParams p, CombineParams c, const int32_t *topk_idx, int shared, int items_known, int ks) {
  constexpr bool FP4 = FMT == COLI_FMT_NVFP4;
  constexpr int QB = FP4 ? 64 : 128, SB = FP4 ? 8 : 0, Q = 16 * QB, SLOT = 16 * (QB + SB);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), rows = (int)blockDim.x >> 5;
  const int K = p.I, KT = (K + 127) >> 7, Op = (p.H + 15) & ~15, r0 = (int)blockIdx.x * 16;
  float *ys = reinterpret_cast<float *>(smem_raw + (size_t)rows * kOneStages * SLOT);  // [rows][16]
  float *sums = ys + rows * 16 + warp * (4 * 16);                                      // [ks][16], ks <= 4 with so few k-tiles
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem_raw) + warp * (kOneStages * SLOT);
  if (!items_known) coli_grid_wait();
  const int ex = warp < c.k ? __ldcg(topk_idx + warp) : shared;
  const int row = warp < c.k ? __ldcg(c.slot + warp) : c.k;
  const WeightRef w = p.down[ex];
  int kf = 0;  // the k-tile that is fetched next
  auto issue = [&]() {
    if (kf < KT) {
      const uint32_t d = ring + (kf % kOneStages) * SLOT + lane * 16;
      const uint8_t *q = w.q + ((size_t)kf * Op + r0) * QB + lane * 16;
#pragma unroll
      for (int i = 0; i < Q / 512; ++i) cp_async16(d + i * 512, q + i * 512);
      if (FP4 && lane < 8) cp_async16(d + Q, w.s + ((size_t)kf * Op + r0) * SB + lane * 16);
      ++kf;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int i = 0; i < kOneStages; ++i) issue();
  if (items_known) coli_grid_wait();
  coli_grid_trigger();
  const __half *h = p.h + (size_t)row * K + t * 32;  // column 0, the token, is read by the lanes of g = 0
  auto load_x = [&](uint4 (&x)[2][4], int kt) {      // of k-tiles kt and kt + 1
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = (kt + j) * 128 + 8 * i;
        x[j][i] = make_uint4(0, 0, 0, 0);
        if (g == 0 && k + t * 32 + 8 <= K) x[j][i] = *reinterpret_cast<const uint4 *>(h + k);
      }
  };
  uint4 xn[2][4];
  load_x(xn, 0);
  float acc[2][4] = {};
  const uint32_t code_off = FP4 ? g * 64 + coli_fp4_chunk(g, t) * 16 : g * 128 + coli_fp8_chunk(g, 2 * t) * 16;
#pragma unroll 1
  for (int kt = 0; kt < KT; kt += 2) {  // (behind an odd last k-tile the other half of the pair is not used)
    asm volatile("cp.async.wait_group %0;" ::"n"(kOneStages - 2) : "memory");
    __syncwarp();  // these k-tiles have arrived for every lane
    uint4 x[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) x[j][i] = xn[j][i];
    if (kt + 2 < KT) load_x(xn, kt + 2);
    AFrag<FMT> f[2];
    AScale asc[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t base = ring + ((kt + j) % kOneStages) * SLOT;
      if constexpr (FP4) {
        f[j].lo[0] = lds128(base + code_off);
        f[j].hi[0] = lds128(base + 512 + code_off);
        uint16_t a, b;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(a) : "r"(base + Q + lane * 2) : "memory");
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(b) : "r"(base + Q + 64 + lane * 2) : "memory");
        f[j].sc = (uint32_t)a | ((uint32_t)b << 16);
      } else {
        f[j].lo[0] = lds128(base + code_off);
        f[j].lo[1] = lds128(base + (code_off ^ 16));
        f[j].hi[0] = lds128(base + 1024 + code_off);
        f[j].hi[1] = lds128(base + 1024 + (code_off ^ 16));
        f[j].sc = 0;
      }
      asc[j] = decode_scales<FMT>(f[j]);
    }
    float *sum[2];  // (of lanes with t = 0: column 0, elements 0 and 2, is the token)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      sum[j] = sums + ((kt + j) & (ks - 1)) * 16 + g;
      if (!CHAIN || FMT == COLI_FMT_FP8_B128) {
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.0f;
      }
      if (!CHAIN && FMT != COLI_FMT_FP8_B128 && kt + j >= ks && t == 0) {
        acc[j][0] = sum[j][0];
        acc[j][2] = sum[j][8];
      }
    }
    auto mma = [&](int j, int to, int s) {
      const uint4 &xv = x[j][s >> 1];
      uint32_t a[4];
      decode_a<FMT>(f[j], asc[j], s, a);
      mma_f16_16816(acc[to], a, (s & 1) ? xv.z : xv.x, (s & 1) ? xv.w : xv.y);
    };
    if constexpr (CHAIN && FMT != COLI_FMT_FP8_B128) {
#pragma unroll
      for (int s = 0; s < 8; ++s) mma(0, 0, s);
      if (kt + 1 < KT) {
#pragma unroll
        for (int s = 0; s < 8; ++s) mma(1, 0, s);
      }
    } else {
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        mma(0, 0, s);
        mma(1, 1, s);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (t != 0 || kt + j >= KT) continue;
        if (FMT == COLI_FMT_FP8_B128) {  // one f32 scale per (128-row block, k-tile): convert.rs:731-741
          const float sc = __ldg(reinterpret_cast<const float *>(w.s) + (size_t)(r0 >> 7) * KT + kt + j);
          const bool first = kt + j < ks;
          sum[j][0] = fmaf(sc, acc[j][0], first ? 0.0f : sum[j][0]);
          sum[j][8] = fmaf(sc, acc[j][2], first ? 0.0f : sum[j][8]);
        } else {
          sum[j][0] = acc[j][0];
          sum[j][8] = acc[j][2];
        }
      }
    }
    __syncwarp();  // these slots have been read by all
    issue();
    issue();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (t == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int o = r0 + g + 8 * i;
      float v = 0.0f;
      if (CHAIN && FMT != COLI_FMT_FP8_B128)
        v = acc[0][2 * i];
      else
        for (int j = 0; j < ks; ++j) v += sums[j * 16 + g + 8 * i];
      if (FP4) v *= w.g;
      if (FMT == COLI_FMT_E4M3_ROW) v *= o < p.H ? reinterpret_cast<const float *>(w.s)[o] : 0.0f;
      ys[warp * 16 + g + 8 * i] = __bfloat162float(__float2bfloat16_rn(v));
    }
  }
  __syncthreads();
  const int o = r0 + (int)threadIdx.x;
  if (threadIdx.x >= 16 || o >= p.H) return;
  float sum = 0.0f;
  for (int kk = 0; kk < c.k; ++kk) sum = fmaf(c.topk_w[kk], ys[kk * 16 + threadIdx.x], sum);
  if (rows > c.k) sum += ys[c.k * 16 + threadIdx.x];
  if (c.resid) sum = c.resid[o] + sum;
  if (c.out32)
    c.out32[o] = sum;
  else
    c.out[o] = __float2bfloat16_rn(sum);
}
bool down_combine_one_ok(int rows, int H, int I) { return rows <= kOneRows && (H + 15) / 16 <= COLI_SMS && (I + 127) / 128 <= kOneTiles; }
template <int FMT, bool CHAIN>
static int launch_one_token_as(const FfnParams &p, const CombineParams &c, const int32_t *topk_idx, int shared, bool items_known, int ks, cudaStream_t st) {
  const int rows = c.k + c.has_shared;
  static ColiPerDeviceOnce once;
  if (!coli_set_smem_limit(once, k_down_combine_one<FMT, CHAIN>, one_smem<FMT>(kOneRows), "down of one token: shared-memory attribute")) return 0;
  coli_count_launch(1);
  return coli_cuda_check(launch_dependent(k_down_combine_one<FMT, CHAIN>, dim3((p.H + 15) / 16), dim3(32 * rows), one_smem<FMT>(rows), st, p, c, topk_idx, shared,
                                          items_known ? 1 : 0, ks),
                         "down of one token")
             ? 1
             : 0;
}
template <int FMT>
static int launch_one_token(const FfnParams &p, const CombineParams &c, const int32_t *topk_idx, int shared, bool items_known, cudaStream_t st) {
  const int ks = split_of_k(p.items_expected, p.H, p.I);
  return ks > 1 ? launch_one_token_as<FMT, false>(p, c, topk_idx, shared, items_known, ks, st)
                : launch_one_token_as<FMT, true>(p, c, topk_idx, shared, items_known, 1, st);
}
int launch_down_combine_one(const FfnParams &p, const CombineParams &c, const int32_t *topk_idx, int shared, bool items_known, cudaStream_t st) {
  switch (p.fmt) {
    case COLI_FMT_NVFP4:
      return launch_one_token<COLI_FMT_NVFP4>(p, c, topk_idx, shared, items_known, st);
    case COLI_FMT_FP8_B128:
      return launch_one_token<COLI_FMT_FP8_B128>(p, c, topk_idx, shared, items_known, st);
    case COLI_FMT_E4M3_ROW:
      return launch_one_token<COLI_FMT_E4M3_ROW>(p, c, topk_idx, shared, items_known, st);
  }
  coli_set_error("expert ffn: unsupported weight format %d", p.fmt);
  return 0;
}

template <int FMT, int NB>
static int launch_one(const FfnParams &p, cudaStream_t st) {
  const int row_tiles = (p.H + 15) / 16;
  const int W = split_of_k(p.items_expected, p.H, p.I);
  if (W > 1) {
    dim3 grid(row_tiles, p.max_items);
    const size_t sm = (size_t)W * NB * 4 * 32 * sizeof(float);
    const cudaError_t e = launch_dependent(k_ffn_mm<FMT, NB, true>, grid, dim3(W * 32), sm, st, p);
    coli_count_launch(1);
    return coli_cuda_check(e, "expert ffn launch") ? 1 : 0;
  } else {
    // two warps per CTA keep the per-SM share of tasks even; the grid covers what fits at once
    constexpr int W = 2;
    // resident CTAs per kernel variant and device ordinal (an occupancy figure belongs to one device)
    static int resident_tab[32];
    int dev = 0;
    if (!coli_cuda_check(cudaGetDevice(&dev), "device query")) return 0;
    int uncached = 0;
    int &resident_slot = (dev >= 0 && dev < 32) ? resident_tab[dev] : uncached;
    if (resident_slot == 0) {
      int sms = 0, per_sm = 0;
      if (!coli_cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "device query")) return 0;
      const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_ffn_mm<FMT, NB, false>, W * 32, 0);
      if (!coli_cuda_check(e, "occupancy query")) return 0;
      resident_slot = sms * (per_sm > 0 ? per_sm : 1);
    }
    const int resident_ctas = resident_slot;
    const long max_ctas = ((long)row_tiles * p.max_items + W - 1) / W;
    const int grid = (int)(max_ctas < resident_ctas ? max_ctas : resident_ctas);
    const cudaError_t e = launch_dependent(k_ffn_mm<FMT, NB, false>, dim3(grid), dim3(W * 32), 0, st, p);
    coli_count_launch(1);
    return coli_cuda_check(e, "expert ffn launch") ? 1 : 0;
  }
}

// rows_per_item the caller cut the work list with selects NB (8 * NB >= rows per item).
// items_known: a gate/up launch of the streaming kernel stands between the work list and this one.
static int launch_ffn_stage(const FfnParams &p, bool gated, bool items_known, cudaStream_t st) {
  if (p.max_items <= 0) return 1;
  if (p.H % 8 || p.I % 8) {
    coli_set_error("expert ffn: H=%d and I=%d must be multiples of 8", p.H, p.I);
    return 0;
  }
  if (p.rows_per_item > (gated ? 8 : 32)) {
    coli_set_error("expert ffn: rows_per_item=%d exceeds %d", p.rows_per_item, gated ? 8 : 32);
    return 0;
  }
  const int nb = p.rows_per_item <= 8 ? 1 : p.rows_per_item <= 16 ? 2 : 4;
#define COLI_DISPATCH(F) \
  (nb == 1 ? launch_stream_rows<F>(p, gated, items_known, st) : nb == 2 ? launch_one<F, 2>(p, st) : launch_one<F, 4>(p, st))
  switch (p.fmt) {
    case COLI_FMT_NVFP4:
      return COLI_DISPATCH(COLI_FMT_NVFP4);
    case COLI_FMT_FP8_B128:
      return COLI_DISPATCH(COLI_FMT_FP8_B128);
    case COLI_FMT_E4M3_ROW:
      return COLI_DISPATCH(COLI_FMT_E4M3_ROW);
    default:
      coli_set_error("expert ffn: unsupported weight format %d", p.fmt);
      return 0;
  }
#undef COLI_DISPATCH
}

int launch_gate_up_small(const FfnParams &p, cudaStream_t st) { return launch_ffn_stage(p, true, false, st); }
int launch_down_small(const FfnParams &p, bool behind_gate_up, cudaStream_t st) { return launch_ffn_stage(p, false, behind_gate_up, st); }
int launch_ffn_small(const FfnParams &p, cudaStream_t st) {
  return launch_gate_up_small(p, st) && launch_down_small(p, true, st);
}

}  // namespace colib
