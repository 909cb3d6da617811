// Grouped expert GEMM on the 5th-generation tensor cores, NVFP4 weights x fp16 activations (W4A16).
//
// Tokens arrive sorted by expert (`offsets[e]` .. `offsets[e+1]` are the rows of local expert e in the
// permuted activation matrix).  A persistent grid walks the (token tile of an expert, weight tile) pairs
// that have rows, dealt out in turn, so that every CTA has the same number of them whichever experts were chosen:
//
//   TMA warp         activation tile [BT tokens x 64 k] fp16, 128-byte swizzle
//   weight warp      e2m1 codes of 128 weight rows x 256 k by TMA (a 128-byte line a row), their e4m3 group scales by cp.async
//   dequant warps    codes and scales -> fp16 straight into tensor memory: a TMEM lane is a weight row, 64 k are 32 columns
//   MMA warp         tcgen05.mma kind::f16, weights from tensor memory and activations from shared memory, as many token columns
//                    as the tile has rows (in sixteens)
//   epilogue warps   FC1: a warp's lanes hold sixteen gate rows and the up rows of the same features, one shuffle brings a
//                    feature's two products together for SwiGLU with clamp, stored as fp16;
//                    FC2: scaled bf16 store.  Rows past the expert's last token are masked.
//
// e2m1 x e4m3 is exact in fp16, the per-matrix fp32 scale is applied in the epilogue.
//
// What bounds it.  Few rows: memory; the bytes in flight have to cover the trip (the ring holds 108 KB an SM and more; codes fetched
// into registers by the converting warps were 16 KB), and the issuing warp may not be in the way: a wait for a barrier that has long
// completed takes it 70 to 95 cycles, so a K step's barriers are looked at while the step before is issued, and its products are issued by
// one lane (N / 2 + 10 cycles each with weights in tensor memory; 82 to 90 under a lane predicate).  Many rows: a step of 2 x 128
// weight rows x 64 k and 128 tokens is 512 tensor-core cycles, 24 KB from L2 (550 cycles when every SM asks) and 300 cycles of
// conversion, which overlap as far as four steps in tensor memory allow.  Converted weights do not pass through shared memory.
// Measured (hidden 4096, 2048 rows an expert, top 6; device time of the first + the second product, us; before: operands converted
// into shared memory from codes in registers):
//   64 tokens, 256 experts    632 + 302 before, 350 + 193 now (5.3 TB/s)
//   4096 tokens, 256 experts  2409 + 1241, 1105 + 590
//   4096 tokens, 32 experts   756 + 398 now (1090 TFLOP/s); one weight tile x 256 tokens a unit: 1542 us for the whole, 1310 as it is
//
// This is the engine's counterpart of the reference's fused W4A16 MoE kernel and, for the
// expert-parallel layout, of its mega-MoE grouped GEMM (overlay/nvidia_model.py:227-559).
#include "codes.cuh"
#include "common.cuh"

namespace stk {

int make_tmap_2d(CUtensorMap* tm, const void* base, int elem_bytes, long long rows, long long cols, long long ld,
                 int box_rows);

struct MoeGArgs {
  const uint8_t* w;        // [E_l, rows, K/2]
  const uint8_t* s;        // [E_l, rows, K/16]
  const float* gscale;     // [E_l]
  const int* offsets;      // [E_l + 1]
  int e_local;
  int rows;                // weight rows per expert (2I for FC1, H for FC2)
  int n_out;               // output features per token (I for FC1, H for FC2)
  int K;
  void* out;               // FC1: fp16 [P, I]; FC2: bf16 [P, H]
  float limit;
  int scale_copy;          // bytes of one copy of scales: 16, 4 or (unaligned scales) 1
  int* status;
  // Expert-parallel mode: rows of expert e are pushed into the activation matrix by peers (and by this
  // GPU's own dispatch); `arrived[e]` counts the rows that have landed.  nullptr = rows are already there.
  const uint32_t* arrived;
  uint32_t spin_budget;
};

constexpr int kMoeMaxExperts = 2048;     // of one launch (the lists of tiles lie in shared memory)
constexpr int kMoeK = 256;               // K of a weight stage: a 128-byte line of codes and 16 scales per weight row
constexpr int kMoeSlots = 8;             // operand slots in tensor memory: 32 columns (64 K) of a weight tile each
constexpr int kMoeThreads = 768;         // activations, products, weights, (idle), 4 epilogue warps, 4 x 4 dequant warps

// kTiles: weight tiles (128 TMEM lanes each) of a unit
template <int BT, int kTiles_>
struct MoeGCfg {
  static constexpr int kTiles = kTiles_;
  static constexpr int kBoxRows = BT < 32 ? BT : 32;                    // token rows of one activation copy
  static constexpr int kCodeBytes = 128 * 128, kScaleBytes = 128 * 16;  // of a weight tile in a stage
  static constexpr int kSteps = kMoeSlots / kTiles;                     // K steps of 64 whose operands are ready or being written
  static constexpr int kXBytes = BT * 128, kXStages = BT == 128 ? 6 : 8;
  static constexpr int kWStages = kTiles == 2 ? (BT == 128 ? 3 : BT == 16 ? 5 : 4) : (BT == 128 ? 6 : 8);
  static constexpr int kRingBytes = kWStages * kTiles * (kCodeBytes + kScaleBytes) + kXStages * kXBytes;
  static constexpr int kAccCols = kTiles * BT;
  static constexpr int kAccBufs = 2 * kAccCols + kMoeSlots * 32 <= 512 ? 2 : 1;
  static_assert(kAccBufs * kAccCols + kMoeSlots * 32 <= 512, "tensor memory");
};

struct alignas(8) MoeGBars {
  uint64_t w_full[8], w_empty[8];
  uint64_t x_full[8], x_empty[8];
  uint64_t s_full[kMoeSlots], s_empty[kMoeSlots];     // a step's converted weights
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  int n_experts;                  // that have rows
};

__device__ __forceinline__ void moe_tmem_st_32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
      "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void moe_tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 e2m1 codes (16 bytes) and their two scales -> 16 words of fp16 pairs
__device__ __forceinline__ void moe_dequant(const uint4& codes, __half2 sc, uint32_t* out) {
  const uint32_t words[4] = {codes.x, codes.y, codes.z, codes.w};
  const __half2 sc2[2] = {__low2half2(sc), __high2half2(sc)};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    __half2 h[4];
    e2m1x8_to_half(words[i], h);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const __half2 v = __hmul2(h[b], sc2[i >> 1]);
      out[4 * i + b] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
}

// D[tmem] (+)= A[tmem] * B[smem], in code that one lane runs.  With the operands in tensor memory a product takes N / 2 + 10 cycles this
// way; issued by a converged warp under a lane predicate (mma_ts) it takes 82 to 90 however few columns it has.
__device__ __forceinline__ void moe_mma(uint32_t d, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
      ::"r"(d), "r"(a_tmem), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(acc)
      : "memory");
}

// Whether the phase has completed, without waiting for it
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}

// Row of a stage that TMEM lane 32 q4 + lane holds.  FC1: sixteen gate rows (rows 0..63 of the stage) and the up rows of the same
// features (64..127) side by side in a warp, so that one shuffle brings a feature's two products together.
template <bool kFc1>
__device__ __forceinline__ int moe_lane_row(int q4, int lane) {
  return kFc1 ? (lane >> 4) * 64 + q4 * 16 + (lane & 15) : q4 * 32 + lane;
}

template <int BT, bool kFc1, int kTiles>
__global__ void __launch_bounds__(kMoeThreads, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const MoeGArgs a) {
  using Cfg = MoeGCfg<BT, kTiles>;
  constexpr int kWStages = Cfg::kWStages, kXStages = Cfg::kXStages, kSteps = Cfg::kSteps, kAccBufs = Cfg::kAccBufs;
  constexpr int kWCodes = kTiles * Cfg::kCodeBytes, kWScales = kTiles * Cfg::kScaleBytes;      // of a weight stage
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_w = smem;                                        // kWStages x kTiles x 16 KB of codes
  uint8_t* smem_x = smem_w + kWStages * kWCodes;                 // kXStages x BT x 128 B
  uint8_t* smem_s = smem_x + kXStages * Cfg::kXBytes;            // kWStages x kTiles x 2 KB of scales
  MoeGBars* bars = reinterpret_cast<MoeGBars*>(smem_s + kWStages * kWScales);
  int* first_tile = reinterpret_cast<int*>(bars + 1);            // [experts with rows + 1] token tiles of those before
  int* expert_of = first_tile + a.e_local + 1;                   // [experts with rows]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kWStages; ++s) {
      mbar_init(&bars->w_full[s], 1 + 32);        // TMA arrive (+tx bytes) and the lanes that copy scales
      mbar_init(&bars->w_empty[s], 16);           // dequant warps
    }
    for (int s = 0; s < kXStages; ++s) {
      mbar_init(&bars->x_full[s], 1);
      mbar_init(&bars->x_empty[s], 1);
    }
    for (int s = 0; s < kSteps; ++s) {
      mbar_init(&bars->s_full[s], 4 * kTiles);    // the four warps of each tile's dequant group
      mbar_init(&bars->s_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], 4);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmX);
      tma_prefetch_desc(&tmW);
    }
    // experts that have rows, and the token tiles in front of each
    int n = 0, tiles = 0;
    for (int e0 = 0; e0 < a.e_local; e0 += 32) {
      const int e = e0 + lane;
      const int cnt = e < a.e_local ? a.offsets[e + 1] - a.offsets[e] : 0;
      const int mine = cnt > 0 ? (cnt + BT - 1) / BT : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const int up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
      }
      const uint32_t some = __ballot_sync(0xffffffffu, mine > 0);
      if (mine > 0) {
        const int i = n + __popc(some & ((1u << lane) - 1u));
        expert_of[i] = e;
        first_tile[i] = tiles + sum - mine;
      }
      n += __popc(some);
      tiles += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) {
      first_tile[n] = tiles;
      bars->n_experts = n;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  const uint32_t tmem_slots = tmem_base + kAccBufs * Cfg::kAccCols;

  const int tiles_n = a.rows / (128 * kTiles);
  const int n_experts = bars->n_experts;
  const int units = first_tile[n_experts] * tiles_n;
  const int stages_k = (a.K + kMoeK - 1) / kMoeK;               // weight stages of a tile
  const int steps_k = a.K / 64;                                 // K steps of a unit
  // Buffers of K step kb of this CTA's i-th unit, and their phase.  Four of them: those of the step's place in a weight stage (a dequant
  // group then sees every use of its buffers, which a wait by parity needs, also where a unit's last stage is not whole).  Eight: in turn.
  // There a group does not see every use, but its own steps are at most seven apart (seven steps a unit: 3, 10), so its last wait, for the
  // products of a step at most fifteen back, tells it that those of sixteen back are done, and parity can only mean those of eight back.
  struct Step { int buf; uint32_t phase; };
  auto step_at = [&](int i, int kb) {
    if constexpr (kSteps == 4) {
      const int q = kb & 3, use = i * ((steps_k + 3 - q) >> 2) + (kb >> 2);
      return Step{q, static_cast<uint32_t>(use) & 1u};
    } else {
      const int n = i * steps_k + kb;
      return Step{n & (kSteps - 1), static_cast<uint32_t>(n / kSteps) & 1u};
    }
  };

  struct Unit { int e, tn, r0, rows; };             // expert, weight tile, first row and rows of the token tile
  auto unit_at = [&](int u) {
    Unit x;
    const int j = u / tiles_n;
    x.tn = u - j * tiles_n;
    int lo = 0, hi = n_experts - 1;                 // last expert whose first tile is not behind j
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first_tile[mid] <= j) lo = mid;
      else hi = mid - 1;
    }
    x.e = expert_of[lo];
    const int tt = j - first_tile[lo];
    x.r0 = a.offsets[x.e] + tt * BT;
    x.rows = min(BT, a.offsets[x.e + 1] - x.r0);
    return x;
  };

  if (warp == 0) {
    // ------------------------------ TMA producer (activations) ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const Unit x = unit_at(u);
        if (a.arrived != nullptr) {
          // rows of this expert come over NVLink: start as soon as they are all here (bounded wait)
          const uint32_t want = static_cast<uint32_t>(a.offsets[x.e + 1] - a.offsets[x.e]);
          bool here = false;
          for (uint32_t i = 0; i < a.spin_budget; ++i) {
            uint32_t got;
            asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(got) : "l"(a.arrived + x.e) : "memory");
            if (got >= want) { here = true; break; }
            if (i > 64) __nanosleep(64);
          }
          if (!here) { set_status(a.status, kTimeoutPeerFlag, 760); ok = false; break; }
          asm volatile("fence.proxy.async.global;" ::: "memory");      // peer stores (generic proxy) -> TMA reads
        }
        const int boxes = (x.rows + Cfg::kBoxRows - 1) / Cfg::kBoxRows;      // only what has rows
        for (int kb = 0; kb < steps_k; ++kb) {
          if (!mbar_wait(&bars->x_empty[stage], phase ^ 1, a.status, 700 + stage)) { ok = false; break; }
          mbar_expect_tx(&bars->x_full[stage], boxes * Cfg::kBoxRows * 128);
          for (int j = 0; j < boxes; ++j)
            tma_load_2d(smem_x + stage * Cfg::kXBytes + j * Cfg::kBoxRows * 128, &tmX, &bars->x_full[stage], kb * 64, x.r0 + j * Cfg::kBoxRows);
          if (++stage == kXStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t slots = tm + kAccBufs * Cfg::kAccCols, x_lo = desc_lo(smem_u32(smem_x));
    int ab = 0, n = 0, stage = 0;
    uint32_t aphase = 0, xphase = 0, phases = 0;               // kSteps == 4: phase of each buffer; else buffers are taken in turn, n counts steps
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const Unit x = unit_at(u);
      const uint32_t idesc = umma_idesc(0u, 0u, 128, 0) | static_cast<uint32_t>(((x.rows + 15) >> 4) << 1) << 17;   // fp16 x fp16 -> fp32
      ok = mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 705 + ab);
      if (!ok) break;
      tc_fence_after();
      const uint32_t acc = tm + ab * Cfg::kAccCols;
      bool ready = false;                          // the next step's barriers were seen complete while this step's products were issued
      for (int kb0 = 0; kb0 < steps_k && ok; kb0 += 4) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (kb0 + q >= steps_k) break;
          const int buf = kSteps == 4 ? q : n & (kSteps - 1);
          const uint32_t phase = kSteps == 4 ? (phases >> q) & 1u : static_cast<uint32_t>(n / kSteps) & 1u;
          if (!__all_sync(0xffffffffu, ready)) {
            ok = mbar_wait(&bars->x_full[stage], xphase, a.status, 710 + stage) && mbar_wait(&bars->s_full[buf], phase, a.status, 720 + buf);
            if (!ok) break;
          }
          const uint32_t bl = x_lo + stage * (Cfg::kXBytes >> 4), al = slots + buf * (kTiles * 32);
          uint64_t* const x_done = &bars->x_empty[stage];
          if (++stage == kXStages) { stage = 0; xphase ^= 1; }
          ++n;
          phases ^= 1u << q;
          const int after = kSteps == 4 ? (q + 1) & 3 : n & (kSteps - 1);
          ready = mbar_test(&bars->s_full[after], kSteps == 4 ? (phases >> after) & 1u : static_cast<uint32_t>(n / kSteps) & 1u);
          ready = mbar_test(&bars->x_full[stage], xphase) && ready && kb0 + q + 1 < steps_k;
          tc_fence_after();
          if (lead) {
#pragma unroll
            for (int t = 0; t < kTiles; ++t)
#pragma unroll
              for (int k = 0; k < 4; ++k) moe_mma(acc + t * BT, al + t * 32 + k * 8, bl + 2 * k, idesc, (q > 0 || k > 0) ? 1u : (kb0 > 0 ? 1u : 0u));
            umma_commit(&bars->s_empty[buf]);
            umma_commit(x_done);
          }
          __syncwarp();
        }
      }
      if (ok) {
        if (lead) umma_commit(&bars->tmem_full[ab]);
        __syncwarp();
        if (++ab == kAccBufs) { ab = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------ weight producer (codes by TMA, scales by asynchronous copies) ------------------------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const long long sstride = a.K / 16;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const Unit x = unit_at(u);
      for (int sb = 0; sb < stages_k; ++sb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->w_empty[stage], phase ^ 1, a.status, 740 + stage));
        if (!ok) break;
        const int steps = min(4, steps_k - 4 * sb);
        if (lane == 0) mbar_expect_tx(&bars->w_full[stage], kWCodes);
#pragma unroll
        for (int t = 0; t < kTiles; ++t) {
          const int tile = x.tn * kTiles + t;
          const int row0 = x.e * a.rows + tile * (kFc1 ? 64 : 128), row1 = row0 + (kFc1 ? a.rows / 2 : 64);
          if (lane == 0) {
            uint8_t* to = smem_w + stage * kWCodes + t * Cfg::kCodeBytes;
            tma_load_2d(to, &tmW, &bars->w_full[stage], sb * (kMoeK / 2), row0);
            tma_load_2d(to + 64 * 128, &tmW, &bars->w_full[stage], sb * (kMoeK / 2), row1);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int r = i * 32 + lane;
            const uint8_t* src = a.s + ((r < 64 ? row0 + r : row1 + r - 64)) * sstride + sb * 16;
            uint8_t* dst = smem_s + stage * kWScales + t * Cfg::kScaleBytes + r * 16;
            if (a.scale_copy == 16) {
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
            } else if (a.scale_copy == 4) {
              for (int j = 0; j < steps; ++j)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + 4 * j)), "l"(src + 4 * j) : "memory");
            } else {
              for (int j = 0; j < 4 * steps; ++j) dst[j] = src[j];
            }
          }
        }
        if (a.scale_copy != 1)
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bars->w_full[stage])) : "memory");
        else
          mbar_arrive(&bars->w_full[stage]);
        if (++stage == kWStages) { stage = 0; phase ^= 1; }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= 4 && warp < 8) {
    // ------------------------------ epilogue ------------------------------
    const int q4 = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(q4 * 32) << 16;
    int ab = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const Unit x = unit_at(u);
      const float gs = a.gscale[x.e];
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[ab], aphase, a.status, 730 + ab));
      if (!ok) break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < x.rows; c0 += 16) {
#pragma unroll
        for (int t = 0; t < kTiles; ++t) {
          uint32_t r[16];
          tmem_ld_32x16(tmem_base + ab * Cfg::kAccCols + t * BT + c0 + lane_addr, r);
          tmem_ld_wait();
          const int tile = x.tn * kTiles + t;
          if constexpr (kFc1) {
            // gate products in lanes 0..15, up products of the same features in lanes 16..31: the lower lanes finish columns
            // 0..7, the upper ones 8..15
            const bool upper = lane >= 16;
            const int c = c0 + (upper ? 8 : 0);
            __half* o = reinterpret_cast<__half*>(a.out) + static_cast<long long>(x.r0 + c) * a.n_out + tile * 64 + q4 * 16 + (lane & 15);
            __half v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? r[j] : r[j + 8], 16);
              float g = __uint_as_float(upper ? got : r[j]) * gs, up = __uint_as_float(upper ? r[j + 8] : got) * gs;
              if (a.limit > 0.f) {
                g = fminf(g, a.limit);
                up = fminf(fmaxf(up, -a.limit), a.limit);
              }
              // the quotient of the reciprocal's unit, 2 ulp of fp32 under a rounding to fp16:
              // against 64 bits the same error as a rounded division, which took 130 us of 2084 (4096 tokens, 256 experts)
              v[j] = __float2half(__fdividef(g, 1.f + __expf(-g)) * up);
            }
            if (c0 + 16 <= x.rows) {
#pragma unroll
              for (int j = 0; j < 8; ++j) o[j * a.n_out] = v[j];
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (c + j < x.rows) o[j * a.n_out] = v[j];
            }
          } else {
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + static_cast<long long>(x.r0 + c0) * a.n_out + tile * 128 + q4 * 32 + lane;
            __nv_bfloat16 v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __float2bfloat16(__uint_as_float(r[j]) * gs);
            if (c0 + 16 <= x.rows) {
#pragma unroll
              for (int j = 0; j < 16; ++j) o[j * a.n_out] = v[j];
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (c0 + j < x.rows) o[j * a.n_out] = v[j];
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->tmem_empty[ab]);
      if (++ab == kAccBufs) { ab = 0; aphase ^= 1; }
    }
  } else if (warp >= 8) {
    // ------------------------------ dequant (weights) ------------------------------
    // A tile has 4 / kTiles groups of four warps, which take its K steps in turn; a thread has one weight row.  Operands are converted
    // before their place in tensor memory is waited for.
    constexpr int kTurns = 4 / kTiles;
    const int group = (warp - 8) >> 2, t = group % kTiles, turn = group / kTiles, q4 = warp & 3;
    const uint32_t to = tmem_slots + t * 32 + (static_cast<uint32_t>(q4 * 32) << 16);
    const int row = moe_lane_row<kFc1>(q4, lane);
    const uint32_t code_at = t * Cfg::kCodeBytes + row * 128, scale_at = t * Cfg::kScaleBytes + row * 16, swap = (row & 7) << 4;
    int stage = 0, i = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x, ++i) {
      for (int sb = 0; sb < stages_k && ok; ++sb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->w_full[stage], phase, a.status, 770 + stage));
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < kTiles; ++j) {
          const int q = j * kTurns + turn;
          const bool mine = 4 * sb + q < steps_k;
          uint32_t o[32];
          if (mine) {
            const uint8_t* codes = smem_w + stage * kWCodes + code_at;
            const uint4 c0 = *reinterpret_cast<const uint4*>(codes + ((2 * q) << 4 ^ swap)), c1 = *reinterpret_cast<const uint4*>(codes + ((2 * q + 1) << 4 ^ swap));
            const uint32_t sc = *reinterpret_cast<const uint32_t*>(smem_s + stage * kWScales + scale_at + q * 4);
            __half2 s0, s1;
            e4m3x4_to_half(sc, s0, s1);
            moe_dequant(c0, s0, o);
            moe_dequant(c1, s1, o + 16);
          }
          if (j == kTiles - 1) {                                 // the last of this warp's parts of the stage
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->w_empty[stage]);
          }
          if (mine) {
            const Step st = step_at(i, 4 * sb + q);
            ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_empty[st.buf], st.phase ^ 1, a.status, 780 + st.buf));
            if (!ok) break;
            tc_fence_after();
            moe_tmem_st_32(to + st.buf * (kTiles * 32), o);
            moe_tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->s_full[st.buf]);
          }
        }
        if (++stage == kWStages) { stage = 0; phase ^= 1; }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// sorted row q <- activations of token sorted[q] / topk, converted to fp16.
__global__ void moe_permute_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const int* __restrict__ sorted,
                                   const int* __restrict__ offsets, int e_local, int topk, __half* __restrict__ xs, int H) {
  const int q = blockIdx.x;
  if (q >= offsets[e_local]) return;
  const int t = sorted[q] / topk;
  const uint4* src = reinterpret_cast<const uint4*>(x + t * ldx);
  uint4* dst = reinterpret_cast<uint4*>(xs + static_cast<long long>(q) * H);
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    const uint4 v = __ldg(src + i);
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
    const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int j = 0; j < 4; ++j) oh[j] = __float22half2_rn(__bfloat1622float2(b[j]));
    dst[i] = o;
  }
}

template <int BT, bool kFc1, int kTiles>
static int launch_moe_grouped(const CUtensorMap& tx, const CUtensorMap& tw, const MoeGArgs& a, int grid, cudaStream_t st) {
  using Cfg = MoeGCfg<BT, kTiles>;
  constexpr int kFixed = Cfg::kRingBytes + static_cast<int>(sizeof(MoeGBars)) + 1024;
  constexpr int kMost = kFixed + (2 * kMoeMaxExperts + 1) * 4;
  static_assert(kMost <= 227 * 1024, "shared memory");
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(moe_grouped_kernel<BT, kFc1, kTiles>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost) != cudaSuccess)
      return -3;
    configured = true;
  }
  moe_grouped_kernel<BT, kFc1, kTiles><<<grid, kMoeThreads, kFixed + (2 * a.e_local + 1) * 4, st>>>(tx, tw, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace stk

using namespace stk;

STK_API int stk_moe_permute(const void* x, long long ldx, const int* sorted, const int* offsets, int e_local, int topk,
                            void* xs, int max_rows, int H, void* stream) {
  if (max_rows <= 0) return 0;
  if (H % 8 || (ldx % 8)) return -1;
  moe_permute_kernel<<<max_rows, 128, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)x, ldx, sorted, offsets, e_local, topk,
                                                               (__half*)xs, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// xs: fp16 [xs_rows, K] sorted activations (xs_rows >= total rows + bt, tail readable).
// fc1 = 1: w rows = 2*n_out (gate rows then up rows), out fp16 [P, n_out] = swiglu;  fc1 = 0: w rows = n_out, out bf16.
static int moe_grouped_launch(const void* xs, long long xs_rows, const void* w, const void* s, const float* gscale,
                              const int* offsets, int e_local, int n_out, int K, void* out, int fc1, float limit, int bt,
                              int* status, int sm_count, const uint32_t* arrived, uint32_t spin_budget, void* stream) {
  if (e_local <= 0) return 0;
  if (K % 64 || n_out % 128 || (bt != 16 && bt != 32 && bt != 64 && bt != 128)) return -1;
  CUtensorMap tx;
  if (make_tmap_2d(&tx, xs, 2, xs_rows, K, K, bt < 32 ? bt : 32) != 0) return -2;
  MoeGArgs a;
  a.rows = fc1 ? 2 * n_out : n_out; a.n_out = n_out; a.K = K; a.out = out; a.limit = limit; a.status = status;
  a.spin_budget = spin_budget;
  const bool two = fc1 || n_out % 256 == 0;
  cudaStream_t st = (cudaStream_t)stream;
  for (int e0 = 0; e0 < e_local; e0 += kMoeMaxExperts) {
    a.e_local = e_local - e0 < kMoeMaxExperts ? e_local - e0 : kMoeMaxExperts;
    a.w = (const uint8_t*)w + static_cast<long long>(e0) * a.rows * (K / 2);
    a.s = (const uint8_t*)s + static_cast<long long>(e0) * a.rows * (K / 16);
    a.scale_copy = K % 256 == 0 && (reinterpret_cast<uintptr_t>(a.s) & 15) == 0 ? 16 : (reinterpret_cast<uintptr_t>(a.s) & 3) == 0 ? 4 : 1;
    CUtensorMap tw;
    if (make_tmap_2d(&tw, a.w, 1, static_cast<long long>(a.e_local) * a.rows, K / 2, K / 2, 64) != 0) return -2;
    a.gscale = gscale + e0;
    a.offsets = offsets + e0;
    a.arrived = arrived != nullptr ? arrived + e0 : nullptr;
    int rc;
#define STK_MG(BT_) (fc1 ? launch_moe_grouped<BT_, true, 2>(tx, tw, a, sm_count, st) \
                         : two ? launch_moe_grouped<BT_, false, 2>(tx, tw, a, sm_count, st) : launch_moe_grouped<BT_, false, 1>(tx, tw, a, sm_count, st))
    switch (bt) {
      case 16: rc = STK_MG(16); break;
      case 32: rc = STK_MG(32); break;
      case 64: rc = STK_MG(64); break;
      default: rc = STK_MG(128); break;
    }
#undef STK_MG
    if (rc != 0) return rc;
  }
  return 0;
}

STK_API int stk_moe_grouped(const void* xs, long long xs_rows, const void* w, const void* s, const float* gscale,
                            const int* offsets, int e_local, int n_out, int K, void* out, int fc1, float limit, int bt,
                            int* status, int sm_count, void* stream) {
  return moe_grouped_launch(xs, xs_rows, w, s, gscale, offsets, e_local, n_out, K, out, fc1, limit, bt, status, sm_count,
                            nullptr, 0u, stream);
}

// Expert-parallel FC1: the activation rows of local expert e are complete once arrived[e] reaches the expert's row
// count; the producer warp waits for that per expert, so tiles of early experts run while later rows are in flight.
STK_API int stk_moe_grouped_ep(const void* xs, long long xs_rows, const void* w, const void* s, const float* gscale,
                               const int* offsets, int e_local, int n_out, int K, void* out, int fc1, float limit, int bt,
                               int* status, int sm_count, const void* arrived, int spin_budget, void* stream) {
  return moe_grouped_launch(xs, xs_rows, w, s, gscale, offsets, e_local, n_out, K, out, fc1, limit, bt, status, sm_count,
                            (const uint32_t*)arrived, static_cast<uint32_t>(spin_budget), stream);
}
