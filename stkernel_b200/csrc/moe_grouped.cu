// Grouped expert GEMM on the 5th-generation tensor cores, NVFP4 weights x fp16 activations (W4A16).
//
// Tokens arrive sorted by expert (`offsets[e]` .. `offsets[e+1]` are the rows of local expert e in the
// permuted activation matrix).  A persistent grid walks the (token tile of an expert, weight tile) pairs
// that have rows, dealt out in turn, so that every CTA has the same number of them whichever experts were chosen:
//
//   TMA warp         activation tile [BT tokens x 64 k] fp16, 128-byte swizzle
//   dequant warps    e2m1 codes and e4m3 group scales -> fp16 written straight into the swizzled K-major
//                    operand tile
//   MMA warp         tcgen05.mma kind::f16 into TMEM (double-buffered accumulators), as many token columns as
//                    the tile has rows (in sixteens)
//   epilogue warps   FC1: gate and up tiles sit side by side in TMEM, so one thread holds both values
//                    of an output and applies SwiGLU with clamp before storing fp16;
//                    FC2: scaled bf16 store.  Rows past the expert's last token are masked.
//
// e2m1 x e4m3 is exact in fp16, the per-matrix fp32 scale is applied in the epilogue.
//
// What bounds it: a K block of 256 weight rows is 16384 codes to convert and 9.2 KB to fetch, for eight products of 40 to 65
// tensor-core cycles.  Four groups of four dequant warps (one per scheduler) convert every fourth K block each, so the waits,
// fences and load latency of a block are paid once per 128 codes of a thread and hidden by the other three groups; with all
// sixteen warps on the same block (32 codes each) the same conversions took 2500 cycles per block at 128 tokens and 1040 at 16.
// Codes are fetched two own blocks ahead, past the ends of tiles.
// Measured (hidden 4096, 2048 rows an expert, top 6; device time of the first + the second product, us):
//   64 tokens, 256 experts    849 + 529 with all warps on one block, 632 + 302 now
//   4096 tokens, 256 experts  2772 + 1512, 2399 + 1233
//   4096 tokens, 64 experts   1901 + 1033, 1005 + 540
//
// This is the engine's counterpart of the reference's fused W4A16 MoE kernel and, for the
// expert-parallel layout, of its mega-MoE grouped GEMM (overlay/nvidia_model.py:227-559).
#include <cuda_fp4.h>

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
  int* status;
  // Expert-parallel mode: rows of expert e are pushed into the activation matrix by peers (and by this
  // GPU's own dispatch); `arrived[e]` counts the rows that have landed.  nullptr = rows are already there.
  const uint32_t* arrived;
  uint32_t spin_budget;
};

constexpr int kMoeMaxExperts = 2048;     // of one launch (the lists of tiles lie in shared memory)
constexpr int kMoeGroups = 4;            // dequant warps: groups x 4

// kATiles: 128-row weight tiles of a unit (FC1: gate and up; FC2: two neighbours where the rows allow it)
template <int BT, int kATiles_>
struct MoeGCfg {
  static constexpr int kATiles = kATiles_;
  static constexpr int kStageBytes = kATiles * 128 * 128 + BT * 128;
  static constexpr int kStagesRaw = (196 * 1024) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 6 ? 6 : kStagesRaw;
  // A dequant group waits for a free stage by parity, which cannot tell "free" from "two rounds behind".  At block i it knows that
  // block i - kMoeGroups - kStages was multiplied (its last wait); the stage is at most one round behind if that is not before
  // block i - 2 kStages.
  static_assert(kStages >= kMoeGroups, "stages of the ring");
  static constexpr int kAccCols = kATiles * BT;
  static constexpr int kTmemCols = (2 * kAccCols <= 32) ? 32 : (2 * kAccCols <= 64) ? 64 : (2 * kAccCols <= 128) ? 128
                                   : (2 * kAccCols <= 256) ? 256 : 512;
};

struct alignas(8) MoeGBars {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int n_experts;                  // that have rows
};

// Half of a weight row's K block: 32 e2m1 codes (16 bytes) and their two e4m3 group scales.
struct RawRow {
  uint4 w;
  uint32_t sc;
};

__device__ __forceinline__ void load_raw(RawRow& r, const uint8_t* w, const uint8_t* s) {
  // codes pass by the first-level cache, which is left to the scales (a sector of them serves eight K blocks)
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r.w.x), "=r"(r.w.y), "=r"(r.w.z), "=r"(r.w.w) : "l"(w));
  r.sc = __ldg(reinterpret_cast<const uint16_t*>(s));
}

// 32 values of one weight row -> 64 bytes of fp16, chunk i (eight values) at line + at[i].
__device__ __forceinline__ void dequant_store(const RawRow& r, uint8_t* line, const uint32_t (&at)[4]) {
  const uint32_t words[4] = {r.w.x, r.w.y, r.w.z, r.w.w};
  const __half2_raw sraw = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(r.sc), __NV_E4M3);
  const __half2 sc = *reinterpret_cast<const __half2*>(&sraw);
  const __half2 sc2[2] = {__low2half2(sc), __high2half2(sc)};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 o;
    __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const __half2_raw hr = __nv_cvt_fp4x2_to_halfraw2(static_cast<__nv_fp4x2_storage_t>((words[i] >> (8 * b)) & 0xff), __NV_E2M1);
      oh[b] = __hmul2(*reinterpret_cast<const __half2*>(&hr), sc2[i >> 1]);
    }
    *reinterpret_cast<uint4*>(line + at[i]) = o;
  }
}

template <int BT, bool kFc1, int kATiles>
__global__ void __launch_bounds__(704, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap tmX, const MoeGArgs a) {
  using Cfg = MoeGCfg<BT, kATiles>;
  constexpr int kStages = Cfg::kStages;
  constexpr int CW = (BT >= 32 && kATiles == 1) ? 32 : 16;     // columns of an epilogue step
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;                                        // kStages x kATiles x 16 KB
  uint8_t* smem_b = smem + kStages * kATiles * 128 * 128;        // kStages x BT*128
  MoeGBars* bars = reinterpret_cast<MoeGBars*>(smem_b + kStages * BT * 128);
  int* first_tile = reinterpret_cast<int*>(bars + 1);            // [experts with rows + 1] token tiles of those before
  int* expert_of = first_tile + a.e_local + 1;                   // [experts with rows]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1 + 4);           // TMA arrive (+tx bytes) and the four warps of a dequant group
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], 4);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, Cfg::kTmemCols);
    tmem_relinquish();
  }
  if (warp == 0) {
    if (lane == 0) tma_prefetch_desc(&tmX);
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

  const int tiles_n = a.rows / (128 * kATiles);     // FC1: tiles over I; FC2: tiles over H
  const int n_experts = bars->n_experts;
  const int units = first_tile[n_experts] * tiles_n;
  const int k_blocks = a.K / 64;

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
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 700 + stage)) { ok = false; break; }
          mbar_expect_tx(&bars->full[stage], BT * 128);
          tma_load_2d(smem_b + stage * BT * 128, &tmX, &bars->full[stage], kb * 64, x.r0);
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t a_lo = desc_lo(smem_u32(smem_a)), b_lo = desc_lo(smem_u32(smem_b));
    int stage = 0;
    uint32_t phase = 0;
    int ab = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const Unit x = unit_at(u);
      const uint32_t idesc = umma_idesc(0u, 0u, 128, 0) | static_cast<uint32_t>(((x.rows + 15) >> 4) << 1) << 17;   // fp16 x fp16 -> fp32
      ok = mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 710 + ab);
      if (!ok) break;
      tc_fence_after();
      for (int kb = 0; kb < k_blocks; ++kb) {
        ok = mbar_wait(&bars->full[stage], phase, a.status, 720 + stage);
        if (!ok) break;
        tc_fence_after();
        const uint32_t bl = b_lo + stage * (BT * 8), al = a_lo + stage * (kATiles * 1024);
#pragma unroll
        for (int at = 0; at < kATiles; ++at)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_ss(tm + ab * Cfg::kAccCols + at * BT, al + at * 1024 + 2 * k, bl + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u, lead);
        mma_commit(&bars->empty[stage], lead);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
      if (ok) {
        mma_commit(&bars->tmem_full[ab], lead);
        if (++ab == 2) { ab = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp < 6) {
    // ------------------------------ epilogue ------------------------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    int ab = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const Unit x = unit_at(u);
      const float gs = a.gscale[x.e];
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[ab], aphase, a.status, 730 + ab));
      if (!ok) break;
      tc_fence_after();
      const int n = x.tn * (kFc1 ? 128 : 128 * kATiles) + row;      // (first) output feature of this thread
#pragma unroll 1
      for (int c0 = 0; c0 < x.rows; c0 += CW) {
        uint32_t r[kATiles][32];
#pragma unroll
        for (int at = 0; at < kATiles; ++at) {
          const uint32_t base = tmem_base + ab * Cfg::kAccCols + at * BT + c0 + lane_addr;
          if constexpr (CW == 32) {
            tmem_ld_32x32(base, r[at]);
          } else {
            uint32_t t16[16];
            tmem_ld_32x16(base, t16);
#pragma unroll
            for (int i = 0; i < 16; ++i) r[at][i] = t16[i];
          }
        }
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          if (c0 + j < x.rows) {
            const long long o = static_cast<long long>(x.r0 + c0 + j) * a.n_out + n;
            if constexpr (kFc1) {
              float g = __uint_as_float(r[0][j]) * gs, up = __uint_as_float(r[1][j]) * gs;
              if (a.limit > 0.f) {
                g = fminf(g, a.limit);
                up = fminf(fmaxf(up, -a.limit), a.limit);
              }
              reinterpret_cast<__half*>(a.out)[o] = __float2half(g / (1.f + __expf(-g)) * up);
            } else {
#pragma unroll
              for (int at = 0; at < kATiles; ++at)
                reinterpret_cast<__nv_bfloat16*>(a.out)[o + at * 128] = __float2bfloat16(__uint_as_float(r[at][j]) * gs);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->tmem_empty[ab]);
      if (++ab == 2) { ab = 0; aphase ^= 1; }
    }
  } else {
    // ------------------------------ dequant producers (weights) ------------------------------
    // Group g converts every fourth K block of the CTA's sequence of units.  A lane pair shares a weight row (32 codes each);
    // a thread has the same half of 2 kATiles rows, 64 apart.
    constexpr int kMine = 2 * kATiles;
    const int group = (warp - 6) >> 2, gt = ((warp - 6) & 3) * 32 + lane;
    const int half = gt & 1, r16 = gt >> 1;
    uint32_t at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) at[i] = static_cast<uint32_t>(r16 * 128 + (((half * 4 + i) ^ (r16 & 7)) << 4));
    const long long wstride = a.K / 2, sstride = a.K / 16;
    const long long second = (kFc1 ? a.rows / 2 : 128);             // rows between the first and the second tile
    struct Cursor {
      int u, kb;
      const uint8_t* w;
      const uint8_t* s;
    } ld{static_cast<int>(blockIdx.x), group, nullptr, nullptr};
    auto enter = [&]() {                                             // pointers of the cursor's unit
      if (ld.u >= units) return;
      const Unit x = unit_at(ld.u);
      const long long row = static_cast<long long>(x.e) * a.rows + x.tn * (kFc1 ? 128 : 128 * kATiles) + r16;
      ld.w = a.w + row * wstride + half * 16;
      ld.s = a.s + row * sstride + half * 2;
    };
    auto settle = [&]() {                                            // the K block may lie in a later unit
      while (ld.kb >= k_blocks && ld.u < units) {
        ld.kb -= k_blocks;
        ld.u += gridDim.x;
        if (ld.kb < k_blocks) enter();
      }
    };
    RawRow raw[2][kMine];
    auto load = [&](RawRow (&r)[kMine]) {                            // the cursor's block, then on by a group's stride
      if (ld.u < units) {
#pragma unroll
        for (int j = 0; j < kMine; ++j) {
          const long long rows = (j & 1) * 64 + (j >> 1) * second;
          load_raw(r[j], ld.w + rows * wstride + ld.kb * 32, ld.s + rows * sstride + ld.kb * 4);
        }
        ld.kb += kMoeGroups;
        settle();
      }
    };
    enter();
    settle();
    load(raw[0]);
    load(raw[1]);
    // blocks of this CTA's whole sequence: units, each k_blocks long
    const long long mine = static_cast<int>(blockIdx.x) < units ? (units - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;
    const long long total = mine * k_blocks;
    int stage = group % kStages;
    uint32_t phase = static_cast<uint32_t>(group / kStages) & 1u;
    bool ok = true;
    auto step = [&](RawRow (&r)[kMine]) {
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 740 + stage));
      if (!ok) return;
#pragma unroll
      for (int j = 0; j < kMine; ++j)
        dequant_store(r[j], smem_a + (stage * kATiles + (j >> 1)) * 128 * 128 + (j & 1) * 64 * 128, at);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->full[stage]);
      load(r);
      stage += kMoeGroups;
      while (stage >= kStages) { stage -= kStages; phase ^= 1; }
    };
    for (long long i = group; i < total && ok; i += 2 * kMoeGroups) {
      step(raw[0]);
      if (ok && i + kMoeGroups < total) step(raw[1]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
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

template <int BT, bool kFc1, int kATiles>
static int launch_moe_grouped(const CUtensorMap& tx, const MoeGArgs& a, int grid, cudaStream_t st) {
  using Cfg = MoeGCfg<BT, kATiles>;
  constexpr int kFixed = Cfg::kStages * Cfg::kStageBytes + static_cast<int>(sizeof(MoeGBars)) + 1024;
  constexpr int kMost = kFixed + (2 * kMoeMaxExperts + 1) * 4;
  static_assert(kMost <= 227 * 1024, "shared memory");
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(moe_grouped_kernel<BT, kFc1, kATiles>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost) != cudaSuccess)
      return -3;
    configured = true;
  }
  moe_grouped_kernel<BT, kFc1, kATiles><<<grid, 704, kFixed + (2 * a.e_local + 1) * 4, st>>>(tx, a);
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
  if (make_tmap_2d(&tx, xs, 2, xs_rows, K, K, bt) != 0) return -2;
  MoeGArgs a;
  a.rows = fc1 ? 2 * n_out : n_out; a.n_out = n_out; a.K = K; a.out = out; a.limit = limit; a.status = status;
  a.spin_budget = spin_budget;
  const bool two = fc1 || n_out % 256 == 0;
  cudaStream_t st = (cudaStream_t)stream;
  for (int e0 = 0; e0 < e_local; e0 += kMoeMaxExperts) {
    a.e_local = e_local - e0 < kMoeMaxExperts ? e_local - e0 : kMoeMaxExperts;
    a.w = (const uint8_t*)w + static_cast<long long>(e0) * a.rows * (K / 2);
    a.s = (const uint8_t*)s + static_cast<long long>(e0) * a.rows * (K / 16);
    a.gscale = gscale + e0;
    a.offsets = offsets + e0;
    a.arrived = arrived != nullptr ? arrived + e0 : nullptr;
    int rc;
#define STK_MG(BT_) (fc1 ? launch_moe_grouped<BT_, true, 2>(tx, a, sm_count, st) \
                         : two ? launch_moe_grouped<BT_, false, 2>(tx, a, sm_count, st) : launch_moe_grouped<BT_, false, 1>(tx, a, sm_count, st))
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
