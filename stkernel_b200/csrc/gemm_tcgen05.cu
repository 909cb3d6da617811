// Dense linear layer on the 5th-generation tensor cores:  out[T, N] = X[T, K] * W[N, K]^T
//
// * Operands arrive by TMA (128-byte swizzle) into a multi-stage shared-memory ring.
// * One elected thread issues tcgen05.mma; the accumulator lives in TMEM (double buffered).
// * The weight tile is the 128-row "M" operand and the token tile is the "N" operand
//   (16..256 tokens), so decode-sized batches still use full-height MMAs and each epilogue
//   thread owns one output feature, which makes the global stores contiguous across a warp.
// * bf16 operands: one accumulation over all of K, epilogue once per tile.
// * fp8 e4m3 operands with 128x128 weight scales and 1x128 activation scales: one TMEM
//   accumulation per 128-wide K block; the epilogue warps fold `w_scale * x_scale` into
//   fp32 register accumulators while the next block's MMAs run (two-level accumulation).
// * Split-K for skinny problems: partial tiles go to an fp32 workspace, the last CTA to
//   finish a tile sums the partials in split order (deterministic) and writes the output.
// * Persistent grid: one CTA per SM walks the (split, token-tile, feature-tile) list.
//
// Covers the reference's DeepGEMM fp8_gemm_nt call sites (overlay/dspark_v2.py:92-107,
// probes/oproj_prof.py:65-71) and its bf16 cuBLAS projections.
#include <string.h>

#define STK_PDL_CLASS 8      // bit of this file's kernels in the PDL mask (STK_PDL, stk_set_pdl_mask)
#include <stdlib.h>

#include "common.cuh"
#include "pairs.cuh"
#include "stk_c_api.h"
#include "symm.cuh"

namespace stk {

struct GemmArgs {
  int T, N;
  int k_blocks;          // K extent in 128-byte blocks
  int splits;            // split-K factor (>= 1)
  int tiles_n, tiles_t;
  void* out;             // [T, ldo]
  long long ldo;
  int out_fp32;
  const float* w_scale;  // fp8 only: [ceil(N/128), w_scale_ld]
  int w_scale_ld;
  const float* x_scale;  // fp8 only: [k_blocks, x_scale_ld]  (token index contiguous)
  int x_scale_ld;
  float* workspace;      // split-K partials [splits, T, N]
  int* counters;         // one per output tile; zero on entry, zero again on exit
  int* status;
  // Grouped mode (block-diagonal weights, e.g. the per-o-group low-rank projection): feature tile
  // `tn` belongs to group tn / group_tiles and reads X columns starting at group * group_k_elems.
  int group_tiles;       // 0 = plain GEMM
  int group_k_elems;
  // Fused all-reduce (row-parallel layers): every rank pushes its partial output tile into all
  // peers' slots as soon as the tile's accumulation ends, then sums the tiles it received in
  // rank order.  The transfer of tile i overlaps the MMAs of tile i+1 of the same CTA and of
  // all other CTAs.
  int ar_enabled;
  SymmCtx ar;
  // Arrival-gated activations (all-gather -> GEMM): X is the gathered matrix in this rank's symmetric region,
  // rows [s * gate_rows, (s+1) * gate_rows) are pushed by rank s and are complete once flag (kAgKind, 0, s)
  // carries the current epoch.  Token tiles are visited starting with this rank's own shard.
  int gate_enabled;
  int gate_rows;
  // Whether the split-K reduction may write `out` with 16-byte (fp32) / 4-byte (bf16) vector stores: the host sets
  // it from the alignment of `out` and `ldo`; otherwise the reduction writes element by element.
  int out_vec_ok;
};

constexpr int kArKind = 3;
constexpr int kGateKind = 4;      // flags written by the all-gather push kernel (symm.cu)

template <int BT>
struct GemmCfg {
  static constexpr int kStageBytes = 128 * 128 + BT * 128;
  // bf16 staging tile [BT][128] for the fused all-reduce epilogue (token tiles up to 128)
  static constexpr int kArTileBytes = BT <= 128 ? BT * 256 : 0;
  static constexpr int kStagesRaw = (196 * 1024) / kStageBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  static constexpr int kTmemCols = (2 * BT <= 32) ? 32 : (2 * BT <= 64) ? 64 : (2 * BT <= 128) ? 128 : (2 * BT <= 256) ? 256 : 512;
  static constexpr int kChunk = BT >= 32 ? 32 : 16;
};

struct alignas(8) GemmBarriers {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int last_flag;
};

template <int CW>
__device__ __forceinline__ void tmem_ld_chunk(uint32_t taddr, uint32_t (&r)[32]) {
  if constexpr (CW == 32) {
    tmem_ld_32x32(taddr, r);
  } else {
    uint32_t t[16];
    tmem_ld_32x16(taddr, t);
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = t[i];
  }
}

__device__ __forceinline__ void epi_bar_sync(int nthreads) {
  asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
}

template <int BT, bool kFp8>
__global__ void __launch_bounds__(kFp8 ? 320 : 192, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const GemmArgs a) {
  using Cfg = GemmCfg<BT>;
  constexpr int kStages = Cfg::kStages;
  constexpr int CW = Cfg::kChunk;
  // epilogue warps: fp8 with wide tiles splits the columns over two warps per lane quarter
  constexpr int kEpiWarps = (kFp8 && BT >= 64) ? 8 : 4;
  constexpr int kColsPerWarp = (kEpiWarps == 8) ? BT / 2 : BT;
  constexpr int kChunksPerWarp = kColsPerWarp / CW;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_a = smem;                                  // kStages x 16 KB
  uint8_t* smem_b = smem + kStages * 128 * 128;            // kStages x BT*128
  GemmBarriers* bars = reinterpret_cast<GemmBarriers*>(smem_b + kStages * BT * 128);
  __nv_bfloat16* ar_tile = reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<uint8_t*>(bars) + 256);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], kEpiWarps);
    }
    bars->last_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, Cfg::kTmemCols);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  // Launched with programmatic serialization (plain GEMMs only): barriers, TMEM and descriptors are set up and the
  // first weight tiles of this CTA are on their way to L2 while the previous kernel finishes; activations, split-K
  // counters and epochs are touched only after the wait.
  if (warp == 0 && lane == 0 && static_cast<int>(blockIdx.x) < a.splits * a.tiles_t * a.tiles_n) {
    const int u = blockIdx.x;
    const int tn = u % a.tiles_n;
    const int sp = u / (a.tiles_n * a.tiles_t);
    const int kbs = (a.k_blocks + a.splits - 1) / a.splits;
    const int kb0 = sp * kbs;
    const int kb1 = min(a.k_blocks, min(kb0 + kbs, kb0 + 8));
    for (int kb = kb0; kb < kb1; ++kb) tma_prefetch_2d(&tmW, kb * (kFp8 ? 128 : 64), tn * 128);
  }
  pdl_wait();
  pdl_trigger();
  uint32_t ar_epoch = 0;
  if (a.ar_enabled) ar_epoch = *epoch_ptr(a.ar, kArKind, 0) + 1;   // bumped only after every CTA has finished

  uint32_t gate_epoch = 0;
  int tt_rot = 0;
  if (a.gate_enabled) {
    gate_epoch = *epoch_ptr(a.ar, kGateKind, 0);                   // the push of this call has already run on this rank
    tt_rot = (a.ar.rank * a.gate_rows) / BT;
  }
  const int units = a.splits * a.tiles_t * a.tiles_n;
  const int kb_per_split = (a.k_blocks + a.splits - 1) / a.splits;
  constexpr uint32_t kIdesc = umma_idesc(kFp8 ? 0u : 1u, kFp8 ? 0u : 1u, 128, BT);
  constexpr uint32_t kTxBytes = 128 * 128 + BT * 128;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int issued = 0;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const int tn = u % a.tiles_n;
        const int tt = ((u / a.tiles_n) % a.tiles_t + tt_rot) % a.tiles_t;
        const int sp = u / (a.tiles_n * a.tiles_t);
        const int kb0 = sp * kb_per_split;
        const int kb1 = min(a.k_blocks, kb0 + kb_per_split);
        if (a.gate_enabled) {
          // the rows of this token tile come from one or two source ranks: wait (bounded) for their pushes
          const int s0 = (tt * BT) / a.gate_rows;
          const int s1 = min(a.ar.world - 1, (min(a.T, (tt + 1) * BT) - 1) / a.gate_rows);
          for (int sr = s0; sr <= s1 && ok; ++sr) {
            if (sr == a.ar.rank) continue;
            if (!wait_flag(flag_ptr(a.ar, a.ar.rank, kGateKind, 0, sr), gate_epoch, a.ar.spin_budget, a.status, 600 + sr))
              ok = false;
          }
          if (!ok) break;
          asm volatile("fence.proxy.async.global;" ::: "memory");    // peer stores (generic proxy) -> TMA reads
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 100 + stage)) { ok = false; break; }
          mbar_expect_tx(&bars->full[stage], kTxBytes);
          const int kx = kb * (kFp8 ? 128 : 64);
          const int gx = a.group_tiles ? (tn / a.group_tiles) * a.group_k_elems : 0;
          tma_load_2d(smem_a + stage * 128 * 128, &tmW, &bars->full[stage], kx, tn * 128);
          tma_load_2d(smem_b + stage * BT * 128, &tmX, &bars->full[stage], gx + kx, tt * BT);
          ++issued;
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // Drain: wait (bounded) until every load issued to the ring has landed.
        const int pending = issued < kStages ? issued : kStages;
        int s = stage;
        uint32_t ph = phase;
        for (int i = 0; i < pending; ++i) {
          if (--s < 0) { s = kStages - 1; ph ^= 1; }
          mbar_wait(&bars->full[s], ph, nullptr, 0);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int ab = 0;
      uint32_t aphase = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const int sp = u / (a.tiles_n * a.tiles_t);
        const int kb0 = sp * kb_per_split;
        const int kb1 = min(a.k_blocks, kb0 + kb_per_split);
        if constexpr (!kFp8) {
          if (!mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 200 + ab)) { ok = false; break; }
          tc_fence_after();
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if constexpr (kFp8) {
            if (!mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 200 + ab)) { ok = false; break; }
          }
          if (!mbar_wait(&bars->full[stage], phase, a.status, 300 + stage)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem_base + ab * BT;
          const uint64_t adesc = umma_desc_sw128(smem_u32(smem_a + stage * 128 * 128));
          const uint64_t bdesc = umma_desc_sw128(smem_u32(smem_b + stage * BT * 128));
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            // advance 32 bytes along K inside the swizzled 128-byte row (encoded >> 4)
            const uint32_t acc = kFp8 ? (k > 0) : (kb > kb0 || k > 0);
            if constexpr (kFp8) umma_f8(d, adesc + 2 * k, bdesc + 2 * k, kIdesc, acc);
            else umma_f16(d, adesc + 2 * k, bdesc + 2 * k, kIdesc, acc);
          }
          umma_commit(&bars->empty[stage]);
          if constexpr (kFp8) {
            umma_commit(&bars->tmem_full[ab]);
            if (++ab == 2) { ab = 0; aphase ^= 1; }
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
        if constexpr (!kFp8) {
          if (ok) {
            umma_commit(&bars->tmem_full[ab]);
            if (++ab == 2) { ab = 0; aphase ^= 1; }
          }
        }
      }
    }
  } else if (warp - 2 < kEpiWarps) {
    // ------------------------------ epilogue -----------------------------------
    const int e = warp - 2;
    const int q = warp & 3;                         // TMEM lane quarter this warp may read
    const int col_base = (kEpiWarps == 8) ? (e >> 2) * kColsPerWarp : 0;
    const int row = q * 32 + lane;
    int ab = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int tn = u % a.tiles_n;
      const int tt = ((u / a.tiles_n) % a.tiles_t + tt_rot) % a.tiles_t;
      const int sp = u / (a.tiles_n * a.tiles_t);
      const int kb0 = sp * kb_per_split;
      const int kb1 = min(a.k_blocks, kb0 + kb_per_split);
      const int n = tn * 128 + row;
      const int t0 = tt * BT + col_base;
      const bool n_ok = n < a.N;

      const int ar_par = ar_epoch & 1;
      const long long ar_slot = a.ar.gemm_bytes / 2;      // bf16 elements per (parity, source) slot
      auto ar_push = [&](int t, float v) {
        if constexpr (Cfg::kArTileBytes > 0) ar_tile[(t - tt * BT) * 128 + row] = __float2bfloat16(v);
      };
      // copy the staged tile to every rank with 16-byte stores, signal it, wait (bounded) for every
      // rank's tile, and sum the tiles in rank order
      auto ar_finish = [&]() -> bool {
        const int tile = (tt * a.tiles_n + tn) & 4095;
        const int et = threadIdx.x - 64;
        const int nthr = kEpiWarps * 32;
        const int rows_valid = min(BT, a.T - tt * BT);
        const int nvec = rows_valid * 16;
        epi_bar_sync(nthr);
        for (int p = 0; p < a.ar.world; ++p) {
          const int peer = (a.ar.rank + p) % a.ar.world;
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.ar.base[peer] + a.ar.off_gemm) +
                               (static_cast<long long>(ar_par) * a.ar.world + a.ar.rank) * ar_slot;
          for (int v = et; v < nvec; v += nthr) {
            const int r = v >> 4, cvec = v & 15;
            const uint4 val = *reinterpret_cast<const uint4*>(ar_tile + r * 128 + cvec * 8);
            *reinterpret_cast<uint4*>(dst + static_cast<long long>(tt * BT + r) * a.N + tn * 128 + cvec * 8) = val;
          }
        }
        epi_bar_sync(nthr);
        if (et < a.ar.world) {
          __threadfence_system();      // cumulative with the barrier: orders every thread's pushes before the flag
          st_release_sys(flag_ptr(a.ar, et, kArKind, tile, a.ar.rank), ar_epoch);
        }
        if (et == 0) bars->last_flag = 1;
        epi_bar_sync(nthr);
        if (et < a.ar.world) {
          if (!wait_flag(flag_ptr(a.ar, a.ar.rank, kArKind, tile, et), ar_epoch, a.ar.spin_budget, a.status, 500 + et))
            bars->last_flag = 0;
        }
        epi_bar_sync(nthr);
        const bool got = bars->last_flag != 0;
        if (got) {
          const __nv_bfloat16* slots = reinterpret_cast<const __nv_bfloat16*>(a.ar.base[a.ar.rank] + a.ar.off_gemm) +
                                       static_cast<long long>(ar_par) * a.ar.world * ar_slot;
          for (int v = et; v < nvec; v += nthr) {
            const int r = v >> 4, cvec = v & 15;
            const long long off = static_cast<long long>(tt * BT + r) * a.N + tn * 128 + cvec * 8;
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int rk = 0; rk < a.ar.world; ++rk) {
              const uint4 val = __ldcg(reinterpret_cast<const uint4*>(slots + rk * ar_slot + off));
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&val);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                acc[2 * i] += __low2float(h[i]);
                acc[2 * i + 1] += __high2float(h[i]);
              }
            }
            if (a.out_fp32) {
              float* o = reinterpret_cast<float*>(a.out) + static_cast<long long>(tt * BT + r) * a.ldo + tn * 128 + cvec * 8;
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = acc[i];
            } else {
              uint4 ov;
              __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
              for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + static_cast<long long>(tt * BT + r) * a.ldo +
                                        tn * 128 + cvec * 8) = ov;
            }
          }
        }
        epi_bar_sync(nthr);
        return got;
      };
      auto store = [&](int t, float v) {
        if (n_ok && t < a.T) {
          if (a.splits > 1) {
            a.workspace[(static_cast<long long>(sp) * a.T + t) * a.N + n] = v;
          } else if (a.ar_enabled) {
            ar_push(t, v);
          } else if (a.out_fp32) {
            reinterpret_cast<float*>(a.out)[t * a.ldo + n] = v;
          } else {
            reinterpret_cast<__nv_bfloat16*>(a.out)[t * a.ldo + n] = __float2bfloat16(v);
          }
        }
      };

      if constexpr (kFp8) {
        float acc[kColsPerWarp];
#pragma unroll
        for (int j = 0; j < kColsPerWarp; ++j) acc[j] = 0.f;
        for (int kb = kb0; kb < kb1 && ok; ++kb) {
          const float sw = a.w_scale[tn * a.w_scale_ld + kb];
          const int gkb = a.group_tiles ? (tn / a.group_tiles) * a.k_blocks : 0;
          const float* xs = a.x_scale + static_cast<long long>(gkb + kb) * a.x_scale_ld;
          if (!mbar_wait(&bars->tmem_full[ab], aphase, a.status, 400 + ab)) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < kChunksPerWarp; ++c) {
            uint32_t r[32];
            tmem_ld_chunk<CW>(tmem_base + ab * BT + col_base + c * CW + (static_cast<uint32_t>(q * 32) << 16), r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < CW; j += 4) {
              const int t = t0 + c * CW + j;
              float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
              if (t + 4 <= a.x_scale_ld) s4 = __ldg(reinterpret_cast<const float4*>(xs + t));
              acc[c * CW + j + 0] = fmaf(__uint_as_float(r[j + 0]), sw * s4.x, acc[c * CW + j + 0]);
              acc[c * CW + j + 1] = fmaf(__uint_as_float(r[j + 1]), sw * s4.y, acc[c * CW + j + 1]);
              acc[c * CW + j + 2] = fmaf(__uint_as_float(r[j + 2]), sw * s4.z, acc[c * CW + j + 2]);
              acc[c * CW + j + 3] = fmaf(__uint_as_float(r[j + 3]), sw * s4.w, acc[c * CW + j + 3]);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->tmem_empty[ab]);
          if (++ab == 2) { ab = 0; aphase ^= 1; }
        }
        if (ok) {
#pragma unroll
          for (int j = 0; j < kColsPerWarp; ++j) store(t0 + j, acc[j]);
        }
      } else {
        if (!mbar_wait(&bars->tmem_full[ab], aphase, a.status, 400 + ab)) { ok = false; break; }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < kChunksPerWarp; ++c) {
          uint32_t r[32];
          tmem_ld_chunk<CW>(tmem_base + ab * BT + col_base + c * CW + (static_cast<uint32_t>(q * 32) << 16), r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < CW; ++j) store(t0 + c * CW + j, __uint_as_float(r[j]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->tmem_empty[ab]);
        if (++ab == 2) { ab = 0; aphase ^= 1; }
      }

      if (a.ar_enabled && a.splits == 1 && ok) ok = ar_finish();
      if (a.splits > 1 && ok) {
        // Publish this split's partial; the CTA that completes the tile reduces it.
        __threadfence();
        epi_bar_sync(kEpiWarps * 32);
        if (threadIdx.x == 64) {
          const int prev = atomicAdd(&a.counters[tt * a.tiles_n + tn], 1);
          bars->last_flag = (prev == a.splits - 1);
          if (prev == a.splits - 1) a.counters[tt * a.tiles_n + tn] = 0;
        }
        epi_bar_sync(kEpiWarps * 32);
        const bool last = bars->last_flag != 0;
        epi_bar_sync(kEpiWarps * 32);
        if (last) {
          __threadfence();
          // Cooperative reduction: the tile's partials are [split][token][128 features] fp32 rows of
          // 512 contiguous bytes; every epilogue thread sums float4 vectors (all loads independent).
          {
            const int et2 = threadIdx.x - 64;
            const int nthr2 = kEpiWarps * 32;
            const int rows_valid = min(BT, a.T - tt * BT);
            const int cols_valid = min(128, a.N - tn * 128);
            const int cv = cols_valid >> 2;                  // vectors of a row (a tile at the edge of N has fewer than 32)
            const bool vec_ok = ((a.N & 3) == 0) && (a.out_vec_ok || a.ar_enabled);
            if (vec_ok) {
              // four output vectors per thread at a time, so that 4 x (unrolled splits) loads are in flight: one vector
              // at a time left a reducing CTA at a few dozen GB/s
              const int total = rows_valid * cv;
              for (int v0 = et2; v0 < total; v0 += nthr2 * 4) {
                float4 s4[4];
                int row4[4], col4[4];
                const float* src[4];                        // the vector's place in split 0 (the last one's past the end)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  s4[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                  const int v = min(v0 + u * nthr2, total - 1);
                  row4[u] = cv == 32 ? v >> 5 : v / cv;
                  col4[u] = (v - row4[u] * cv) * 4;
                  src[u] = a.workspace + static_cast<long long>(tt * BT + row4[u]) * a.N + tn * 128 + col4[u];
                }
                const long long split_step = static_cast<long long>(a.T) * a.N;
#pragma unroll 4
                for (int p = 0; p < a.splits; ++p) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) {
                    const float4 x = __ldcg(reinterpret_cast<const float4*>(src[u] + p * split_step));
                    s4[u].x += x.x; s4[u].y += x.y; s4[u].z += x.z; s4[u].w += x.w;
                  }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                  if (v0 + u * nthr2 >= total) break;
                  const int r = row4[u], c4 = col4[u];
                  const int t = tt * BT + r;
                  if (a.ar_enabled) {
                    if constexpr (Cfg::kArTileBytes > 0) {
                      __nv_bfloat162* d = reinterpret_cast<__nv_bfloat162*>(ar_tile + r * 128 + c4);
                      d[0] = __floats2bfloat162_rn(s4[u].x, s4[u].y);
                      d[1] = __floats2bfloat162_rn(s4[u].z, s4[u].w);
                    }
                  } else if (a.out_fp32) {
                    *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + t * a.ldo + tn * 128 + c4) = s4[u];
                  } else {
                    __nv_bfloat162* d = reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(a.out) + t * a.ldo + tn * 128 + c4);
                    d[0] = __floats2bfloat162_rn(s4[u].x, s4[u].y);
                    d[1] = __floats2bfloat162_rn(s4[u].z, s4[u].w);
                  }
                }
              }
            } else {
              for (int v = et2; v < rows_valid * cols_valid; v += nthr2) {
                const int r = v / cols_valid, cc = v % cols_valid;
                const int t = tt * BT + r, nn = tn * 128 + cc;
                float sacc = 0.f;
                for (int p = 0; p < a.splits; ++p) sacc += __ldcg(&a.workspace[(static_cast<long long>(p) * a.T + t) * a.N + nn]);
                if (a.ar_enabled) {
                  if constexpr (Cfg::kArTileBytes > 0) ar_tile[r * 128 + cc] = __float2bfloat16(sacc);
                } else if (a.out_fp32) {
                  reinterpret_cast<float*>(a.out)[t * a.ldo + nn] = sacc;
                } else {
                  reinterpret_cast<__nv_bfloat16*>(a.out)[t * a.ldo + nn] = __float2bfloat16(sacc);
                }
              }
            }
          }
          if (a.ar_enabled) ok = ar_finish();
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
  if (a.ar_enabled && threadIdx.x == 0) {
    // the last CTA to leave advances the epoch for the next call
    __threadfence();
    uint32_t* done = epoch_ptr(a.ar, kArKind, 1);
    if (atomicAdd(done, 1u) == gridDim.x - 1) {
      *done = 0;
      *epoch_ptr(a.ar, kArKind, 0) = ar_epoch;
      __threadfence();
    }
  }
}

// ---- clusters that split K ---------------------------------------------------------
__device__ __forceinline__ uint32_t peer_addr(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---------------------------------------------------------------------------------
// Wide tile for large bf16 problems: one CTA owns 256 tokens x 256 weight rows (token-major: TMEM lanes are tokens,
// so an epilogue thread writes 64 contiguous bytes of its token's output row per chunk).
//
// Measured on the 128 x 256 tile above (4096 x 4096 x 8192, ncu): tensor pipe 31 % active, no unit saturated; the
// kernel is paced by operand delivery (48 KB per 512 tensor-core cycles per SM, 7.9 TB/s out of L2 over all SMs), and
// adding L2 prefetch requests made it slower -- it is the L2 -> SM path that is short, not DRAM.  Two 128-token MMAs that
// share one 256-row weight stage need 64 KB per 1024 cycles: two thirds of the traffic per FLOP, and the three-stage
// ring covers 3072 tensor-core cycles instead of 2048.  The two accumulators take all 512 TMEM columns, so the
// epilogue of a tile is not overlapped with the next tile's MMAs; eight epilogue warps with 16-byte stores keep it short.
// ---------------------------------------------------------------------------------
struct WideArgs {
  int T, N, k_blocks, tiles_n, tiles_t;
  void* out;
  long long ldo;
  int out_fp32;
  int* status;
  // block-diagonal weights: tn / group_tiles is the block, its X columns start at that times group_k (0: one block)
  int group_tiles, group_k;
};

constexpr int kWideStages = 3;
constexpr int kWideStageBytes = 2 * 128 * 128 + 256 * 128;       // two weight tiles + one token tile = 64 KB

// A cluster of four CTAs shares a tile, each with its part of K.  CTA j writes piece j of the tile (128 tokens x 128 weight rows); the
// others bring it their partial sums through distributed shared memory, into the operand ring that is free by then.  Sums are formed in
// the order of the CTAs' ranks.  (Tiles that one or two CTAs can have to themselves are left to the pairs below.)
__global__ void __launch_bounds__(320, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const WideArgs a) {
  constexpr int S = 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  GemmBarriers* bars = reinterpret_cast<GemmBarriers*>(smem + kWideStages * kWideStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kWideStages; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    mbar_init(&bars->tmem_full[0], 1);
    mbar_init(&bars->tmem_empty[0], 8);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();
  pdl_trigger();
  const int units = a.tiles_n * a.tiles_t;
  constexpr uint32_t kIdesc = umma_idesc(1u, 1u, 128, 256);
  const int rank = static_cast<int>(blockIdx.x) % S;
  const int per = (a.k_blocks + S - 1) / S, k_begin = rank * per, k_end = min(a.k_blocks, k_begin + per);
  const int u_first = blockIdx.x / S, u_step = gridDim.x / S;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = u_first; u < units && ok; u += u_step) {
        const int tn = u % a.tiles_n, tt = u / a.tiles_n;
        const int gx = a.group_tiles ? tn / a.group_tiles * a.group_k : 0;
        for (int kb = k_begin; kb < k_end; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 100 + stage)) { ok = false; break; }
          mbar_expect_tx(&bars->full[stage], kWideStageBytes);
          uint8_t* st = smem + stage * kWideStageBytes;
          // token-major: the two A operands are 128-token tiles (TMEM lanes = tokens), B is the 256-row weight tile
          const int kx = kb * 64 + gx;
          tma_load_2d(st, &tmX, &bars->full[stage], kx, tt * 256);
          tma_load_2d(st + 128 * 128, &tmX, &bars->full[stage], kx, tt * 256 + 128);
          tma_load_2d(st + 2 * 128 * 128, &tmW, &bars->full[stage], kb * 64, tn * 256);
          ++issued;
          if (++stage == kWideStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // drain: wait (bounded) until every load issued to the ring has landed
        const int pending = issued < kWideStages ? issued : kWideStages;
        int s = stage;
        uint32_t ph = phase;
        for (int i = 0; i < pending; ++i) {
          if (--s < 0) { s = kWideStages - 1; ph ^= 1; }
          mbar_wait(&bars->full[s], ph, nullptr, 0);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0), s_lo = desc_lo(smem_u32(smem));
    int stage = 0;
    uint32_t phase = 0, aphase = 0;
    bool ok = true;
    for (int u = u_first; u < units && ok; u += u_step) {
      ok = mbar_wait(&bars->tmem_empty[0], aphase ^ 1, a.status, 200);
      if (!ok) break;
      tc_fence_after();
      for (int kb = k_begin; kb < k_end; ++kb) {
        ok = mbar_wait(&bars->full[stage], phase, a.status, 300 + stage);
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = s_lo + stage * (kWideStageBytes >> 4);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t acc = (kb > k_begin || k > 0) ? 1u : 0u;
          mma_ss(tm, st + 2 * k, st + 2048 + 2 * k, kIdesc, acc, lead);
          mma_ss(tm + 256, st + 1024 + 2 * k, st + 2048 + 2 * k, kIdesc, acc, lead);
        }
        mma_commit(&bars->empty[stage], lead);
        if (++stage == kWideStages) { stage = 0; phase ^= 1; }
      }
      if (ok) mma_commit(&bars->tmem_full[0], lead);
      aphase ^= 1;
    }
    __syncwarp();
  } else {
    // eight epilogue warps: lane quarter q = warp % 4 (the TMEM lanes a warp may read), column half h
    const int e = warp - 2;
    const int q = warp & 3, h = e >> 2;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    uint32_t aphase = 0;
    bool ok = true;
    for (int u = u_first; u < units && ok; u += u_step) {
      const int tn = u % a.tiles_n, tt = u / a.tiles_n;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[0], aphase, a.status, 400));
      tc_fence_after();
      // a thread owns one token row and, per chunk, 32 consecutive output features: 64 contiguous bytes of bf16
      const bool vec_ok = !a.out_fp32 && (a.ldo % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.out) & 15) == 0);
      const bool vec32_ok = (a.ldo % 4 == 0) && ((reinterpret_cast<uintptr_t>(a.out) & 15) == 0);
      auto store32 = [&](int m, int col, const uint32_t (&r)[32]) {
        const int t = tt * 256 + m * 128 + q * 32 + lane;
        const bool t_ok = t < a.T;
        const int n0 = tn * 256 + col;
        if (t_ok) {
          if (vec_ok && n0 + 32 <= a.N) {
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + static_cast<long long>(t) * a.ldo + n0;
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
              uint4 ov;
              __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
              for (int i = 0; i < 4; ++i)
                oh[i] = __floats2bfloat162_rn(__uint_as_float(r[j + 2 * i]), __uint_as_float(r[j + 2 * i + 1]));
              *reinterpret_cast<uint4*>(o + j) = ov;
            }
          } else if (a.out_fp32) {
            float* o = reinterpret_cast<float*>(a.out) + static_cast<long long>(t) * a.ldo + n0;
            if (vec32_ok && n0 + 32 <= a.N) {
#pragma unroll
              for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(o + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (n0 + j < a.N) o[j] = __uint_as_float(r[j]);
            }
          } else {
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + static_cast<long long>(t) * a.ldo + n0;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (n0 + j < a.N) o[j] = __float2bfloat16(__uint_as_float(r[j]));
          }
        }
      };
      {
        // piece j: token tile m_of(j), columns from c_of(j); this warp's share of a piece is kShare columns of its lane quarter
        constexpr int kCols = 512 / S, kShare = kCols / 2;
        auto m_of = [](int j) { return j >> 1; };
        auto c_of = [](int j) { return (j & 1) * 128; };
        const uint32_t line = smem_u32(smem) + (q * 32 + lane) * 16;      // [slot][column / 4][token] of 16 bytes
        cluster_sync_all();                                               // every CTA's products are done: the rings are free
#pragma unroll 1
        for (int d = 1; d < S; ++d) {
          const int j = (rank + d) % S;
          const uint32_t to = peer_addr(line + (rank < j ? rank : rank - 1) * (kCols * 512), j);
#pragma unroll 1
          for (int c = 0; c < kShare; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(tmem_base + m_of(j) * 256 + c_of(j) + h * kShare + c + lane_addr, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                           ::"r"(to + (h * kShare + c + i) / 4 * 2048), "r"(r[i]), "r"(r[i + 1]), "r"(r[i + 2]), "r"(r[i + 3]) : "memory");
          }
        }
        cluster_sync_all();                                               // all pieces have arrived
#pragma unroll 1
        for (int c = 0; c < kShare; c += 32) {
          uint32_t r[32];
          float v[32];
          tmem_ld_32x32(tmem_base + m_of(rank) * 256 + c_of(rank) + h * kShare + c + lane_addr, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0.f;
#pragma unroll
          for (int j = 0; j < S; ++j) {
            if (j == rank) {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] += __uint_as_float(r[i]);
            } else {
              const uint32_t from = line + (j < rank ? j : j - 1) * (kCols * 512) + (h * kShare + c) / 4 * 2048;
#pragma unroll
              for (int i = 0; i < 32; i += 4) {
                float x0, x1, x2, x3;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x0), "=f"(x1), "=f"(x2), "=f"(x3) : "r"(from + i / 4 * 2048));
                v[i] += x0; v[i + 1] += x1; v[i + 2] += x2; v[i + 3] += x3;
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(v[i]);
          store32(m_of(rank), c_of(rank) + h * kShare + c, r);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->tmem_empty[0]);
      aphase ^= 1;
    }
  }
  if (warp < 2) {
    // the CTAs of a cluster meet twice (one tile each)
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------
// fp8, token-major (from nine tokens on, see fp8_tokens_split): TMEM lanes are tokens, columns are weight rows, so the scale of a K
// block is one multiplier per thread.  One CTA owns 128 tokens x 128 weight rows.
//
// What bounds it: a K block is 259 tensor-core cycles, and its 128 x 128 results have to be read back from TMEM, scaled and added
// to the second-level accumulators (fp32, in registers).  The scales of a block are asked for four blocks ahead (loaded when their
// block's products were done, they held every block up for a trip to memory), four accumulators are in flight, and a buffer is given
// back as soon as it has been read.  Operands are 32 KB a block; at 4096 tokens 2.1 GB of them leave L2 in 172 us.
// Measured (4096 tokens, 4096 x 8192): 241 us with scales loaded on demand, 172 us now.  Sixteen epilogue warps instead of eight
// took 238 us, 256 tokens a CTA 193 us.
// ---------------------------------------------------------------------------------
struct Fp8Args {
  int T, N, k_blocks, tiles_t, tiles_n;
  void* out;
  long long ldo;
  int out_fp32;
  const float* w_scale;
  int w_scale_ld;
  const float* x_scale;
  int x_scale_ld;
  int* status;
};

constexpr int kFp8StageBytes = 2 * 128 * 128, kFp8Stages = 6;
constexpr int kFp8Bufs = 4;                                    // accumulators in TMEM, 128 columns each
constexpr int kFp8EpiWarps = 8, kFp8Threads = 32 * (2 + kFp8EpiWarps);

struct alignas(8) Fp8Bars {
  uint64_t full[6], empty[6], tmem_full[4], tmem_empty[4];
  uint32_t tmem_base;
};

// D[tmem] (+)= A[smem] * B[smem], e4m3 operands, issued by a converged warp (see common.cuh)
__device__ __forceinline__ void mma_ss_f8(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %4, p;\n\t}"
      ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(acc), "r"(lead)
      : "memory");
}

// S > 1: a cluster of S CTAs shares a tile, each with its part of K; CTA j writes kCols / S columns of every epilogue thread, to
// which the others' sums come through distributed shared memory (into the operand ring, free by then), added in rank order.
template <int S>
__global__ void __launch_bounds__(kFp8Threads, 1)
gemm_fp8_tokens_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Fp8Args a) {
  constexpr int kStages = kFp8Stages, kBufs = kFp8Bufs, kCols = 64;       // columns of an epilogue warp
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Fp8Bars* bars = reinterpret_cast<Fp8Bars*>(smem + kStages * kFp8StageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], kFp8EpiWarps);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();
  pdl_trigger();
  const int units = a.tiles_t * a.tiles_n;
  const int rank = S > 1 ? static_cast<int>(blockIdx.x) % S : 0;
  const int per = (a.k_blocks + S - 1) / S, k_begin = min(a.k_blocks, rank * per), k_end = min(a.k_blocks, k_begin + per);
  const int u_first = blockIdx.x / S, u_step = gridDim.x / S;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = u_first; u < units && ok; u += u_step) {
        const int tt = u % a.tiles_t, tn = u / a.tiles_t;
        for (int kb = k_begin; kb < k_end; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 100 + stage)) { ok = false; break; }
          mbar_expect_tx(&bars->full[stage], kFp8StageBytes);
          uint8_t* st = smem + stage * kFp8StageBytes;
          tma_load_2d(st, &tmX, &bars->full[stage], kb * 128, tt * 128);
          tma_load_2d(st + 128 * 128, &tmW, &bars->full[stage], kb * 128, tn * 128);
          ++issued;
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // drain: wait (bounded) until every load issued to the ring has landed
        const int pending = issued < kStages ? issued : kStages;
        int s = stage;
        uint32_t ph = phase;
        for (int i = 0; i < pending; ++i) {
          if (--s < 0) { s = kStages - 1; ph ^= 1; }
          mbar_wait(&bars->full[s], ph, nullptr, 0);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0), s_lo = desc_lo(smem_u32(smem));
    constexpr uint32_t kIdesc = umma_idesc(0u, 0u, 128, 128);
    const long long total = units > u_first ? ((units - 1 - u_first) / u_step + 1LL) * (k_end - k_begin) : 0;
    int stage = 0, ab = 0;
    uint32_t phase = 0, aphase = 0;
    for (long long i = 0; i < total; ++i) {
      if (!mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 200 + ab) || !mbar_wait(&bars->full[stage], phase, a.status, 300 + stage)) break;
      tc_fence_after();
      const uint32_t st = s_lo + stage * (kFp8StageBytes >> 4), d = tm + ab * 128;
#pragma unroll
      for (int k = 0; k < 4; ++k) mma_ss_f8(d, st + 2 * k, st + 1024 + 2 * k, kIdesc, k > 0 ? 1u : 0u, lead);
      mma_commit(&bars->empty[stage], lead);
      mma_commit(&bars->tmem_full[ab], lead);
      if (++stage == kStages) { stage = 0; phase ^= 1; }
      if (++ab == kBufs) { ab = 0; aphase ^= 1; }
    }
    __syncwarp();
  } else {
    // ------------------------------ epilogue -----------------------------------
    // a thread owns one token and kCols weight rows
    const int e = warp - 2, q = warp & 3, col0 = (e >> 2) * kCols;
    const uint32_t tile = tmem_base + col0 + (static_cast<uint32_t>(q * 32) << 16);
    int ab = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int u = u_first; u < units && ok; u += u_step) {
      const int tt = u % a.tiles_t, tn = u / a.tiles_t;
      const int t = tt * 128 + q * 32 + lane;
      const bool t_ok = t < a.T;
      const bool live = tt * 128 + q * 32 < a.T;         // some lane of this warp has a token
      const float* xs = a.x_scale + (t_ok ? t : 0);
      const float* ws = a.w_scale + static_cast<long long>(tn) * a.w_scale_ld;
      constexpr int kAhead = 4;
      float sx[kAhead], sw[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int kb = min(k_begin + i, a.k_blocks - 1);
        sx[i] = __ldg(xs + static_cast<long long>(kb) * a.x_scale_ld);
        sw[i] = __ldg(ws + kb);
      }
      uint64_t acc[kCols / 2];
#pragma unroll
      for (int j = 0; j < kCols / 2; ++j) acc[j] = 0ull;
      for (int kb0 = k_begin; kb0 < k_end && ok; kb0 += kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int kb = kb0 + i;
          if (kb >= k_end || !ok) break;
          const float s = sx[i] * sw[i];
          const uint64_t s2 = pack2(s, s);
          const int next = min(kb + kAhead, a.k_blocks - 1);
          sx[i] = __ldg(xs + static_cast<long long>(next) * a.x_scale_ld);
          sw[i] = __ldg(ws + next);
          ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[ab], aphase, a.status, 400 + ab));
          if (!ok) break;
          tc_fence_after();
          uint32_t r[2][32];
          if (live) {
            tmem_ld_32x32(tile + ab * 128, r[0]);
            tmem_ld_32x32(tile + ab * 128 + 32, r[1]);
            tmem_ld_wait();
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->tmem_empty[ab]);
          if (live) {
#pragma unroll
            for (int j = 0; j < kCols; j += 2)
              acc[j / 2] = fma2(pack2(__uint_as_float(r[j / 32][j % 32]), __uint_as_float(r[j / 32][j % 32 + 1])), s2, acc[j / 2]);
          }
          if (++ab == kBufs) { ab = 0; aphase ^= 1; }
        }
      }
      const bool aligned = (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 && a.ldo % (a.out_fp32 ? 4 : 8) == 0;
      auto store8 = [&](int c, const float (&v)[8]) {               // columns c .. c + 7 of this thread
        const int n = tn * 128 + col0 + c;
        const long long o0 = static_cast<long long>(t) * a.ldo + n;
        if (!t_ok) return;
        if (aligned && n + 8 <= a.N) {
          if (a.out_fp32) {
            float* o = reinterpret_cast<float*>(a.out) + o0;
            *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
          } else {
            uint4 ov;
            __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
            for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + o0) = ov;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (n + i < a.N) {
              if (a.out_fp32) reinterpret_cast<float*>(a.out)[o0 + i] = v[i];
              else reinterpret_cast<__nv_bfloat16*>(a.out)[o0 + i] = __float2bfloat16(v[i]);
            }
          }
        }
      };
      auto take8 = [&](int c, float (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 8; i += 2) unpack2(acc[(c + i) / 2], v[i], v[i + 1]);
      };
      if constexpr (S == 1) {
        if (ok) {
#pragma unroll
          for (int c = 0; c < kCols; c += 8) {
            float v[8];
            take8(c, v);
            store8(c, v);
          }
        }
      } else {
        constexpr int kShare = kCols / S;
        static_assert(kShare % 8 == 0, "columns of a CTA");
        const uint32_t line = smem_u32(smem) + e * 512 + lane * 16;                     // [sender][column / 4][thread] of 16 bytes
        cluster_sync_all();                                                             // every CTA is done with its ring
#pragma unroll
        for (int j = 0; j < S; ++j) {
          if (j != rank && live) {
            const uint32_t to = peer_addr(line + (rank < j ? rank : rank - 1) * (kShare / 4 * 4096), j);
#pragma unroll
            for (int c = 0; c < kShare; c += 8) {
              float v[8];
              take8(j * kShare + c, v);
#pragma unroll
              for (int i = 0; i < 8; i += 4)
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
                             ::"r"(to + (c + i) / 4 * 4096), "f"(v[i]), "f"(v[i + 1]), "f"(v[i + 2]), "f"(v[i + 3]) : "memory");
            }
          }
        }
        cluster_sync_all();                                                             // all sums have arrived
#pragma unroll
        for (int own = 0; own < S; ++own) {
          if (own == rank && live && ok) {
#pragma unroll
            for (int c = 0; c < kShare; c += 8) {
              float v[8], mine[8];
              take8(own * kShare + c, mine);
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = 0.f;
#pragma unroll
              for (int j = 0; j < S; ++j) {
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                  float4 x = make_float4(mine[i], mine[i + 1], mine[i + 2], mine[i + 3]);
                  if (j != own)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                                 : "r"(line + (j < own ? j : j - 1) * (kShare / 4 * 4096) + (c + i) / 4 * 4096));
                  v[i] += x.x; v[i + 1] += x.y; v[i + 2] += x.z; v[i + 3] += x.w;
                }
              }
              store8(own * kShare + c, v);
            }
          }
        }
      }
    }
  }
  if (S > 1 && warp < 2) {
    // the CTAs of a cluster meet twice (one tile each)
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------
// fp8, a pair of CTAs on 256 tokens x 256 weight rows: each holds 128 tokens and half of the weight rows of a K block, one product of
// the pair reads both halves (cta_group::2), and each CTA's accumulators are its own tokens x all 256 weight rows.
//
// What bounds it: the single CTAs above fetch 32 KB of operands per 128 x 128 x 128 products, 2.1 GB for 4096 x 4096 x 8192, near the
// 12 TB/s that L2 gives; a pair fetches the same 32 KB per CTA for twice the products (512 tensor-core cycles).  Each epilogue warp
// adds 128 columns to its fp32 sums in that time, 360 cycles and as much again for hand-overs; packed multiply-adds took 760.  Large
// products meet the power limit first.
// ---------------------------------------------------------------------------------
constexpr int kPairStages = 6, kPairStageBytes = 2 * 128 * 128;
constexpr int kPairThreads = 384;      // four warps that issue, eight that add up; registers follow (of 384 x 168: 128 x 40 + 256 x 232)

struct alignas(8) PairBars {
  uint64_t full[6], empty[6], tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
};

// Copy into this CTA's shared memory whose bytes count on a barrier of the pair's first CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void mma_pair_f8(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], a, b, %4, p;\n\t}"
      ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(acc), "r"(lead)
      : "memory");
}
// The barrier at this offset in both CTAs of the pair counts one arrival when the products issued so far are done.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t.reg .b16 both;\n\tsetp.ne.b32 q, %1, 0;\n\tmov.b16 both, 3;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], both;\n\t}"
      ::"r"(smem_u32(bar)), "r"(lead) : "memory");
}
// (What these arrivals order is reads of tensor memory, which the fence in front of them covers; with cluster-wide release they waited
// for the scales in flight, 1300 cycles a K block.)
__device__ __forceinline__ void mbar_arrive_at(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
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

__global__ void __launch_bounds__(kPairThreads, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Fp8Args a) {
  constexpr int kCols = 128;                             // weight rows of an epilogue warp
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  PairBars* bars = reinterpret_cast<PairBars*>(smem + kPairStages * kPairStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1u;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPairStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], 16);             // epilogue warps of both CTAs
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                    // the other CTA's barriers are ready
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();
  pdl_trigger();
  const int units = a.tiles_t * a.tiles_n;
  const int u_first = blockIdx.x >> 1, u_step = gridDim.x >> 1;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
      // ------------------------------ TMA producer: this CTA's tokens and half of the weight rows ------------------------------
      if (lane == 0) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int u = u_first; u < units && ok; u += u_step) {
          const int tt = u % a.tiles_t, tn = u / a.tiles_t;
          for (int kb = 0; kb < a.k_blocks; ++kb) {
            if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 100 + stage)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(&bars->full[stage], 2 * kPairStageBytes);
            const uint32_t st = smem_u32(smem + stage * kPairStageBytes), full = peer_addr(smem_u32(&bars->full[stage]), 0);
            tma_load_2d_pair(st, &tmX, full, kb * 128, tt * 256 + rank * 128);
            tma_load_2d_pair(st + 128 * 128, &tmW, full, kb * 128, tn * 256 + rank * 128);
            if (++stage == kPairStages) { stage = 0; phase ^= 1; }
          }
        }
      }
    } else if (warp == 1 && rank == 0) {
      // ------------------------------ MMA issuer (first CTA) --------------------------------
      const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0), s_lo = desc_lo(smem_u32(smem));
      constexpr uint32_t kIdesc = umma_idesc(0u, 0u, 256, 256);
      const long long total = units > u_first ? ((units - 1 - u_first) / u_step + 1LL) * a.k_blocks : 0;
      int stage = 0, ab = 0;
      uint32_t phase = 0, aphase = 0;
      for (long long i = 0; i < total; ++i) {
        if (!mbar_wait(&bars->full[stage], phase, a.status, 300 + stage) || !mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 200 + ab)) break;
        tc_fence_after();
        const uint32_t st = s_lo + stage * (kPairStageBytes >> 4), d = tm + ab * 256;
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_pair_f8(d, st + 2 * k, st + 1024 + 2 * k, kIdesc, k > 0 ? 1u : 0u, lead);
        mma_commit_pair(&bars->tmem_full[ab], lead);
        mma_commit_pair(&bars->empty[stage], lead);
        if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        if (++ab == 2) { ab = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    // ------------------------------ epilogue: a thread owns one token and kCols weight rows -----------------------------------
    const int q = warp & 3, col0 = ((warp - 4) >> 2) * kCols;
    const uint32_t tile = tmem_base + col0 + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t empty0 = peer_addr(smem_u32(&bars->tmem_empty[0]), 0);
    int ab = 0;
    uint32_t aphase = 0;
    bool ok = true, ready = false;
    for (int u = u_first; u < units && ok; u += u_step) {
      const int tt = u % a.tiles_t, tn = u / a.tiles_t;
      const int t0 = tt * 256 + static_cast<int>(rank) * 128 + q * 32, t = t0 + lane, n0 = tn * 256 + col0;
      const bool t_ok = t < a.T;
      const bool live = t0 < a.T && n0 < a.N;             // some lane of this warp has a token, some column a weight row
      const float* xs = a.x_scale + (t_ok ? t : 0);
      const float* ws = a.w_scale + (live ? static_cast<long long>(n0 / 128) * a.w_scale_ld : 0LL);
      constexpr int kAhead = 4;
      float sx[kAhead], sw[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int kb = min(i, a.k_blocks - 1);
        sx[i] = __ldg(xs + static_cast<long long>(kb) * a.x_scale_ld);
        sw[i] = __ldg(ws + kb);
      }
      float acc[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
      for (int kb0 = 0; kb0 < a.k_blocks && ok; kb0 += kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
          const int kb = kb0 + i;
          if (kb >= a.k_blocks || !ok) break;
          const float s = sx[i] * sw[i];
          const int next = min(kb + kAhead, a.k_blocks - 1);
          sx[i] = __ldg(xs + static_cast<long long>(next) * a.x_scale_ld);
          sw[i] = __ldg(ws + next);
          if (!__all_sync(0xffffffffu, ready)) {
            ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[ab], aphase, a.status, 400 + ab));
            if (!ok) break;
          }
          tc_fence_after();
          if (live) {
#pragma unroll
            for (int c = 0; c < kCols; c += 64) {
              uint32_t r[2][32];
              tmem_ld_32x32(tile + ab * 256 + c, r[0]);
              tmem_ld_32x32(tile + ab * 256 + c + 32, r[1]);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 64; ++j) acc[c + j] = fmaf(__uint_as_float(r[j / 32][j % 32]), s, acc[c + j]);
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_at(empty0 + ab * 8);
          if (++ab == 2) { ab = 0; aphase ^= 1; }
          ready = mbar_test(&bars->tmem_full[ab], aphase);
        }
      }
      if (ok && t_ok) {
        const bool aligned = (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 && a.ldo % (a.out_fp32 ? 4 : 8) == 0;
        if (aligned && n0 + kCols <= a.N) {
#pragma unroll
          for (int c = 0; c < kCols; c += 8) {
            const float* v = acc + c;
            const long long o0 = static_cast<long long>(t) * a.ldo + n0 + c;
            if (a.out_fp32) {
              float* o = reinterpret_cast<float*>(a.out) + o0;
              *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
              *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
            } else {
              uint4 ov;
              __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
              for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(a.out) + o0) = ov;
            }
          }
        } else {
#pragma unroll
          for (int c = 0; c < kCols; ++c) {
            if (n0 + c < a.N) {
              const long long o = static_cast<long long>(t) * a.ldo + n0 + c;
              if (a.out_fp32) reinterpret_cast<float*>(a.out)[o] = acc[c];
              else reinterpret_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16(acc[c]);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                    // nobody reads this CTA's operands or arrives at its barriers any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------------------------
// bf16, a pair of CTAs on 256 tokens x 256 weight rows (operands as in the fp8 pair): a CTA's accumulators are its 128 tokens x 256
// weight rows, half of its tensor memory, so the epilogue of a tile runs under the products of the next, and a tile that would leave
// SMs idle is shared by two CTAs without partial sums to exchange.
//
// What bounds it: 32 KB of operands per CTA and 512 tensor-core cycles, as for the wide tile above; large products meet the power limit.
// Measured, us, wide tile (with its split) / pair: 777 x 4096 x 4096: 31.5 / 27.1;  1904 x 11264 x 2048: 82 / 64;
//   4096 x 8192 x 2048: 121 / 90;  4096 x 32768 x 1536: 372 / 318;  4096 x 4096 x 2048: 82 / 72;  4096 x 4096 x 8192: 236 / 229.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ void mma_pair_f16(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t acc, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
      "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n\t}"
      ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(kDescHi), "r"(idesc), "r"(acc), "r"(lead)
      : "memory");
}

__global__ void __launch_bounds__(320, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const WideArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  PairBars* bars = reinterpret_cast<PairBars*>(smem + kPairStages * kPairStageBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1u;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kPairStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tmem_full[i], 1);
      mbar_init(&bars->tmem_empty[i], 16);             // epilogue warps of both CTAs
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                    // the other CTA's barriers are ready
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();
  pdl_trigger();
  const int units = a.tiles_t * a.tiles_n;
  const int u_first = blockIdx.x >> 1, u_step = gridDim.x >> 1;

  if (warp == 0) {
    // ------------------------------ TMA producer: this CTA's tokens and half of the weight rows ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = u_first; u < units && ok; u += u_step) {
        const int tn = u % a.tiles_n, tt = u / a.tiles_n;
        const int gx = a.group_tiles ? tn / a.group_tiles * a.group_k : 0;
        for (int kb = 0; kb < a.k_blocks; ++kb) {
          if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 100 + stage)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&bars->full[stage], 2 * kPairStageBytes);
          const uint32_t st = smem_u32(smem + stage * kPairStageBytes), full = peer_addr(smem_u32(&bars->full[stage]), 0);
          tma_load_2d_pair(st, &tmX, full, kb * 64 + gx, tt * 256 + rank * 128);
          tma_load_2d_pair(st + 128 * 128, &tmW, full, kb * 64, tn * 256 + rank * 128);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (first CTA) --------------------------------
    if (rank == 0) {
      const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0), s_lo = desc_lo(smem_u32(smem));
      constexpr uint32_t kIdesc = umma_idesc(1u, 1u, 256, 256);
      int stage = 0, ab = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      for (int u = u_first; u < units && ok; u += u_step) {
        ok = mbar_wait(&bars->tmem_empty[ab], aphase ^ 1, a.status, 200 + ab);
        if (!ok) break;
        for (int kb = 0; kb < a.k_blocks; ++kb) {
          ok = mbar_wait(&bars->full[stage], phase, a.status, 300 + stage);
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = s_lo + stage * (kPairStageBytes >> 4), d = tm + ab * 256;
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_pair_f16(d, st + 2 * k, st + 1024 + 2 * k, kIdesc, (kb > 0 || k > 0) ? 1u : 0u, lead);
          mma_commit_pair(&bars->empty[stage], lead);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
        if (ok) mma_commit_pair(&bars->tmem_full[ab], lead);
        if (++ab == 2) { ab = 0; aphase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------ epilogue: a thread owns one token and half of the weight rows -----------------------------
    const int q = warp & 3, h = (warp - 2) >> 2;
    const uint32_t tile = tmem_base + h * 128 + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t empty0 = peer_addr(smem_u32(&bars->tmem_empty[0]), 0);
    const bool vec_ok = (a.ldo % (a.out_fp32 ? 4 : 8) == 0) && ((reinterpret_cast<uintptr_t>(a.out) & 15) == 0);
    int ab = 0;
    uint32_t aphase = 0;
    for (int u = u_first; u < units; u += u_step) {
      const int tn = u % a.tiles_n, tt = u / a.tiles_n;
      const int t = tt * 256 + static_cast<int>(rank) * 128 + q * 32 + lane, n0 = tn * 256 + h * 128;
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[ab], aphase, a.status, 400 + ab))) break;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < 128; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32(tile + ab * 256 + c, r);
        tmem_ld_wait();
        if (c == 96) {                                     // all of this warp's columns have been read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_at(empty0 + ab * 8);
        }
        const int n = n0 + c;
        if (t < a.T) {
          const long long o0 = static_cast<long long>(t) * a.ldo + n;
          if (vec_ok && n + 32 <= a.N) {
            if (a.out_fp32) {
              float* o = reinterpret_cast<float*>(a.out) + o0;
#pragma unroll
              for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(o + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
            } else {
              __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(a.out) + o0;
#pragma unroll
              for (int j = 0; j < 32; j += 8) {
                uint4 ov;
                __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&ov);
#pragma unroll
                for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(__uint_as_float(r[j + 2 * i]), __uint_as_float(r[j + 2 * i + 1]));
                *reinterpret_cast<uint4*>(o + j) = ov;
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (n + j < a.N) {
                if (a.out_fp32) reinterpret_cast<float*>(a.out)[o0 + j] = __uint_as_float(r[j]);
                else reinterpret_cast<__nv_bfloat16*>(a.out)[o0 + j] = __float2bfloat16(__uint_as_float(r[j]));
              }
            }
          }
        }
      }
      if (++ab == 2) { ab = 0; aphase ^= 1; }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                    // nobody reads this CTA's operands or arrives at its barriers any more
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------------------------
// bf16, up to 128 tokens under weights of few 128-row tiles: a cluster of S CTAs shares a tile, each with its part of K.  TMEM lanes are
// weight rows, columns tokens; CTA j finishes the j-th part of the tokens, to which the others bring their sums through distributed
// shared memory, added in the order of the ranks.
//
// What bounds it: at 17 MB of weights (2.6 us of memory) the fixed costs, of which the meeting in an fp32 workspace -- sums out, a
// counter, the last CTA reading them all back -- was the largest.  Measured, us, workspace splits / cluster:
//   9 tokens x 1024 x 4096: 9.5 / 4.8;  32 x 4096 x 2048: 12.1 / 6.1;  x 4096 x 8192: 20.5 / 14.1;
//   64 x 1024 x 4096: 22.4 / 6.6;  x 2048 x 4096: 19.8 / 8.8;  x 8192 x 2048: 20.6 / 10.2.
// 256 x 256 tiles / cluster: 128 x 1024 x 4096: 19.7 / 8.8;  x 2048 x 4096: 20.4 / 11.2;  x 4096 x 2048: 16.2 / 10.0;
//   x 4096 x 8192: 31.7 / 18.4.
// ---------------------------------------------------------------------------------
struct SmallArgs {
  int T, N, k_blocks;
  void* out;
  long long ldo;
  int out_fp32;
  int* status;
  int group_tiles, group_k;            // block-diagonal weights: tile / group_tiles is the block (0: one block)
};

template <int BT, int S>
struct SmallCfg {
  static constexpr int kStageBytes = 128 * 128 + BT * 128;
  static constexpr int kStages = BT == 128 ? 5 : BT == 64 ? 6 : 8;
  static constexpr int kShare = BT / S;                                 // token columns that a CTA finishes
  static constexpr int kMeetBytes = (S - 1) * kShare * 128 * 4;         // [sender][column][weight row]
  static constexpr int kSmem = kStages * kStageBytes + kMeetBytes + 256 + 1024;
  static_assert(kSmem <= 227 * 1024, "shared memory");
};

template <int BT, int S>
__global__ void __launch_bounds__(192, 1)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const SmallArgs a) {
  using Cfg = SmallCfg<BT, S>;
  constexpr int kStages = Cfg::kStages, kShare = Cfg::kShare;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_x = smem + kStages * 128 * 128;
  uint8_t* meet = smem_x + kStages * BT * 128;
  GemmBarriers* bars = reinterpret_cast<GemmBarriers*>(meet + Cfg::kMeetBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x) % S, tile = static_cast<int>(blockIdx.x) / S;
  const int per = (a.k_blocks + S - 1) / S, k_begin = min(a.k_blocks, rank * per), k_end = min(a.k_blocks, k_begin + per);
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    mbar_init(&bars->tmem_full[0], 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&bars->tmem_base, BT < 32 ? 32 : BT);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    // weights are immutable: this CTA's first tiles are on their way to L2 while the kernel before finishes
    for (int kb = k_begin; kb < min(k_end, k_begin + kStages); ++kb) tma_prefetch_2d(&tmW, kb * 64, tile * 128);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  pdl_wait();
  pdl_trigger();
  if (warp == 0) {
    if (lane == 0) {
      const int gx = a.group_tiles ? tile / a.group_tiles * a.group_k : 0;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = k_begin; kb < k_end; ++kb) {
        if (!mbar_wait(&bars->empty[stage], phase ^ 1, a.status, 100 + stage)) break;
        mbar_expect_tx(&bars->full[stage], Cfg::kStageBytes);
        tma_load_2d(smem + stage * 128 * 128, &tmW, &bars->full[stage], kb * 64, tile * 128);
        tma_load_2d(smem_x + stage * BT * 128, &tmX, &bars->full[stage], gx + kb * 64, 0);
        if (++stage == kStages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t lead = elect_one() ? 1u : 0u, tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t w_lo = desc_lo(smem_u32(smem)), x_lo = desc_lo(smem_u32(smem_x));
    constexpr uint32_t kIdesc = umma_idesc(1u, 1u, 128, BT);
    int stage = 0;
    uint32_t phase = 0;
    for (int kb = k_begin; kb < k_end; ++kb) {
      if (!mbar_wait(&bars->full[stage], phase, a.status, 300 + stage)) break;
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < 4; ++k)
        mma_ss(tm, w_lo + stage * 1024 + 2 * k, x_lo + stage * (BT * 8) + 2 * k, kIdesc, (kb > k_begin || k > 0) ? 1u : 0u, lead);
      mma_commit(&bars->empty[stage], lead);
      if (++stage == kStages) { stage = 0; phase ^= 1; }
    }
    mma_commit(&bars->tmem_full[0], lead);
    __syncwarp();
  }
  cluster_sync_all();                                      // every CTA runs: its meeting place may be written
  bool ok = true;
  const int q = warp & 3, row = q * 32 + lane;
  uint32_t r[BT];
  if (warp >= 2) {
    ok = __all_sync(0xffffffffu, mbar_wait(&bars->tmem_full[0], 0, a.status, 400));
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < BT; c += 16) {
      uint32_t t16[16];
      tmem_ld_32x16(tmem_base + c + (static_cast<uint32_t>(q * 32) << 16), t16);
#pragma unroll
      for (int i = 0; i < 16; ++i) r[c + i] = t16[i];
    }
    tmem_ld_wait();
    if (k_begin < k_end) {
#pragma unroll
      for (int j = 0; j < S; ++j) {
        if (j != rank) {
          const uint32_t to = peer_addr(smem_u32(meet) + ((rank < j ? rank : rank - 1) * kShare * 128 + row) * 4, j);
#pragma unroll
          for (int c = 0; c < kShare; ++c) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(to + c * 512), "r"(r[j * kShare + c]) : "memory");
        }
      }
    }
  }
  cluster_sync_all();                                      // all sums have arrived
  if (warp >= 2 && ok) {
    const int n = tile * 128 + row;
    float v[kShare];
#pragma unroll
    for (int c = 0; c < kShare; ++c) v[c] = 0.f;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      if (j * per >= a.k_blocks) continue;                 // a part of K without blocks
      if (j == rank) {
#pragma unroll
        for (int o = 0; o < S; ++o)
          if (o == rank) {
#pragma unroll
            for (int c = 0; c < kShare; ++c) v[c] += __uint_as_float(r[o * kShare + c]);
          }
      } else {
        const float* from = reinterpret_cast<const float*>(meet) + (j < rank ? j : j - 1) * kShare * 128 + row;
#pragma unroll
        for (int c = 0; c < kShare; ++c) v[c] += from[c * 128];
      }
    }
    if (n < a.N) {
#pragma unroll
      for (int c = 0; c < kShare; ++c) {
        const int t = rank * kShare + c;
        if (t < a.T) {
          const long long o = static_cast<long long>(t) * a.ldo + n;
          if (a.out_fp32) reinterpret_cast<float*>(a.out)[o] = v[c];
          else reinterpret_cast<__nv_bfloat16*>(a.out)[o] = __float2bfloat16(v[c]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BT < 32 ? 32 : BT);
  }
}

// ---------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  }
  return fn;
}

// 2-D row-major [rows, cols] tensor with `ld` elements between rows; box = [box_rows, 128 bytes].
int make_tmap_2d(CUtensorMap* tm, const void* base, int elem_bytes, long long rows, long long cols, long long ld,
                 int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return -1;
  CUtensorMapDataType dt = elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                         : elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                           : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * elem_bytes};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem_bytes), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(tm, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Paged uint8 tensor [pages][rows_per_page][128 B] with `page_stride` bytes between pages; box = one page's rows.
int make_tmap_pages(CUtensorMap* tm, const void* base, long long pages, int rows_per_page, long long page_stride) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return -1;
  cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(rows_per_page), static_cast<cuuint64_t>(pages)};
  cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(page_stride)};
  cuuint32_t box[3] = {128, static_cast<cuuint32_t>(rows_per_page), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// Clusters of `cluster` CTAs, with the programmatic-serialization attribute where `launch_pdl` would use it
template <typename... KArgs, typename... Args>
static int launch_cluster(void (*kernel)(KArgs...), int cluster, int grid, int threads, int smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_use(st, STK_PDL_CLASS) ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...) == cudaSuccess ? 0 : -4;
}

template <int BT, bool kFp8>
static int launch_gemm(const CUtensorMap& tw, const CUtensorMap& tx, const GemmArgs& a, int grid, cudaStream_t st) {
  using Cfg = GemmCfg<BT>;
  const int smem = Cfg::kStages * Cfg::kStageBytes + 256 + Cfg::kArTileBytes + 1024;
  static_assert(sizeof(GemmBarriers) <= 256, "barrier block");
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_kernel<BT, kFp8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return -3;
    configured = true;
  }
  if (a.ar_enabled || a.gate_enabled) {
    gemm_kernel<BT, kFp8><<<grid, kFp8 ? 320 : 192, smem, st>>>(tw, tx, a);      // waits on peers: plain launch
  } else {
    launch_pdl(gemm_kernel<BT, kFp8>, dim3(grid), dim3(kFp8 ? 320 : 192), smem, st, tw, tx, a);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

template <int S>
static int launch_fp8_tokens(const CUtensorMap& tx, const CUtensorMap& tw, const Fp8Args& a, int sm_count, cudaStream_t st) {
  constexpr int smem = kFp8Stages * kFp8StageBytes + static_cast<int>(sizeof(Fp8Bars)) + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_fp8_tokens_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
    configured = true;
  }
  const int units = a.tiles_t * a.tiles_n;
  return launch_cluster(gemm_fp8_tokens_kernel<S>, S, S > 1 ? units * S : units < sm_count ? units : sm_count, kFp8Threads, smem, st, tx, tw, a);
}

static int launch_fp8_pair(const CUtensorMap& tx, const CUtensorMap& tw, const Fp8Args& a, int sm_count, cudaStream_t st) {
  constexpr int smem = kPairStages * kPairStageBytes + static_cast<int>(sizeof(PairBars)) + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_fp8_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
    configured = true;
  }
  const int units = a.tiles_t * a.tiles_n, pairs = sm_count / 2;
  return launch_cluster(gemm_fp8_pair_kernel, 2, 2 * (units < pairs ? units : pairs), kPairThreads, smem, st, tx, tw, a);
}

}  // namespace stk

using namespace stk;

STK_API int stk_gemm_pick_bt(int T, int is_fp8) {
  const int cap = is_fp8 ? 128 : 256;
  int bt = 16;
  while (bt < T && bt < cap) bt *= 2;
  return bt;
}

// Suggested split-K factor so that a skinny problem still fills the SMs (through the fp32 workspace of the 128-row tiles).
STK_API int stk_gemm_pick_splits(int T, int N, int K, int is_fp8, int sm_count) {
  const int bt = stk_gemm_pick_bt(T, is_fp8);
  const int tiles = ((N + 127) / 128) * ((T + bt - 1) / bt);
  const int kb = (K * (is_fp8 ? 1 : 2) + 127) / 128;
  if (tiles >= sm_count || T > 128) return 1;
  int s = sm_count / tiles;
  if (s > kb / 4) s = kb / 4;      // keep at least four K blocks per split
  if (s > 16) s = 16;
  return s < 1 ? 1 : s;
}

STK_API long long stk_gemm_workspace_bytes(int T, int N, int splits) {
  return splits > 1 ? static_cast<long long>(splits) * T * N * 4 : 0;
}

// CTAs that share a 256 x 256 tile of a token-major kernel: four with a part of K each where that keeps the SMs to one round (with at
// least four K blocks each), else a pair (1 and 2 here); or 0 up to 64 tokens, where a tile would be mostly padding.  Up to 128 tokens
// clusters on 128-row tiles come first where those leave SMs idle (small_split_of).  A call that asks for workspace splits keeps the
// kernel above.  Measured, us, kernel above with the split that it would ask for / these:
//   80 tokens x 32768 x 1536: 66 / 24;  777 x 4096 x 4096: 66 / 27;  1500 x 4096 x 4096: 113 / 47.
static int wide_split_of(int T, int N, int K, int sm_count) {
  if (T <= 64) return 0;
  const int units = ((T + 255) / 256) * ((N + 255) / 256), kb = (K * 2 + 127) / 128;
  int s = 4;
  while (s > 1 && (units * s > sm_count || kb < 4 * s)) s /= 2;
  return s;
}

static int launch_wide(const CUtensorMap& tx, const CUtensorMap& tw, const WideArgs& a, cudaStream_t st) {
  constexpr int smem = kWideStages * kWideStageBytes + 256 + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
    configured = true;
  }
  return launch_cluster(gemm_wide_kernel, 4, a.tiles_n * a.tiles_t * 4, 320, smem, st, tw, tx, a);
}

template <int BT, int S>
static int launch_small_s(const CUtensorMap& tw, const CUtensorMap& tx, const SmallArgs& a, int tiles, cudaStream_t st) {
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_small_kernel<BT, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmallCfg<BT, S>::kSmem) != cudaSuccess) return -3;
    configured = true;
  }
  return launch_cluster(gemm_small_kernel<BT, S>, S, tiles * S, 192, SmallCfg<BT, S>::kSmem, st, tw, tx, a);
}
template <int BT>
static int launch_small(const CUtensorMap& tw, const CUtensorMap& tx, const SmallArgs& a, int split, int tiles, cudaStream_t st) {
  if (split == 8) return launch_small_s<BT, 8>(tw, tx, a, tiles, st);
  if (split == 4) return launch_small_s<BT, 4>(tw, tx, a, tiles, st);
  return launch_small_s<BT, 2>(tw, tx, a, tiles, st);
}

static int launch_pair(const CUtensorMap& tx, const CUtensorMap& tw, const WideArgs& a, int sm_count, cudaStream_t st) {
  constexpr int smem = kPairStages * kPairStageBytes + static_cast<int>(sizeof(PairBars)) + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -3;
    configured = true;
  }
  const int units = a.tiles_n * a.tiles_t, pairs = sm_count >= 2 ? sm_count / 2 : 1;
  return launch_cluster(gemm_pair_kernel, 2, 2 * (units < pairs ? units : pairs), 320, smem, st, tx, tw, a);
}

// STK_GEMM_WIDE=0 keeps large bf16 problems on the 128 x 256 tile (A/B runs)
static bool gemm_wide_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("STK_GEMM_WIDE");
    v = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

// CTAs that share a tile of the fp8 token-major kernel (as many as keep the SMs to one round, with at least four K blocks each), or 0
// where the kernel above is better: few tokens under a weight whose tiles fill the SMs.  Measured, us, kernel above / this one:
//   64 tokens x 4096 x 8192: 18.9 / 11.5;  x 2048 x 4096: 14.2 / 7.7;  x 40960 x 1536: 32.7 / 20.2;  x 129280 x 4096: 143 / 101;
//   12 tokens x 4096 x 8192: 13.9 / 11.8;  x 129280 x 4096: 106 / 137.
static int fp8_tokens_split(int T, int N, int K, int sm_count) {
  if (T <= 8) return 0;
  const int units = ((N + 127) / 128) * ((T + 127) / 128), kb = (K + 127) / 128;
  int s = 4;
  while (s > 1 && (units * s > sm_count || kb < 4 * s)) s /= 2;
  return s > 1 || T >= 48 ? s : 0;
}

// Whether pairs of CTAs take a product that the single CTAs above would take without splitting K.  A round of pairs does the work of two
// rounds of single CTAs in 1.62 to 1.92 times the time of one, so they are taken where they need no more than half the rounds.
// Measured, us, single / pair (rounds): 512 tokens x 16384 x 4096: 59 / 50 (4 / 2);  3000 x 4096 x 4096: 84 / 70 (6 / 3);
//   4096 x 1024 x 8192: 55 / 46 (2 / 1);  4096 x 40960 x 1536: 456 / 424 (70 / 35);  1500 x 4096 x 8192: 79 / 86 (3 / 2);
//   4096 x 4096 x 8192: 176 / 192 (7 / 4): at K = 8192 both run into the power limit (single CTAs: 1.66 to 1.70 GHz
//   sampled at 1000 W).
static bool fp8_pair_serves(int T, int N, int sm_count) {
  const int pairs = sm_count / 2;
  if (pairs < 1) return false;
  const long long single = (static_cast<long long>((T + 127) / 128) * ((N + 127) / 128) + sm_count - 1) / sm_count;
  const long long paired = (static_cast<long long>((T + 255) / 256) * ((N + 255) / 256) + pairs - 1) / pairs;
  return 2 * paired <= single;
}

// CTAs that share a 128-row tile of up to 128 tokens (as many as keep the SMs to one round, with at least four K blocks each), or 1: no
// split, the persistent kernel above.  Clusters of eight only where they ask for half of the SMs: sixteen of them do not run at once
// (2048 x 4096, 9 tokens: 9.6 us against 4.8 for eight of them on 1024 x 4096).
static int small_split_of(int T, int N, int K, int sm_count) {
  if (T > 128) return 1;
  const int tiles = (N + 127) / 128, kb = (K * 2 + 127) / 128;
  int s = tiles * 16 <= sm_count ? 8 : 4;
  while (s > 1 && (tiles * s > sm_count || kb < 4 * s)) s /= 2;
  return s;
}

// The kernel of a plain product (no fused collective, no workspace splits) and the CTAs that share a tile of it
enum GemmKind { kGemmTiles, kGemmFp8Tokens, kGemmFp8Pair, kGemmSmall, kGemmWide, kGemmPair };
struct GemmPlan { int kind, ctas; };
static GemmPlan gemm_plan(int T, int N, int K, int groups, int is_fp8, int sm_count) {
  if (is_fp8) {
    const int s = groups == 1 ? fp8_tokens_split(T, N, K, sm_count) : 0;
    if (s == 1 && fp8_pair_serves(T, N, sm_count)) return {kGemmFp8Pair, 2};
    return s > 0 ? GemmPlan{kGemmFp8Tokens, s} : GemmPlan{kGemmTiles, 1};
  }
  if (!gemm_wide_enabled()) return {kGemmTiles, 1};
  // block-diagonal weights take clusters and wide tiles where blocks are whole tiles and whole 128-byte steps of K
  const int small = groups == 1 || (N % (128 * groups) == 0 && K % 64 == 0) ? small_split_of(T, N, K, sm_count) : 1;
  if (small > 1) return {kGemmSmall, small};
  const int wide = groups == 1 || (N % (256 * groups) == 0 && K % 64 == 0) ? wide_split_of(T, N, K, sm_count) : 0;
  return wide == 4 ? GemmPlan{kGemmWide, 4} : wide > 0 ? GemmPlan{kGemmPair, 2} : GemmPlan{kGemmTiles, 1};
}
// 16 x kind + CTAs
STK_API int stk_gemm_plan(int T, int N, int K, int groups, int is_fp8, int sm_count) {
  const GemmPlan p = gemm_plan(T, N, K, groups < 1 ? 1 : groups, is_fp8, sm_count);
  return 16 * p.kind + p.ctas;
}

// Whether a plain product does without workspace splits (not 0: it leaves the 128-row tiles of one CTA each).  Which kernel takes it is
// gemm_plan's answer; this one does not look at small clusters from 65 tokens on, where the wide tiles serve as well.
STK_API int stk_gemm_token_tile_ctas(int T, int N, int K, int is_fp8, int sm_count) {
  if (is_fp8) return fp8_tokens_split(T, N, K, sm_count);
  if (!gemm_wide_enabled()) return 0;
  const int small = T <= 64 ? small_split_of(T, N, K, sm_count) : 1;
  return small > 1 ? small : wide_split_of(T, N, K, sm_count);
}

static int gemm_launch(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N,
                       int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld, const float* x_scale,
                       int x_scale_ld, int splits, float* workspace, int* counters, int* status, int sm_count,
                       int groups, const void* ar_ctx, const void* gate_ctx, int gate_rows, void* stream, int bt_override = 0) {
  if (T <= 0 || N <= 0 || K <= 0) return 0;
  const int es = is_fp8 ? 1 : 2;
  if ((ldw * es) % 16 || (ldx * es) % 16 || (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(X) & 15))
    return -10;
  if (is_fp8 && (w_scale == nullptr || x_scale == nullptr || (x_scale_ld & 3))) return -11;
  if (splits > 1 && (workspace == nullptr || counters == nullptr)) return -12;
  if (groups < 1) groups = 1;
  // an explicit split goes through the workspace
  const bool plain = splits <= 1 && ar_ctx == nullptr && gate_ctx == nullptr && (is_fp8 || bt_override == 0);
  const GemmPlan plan = plain ? gemm_plan(T, N, K, groups, is_fp8, sm_count) : GemmPlan{kGemmTiles, 1};
  if (plan.kind == kGemmFp8Tokens || plan.kind == kGemmFp8Pair) {
    CUtensorMap ta, tb;
    if (make_tmap_2d(&ta, X, 1, T, K, ldx, 128) != 0) return -13;        // lanes: tokens
    if (make_tmap_2d(&tb, W, 1, N, K, ldw, 128) != 0) return -14;        // columns: weight rows
    Fp8Args a;
    memset(&a, 0, sizeof(a));
    a.T = T; a.N = N;
    a.k_blocks = (K + 127) / 128;
    a.tiles_n = (N + 127) / 128;
    a.out = out; a.ldo = ldo; a.out_fp32 = out_fp32;
    a.w_scale = w_scale; a.w_scale_ld = w_scale_ld;
    a.x_scale = x_scale; a.x_scale_ld = x_scale_ld;
    a.status = status;
    a.tiles_t = (T + 127) / 128;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (plan.kind == kGemmFp8Pair) {
      a.tiles_t = (T + 255) / 256;
      a.tiles_n = (N + 255) / 256;
      return launch_fp8_pair(ta, tb, a, sm_count, st);
    }
    switch (plan.ctas) {
      case 4: return launch_fp8_tokens<4>(ta, tb, a, sm_count, st);
      case 2: return launch_fp8_tokens<2>(ta, tb, a, sm_count, st);
      default: return launch_fp8_tokens<1>(ta, tb, a, sm_count, st);
    }
  }
  if (plan.kind == kGemmSmall) {
    const int tiles = (N + 127) / 128, columns = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : 128;
    CUtensorMap tw3, tx3;
    if (make_tmap_2d(&tw3, W, 2, N, K, ldw, 128) != 0) return -13;
    if (make_tmap_2d(&tx3, X, 2, T, static_cast<long long>(K) * groups, ldx, columns) != 0) return -14;
    SmallArgs sa;
    sa.T = T; sa.N = N;
    sa.k_blocks = (K * 2 + 127) / 128;
    sa.out = out; sa.ldo = ldo; sa.out_fp32 = out_fp32; sa.status = status;
    sa.group_tiles = groups > 1 ? N / groups / 128 : 0;
    sa.group_k = K;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (columns == 16) return launch_small<16>(tw3, tx3, sa, plan.ctas, tiles, st);
    if (columns == 32) return launch_small<32>(tw3, tx3, sa, plan.ctas, tiles, st);
    if (columns == 64) return launch_small<64>(tw3, tx3, sa, plan.ctas, tiles, st);
    return launch_small<128>(tw3, tx3, sa, plan.ctas, tiles, st);
  }
  if (plan.kind == kGemmWide || plan.kind == kGemmPair) {
    CUtensorMap tw2, tx2;
    if (make_tmap_2d(&tw2, W, 2, N, K, ldw, plan.kind == kGemmWide ? 256 : 128) != 0) return -13;                       // B operand: 256 weight rows, or a CTA's half
    if (make_tmap_2d(&tx2, X, 2, T, static_cast<long long>(K) * groups, ldx, 128) != 0) return -14;              // A operands: 128 tokens each
    WideArgs wa;
    wa.T = T; wa.N = N;
    wa.k_blocks = (K * 2 + 127) / 128;
    wa.tiles_n = (N + 255) / 256;
    wa.tiles_t = (T + 255) / 256;
    wa.out = out; wa.ldo = ldo; wa.out_fp32 = out_fp32; wa.status = status;
    wa.group_tiles = groups > 1 ? N / groups / 256 : 0;
    wa.group_k = K;
    if (plan.kind == kGemmWide) return launch_wide(tx2, tw2, wa, reinterpret_cast<cudaStream_t>(stream));
    return launch_pair(tx2, tw2, wa, sm_count, reinterpret_cast<cudaStream_t>(stream));
  }
  int bt = stk_gemm_pick_bt(T, is_fp8);
  if (!is_fp8 && T > 128 && groups == 1) {
    // bf16 products that the wide tiles do not take (those fused with a collective): split-K through the fp32 workspace costs more
    // than it gains above 128 tokens (measured), so parallelism comes from narrower token tiles until about 0.7 x the SMs have one
    const int wt = (N + 127) / 128;
    while (bt > 64 && wt * ((T + bt - 1) / bt) * 10 < sm_count * 7) bt /= 2;
  }
  if (bt_override == 16 || bt_override == 32 || bt_override == 64 || bt_override == 128) bt = bt_override;
  CUtensorMap tw, tx;
  if (make_tmap_2d(&tw, W, es, N, K, ldw, 128) != 0) return -13;
  if (groups > 1 && ((K * es) % 128 || N % (128 * groups))) return -17;   // groups must split on tile boundaries
  if (make_tmap_2d(&tx, X, es, T, static_cast<long long>(K) * groups, ldx, bt) != 0) return -14;
  GemmArgs a;
  a.T = T; a.N = N;
  a.k_blocks = (K * es + 127) / 128;
  a.splits = splits < 1 ? 1 : splits;
  if (a.splits > a.k_blocks) a.splits = a.k_blocks;
  {  // no split may own an empty K range: its accumulator would never be written
    const int per = (a.k_blocks + a.splits - 1) / a.splits;
    a.splits = (a.k_blocks + per - 1) / per;
  }
  a.tiles_n = (N + 127) / 128;
  a.tiles_t = (T + bt - 1) / bt;
  a.out = out; a.ldo = ldo; a.out_fp32 = out_fp32;
  a.w_scale = w_scale; a.w_scale_ld = w_scale_ld;
  a.x_scale = x_scale; a.x_scale_ld = x_scale_ld;
  a.workspace = workspace; a.counters = counters; a.status = status;
  a.group_tiles = groups > 1 ? (N / groups) / 128 : 0;
  a.group_k_elems = K;
  {
    const uintptr_t o = reinterpret_cast<uintptr_t>(out);
    a.out_vec_ok = out_fp32 ? ((o & 15) == 0 && (ldo & 3) == 0) : ((o & 3) == 0 && (ldo & 1) == 0);
  }
  a.ar_enabled = 0;
  memset(&a.ar, 0, sizeof(a.ar));
  if (ar_ctx != nullptr) {
    memcpy(&a.ar, ar_ctx, sizeof(a.ar));
    if (static_cast<long long>(T) * N * 2 > a.ar.gemm_bytes || ldo % 8 || N % 128 || bt > 128 ||
        (reinterpret_cast<uintptr_t>(out) & 15))
      return -18;
    a.ar_enabled = 1;
  }
  a.gate_enabled = 0;
  a.gate_rows = 0;
  if (gate_ctx != nullptr) {
    if (ar_ctx != nullptr || gate_rows <= 0 || a.splits != 1) return -19;
    memcpy(&a.ar, gate_ctx, sizeof(a.ar));
    a.gate_enabled = 1;
    a.gate_rows = gate_rows;
  }
  const int units = a.splits * a.tiles_n * a.tiles_t;
  const int grid = units < sm_count ? units : sm_count;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
#define STK_LAUNCH(BT_) (is_fp8 ? launch_gemm<BT_, true>(tw, tx, a, grid, st) : launch_gemm<BT_, false>(tw, tx, a, grid, st))
  switch (bt) {
    case 16: return STK_LAUNCH(16);
    case 32: return STK_LAUNCH(32);
    case 64: return STK_LAUNCH(64);
    case 128: return STK_LAUNCH(128);
    case 256: return is_fp8 ? -15 : launch_gemm<256, false>(tw, tx, a, grid, st);
  }
#undef STK_LAUNCH
  return -16;
}

STK_API int stk_gemm(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N,
                     int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld, const float* x_scale,
                     int x_scale_ld, int splits, float* workspace, int* counters, int* status, int sm_count,
                     int groups, const void* ar_ctx, void* stream) {
  return gemm_launch(W, ldw, X, ldx, out, ldo, T, N, K, is_fp8, out_fp32, w_scale, w_scale_ld, x_scale, x_scale_ld, splits,
                     workspace, counters, status, sm_count, groups, ar_ctx, nullptr, 0, stream);
}

// Plain GEMM with an explicit token-tile width (16/32/64/128): narrow weights with many tokens get their parallelism
// from token tiles instead of split-K (e.g. the 24-row hyper-connection mix projection over [T, 16384]).
STK_API int stk_gemm_tile(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T, int N,
                          int K, int out_fp32, int bt, int splits, float* workspace, int* counters, int* status,
                          int sm_count, void* stream) {
  return gemm_launch(W, ldw, X, ldx, out, ldo, T, N, K, 0, out_fp32, nullptr, 0, nullptr, 0, splits < 1 ? 1 : splits,
                     workspace, counters, status, sm_count, 1, nullptr, nullptr, 0, stream, bt);
}

// All-gather -> GEMM: X is the gathered [T, K] matrix inside this rank's symmetric region (filled by
// stk_symm_ag_push on every rank, `gate_rows` rows per source rank); tiles wait only for the shards they read.
STK_API int stk_gemm_gated(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo, int T,
                           int N, int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld,
                           const float* x_scale, int x_scale_ld, int* status, int sm_count, const void* gate_ctx,
                           int gate_rows, void* stream) {
  return gemm_launch(W, ldw, X, ldx, out, ldo, T, N, K, is_fp8, out_fp32, w_scale, w_scale_ld, x_scale, x_scale_ld, 1,
                     nullptr, nullptr, status, sm_count, 1, nullptr, gate_ctx, gate_rows, stream);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free entry point (declared in stk_no_alloc.h).
// ---------------------------------------------------------------------------------------------
namespace {
constexpr long long kNoAllocWorkspaceBytes = 8ll << 20;      // split-K partials: splits * T * N * 4 bytes
constexpr int kNoAllocCounters = 4096;                        // one per output tile
constexpr long long kNoAllocBytes = kNoAllocWorkspaceBytes + kNoAllocCounters * 4;
// Lives in every context that loads the library until the process exits.  Zero-initialised by the
// loader; the GEMM leaves its tile counters at zero when it finishes.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];
constexpr int kMaxDevices = 64;
static void* g_noalloc_ptr[kMaxDevices] = {};
}  // namespace

STK_API long long stk_gemm_noalloc_max_workspace_bytes() { return kNoAllocWorkspaceBytes; }

static int noalloc_resolve(unsigned char** base) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return -30;
  if (g_noalloc_ptr[dev] == nullptr) {
    // First call on this device: resolve the device address of the static array.  In host code the
    // array's name is only a handle for this query, never a pointer a kernel may be given.
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) return -31;
    g_noalloc_ptr[dev] = p;
  }
  *base = static_cast<unsigned char*>(g_noalloc_ptr[dev]);
  return 0;
}

// Zeroes the built-in tile counters on `stream` (a memset node, no allocation).  Needed only after a call whose
// status word came back non-zero: a split that gave up a wait never counted itself in, so its tile's counter is
// left between 1 and splits-1 and the next split-K call on that tile would reduce too early.
STK_API int stk_gemm_noalloc_reset(void* stream) {
  unsigned char* base = nullptr;
  const int rc = noalloc_resolve(&base);
  if (rc != 0) return rc;
  return cudaMemsetAsync(base + kNoAllocWorkspaceBytes, 0, kNoAllocCounters * 4, reinterpret_cast<cudaStream_t>(stream)) ==
                 cudaSuccess ? 0 : -34;
}

STK_API int stk_gemm_noalloc(const void* W, long long ldw, const void* X, long long ldx, void* out, long long ldo,
                             int T, int N, int K, int is_fp8, int out_fp32, const float* w_scale, int w_scale_ld,
                             const float* x_scale, int x_scale_ld, int splits, int* status, int sm_count, void* stream) {
  unsigned char* base = nullptr;
  const int rc = noalloc_resolve(&base);
  if (rc != 0) return rc;
  if (splits < 1) splits = 1;
  const int bt = stk_gemm_pick_bt(T, is_fp8);
  const long long tiles = static_cast<long long>((N + 127) / 128) * ((T + bt - 1) / bt);
  if (splits > 1) {
    if (static_cast<long long>(splits) * T * N * 4 > kNoAllocWorkspaceBytes) return -32;   // beyond the built-in scratch
    if (tiles > kNoAllocCounters) return -33;
  }
  float* workspace = reinterpret_cast<float*>(base);
  int* counters = reinterpret_cast<int*>(base + kNoAllocWorkspaceBytes);
  return stk_gemm(W, ldw, X, ldx, out, ldo, T, N, K, is_fp8, out_fp32, w_scale, w_scale_ld, x_scale, x_scale_ld, splits,
                  workspace, counters, status, sm_count, 1, nullptr, stream);
}
