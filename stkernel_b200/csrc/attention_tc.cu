// Sparse multi-head latent attention on the 5th-generation tensor cores (fp8_ds_mla rows, D = 512).
//
// One CTA per SM, which walks through (query token, row split) items.  The row list (SWA window rows, then top-k compressed rows)
// is walked in blocks of 128 rows:
//
//   producer warps   gather the 584-byte rows by slot id, dequantise fp8 x UE8M0 -> fp16 and write them
//                    into shared memory as 8 panels of [128 rows x 64 dims], 128-byte swizzled
//   MMA warp         S^T[row, head] = K_block . Q^T      (K panels as the K-major A operand)
//                    O^T[dim, head] += V^T . P           (the same panels as the MN-major A operand:
//                                                         K = V = the latent row, stored once)
//   softmax warps    read S^T from TMEM (one row and half of the heads per thread), write P as the K-major B
//                    operand, rescale in TMEM the columns of O whose head's maximum moved
//
// Operands are fp16: weights keep three bits more than bf16 leaves them, and values from 2^-14 to 2^16 all of theirs.  A row, or a
// head's queries, whose largest magnitude lies outside 2^-8 .. 2^16 is divided by a power of two that brings it back (`range_shift`):
// its scores get it back, and a row's weights carry it to the values (`lift`).  What is below 2^-14 beside something large in the same
// row or head is held to 2^-25, a group of codes with a scale below 2^-24 to 2^-16: at most 2^-17 of the largest.
//
// What bounds it: the key block (128 KB in fp16) and Q (64 KB) fill shared memory, so there is one key buffer, and a block is
// scores -> softmax -> values in turn.  Everything else is taken off that chain:
//   * panels change hands one by one: scores start on the first panel that has landed, and a pair of panels goes back to the
//     producers as soon as its 128 output dims are accumulated, so the next block is written under the value products;
//   * sixteen producer warps hold the codes of the whole next block in registers, so no gather latency is on the chain (eight
//     warps with twice the rows each left the conversions waiting for their own results); a load instruction takes 64 contiguous
//     bytes of eight rows, and its two stores per lane hit every bank once;
//   * of O only the columns of the heads whose maximum moved are rescaled, one head at a time (a few of a block's 64; two at a time
//     took 2753 us, four 2894, all of them 3182), and that only in blocks where a weight would pass 2^kSlack: the others cost one
//     look at the scores and a vote.  The row sums of P stay in registers (one per head and row) and are reduced once per CTA.
// The value products read 6 KB of shared memory each and the next block's panels are written under them: 2500 cycles alone, 5600
// with the writes.  The beginning and the end of a token (queries, first gather, output) were 26000 cycles with a thread block per
// token, a block is 8200: thread blocks stay and walk through tokens, the next one's queries and first codes are fetched under this
// one's last softmax, value products and output.
// Measured (4096 tokens, 64 heads, 128 + 2048 rows): 5162 us with one thread block of thirteen warps working through
// load -> scores -> softmax -> values without overlap, 2677 with bf16 operands, exact maxima in every block and a branch per stored
// value, 2403 now, 16 of them for looking at ranges; 128 rows alone: 576 -> 281.
//
// Accumulators live in TMEM: S (NH columns) and four O^T tiles of [128 dims x NH heads].
// A CTA of a split writes an un-normalised partial (o, m, l) that `sparse_mla_combine` merges with the sink.
// Every mbarrier wait is bounded; on expiry the status word is set and the CTA drains and exits.
//
// Replaces the reference's FlashInfer sparse-MLA decode/prefill kernels
// (overlay/flashinfer_sparse.py:323-541).
#define STK_PDL_CLASS 128      // bit of this file's kernels in the PDL mask (STK_PDL, stk_set_pdl_mask)
#include "codes.cuh"
#include "common.cuh"
#include "pairs.cuh"
#include "warp_reduce.cuh"

#include <type_traits>

namespace stk {

struct MlaTcArgs {
  const __nv_bfloat16* q;      // [T, nh, 512]
  long long ldt;
  const uint8_t* swa_base; long long swa_stride;
  const uint8_t* comp_base; long long comp_stride;
  const int* swa_slots; int swa_ld; const int* swa_lens;
  const int* topk_slots; int topk_ld; const int* topk_lens;   // may be null
  float* partial;              // [T, n_splits, nh, 514]
  // Direct output (n_splits == 1 only, out != nullptr): the CTA merges the sink, normalises, applies the inverse
  // RoPE to the rope dims and writes bf16 [T, nh, 512] itself; no partial is written and no combine pass runs.
  __nv_bfloat16* out; long long ldo;
  const float* sink;           // [nh] or null
  const int64_t* positions;    // [T] or null (no inverse RoPE)
  const float* inv_freq;       // [32]
  int T, nh, n_splits, rows_per_split;
  float scale;
  int* status;
  unsigned long long* trace;   // optional [8] stage timestamps (ns) of CTA (0,0): a device-side stage trace
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define STK_TRACE(slot) do { if (a.trace && blockIdx.x == 0) a.trace[slot] = global_ns(); } while (0)

constexpr int kD = 512, kR = 64, kNope = 448, kDataBytes = 576, kPanels = 8, kRows = 128;
constexpr int kPanelBytes = kRows * 128;                 // 16 KB
constexpr int kProducerWarps = 16;

// Warpgroups: the first issues products (one warp of it), then the softmax warps, then the producers.  From 32 heads on two
// softmax warps share a lane quarter of TMEM and take half of the heads each.  Registers follow the roles: what the first
// warpgroup gives back (of 896 x 72 or 768 x 80 at launch) pays for the sums that the softmax warps hold.
template <int NH>
struct MlaCfg {
  static constexpr int kHalves = NH >= 32 ? 2 : 1;
  static constexpr int kHeads = NH / kHalves;            // heads per softmax thread
  static constexpr int kSoftmaxWarps = 4 * kHalves;
  static constexpr int kThreads = 32 * (4 + kSoftmaxWarps + kProducerWarps);
  static constexpr int kLaunchRegs = kThreads > 768 ? 72 : 80;
  static constexpr int kIssueRegs = 24, kSoftmaxRegs = kHalves == 2 ? 96 : 128, kProducerRegs = 72;
  static_assert(128 * kIssueRegs + 32 * kSoftmaxWarps * kSoftmaxRegs + 32 * kProducerWarps * kProducerRegs <= kThreads * kLaunchRegs,
                "register split");
  static constexpr int kTmemCols = (5 * NH <= 128) ? 128 : (5 * NH <= 256) ? 256 : 512;
};

constexpr int kBarBytes = 192;
constexpr int kNoRow = 1 << 20;       // `lift` of a place in the list without a row
constexpr float kSlack = 1.5f;        // powers of two by which weights may pass the maxima in use before these are taken anew
// Order in which panels are written and scored, and in which pairs of them are summed and freed: the rotated part (panel 7)
// is freed first and needed last.
__device__ __forceinline__ constexpr int panel_at(int i) { return i == 0 ? 6 : i == 7 ? 7 : i - 1; }
__device__ __forceinline__ constexpr int pair_at(int i) { return i == 0 ? 3 : i - 1; }

template <int N>
__device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

struct alignas(8) MlaBars {
  uint64_t k_full[5];              // panels 0 + 1, 2 + 3, 4 + 5, 6, 7 of the block are in shared memory
  uint64_t k_free[kPanels / 2];    // the value products of a pair of panels are done
  uint64_t s_full, p_full, pv_done, q_full;
  uint32_t tmem_base;
  uint32_t moved[2];               // heads whose maximum the last block that took maxima moved, by halves of 32
  uint32_t unset[2];               // heads that have none yet
};
static_assert(sizeof(MlaBars) <= kBarBytes, "barrier block");

// one column: 32 lanes x 32 bits
__device__ __forceinline__ void tmem_ld_32x1(uint32_t taddr, uint32_t& r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_32x1(uint32_t taddr, uint32_t r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(r) : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void put16(uint32_t smem_addr, uint32_t v) {
  asm volatile("st.shared.b16 [%0], %1;" ::"r"(smem_addr), "h"(static_cast<unsigned short>(v)) : "memory");
}

// barrier `id` of n threads; whether any of them came with `pred`
__device__ __forceinline__ bool bar_any(int id, int n, bool pred) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.or.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(id), "r"(n), "r"(pred ? 1u : 0u) : "memory");
  return r != 0;
}
__device__ __forceinline__ void named_bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// Eight bf16 values (16 bytes) times a power of two -> fp16
__device__ __forceinline__ uint4 bf16x8_to_half(const uint4& v, float f) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
  uint4 o;
  __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
  for (int i = 0; i < 4; ++i) oh[i] = __floats2half2_rn(__uint_as_float(w[i] << 16) * f, __uint_as_float(w[i] & 0xffff0000u) * f);
  return o;
}

constexpr int kMostExponent = 142, kLeastExponent = 119;      // 2^15, 2^-8
// Power of two that a row or a head is divided by, from the biased exponent of its largest magnitude: none from 2^-8 to below 2^16,
// else what brings that to 2^15 or 2^1 (a row lifted no higher than ordinary ones leaves fp16's range to their weights).  `low`: it
// holds a scale that fp16 does not, which asks for 2^1 as well.  Below 2^-98 it stays where 2^100 puts it: sums of weights times that
// have to be finite in fp32.
__device__ __forceinline__ int range_shift(int e, bool low) {
  return e > kMostExponent ? e - kMostExponent : e >= (low ? 128 : kLeastExponent) || e == 0 ? 0 : max(e - 128, -100);
}
__device__ __forceinline__ float power_of_two(int e) { return __int_as_float((127 + e) << 23); }

__device__ __forceinline__ uint32_t half2_bits(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }

// Eight bf16 values times a power of two (exact, but for what falls below bf16's own range)
__device__ __forceinline__ uint4 bf16x8_times(uint4 v, float f) {
  const __nv_bfloat162 f2 = __float2bfloat162_rn(f);
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __hmul2(h[i], f2);
  return v;
}

// Larger of the magnitudes of two words of bf16 pairs, by halves (their bits order as the magnitudes do)
__device__ __forceinline__ uint32_t bf16x2_absmax(uint32_t a, uint32_t b) { return __vmaxu2(a & 0x7fff7fffu, b & 0x7fff7fffu); }

template <int NH>
__global__ void __launch_bounds__(MlaCfg<NH>::kThreads, 1)
sparse_mla_tc_kernel(const MlaTcArgs a) {
  pdl_wait();
  pdl_trigger();
  using Cfg = MlaCfg<NH>;
  constexpr int kThreads = Cfg::kThreads, kSoftmaxWarps = Cfg::kSoftmaxWarps, kHeads = Cfg::kHeads;
  constexpr int kSoftmaxThreads = kSoftmaxWarps * 32;
  constexpr int kQBytes = kPanels * NH * 128;
  constexpr int kPBytes = 2 * NH * 128;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* k_s = smem;                                   // 8 panels x 16 KB
  uint8_t* q_s = k_s + kPanels * kPanelBytes;            // 8 panels x NH x 128 B
  uint8_t* p_s = q_s + kQBytes;                          // 2 panels x NH x 128 B
  MlaBars* bars = reinterpret_cast<MlaBars*>(p_s + kPBytes);
  float* smax = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + kBarBytes);  // [4][NH], row sums at the end
  float* m_run = smax + 4 * NH;                          // [NH] the maxima in use, in powers of two
  float* minus_m = m_run + NH;                           // [NH] their negatives (0 for none yet)
  float* alpha_s = minus_m + NH;                         // [NH]
  int* lift_s = reinterpret_cast<int*>(alpha_s + NH);    // [kRows] what the block's rows were divided by, in powers of two; kNoRow: no row
  float* q_mul = reinterpret_cast<float*>(lift_s + kRows);      // [2][NH] what the heads' queries were divided by, items in turn

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) STK_TRACE(0);
  // Items of this CTA: a token and its part of the row list.  Every role walks through those that have rows.
  const int items = a.T * a.n_splits;
  struct Item { int i, t, sp, n_swa, r_begin, r_end, n_blocks; };
  auto item_at = [&](int i) {
    Item w;
    w.i = i;
    w.sp = i / a.T;
    w.t = i - w.sp * a.T;
    w.n_swa = a.swa_lens[w.t];
    const int L = w.n_swa + (a.topk_slots ? a.topk_lens[w.t] : 0);
    w.r_begin = w.sp * a.rows_per_split;
    w.r_end = min(L, w.r_begin + a.rows_per_split);
    w.n_blocks = w.r_end > w.r_begin ? (w.r_end - w.r_begin + kRows - 1) / kRows : 0;
    return w;
  };
  auto item_from = [&](int i) {                          // the first that has rows from i on; i >= items: none left
    Item w;
    w.i = i;
    w.n_blocks = 0;
    for (; i < items; i += gridDim.x) {
      w = item_at(i);
      if (w.n_blocks > 0) return w;
    }
    w.i = i;
    return w;
  };

  if (threadIdx.x == 0) {
    for (int p = 0; p < 5; ++p) mbar_init(&bars->k_full[p], kProducerWarps);
    for (int j = 0; j < kPanels / 2; ++j) mbar_init(&bars->k_free[j], 1);
    bars->unset[0] = bars->unset[1] = 0;
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->p_full, kSoftmaxWarps);
    mbar_init(&bars->pv_done, 1);
    mbar_init(&bars->q_full, kProducerWarps);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_base, Cfg::kTmemCols);
    tmem_relinquish();
  }
  // every warp passes this once its part of the prologue is done
  auto begin = [&]() {
    fence_proxy_async();
    tc_fence_before();
    named_bar_sync(1, kThreads);
    tc_fence_after();
  };
  // Q of a token -> shared memory, K-major panels [NH x 64 dims], 128-byte swizzled; heads >= nh are zero.  `who` of kLoaders threads,
  // a warp to a head; `turn`: which of the two lists of powers of two the token's heads get.
  auto load_q = [&](int t, int who, uint32_t turn, auto loaders) {
    constexpr int kLoaders = decltype(loaders)::value, kWarps = kLoaders / 32, kMine = NH / kWarps;
    static_assert(NH % kWarps == 0, "heads of a warp");
    const int w = who >> 5, lane = who & 31;
    uint4 qv[kMine][2];
#pragma unroll
    for (int j = 0; j < kMine; ++j) {
      const int h = w + j * kWarps;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        qv[j][i] = make_uint4(0, 0, 0, 0);
        if (h < a.nh) qv[j][i] = __ldg(reinterpret_cast<const uint4*>(a.q + t * a.ldt + static_cast<long long>(h) * kD + (i * 32 + lane) * 8));
      }
    }
    // Largest magnitudes of the lane's parts.  Whether heads need a power of two is voted on; which one is asked only then (with the
    // reductions and products for all, 4096 tokens took 29 us more).
    uint32_t big[kMine], all = 0;
    bool shifted = false;
#pragma unroll
    for (int j = 0; j < kMine; ++j) {
      big[j] = __vmaxu2(__vmaxu2(bf16x2_absmax(qv[j][0].x, qv[j][0].y), bf16x2_absmax(qv[j][0].z, qv[j][0].w)),
                        __vmaxu2(bf16x2_absmax(qv[j][1].x, qv[j][1].y), bf16x2_absmax(qv[j][1].z, qv[j][1].w)));
      all = __vmaxu2(all, big[j]);
      shifted |= !__any_sync(0xffffffffu, w + j * kWarps >= a.nh || max(big[j] & 0xffffu, big[j] >> 16) >= kLeastExponent << 7);
    }
    shifted |= __any_sync(0xffffffffu, max(all & 0xffffu, all >> 16) > (kMostExponent << 7 | 127));
#pragma unroll
    for (int j = 0; j < kMine; ++j) {
      const int h = w + j * kWarps;
      int shift = 0;
      if (shifted) {
        const uint32_t most = __reduce_max_sync(0xffffffffu, max(big[j] & 0xffffu, big[j] >> 16));
        shift = range_shift(static_cast<int>(most >> 7), false);
#pragma unroll
        for (int i = 0; i < 2; ++i) qv[j][i] = bf16x8_times(qv[j][i], power_of_two(-shift));
      }
      if (lane == 0) q_mul[turn * NH + h] = power_of_two(shift);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int c8 = i * 32 + lane;
        *reinterpret_cast<uint4*>(q_s + (c8 >> 3) * (NH * 128) + h * 128 + (((c8 & 7) ^ (h & 7)) << 4)) = bf16x8_to_half(qv[j][i], 1.f);
      }
    }
  };
  if (warp < 4) {
    reg_dec<Cfg::kIssueRegs>();
    begin();
    if (threadIdx.x == 0) STK_TRACE(1);
    if (warp == 0) {
      // ------------------------------- MMA issuer -------------------------------
      const uint32_t tmem_s = bars->tmem_base, tmem_o = tmem_s + NH;
      const uint32_t lead = elect_one() ? 1u : 0u, ts = __shfl_sync(0xffffffffu, tmem_s, 0), to = __shfl_sync(0xffffffffu, tmem_o, 0);
      constexpr uint32_t kIdescQK = umma_idesc(0u, 0u, 128, NH);
      constexpr uint32_t kIdescPV = umma_idesc(0u, 0u, 128, NH) | (1u << 15);     // A is MN-major
      constexpr uint32_t kStep = kPanelBytes >> 4, kQStep = (NH * 128) >> 4;      // panels in descriptor units
      const uint32_t k_lo = desc_lo(smem_u32(k_s)), v_lo = desc_lo(smem_u32(k_s), kPanelBytes);
      const uint32_t q_lo = desc_lo(smem_u32(q_s)), p_lo = desc_lo(smem_u32(p_s));
      bool ok = true;
      uint32_t g = 0, k = 0;                                   // blocks and items before this one: phases of their barriers
      for (int at = blockIdx.x; at < items && ok; at += gridDim.x) {
      const int n_blocks = item_at(at).n_blocks;
      if (n_blocks == 0) continue;
      if (k > 0) ok = mbar_wait(&bars->q_full, (k - 1) & 1, a.status, 603);
      for (int b = 0; b < n_blocks && ok; ++b, ++g) {
        const uint32_t ph = g & 1;
#pragma unroll 1
        for (int i = 0; i < kPanels; ++i) {
          const int p = panel_at(i);
          if (i != 2 && i != 4 && i != 6) {
            ok = ok && mbar_wait(&bars->k_full[p < 6 ? p >> 1 : p - 3], ph, a.status, 600);
            if (!ok) break;
            tc_fence_after();
          }
          if (b == 0 && i == 0 && lane == 0) STK_TRACE(2);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_ss(ts, k_lo + p * kStep + 2 * k, q_lo + p * kQStep + 2 * k, kIdescQK, (i | k) != 0 ? 1u : 0u, lead);
        }
        if (!ok) break;
        mma_commit(&bars->s_full, lead);
        ok = mbar_wait(&bars->p_full, ph, a.status, 601);
        if (!ok) break;
        tc_fence_after();
        if (b == 0 && lane == 0) STK_TRACE(4);
#pragma unroll 1
        for (int i = 0; i < kPanels / 2; ++i) {
          const int j = pair_at(i);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            mma_ss(to + j * NH, v_lo + 2 * j * kStep + kk * 128, p_lo + (kk >> 2) * kQStep + 2 * (kk & 3), kIdescPV, (b > 0 || kk > 0) ? 1u : 0u, lead);
          mma_commit(&bars->k_free[j], lead);
        }
      }
      mma_commit(&bars->pv_done, lead);
      ++k;
      }
      // what was issued completes before the tensor memory goes away
      if (k > 0) mbar_wait(&bars->pv_done, (k - 1) & 1, a.status, 602);
      __syncwarp();
    }
  } else if (warp < 4 + kSoftmaxWarps) {
    // ------------------------------- softmax / epilogue -------------------------------
    if constexpr (Cfg::kSoftmaxRegs > Cfg::kLaunchRegs) reg_inc<Cfg::kSoftmaxRegs>();
    int at = blockIdx.x, n_blocks = 0;                    // this item, and its blocks
    {
      const Item e = item_from(at);
      at = e.i;
      n_blocks = e.n_blocks;
    }
    if (at < items) load_q(at % a.T, threadIdx.x - 128, 0, std::integral_constant<int, kSoftmaxThreads>{});
    begin();
    const uint32_t tmem_s = bars->tmem_base, tmem_o = tmem_s + NH;       // S^T: NH columns; O^T: 4 x NH columns
    const int q4 = warp & 3;                              // TMEM lane quarter
    const int row = q4 * 32 + lane;                       // row of the block owned by this thread
    const int h0 = ((warp - 4) >> 2) * kHeads;            // its first head
    const uint32_t lane_addr = static_cast<uint32_t>(q4 * 32) << 16;
    const float sl2 = a.scale * 1.4426950408889634f;
    const int own = threadIdx.x - 128;                   // owner thread of head `own` when < NH
    uint64_t lp[kHeads / 2];                              // sums of this row's weights, two heads each
    // this row's place in a head's line of P: the 16-byte chunk number is turned by the head's low bits
    uint32_t pdst[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      pdst[i] = smem_u32(p_s) + (row >> 6) * (NH * 128) + (h0 + i) * 128 + ((((row & 63) >> 3) ^ i) << 4) + (row & 7) * 2;
    // items without rows: only the sink takes probability mass, the output is zero
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
      const Item e = item_at(i);
      if (e.n_blocks > 0) continue;
      if (a.out != nullptr) {
        __nv_bfloat16* orow = a.out + static_cast<long long>(e.t) * a.ldo;
        for (int j = own; j < a.nh * kD; j += kSoftmaxThreads) orow[j] = __float2bfloat16(0.f);
      } else {
        float* prow = a.partial + (static_cast<long long>(e.t) * a.n_splits + e.sp) * a.nh * (kD + 2);
        for (int j = own; j < a.nh * (kD + 2); j += kSoftmaxThreads) prow[j] = j % (kD + 2) == kD ? -INFINITY : 0.f;
      }
    }
    bool ok = true;                                       // the same in every lane; barriers are passed either way
    auto scores = [&](int c, uint32_t (&r16)[16]) {       // sixteen heads' products of this row
      tmem_ld_32x16(tmem_s + lane_addr + h0 + c, r16);
      tmem_ld_wait();
    };
    uint32_t g = 0, k = 0;
    for (; at < items; ++k) {
#pragma unroll
    for (int i = 0; i < kHeads / 2; ++i) lp[i] = 0ull;
    if (own < NH) m_run[own] = -INFINITY;
    bool lifted = false;                                  // a row of this item so far has a power of two (the same in every warp)
    bool q_lifted = false;                                // a head of this warp has
    const float* const qm = q_mul + (k & 1) * NH + h0;
    for (int b = 0; b < n_blocks; ++b, ++g) {
      const uint32_t ph = g & 1;
      // (the row's power of two was left before the first panel was handed over: a barrier that has long completed)
      ok = __all_sync(0xffffffffu, ok && mbar_wait(&bars->s_full, ph, a.status, 610) && mbar_wait(&bars->k_full[3], ph, a.status, 612));
      if (b == 0 && threadIdx.x == 128) STK_TRACE(3);
      tc_fence_after();
      const int row_lift = lift_s[row];
      const bool valid = row_lift != kNoRow, has_lift = valid && row_lift != 0;
      if (b == 0) q_lifted = __any_sync(0xffffffffu, qm[lane & (kHeads - 1)] != 1.f);
      // Whether a weight would pass 2^kSlack with the maxima in use (not asked where powers of two are about)
      bool over = b == 0 || (bars->unset[0] | bars->unset[1]) != 0 || lifted || q_lifted;
      if (!over) {
        const uint64_t sl22 = pack2(sl2, sl2);
        float top = -INFINITY;
#pragma unroll
        for (int c = 0; c < kHeads; c += 16) {
          uint32_t r16[16];
          scores(c, r16);
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const ulonglong2 m4 = *reinterpret_cast<const ulonglong2*>(minus_m + h0 + c + i);
            float x, y;
            unpack2(fma2(pack2(__uint_as_float(r16[i]), __uint_as_float(r16[i + 1])), sl22, m4.x), x, y);
            top = fmaxf(top, fmaxf(x, y));
            unpack2(fma2(pack2(__uint_as_float(r16[i + 2]), __uint_as_float(r16[i + 3])), sl22, m4.y), x, y);
            top = fmaxf(top, fmaxf(x, y));
          }
        }
        over = (valid && !(top <= kSlack)) || has_lift;
      }
      if (bar_any(2, kSoftmaxThreads, over)) {
      // exact maxima of this block's rows per head, and the running ones
      {
        uint32_t raw[kHeads / 16][16];
        float s[kHeads];
#pragma unroll
        for (int c = 0; c < kHeads / 16; ++c) tmem_ld_32x16(tmem_s + lane_addr + h0 + 16 * c, raw[c]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < kHeads; ++i) s[i] = valid ? __uint_as_float(raw[i / 16][i % 16]) * sl2 : -INFINITY;
        if (q_lifted) {
#pragma unroll
          for (int i = 0; i < kHeads; i += 4) {
            const float4 q4m = *reinterpret_cast<const float4*>(qm + i);
            s[i] *= q4m.x;
            s[i + 1] *= q4m.y;
            s[i + 2] *= q4m.z;
            s[i + 3] *= q4m.w;
          }
        }
        if (has_lift) {
          const float f = power_of_two(row_lift), l = static_cast<float>(row_lift);
#pragma unroll
          for (int i = 0; i < kHeads; ++i) s[i] = fmaf(s[i], f, l);
        }
        bfly_reduce_store<kHeads, true>(s, smax + q4 * NH + h0, lane);
      }
      lifted = bar_any(2, kSoftmaxThreads, has_lift) || lifted;
      if (own < (NH < 32 ? 32 : NH)) {                     // whole warps
        bool moved = false, unset = false;
        if (own < NH) {
          const float bm = fmaxf(fmaxf(smax[own], smax[NH + own]), fmaxf(smax[2 * NH + own], smax[3 * NH + own]));
          const float mo = m_run[own], mn = fmaxf(mo, bm);
          moved = mn != mo && mo != -INFINITY;
          alpha_s[own] = moved ? exp2f(mo - mn) : 1.f;
          m_run[own] = mn;
          unset = mn == -INFINITY;
          minus_m[own] = unset ? 0.f : -mn;
        }
        const uint32_t some = __ballot_sync(0xffffffffu, moved), none = __ballot_sync(0xffffffffu, unset);
        if (lane == 0) {
          bars->moved[own >> 5] = some;
          bars->unset[own >> 5] = none;
        }
      }
      named_bar_sync(2, kSoftmaxThreads);
      // heads whose maximum moved: their sums, and their columns of O (this block's scores were issued behind the previous block's
      // value products: those are complete)
      uint32_t mask = bars->moved[h0 >> 5] >> (h0 & 31);
      if constexpr (kHeads < 32) mask &= (1u << kHeads) - 1u;
      if (mask != 0) {
#pragma unroll
        for (int i = 0; i < kHeads; i += 4) {
          const ulonglong2 f4 = *reinterpret_cast<const ulonglong2*>(alpha_s + h0 + i);
          lp[i / 2] = mul2(lp[i / 2], f4.x);
          lp[i / 2 + 1] = mul2(lp[i / 2 + 1], f4.y);
        }
        const uint32_t o_at = tmem_o + h0 + lane_addr;
        while (mask != 0) {
          const int h = __ffs(mask) - 1;
          mask &= mask - 1;
          uint32_t r[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) tmem_ld_32x1(o_at + j * NH + h, r[j]);
          const float f = alpha_s[h0 + h];
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 4; ++j) tmem_st_32x1(o_at + j * NH + h, __float_as_uint(__uint_as_float(r[j]) * f));
        }
        tmem_st_wait();
      }
      }
      // P = exp2(s - m), fp16, written as the K-major B operand [head][row].  The sums take the rounded values, unless powers of two are
      // about: these move a maximum away from the largest weight, which may then be below what fp16 holds.
      auto weights = [&](auto plain) {
        constexpr bool kPlain = decltype(plain)::value;
        const int lift = kPlain || !valid ? 0 : row_lift;
        const float sl = sl2 * power_of_two(lift), liftf = static_cast<float>(lift), back = power_of_two(-lift);
        const uint64_t sl22 = pack2(sl, sl), lift2 = pack2(liftf, liftf), back2 = pack2(back, back);
#pragma unroll
        for (int c = 0; c < kHeads; c += 16) {
          uint32_t r16[16];
          scores(c, r16);
          if (valid) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const ulonglong2 m4 = *reinterpret_cast<const ulonglong2*>(minus_m + h0 + c + i);
              ulonglong2 q4m = make_ulonglong2(0ull, 0ull);
              if constexpr (!kPlain) q4m = *reinterpret_cast<const ulonglong2*>(qm + c + i);
#pragma unroll
              for (int j = 0; j < 4; j += 2) {
                const uint64_t r2 = pack2(__uint_as_float(r16[i + j]), __uint_as_float(r16[i + j + 1])), m2 = j ? m4.y : m4.x;
                float x, y;
                if constexpr (kPlain) unpack2(fma2(r2, sl22, m2), x, y);
                else unpack2(fma2(r2, mul2(sl22, j ? q4m.y : q4m.x), add2(m2, lift2)), x, y);
                const float ex = ex2_approx(x), ey = ex2_approx(y);
                const __half2 p = __floats2half2_rn(ex, ey);
                const uint32_t u = half2_bits(p);
                uint64_t& sum = lp[(c + i + j) / 2];
                if constexpr (kPlain) {
                  const float2 pf = __half22float2(p);
                  sum = add2(sum, pack2(pf.x, pf.y));
                } else {
                  sum = fma2(pack2(ex, ey), back2, sum);
                }
                put16(pdst[(i + j) & 7] + (c + ((i + j) & 8)) * 128, u);
                put16(pdst[(i + j + 1) & 7] + (c + ((i + j) & 8)) * 128, u >> 16);
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) put16(pdst[i & 7] + (c + (i & 8)) * 128, 0u);
          }
        }
      };
      if (lifted || q_lifted) weights(std::false_type{});
      else weights(std::true_type{});
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_full);
    }
    // ---- epilogue: wait for the last value products, reduce the row sums ----
    const int sp = at / a.T, t = at - sp * a.T;
    float* prow = a.partial + (static_cast<long long>(t) * a.n_splits + sp) * a.nh * (kD + 2);
    {
      const Item e = item_from(at + gridDim.x);
      at = e.i;
      n_blocks = e.n_blocks;
    }
    ok = __all_sync(0xffffffffu, ok && mbar_wait(&bars->pv_done, k & 1, a.status, 611));
    if (threadIdx.x == 128) STK_TRACE(5);
    tc_fence_after();
#pragma unroll
    for (int c = 0; c < kHeads; c += 16) {
      float l16[16];
#pragma unroll
      for (int i = 0; i < 16; i += 2) unpack2(lp[(c + i) / 2], l16[i], l16[i + 1]);
      bfly_reduce_store<16, false>(l16, smax + q4 * NH + h0 + c, lane);
    }
    named_bar_sync(2, kSoftmaxThreads);
    const float l_own = own < NH ? (smax[own] + smax[NH + own]) + (smax[2 * NH + own] + smax[3 * NH + own]) : 0.f;
    if (a.out != nullptr) {
      // direct output: per-head factor exp(m - M) / (exp(sink - M) + l * exp(m - M)) with M = max(sink, m)
      if (own < NH) {
        const float m_nat = m_run[own] * 0.6931471805599453f;
        const float sk = (a.sink != nullptr && own < a.nh) ? a.sink[own] : -INFINITY;
        const float M = fmaxf(sk, m_nat);
        float f = 0.f;
        if (m_nat != -INFINITY) {
          const float w = __expf(m_nat - M);
          const float denom = (sk != -INFINITY ? __expf(sk - M) : 0.f) + l_own * w;
          f = denom > 0.f ? w / denom : 0.f;
        }
        alpha_s[own] = f;
      }
      named_bar_sync(2, kSoftmaxThreads);
    }
    if (ok && a.out != nullptr) {
      // 64 bytes of a row a store: without a branch per value these are as fast as a turn through shared memory (with one per value
      // they took 16000 cycles a token)
      __nv_bfloat16* orow = a.out + static_cast<long long>(t) * a.ldo;
      const float pos = a.positions != nullptr ? static_cast<float>(a.positions[t]) : 0.f;
#pragma unroll 1
      for (int j = 0; j < 4; ++j) {
        const int d = j * 128 + row;
        const bool rot = a.positions != nullptr && j == 3 && q4 >= 2;      // d >= 448: warp-uniform
        float sn = 0.f, cs = 1.f;
        if (rot) sincosf(pos * a.inv_freq[(d - kNope) >> 1], &sn, &cs);
#pragma unroll 1
        for (int c = 0; c < kHeads; c += 16) {
          uint32_t r16[16];
          tmem_ld_32x16(tmem_o + j * NH + h0 + c + lane_addr, r16);
          tmem_ld_wait();
          float v[16];
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            const float4 f4 = *reinterpret_cast<const float4*>(alpha_s + h0 + c + i);
            v[i] = __uint_as_float(r16[i]) * f4.x;
            v[i + 1] = __uint_as_float(r16[i + 1]) * f4.y;
            v[i + 2] = __uint_as_float(r16[i + 2]) * f4.z;
            v[i + 3] = __uint_as_float(r16[i + 3]) * f4.w;
          }
          if (rot) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              // the pair (even d, d + 1) sits in neighbouring lanes
              const float p = __shfl_xor_sync(0xffffffffu, v[i], 1);
              v[i] = (d & 1) ? (-p * sn + v[i] * cs) : (v[i] * cs + p * sn);
            }
          }
          __nv_bfloat16* o = orow + (h0 + c) * kD + d;
          if (h0 + c + 16 <= a.nh) {
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i * kD] = __float2bfloat16(v[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (h0 + c + i < a.nh) o[i * kD] = __float2bfloat16(v[i]);
          }
        }
      }
    } else if (ok) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int c = 0; c < kHeads; c += 16) {
          uint32_t r16[16];
          tmem_ld_32x16(tmem_o + j * NH + h0 + c + lane_addr, r16);
          tmem_ld_wait();
          float* o = prow + (h0 + c) * (kD + 2) + j * 128 + row;
          if (h0 + c + 16 <= a.nh) {                       // without a branch per value
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i * (kD + 2)] = __uint_as_float(r16[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (h0 + c + i < a.nh) o[i * (kD + 2)] = __uint_as_float(r16[i]);
          }
        }
      }
      if (own < a.nh) {
        prow[own * (kD + 2) + kD] = m_run[own] * 0.6931471805599453f;      // back to natural-log units
        prow[own * (kD + 2) + kD + 1] = l_own;
      }
    }
    // O has been read: the next item's value products wait for its weights, which come behind this fence
    tc_fence_before();
    }
  } else {
    // ------------------------------- producers -------------------------------
    // Warp pw owns rows 8 pw .. 8 pw + 7 of every block; a lane holds 16 bytes of each 64-byte segment of one row's codes, and the
    // row's scale bytes.
    const int pw = warp - 4 - kSoftmaxWarps, l4 = lane & 3, row = 8 * pw + (lane >> 2);
    uint8_t* const line = k_s + row * 128;
    const uint32_t turn = (row & 7) << 4;
    uint4 raw[7], rot[2];                                  // codes, and the rotated part (bf16)
    uint2 sc8;
    const uint8_t* src_row;                                // row whose codes are in `raw`; nullptr: none
    // The item, its blocks, and the list's next row of this lane (registers are short here: no more is kept)
    int at, t = 0, n_swa = 0, r_end = 0, n_blocks = 0, li = 0, next_slot = -1;
    uint32_t turn_q = 0;                                   // list of the powers of two of this item's queries
    constexpr int kWindow = 1 << 30;                       // marks a slot of the first cache (a slot is far below)
    auto look_up = [&]() {                                 // li -> next_slot, and on to the same row of the next block
      next_slot = -1;
      if (li < n_swa && li < r_end) next_slot = a.swa_slots[static_cast<long long>(t) * a.swa_ld + li] | kWindow;
      else if (li < r_end) next_slot = a.topk_slots[static_cast<long long>(t) * a.topk_ld + (li - n_swa)];
      li += kRows;
    };
    auto enter = [&](int from) {
      const Item w = item_from(from);
      at = w.i;
      if (at >= items) return;
      t = w.t;
      n_swa = w.n_swa;
      r_end = w.r_end;
      n_blocks = w.n_blocks;
      li = w.r_begin + row;
      look_up();
    };
    enter(blockIdx.x);
    auto next_row = [&]() {                                // next_slot -> row to be fetched; slot of the block after
      const int slot = next_slot & ~kWindow;
      const bool swa = (next_slot & kWindow) != 0;
      src_row = nullptr;
      sc8 = make_uint2(0, 0);
      if (next_slot >= 0) {
        const uint8_t* page = (swa ? a.swa_base : a.comp_base) + static_cast<long long>(slot >> 6) * (swa ? a.swa_stride : a.comp_stride);
        src_row = page + (slot & 63) * kDataBytes + l4 * 16;
        sc8 = *reinterpret_cast<const uint2*>(page + 64 * kDataBytes + (slot & 63) * 8);
      }
      look_up();
    };
    auto fetch = [&](int seg) {
      raw[seg] = make_uint4(0, 0, 0, 0);
      if (src_row != nullptr) raw[seg] = __ldg(reinterpret_cast<const uint4*>(src_row + seg * 64));
    };
    auto fetch_rot = [&]() {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        rot[i] = make_uint4(0, 0, 0, 0);
        if (src_row != nullptr) rot[i] = __ldg(reinterpret_cast<const uint4*>(src_row + kNope + i * 64));
      }
    };
    auto fetch_row = [&]() {
      next_row();
#pragma unroll
      for (int i = 0; i < 7; ++i) fetch(panel_at(i));
      fetch_rot();
    };
    if (at < items) fetch_row();
    begin();
    bool ok = true;
    uint32_t g = 0;
    while (at < items) {
      const uint2 sc = sc8;
      // The row's largest magnitude: a code's is below 2^9.  Scales (by halves: bytes 0 2, 1 3, 4 6, 5 -)
      const uint32_t s0 = sc.x & 0x00ff00ffu, s1 = (sc.x >> 8) & 0x00ff00ffu, s2 = sc.y & 0x00ff00ffu, s3 = (sc.y >> 8) & 0x000000ffu;
      const uint32_t top = __vmaxu2(__vmaxu2(s0, s1), __vmaxu2(s2, s3)), low = __vminu2(__vminu2(s0, s1), __vminu2(s2, s3 | 0x00ff0000u));
      uint32_t big = __vmaxu2(__vmaxu2(bf16x2_absmax(rot[0].x, rot[0].y), bf16x2_absmax(rot[0].z, rot[0].w)),
                              __vmaxu2(bf16x2_absmax(rot[1].x, rot[1].y), bf16x2_absmax(rot[1].z, rot[1].w)));
      big = __vmaxu2(big, __shfl_xor_sync(0xffffffffu, big, 1));
      big = __vmaxu2(big, __shfl_xor_sync(0xffffffffu, big, 2));
      const int lift = range_shift(max(max(static_cast<int>(top & 0xffff), static_cast<int>(top >> 16)) + 8, static_cast<int>(max(big & 0xffff, big >> 16) >> 7)),
                                   min(low & 0xffff, low >> 16) < 103);
      const float back = power_of_two(-lift);
#pragma unroll
      for (int i = 0; i < kPanels; ++i) {
        const int p = panel_at(i);
        if (g > 0 && (i == 0 || i == 1 || i == 3 || i == 5)) {
          ok = __all_sync(0xffffffffu, ok && mbar_wait(&bars->k_free[p >> 1], (g - 1) & 1, a.status, 620));
          if (!ok) break;
        }
        if (i == 0 && l4 == 0) lift_s[row] = src_row != nullptr ? lift : kNoRow;
        uint4 o0, o1;
        uint32_t at0, at1;
        if (p < 7) {
          const uint32_t w = p < 4 ? sc.x : sc.y;
          const float f = __uint_as_float(((p & 3) == 3 ? w >> 1 : w << (23 - 8 * (p & 3))) & 0x7f800000u) * back;      // 2^(byte - 127 - lift)
          const __half2 f2 = __float2half2_rn(f);
          const uint32_t codes[4] = {raw[p].x, raw[p].y, raw[p].z, raw[p].w};
          __half2 h[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            e4m3x4_to_half(codes[j], h[2 * j], h[2 * j + 1]);
            h[2 * j] = __hmul2(h[2 * j], f2);
            h[2 * j + 1] = __hmul2(h[2 * j + 1], f2);
          }
          o0 = make_uint4(half2_bits(h[0]), half2_bits(h[1]), half2_bits(h[2]), half2_bits(h[3]));
          o1 = make_uint4(half2_bits(h[4]), half2_bits(h[5]), half2_bits(h[6]), half2_bits(h[7]));
          at0 = (l4 << 5) ^ turn;
          at1 = ((l4 << 5) + 16) ^ turn;
        } else {
          o0 = bf16x8_to_half(rot[0], back);
          o1 = bf16x8_to_half(rot[1], back);
          at0 = (l4 << 4) ^ turn;
          at1 = ((4 + l4) << 4) ^ turn;
        }
        *reinterpret_cast<uint4*>(line + p * kPanelBytes + at0) = o0;
        *reinterpret_cast<uint4*>(line + p * kPanelBytes + at1) = o1;
        if (i == 0 || i == 2 || i == 4 || i == 6 || i == 7) {
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->k_full[p < 6 ? p >> 1 : p - 3]);
        }
      }
      if (!ok) break;
      ++g;
      if (--n_blocks == 0) {
        // the next item's queries as soon as this one's last scores have been formed, under its softmax, value products and output
        enter(at + gridDim.x);
        if (at >= items) break;
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_full, (g - 1) & 1, a.status, 621));
        if (!ok) break;
        turn_q ^= 1;
        load_q(t, threadIdx.x - (4 + kSoftmaxWarps) * 32, turn_q, std::integral_constant<int, 32 * kProducerWarps>{});
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->q_full);
      }
      // the next block's codes: asked for once all of this one is handed over, they arrive under its softmax
      fetch_row();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0) STK_TRACE(6);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(bars->tmem_base, Cfg::kTmemCols);
  }
}

template <int NH>
static int launch_mla_tc(const MlaTcArgs& a, cudaStream_t st) {
  const int smem = kPanels * kPanelBytes + kPanels * NH * 128 + 2 * NH * 128 + kBarBytes + 9 * NH * 4 + kRows * 4 + 1024;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(sparse_mla_tc_kernel<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
      return -3;
    configured = true;
  }
  int device = 0, sms = 1;
  if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return -5;
  const long long items = static_cast<long long>(a.T) * a.n_splits;
  if (items > 0x7fffffffLL - sms) return -6;
  launch_pdl(sparse_mla_tc_kernel<NH>, dim3(static_cast<unsigned>(items < sms ? items : sms)), dim3(MlaCfg<NH>::kThreads), smem, st, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace stk

using namespace stk;

static int mla_tc_run(const void* q, long long ldt, const void* swa_cache, long long swa_stride, const void* comp_cache,
                      long long comp_stride, const int* swa_slots, int swa_ld, const int* swa_lens, const int* topk_slots,
                      int topk_ld, const int* topk_lens, float* workspace, int n_splits, int T, int nh, int D, int R,
                      int max_rows, float scale, void* out, long long ldo, const float* sink, const int64_t* positions,
                      const float* inv_freq, int* status, void* trace, void* stream) {
  if (T <= 0) return 0;
  if (D != kD || R != kR || nh > 64 || nh < 1) return -20;
  if ((reinterpret_cast<uintptr_t>(q) & 15) || (ldt % 8)) return -21;
  if (out != nullptr && n_splits != 1) return -22;
  MlaTcArgs a;
  a.q = (const __nv_bfloat16*)q; a.ldt = ldt;
  a.swa_base = (const uint8_t*)swa_cache; a.swa_stride = swa_stride;
  a.comp_base = (const uint8_t*)comp_cache; a.comp_stride = comp_stride;
  a.swa_slots = swa_slots; a.swa_ld = swa_ld; a.swa_lens = swa_lens;
  a.topk_slots = topk_slots; a.topk_ld = topk_ld; a.topk_lens = topk_lens;
  a.partial = workspace; a.T = T; a.nh = nh; a.n_splits = n_splits;
  a.out = (__nv_bfloat16*)out; a.ldo = ldo; a.sink = sink; a.positions = positions; a.inv_freq = inv_freq;
  const int rps = (max_rows + n_splits - 1) / n_splits;
  a.rows_per_split = ((rps + kRows - 1) / kRows) * kRows;
  a.scale = scale; a.status = status; a.trace = (unsigned long long*)trace;
  cudaStream_t st = (cudaStream_t)stream;
  if (nh <= 16) return launch_mla_tc<16>(a, st);
  if (nh <= 32) return launch_mla_tc<32>(a, st);
  return launch_mla_tc<64>(a, st);
}

// Same contract as stk_sparse_mla (partials + combine), restricted to fp8_ds_mla rows with D = 512,
// R = 64 and at most 64 local heads.  Returns -20 for shapes it does not cover.
STK_API int stk_sparse_mla_tc(const void* q, long long ldt, const void* swa_cache, long long swa_stride,
                              const void* comp_cache, long long comp_stride, const int* swa_slots, int swa_ld,
                              const int* swa_lens, const int* topk_slots, int topk_ld, const int* topk_lens,
                              float* workspace, int n_splits, int T, int nh, int D, int R, int max_rows, float scale,
                              int* status, void* trace, void* stream) {
  return mla_tc_run(q, ldt, swa_cache, swa_stride, comp_cache, comp_stride, swa_slots, swa_ld, swa_lens, topk_slots,
                    topk_ld, topk_lens, workspace, n_splits, T, nh, D, R, max_rows, scale, nullptr, 0, nullptr, nullptr,
                    nullptr, status, trace, stream);
}

// An item is a token's whole row list, final output written by the kernel (sink merged, normalised, inverse
// RoPE on the rope dims when positions != null): for steps with enough tokens to fill the GPU without row splits.
STK_API int stk_sparse_mla_tc_out(const void* q, long long ldt, const void* swa_cache, long long swa_stride,
                                  const void* comp_cache, long long comp_stride, const int* swa_slots, int swa_ld,
                                  const int* swa_lens, const int* topk_slots, int topk_ld, const int* topk_lens, int T,
                                  int nh, int D, int R, int max_rows, float scale, void* out, long long ldo,
                                  const float* sink, const int64_t* positions, const float* inv_freq, int* status,
                                  void* stream) {
  if (out == nullptr) return -23;
  return mla_tc_run(q, ldt, swa_cache, swa_stride, comp_cache, comp_stride, swa_slots, swa_ld, swa_lens, topk_slots,
                    topk_ld, topk_lens, nullptr, 1, T, nh, D, R, max_rows, scale, out, ldo, sink, positions, inv_freq,
                    status, nullptr, stream);
}
