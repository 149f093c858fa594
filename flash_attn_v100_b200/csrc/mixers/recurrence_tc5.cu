// Gated linear recurrences over prompts on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a: heads of up to 128 key
// columns and any number of value columns, bfloat16 activations.
//
// In chunks of C = 128 tokens, with L the running sum of la inside the chunk and S the state before it:
//     A  = Q K^T                           O1 = Q S                  S enters as two bfloat16 parts (high, low: about 17 bits)
//     P_ij = A_ij e^(L_i - L_j) b_j, j <= i, as two bfloat16 parts    O2 = P V           P is read from tensor memory
//     o_i = e^(L_i) O1_i + O2_i            dS = K^T V'               v'_j = e^(L_C - L_j) b_j v_j, two bfloat16 parts
//     S  <- e^(L_C) S + dS                 S stays in the threads' registers, fp32
// Decays and weights act on rows of V' and P and on columns of S only, never on Q and K: the 128 value columns of a CTA can
// belong to two heads with the same queries and keys (NH = 2, heads of up to 64 value columns), which share A.
// The normaliser (NORM), n <- e^(L_C) n + sum_j w_j k_j with the weights w of V', is a column beside the state's: n_i . q_i = e^(L_i) (n . q_i) +
// sum_j P_ij, the second sum from the P in registers. n and w enter their products as three bfloat16 parts each, which hold all 24 bits, in columns 0-2
// and 16-18 of a tile of their own (two products of N = 32); n stays in registers, fp32.  (As sums in the threads, which read Q and K from shared
// memory once more, they took 2950 cycles of a chunk.)
//
// CTA = (segment of a sequence, head or pair of heads, 128 value columns), eighteen warps and two idle ones.  Sixteen compute: a warp owns 32 lanes (rows) x 32 columns of
// whatever is in tensor memory.  One issues the MMAs and one the copies, and works out the gates of the next chunk.  They meet at mbarriers, the four warps
// that share rows at named ones: with the MMAs issued by one of the computing warps and all of them at block barriers, everybody waited for that warp at
// every hand-over, since an issue blocks while the tensor queue is full.  16 x 1024 tokens, 32 heads of 128, with the normaliser's sums moved to the MMAs
// and Q K^T of the next chunk issued behind the state's product: 235 -> 209 us for gates and recurrence.  The least divisor of every token comes with the
// gates, too: as a load in the computing warps, whose registers are full, it held them up for a trip to memory per chunk; 209 -> 200 us.  Registers that the
// other warps hand in (a thread may have 96 at the launch, the computing warps then have 104, with next to no spills): 200 -> 193 us; 7500 cycles per chunk
// where it took 8700 (11 700 at first).  What bounds it now: the chain S -> tiles -> V' -> state of a chunk, its shared-memory traffic (a third of the
// cycles), and 6 of the 40 us of a CTA before its first and behind its last chunk.
// Segments let few long sequences fill the GPU: a first launch computes what every segment adds to the state, a scan over the segments turns that into
// the state at the start of each, and the main launch then runs all segments side by side.
//
// Tensor memory, 512 columns: A / P of the first head [0, 128)  O1 [128, 256)  O2 [256, 384), before P V the normaliser's products  P of the second head / dS
// [384, 512).
// Shared memory: six tiles of 128 x 128 bfloat16, each two 128-byte-swizzled slabs of 64 columns: Q, K twice, V, and S high and low,
// whose place V' takes once O1 is done.  Q, K and V come by TMA (the next K while this chunk is computed, the next Q once O1 is done,
// the next V once the output, which takes V's place, has been stored, also by TMA).  Rows past a sequence's end have the weight 0.
// Waits are bounded: one that runs out sets the status word, and every role runs on to its end without waiting.
#include "../hybrid/hybrid_common.cuh"
#include "../tc5.cuh"
#include "../tma3.cuh"
#include "recurrence.cuh"

namespace fa {
namespace mixers {

using hybrid::bf16;

namespace {

constexpr int C = 128;         // tokens per chunk
constexpr int N = 128;         // key and value columns per CTA (padded with zeros)
constexpr int kCompute = 512;  // threads that compute
constexpr int kThreads = kCompute + 128;
static_assert(kCompute * 104 + 128 * 64 <= kThreads * 96, "registers");   // (launched with 96 a thread)
constexpr int SLAB = 128 * 128;
constexpr int TILE = 2 * SLAB;
constexpr float kLog2e = 1.4426950408889634f;

struct Small {                 // behind the tiles
  float2 lb[2][2][C];          // [buffer][head]: running log2 decay and weight of every token
  float wk[2][2][C];           // weight of every token in the state after the chunk
  float wb[2][2][C];           // ... and in the row at the end of its block of 32 tokens, without what is decayed by then
  float dec[2][2];             // log2 decay over the chunk
  float floor[2][C];           // (NORM) least divisor of every token
  float den[4][C];             // partial n . q of every row, by column group
  uint64_t bars[16];
  uint32_t tmem_slot;
  volatile int gave_up;
  int grows[2];                // [buffer] (pairs of heads) some log decay of the chunk is above 0
};
// Barriers: a copy has landed; MMAs are done; the computing warps have written (or, the last, may be read) what the name says; gates are there.
enum Bar { kFullQ, kFullV, kFullK, kScores = kFullK + 2, kOld, kNew, kState, kStateIn, kWeights, kValues, kOut, kGates, kDrain = kGates + 2, kBars };
static_assert(kBars <= 16, "barriers");
constexpr int kTiles = 6;
constexpr int smem_bytes(bool norm) { return 1024 + kTiles * TILE + (norm ? SLAB : 0) + (int)sizeof(Small); }
static_assert(smem_bytes(true) <= 227 * 1024, "shared memory plan exceeds the SM");

// Byte offset of 16-byte unit `u` (0..15) of row `row` in a tile.
__device__ __forceinline__ uint32_t tile_off(int row, int u) {
  return (uint32_t)((u >> 3) * SLAB + row * 128 + ((u ^ row) & 7) * 16);
}
__device__ __forceinline__ void st_shared(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 ld_shared(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 unpack2(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}
// Two fp32 numbers as packed (high, low) bfloat16 parts.
__device__ __forceinline__ void split2(float2 v, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf162(v.x, v.y);
  const float2 r = ffma2(unpack2(hi), make_float2(-1.f, -1.f), v);
  lo = pack_bf162(r.x, r.y);
}
// One fp32 number as the sum of three bfloat16 numbers, the first three of a unit.
__device__ __forceinline__ uint4 split3(float v) {
  const float hi = __bfloat162float(__float2bfloat16_rn(v)), mid = __bfloat162float(__float2bfloat16_rn(v - hi));
  return make_uint4(pack_bf162(hi, mid), pack_bf162((v - hi) - mid, 0.f), 0u, 0u);
}

template <bool STATE_ONLY, int NH, bool NORM>
__global__ void __launch_bounds__(kThreads, 1)
recurrence_tc5_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                      const __grid_constant__ CUtensorMap omap, const RecurrenceArgs a) {
  static_assert(NH == 1 || !NORM, "a pair of heads has no normaliser");
  // instruction descriptors: fp32 accumulators, bfloat16 operands, M = 128, N at bit 17; bit 15: A MN-major, bit 16: B MN-major
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24);
  constexpr uint32_t N128 = (uint32_t)(N >> 3) << 17, NPV = (uint32_t)((N / NH) >> 3) << 17;
  constexpr uint32_t IDESC_QK = IDESC | N128, IDESC_B = IDESC | N128 | (1u << 16), IDESC_PV = IDESC | NPV | (1u << 16),
                     IDESC_AB = IDESC | N128 | (1u << 15) | (1u << 16);
  constexpr uint32_t N32 = (uint32_t)(32 >> 3) << 17, IDESC_B32 = IDESC | N32 | (1u << 16), IDESC_AB32 = IDESC | N32 | (1u << 15) | (1u << 16);
  extern __shared__ uint8_t smem_dyn[];
  const uint32_t raw_base = smem_u32(smem_dyn);
  uint8_t* smem = smem_dyn + ((1024u - (raw_base & 1023u)) & 1023u);
  const uint32_t sQ = smem_u32(smem), sK0 = sQ + TILE, sV = sK0 + 2 * TILE, sSh = sV + TILE, sSl = sSh + TILE, sE = sSl + TILE;
  Small& sm = *reinterpret_cast<Small*>(smem + kTiles * TILE + (NORM ? SLAB : 0));
  auto bar = [&](int i) { return smem_u32(&sm.bars[i]); };

  const int seq = blockIdx.x / a.max_segs, seg = blockIdx.x - seq * a.max_segs;
  const int head0 = blockIdx.y * NH, c0 = blockIdx.z * N, grp = head0 / a.kv_rep;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  long long t0 = a.cu[seq], t1 = a.cu[seq + 1];
  if (t0 < 0) t0 = 0;
  if (t1 > a.total) t1 = a.total;
  const long long seq_end = t1;
  const int seq_len = (int)(t1 - t0);
  t0 += (long long)seg * a.seg_len;
  if (t0 >= t1) return;
  if (t1 > t0 + a.seg_len) t1 = t0 + a.seg_len;
  const bool last_seg = t1 == seq_end;
  if (STATE_ONLY && last_seg) return;              // nothing follows it
  const int n_tok = (int)(t1 - t0), n_chunk = (n_tok + C - 1) / C;

  const int slot = a.slots[seq];
  const bool slot_ok = slot >= 0 && slot < a.n_slots;
  if (!slot_ok && tid == 0) atomicOr(a.status, kStatusBadPageId);
  const long long hs = (long long)a.dk * a.dv;
  const bool segmented = a.max_segs > 1;
  const long long seg_at = ((long long)seq * a.max_segs + seg) * a.heads;      // + head

  // ---- roles: the first sixteen warps compute, then one issues the MMAs and one the copies (and works out the gates) ----------
  const bool wide_k = a.dk > 64, wide_v = NH == 2 || a.dv - c0 > 64;           // the tile's second slab has columns
  const bool mma_warp = warp == kCompute / 32, copy_warp = warp == kCompute / 32 + 1;
  auto load_tile = [&](const CUtensorMap* map, uint32_t dst, uint32_t full, bool wide, int col, int head, int col2, int head2, long long t) {
    mbar_expect_tx(full, wide ? TILE : SLAB);
    tma_load_3d(dst, map, col, head, (int)t, full);
    if (wide) tma_load_3d(dst + SLAB, map, col2, head2, (int)t, full);
  };
  auto load_q = [&](int chunk) { load_tile(&qmap, sQ, bar(kFullQ), wide_k, 0, grp, 64, grp, t0 + (long long)chunk * C); };
  auto load_k = [&](int chunk) {
    load_tile(&kmap, sK0 + (chunk & 1) * TILE, bar(kFullK + (chunk & 1)), wide_k, 0, grp, 64, grp, t0 + (long long)chunk * C);
  };
  auto load_v = [&](int chunk) {
    if (NH == 2) load_tile(&vmap, sV, bar(kFullV), true, 0, head0, 0, head0 + 1, t0 + (long long)chunk * C);
    else load_tile(&vmap, sV, bar(kFullV), wide_v, c0, head0, c0 + 64, head0, t0 + (long long)chunk * C);
  };
  if (copy_warp && lane == 0) {
    for (int i = 0; i < kBars; ++i) mbar_init(bar(i), i >= kStateIn && i < kStateIn + 4 ? kCompute / 32 : 1);
    sm.gave_up = 0;
    mbar_fence_init();
    fence_proxy_async();
    if (!STATE_ONLY) load_q(0);
    load_k(0);
    load_v(0);
  }
  if (mma_warp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }

  // ---- decays: la and b of a chunk turned into sums, four tokens per lane -----
  float gl[NH][4], gb[NH][4], gf[4];
  auto fetch_gates = [&](int chunk) {
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      const long long tb = t0 + (long long)chunk * C + lane * 4, at = (long long)(head0 + h) * a.total + tb;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool in = tb + i < t1;
        gl[h][i] = in ? a.la[at + i] : 0.f;
        gb[h][i] = in ? a.b[at + i] : 0.f;
        if (NORM && !STATE_ONLY) gf[i] = in ? a.floor[at + i] : 0.f;
      }
    }
  };
  auto put_gates = [&](int buf) {
    if (NH == 2 && !STATE_ONLY) {
      bool up = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) up |= gl[0][i] > 0.f || gl[NH - 1][i] > 0.f;
      up = __any_sync(0xffffffffu, up);
      if (lane == 0) sm.grows[buf] = up ? 1 : 0;
    }
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      float* g = gl[h];
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] *= kLog2e;
      float up = g[0] + g[1] + g[2] + g[3], down = up;         // sums up to my last token, and from my first token on
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, up, o), d = __shfl_down_sync(0xffffffffu, down, o);
        if (lane >= o) up += u;
        if (lane + o < 32) down += d;
      }
      if (lane == 31) sm.dec[buf][h] = up;
      float before = __shfl_up_sync(0xffffffffu, up, 1), after = __shfl_down_sync(0xffffffffu, down, 1);
      if (lane == 0) before = 0.f;
      if (lane == 31) after = 0.f;
      float own[4];                                             // running decay at my tokens
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        before += g[i];
        sm.lb[buf][h][lane * 4 + i] = make_float2(before, gb[h][i]);
        own[i] = before;
      }
      if (NH == 2 && !STATE_ONLY) {
        const float end = __shfl_sync(0xffffffffu, before, lane | 7);
        *reinterpret_cast<float4*>(&sm.wb[buf][h][lane * 4]) = make_float4(fast_exp2(end - own[0]) * gb[h][0], fast_exp2(end - own[1]) * gb[h][1],
                                                                           fast_exp2(end - own[2]) * gb[h][2], fast_exp2(end - own[3]) * gb[h][3]);
      }
#pragma unroll
      for (int i = 3; i >= 0; --i) {                            // (summed from the end: the tokens that matter have small sums)
        sm.wk[buf][h][lane * 4 + i] = fast_exp2(after) * gb[h][i];
        after += g[i];
      }
      if (NORM && !STATE_ONLY) *reinterpret_cast<float4*>(&sm.floor[buf][lane * 4]) = make_float4(gf[0], gf[1], gf[2], gf[3]);
    }
  };
  if (copy_warp) {
    fetch_gates(0);
    put_gates(0);
    if (n_chunk > 1) fetch_gates(1);
  }
  if (NORM && tid < kCompute) {                                // the columns that are never written
    for (int i = tid; i < SLAB / 16; i += kCompute) st_shared(sE + i * 16, make_uint4(0, 0, 0, 0));
    fence_proxy_async();
  }
  if ((!wide_k || !wide_v) && tid < kCompute) {                // slabs that no copy fills
    const uint4 z = make_uint4(0, 0, 0, 0);
    for (int i = tid; i < SLAB / 16; i += kCompute) {
      if (!wide_k) {
        st_shared(sQ + SLAB + i * 16, z);
        st_shared(sK0 + SLAB + i * 16, z);
        st_shared(sK0 + TILE + SLAB + i * 16, z);
      }
      if (!wide_v) st_shared(sV + SLAB + i * 16, z);
    }
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_slot;

  // A wait that runs out, here or elsewhere in the CTA, turns `ok` false; the role goes on without waiting (the computing warps meet at barriers),
  // arriving or copying.
  bool ok = true;
  auto wait = [&](int which, uint32_t parity) {
    if (!ok) return;
    for (uint32_t i = 0; i < kMaxBarrierPolls; ++i) {
      if (mbar_try_wait(bar(which), parity)) return;
      if ((i & 255u) == 255u && sm.gave_up) break;
    }
    sm.gave_up = 1;
    ok = false;
  };
  // Every barrier below completes one phase per chunk, that of chunk c with parity c & 1; the two that alternate (K, gates) one per two chunks.
  if (mma_warp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    const uint64_t qd = smem_desc(sQ, 16, 1024), qkd = smem_desc(sK0, 16, 1024), khd = smem_desc(sK0, SLAB, 1024), vd = smem_desc(sV, SLAB, 1024);
    const uint64_t shd = smem_desc(sSh, SLAB, 1024), ed = smem_desc(sE, SLAB, 1024);
    auto issue_scores = [&](int c) {
      wait(kFullQ, (uint32_t)c & 1u);
      wait(kFullK + (c & 1), (uint32_t)(c >> 1) & 1u);
      tc_fence_after();
      __syncwarp();
      tc_mma_ss8<StepsAlongK<SLAB, SLAB>>(tmem, qd, qkd + (uint64_t)((c & 1) * (TILE >> 4)), IDESC_QK, 0u);
      tc_commit(bar(kScores));
    };
    if constexpr (!STATE_ONLY) issue_scores(0);
#pragma unroll 1
    for (int c = 0; c < n_chunk; ++c) {
      const uint32_t ph = (uint32_t)c & 1u;
      const uint64_t kc = khd + (uint64_t)((c & 1) * (TILE >> 4));
      if constexpr (!STATE_ONLY) {
        wait(kStateIn, ph);
        tc_fence_after();
        __syncwarp();
        tc_mma_ss8_parts<StepsByRowsB<SLAB>, 0, (TILE >> 4)>(tmem + 128u, qd, shd, IDESC_B, 0u);
        if constexpr (NORM) {
          tc_mma_ss8<StepsByRowsB<SLAB>>(tmem + 256u, qd, ed, IDESC_B32, 0u);
          tc_mma_ss8<StepsByRows>(tmem + 288u, kc, ed, IDESC_AB32, 0u);
        }
        tc_commit(bar(kOld));
        wait(kWeights, ph);
        wait(kFullV, ph);
        tc_fence_after();
        __syncwarp();
#pragma unroll
        for (int hh = 0; hh < NH; ++hh) {
          const uint64_t vh = vd + (uint64_t)(hh * (SLAB >> 4));
          const uint32_t d = tmem + 256u + (uint32_t)hh * 64u, p = tmem + (uint32_t)hh * 384u;
          tc_mma_ts8_parts<StepsTmemA<>, 64>(d, p, vh, IDESC_PV, 0u);
        }
        tc_commit(bar(kNew));
      }
      wait(kValues, ph);
      if constexpr (STATE_ONLY) wait(kFullK + (c & 1), (uint32_t)(c >> 1) & 1u);
      tc_fence_after();
      __syncwarp();
      tc_mma_ss8_parts<StepsByRows, 0, (TILE >> 4)>(tmem + 384u, kc, shd, IDESC_AB, 0u);       // (in order behind the products that read the second head's P there)
      if constexpr (NORM && STATE_ONLY) tc_mma_ss8<StepsByRows>(tmem + 288u, kc, ed, IDESC_AB32, 0u);
      tc_commit(bar(kState));
      if constexpr (!STATE_ONLY)
        if (c + 1 < n_chunk) issue_scores(c + 1);               // over P, in order behind P V
    }
    // every MMA is done before shared and tensor memory are given up
    tc_commit(bar(kDrain));
    if (!mbar_wait(bar(kDrain), 0u)) sm.gave_up = 1;
  } else if (copy_warp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    int n_q = 1, n_v = 1, n_k = 1;                              // loads issued
#pragma unroll 1
    for (int c = 0; c < n_chunk; ++c) {
      const uint32_t ph = (uint32_t)c & 1u;
      const bool more = c + 1 < n_chunk;
      wait(STATE_ONLY ? kValues : kStateIn, ph);                // every warp has begun the chunk: what only the one before used is free
      ok = __all_sync(0xffffffffu, ok);
      if (more) {
        if (lane == 0 && ok) { load_k(c + 1); ++n_k; }
        __syncwarp();
        put_gates((c + 1) & 1);
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(bar(kGates + ((c + 1) & 1)));
        if (c + 2 < n_chunk) fetch_gates(c + 2);
      }
      if constexpr (STATE_ONLY) {
        if (more && lane == 0 && ok) { load_v(c + 1); ++n_v; }  // V has become V'
      } else {
        if (more) {
          wait(kOld, ph);
          ok = __all_sync(0xffffffffu, ok);
          if (lane == 0 && ok) { load_q(c + 1); ++n_q; }
        }
        wait(kOut, ph);
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0 && ok) {
          const long long tb = t0 + (long long)c * C;
          if (n_tok - c * C >= C) {
            if (NH == 2) {
              tma_store_3d(&omap, 0, head0, (int)tb, sV);
              tma_store_3d(&omap, 0, head0 + 1, (int)tb, sV + SLAB);
            } else {
              tma_store_3d(&omap, c0, head0, (int)tb, sV);
              if (wide_v) tma_store_3d(&omap, c0 + 64, head0, (int)tb, sV + SLAB);
            }
            tma_store_commit();
          }
          if (more) {
            tma_store_wait_read();
            load_v(c + 1);
            ++n_v;
          }
        }
      }
      __syncwarp();
    }
    if (lane == 0) {                                            // copies into and out of this CTA's shared memory
      bool in = STATE_ONLY || mbar_wait(bar(kFullQ), (uint32_t)(n_q - 1) & 1u);
      in = mbar_wait(bar(kFullK + ((n_k - 1) & 1)), (uint32_t)((n_k - 1) >> 1) & 1u) && in;
      in = mbar_wait(bar(kFullV), (uint32_t)(n_v - 1) & 1u) && in;
      if (!in) sm.gave_up = 1;
      tma_store_wait_read();
    }
  } else if (tid >= kCompute) {                                // (two warps that only hand in their registers)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // my place in tensor memory: lane (row) and 32 columns
    const int row = (warp & 3) * 32 + lane, cg = warp >> 2;
    const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cg * 32u;
    const uint32_t tA = tl, tO1 = tl + 128u, tO2 = tl + 256u, tS = tl + 384u;
    const uint32_t tP = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)cg * 16u;     // high part; low part 64 columns on
    // ... and what the columns are: a head and its columns from mc on
    const int mh = NH == 2 ? cg >> 1 : 0, mc = NH == 2 ? (cg & 1) * 32 : c0 + cg * 32;
    auto row_sync = [&]() {                                     // the four warps that share my rows
      tc_fence_before();
      asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp & 3)) : "memory");
      tc_fence_after();
    };
    auto done = [&](int which) {                                // one arrival per warp, behind its writes of shared and tensor memory
      tc_fence_before();
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(bar(which));
    };

    // ---- state: row `row`, my columns ----------------------------------------------------------------
    float* cache = slot_ok ? a.state + ((long long)slot * a.heads + head0 + mh) * hs + (long long)row * a.dv : nullptr;
    float* segst = segmented ? a.seg_state + (seg_at + head0 + mh) * hs + (long long)row * a.dv : nullptr;
    float S[32];
    {
      const float* init = nullptr;
      if (!STATE_ONLY) {
        if (segmented) init = segst;
        else if (a.starts[seq] != 0) init = cache;
      }
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 v = init != nullptr && row < a.dk && mc + i < a.dv ? *reinterpret_cast<const float4*>(init + mc + i)
                                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
        S[i] = v.x; S[i + 1] = v.y; S[i + 2] = v.z; S[i + 3] = v.w;
      }
    }
    // normaliser: the first 128 threads hold column `row` of it
    float nrm = 0.f;
    auto put_ext = [&](int unit, float v) { st_shared(sE + (uint32_t)(row * 128 + ((unit ^ row) & 7) * 16), split3(v)); };
    if (NORM && !STATE_ONLY && cg == 0 && row < a.dk)
      nrm = segmented ? a.seg_norm[(seg_at + head0) * a.dk + row] : a.n0[((long long)seq * a.heads + head0) * a.dk + row];

    // 16-byte unit n of mine where tiles are worked on row by row: row urow + 32 n, unit tid & 15
    const int cu8 = (tid & 15) * 8, urow = tid >> 4;
    const int uh = NH == 2 ? cu8 >> 6 : 0, uc = NH == 2 ? cu8 & 63 : c0 + cu8;   // as value columns: a head and its columns
    const float skip = a.skip != nullptr ? a.skip[head0 + mh] : 0.f;
    float log_sum = 0.f;                                        // (STATE_ONLY) log2 decay over the segment

#pragma unroll 1
    for (int c = 0; c < n_chunk; ++c) {
      const int buf = c & 1;
      const uint32_t ph = (uint32_t)buf;
      // v' = weight * v of the units of mine, high and low part, to the state's tiles
      auto put_weighted = [&]() {
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const uint32_t off = tile_off(urow + 32 * n, tid & 15);
          const float w1 = sm.wk[buf][uh][urow + 32 * n];
          const float2 w = make_float2(w1, w1);
          const uint4 v = ld_shared(sV + off);
          uint4 h, l;
          split2(fmul2(unpack2(v.x), w), h.x, l.x);
          split2(fmul2(unpack2(v.y), w), h.y, l.y);
          split2(fmul2(unpack2(v.z), w), h.z, l.z);
          split2(fmul2(unpack2(v.w), w), h.w, l.w);
          st_shared(sSh + off, h);
          st_shared(sSl + off, l);
        }
      };
      if (c > 0) wait(kGates + buf, (uint32_t)((c - 1) >> 1) & 1u);
      if (NORM && cg == 0) put_ext(2, sm.wk[buf][0][row]);
      if constexpr (!STATE_ONLY) {
        // ---- the state's tiles ------------------------------------------------------------------------
        if (NORM && cg == 0) put_ext(0, nrm);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          uint4 h, l;
          split2(make_float2(S[8 * u], S[8 * u + 1]), h.x, l.x);
          split2(make_float2(S[8 * u + 2], S[8 * u + 3]), h.y, l.y);
          split2(make_float2(S[8 * u + 4], S[8 * u + 5]), h.z, l.z);
          split2(make_float2(S[8 * u + 6], S[8 * u + 7]), h.w, l.w);
          const uint32_t off = tile_off(row, cg * 4 + u);
          st_shared(sSh + off, h);
          st_shared(sSl + off, l);
        }
        fence_proxy_async();
        done(kStateIn);
        float den = 0.f;
        // ---- A -> P ------------------------------------------------------------------------------------
        wait(kScores, ph);
        __syncwarp();
        tc_fence_after();
        float s[32];
        tc_ld32(tA, s);
        tc_wait_ld();
        row_sync();                                             // P is written over the other warps' part of A
        const int over = row - cg * 32;                         // my columns up to this one are at or before my row
        const bool below = __any_sync(0xffffffffu, over >= 0);
        // All of my columns' tokens are in blocks before my row's: e^(L_i - L_j) is a factor per row, from the end of the columns' block on, and one per column,
        // which come with the gates, in place of an exponential per element and head.  Both are at most 1 where nothing grows; a chunk with a log decay above 0 goes by the
        // differences, as a factor could overflow where they do not.  Pairs of heads, 8 x 2048 tokens of 64 heads: 166 -> 154 us,
        // 8 x 1024 of 32 48.4 -> 46.9; with one head per CTA the exponentials are not what a chunk waits for (157.4 and 156.3 us, long sequences 2 % slower).
        const bool apart = NH == 2 && cg < (warp & 3) && sm.grows[buf] == 0;
#pragma unroll
        for (int hh = 0; hh < NH; ++hh) {
          const float2* lb = sm.lb[buf][hh] + cg * 32;
          const float li = sm.lb[buf][hh][row].x;
          const float *wb = sm.wb[buf][hh] + cg * 32, e1 = apart ? fast_exp2(li - lb[31].x) : 0.f;
          const float2 e_end = make_float2(e1, e1);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t hi[8], lo[8];
            if (apart) {
#pragma unroll
              for (int i = 0; i < 8; i += 2) {
                const int j = h * 16 + 2 * i;
                const float4 w = *reinterpret_cast<const float4*>(wb + j);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const float2 p = fmul2(make_float2(s[j + 2 * u], s[j + 2 * u + 1]), fmul2(e_end, u == 0 ? make_float2(w.x, w.y) : make_float2(w.z, w.w)));
                  if constexpr (NORM) den += p.x + p.y;
                  split2(p, hi[i + u], lo[i + u]);
                }
              }
            } else if (below) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int j = h * 16 + 2 * i;
                const float4 w = *reinterpret_cast<const float4*>(lb + j);
                const float2 e = make_float2(fast_exp2(li - w.x), fast_exp2(li - w.z));
                float2 p = fmul2(make_float2(s[j], s[j + 1]), fmul2(e, make_float2(w.y, w.w)));
                p.x = j <= over ? p.x : 0.f;                    // (a selection: what is dropped may have overflowed)
                p.y = j + 1 <= over ? p.y : 0.f;
                if constexpr (NORM) den += p.x + p.y;
                split2(p, hi[i], lo[i]);
              }
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) hi[i] = lo[i] = 0u;
            }
            tc_st8(tP + hh * 384u + h * 8u, hi);
            tc_st8(tP + hh * 384u + 64u + h * 8u, lo);
          }
        }
        wait(kOld, ph);
        __syncwarp();
        tc_fence_after();
        if constexpr (NORM) {
          if (cg == 0) {                                        // n . q and what the chunk adds to n, from where the first columns of P V will be
            float nq[8], add[8];
            tc_ld8(tO2, nq);
            tc_ld8(tO2 + 48u, add);
            tc_wait_ld();
            den += (nq[0] + nq[1] + nq[2]) * fast_exp2(sm.lb[buf][0][row].x);
            nrm = nrm * fast_exp2(sm.dec[buf][0]) + (add[0] + add[1] + add[2]);
          }
          sm.den[cg][row] = den;
        }
        tc_wait_st();
        done(kWeights);
        // ---- V' over the state's tiles ----------------------------------------------------------------
        wait(kFullV, ph);
        __syncwarp();
        put_weighted();
        fence_proxy_async();
        done(kValues);
        // ---- output, over V --------------------------------------------------------------------------------
        const float e = fast_exp2(sm.lb[buf][mh][row].x) * a.q_scale;
        float f2 = a.q_scale, f1 = e;
        if constexpr (NORM) {
          row_sync();
          const float dn = a.q_scale * (sm.den[0][row] + sm.den[1][row] + sm.den[2][row] + sm.den[3][row]);
          const float inv = 1.f / (fmaxf(fabsf(dn), sm.floor[buf][row]) + a.norm_eps);
          f1 *= inv;
          f2 *= inv;
        }
        wait(kValues, ph);                                      // every warp has read V
        wait(kNew, ph);
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float x[16], y[16];
          tc_ld16(tO1 + h * 16u, x);
          tc_ld16(tO2 + h * 16u, y);
          tc_wait_ld();
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const uint32_t off = tile_off(row, cg * 4 + h * 2 + u);
            uint32_t p[4];
            uint4 vu = make_uint4(0, 0, 0, 0);
            if (!NORM) vu = ld_shared(sV + off);
            const uint32_t vv[4] = {vu.x, vu.y, vu.z, vu.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int j = u * 8 + 2 * i;
              float2 r = ffma2(make_float2(x[j], x[j + 1]), make_float2(f1, f1), fmul2(make_float2(y[j], y[j + 1]), make_float2(f2, f2)));
              if (!NORM) r = ffma2(unpack2(vv[i]), make_float2(skip, skip), r);
              p[i] = pack_bf162(r.x, r.y);
            }
            st_shared(sV + off, make_uint4(p[0], p[1], p[2], p[3]));
          }
        }
        fence_proxy_async();
        done(kOut);
      } else {
        wait(kFullV, ph);
        __syncwarp();
        put_weighted();
        fence_proxy_async();
        done(kValues);
      }
      // ---- state ---------------------------------------------------------------------------------------
      wait(kState, ph);
      __syncwarp();
      tc_fence_after();
      {
        const float ld = sm.dec[buf][mh], dc = fast_exp2(ld);
        if (STATE_ONLY) log_sum += ld;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float t[16];
          tc_ld16(tS + h * 16u, t);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float2 r = ffma2(make_float2(S[h * 16 + i], S[h * 16 + i + 1]), make_float2(dc, dc), make_float2(t[i], t[i + 1]));
            S[h * 16 + i] = r.x;
            S[h * 16 + i + 1] = r.y;
          }
        }
        if (NORM && STATE_ONLY && cg == 0) {
          float add[8];
          tc_ld8(tO2 + 48u, add);
          tc_wait_ld();
          nrm = nrm * dc + (add[0] + add[1] + add[2]);
        }
      }
      if constexpr (!STATE_ONLY) {
        const int rows = n_tok - c * C;
        if (rows < C) {                                         // the last chunk of a sequence: its rows only
          wait(kOut, ph);
          bf16* p = static_cast<bf16*>(a.out) + (t0 + (long long)c * C + urow) * ((long long)a.heads * a.dv) + (long long)(head0 + uh) * a.dv + uc;
#pragma unroll
          for (int n = 0; n < 4; ++n)
            if (uc < a.dv && urow + 32 * n < rows)
              *reinterpret_cast<uint4*>(p + (long long)(32 * n) * a.heads * a.dv) = ld_shared(sV + tile_off(urow + 32 * n, tid & 15));
        }
      }
    }
    // The state leaves by way of the tiles' place, whose last readers are done: a row per lane is 16 bytes in each of 32 sectors, and took 3 us (the whole
    // kernel, with four CTAs one after the other on an SM: 163 -> 158 us).
    float* dst = STATE_ONLY ? a.seg_state + seg_at * hs : (last_seg && slot_ok ? a.state + (long long)slot * a.heads * hs : nullptr);
    if (dst != nullptr) {
      const int turn = lane & 7;                                // the lanes of eight rows at different units, without conflicts
#pragma unroll
      for (int b = 1; b < 8; b <<= 1) {
        float t[4 * 4];
#pragma unroll
        for (int i = 0; i < 4 * b; ++i) t[i] = S[i];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float from = i + 4 * b < 32 ? S[i + 4 * b] : t[i + 4 * b - 32];
          S[i] = (turn & b) ? from : S[i];
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i)
        st_shared(sSh + (uint32_t)(row * 512 + cg * 128 + ((i + turn) & 7) * 16),
                  make_uint4(__float_as_uint(S[4 * i]), __float_as_uint(S[4 * i + 1]), __float_as_uint(S[4 * i + 2]), __float_as_uint(S[4 * i + 3])));
      asm volatile("bar.sync 5, 512;" ::: "memory");
      const int unit = tid & 31, oh = NH == 2 ? unit >> 4 : 0, oc = NH == 2 ? (unit & 15) * 4 : c0 + unit * 4;
      dst += (long long)(head0 + oh) * hs + oc;
      if (oc < a.dv)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 16 + (tid >> 5);
          if (r < a.dk) *reinterpret_cast<uint4*>(dst + (long long)r * a.dv) = ld_shared(sSh + (uint32_t)(r * 512 + unit * 16));
        }
    }
    if (STATE_ONLY && blockIdx.z == 0 && row == 0 && (NH == 2 ? (cg & 1) == 0 : cg == 0)) a.seg_log[seg_at + head0 + mh] = log_sum;
    if (NORM && blockIdx.z == 0 && tid < a.dk) {
      if (STATE_ONLY) a.seg_norm[(seg_at + head0) * a.dk + tid] = nrm;
      else if (last_seg && slot_ok)
        a.norm[(((long long)slot * 2 + ((a.starts[seq] + seq_len - 1) & 1)) * a.heads + head0) * a.dk + tid] = nrm;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && sm.gave_up) atomicOr(a.status, kStatusWaitTimeout);
  if (mma_warp) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// seg_state[seq, s] (and seg_norm) holds what segment s adds; turned in place into the state at the start of segment s.
__global__ void __launch_bounds__(256) recurrence_segment_scan_kernel(const RecurrenceArgs a) {
  const long long hs = (long long)a.dk * a.dv;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const int head = blockIdx.y, seq = blockIdx.z;
  const bool norm = i >= hs;
  if (i >= hs + (a.floor != nullptr ? a.dk : 0)) return;
  const long long n = a.cu[seq + 1] - (long long)a.cu[seq];
  const int n_seg = (int)((n + a.seg_len - 1) / a.seg_len);
  const int slot = a.slots[seq];
  float s = 0.f;
  if (norm) s = a.n0[((long long)seq * a.heads + head) * a.dk + i - hs];
  else if (a.starts[seq] != 0 && slot >= 0 && slot < a.n_slots) s = a.state[((long long)slot * a.heads + head) * hs + i];
  const long long at = (long long)seq * a.max_segs * a.heads + head;
  float* p = norm ? a.seg_norm + at * a.dk + i - hs : a.seg_state + at * hs + i;
  const long long step = (long long)a.heads * (norm ? a.dk : hs);
  const float* lg = a.seg_log + at;
  for (int k = 0; k < n_seg && k < a.max_segs; ++k, p += step, lg += a.heads) {
    const bool more = k + 1 < n_seg;                // the last segment's slot was not written
    const float add = more ? *p : 0.f;
    *p = s;
    s = more ? fast_exp2(*lg) * s + add : s;
  }
}

// Heads per CTA.
int tile_heads(int heads, int kv_rep, int dv, bool norm) { return !norm && dv <= 64 && kv_rep % 2 == 0 && heads % 2 == 0 ? 2 : 1; }

template <int NH, bool NORM>
cudaError_t launch_t(const RecurrenceArgs& a, EncodeTiledFn enc, cudaStream_t stream) {
  const dim3 grid((unsigned)(a.n_seq * a.max_segs), (unsigned)(a.heads / NH), (unsigned)((a.dv + N - 1) / N));
  const auto* x = static_cast<const bf16*>(a.qkv);
  const int groups = a.heads / a.kv_rep;
  CUtensorMap qmap, kmap, vmap, omap;
  if (!make_map3(enc, &qmap, x + a.off_q, a.dk, groups, a.total, a.dk, a.stride) ||
      !make_map3(enc, &kmap, x + a.off_k, a.dk, groups, a.total, a.dk, a.stride) ||
      !make_map3(enc, &vmap, x + a.off_v, a.dv, a.heads, a.total, a.dv, a.stride) ||
      !make_map3(enc, &omap, a.out, a.dv, a.heads, a.total, a.dv, (long long)a.heads * a.dv))
    return cudaErrorInvalidValue;
  cudaError_t e;
  if (a.max_segs > 1) {
    e = cudaFuncSetAttribute(recurrence_tc5_kernel<true, NH, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(NORM));
    if (e != cudaSuccess) return e;
    recurrence_tc5_kernel<true, NH, NORM><<<grid, kThreads, smem_bytes(NORM), stream>>>(qmap, kmap, vmap, omap, a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long long n = (long long)a.dk * a.dv + (NORM ? a.dk : 0);
    recurrence_segment_scan_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)a.heads, (unsigned)a.n_seq), 256, 0, stream>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  e = cudaFuncSetAttribute(recurrence_tc5_kernel<false, NH, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(NORM));
  if (e != cudaSuccess) return e;
  recurrence_tc5_kernel<false, NH, NORM><<<grid, kThreads, smem_bytes(NORM), stream>>>(qmap, kmap, vmap, omap, a);
  return cudaGetLastError();
}

}  // namespace

int recurrence_segments(int n_seq, int heads, int kv_rep, int dk, int dv, int max_len, int sm_count, int* seg_len) {
  // one CTA per SM, in segments of at least 512 tokens: a segment's keys and values are read twice, which only pays while SMs
  // would stay empty.  (Heads with a normaliser never share a CTA; counting them as if they did only makes more segments.)
  (void)dk;
  const int nh = tile_heads(heads, kv_rep, dv, false);
  const long long tasks = (long long)n_seq * (heads / nh) * ((dv + N - 1) / N);
  const long long segs = tasks * 2 > sm_count ? 1 : sm_count / tasks;
  long long len = (max_len + segs - 1) / segs;
  if (len < 512) len = 512;
  len = (len + C - 1) / C * C;
  *seg_len = (int)len;
  return (int)((max_len + len - 1) / len);
}

bool recurrence_tc5_supported(const RecurrenceArgs& a) {
  return a.cu != nullptr && a.dk <= N && a.dk % 8 == 0 && a.dv % 8 == 0 && a.stride % 8 == 0 && a.off_q % 8 == 0 && a.off_k % 8 == 0 &&
         a.off_v % 8 == 0 && (reinterpret_cast<uintptr_t>(a.qkv) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(a.state) & 15) == 0 && (a.floor == nullptr || a.skip == nullptr);
}

cudaError_t launch_recurrence_tc5(const RecurrenceArgs& a, void* encode_fn, cudaStream_t stream) {
  if (a.n_seq == 0) return cudaSuccess;
  EncodeTiledFn enc = reinterpret_cast<EncodeTiledFn>(encode_fn);
  if (a.floor != nullptr) return launch_t<1, true>(a, enc, stream);
  return tile_heads(a.heads, a.kv_rep, a.dv, false) == 2 ? launch_t<2, false>(a, enc, stream) : launch_t<1, false>(a, enc, stream);
}

}  // namespace mixers
}  // namespace fa
