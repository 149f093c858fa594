// Attention in the latent space on the 5th-generation tensor cores (tcgen05 + TMEM), sm_100a, bfloat16 operands: decode steps and short portions
// of prompts, latents of 128 to 512 columns in blocks of 128, rotated parts of up to 64 columns.  Other sizes: latent_decode.cu.
//
// What bounds it: the ring of tiles and the few small MMAs that go through it.  A tile of 64 keys is 72 KB at 512 + 64 columns, 3250 cycles of an SM's share of
// HBM; it takes 52 MMAs of 45 cycles, whatever their size up to 64 columns, and two and a half tiles fit.  So the keys, and then the latent columns, are the
// rows of the MMAs and the heads their columns (16 to 64 of them, which cost little):
//     S^T [64 keys, heads] = K Q^T          O^T [latent columns, heads] += V^T P^T          V = the first columns of K, the same tile
// and all heads of the block use a tile while it is there.  (With the heads in the rows, on mma.sync, every warp reads the queries again for each
// tile and its ldmatrix instructions were the bound.)  O^T of 512 columns and 64 heads is 256 columns of tensor memory beside two score
// buffers; P^T goes through shared memory with the heads contiguous, as the thread of a key writes it.  Maxima are exact and running; O is rescaled
// in tensor memory by the heads whose maximum grew.
//
// The (row, key tile) units of the batch are cut into equal runs, one per CTA (latent_run.cuh); a row that is cut leaves partial sums for the merge
// of latent_decode.cu.
//
// Measured, us (the mma.sync kernel of latent_decode.cu): 64 rows of 2048 to 4096 cached tokens, 32 heads of 512 + 64 60.6 (87.5), L2 flushed in between 71.6 (96.2); flushed, 64
// heads 90 (164), 16 heads 65 (69); 256 + 32 and 8192 tokens, 32 heads 70 (115), 64 heads 106 (207); 256 rows of 256 tokens 45 (61); 5 rows of 700, 64 heads 24.5 (22.5).
// Tried: pages brought to L2 by bulk prefetches four tiles ahead, 79; one thread that issues all copies, 88; one warp for both products 68 to 70.
//
// Warps: 0 and those from 11 on copy (TMA, a box of 16 rows x 64 columns per page and slab), 1 issues the products for the scores, 2 those with the values, 4-7 softmax,
// rescale and output, 3, 8, 9 and 10 stage the queries (the next row's wait in registers).  A ring of slots of 64 keys x 256 (128) columns holds the latents and
// a smaller one the rotated parts, so copies run on while a tile is in the softmax.  (With one warp that issued both products, whichever was ready,
// its polls and waits were the bound: 4700 cycles per tile, 500 to 600 of them between any two runs of MMAs.)  Waits are bounded; one that runs out sets the
// status word, and all roles leave.
#include <math_constants.h>

#include "../common.cuh"
#include "../smem_limit.cuh"
#include "../tc5.cuh"
#include "hybrid_common.cuh"
#include "latent_run.cuh"

namespace fa {
namespace hybrid {
namespace {

constexpr int kQThreads = 128;         // threads that stage queries
constexpr int kSlab = KT * 128;        // bytes of 64 keys x 64 columns

// Shared memory of NB blocks of 128 latent columns and N heads.
template <int NB, int N>
struct Plan {
  static constexpr int kCtas = NB <= 2 && N <= 32 ? 2 : 1;             // resident CTAs per SM
  static constexpr int kCopyWarps = kCtas == 2 ? 2 : 4;
  static constexpr int kThreads = 320 + 32 * kCopyWarps;
  static constexpr int kBudget = kCtas == 2 ? 113 * 1024 : 226 * 1024;
  static constexpr int NR = NB == 4 && N == 64 ? 1 : 2;                // slabs of rotated parts
  static constexpr int kQ = (2 * NB + 1) * N * 128;
  static constexpr int kP = KT * 128;
  static constexpr int kMisc = 5 * 4 * N * 4 + 512;    // maxima, references, factors and sums; barriers and the rest
  static constexpr int SB = NB % 2 == 0 ? 2 : 1;                        // blocks per slot: few waits and commits for few MMAs
  static constexpr int kSlot = SB * 2 * kSlab;
  static constexpr int kFit = (kBudget - NR * kSlab - kQ - kP - kMisc) / kSlot;
  static constexpr int NV = kFit > 12 ? 12 : kFit;                     // slots
  static constexpr int kSmem = NV * kSlot + NR * kSlab + kQ + kP + kMisc;
  static constexpr int kTmemNeed = (NB + 2) * N;                       // O^T, two score buffers
  static constexpr int kTmem = kTmemNeed <= 64 ? 64 : (kTmemNeed <= 128 ? 128 : (kTmemNeed <= 256 ? 256 : 512));
  static_assert(NV >= NB / SB + 1, "a tile and a slot at least");
};

template <int NH>
__device__ __forceinline__ void tc_ld_split(uint32_t taddr, float (&v)[NH]);
// 16 lanes of tensor memory: threads 0-15 read NH columns from `taddr`, threads 16-31 the NH columns behind them.
template <>
__device__ __forceinline__ void tc_ld_split<8>(uint32_t taddr, float (&v)[8]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.16x32bx2.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], 8;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
template <>
__device__ __forceinline__ void tc_ld_split<16>(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x32bx2.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16], 16;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
template <>
__device__ __forceinline__ void tc_ld_split<32>(uint32_t taddr, float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x32bx2.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32], 32;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// Reduction of v[h] over the 16 lanes of a half warp: in each of four exchanges a lane keeps half of its values, so that it ends with the
// totals of N / 32 (at least one) heads, the first of them own_head<NH>(lane).
template <int NH, bool MAX>
__device__ __forceinline__ void spread_reduce(float (&v)[NH], int lane) {
#pragma unroll
  for (int s = 8, n = NH; s >= 1; s >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = (lane & s) != 0;
#pragma unroll
      for (int i = 0; i < NH / 2; ++i) {
        if (i < n) {
          const float send = up ? v[i] : v[n + i], keep = up ? v[n + i] : v[i];
          const float got = __shfl_xor_sync(0xffffffffu, send, s);
          v[i] = MAX ? fmaxf(keep, got) : keep + got;
        }
      }
    } else {
      const float got = __shfl_xor_sync(0xffffffffu, v[0], s);
      v[0] = MAX ? fmaxf(v[0], got) : v[0] + got;
    }
  }
}
template <int NH>
__device__ __forceinline__ int own_head(int lane) {
  return (lane >> 4) * NH + (NH == 32 ? (lane & 15) * 2 : (NH == 16 ? (lane & 15) : (lane & 15) >> 1));
}

template <int NB, int N>
__global__ void __launch_bounds__((Plan<NB, N>::kThreads), (Plan<NB, N>::kCtas)) latent_decode_tc5_kernel(const __grid_constant__ CUtensorMap pool_map,
                                                                                           const LatentAttentionArgs a) {
  using P = Plan<NB, N>;
  constexpr int NV = P::NV, NR = P::NR, CW = P::kCopyWarps, kThreads = P::kThreads, SB = P::SB, kSlot = P::kSlot;
  constexpr int NH = N / 2;                        // heads per softmax thread
  constexpr int OWN = NH == 32 ? 2 : 1;            // heads whose totals a lane holds
  constexpr int R = NB * 128;
  enum Bar { kVFull = 0, kVEmpty = NV, kRFull = 2 * NV, kREmpty = kRFull + NR, kQFull = kREmpty + NR, kQEmpty, kSFull, kPFull = kSFull + 2, kDrain = kPFull + 2,
             kBars = kDrain + 2 };
  static_assert(kBars * 8 + (kThreads / 32 + 8) * 4 <= 512, "barriers and the rest");
  extern __shared__ __align__(1024) uint8_t sm[];
  const uint32_t sV = smem_u32(sm), sR = sV + NV * kSlot, sQ = sR + NR * kSlab, sP = sQ + P::kQ;
  float* red = reinterpret_cast<float*>(sm + NV * kSlot + NR * kSlab + P::kQ + P::kP);       // [tile & 1][warp][N]
  float* refs = red + 2 * 4 * N;                   // [warp][N] references of the tile
  float* factors = refs + 4 * N;                   // [warp][N] what the sums so far are multiplied by
  float* sums = factors + 4 * N;                   // [warp][N] sums of the weights
  uint64_t* bars = reinterpret_cast<uint64_t*>(sums + 4 * N);
  int* scan_buf = reinterpret_cast<int*>(bars + kBars);
  int* found = scan_buf + kThreads / 32;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(found + 2);
  volatile int* gave_up = reinterpret_cast<volatile int*>(found + 3);
  auto bar = [&](int i) -> uint32_t { return smem_u32(bars + i); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cta = blockIdx.x, h0 = blockIdx.y * N;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the merge may be launched (it waits for this grid's end)

  int u0, u1;
  if (!find_run<kThreads>(a, scan_buf, found, u0, u1)) return;
  const int first_row = found[0];
  Cursor start;
  start_row(a, start, first_row);
  start.tile = u0 - found[1];
  if (tid == 0) {
    for (int i = 0; i < NV; ++i) {
      mbar_init(bar(kVFull + i), 8 * SB);          // one arrival per box
      mbar_init(bar(kVEmpty + i), 1);
    }
    for (int i = 0; i < NR; ++i) {
      mbar_init(bar(kRFull + i), 4);
      mbar_init(bar(kREmpty + i), 1);
    }
    mbar_init(bar(kQFull), kQThreads / 32);
    mbar_init(bar(kQEmpty), 1);
    mbar_init(bar(kSFull), 1);
    mbar_init(bar(kSFull + 1), 1);
    mbar_init(bar(kPFull), 4);                     // two: warp 1 may look at a tile's after the next tile's is there
    mbar_init(bar(kPFull + 1), 4);
    mbar_init(bar(kDrain), 1);
    mbar_init(bar(kDrain + 1), 1);
    *gave_up = (sV & 1023u) != 0u ? 1 : 0;
    mbar_fence_init();
    fence_proxy_async();
    tma_prefetch_desc(&pool_map);
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(P::kTmem) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tS = tmem + NB * N;      // O^T block b at b * N, scores of tile u at tS + (u & 1) * N
  // False once a wait has run out, here or elsewhere in the CTA: the role leaves.
  auto wait = [&](uint32_t b, uint32_t parity) -> bool {
    for (uint32_t i = 0; i < kMaxBarrierPolls; ++i) {
      if (mbar_try_wait(b, parity)) return true;
      if ((i & 255u) == 255u && *gave_up) return false;
    }
    *gave_up = 1;
    return false;
  };

  constexpr uint32_t kTypes = (1u << 4) | (1u << 7) | (1u << 10);                       // fp32 sums of bfloat16 products
  constexpr uint32_t IDESC_QK = kTypes | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(KT >> 4) << 24);
  constexpr uint32_t IDESC_PV = kTypes | (1u << 15) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | (8u << 24);     // both operands along their rows
  if (*gave_up) {
    // (shared memory does not start on a swizzle atom: reported below)
  } else if (warp == 0 || warp > 10) {
    // ---- copies.  A copy warp has 4 / CW pages of every tile; a lane issues the box of a page and slab.  (A box takes a warp 61 cycles to issue, 110 if one
    // thread issues them all: the 36 of a tile of 512 + 64 columns, 2200, were most of its 3250 cycles with one copy warp.) ----------------
    constexpr int PP = 4 / CW;
    const int cw = warp == 0 ? 0 : warp - 10, pg = cw * PP + lane % PP, sl = lane / PP;      // my page of a tile, my slab of a slot
    bool bad = false, ok = true;
    uint32_t slot = 0, use = 0, rslot = 0, ruse = 0;         // next slots and how often they were used
    Cursor c = start;
    int page = page_of(a, c, pg);
#pragma unroll 1
    for (int u = u0; u < u1 && ok; ++u) {
      if (page < 0 || page >= a.n_blocks) {
        bad = true;
        page = 0;
      }
#pragma unroll
      for (int b = 0; b < NB; b += SB) {
        if (use > 0) ok = ok && wait(bar(kVEmpty + slot), (use - 1) & 1u);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
          if (sl < 2 * SB) {
            mbar_expect_tx(bar(kVFull + slot), 2048);
            tma_load_2d_nohint(sV + slot * kSlot + sl * kSlab + pg * 2048, &pool_map, b * 128 + sl * 64, page * 16, bar(kVFull + slot));
          }
          if (++slot == NV) { slot = 0; ++use; }
        }
      }
      if (ruse > 0) ok = ok && wait(bar(kREmpty + rslot), (ruse - 1) & 1u);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        if (sl == 0) {
          mbar_expect_tx(bar(kRFull + rslot), 2048);
          tma_load_2d_nohint(sR + rslot * kSlab + pg * 2048, &pool_map, R, page * 16, bar(kRFull + rslot));
        }
        if (++rslot == NR) { rslot = 0; ++ruse; }
      }
      if (u + 1 < u1) {
        advance(a, c);
        page = page_of(a, c, pg);
      }
    }
    // leave only when every copy has landed
    for (uint32_t i = 0; i < NV; ++i)
      if ((use > 0 || i < slot) && !mbar_wait(bar(kVFull + i), (i < slot ? use : use - 1) & 1u)) *gave_up = 1;
    for (uint32_t i = 0; i < NR; ++i)
      if ((ruse > 0 || i < rslot) && !mbar_wait(bar(kRFull + i), (i < rslot ? ruse : ruse - 1) & 1u)) *gave_up = 1;
    if (bad) atomicOr(a.status, kStatusBadPageId);
  } else if (warp == 1) {
    // ---- scores.  Those of tile u go where the softmax has read tile u - 2's, which its weights imply ----------------------
    const uint64_t kd = smem_desc(sV, 16, 1024), rd = smem_desc(sR, 16, 1024), qd = smem_desc(sQ, 16, 1024);
    Cursor c = start;
    uint32_t slot = 0, use = 0, rslot = 0, ruse = 0, rows = 0;           // next slots and how often they were used; rows whose scores are done
    bool ok = true;
#pragma unroll 1
    for (int u = u0; u < u1 && ok; ++u) {
      const int k = u - u0;
      if (u == u0 || c.tile == 0) ok = ok && wait(bar(kQFull), rows & 1u);
      if (k >= 2) ok = ok && wait(bar(kPFull + (k & 1)), (uint32_t)((k - 2) >> 1) & 1u);
      const uint32_t d = tS + (uint32_t)(k & 1) * N;
#pragma unroll
      for (int b = 0; b < NB; b += SB) {
        ok = ok && wait(bar(kVFull + slot), use & 1u);
        tc_fence_after();
        __syncwarp();
#pragma unroll
        for (int i = 0; i < SB; ++i)
          tc_mma_ss8<StepsAlongK<kSlab, N * 128>>(d, kd + (uint64_t)(slot * (kSlot >> 4) + i * (2 * kSlab >> 4)),
                                                  qd + (uint64_t)((uint32_t)(b + i) * 2u * (N * 128 >> 4)), IDESC_QK, b + i ? 1u : 0u);
        if (++slot == NV) { slot = 0; ++use; }
      }
      ok = ok && wait(bar(kRFull + rslot), ruse & 1u);
      tc_fence_after();
      __syncwarp();
      tc_mma_ss4<StepsAlongK<kSlab, N * 128>>(d, rd + (uint64_t)(rslot * (kSlab >> 4)), qd + (uint64_t)((uint32_t)NB * 2u * (N * 128 >> 4)), IDESC_QK, 1u);
      tc_commit(bar(kSFull + (k & 1)));
      if (++rslot == NR) { rslot = 0; ++ruse; }
      if (c.tile + 1 == c.tiles || u + 1 == u1) {
        tc_commit(bar(kQEmpty));
        ++rows;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (u + 1 < u1) advance(a, c);
    }
    // every MMA is done before shared and tensor memory are given up
    __syncwarp();
    tc_commit(bar(kDrain));
    if (!mbar_wait(bar(kDrain), 0u)) *gave_up = 1;
  } else if (warp == 2) {
    // ---- values ---------------------------------------------------------------------------------------
    const uint64_t vd = smem_desc(sV, kSlab, 1024), pd = smem_desc(sP, 16, 1024);
    Cursor c = start;
    uint32_t slot = 0;
    bool ok = true;
#pragma unroll 1
    for (int u = u0; u < u1 && ok; ++u) {
      ok = __all_sync(0xffffffffu, wait(bar(kPFull + ((u - u0) & 1)), (uint32_t)((u - u0) >> 1) & 1u));       // (which implies that the tile is there)
      tc_fence_after();
      __syncwarp();
      const uint32_t fresh = u == u0 || c.tile == 0 ? 0u : 1u;
#pragma unroll
      for (int b = 0; b < NB; b += SB) {
#pragma unroll
        for (int i = 0; i < SB; ++i)
          tc_mma_ss4<StepsByRows>(tmem + (b + i) * N, vd + (uint64_t)(slot * (kSlot >> 4) + i * (2 * kSlab >> 4)), pd, IDESC_PV, fresh);
        tc_commit(bar(kVEmpty + slot));
        if (++slot == NV) slot = 0;
      }
      if (u + 1 < u1) advance(a, c);
    }
    __syncwarp();
    tc_commit(bar(kDrain + 1));
    if (!mbar_wait(bar(kDrain + 1), 0u)) *gave_up = 1;
  } else if (warp >= 4 && warp < 8) {
    // ---- softmax: a thread has one key (with its half of the heads); output: a thread has one latent column of every block ---------------
    const int wq = warp - 4, key = wq * 16 + (lane & 15), hh = (lane >> 4) * NH, own = own_head<NH>(lane);
    const uint32_t lanes = (uint32_t)(wq * 32) << 16;
    const float sc = a.scale * 1.4426950408889634f;
    float* my_refs = refs + wq * N;
    float* my_factors = factors + wq * N;
    // the 16-byte units of my key's row of P^T that hold my heads
    const uint32_t p_row = sP + (uint32_t)(key * 128);
    float m_run[OWN], l[NH];
#pragma unroll
    for (int i = 0; i < OWN; ++i) m_run[i] = -CUDART_INF_F;
#pragma unroll
    for (int i = 0; i < NH; ++i) l[i] = 0.f;
    Cursor c = start;
    int piece_tile0 = c.tile;
    // Tile k's products with V are done when its last slot is free.
    auto wait_values = [&](int k) -> bool {
      const uint32_t n = (uint32_t)((k + 1) * (NB / SB) - 1);
      return wait(bar(kVEmpty + n % NV), (n / NV) & 1u);
    };
    bool ok = true;                                // (after a wait that ran out this role goes on without waiting or arriving: its warps meet at a barrier)
#pragma unroll 1
    for (int u = u0; u < u1; ++u) {
      const int k = u - u0, buf = k & 1;
      ok = ok && wait(bar(kSFull + buf), (uint32_t)(k >> 1) & 1u);
      __syncwarp();
      if (ok && wq == 0 && lane == 0) mbar_arrive(bar(kREmpty + k % NR));       // (the rotated parts have been read)
      tc_fence_after();
      float s[NH];
      tc_ld_split<NH>(tS + lanes + buf * N, s);
      tc_wait_ld();
      const bool seen = c.tile * KT + key < c.n;
      float v[NH];
#pragma unroll
      for (int i = 0; i < NH; ++i) {
        s[i] = seen ? s[i] * sc : -CUDART_INF_F;
        v[i] = s[i];
      }
      spread_reduce<NH, true>(v, lane);
      float* part = red + buf * 4 * N;
#pragma unroll
      for (int i = 0; i < OWN; ++i) part[wq * N + own + i] = v[i];
      asm volatile("bar.sync 1, 128;" ::: "memory");
      bool grown = false;
#pragma unroll
      for (int i = 0; i < OWN; ++i) {
        const float* p = part + own + i;
        const float m_new = fmaxf(fmaxf(m_run[i], fmaxf(p[0], p[N])), fmaxf(p[2 * N], p[3 * N]));
        const float ref = m_new == -CUDART_INF_F ? 0.f : m_new;
        const float f = fast_exp2(m_run[i] - ref);   // 0 at the piece's first tile
        my_refs[own + i] = ref;
        my_factors[own + i] = f;
        grown |= f != 1.f;
        m_run[i] = m_new;
      }
      grown = __any_sync(0xffffffffu, grown);
      __syncwarp();                                // references and factors are there
      uint32_t pk[NH / 2];
#pragma unroll
      for (int i = 0; i < NH; i += 4) {
        const float4 r4 = *reinterpret_cast<const float4*>(my_refs + hh + i);
        s[i] = fast_exp2(s[i] - r4.x);
        s[i + 1] = fast_exp2(s[i + 1] - r4.y);
        s[i + 2] = fast_exp2(s[i + 2] - r4.z);
        s[i + 3] = fast_exp2(s[i + 3] - r4.w);
        pk[i / 2] = pack_bf162(s[i], s[i + 1]);
        pk[i / 2 + 1] = pack_bf162(s[i + 2], s[i + 3]);
      }
      if (grown) {
#pragma unroll
        for (int i = 0; i < NH; i += 4) {
          const float4 f4 = *reinterpret_cast<const float4*>(my_factors + hh + i);
          l[i] *= f4.x;
          l[i + 1] *= f4.y;
          l[i + 2] *= f4.z;
          l[i + 3] *= f4.w;
        }
      }
#pragma unroll
      for (int i = 0; i < NH; ++i) l[i] += s[i];
      if (k > 0) ok = ok && wait_values(k - 1);      // P's place is free, O holds the tiles before
      __syncwarp();
      if (grown && k > 0 && c.tile != piece_tile0) {
        tc_fence_after();
        constexpr int G = NB <= 2 || N == 64 ? 8 : 16;         // heads at a time
#pragma unroll 1
        for (int j = 0; j < N; j += G) {
          float f[G];
          bool any = false;
#pragma unroll
          for (int i = 0; i < G; i += 4) {
            const float4 f4 = *reinterpret_cast<const float4*>(my_factors + j + i);
            f[i] = f4.x; f[i + 1] = f4.y; f[i + 2] = f4.z; f[i + 3] = f4.w;
            any |= f4.x != 1.f || f4.y != 1.f || f4.z != 1.f || f4.w != 1.f;
          }
          if (__any_sync(0xffffffffu, any)) {
            float o[NB][G];
#pragma unroll
            for (int b = 0; b < NB; ++b) {
              if constexpr (G == 16) tc_ld16(tmem + lanes + b * N + j, o[b]);
              else tc_ld8(tmem + lanes + b * N + j, o[b]);
            }
            tc_wait_ld();
#pragma unroll
            for (int b = 0; b < NB; ++b) {
#pragma unroll
              for (int i = 0; i < G; ++i) o[b][i] *= f[i];
              if constexpr (G == 16) tc_st16(tmem + lanes + b * N + j, reinterpret_cast<const uint32_t(&)[16]>(o[b]));
              else tc_st8(tmem + lanes + b * N + j, reinterpret_cast<const uint32_t(&)[8]>(o[b]));
            }
          }
        }
        tc_wait_st();
      }
#pragma unroll
      for (int i = 0; i < NH / 8; ++i)
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(p_row + ((uint32_t)((hh / 8 + i) ^ (key & 7)) * 16)), "r"(pk[4 * i]), "r"(pk[4 * i + 1]),
                     "r"(pk[4 * i + 2]), "r"(pk[4 * i + 3])
                     : "memory");
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (ok && lane == 0) mbar_arrive(bar(kPFull + buf));
      // ---- end of a row or of my run ------------------------------------------------------------------
      const bool row_end = c.tile + 1 == c.tiles;
      if (row_end || u + 1 == u1) {
        const bool whole = row_end && piece_tile0 == 0;
        const int which = c.row == first_row ? 0 : 1;
        spread_reduce<NH, false>(l, lane);
#pragma unroll
        for (int i = 0; i < OWN; ++i) sums[wq * N + own + i] = l[i];
        asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
        for (int i = 0; i < OWN; ++i) {
          const float* p = sums + own + i;
          const float total = (p[0] + p[N]) + (p[2 * N] + p[3 * N]);
          const int head = h0 + own + i;
          float f = 1.f;
          if (head < a.heads) {
            if (whole) {
              f = total > 0.f ? 1.f / total : 0.f;
              if (a.gate != nullptr) f *= sigmoid_f(to_f(static_cast<const bf16*>(a.gate)[(long long)c.row * a.gate_stride + head]));
            } else if (wq == 0) {
              float* ml = a.part_ml + (((long long)cta * 2 + which) * a.heads + head) * 2;
              ml[0] = m_run[i];
              ml[1] = total;
            }
          }
          my_factors[own + i] = f;
          m_run[i] = -CUDART_INF_F;
        }
        __syncwarp();
        ok = ok && wait_values(k);
        __syncwarp();
        tc_fence_after();
        const int col = wq * 32 + lane;
#pragma unroll 1
        for (int j = 0; j < N; j += 8) {
          if (h0 + j >= a.heads) break;
          float o[NB][8];
#pragma unroll
          for (int b = 0; b < NB; ++b) tc_ld8(tmem + lanes + b * N + j, o[b]);
          tc_wait_ld();
          if (whole) {
            bf16* out = static_cast<bf16*>(a.out) + ((long long)c.row * a.heads + h0 + j) * R + (col & ~1);
            const bool odd = lane & 1;
#pragma unroll
            for (int i = 0; i < 8; i += 2) {       // the even thread of two stores both columns of head j + i, the odd one those of the next head
              const float f0 = my_factors[j + i], f1 = my_factors[j + i + 1];
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                const float x = o[b][i] * f0, y = o[b][i + 1] * f1;
                const float got = __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
                if (h0 + j + i + odd < a.heads)
                  *reinterpret_cast<uint32_t*>(out + (long long)(i + odd) * R + b * 128) = odd ? pack_bf162(got, y) : pack_bf162(x, got);
              }
            }
          } else {
            float* out = a.part_o + (((long long)cta * 2 + which) * a.heads + h0 + j) * R + col;
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (h0 + j + i < a.heads)
#pragma unroll
                for (int b = 0; b < NB; ++b) out[(long long)i * R + b * 128] = o[b][i];
          }
        }
        tc_fence_before();
        __syncwarp();                              // the factors have been read
#pragma unroll
        for (int i = 0; i < NH; ++i) l[i] = 0.f;
        piece_tile0 = 0;
      }
      if (u + 1 < u1) advance(a, c);
    }
  } else {
    // ---- queries: 16-byte units of the row's latent parts wait in registers until the scores of the row before are done; rotated parts --------------
    const int qi = warp == 3 ? lane : tid - 224;     // 0 .. 127
    constexpr int UNITS = NB * 16, NQ = N * UNITS / kQThreads;
    constexpr int NW = NQ > 18 ? NQ / 2 : NQ;      // those that wait in registers
    constexpr int NROT = (N * 4 + kQThreads - 1) / kQThreads;          // pairs of units: 8 frequencies of a head
    const int half = a.rot_dim / 2, hu = half / 8;
    auto place = [&](int head, int u) -> uint32_t { return sQ + (uint32_t)((u >> 3) * (N * 128) + head * 128 + (((u ^ head) & 7) * 16)); };
    auto put = [&](uint32_t dst, const uint4& v) {
      asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
    };
    for (int i = qi; i < N * 8; i += kQThreads)    // columns past the rotated part stay zero, and so do heads past the last
      put(place(i >> 3, UNITS + (i & 7)), make_uint4(0, 0, 0, 0));
    asm volatile("bar.sync 2, 128;" ::: "memory");
    int row = first_row, left = u1 - u0 + start.tile;        // units from this row's first one to the end of the run
#pragma unroll 1
    for (uint32_t r = 0;; ++r, ++row) {
      uint4 v[NW];
      auto fetch = [&](int i0) {
#pragma unroll
        for (int i = 0; i < NW; ++i) {
          const int idx = qi + (i0 + i) * kQThreads, head = h0 + idx / UNITS;
          v[i] = head < a.heads ? __ldg(reinterpret_cast<const uint4*>(static_cast<const bf16*>(a.q_abs) + ((long long)row * a.heads + head) * R) + idx % UNITS)
                                : make_uint4(0, 0, 0, 0);
        }
      };
      auto store = [&](int i0) {
#pragma unroll
        for (int i = 0; i < NW; ++i) {
          const int idx = qi + (i0 + i) * kQThreads;
          put(place(idx / UNITS, idx % UNITS), v[i]);
        }
      };
      fetch(0);
      uint4 lo[NROT], hi[NROT];
#pragma unroll
      for (int i = 0; i < NROT; ++i) {
        const int idx = qi + i * kQThreads, head = h0 + idx / 4, f0 = (idx & 3) * 8;
        if (idx < N * 4 && head < a.heads && f0 < half) {
          const bf16* q = static_cast<const bf16*>(a.q) + ((long long)row * a.heads + head) * a.q_stride + a.q_off + f0;
          float x[8], y[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float cs = a.cos_t[(long long)row * half + f0 + j], sn = a.sin_t[(long long)row * half + f0 + j];
            const float p = to_f(q[j]), w = to_f(q[half + j]);
            x[j] = p * cs - w * sn;
            y[j] = w * cs + p * sn;
          }
          lo[i] = make_uint4(pack_bf162(x[0], x[1]), pack_bf162(x[2], x[3]), pack_bf162(x[4], x[5]), pack_bf162(x[6], x[7]));
          hi[i] = make_uint4(pack_bf162(y[0], y[1]), pack_bf162(y[2], y[3]), pack_bf162(y[4], y[5]), pack_bf162(y[6], y[7]));
        }
      }
      if (r > 0) {                                 // (a long wait: it sleeps between its looks, which would take cycles from the other warps)
        bool there = false;
        for (uint32_t i = 0; i < kMaxBarrierPolls / 8 && !there && *gave_up == 0; ++i) {
          there = mbar_test_wait(bar(kQEmpty), (r - 1) & 1u) != 0u;
          if (!there) __nanosleep(200);
        }
        if (!there) *gave_up = 1;
        if (!__all_sync(0xffffffffu, there)) break;
      }
      store(0);
      if constexpr (NW < NQ) {
        fetch(NW);
        store(NW);
      }
#pragma unroll
      for (int i = 0; i < NROT; ++i) {
        const int idx = qi + i * kQThreads, head = idx / 4, f = idx & 3;
        if (idx < N * 4 && h0 + head < a.heads && f < hu) {
          put(place(head, UNITS + f), lo[i]);
          put(place(head, UNITS + hu + f), hi[i]);
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kQFull));
      left -= row_tiles_of(a, row);
      if (left <= 0) break;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *gave_up) atomicOr(a.status, kStatusWaitTimeout);
  if (warp == 2) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(P::kTmem) : "memory");
  }
}

template <int NB, int N>
cudaError_t launch_t(const LatentAttentionArgs& a, const CUtensorMap& map, cudaStream_t s) {
  constexpr int smem = Plan<NB, N>::kSmem;
  static SharedMemoryLimit limit;
  cudaError_t e = limit.raise(reinterpret_cast<const void*>(latent_decode_tc5_kernel<NB, N>), smem);
  if (e != cudaSuccess) return e;
  latent_decode_tc5_kernel<NB, N><<<dim3((unsigned)a.n_cta, (unsigned)((a.heads + N - 1) / N)), Plan<NB, N>::kThreads, smem, s>>>(map, a);
  return cudaGetLastError();
}
template <int NB>
cudaError_t launch_n(const LatentAttentionArgs& a, const CUtensorMap& map, cudaStream_t s) {
  switch (a.block_heads) {
    case 16: return launch_t<NB, 16>(a, map, s);
    case 32: return launch_t<NB, 32>(a, map, s);
    default: return launch_t<NB, 64>(a, map, s);
  }
}

}  // namespace

bool latent_decode_tc5_supported(int kv_rank, int rot_dim) {
  return kv_rank % 128 == 0 && kv_rank <= 512 && rot_dim > 0 && rot_dim <= 64 && rot_dim % 16 == 0;
}

int latent_decode_tc5_ctas(int heads, int kv_rank, int block_heads, int sm_count) {
  const int blocks = (heads + block_heads - 1) / block_heads, per_sm = kv_rank <= 256 && block_heads <= 32 ? 2 : 1;
  const int n = sm_count * per_sm / blocks;
  return n > 0 ? n : 1;
}

cudaError_t launch_latent_decode_tc5(const LatentAttentionArgs& a, const CUtensorMap& map, cudaStream_t s) {
  switch (a.kv_rank / 128) {
    case 1: return launch_n<1>(a, map, s);
    case 2: return launch_n<2>(a, map, s);
    case 3: return launch_n<3>(a, map, s);
    default: return launch_n<4>(a, map, s);
  }
}

}  // namespace hybrid
}  // namespace fa
