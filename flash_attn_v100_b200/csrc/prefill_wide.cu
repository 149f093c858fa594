// Causal / non-causal GQA prefill of wide heads (128 < D <= 256) on tcgen05, sm_100a.
//
// Replaces the reference's prefill kernels (flash_attn_kernel.cu:1138-1299, 2471-2605, 3005-3148) for those head dimensions, dense
// [B,H,N,D] and packed varlen [total,H,D], fp16 operands.
//
// What bounds it: the softmax of a step, then the tensor cores.  A step of 128 rows x 128 keys is 1024 cycles of QK and 2048 of PV at D = 256 (the
// weights and their rests, below) against 1024 cycles of exponentials, so one 128-row query tile per CTA keeps the tensor pipe busy if the softmax
// of one step runs under the MMAs of its neighbours; and one tile is what tensor memory holds (an output of 256 columns and two score buffers of 128 fill
// its 512).  The issue order is QK(j+1), PV(j), QK(j+2), ...: from the end of QK(j) to the start of PV(j) the softmax has the length of PV(j-1) and
// QK(j+1).  P is handed over in two halves of 64 keys, so that PV(j) starts while the second half is exponentiated.
//
// Weights in two fp16 terms.  A row's reference exponent lags behind its maximum (see the softmax), so the largest weight is not exactly 1, as it is
// under an exact running maximum, and rounding the weights to fp16 alone costs 2 to 4 % of the error against 64 bits, 20 % with peaked scores, above the mma.sync
// kernel's.  What the rounding leaves is a second operand beside the first: 0.73 to 0.94 of the mma.sync kernel's error, for 128 to 8192 tokens,
// 136 to 256 columns, flat and peaked scores.  The other way, an exact maximum with O scaled in tensor memory before every PV, is as slow: PV, scale, PV is a
// serial chain (1 x 4096 tokens, 16 heads on 8, not causal: 375 us; two terms 374; one term 252).
//
// Measured: 2 x 2048 tokens, 16 heads on 8 of 256, causal: 112 us against 401 of the mma.sync kernel (prefill_mma.cu); 1 x 2048 48 and 229.  The smallest launch takes 12 us.  Releasing every unit with a commit of its own, earlier, changed nothing.
//
// Warps: 0 copies (TMA), 1 issues the MMAs, 2 owns tensor memory and takes work items, 4-7 and 8-11 softmax of the even and of the odd steps (a
// thread per row, its 128 scores in registers), 12-15 write the output of a finished tile while the softmax is on the next one.  (With one
// softmax group a step took 3800 cycles: a single warp per scheduler waits for its own loads, maxima and stores.)  Shared memory: Q (64 KB) and a ring of
// five units of 32 KB.  A K unit is 128 keys x 128 columns (QK accumulates over two units), a V unit 64 keys x all columns, so that every
// MMA has its full N and units of both kinds fill one ring in the order of use.  No barrier is committed for a unit: the copy lane waits for
// the MMA batch that read it (a tcgen05.commit costs the tensor pipe about as much as an MMA).
#include "prefill.cuh"
#include "prefill_tc5_kernel.cuh"
#include "smem_limit.cuh"

namespace fa {

namespace {

constexpr int kWideThreads = 512;
constexpr int kUnits = 5;
constexpr int kUnitBytes = 32 * 1024;
constexpr int kSlabK = 128 * 128, kSlabV = 64 * 128;      // bytes of 64 columns of a K (or Q) and of a V unit
constexpr int kQBytes = 64 * 1024;
constexpr int kWideItemQ = 4;
constexpr int kWideConsumers = 1 + 1 + 8 + 4;             // copy lane, MMA warp, softmax and output warps
enum WideBar { kQFull = 0, kUFull = 1, kSFull = kUFull + kUnits, kPLo = kSFull + 2, kPHi = kPLo + 2, kODone = kPHi + 2, kOEmpty = kODone + 2, kLFull, kMReady,
               kIFull = kMReady + 2, kIEmpty = kIFull + kWideItemQ, kClaim = kIEmpty + kWideItemQ, kTaken, kWideBars };
constexpr int kWideSmem = kQBytes + kUnits * kUnitBytes + 16 + kWideBars * 8 + kWideItemQ * 16 + 4 * 128 * 4 + 16;
static_assert(kWideSmem <= 227 * 1024, "shared memory plan exceeds the SM");

struct WideParams {
  __half* out;
  const int32_t* cu_seqlens;
  int batch, H_Q, H_KV, N, max_seqlen;
  long long total;
  long long o_batch_stride, o_head_stride, o_tok_stride;
  int causal, D_real, dense, out_bf16;
  int n_rb;                                // row blocks of the item grid (items = n_rb * batch * H_Q)
  long long n_grid;                        // items that the grid is made for (items_of_grid)
  int take_over;                           // CTAs go on with the items of CTAs that have not started (see take_item)
  int* status;
  float scale_log2;
};

struct WideItem {
  int head, row0, len, n_kv, seq;
  int q_c1, q_c2, kv_c1, kv_c2;
  long long tok0;
};

// (The heads of a group are neighbours in the order of the items, so they read K and V from L2 together.)
__device__ __forceinline__ void wide_item(const WideParams& p, const ItemPlace& at, WideItem& it) {
  it.head = at.hg;
  it.seq = at.seq;
  it.row0 = at.rb * 128;
  const int h_kv = it.head / (p.H_Q / p.H_KV);
  if (p.cu_seqlens != nullptr) {
    int a;
    it.len = packed_rows(p, it.seq, a);
    it.tok0 = a;
  } else {
    it.tok0 = 0;
    it.len = p.N;
  }
  const int kv_end = p.causal && it.row0 + 128 < it.len ? it.row0 + 128 : it.len;
  it.n_kv = (kv_end + 127) / 128;
  if (p.dense) {
    it.q_c1 = it.kv_c1 = 0;
    it.q_c2 = (it.seq * p.H_Q + it.head) * p.N + it.row0;
    it.kv_c2 = (it.seq * p.H_KV + h_kv) * p.N;
  } else {
    it.q_c1 = it.head;
    it.kv_c1 = h_kv;
    it.q_c2 = (int)it.tok0 + it.row0;
    it.kv_c2 = (int)it.tok0;
  }
}

// One 32-column chunk of a score row: P = exp2(s * scale - m) in two fp16 terms, the weight and what its rounding left, written to tensor memory
// at `taddr` and 32 columns on (16 columns each); the fp32 sum of the chunk is added to `rs`.
__device__ __forceinline__ void exp_chunk_two(const float (&s)[32], float2 sc2, float2 nm2, float2& rs, uint32_t taddr) {
  uint32_t hi[16], lo[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float2 x = ffma2(make_float2(s[2 * i], s[2 * i + 1]), sc2, nm2);
    const float2 e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
    rs = fadd2(rs, e);
    hi[i] = pack_half2(e.x, e.y);
    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&hi[i]));
    lo[i] = pack_half2(e.x - h.x, e.y - h.y);
  }
  tc_st16(taddr, hi);
  tc_st16(taddr + 32, lo);
}

__global__ void __launch_bounds__(kWideThreads, 1)
prefill_wide_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
                    const __grid_constant__ CUtensorMap vmap, const WideParams p) {
  extern __shared__ __align__(1024) uint8_t smem_wide[];     // (no room for a slack: the only shared memory, so it starts aligned)
  uint8_t* smem = smem_wide;
  const uint32_t sQ = smem_u32(smem), sU = sQ + kQBytes;
  if ((sQ & 1023u) != 0u) {
    wait_for_clear();
    if (threadIdx.x == 0) atomicOr(p.status, kStatusWaitTimeout);
    return;
  }
  const uint32_t reply = sU + kUnits * kUnitBytes;             // of take_item
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kQBytes + kUnits * kUnitBytes + 16);
  volatile int* item_slot = reinterpret_cast<volatile int*>(bars + kWideBars);   // [kWideItemQ][4]
  float* l_rows = reinterpret_cast<float*>(bars + kWideBars + 2 * kWideItemQ);   // [softmax group][row]: parts of the row sums
  float* m_rows = l_rows + 256;                                                  // [step & 1][row]: reference exponents
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(m_rows + 256);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  auto bar = [&](int i) -> uint32_t { return smem_u32(bars + i); };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_slab = (p.D_real + 63) >> 6;         // 3 or 4 slabs of 64 columns

  if (threadIdx.x == 0) {
    mbar_init(bar(kQFull), 1);
    for (int i = 0; i < kUnits; ++i) mbar_init(bar(kUFull + i), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar(kSFull + b), 1);
      mbar_init(bar(kPLo + b), 4);
      mbar_init(bar(kPHi + b), 4);
      mbar_init(bar(kMReady + b), 4);
      mbar_init(bar(kODone + b), 1);
    }
    mbar_init(bar(kOEmpty), 4);
    mbar_init(bar(kClaim), 1);
    mbar_init(bar(kTaken), 1);
    mbar_init(bar(kLFull), 8);
    for (int i = 0; i < kWideItemQ; ++i) {
      item_slot[4 * i] = -1;                       // (a role that gave up waiting reads a place that is none, or an earlier one)
      mbar_init(bar(kIFull + i), 1);
      mbar_init(bar(kIEmpty + i), kWideConsumers);
    }
    *abort_flag = 0;
    mbar_fence_init();
    fence_proxy_async();
    tma_prefetch_desc(&qmap);
    tma_prefetch_desc(&kmap);
    tma_prefetch_desc(&vmap);
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;                // S_0 [0,128) S_1 [128,256) O [256,512); P over its S: per 64 keys 32 columns and 32 of their rests
  auto next_item = [&](uint32_t ic) -> ItemPlace {
    const int slot = ic % kWideItemQ;
    wait_or_abort(bar(kIFull + slot), (ic / kWideItemQ) & 1u, abort_flag);
    return read_place(item_slot + 4 * slot);
  };
  auto release_item = [&](uint32_t ic) { mbar_arrive(bar(kIEmpty + (int)(ic % kWideItemQ))); };

  // Running numbers, the same in every role: ic items, cnt KV steps of all items so far (S buffer cnt & 1; SFull, PLo, PHi and
  // ODone of step cnt complete phase cnt >> 1 of barrier cnt & 1), un units of the ring.  Waits by phase parity are safe: no role can fall two
  // phases behind, because step cnt + 2 needs what the role that waits for step cnt does next (a unit, a half of P, an emptied O).
  if (warp == 0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (lane == 0) {
      uint32_t cnt = 0, un = 0;
      // what the units of the ring hold: step << 1 | (0: K, read by QK(step); 1: V, read by PV(step)), as a small shift register
      uint32_t held[kUnits];
#pragma unroll
      for (int i = 0; i < kUnits; ++i) held[i] = 0;
      uint32_t q_cnt = 0;
      auto claim = [&](uint32_t what) -> uint32_t {          // a place for the next unit, once its last reader is done
        if (un >= kUnits) {
          const uint32_t c = held[0] >> 1;
          wait_or_abort(bar(((held[0] & 1u) ? kODone : kSFull) + (int)(c & 1u)), (c >> 1) & 1u, abort_flag);
        }
#pragma unroll
        for (int i = 0; i + 1 < kUnits; ++i) held[i] = held[i + 1];
        held[kUnits - 1] = what;
        return un++ % kUnits;
      };
      for (uint32_t ic = 0;; ++ic) {
        if (*abort_flag) break;
        const ItemPlace item = next_item(ic);
        release_item(ic);
        if (item.rb < 0) break;
        WideItem it;
        wide_item(p, item, it);
        if (cnt > 0) wait_or_abort(bar(kSFull + ((cnt - 1) & 1u)), ((cnt - 1) >> 1) & 1u, abort_flag);   // Q has been read
        mbar_expect_tx(bar(kQFull), n_slab * kSlabK);
        for (int s = 0; s < n_slab; ++s) tma_load_3d(sQ + s * kSlabK, &qmap, s * 64, it.q_c1, it.q_c2, bar(kQFull));
        ++q_cnt;
        auto load_k = [&](int j) {
          for (int half = 0; half < 2; ++half) {
            const uint32_t u = claim((cnt + j) << 1);
            const int s1 = half == 0 ? 2 : n_slab;
            mbar_expect_tx(bar(kUFull + u), (s1 - 2 * half) * kSlabK);
            for (int s = 2 * half; s < s1; ++s)
              tma_load_3d(sU + u * kUnitBytes + (s - 2 * half) * kSlabK, &kmap, s * 64, it.kv_c1, it.kv_c2 + j * 128, bar(kUFull + u));
          }
        };
        auto load_v = [&](int j) {
          for (int half = 0; half < 2; ++half) {
            const uint32_t u = claim((cnt + j) << 1 | 1u);
            mbar_expect_tx(bar(kUFull + u), n_slab * kSlabV);
            for (int s = 0; s < n_slab; ++s)
              tma_load_3d(sU + u * kUnitBytes + s * kSlabV, &vmap, s * 64, it.kv_c1, it.kv_c2 + j * 128 + half * 64, bar(kUFull + u));
          }
        };
        load_k(0);
        for (int j = 0; j < it.n_kv; ++j) {
          if (j == (it.n_kv > 2 ? it.n_kv - 3 : 0)) mbar_arrive(bar(kClaim));
          if (j + 1 < it.n_kv) load_k(j + 1);
          load_v(j);
        }
        cnt += (uint32_t)it.n_kv;
      }
      // every copy has landed before shared memory is given up
      for (uint32_t i = 0; i < kUnits; ++i)
        if (un > i) drain_wait(bar(kUFull + i), ((un - 1 - i) / kUnits) & 1u, abort_flag);
      if (q_cnt > 0) drain_wait(bar(kQFull), (q_cnt - 1) & 1u, abort_flag);
    }
  } else if (warp == 1) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    constexpr uint32_t IDESC_QK = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t idesc_pv = (1u << 4) | (1u << 16) | ((uint32_t)(n_slab * 8) << 17) | ((128u >> 4) << 24);
    const uint64_t qd = smem_desc(sQ, 16, 1024), kd = smem_desc(sU, 16, 1024), vd = smem_desc(sU, kSlabV, 1024);
    uint32_t cnt = 0, un = 0;
    uint32_t ic = 0;
    for (;; ++ic) {
      if (*abort_flag) break;
      const ItemPlace item = next_item(ic);
      __syncwarp();
      if (lane == 0) release_item(ic);
      if (item.rb < 0) break;
      WideItem it;
      wide_item(p, item, it);
      auto take_unit = [&]() -> uint32_t {
        const uint32_t u = un % kUnits;
        wait_or_abort(bar(kUFull + u), (un / kUnits) & 1u, abort_flag);
        ++un;
        return u;
      };
      auto issue_qk = [&](uint32_t c) {
        const uint32_t d = tmem + (c & 1u) * 128u;
        for (int half = 0; half < 2; ++half) {
          const uint32_t u = take_unit();
          tc_fence_after();
          __syncwarp();
          const uint64_t a = qd + (uint64_t)((uint32_t)half * 2u * (kSlabK >> 4)), b = kd + (uint64_t)(u * (kUnitBytes >> 4));
          if (half == 0 || n_slab == 4) tc_mma_ss8<StepsAlongK<kSlabK, kSlabK>>(d, a, b, IDESC_QK, (uint32_t)half);
          else tc_mma_ss4<StepsAlongK<kSlabK, kSlabK>>(d, a, b, IDESC_QK, 1u);
        }
        tc_commit(bar(kSFull + (c & 1u)));
      };
      wait_or_abort(bar(kQFull), ic & 1u, abort_flag);
      issue_qk(cnt);
      for (int j = 0; j < it.n_kv; ++j, ++cnt) {
        if (j + 1 < it.n_kv) issue_qk(cnt + 1);
        if (j == 0 && ic > 0) wait_or_abort(bar(kOEmpty), (ic - 1) & 1u, abort_flag);
        for (int half = 0; half < 2; ++half) {
          const uint32_t u = take_unit();
          // rows past the end of the sequence: zeros, since what lies there (another sequence) may not be a number and 0 * NaN is NaN
          const int rows = it.len - (j * 128 + half * 64);
          if (rows < 64) {
            uint8_t* v = smem + kQBytes + u * kUnitBytes + (lane >> 3) * kSlabV + (lane & 7) * 16;
            if ((lane >> 3) < n_slab)
              for (int r = rows > 0 ? rows : 0; r < 64; ++r) *reinterpret_cast<uint4*>(v + r * 128) = make_uint4(0u, 0u, 0u, 0u);
            fence_proxy_async();
          }
          wait_or_abort(bar((half ? kPHi : kPLo) + (int)(cnt & 1u)), (cnt >> 1) & 1u, abort_flag);
          tc_fence_after();
          __syncwarp();
          const uint32_t a = tmem + (cnt & 1u) * 128u + (uint32_t)half * 64u;
          // the weights, and their rests, by the same rows of V
          tc_mma_ts8<StepsTmemA<4>>(tmem + 256u, a, vd + (uint64_t)(u * (kUnitBytes >> 4)), idesc_pv, (j | half) ? 1u : 0u);
        }
        tc_commit(bar(kODone + (int)(cnt & 1u)));
      }
    }
    // The commits of the last step cover every MMA issued; on a regular exit that step's batch is the last phase of ODone.
    if (cnt > 0) drain_wait(bar(kODone + (int)((cnt - 1) & 1u)), ((cnt - 1) >> 1) & 1u, abort_flag);
  } else if (warp == 2) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    ItemWalk walk;
    auto blocks_of = [&](int s) {
      int a;
      return (packed_rows(p, s, a) + 127) / 128;
    };
    uint32_t taken = 0;
    auto take = [&]() { return p.take_over ? take_item(reply, bar(kTaken), taken, abort_flag) : -1ll; };
    const bool packed = p.cu_seqlens != nullptr;
    if (packed) walk.start(p.batch, blocks_of);
    const long long count = packed ? walk.blocks * p.H_Q : p.n_grid;
    long long number = first_item();
    for (uint32_t ic = 0;; ++ic) {
      if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
      // an item is taken when the copies of the last steps of the one before begin: taken earlier, items were dealt out in turn, whatever they cost
      if (ic > 0) wait_or_abort(bar(kClaim), (ic - 1) & 1u, abort_flag);
      __syncwarp();
      const ItemPlace at = next_place(walk, ic == 0, number, count, p.n_grid, packed, p.n_rb, p.batch, p.H_Q, take, blocks_of);
      const int slot = ic % kWideItemQ;
      if (ic >= kWideItemQ) wait_or_abort(bar(kIEmpty + slot), ((ic / kWideItemQ) & 1u) ^ 1u, abort_flag);
      __syncwarp();
      if (lane == 0) {
        write_place(item_slot + 4 * slot, at);
        mbar_arrive(bar(kIFull + slot));
      }
      __syncwarp();
      if (at.rb < 0) break;
    }
  } else if (warp == 3) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  } else if (warp < 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 176;");
    // ---- softmax: thread = row.  m is the reference exponent of the row (raised, with O rescaled, when the maximum grows by more than
    // 2^8: P stays within fp16, and a stale reference cancels in O / l up to the rounding of P, which the second term takes in); l is this group's part of the row sum, relative to its last m.  The
    // groups take turns: a step's reference comes from the step before through shared memory, as soon as that step has its maximum.
    const int grp = (warp - 4) >> 2, wq = warp & 3;
    const int row = wq * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(wq * 32) << 16);
    const uint32_t tS = lanes + (uint32_t)grp * 128u;
    const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
    uint32_t cnt0 = 0;
    for (uint32_t ic = 0;; ++ic) {
      if (*abort_flag) break;
      const ItemPlace item = next_item(ic);
      __syncwarp();
      if (lane == 0) release_item(ic);
      if (item.rb < 0) break;
      WideItem it;
      wide_item(p, item, it);
      const int grow = it.row0 + row;
      float m = -INFINITY;
      float2 l2 = make_float2(0.f, 0.f);
      for (int j = (int)((cnt0 ^ (uint32_t)grp) & 1u); j < it.n_kv; j += 2) {
        const uint32_t cnt = cnt0 + (uint32_t)j, ph = (cnt >> 1) & 1u;
        wait_or_abort(bar(kSFull + grp), ph, abort_flag);
        tc_fence_after();
        float s[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tc_ld32(tS + c * 32, s[c]);
        tc_wait_ld();
        const int k0 = j * 128;
        if (k0 + 128 > it.len || (p.causal && k0 + 127 > it.row0)) {
          int lim = it.len - k0;
          if (p.causal && grow - k0 + 1 < lim) lim = grow - k0 + 1;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i >= lim) s[c][i] = -INFINITY;
        }
        float a[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) a[c] = fmaxf(s[c][0], s[c][1]);
#pragma unroll
        for (int i = 2; i < 32; i += 2)
#pragma unroll
          for (int c = 0; c < 4; ++c) a[c] = fmax3(a[c], s[c][i], s[c][i + 1]);
        const float mx = fmaxf(fmaxf(a[0], a[1]), fmaxf(a[2], a[3])) * p.scale_log2;
        float m_ref = mx;                              // the reference of this step
        if (j > 0) {
          wait_or_abort(bar(kMReady + (grp ^ 1)), ((cnt - 1) >> 1) & 1u, abort_flag);
          const float m_prev = m_rows[(grp ^ 1) * 128 + row];
          const bool raise = mx > m_prev + 8.f;
          if (!raise) m_ref = m_prev;
          m_rows[grp * 128 + row] = m_ref;
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(kMReady + grp));
          if (__any_sync(0xffffffffu, raise)) {
            const float alpha = raise ? fast_exp2(m_prev - mx) : 1.f;
            wait_or_abort(bar(kODone + (grp ^ 1)), ((cnt - 1) >> 1) & 1u, abort_flag);
            tc_fence_after();
            for (int c = 0; c < n_slab * 8; ++c) {
              float o[8];
              tc_ld8(lanes + 256u + c * 8, o);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] *= alpha;
              tc_st8(lanes + 256u + c * 8, reinterpret_cast<const uint32_t(&)[8]>(o));
            }
          }
        } else {
          m_rows[grp * 128 + row] = m_ref;
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(kMReady + grp));
        }
        if (m_ref != m) {                              // (from -inf at the group's first step: the sum is zero)
          const float f = fast_exp2(m - m_ref);
          l2 = m == -INFINITY ? make_float2(0.f, 0.f) : make_float2(l2.x * f, l2.y * f);
          m = m_ref;
        }
        const float neg_m = m == -INFINITY ? 0.f : -m;
        const float2 nm2 = make_float2(neg_m, neg_m);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          exp_chunk_two(s[c], sc2, nm2, l2, tS + (c >> 1) * 64 + (c & 1) * 16);
          if (c & 1) {
            tc_wait_st();                              // O's rescale as well
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar((c == 1 ? kPLo : kPHi) + grp));
          }
        }
      }
      cnt0 += (uint32_t)it.n_kv;
      float l = l2.x + l2.y;
      if (it.n_kv > 1 && ((cnt0 - 1u) & 1u) != (uint32_t)grp) {      // O is relative to the other group's last reference
        wait_or_abort(bar(kMReady + (grp ^ 1)), ((cnt0 - 1u) >> 1) & 1u, abort_flag);
        const float m_last = m_rows[(grp ^ 1) * 128 + row];
        if (m_last != m) l = m == -INFINITY ? 0.f : l * fast_exp2(m - m_last);
      }
      if (ic > 0) wait_or_abort(bar(kOEmpty), (ic - 1u) & 1u, abort_flag);       // the previous item's sums have been read
      l_rows[grp * 128 + row] = l;
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(kLFull));
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    // ---- output: O / l -> 16 bits -> global; eight lanes store 128 contiguous bytes of a row (see prefill_tc5_kernel.cuh)
    const int wq = warp & 3, row = wq * 32 + lane;
    const uint32_t tO = tmem + 256u + ((uint32_t)(wq * 32) << 16);
    uint32_t cnt = 0;
    wait_for_clear();
    for (uint32_t ic = 0;; ++ic) {
      if (*abort_flag) break;
      const ItemPlace item = next_item(ic);
      __syncwarp();
      if (lane == 0) release_item(ic);
      if (item.rb < 0) break;
      WideItem it;
      wide_item(p, item, it);
      cnt += (uint32_t)it.n_kv;
      wait_or_abort(bar(kLFull), ic & 1u, abort_flag);
      const float l = l_rows[row] + l_rows[128 + row];
      const float inv = l > 0.f ? 1.f / l : 0.f;
      wait_or_abort(bar(kODone + (int)((cnt - 1) & 1u)), ((cnt - 1) >> 1) & 1u, abort_flag);
      tc_fence_after();
      __half* obase = p.dense ? p.out + (long long)it.seq * p.o_batch_stride : p.out + it.tok0 * p.o_tok_stride;
      obase += (long long)it.head * p.o_head_stride;
      const int gi = lane & 7;
      for (int c = 0; c < n_slab; ++c) {
        uint32_t u[8][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float o[32];
          tc_ld32(tO + c * 64 + h * 32, o);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) u[h * 4 + (i >> 2)][i & 3] = pack_out16x2(o[2 * i] * inv, o[2 * i + 1] * inv, p.out_bf16 != 0);
        }
        if (c + 1 == n_slab) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(kOEmpty));
        }
#pragma unroll
        for (int sft = 4; sft >= 1; sft >>= 1) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            if (k & sft) continue;
            const bool up = (gi & sft) != 0;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const uint32_t send = up ? u[k][w] : u[k | sft][w];
              const uint32_t got = __shfl_xor_sync(0xffffffffu, send, sft);
              if (up) u[k][w] = got; else u[k | sft][w] = got;
            }
          }
        }
        const int col = c * 64 + gi * 8;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int r = it.row0 + wq * 32 + (lane - gi) + k;
          if (r < it.len && col < p.D_real)
            *reinterpret_cast<uint4*>(obase + (long long)r * p.o_tok_stride + col) = make_uint4(u[k][0], u[k][1], u[k][2], u[k][3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicOr(p.status, kStatusWaitTimeout);
  if (warp == 2) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

}  // namespace

bool prefill_wide_supported(const PrefillParams& p) {
  const long long qrows = p.cu_seqlens ? p.total : (long long)p.batch * p.H_Q * p.N;
  return p.D_real > 128 && p.D_real <= 256 && p.D_real % 8 == 0 && !p.in_bf16 && qrows < (1ll << 31);
}

cudaError_t launch_prefill_wide(const PrefillParams& pp, int sm_count, void* encode_fn, cudaStream_t stream) {
  EncodeTiledFn enc = reinterpret_cast<EncodeTiledFn>(encode_fn);
  const bool dense = pp.cu_seqlens == nullptr;
  const int Dr = pp.D_real;
  CUtensorMap qmap, kmap, vmap;
  bool ok;
  if (dense) {
    const long long qrows = (long long)pp.batch * pp.H_Q * pp.N, krows = (long long)pp.batch * pp.H_KV * pp.N;
    ok = make_map3(enc, &qmap, pp.q, Dr, 1, qrows, Dr, Dr) && make_map3(enc, &kmap, pp.k, Dr, 1, krows, Dr, Dr) &&
         make_map3(enc, &vmap, pp.v, Dr, 1, krows, Dr, Dr, 64);
  } else {
    ok = make_map3(enc, &qmap, pp.q, Dr, pp.H_Q, pp.total, Dr, (long long)pp.H_Q * Dr) &&
         make_map3(enc, &kmap, pp.k, Dr, pp.H_KV, pp.total, Dr, (long long)pp.H_KV * Dr) &&
         make_map3(enc, &vmap, pp.v, Dr, pp.H_KV, pp.total, Dr, (long long)pp.H_KV * Dr, 64);
  }
  if (!ok) return cudaErrorInvalidValue;
  WideParams p{};
  p.out = pp.out;
  p.cu_seqlens = pp.cu_seqlens;
  p.batch = pp.batch; p.H_Q = pp.H_Q; p.H_KV = pp.H_KV; p.N = pp.N; p.max_seqlen = pp.max_seqlen;
  p.total = pp.total;
  p.o_batch_stride = pp.q_batch_stride; p.o_head_stride = pp.q_head_stride; p.o_tok_stride = pp.q_tok_stride;
  p.causal = pp.causal; p.D_real = Dr; p.dense = dense ? 1 : 0; p.out_bf16 = pp.out_bf16;
  p.scale_log2 = pp.scale_log2;
  p.n_rb = ((dense ? pp.N : pp.max_seqlen) + 127) / 128;
  cudaError_t e = prefill_status_ptr(&p.status);
  if (e != cudaSuccess) return e;
  static SharedMemoryLimit limit;
  e = limit.raise(reinterpret_cast<const void*>(prefill_wide_kernel), kWideSmem);
  if (e != cudaSuccess) return e;
  const long long n_items = items_of_grid(!dense, pp.total, 128, pp.batch, p.n_rb, pp.H_Q);
  p.n_grid = n_items;
  p.take_over = n_items > sm_count ? 1 : 0;
  return launch_attention(pp.after_clear != 0, prefill_wide_kernel, item_grid(n_items), kWideThreads, kWideSmem, stream, qmap, kmap, vmap, p);
}

}  // namespace fa
