// Zeros in the rows of a packed output that no sequence covers, sm_100a.
#include "prefill.cuh"

namespace fa {
namespace {

constexpr int kThreads = 256, kRows = 1024, kAhead = 4;      // kRows: rows that a block looks at together

// Gap 0 lies before the first sequence, gap g in 1 .. batch behind the first max_seqlen rows of sequence g - 1 (from its start on, where
// that lies below row 0: it has no rows), gap batch + 1 behind the last sequence.  A block has an equal share of the rows, marks which of them lie in a gap and clears those, a warp per row: one gap that is most
// of the output, as a buffer padded to a fixed size has it, then keeps every SM writing.  (65536 rows of 32 heads of 128, 300 sequences of 4
// tokens at their start: the packed prefill takes 290 us so, 340 over a fill of the whole output, and took 4400 with the blocks dealt out to the gaps, two
// for each.)  Every gap is looked at, not searched for, so offsets in any order are served as they were by a fill; the attention waits for
// this one before it stores, so where offsets overlap its rows win.  Usually all gaps are empty: 16 prompts of up to 4096 tokens, 32 heads of 128, took 1046 us with the
// fill, 67 of them the fill, and the clear takes 3.
__global__ void __launch_bounds__(kThreads)
varlen_clear_kernel(uint4* out, const int32_t* cu, int batch, long long total, int max_seqlen, long long units, long long share) {
  __shared__ uint32_t in_gap[kRows / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the attention may be launched (see launch_attention)
  const long long first = (long long)blockIdx.x * share, end = first + share < total ? first + share : total;
  for (long long r0 = first; r0 < end; r0 += kRows) {
    const int n = (int)(end - r0 < kRows ? end - r0 : kRows);
    if (threadIdx.x < kRows / 32) in_gap[threadIdx.x] = 0u;
    __syncthreads();
    bool any = false;
    for (int g0 = threadIdx.x; g0 < batch + 2; g0 += kThreads * kAhead) {
      long long from[kAhead], to[kAhead];
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {             // the offsets of several gaps are under way together
        const int g = g0 + i * kThreads;
        from[i] = 0;
        to[i] = g < batch + 2 ? total : 0;
        if (g > 0 && g < batch + 2) from[i] = __ldg(cu + g - 1);
        if (g <= batch) to[i] = __ldg(cu + g);
      }
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        const int g = g0 + i * kThreads;
        if (g > 0 && g <= batch && from[i] >= 0) from[i] += max_seqlen;
        const long long lo = from[i] > r0 ? from[i] - r0 : 0, hi = to[i] < r0 + n ? to[i] - r0 : n;
        if (lo >= hi) continue;
        any = true;
        for (int w = (int)(lo >> 5); w <= (int)((hi - 1) >> 5); ++w) {
          const int a = (int)lo - w * 32, e = (int)hi - w * 32;
          const uint32_t upto = e >= 32 ? 0xffffffffu : (1u << e) - 1u;
          atomicOr(in_gap + w, a > 0 ? upto & ~((1u << a) - 1u) : upto);
        }
      }
    }
    if (!__syncthreads_or(any)) continue;
    for (int r = warp; r < n; r += kThreads / 32) {
      if (!((in_gap[r >> 5] >> (r & 31)) & 1u)) continue;
      uint4* row = out + (r0 + r) * units;
#pragma unroll 4
      for (long long u = lane; u < units; u += 32) row[u] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();                               // the marks have been read
  }
}

}  // namespace

cudaError_t launch_varlen_clear(void* out, const int32_t* cu, int batch, long long total, int max_seqlen, long long row_bytes, int sm_count,
                                cudaStream_t stream) {
  // shares of 16 KB, or as many blocks as run at a time (eight per SM)
  long long blocks = (total * row_bytes + (16 * 1024 - 1)) / (16 * 1024);
  if (blocks > sm_count * 8ll) blocks = sm_count * 8ll;
  const long long share = (total + blocks - 1) / blocks;
  blocks = (total + share - 1) / share;
  varlen_clear_kernel<<<(unsigned)blocks, kThreads, 0, stream>>>(static_cast<uint4*>(out), cu, batch, total, max_seqlen, row_bytes / 16, share);
  return cudaGetLastError();
}

}  // namespace fa
