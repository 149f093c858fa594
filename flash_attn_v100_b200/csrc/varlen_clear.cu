// Zeros in the rows of a packed output that no sequence covers, sm_100a.
#include "prefill.cuh"

namespace fa {
namespace {

// Blocks of column x take the gaps x, x + gridDim.x, ...: gap 0 lies before the first sequence, gap g in 1 .. batch behind the first max_seqlen
// rows of sequence g - 1, gap batch + 1 behind the last sequence.  Usually all are empty and the launch takes 3 us; a fill of the whole output
// before the attention took 67 us of 1046 for 16 prompts of up to 4096 tokens, 32 heads of 128.  (The attention is launched behind this one, so
// where offsets overlap its rows win, as they do over a fill.)
__global__ void __launch_bounds__(256) varlen_clear_kernel(uint4* out, const int32_t* cu, int batch, long long total, int max_seqlen, long long units) {
  for (int g = blockIdx.x; g < batch + 2; g += gridDim.x) {
    long long lo, hi;
    if (g == 0) {
      lo = 0;
      hi = __ldg(cu);
    } else if (g <= batch) {
      lo = (long long)__ldg(cu + g - 1) + max_seqlen;
      hi = __ldg(cu + g);
    } else {
      lo = __ldg(cu + batch);
      hi = total;
    }
    if (lo < 0) lo = 0;
    if (hi > total) hi = total;
    for (long long i = lo * units + (long long)blockIdx.y * blockDim.x + threadIdx.x; i < hi * units; i += (long long)gridDim.y * blockDim.x)
      out[i] = make_uint4(0u, 0u, 0u, 0u);
  }
}

}  // namespace

cudaError_t launch_varlen_clear(void* out, const int32_t* cu, int batch, long long total, int max_seqlen, long long row_bytes, cudaStream_t stream) {
  // one column per gap up to 256, and enough blocks in a column for one gap that is the whole output
  const unsigned x = (unsigned)(batch + 2 < 256 ? batch + 2 : 256);
  const long long per = (total * row_bytes + (256 * 16 * 8 - 1)) / (256 * 16 * 8);        // blocks that would each write 32 KB
  const long long most = 592 / x > 1 ? 592 / x : 1;
  varlen_clear_kernel<<<dim3(x, (unsigned)(per < most ? (per > 0 ? per : 1) : most)), 256, 0, stream>>>(static_cast<uint4*>(out), cu, batch, total, max_seqlen, row_bytes / 16);
  return cudaGetLastError();
}

}  // namespace fa
