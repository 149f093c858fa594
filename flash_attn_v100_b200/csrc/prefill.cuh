// Prefill parameter block shared by the prefill kernels and the C-ABI layer.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fa {

struct PrefillParams {
  const __half* q;
  const __half* k;
  const __half* v;
  __half* out;                // fp16, or bfloat16 bits when out_bf16 is set
  int out_bf16;
  int in_bf16;                // q, k, v are bfloat16 (tcgen05 kernel only: bfloat16 MMAs, P rounded to bfloat16)
  const int32_t* cu_seqlens;  // null => dense [B,H,N,D]; else packed [total,H,D]
  int batch;                  // sequences (dense: B)
  int H_Q, H_KV;
  int N;                      // dense sequence length (unused when packed)
  int max_seqlen;             // packed: grid bound; dense: N
  long long total;            // packed: rows in q/k/v
  long long q_batch_stride, q_head_stride, q_tok_stride;     // elements
  long long kv_batch_stride, kv_head_stride, kv_tok_stride;  // elements
  int causal;
  int D_real;                 // head dimension of the tensors; the kernels are built for 64 / 128 / 256 columns
                              // and take the columns [D_real, D) as zeros
  float scale_log2;           // log2(e) / sqrt(D_real)
  int after_clear;            // launched directly behind launch_varlen_clear on the same stream
};

// Launch of an attention kernel; `overlap`: beside the end of the clear in front of it, which lets its successor start as soon as its own blocks have.  That clear
// started behind everything before it, so the attention may read its inputs at once; before its first store it waits for the clear (wait_for_clear), whose rows it
// may share where offsets overlap, and every thread does before it leaves: what follows on the stream waits for the attention alone.
template <class Kernel, class... Args>
cudaError_t launch_attention(bool overlap, Kernel kern, dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

cudaError_t launch_prefill_mma(const PrefillParams& p, int D, cudaStream_t stream);

// tcgen05 / TMEM kernel (D = 64 or 128).  `encode_fn` is cuTensorMapEncodeTiled.
bool prefill_tc5_supported(const PrefillParams& p, int D);
cudaError_t launch_prefill_tc5(const PrefillParams& p, int D, void* encode_fn, cudaStream_t stream);
void prefill_tc5_set_poly(bool on);
// tcgen05 kernel of wide heads: 128 < D_real <= 256, fp16.
bool prefill_wide_supported(const PrefillParams& p);
cudaError_t launch_prefill_wide(const PrefillParams& p, int sm_count, void* encode_fn, cudaStream_t stream);
// Zeros in the rows of a packed [total, row_bytes] output that no sequence covers.
cudaError_t launch_varlen_clear(void* out, const int32_t* cu_seqlens, int batch, long long total, int max_seqlen, long long row_bytes,
                                int sm_count, cudaStream_t stream);
cudaError_t prefill_status(int* host_out, cudaStream_t stream);
cudaError_t prefill_status_ptr(int** out);  // device address of the status word (current device)
cudaError_t prefill_status_clear(cudaStream_t stream);

}  // namespace fa
