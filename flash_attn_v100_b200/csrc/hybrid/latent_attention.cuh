// Attention over the cached latent rows (see latent_attention.cu, latent_decode.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fa {
namespace hybrid {

struct LatentAttentionArgs {
  const void* q_abs;         // T [rows, heads, kv_rank]: unrotated query part, multiplied into the latent space
  const void* q;             // T [rows, heads, q_stride]: the rotated query part before its rotation, at column q_off
  int q_stride, q_off;
  const float *cos_t, *sin_t;    // [rows, rot_dim / 2]
  const void* pool;          // T [n_blocks, 16, pool_stride]: latent | rotated key part
  int pool_stride, n_blocks;
  const int32_t* block_table;    // [n_seq, max_blocks]
  int max_blocks, n_seq;
  const int32_t* tok_seq;    // [rows]
  const int32_t* positions;  // [rows]: the row sees the keys 0 .. position
  const void* gate;          // T [rows, gate_stride]: head h's output is multiplied by sigmoid(gate[h]); or null
  long long gate_stride;
  int heads, kv_rank, rot_dim;
  float scale;
  void* out;                 // T [rows, heads, kv_rank]
  long long rows;
  int* status;
  // tensor-core kernel: work is cut into equal runs of key tiles, one per CTA and head block
  int n_cta;
  int block_heads;           // (see LatentPlan)
  float* part_o;             // [n_cta, 2, heads, kv_rank] unnormalised sums of the rows that are cut
  float* part_ml;            // [n_cta, 2, heads, 2]: their maxima (log2 units) and weights
  int32_t* row_tiles;        // [rows + 1] prefix sums of the rows' key tiles, written by the kernel for the merge
};

// One CTA per (row, head): any size, both types.
template <typename T> cudaError_t launch_latent_attention(const LatentAttentionArgs& a, cudaStream_t s);


// Tensor cores (bfloat16; kv_rank + rot_dim <= 576, both multiples of 8).
bool latent_decode_supported(const LatentAttentionArgs& a);
// Which kernel a call takes, and its grid.
struct LatentPlan {
  int block_heads;           // heads per CTA of the kernel in latent_decode_tc5.cu; 0: the one in latent_decode.cu
  int n_cta;                 // per head block
};
LatentPlan latent_decode_plan(int heads, int kv_rank, int rot_dim, long long rows, int max_blocks, int sm_count);
int latent_decode_max_ctas(int heads, int kv_rank, int rot_dim, int sm_count);   // n_cta of any plan, at most
cudaError_t launch_latent_decode(const LatentAttentionArgs& a, int sm_count, void* encode_fn, cudaStream_t s);   // cuTensorMapEncodeTiled

// The kernel of latents of 128 to 512 columns in blocks of 128, with rotated parts of 16 to 64 columns (latent_decode_tc5.cu).
bool latent_decode_tc5_supported(int kv_rank, int rot_dim);
int latent_decode_tc5_ctas(int heads, int kv_rank, int block_heads, int sm_count);
cudaError_t launch_latent_decode_tc5(const LatentAttentionArgs& a, const CUtensorMap& pool_map, cudaStream_t s);

}  // namespace hybrid
}  // namespace fa
