// attn_prefill_tc.cuh -- host interface of the prompt-chunk attention on tcgen05 (attn_prefill_tc.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ieb {

// Splits of the positions, and partial rows of all of them together, at most. (16 splits of 256 tokens x 80 heads: a chunk with
// more rows fills the GPU with fewer splits. The scratch stays below 171 MB, heads of 128, however long the chunks.)
constexpr uint32_t PT_MAX_SPLITS = 16, PT_MAX_RECORDS = 16u * 256u * 80u;
// Scratch for the partial rows.
size_t attn_prefill_scratch_bytes(uint32_t n_head, uint32_t hd, uint32_t T);
// positions: *d_pos + T as the host knows it, or 0 (the grid is sized for it; the result depends on it to the summation order only).
// The checks of the C entries are in here: the engine's call has them too.
// d_scratch NULL: one split of the positions. d_err (may be NULL): set to 5 if a bounded wait inside the kernel ran out. hd 64 or 128.
int attn_prefill_tc(const float *d_q, const void *d_kc, const void *d_vc, float *d_out, void *d_oq, const uint32_t *d_pos, uint32_t n_head, uint32_t n_kv,
                    uint32_t hd, uint32_t kv_len, uint32_t T, size_t q_stride, size_t out_stride, size_t oq_stride, uint32_t positions, float *d_scratch,
                    uint32_t *d_err, cudaStream_t st);
// The mma.sync form for small chunks (attn_decode.cu); attn_prefill_tc checks the arguments and decides.
int attn_prefill_mma(const float *d_q, const void *d_kc, const void *d_vc, float *d_out, void *d_oq, const uint32_t *d_pos, uint32_t n_head, uint32_t n_kv,
                     uint32_t hd, uint32_t kv_len, uint32_t T, size_t q_stride, size_t out_stride, size_t oq_stride, cudaStream_t st);

}  // namespace ieb
