// row_stage.cuh -- a warp's private stage of raw weights in shared memory: 16 rows x 4 blocks of a row panel, brought by
// cp.async with whole 64- or 128-byte runs of a row per request (one row per lane would touch 32 lines with every request).
// Shared by the multi-token GEMV and the prompt-chunk GEMM.
#pragma once

#include "common.cuh"

namespace ieb {

// Bytes of a stage. Q4_0 / Q4_K / Q6_K: [16 rows][4 x 16 B of nibbles, swizzled] at 0; Q8_0: [16 rows][8 x 16 B, swizzled] at 0.
// Q4_0: four f16 scales per row at 1024. Q8_0: the same at 2048. Q4_K: the super-block header of the row at 1024. Q6_K: high
// bits 4 x 8 B per row at 1024, (sc0 | sc1 << 8) x 4 per row at 1536, at 1664 a 4-byte word per row that holds d.
template <int KIND>
constexpr uint32_t RS_BYTES = KIND == IE_B200_MAT_Q4 ? 1152u : KIND == IE_B200_MAT_Q8 ? 2176u : KIND == IE_B200_MAT_Q4K ? 1280u : 1728u;

// N bytes into shared memory, asynchronously: the first `most` of them from global memory (none if !ok), the rest zeros
template <int N>
__device__ __forceinline__ void rs_cp(uint32_t dst, const void *src, bool ok, uint32_t most = N) {
  const uint32_t sz = ok ? min((uint32_t)N, most) : 0u;
  if (N == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(sz) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(sz) : "memory");
}

// One stage: rows row0 .. + 15, blocks b0 .. b0 + 3 (b0 a multiple of 4). Rows past the matrix and blocks past the row are zeros.
// 16-byte pieces are swizzled so that the eight rows that ldmatrix reads at once lie in different banks.
template <int KIND>
__device__ __forceinline__ void rs_issue(const uint8_t *w, size_t rowb, uint32_t rows, uint32_t nb, uint32_t st, uint32_t row0, uint32_t b0,
                                         int lane) {
  if (KIND == IE_B200_MAT_Q8) {
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
      const uint32_t r = (uint32_t)(lane >> 3) + 4u * k, c = lane & 7u;
      const bool ok = row0 + r < rows && b0 + (c >> 1) < nb;
      rs_cp<16>(st + r * 128u + ((c ^ (r & 7u)) << 4), ok ? w + (size_t)(row0 + r) * rowb + 32u * (size_t)b0 + 16u * c : w, ok);
    }
  } else {
#pragma unroll
    for (uint32_t k = 0; k < 2; k++) {
      const uint32_t r = (uint32_t)(lane >> 2) + 8u * k, c = lane & 3u;
      const bool ok = row0 + r < rows && b0 + c < nb;
      rs_cp<16>(st + r * 64u + ((c ^ ((r >> 1) & 3u)) << 4), ok ? w + (size_t)(row0 + r) * rowb + 16u * (size_t)(b0 + c) : w, ok);
    }
  }
  if (KIND == IE_B200_MAT_Q6K) {
    const uint32_t r = (uint32_t)lane >> 1, c = lane & 1u;
    const bool ok = row0 + r < rows;
    rs_cp<16>(st + 1024u + r * 32u + 16u * c, ok ? w + (size_t)(row0 + r) * rowb + 16u * (size_t)nb + 8u * (size_t)b0 + 16u * c : w, ok);
  }
  if (lane < 16) {
    const bool ok = row0 + lane < rows;
    const uint8_t *rp = w + (size_t)(ok ? row0 + lane : 0u) * rowb;
    if (KIND == IE_B200_MAT_Q4) rs_cp<8>(st + 1024u + 8u * lane, rp + 16u * (size_t)nb + 2u * b0, ok, 2u * (nb - b0));
    if (KIND == IE_B200_MAT_Q8) rs_cp<8>(st + 2048u + 8u * lane, rp + 32u * (size_t)nb + 2u * b0, ok, 2u * (nb - b0));
    if (KIND == IE_B200_MAT_Q4K) rs_cp<16>(st + 1024u + 16u * lane, rp + 16u * (size_t)nb + 16u * (b0 >> 3), ok);
    if (KIND == IE_B200_MAT_Q6K) {
      rs_cp<8>(st + 1536u + 8u * lane, rp + 24u * (size_t)nb + 2u * b0, ok);
      rs_cp<4>(st + 1664u + 4u * lane, rp + 26u * (size_t)nb + ((2u * (b0 >> 3)) & ~3u), ok);
    }
  }
}

// The same stage with the addresses of the rows a lane copies from kept for a whole tile. Rows past the matrix give a copy of its
// last row (the caller does not store their results).
template <int KIND>
struct RsRows {
  static constexpr int N = KIND == IE_B200_MAT_Q8 ? 4 : 2;
  const uint8_t *rp[N];  // the pieces' rows, at the lane's piece
  const uint8_t *hp;     // Q6_K: the high bits of row lane / 2
  const uint8_t *sp;     // lanes 0..15: the scale fields of row `lane`
  __device__ __forceinline__ void set(const uint8_t *w, size_t rowb, uint32_t rows, uint32_t nb, uint32_t row0, int lane) {
#pragma unroll
    for (uint32_t k = 0; k < N; k++) {
      const uint32_t r = KIND == IE_B200_MAT_Q8 ? (uint32_t)(lane >> 3) + 4u * k : (uint32_t)(lane >> 2) + 8u * k;
      rp[k] = w + (size_t)min(row0 + r, rows - 1u) * rowb + 16u * (lane & (KIND == IE_B200_MAT_Q8 ? 7u : 3u));
    }
    if (KIND == IE_B200_MAT_Q6K) hp = w + (size_t)min(row0 + ((uint32_t)lane >> 1), rows - 1u) * rowb + 16u * (size_t)nb + 16u * (lane & 1u);
    sp = w + (size_t)min(row0 + (lane & 15u), rows - 1u) * rowb + (KIND == IE_B200_MAT_Q8 ? 32u : KIND == IE_B200_MAT_Q6K ? 24u : 16u) * (size_t)nb;
  }
};
template <int KIND>
__device__ __forceinline__ void rs_issue_rows(const RsRows<KIND> &rr, uint32_t nb, uint32_t st, uint32_t b0, int lane) {
  if (KIND == IE_B200_MAT_Q8) {
    const uint32_t c = lane & 7u;
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) {
      const uint32_t r = (uint32_t)(lane >> 3) + 4u * k;
      rs_cp<16>(st + r * 128u + ((c ^ (r & 7u)) << 4), rr.rp[k] + 32u * (size_t)b0, b0 + (c >> 1) < nb);
    }
  } else {
    const uint32_t c = lane & 3u;
#pragma unroll
    for (uint32_t k = 0; k < 2; k++) {
      const uint32_t r = (uint32_t)(lane >> 2) + 8u * k;
      rs_cp<16>(st + r * 64u + ((c ^ ((r >> 1) & 3u)) << 4), rr.rp[k] + 16u * (size_t)b0, b0 + c < nb);
    }
  }
  if (KIND == IE_B200_MAT_Q6K) rs_cp<16>(st + 1024u + 16u * lane, rr.hp + 8u * (size_t)b0, true);
  if (lane < 16) {
    if (KIND == IE_B200_MAT_Q4) rs_cp<8>(st + 1024u + 8u * lane, rr.sp + 2u * b0, true, 2u * (nb - b0));
    if (KIND == IE_B200_MAT_Q8) rs_cp<8>(st + 2048u + 8u * lane, rr.sp + 2u * b0, true, 2u * (nb - b0));
    if (KIND == IE_B200_MAT_Q4K) rs_cp<16>(st + 1024u + 16u * lane, rr.sp + 16u * (b0 >> 3), true);
    if (KIND == IE_B200_MAT_Q6K) {
      rs_cp<8>(st + 1536u + 8u * lane, rr.sp + 2u * b0, true);
      rs_cp<4>(st + 1664u + 4u * lane, rr.sp + 2u * (size_t)nb + ((2u * (b0 >> 3)) & ~3u), true);
    }
  }
}

}  // namespace ieb
