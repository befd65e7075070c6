// gemm_tc.cu -- the prompt-chunk GEMM on the 5th-generation tensor cores (tcgen05 + tensor memory):
// Y[T x rows] = X[T x cols] . W^T for the quantised kinds, the role of ie_gemm_q4kr / ie_gemm_q6kr
// (kernels/ie_kernels.c:1315-1465, :2015-2158; dispatch src/hip.c:965-1003).
//
// The quant scales change every 32 columns, so an integer MMA needs a scaling step on the CUDA cores per 32 x row x
// token (the wall the reference's own GEMM hit, and the bound of the mma.sync kernel in gemm_mma.cu). Here nothing is
// scaled inside the main loop: both operands are turned into f16 ONCE and the tensor cores accumulate in fp32 over the
// whole K in tensor memory:
//   activations  a pre-pass expands each token's Q8 row to x = d_a * q (f32) and splits it into two f16 terms
//                x = x_hi + x_lo (22 significant bits), stored in the order the MMA wants (cost ~ T x K, once per chunk);
//   weights      sixteen producer warps bring raw rows by cp.async (64 bytes of a row per request, four blocks at a time, the next
//                four on their way: one row per lane touched 32 lines with every load) and turn 256 rows of the current 32-column
//                block into two f16 terms w = w_hi + w_lo in pairs (tc_convert), straight into shared memory in the canonical
//                K-major core-matrix layout (cost ~ rows x K, once per 256 tokens);
//   MMA          one thread per tile issues, per 16 columns, w_hi x_hi + w_hi x_lo + w_lo x_hi (the dropped w_lo x_lo term is
//                below 2^-22 of a product) as tcgen05.mma kind::f16, M = 128, N = up to 256 tokens, two 128-row tiles per
//                CTA, accumulators in tensor memory (2 x 256 columns). Up to 128 tokens, x_hi and x_lo lie side by side as one
//                operand of twice the width and go into two accumulators: two products of w per 16 columns instead of three;
//   epilogue     the producer warps read the accumulators back (tcgen05.ld, one row and 32 tokens per thread at a time), add bias /
//                residual and store token rows (32 consecutive rows per warp store: coalesced).
// Two rings, handed over with mbarriers (full: sixteen producer warps / the bulk copy's bytes; empty: tcgen05.commit): 32 KB of
// weights and the tokens' 128 bytes each of activations per 32-column stage, as many stages as fit.
// Matrices with few rows (3584 x 18944: 14 CTAs) are split along K over grid.z, every split writing its partial sums to
// scratch, which a second kernel adds in split order (deterministic). Every mbarrier wait is bounded by wall time and reports through the device
// error word; a warp goes on as one, waiting or not, and a CTA that gave up waits for its copies and MMAs on their way before it
// frees its tensor memory and ends.
//
// Half precision has a narrow exponent range, so both sides are scaled by exact powers of two before they are split (a value
// below 2^-14 would lose its low term to the subnormal grid): the weights by 2^S_w, S_w chosen once per matrix from a bound on
// its largest weight (ie_b200_mat_tc_exp), each token by 2^S_n chosen from its largest Q8 scale; the epilogue multiplies row n
// of the result by 2^-(S_w + S_n).
//
// Measured with its pre-pass and reduction, one row per lane from global memory and every weight converted in f32 -> now: 28672 x
// 4096 Q4_0 17 / 77 / 160 / 256 tokens 122 / 134 / 151 / 166 -> 73 / 83 / 106 / 142 us; 37888 x 3584 Q4_K 108 / 115 / 128 / 154 ->
// 79 / 82 / 108 / 146; 3584 x 18944 Q6_K 121 / 129 / 139 / 151 -> 60 / 67 / 78 / 104. At 256 tokens the tensor pipe bounds it (three
// products per weight and token: 126 us of f16 work for the 37888 rows at the measured bf16 burst rate).
//
// Result: equal to the one-token GEMV (which is bit-exact with the CPU) to fp32 rounding: not bit for bit, as the
// reference's GEMM against its GEMV. Relative error against 64 bits (2-norm; the f32 accumulation dominates): Q4_0 4096 columns
// 9.0e-7, 14336 3.0e-6, Q4_K 3584 9.8e-7, Q6_K 18944 4.5e-6 above 128 tokens; with two accumulators 5.9e-7, 1.9e-6, 6.7e-7, 3.0e-6.
#include <cuda_fp16.h>
#include <math.h>
#include <string.h>

#include <algorithm>

#include "common.cuh"
#include "row_stage.cuh"
#include "tc_common.cuh"

namespace ieb {

int gemm_tc_run(int kind, const void *d_w, uint32_t rows, uint32_t cols, int w_exp, const void *d_xq, float *d_y, const float *d_bias, const float *d_res, uint32_t T,
                size_t x_stride, size_t y_stride, size_t res_stride, void *d_scratch, size_t scratch_bytes, uint32_t *d_err, cudaStream_t st, bool act_ready);

constexpr int TC_ROWS = 256, TC_TOK = 256, TC_KS = 32, TC_PROD_WARPS = 16, TC_THREADS = (TC_PROD_WARPS + 3) * 32;
constexpr int TC_A_TILE = 128 * TC_KS * 2;       // one 128-row tile, one f16 term, one stage: 8 KB
constexpr int TC_A_STAGE = 4 * TC_A_TILE;        // two tiles x (hi, lo)
constexpr int TC_TOK_STAGE = 2 * TC_KS * 2;      // one token's two f16 terms of a stage: 128 B
constexpr int TC_MAX_ST = 4;                     // stages of a ring, at most
constexpr uint32_t TC_SMEM = 227u * 1024u - 2048u, TC_BARS = 256u;  // (2 KB stay for the static arrays)
// tokens of tile nt, padded to what an MMA takes
__host__ __device__ inline uint32_t tc_pad(uint32_t T, uint32_t nt) {
  const uint32_t n = T - nt * TC_TOK < (uint32_t)TC_TOK ? T - nt * TC_TOK : (uint32_t)TC_TOK;
  return (n + 15u) & ~15u;
}

struct TcArgs {
  const uint8_t *w;
  size_t rowb;
  uint32_t rows, nb, T;
  uint32_t blocks_per_split;
  const uint8_t *bp;  // expanded activations: [token tile][block][4 chunks][hi | lo][n / 8 groups][8 tokens][8 halves], n = tc_pad
  uint32_t sa, sb;    // stages of the two rings
  float *y;
  const float *bias, *res;
  size_t ys, rs;
  float *partial;     // grid.z > 1: [split][T][rows]
  uint32_t *err;
  float w_scale;      // 2^S_w applied to every weight before the split
  float w_inv;           // 2^-S_w
  const float *tok_inv;  // per token: 2^-S_n
};

// ---- activations: Q8 rows -> f16 hi / lo in MMA order -----------------------------------------------------------------
// grid (groups of 8 tokens, parts of the columns), 256 threads. Warp w of a CTA first looks for the largest Q8 scale of token w
// (every part repeats that: a few KB from L2): S_n such that the largest |d q| 2^S_n lies in [2048, 4096); tok_inv[n] = 2^-S_n.
// Then thread = token and one of 32 blocks at a time: its 32 values as 4 + 4 16-byte pieces, eight tokens side by side. Tokens
// past T are zero. The four columns of an activation word are stored in the order 0, 2, 1, 3, as the producers store the
// weights: a mask takes bytes 0 and 2 of a word into a pair of halves at once, and the order of the columns of a product does
// not matter.
__global__ void __launch_bounds__(256) tc_expand_kernel(const uint8_t *xq, size_t xs, uint32_t T, uint32_t nb, float *tok_inv, uint8_t *bp) {
  __shared__ float scale[8];
  pdl_prologue();
  const uint32_t n0 = blockIdx.x * 8u, nt = n0 / TC_TOK, pad = tc_pad(T, nt);
  {
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u, n = n0 + w;
    float m = 0.0f;
    if (n < T) {
      const float *d = reinterpret_cast<const float *>(xq + xs * n + 32u * (size_t)nb);
#pragma unroll 4
      for (uint32_t b = lane; b < nb; b += 32u) m = fmaxf(m, fabsf(d[b]));
    }
    m = warp_max(m) * 127.0f;
    int e = 0;
    if (m > 0.0f && m < 3.0e38f) {
      int ex;
      frexpf(m, &ex);  // m = f * 2^ex, f in [0.5, 1)
      e = 12 - ex;     // m * 2^e in [2048, 4096)
      e = e > 100 ? 100 : (e < -100 ? -100 : e);
    }
    if (lane == 0) {
      scale[w] = ldexpf(1.0f, e);
      if (blockIdx.y == 0 && n < T) tok_inv[n] = ldexpf(1.0f, -e);
    }
  }
  __syncthreads();
  const uint32_t tok = threadIdx.x & 7u, n = n0 + tok, nl = n - nt * TC_TOK;
  for (uint32_t b = blockIdx.y * 32u + (threadIdx.x >> 3); b < nb; b += gridDim.y * 32u) {
    uint4 hi[4], lo[4];
#pragma unroll
    for (int c = 0; c < 4; c++) hi[c] = lo[c] = make_uint4(0u, 0u, 0u, 0u);
    if (n < T) {
      const uint8_t *row = xq + xs * n;
      const uint4 q0 = *reinterpret_cast<const uint4 *>(row + 32u * (size_t)b), q1 = *reinterpret_cast<const uint4 *>(row + 32u * (size_t)b + 16u);
      const float d = __fmul_rn(*reinterpret_cast<const float *>(row + 32u * (size_t)nb + 4u * b), scale[tok]);  // exact: a power of two
      const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
      for (int c = 0; c < 4; c++) {  // chunk c: values 8c .. 8c + 7 = words 2c, 2c + 1
        uint32_t h[4], l[4];
#pragma unroll
        for (int p = 0; p < 4; p++) {
          const uint32_t wd = qw[2 * c + (p >> 1)];
          const int s0 = (int)(int8_t)(wd >> (8 * (p & 1))), s1 = (int)(int8_t)(wd >> (8 * (p & 1) + 16));
          tc_split2(__fmul_rn(d, (float)s0), __fmul_rn(d, (float)s1), h[p], l[p]);
        }
        hi[c] = make_uint4(h[0], h[1], h[2], h[3]), lo[c] = make_uint4(l[0], l[1], l[2], l[3]);
      }
    }
    uint8_t *base = bp + (size_t)nt * nb * TC_TOK * TC_TOK_STAGE + (size_t)b * pad * TC_TOK_STAGE + nl * 16u;
#pragma unroll
    for (uint32_t c = 0; c < 4; c++) {
      *reinterpret_cast<uint4 *>(base + c * pad * 32u) = hi[c];
      *reinterpret_cast<uint4 *>(base + c * pad * 32u + pad * 16u) = lo[c];
    }
  }
}

// ---- weights: half a block (16 columns) of one row of a raw stage -> two f16 terms, column pairs (0, 2), (1, 3) per word ----
// Q4_0, Q8_0, Q6_K: the integer weight is exact in f16 (a byte ORed into 0x6400 is 1024 + byte), and so is the rest of a
// product of two halves, which one fma gives: hi = rn(s q), lo = s q - hi, two weights per instruction. A Q6_K scale d sc has
// 19 bits: s = s_hi + s_lo, lo = (s_hi q - hi) + s_lo q, the last product as (2^10 s_lo) (2^-10 q): of a super-block far below the
// matrix's largest, s_lo alone would lie on the subnormal grid. Q4_K (d sc q - dmin mn cancels) is worked in f32 and split after.
// About 2 (Q4_0) to 5 (Q4_K) instructions per weight; converting each to f32, scaling and splitting there took more than 10.
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }
__device__ __forceinline__ __half2 u2h(uint32_t u) { return *reinterpret_cast<const __half2 *>(&u); }

template <int KIND>
__device__ __forceinline__ void tc_convert(const uint8_t *raw, uint32_t r, uint32_t i, uint32_t b, uint32_t hf, float w_scale, uint32_t (&hi)[8], uint32_t (&lo)[8]) {
  if (KIND == IE_B200_MAT_Q8) {
    const uint4 v4 = *reinterpret_cast<const uint4 *>(raw + r * 128u + (((2u * i + hf) ^ (r & 7u)) << 4));
    const uint32_t v[4] = {v4.x, v4.y, v4.z, v4.w};
    const __half2 d2 = __float2half2_rn(__fmul_rn(h2f(*reinterpret_cast<const uint16_t *>(raw + 2048u + 8u * r + 2u * i)), w_scale));
    const __half2 off = u2h(0x64806480u);  // 1152
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t u = v[k] ^ 0x80808080u;  // byte + 128
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const __half2 q = __hsub2(u2h(__byte_perm(u, 0x64646464u, p ? 0x4341 : 0x4240)), off), h = __hmul2(d2, q);
        hi[2 * k + p] = h2u(h), lo[2 * k + p] = h2u(__hfma2(d2, q, __hneg2(h)));
      }
    }
    return;
  }
  const uint4 v4 = *reinterpret_cast<const uint4 *>(raw + r * 64u + ((i ^ ((r >> 1) & 3u)) << 4));
  const uint32_t v[4] = {v4.x >> (4u * hf), v4.y >> (4u * hf), v4.z >> (4u * hf), v4.w >> (4u * hf)};
  if (KIND == IE_B200_MAT_Q4) {
    const __half2 d2 = __float2half2_rn(__fmul_rn(h2f(*reinterpret_cast<const uint16_t *>(raw + 1024u + 8u * r + 2u * i)), w_scale));
    const __half2 off = u2h(0x64086408u);  // 1032
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const __half2 q = __hsub2(u2h(((v[k] >> (8 * p)) & 0x000F000Fu) | 0x64006400u), off), h = __hmul2(d2, q);
        hi[2 * k + p] = h2u(h), lo[2 * k + p] = h2u(__hfma2(d2, q, __hneg2(h)));
      }
    }
  } else if (KIND == IE_B200_MAT_Q6K) {
    const uint32_t hw = *reinterpret_cast<const uint32_t *>(raw + 1024u + 32u * r + 8u * i + 4u * hf);
    const uint32_t sc = raw[1536u + 8u * r + 2u * i + hf];
    const float df = h2f(*reinterpret_cast<const uint16_t *>(raw + 1664u + 4u * r + 2u * ((b >> 3) & 1u)));
    const float s = __fmul_rn(__fmul_rn(df, (float)(int8_t)sc), w_scale);
    const __half sh = __float2half_rn(s);
    const __half2 s_hi = __half2half2(sh), s_lo = __float2half2_rn(1024.0f * (s - __half2float(sh))), off = u2h(0x64206420u);  // 1056
    const __half2 down = u2h(0x14001400u), off_d = u2h(0xBC20BC20u);  // 2^-10, -1056 2^-10
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t w6 = (v[k] & 0x0F0F0F0Fu) | (((hw >> (2 * k)) & 0x03030303u) << 4);
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const __half2 x = u2h(((w6 >> (8 * p)) & 0x003F003Fu) | 0x64006400u), q = __hsub2(x, off), h = __hmul2(s_hi, q);
        hi[2 * k + p] = h2u(h), lo[2 * k + p] = h2u(__hfma2(s_lo, __hfma2(x, down, off_d), __hfma2(s_hi, q, __hneg2(h))));
      }
    }
  } else {
    const uint4 hd = *reinterpret_cast<const uint4 *>(raw + 1024u + 16u * r);
    const uint32_t fld = q4k_field(hd, (int)(b & 7u));
    const float s = __fmul_rn(__fmul_rn(h2f((uint16_t)(hd.x & 0xFFFFu)), (float)(fld & 63u)), w_scale);
    const float mm = -__fmul_rn(__fmul_rn(h2f((uint16_t)(hd.x >> 16)), (float)(fld >> 6)), w_scale);
    const f32x2 s2 = pk2(s, s), m2 = pk2(mm, mm), two23 = pk2(-8388608.0f, -8388608.0f), neg = pk2(-1.0f, -1.0f);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const uint32_t u = v[k] & 0x0F0F0F0Fu;
#pragma unroll
      for (int p = 0; p < 2; p++) {  // a byte under 0x4B000000 is the float 2^23 + byte
        const f32x2 q = add2(pk2(__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7440 + p)), __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7442 + p))), two23);
        const f32x2 f = fma2(s2, q, m2);
        float f0, f1;
        unpk2(f, f0, f1);
        const __half2 h = __floats2half2_rn(f0, f1);
        const float2 hf2 = __half22float2(h);
        unpk2(fma2(pk2(hf2.x, hf2.y), neg, f), f0, f1);
        hi[2 * k + p] = h2u(h), lo[2 * k + p] = h2u(__floats2half2_rn(f0, f1));
      }
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(TC_THREADS, 1) gemm_tc_kernel(const TcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_tc[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t m0 = blockIdx.x * TC_ROWS, nt = blockIdx.y, split = blockIdx.z;
  const uint32_t kb0 = split * a.blocks_per_split, kb1 = min(a.nb, kb0 + a.blocks_per_split), n_it = kb1 - kb0;
  const uint32_t n_eff = tc_pad(a.T, nt), b_stage = n_eff * TC_TOK_STAGE;  // MMA N: a multiple of 16
  const uint32_t n_tiles = a.rows - m0 > 128u ? 2u : 1u;
  const bool wide = n_eff <= 128u;                         // w_hi (x_hi | x_lo) as one MMA, into two accumulators
  uint8_t *sA = smem_tc;                                   // [stage][tile][term] 8 KB each
  uint8_t *sB = sA + a.sa * TC_A_STAGE;                    // [stage][4 chunks][hi | lo][tokens][16 B]
  uint8_t *sR = sB + (size_t)a.sb * min(a.T + 15u & ~15u, (uint32_t)TC_TOK) * TC_TOK_STAGE;  // raw weights: two stages per producer warp
  uint64_t *bars = reinterpret_cast<uint64_t *>(sR + TC_PROD_WARPS * 2u * RS_BYTES<KIND>);
  uint64_t *full_a = bars, *empty_a = bars + TC_MAX_ST, *full_b = bars + 2 * TC_MAX_ST, *empty_b = bars + 3 * TC_MAX_ST, *done = bars + 4 * TC_MAX_ST,
           *drained = done + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 4 * TC_MAX_ST + 3);
  __shared__ uint32_t s_abort;
  __shared__ float s_inv[TC_TOK];

  if (tid == 0) {
    s_abort = 0u;
    for (int s = 0; s < TC_MAX_ST; s++) mbar_init(&full_a[s], (uint32_t)TC_PROD_WARPS), mbar_init(&empty_a[s], n_tiles), mbar_init(&full_b[s], 1u), mbar_init(&empty_b[s], n_tiles);
    mbar_init(done, n_tiles), mbar_init(&drained[0], 1u), mbar_init(&drained[1], 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == TC_PROD_WARPS) {  // tensor memory: all 512 columns (two accumulators of up to 256 columns), by one warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();
  // producers: warp w dequantises 16 rows of tile w >> 3, thread = row and column half; the first raw stage (weights) is on
  // its way before the wait for the activations
  const uint32_t t_p = (uint32_t)warp >> 3, row0 = m0 + t_p * 128u + ((uint32_t)warp & 7u) * 16u;
  uint8_t *raw = sR + (uint32_t)warp * 2u * RS_BYTES<KIND>;
  if (warp < TC_PROD_WARPS) {  // (raw stages start at multiples of four blocks; a split may start inside one)
    if (n_it > 0u) rs_issue<KIND>(a.w, a.rowb, a.rows, a.nb, smem_u32(raw + ((kb0 >> 2) & 1u) * RS_BYTES<KIND>), row0, kb0 & ~3u, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  pdl_wait();  // the expanded activations (and the residual) are complete
  for (uint32_t j = tid; j < TC_TOK; j += TC_THREADS) s_inv[j] = nt * TC_TOK + j < a.T ? __fmul_rn(a.tok_inv[nt * TC_TOK + j], a.w_inv) : 0.0f;
  __syncthreads();

  bool gave_up = false;   // of a thread that issues MMAs
  uint32_t issued = 0;    // stages asked for by the thread that copies the activations
  if (warp < TC_PROD_WARPS) {
    // ---------------- producers ----------------
    const uint32_t r = lane & 15u, hf = (uint32_t)lane >> 4, rl = ((uint32_t)warp & 7u) * 16u + r;  // row of the raw stage, column half, row in the tile
    const uint32_t dst0 = t_p * 2 * TC_A_TILE + (rl >> 3) * 128u + (rl & 7u) * 16u + hf * 2u * 2048u;
    uint32_t s = 0, par = 1u;  // the first round finds every stage empty
    for (uint32_t b = kb0; b < kb1; b++) {
      const uint32_t i = b & 3u;  // its place in the raw stage, which lies in place (b / 4) mod 2
      const uint8_t *src = raw + ((b >> 2) & 1u) * RS_BYTES<KIND>;
      if (i == 0u || b == kb0) {  // the next four blocks have arrived; ask for the four after them, whose place all lanes have done with
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        const uint32_t next = (b | 3u) + 1u;
        if (next < kb1) rs_issue<KIND>(a.w, a.rowb, a.rows, a.nb, smem_u32(raw + ((next >> 2) & 1u) * RS_BYTES<KIND>), row0, next, lane);
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      uint32_t hi[8], lo[8];
      tc_convert<KIND>(src, r, i, b, hf, a.w_scale, hi, lo);
      mbar_wait(&empty_a[s], par, &s_abort);  // (after giving up the lanes go on together, without waiting: nobody stores the results)
      uint8_t *dst = sA + s * TC_A_STAGE + dst0;
#pragma unroll
      for (int c = 0; c < 2; c++) {  // 8-column chunks 2 hf + c of the block
        *reinterpret_cast<uint4 *>(dst + c * 2048u) = make_uint4(hi[4 * c], hi[4 * c + 1], hi[4 * c + 2], hi[4 * c + 3]);
        *reinterpret_cast<uint4 *>(dst + TC_A_TILE + c * 2048u) = make_uint4(lo[4 * c], lo[4 * c + 1], lo[4 * c + 2], lo[4 * c + 3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read shared memory through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_a[s]);
      if (++s == a.sa) s = 0u, par ^= 1u;
    }
    // ---------------- epilogue: accumulators -> token rows ----------------
    const bool finished = __all_sync(0xFFFFFFFFu, mbar_wait(done, 0u, &s_abort) && !s_abort);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (finished) {
      // warp w reads lanes 32 (w & 3) .. + 31 of tensor memory (a warp reaches the quarter w mod 4 only): tile (w >> 2) & 1,
      // token columns 32 (w >> 3) + 64 k ..
      const uint32_t q = (uint32_t)warp & 3u, te = ((uint32_t)warp >> 2) & 1u, ch = (uint32_t)warp >> 3;
      const uint32_t row = m0 + te * 128u + q * 32u + lane;
      const float bias = (a.bias && row < a.rows && !a.partial) ? a.bias[row] : 0.0f;
      if (te < n_tiles) {
        for (uint32_t c0 = ch * 32u; c0 < n_eff; c0 += 64u) {
          uint32_t v[32];
          tc_ld32(tmem + ((q * 32u) << 16) + te * TC_TOK + c0, v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (wide) {
            uint32_t v2[32];
            tc_ld32(tmem + ((q * 32u) << 16) + te * TC_TOK + n_eff + c0, v2);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = __float_as_uint(__fadd_rn(__uint_as_float(v[j]), __uint_as_float(v2[j])));
          }
          if (row < a.rows) {
#pragma unroll
            for (int j = 0; j < 32; j++) {
              const uint32_t n = nt * TC_TOK + c0 + j;
              if (n < a.T) {
                float o = __fmul_rn(__uint_as_float(v[j]), s_inv[c0 + j]);
                if (a.partial) {
                  a.partial[((size_t)split * a.T + n) * a.rows + row] = o;
                } else {
                  if (a.bias) o = __fadd_rn(o, bias);
                  if (a.res) o = __fadd_rn(*reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.res) + a.rs * n + 4u * (size_t)row), o);
                  *reinterpret_cast<float *>(reinterpret_cast<char *>(a.y) + a.ys * n + 4u * (size_t)row) = o;
                }
              }
            }
          }
        }
      }
    }
  } else if (warp < TC_PROD_WARPS + 2) {
    // ---------------- MMA issue: one thread per tile ----------------
    // (issuing a stage's products takes one thread longer than the tensor cores need for few tokens: 28672 x 4096, 77 tokens: 125 us
    // with descriptors built for every product, 93 with them stepped by additions, 83 with a thread per tile)
    const uint32_t t = (uint32_t)warp - TC_PROD_WARPS;
    if (lane == 0 && t < n_tiles) {
      // instruction descriptor: D f32, A and B f16, both K-major, M = 128, N
      const uint32_t id0 = (1u << 4) | ((128u >> 4) << 24), id_n = id0 | ((n_eff >> 3) << 17), id_2n = id0 | ((n_eff >> 2) << 17);
      const uint32_t lbo = n_eff * 32u;  // bytes between two 8-column chunks of the activations
      // descriptors: address fields count 16-byte units and never carry out of their 14 bits (shared memory ends at 256 KB), so
      // a stage, a term or a column step is one addition
      const uint64_t da0 = tc_desc(smem_u32(sA) + t * 2u * TC_A_TILE, 2048u, 128u), db0 = tc_desc(smem_u32(sB), lbo, 128u);
      constexpr uint64_t A_LO = TC_A_TILE >> 4, A_J = 4096 >> 4;
      const uint32_t d = tmem + t * TC_TOK;
      const uint64_t b_j = lbo >> 3, b_lo = n_eff;
      uint32_t s = 0, pa = 0, sb = 0, pb = 0;
      for (uint32_t it = 0; it < n_it; it++) {
        if (!mbar_wait(&full_a[s], pa, &s_abort) || !mbar_wait(&full_b[sb], pb, &s_abort)) {
          gave_up = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t da = da0 + s * (uint32_t)(TC_A_STAGE >> 4), db = db0 + sb * (b_stage >> 4);
        const uint32_t acc = it ? 1u : 0u;
        if (wide) {
          tc_mma(d, da, db, id_2n, acc), tc_mma(d, da + A_LO, db, id_n, 1u);
          tc_mma(d, da + A_J, db + b_j, id_2n, 1u), tc_mma(d, da + A_J + A_LO, db + b_j, id_n, 1u);
        } else {
          tc_mma(d, da, db, id_n, acc), tc_mma(d, da, db + b_lo, id_n, 1u), tc_mma(d, da + A_LO, db, id_n, 1u);
          tc_mma(d, da + A_J, db + b_j, id_n, 1u), tc_mma(d, da + A_J, db + b_j + b_lo, id_n, 1u), tc_mma(d, da + A_J + A_LO, db + b_j, id_n, 1u);
        }
        tc_commit(&empty_a[s]), tc_commit(&empty_b[sb]);  // arrive when the MMAs issued so far have completed: the stages may be refilled
        if (++s == a.sa) s = 0u, pa ^= 1u;
        if (++sb == a.sb) sb = 0u, pb ^= 1u;
      }
      if (!gave_up) tc_commit(done);  // (never both tiles' after giving up: the epilogue reads whole results only)
    }
  } else {
    // ---------------- activations: one bulk copy per stage ----------------
    if (lane == 0) {
      for (uint32_t it = 0; it < n_it; it++) {
        const uint32_t s = it % a.sb, round = it / a.sb;
        if (round > 0 && !mbar_wait(&empty_b[s], (round - 1u) & 1u, &s_abort)) break;
        mbar_expect_tx(&full_b[s], b_stage);
        bulk_g2s(sB + s * b_stage, a.bp + (size_t)nt * a.nb * TC_TOK * TC_TOK_STAGE + (size_t)(kb0 + it) * b_stage, b_stage, &full_b[s]);
        issued = it + 1u;
      }
    }
  }
  if (warp < TC_PROD_WARPS) asm volatile("cp.async.wait_group 0;" ::: "memory");  // (after giving up: none is left on its way)
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_abort) {  // (nobody sets it any more) do not leave while MMAs or copies still use this CTA's memory
    if (lane == 0 && warp >= TC_PROD_WARPS && warp < TC_PROD_WARPS + 2 && (uint32_t)warp - TC_PROD_WARPS < n_tiles) {
      uint64_t *bar = &drained[warp - TC_PROD_WARPS];
      tc_commit(bar), mbar_drain(bar, 0u);
    }
    for (uint32_t it = issued > a.sb ? issued - a.sb : 0u; it < issued; it++) mbar_drain(&full_b[it % a.sb], (it / a.sb) & 1u);
    if (tid == 0 && a.err) atomicExch(a.err, 5u);
    __syncthreads();
  }
  __syncwarp();
  if (warp == TC_PROD_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// y[n][row] = sum over the splits (in order) of partial[split][n][row] (+ bias) (+ res).
__global__ void __launch_bounds__(256) tc_reduce_kernel(const float *partial, uint32_t splits, uint32_t T, uint32_t rows, float *y, const float *bias,
                                                        const float *res, size_t ys, size_t rs) {
  pdl_prologue();
  const uint32_t n = blockIdx.y;
  for (uint32_t r = blockIdx.x * 256u + threadIdx.x; r < rows; r += gridDim.x * 256u) {
    float o = 0.0f;
    for (uint32_t s = 0; s < splits; s++) o = __fadd_rn(o, partial[((size_t)s * T + n) * rows + r]);
    if (bias) o = __fadd_rn(o, bias[r]);
    if (res) o = __fadd_rn(*reinterpret_cast<const float *>(reinterpret_cast<const char *>(res) + rs * n + 4u * (size_t)r), o);
    *reinterpret_cast<float *>(reinterpret_cast<char *>(y) + ys * n + 4u * (size_t)r) = o;
  }
}

// The same four rows per thread (rows a multiple of 4, 16-byte aligned rows): all splits' loads on their way at once.
__global__ void __launch_bounds__(128) tc_reduce4_kernel(const float *partial, uint32_t splits, uint32_t T, uint32_t rows, float *y, const float *bias,
                                                         const float *res, size_t ys, size_t rs) {
  pdl_prologue();
  const uint32_t n = blockIdx.y, r = 4u * (blockIdx.x * 128u + threadIdx.x);
  if (r >= rows) return;
  const float4 *src = reinterpret_cast<const float4 *>(partial + (size_t)n * rows + r);
  const size_t step = (size_t)T * rows / 4u;
  float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (uint32_t s0 = 0; s0 < splits; s0 += 4u) {
    float4 p[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; k++)
      if (s0 + k < splits) p[k] = __ldcg(src + (s0 + k) * step);
#pragma unroll
    for (uint32_t k = 0; k < 4; k++)
      if (s0 + k < splits) o.x = __fadd_rn(o.x, p[k].x), o.y = __fadd_rn(o.y, p[k].y), o.z = __fadd_rn(o.z, p[k].z), o.w = __fadd_rn(o.w, p[k].w);
  }
  if (bias) o.x = __fadd_rn(o.x, bias[r]), o.y = __fadd_rn(o.y, bias[r + 1]), o.z = __fadd_rn(o.z, bias[r + 2]), o.w = __fadd_rn(o.w, bias[r + 3]);
  if (res) {
    const float4 v = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(res) + rs * n + 4u * (size_t)r);
    o.x = __fadd_rn(v.x, o.x), o.y = __fadd_rn(v.y, o.y), o.z = __fadd_rn(v.z, o.z), o.w = __fadd_rn(v.w, o.w);
  }
  *reinterpret_cast<float4 *>(reinterpret_cast<char *>(y) + ys * n + 4u * (size_t)r) = o;
}

static uint32_t tc_splits(uint32_t rows, uint32_t nb, uint32_t T) {
  const uint32_t ctas = ((rows + TC_ROWS - 1) / TC_ROWS) * ((T + TC_TOK - 1) / TC_TOK);
  const uint32_t sms = (uint32_t)sm_count();
  if (ctas * 2u > sms) return 1u;
  uint32_t s = sms / ctas;
  if (s > nb / 8u) s = nb / 8u;  // at least 8 blocks (256 columns) per split
  if (s > 16u) s = 16u;
  return s < 1u ? 1u : s;
}

// What one call over T tokens takes of the scratch.
static size_t tc_scratch(uint32_t rows, uint32_t cols, uint32_t T) {
  const uint32_t nb = cols / 32u, nt = (T + TC_TOK - 1) / TC_TOK, splits = tc_splits(rows, nb, T);
  const size_t bp = (size_t)nt * nb * TC_TOK * TC_TOK_STAGE, part = splits > 1u ? (size_t)splits * T * rows * sizeof(float) : 0u;
  const size_t scales = ((size_t)nt * TC_TOK * sizeof(float) + 255u) & ~(size_t)255u;
  return bp + part + scales + 512u;
}

}  // namespace ieb

using namespace ieb;

// Enough for every call of up to T tokens: fewer token tiles mean more splits along K, so a shorter chunk may take more. (Within a
// number of token tiles the splits stay the same and the longest takes the most.)
extern "C" size_t ie_b200_gemm_tc_scratch_bytes(uint32_t rows, uint32_t cols, uint32_t T) {
  size_t most = tc_scratch(rows, cols, T);
  for (uint32_t t = TC_TOK; t < T; t += TC_TOK) most = std::max(most, tc_scratch(rows, cols, t));
  return most;
}

namespace ieb {
// Largest possible |weight| of a matrix from its scale fields: Q4_0 8 |d|; Q4_K 63 (15 |d| + |dmin|); Q6_K 128 * 32 |d|.
template <int KIND>
__global__ void __launch_bounds__(256) tc_wbound_kernel(const uint8_t *w, size_t rowb, uint32_t rows, uint32_t nb, uint32_t *out_bits) {
  float m = 0.0f;
  const uint32_t per = (KIND == IE_B200_MAT_Q4 || KIND == IE_B200_MAT_Q8) ? nb : nb / 8u;
  for (size_t i = (size_t)blockIdx.x * 256u + threadIdx.x; i < (size_t)rows * per; i += (size_t)gridDim.x * 256u) {
    const uint8_t *rp = w + (i / per) * rowb;
    const uint32_t b = (uint32_t)(i % per);
    float v;
    if (KIND == IE_B200_MAT_Q4) {
      v = 8.0f * fabsf(h2f(*reinterpret_cast<const uint16_t *>(rp + 16u * (size_t)nb + 2u * b)));
    } else if (KIND == IE_B200_MAT_Q8) {
      v = 128.0f * fabsf(h2f(*reinterpret_cast<const uint16_t *>(rp + 32u * (size_t)nb + 2u * b)));
    } else if (KIND == IE_B200_MAT_Q4K) {
      const uint32_t dd = *reinterpret_cast<const uint32_t *>(rp + 16u * (size_t)nb + 16u * b);
      v = 63.0f * (15.0f * fabsf(h2f((uint16_t)(dd & 0xFFFFu))) + fabsf(h2f((uint16_t)(dd >> 16))));
    } else {
      v = 4096.0f * fabsf(h2f(*reinterpret_cast<const uint16_t *>(rp + 26u * (size_t)nb + 2u * b)));
    }
    if (v < 3.0e38f) m = fmaxf(m, v);
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) atomicMax(out_bits, __float_as_uint(m));  // non-negative floats order as their bits
}
}  // namespace ieb

extern "C" int ie_b200_mat_tc_exp(int kind, const void *d_w, uint32_t rows, uint32_t cols, int *h_exp, void *stream) {
  if (!d_w || !h_exp) return fail(IE_B200_E_ARG, "ie_b200_mat_tc_exp: NULL pointer");
  if (kind != IE_B200_MAT_Q4 && kind != IE_B200_MAT_Q8 && kind != IE_B200_MAT_Q4K && kind != IE_B200_MAT_Q6K)
    return fail(IE_B200_E_ARG, "ie_b200_mat_tc_exp: matrix kind %d", kind);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint32_t *d_bits = nullptr, bits = 0;
  IEB_CUDA(cudaMalloc(&d_bits, 4));
  IEB_CUDA(cudaMemsetAsync(d_bits, 0, 4, st));
  const uint8_t *w = static_cast<const uint8_t *>(d_w);
  const size_t rowb = row_bytes_of(kind, cols);
  const uint32_t nb = cols / 32u, grid = 592;
  if (kind == IE_B200_MAT_Q4) tc_wbound_kernel<IE_B200_MAT_Q4><<<grid, 256, 0, st>>>(w, rowb, rows, nb, d_bits);
  else if (kind == IE_B200_MAT_Q8) tc_wbound_kernel<IE_B200_MAT_Q8><<<grid, 256, 0, st>>>(w, rowb, rows, nb, d_bits);
  else if (kind == IE_B200_MAT_Q4K) tc_wbound_kernel<IE_B200_MAT_Q4K><<<grid, 256, 0, st>>>(w, rowb, rows, nb, d_bits);
  else tc_wbound_kernel<IE_B200_MAT_Q6K><<<grid, 256, 0, st>>>(w, rowb, rows, nb, d_bits);
  count_launch();
  cudaError_t e = cudaMemcpyAsync(&bits, d_bits, 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(d_bits);
  if (e != cudaSuccess) return cuda_fail(e, "ie_b200_mat_tc_exp");
  float m;
  memcpy(&m, &bits, 4);
  int ex = 0, s = 0;
  if (m > 0.0f) {
    frexpf(m, &ex);  // m < 2^ex
    s = 13 - ex;     // bound * 2^s < 8192
    s = s > 100 ? 100 : (s < -100 ? -100 : s);
  }
  *h_exp = s;
  return IE_B200_OK;
}

// act_ready: the scratch already holds the expanded activations of these Q8 rows (a call with the same columns and tokens was
// launched on the stream before this one, and nothing has written to the scratch since).
int ieb::gemm_tc_run(int kind, const void *d_w, uint32_t rows, uint32_t cols, int w_exp, const void *d_xq, float *d_y, const float *d_bias, const float *d_res,
                     uint32_t T, size_t x_stride, size_t y_stride, size_t res_stride, void *d_scratch, size_t scratch_bytes, uint32_t *d_err, cudaStream_t st,
                     bool act_ready) {
  if (!d_w || !d_xq || !d_y || !d_scratch) return fail(IE_B200_E_ARG, "ie_b200_gemm_tc: NULL pointer");
  if (kind != IE_B200_MAT_Q4 && kind != IE_B200_MAT_Q8 && kind != IE_B200_MAT_Q4K && kind != IE_B200_MAT_Q6K)
    return fail(IE_B200_E_ARG, "ie_b200_gemm_tc: matrix kind %d (Q4_0, Q8_0, Q4_K, Q6_K)", kind);
  if (cols == 0 || cols % ((kind == IE_B200_MAT_Q4 || kind == IE_B200_MAT_Q8) ? 32u : 256u)) return fail(IE_B200_E_SIZE, "ie_b200_gemm_tc: %u columns", cols);
  if (rows == 0 || T == 0) return IE_B200_OK;
  if (!aligned16(d_w) || !aligned16(d_xq) || (x_stride & 15u) || (y_stride & 3u) || (res_stride & 3u) || ((uintptr_t)d_scratch & 255u))
    return fail(IE_B200_E_ARG, "ie_b200_gemm_tc: the matrix and the Q8 rows must be 16-byte aligned, strides multiples of 4, the scratch 256-byte aligned");
  if (scratch_bytes < tc_scratch(rows, cols, T)) return fail(IE_B200_E_SIZE, "ie_b200_gemm_tc: scratch of %zu bytes, %zu needed", scratch_bytes, tc_scratch(rows, cols, T));
  const uint32_t nb = cols / 32u, nt = (T + TC_TOK - 1) / TC_TOK, splits = tc_splits(rows, nb, T);
  if (w_exp < -100 || w_exp > 100) return fail(IE_B200_E_ARG, "ie_b200_gemm_tc: weight exponent %d", w_exp);
  uint8_t *bp = static_cast<uint8_t *>(d_scratch);
  const size_t bp_bytes = ((size_t)nt * nb * TC_TOK * TC_TOK_STAGE + 255u) & ~(size_t)255u, sc_bytes = ((size_t)nt * TC_TOK * sizeof(float) + 255u) & ~(size_t)255u;
  float *tok_inv = reinterpret_cast<float *>(bp + bp_bytes);
  float *partial = splits > 1u ? reinterpret_cast<float *>(bp + bp_bytes + sc_bytes) : nullptr;
  if (!act_ready) {
    // about four CTAs per SM, at least 32 blocks each
    const uint32_t groups = (nt - 1u) * (TC_TOK / 8u) + tc_pad(T, nt - 1u) / 8u, parts = std::min((nb + 31u) / 32u, (4u * sm_count() + groups - 1u) / groups);
    IEB_LAUNCH_PDL("tc_expand_kernel", tc_expand_kernel, dim3(groups, parts), dim3(256), 0, st, static_cast<const uint8_t *>(d_xq), x_stride, T, nb, tok_inv, bp);
  }
  TcArgs a = {};
  a.w = static_cast<const uint8_t *>(d_w), a.rowb = row_bytes_of(kind, cols), a.rows = rows, a.nb = nb, a.T = T;
  // (not rounded up to whole raw stages: a longer accumulation loses more, 4096 x 4096 Q4_0 above 128 tokens 1.60e-6 against 64 bits with
  // 15 blocks per split, 1.74e-6 with 16)
  a.blocks_per_split = (nb + splits - 1u) / splits;
  a.bp = bp, a.y = d_y, a.bias = d_bias, a.res = d_res, a.ys = y_stride, a.rs = res_stride, a.partial = partial, a.err = d_err;
  a.w_scale = ldexpf(1.0f, w_exp), a.w_inv = ldexpf(1.0f, -w_exp), a.tok_inv = tok_inv;
  const uint32_t used_splits = (nb + a.blocks_per_split - 1u) / a.blocks_per_split;
  const dim3 grid((rows + TC_ROWS - 1) / TC_ROWS, nt, partial ? used_splits : 1u);
  void (*k)(TcArgs) = kind == IE_B200_MAT_Q4 ? gemm_tc_kernel<IE_B200_MAT_Q4> : kind == IE_B200_MAT_Q8 ? gemm_tc_kernel<IE_B200_MAT_Q8>
                      : kind == IE_B200_MAT_Q4K ? gemm_tc_kernel<IE_B200_MAT_Q4K> : gemm_tc_kernel<IE_B200_MAT_Q6K>;
  // stages: as many as fit, the activations' ring first (its copies come from L2, the producers are next door)
  const uint32_t bst = std::min((T + 15u) & ~15u, (uint32_t)TC_TOK) * TC_TOK_STAGE;
  const uint32_t raw = TC_PROD_WARPS * 2u * (kind == IE_B200_MAT_Q4 ? RS_BYTES<IE_B200_MAT_Q4> : kind == IE_B200_MAT_Q8 ? RS_BYTES<IE_B200_MAT_Q8>
                                             : kind == IE_B200_MAT_Q4K ? RS_BYTES<IE_B200_MAT_Q4K> : RS_BYTES<IE_B200_MAT_Q6K>);
  auto smem_of = [&](uint32_t sa, uint32_t sb) { return sa * TC_A_STAGE + sb * bst + raw + TC_BARS; };
  a.sa = a.sb = 2u;
  for (int s = 3; s <= TC_MAX_ST; s++) {
    if (smem_of(a.sa, a.sb + 1u) <= TC_SMEM) a.sb++;
    if (smem_of(a.sa + 1u, a.sb) <= TC_SMEM) a.sa++;
  }
  const uint32_t smem = smem_of(a.sa, a.sb);
  if (int r = ensure_dynamic_smem(reinterpret_cast<const void *>(k), smem)) return r;
  IEB_LAUNCH_PDL("gemm_tc_kernel", k, grid, dim3(TC_THREADS), smem, st, a);
  const bool vec = rows % 4u == 0 && !(((uintptr_t)d_y | y_stride | (uintptr_t)d_res | res_stride | (uintptr_t)partial) & 15u);
  if (partial && vec)
    IEB_LAUNCH_PDL("tc_reduce4_kernel", tc_reduce4_kernel, dim3((rows / 4u + 127u) / 128u, T), dim3(128), 0, st, static_cast<const float *>(partial), used_splits, T,
                   rows, d_y, d_bias, d_res, y_stride, res_stride);
  else if (partial)
    IEB_LAUNCH_PDL("tc_reduce_kernel", tc_reduce_kernel, dim3((rows + 255u) / 256u, T), dim3(256), 0, st, static_cast<const float *>(partial), used_splits, T, rows, d_y,
                   d_bias, d_res, y_stride, res_stride);
  return IE_B200_OK;
}

extern "C" int ie_b200_gemm_tc(int kind, const void *d_w, uint32_t rows, uint32_t cols, int w_exp, const void *d_xq, float *d_y, const float *d_bias,
                               const float *d_res, uint32_t T, size_t x_stride, size_t y_stride, size_t res_stride, void *d_scratch, size_t scratch_bytes,
                               uint32_t *d_err, void *stream) {
  return gemm_tc_run(kind, d_w, rows, cols, w_exp, d_xq, d_y, d_bias, d_res, T, x_stride, y_stride, res_stride, d_scratch, scratch_bytes, d_err,
                     static_cast<cudaStream_t>(stream), false);
}
