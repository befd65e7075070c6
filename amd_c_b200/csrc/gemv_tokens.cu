// gemv_tokens.cu -- 2..16 tokens per pass over the weights (drafted tokens checked in one pass, short prompt tails; the role of
// ie_gemv_q4kq8_tr / _ts2 in the reference, kernels/ie_kernels.c:483-628), every token's row bit for bit the one-token GEMV's.
//
// The block dots come from the int8 tensor cores: one mma.sync m16n8k32 is the exact int32 dot of one 32-weight block for 16
// rows x 8 tokens. With dp4a per token the kernel was bound by instruction issue; here the work per block and token is the
// scaling in fp32, two tokens per instruction (f32x2). What bounds it now is still issue: about 55 instructions per 16 rows x one
// block x 8 tokens, 16 warps of 128 registers per SM (24 warps of 80 were slower: 28672 x 4096 24 against 22 us).
// Measured, dp4a -> now, 6 tokens: 28672 x 4096 Q4_0 58 -> 22 us, 4096 x 14336 Q4_0 49 -> 16, 128256 x 4096 Q4_0 222 -> 81, 37888 x
// 3584 Q4_K 86 -> 29, 3584 x 18944 Q6_K 88 -> 28; 2 tokens: 41 -> 21, 35 -> 14, 155 -> 80, 55 -> 28, 58 -> 26; 16 tokens: 154 -> 35,
// 101 -> 30, 646 -> 126, 197 -> 42, 185 -> 50.
// Rows whose activations do not fit (see gemv_tokens_phases) are worked in phases: Q8_0 28672 x 4096 6 / 16 tokens 68 -> 23 / 111 -> 61 us, 5120 x
// 17408 86 -> 32 / 179 -> 63.
//
// Order: the one-token GEMV gives lane l of a warp the blocks l, l + 32, ... in order and adds the 32 lane sums by a tree
// (16, 8, 4, 2, 1). Warp w of the eight that share a 16-row tile keeps the sums of "lanes" 4 w .. 4 w + 3 in registers (four
// adjacent blocks of every 32: 64 contiguous bytes of a row), and the tree over the 32 sums runs through shared memory.
//
// Memory: each warp streams its own blocks through a private ring of cp.async stages (16 rows x 4 blocks each, no barrier
// among warps; ldmatrix hands thread (g, t) word t of row g, which is the A fragment's word), so that 16 warps x 5 stages =
// 90 KB per SM are in flight (Q4_0, up to 8 tokens; 3 stages behind the one being worked for Q6_K, Q8_0 and above 8 tokens); the first stages are asked for before the kernel waits for its predecessor. The activations of a
// CTA are staged in the order of the B fragments; rows longer than fit are worked in phases over the columns.
#include <algorithm>

#include "common.cuh"
#include "row_stage.cuh"

namespace ieb {

constexpr int GT_WARPS = 16, GT_THREADS = GT_WARPS * 32;       // two 16-row tiles of eight warps each
constexpr uint32_t GT_RED_LANE = 176;                          // floats per lane sum of a tile: 8 tokens x 20 (16 rows, padded), 16 mod 32
constexpr uint32_t GT_RED = 32u * GT_RED_LANE * 4u;            // of one tile
constexpr uint32_t GT_SMEM = 227u * 1024u;
constexpr int GT_BIAS = 0x4B400000;                            // 1.5 * 2^23: an int32 |n| < 2^22 added to these bits is the float 12582912 + n

template <int KIND> struct GtKind;  // bytes of a block's scaling data per token tile, stages of a warp's ring (8 tokens)
template <> struct GtKind<IE_B200_MAT_Q4> { static constexpr uint32_t DS = 64, SMAX = 6; };
template <> struct GtKind<IE_B200_MAT_Q8> { static constexpr uint32_t DS = 64, SMAX = 4; };
template <> struct GtKind<IE_B200_MAT_Q4K> { static constexpr uint32_t DS = 64, SMAX = 6; };
template <> struct GtKind<IE_B200_MAT_Q6K> { static constexpr uint32_t DS = 96, SMAX = 4; };

// Stages of a warp's ring: as many as leave room for the activations.
template <int KIND, int NT>
constexpr int GT_STAGES = NT == 1 ? (int)GtKind<KIND>::SMAX : 4;

struct GtArgs {
  const uint8_t *w;
  size_t rowb;
  uint32_t rows, nb, T;
  uint32_t P;  // blocks of a phase (a multiple of 32)
  const uint8_t *xq;
  float *y;
  const float *bias, *res;
  size_t xs, ys, rs;
};

// two int32 sums that were started at GT_BIAS, as floats
__device__ __forceinline__ f32x2 dots2(int a, int b) { return add2(pk2(__int_as_float(a), __int_as_float(b)), pk2(-12582912.0f, -12582912.0f)); }

template <bool UNSIGNED_A>
__device__ __forceinline__ void gt_mma32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int i0, int i1) {
  if (UNSIGNED_A)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(i0), "r"(i1));
  else
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%10,%11};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(i0), "r"(i1));
}
__device__ __forceinline__ void gt_mma16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0, int i0, int i1) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%7,%8};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(i0), "r"(i1));
}
__device__ __forceinline__ void gt_ldm4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}

// The activations of blocks [lo, hi) of tokens t0 .. : B fragments [block][tile][token][t] = words t and t + 4 of the token's
// block, then per (block, tile, t) what the scaling of tokens 2 t and 2 t + 1 needs.
template <int KIND, int NT>
__device__ __forceinline__ void gt_stage_act(const GtArgs &a, uint32_t t0, uint32_t lo, uint32_t hi, uint8_t *sB, uint8_t *sD) {
  const uint32_t nb = a.nb, n = (hi - lo) * 8u * NT;
  for (uint32_t k = threadIdx.x; k < n; k += GT_THREADS) {
    const uint32_t tok = k % (8u * NT), bl = k / (8u * NT), b = lo + bl;
    uint4 q0 = make_uint4(0u, 0u, 0u, 0u), q1 = q0;
    float d = 0.0f;
    int s = 0;
    if (b < nb && t0 + tok < a.T) {
      const uint8_t *row = a.xq + (size_t)(t0 + tok) * a.xs;
      q0 = *reinterpret_cast<const uint4 *>(row + 32u * (size_t)b), q1 = *reinterpret_cast<const uint4 *>(row + 32u * (size_t)b + 16u);
      d = *reinterpret_cast<const float *>(row + 32u * (size_t)nb + 4u * b);
      s = *reinterpret_cast<const int *>(row + 36u * (size_t)nb + 4u * b);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(sB + ((size_t)bl * 8u * NT + tok) * 32u);
    dst[0] = make_uint4(q0.x, q1.x, q0.y, q1.y), dst[1] = make_uint4(q0.z, q1.z, q0.w, q1.w);
    float *ds = reinterpret_cast<float *>(sD + ((size_t)bl * NT + (tok >> 3)) * GtKind<KIND>::DS) + ((tok & 7u) >> 1) * 4u + (tok & 1u);
    ds[0] = d;
    if (KIND == IE_B200_MAT_Q4) ds[2] = __int_as_float(GT_BIAS - 8 * s);
    if (KIND == IE_B200_MAT_Q4K) ds[2] = __fmul_rn(d, (float)s);
    if (KIND == IE_B200_MAT_Q6K) {  // q - 32: the halves' sums of the activations, times 32
      int h0 = __dp4a(0x01010101, (int)q0.x, 0), h1 = __dp4a(0x01010101, (int)q1.x, 0);
      h0 = __dp4a(0x01010101, (int)q0.y, h0), h0 = __dp4a(0x01010101, (int)q0.z, h0), h0 = __dp4a(0x01010101, (int)q0.w, h0);
      h1 = __dp4a(0x01010101, (int)q1.y, h1), h1 = __dp4a(0x01010101, (int)q1.z, h1), h1 = __dp4a(0x01010101, (int)q1.w, h1);
      ds[2] = __int_as_float(GT_BIAS - 32 * h0);
      (reinterpret_cast<int *>(sD + ((size_t)bl * NT + (tok >> 3)) * GtKind<KIND>::DS + 64u))[tok & 7u] = GT_BIAS - 32 * h1;
    }
  }
}

// The four blocks of a stage: acc[i][h][n] += block 4 w + i, rows g + 8 h, tokens 2 t and 2 t + 1 of token tile n.
template <int KIND, int NT>
__device__ __forceinline__ void gt_step(const uint8_t *stp, uint32_t b0, const uint8_t *sB, const uint8_t *sD, f32x2 (&acc)[4][2][NT], int lane) {
  const uint32_t st = smem_u32(stp), g = (uint32_t)lane >> 2, t = lane & 3u;
  const uint32_t lr = lane & 15u;                      // ldmatrix: lanes 0..15 give the rows of the first pair of matrices,
  const uint32_t lh = (uint32_t)lane >> 4;             // lanes 16..31 those of the second
  float s0[2], s1[2];                                  // K kinds: thread t works out the scales of block t for rows g, g + 8
  uint2 sw[2];                                         // Q4_0 / Q8_0: four f16 scales of rows g, g + 8
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t r = g + 8u * h;
    s0[h] = s1[h] = 0.0f, sw[h] = make_uint2(0u, 0u);
    if (KIND == IE_B200_MAT_Q4) sw[h] = *reinterpret_cast<const uint2 *>(stp + 1024u + 8u * r);
    if (KIND == IE_B200_MAT_Q8) sw[h] = *reinterpret_cast<const uint2 *>(stp + 2048u + 8u * r);
    if (KIND == IE_B200_MAT_Q4K) {
      const uint4 hd = *reinterpret_cast<const uint4 *>(stp + 1024u + 16u * r);
      const uint32_t f = q4k_field(hd, (int)((b0 & 7u) + t));
      const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&hd.x));
      s0[h] = __fmul_rn(dd.x, (float)(f & 63u)), s1[h] = -__fmul_rn(dd.y, (float)(f >> 6));
    }
    if (KIND == IE_B200_MAT_Q6K) {
      const uint16_t sc = *reinterpret_cast<const uint16_t *>(stp + 1536u + 8u * r + 2u * t);
      const float df = h2f(*reinterpret_cast<const uint16_t *>(stp + 1664u + 4u * r + 2u * ((b0 >> 3) & 1u)));
      s0[h] = __fmul_rn(df, (float)(int8_t)(sc & 255u)), s1[h] = __fmul_rn(df, (float)(int8_t)(sc >> 8));
    }
  }
  uint32_t m[4];
#pragma unroll
  for (uint32_t i = 0; i < 4; i++) {
    uint32_t a0, a1, a2, a3;
    if (KIND == IE_B200_MAT_Q8) {
      gt_ldm4(st + lr * 128u + (((2u * i + lh) ^ (lr & 7u)) << 4), a0, a1, a2, a3);
    } else {
      if ((i & 1u) == 0u) gt_ldm4(st + lr * 64u + (((i + lh) ^ ((lr >> 1) & 3u)) << 4), m[0], m[1], m[2], m[3]);
      const uint32_t w0 = m[2 * (i & 1u)], w1 = m[2 * (i & 1u) + 1u];
      a0 = w0 & 0x0F0F0F0Fu, a1 = w1 & 0x0F0F0F0Fu, a2 = (w0 >> 4) & 0x0F0F0F0Fu, a3 = (w1 >> 4) & 0x0F0F0F0Fu;
      if (KIND == IE_B200_MAT_Q6K) {
        const uint2 x0 = *reinterpret_cast<const uint2 *>(stp + 1024u + 32u * g + 8u * i), x1 = *reinterpret_cast<const uint2 *>(stp + 1024u + 32u * (g + 8u) + 8u * i);
        a0 |= ((x0.x >> (2u * t)) & 0x03030303u) << 4, a1 |= ((x1.x >> (2u * t)) & 0x03030303u) << 4;
        a2 |= ((x0.y >> (2u * t)) & 0x03030303u) << 4, a3 |= ((x1.y >> (2u * t)) & 0x03030303u) << 4;
      }
    }
    float u0[2], u1[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (KIND == IE_B200_MAT_Q4 || KIND == IE_B200_MAT_Q8) {
        u0[h] = h2f((uint16_t)((i < 2 ? sw[h].x : sw[h].y) >> (16u * (i & 1u)))), u1[h] = 0.0f;
      } else {
        u0[h] = __shfl_sync(0xFFFFFFFFu, s0[h], (lane & 28) | (int)i), u1[h] = __shfl_sync(0xFFFFFFFFu, s1[h], (lane & 28) | (int)i);
      }
    }
#pragma unroll
    for (int n = 0; n < NT; n++) {
      const uint2 bf = *reinterpret_cast<const uint2 *>(sB + (i * NT + n) * 256u + 8u * lane);
      const uint8_t *dp = sD + (i * NT + n) * GtKind<KIND>::DS;
      const float4 ds = *reinterpret_cast<const float4 *>(dp + 16u * t);
      const f32x2 da = pk2(ds.x, ds.y);
      int c[4];
      if (KIND == IE_B200_MAT_Q6K) {
        const int2 i1 = *reinterpret_cast<const int2 *>(dp + 64u + 8u * t);
        int c1[4];
        gt_mma16(c, a0, a1, bf.x, __float_as_int(ds.z), __float_as_int(ds.w));
        gt_mma16(c1, a2, a3, bf.y, i1.x, i1.y);
#pragma unroll
        for (int h = 0; h < 2; h++)  // acc = fma(fma(d sc1, d1, (d sc0) d0), da, acc)
          acc[i][h][n] = fma2(fma2(pk2(u1[h], u1[h]), dots2(c1[2 * h], c1[2 * h + 1]), mul2(pk2(u0[h], u0[h]), dots2(c[2 * h], c[2 * h + 1]))), da, acc[i][h][n]);
      } else if (KIND == IE_B200_MAT_Q4K) {
        gt_mma32<true>(c, a0, a1, a2, a3, bf.x, bf.y, GT_BIAS, GT_BIAS);
#pragma unroll
        for (int h = 0; h < 2; h++)  // acc = fma(-(dmin mn), da asum, fma((d sc) dq, da, acc))
          acc[i][h][n] = fma2(pk2(u1[h], u1[h]), pk2(ds.z, ds.w), fma2(mul2(pk2(u0[h], u0[h]), dots2(c[2 * h], c[2 * h + 1])), da, acc[i][h][n]));
      } else {
        if (KIND == IE_B200_MAT_Q4) gt_mma32<true>(c, a0, a1, a2, a3, bf.x, bf.y, __float_as_int(ds.z), __float_as_int(ds.w));
        else gt_mma32<false>(c, a0, a1, a2, a3, bf.x, bf.y, GT_BIAS, GT_BIAS);
#pragma unroll
        for (int h = 0; h < 2; h++) {  // acc = acc + (dw da) dot, product and sum rounded each (the assembler joins a packed pair of the two into one fma)
          float p0, p1, s0, s1;
          unpk2(mul2(mul2(pk2(u0[h], u0[h]), da), dots2(c[2 * h], c[2 * h + 1])), p0, p1);
          unpk2(acc[i][h][n], s0, s1);
          acc[i][h][n] = pk2(__fadd_rn(s0, p0), __fadd_rn(s1, p1));
        }
      }
    }
  }
}

template <int KIND, int NT>
__global__ void __launch_bounds__(GT_THREADS, 1) gemv_tokens_kernel(const GtArgs a) {
  constexpr int S = GT_STAGES<KIND, NT>;
  constexpr uint32_t STAGE = RS_BYTES<KIND>, DS = GtKind<KIND>::DS;
  extern __shared__ __align__(128) uint8_t smem_gt[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, w = warp & 7, half = warp >> 3;
  uint8_t *ring = smem_gt + (uint32_t)warp * S * STAGE;
  float *red = reinterpret_cast<float *>(smem_gt + GT_WARPS * S * STAGE) + half * 32u * GT_RED_LANE;
  uint8_t *sB = smem_gt + GT_WARPS * S * STAGE + 2u * GT_RED, *sD = sB + (size_t)a.P * NT * 256u;
  pdl_launch_dependents();
  const uint32_t nb = a.nb, tiles = (a.rows + 15u) / 16u, t0 = blockIdx.y * 8u * NT;
  // tiles of this half of the CTA: slot, slot + 2 gridDim.x, ... (the first halves of all CTAs come first)
  const uint32_t slot = half * gridDim.x + blockIdx.x, stride = 2u * gridDim.x;
  const uint32_t mine = slot < tiles ? (tiles - slot + stride - 1u) / stride : 0u, most = (tiles - blockIdx.x + stride - 1u) / stride;
  const uint32_t steps = nb > 4u * w ? (nb - 4u * w + 31u) / 32u : 0u;  // of this warp, per tile
  const uint32_t items = mine * steps;
  // next item to ask for; the rows' addresses are worked out once per tile (rows past the end: copies that are not stored)
  RsRows<KIND> rr;
  uint32_t in = 0, it_tile = slot, it_j = 0, it_stage = 0;
  auto issue = [&]() {
    if (in < items) {
      if (it_j == 0u) rr.set(a.w, a.rowb, a.rows, nb, it_tile * 16u, lane);
      rs_issue_rows<KIND>(rr, nb, smem_u32(ring + it_stage * STAGE), 32u * it_j + 4u * w, lane);
      in++;
      if (++it_j == steps) it_j = 0, it_tile += stride;
    }
    if (++it_stage == S) it_stage = 0;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < S - 1; s++) issue();
  pdl_wait();
  const uint32_t phases = (nb + a.P - 1u) / a.P;
  if (phases == 1u) {
    gt_stage_act<KIND, NT>(a, t0, 0u, (nb + 3u) & ~3u, sB, sD);
    __syncthreads();
  }
  uint32_t stage = 0;
  for (uint32_t k = 0; k < most; k++) {
    f32x2 acc[4][2][NT];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int n = 0; n < NT; n++) acc[i][0][n] = acc[i][1][n] = 0ull;
    for (uint32_t p = 0; p < phases; p++) {
      const uint32_t lo = p * a.P, hi = min(lo + a.P, (nb + 3u) & ~3u);
      if (phases > 1u) {
        __syncthreads();  // the last phase's activations have been read
        gt_stage_act<KIND, NT>(a, t0, lo, hi, sB, sD);
        __syncthreads();
      }
      if (k < mine) {
        for (uint32_t b0 = lo + 4u * w; b0 < hi; b0 += 32u) {
          asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
          __syncwarp();  // every lane's part of the stage has arrived, and the stage before it has been read by all
          issue();
          gt_step<KIND, NT>(ring + stage * STAGE, b0, sB + (size_t)(b0 - lo) * NT * 256u, sD + (size_t)(b0 - lo) * NT * DS, acc, lane);
          if (++stage == S) stage = 0;
        }
      }
    }
    if (k >= mine) continue;
    // ---- the tree over the 32 lane sums, one token tile at a time; warps of this half only
    const uint32_t g = (uint32_t)lane >> 2, t = lane & 3u, row0 = (slot + k * stride) * 16u;
    const uint32_t row = lane & 15u, part = (uint32_t)lane >> 4, tok = (uint32_t)w;  // a warp per token, sixteen rows, two halves of the tree
#pragma unroll
    for (int n = 0; n < NT; n++) {
      asm volatile("bar.sync %0, 256;" ::"r"(1 + half) : "memory");  // the sums before these have been read
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float *dst = red + (4u * w + i) * GT_RED_LANE + 2u * t * 20u + g;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          float v0, v1;
          unpk2(acc[i][h][n], v0, v1);
          dst[8 * h] = v0, dst[20 + 8 * h] = v1;
        }
      }
      asm volatile("bar.sync %0, 256;" ::"r"(1 + half) : "memory");
      float sum[2];
#pragma unroll
      for (int q = 0; q < 2; q++) {  // lanes 4 v + i, v = 0 .. 7, of i = part and part + 2
        const float *src = red + (part + 2u * q) * GT_RED_LANE + tok * 20u + row;
        float x[8];
#pragma unroll
        for (int v = 0; v < 8; v++) x[v] = src[4u * v * GT_RED_LANE];
        sum[q] = __fadd_rn(__fadd_rn(__fadd_rn(x[0], x[4]), __fadd_rn(x[2], x[6])), __fadd_rn(__fadd_rn(x[1], x[5]), __fadd_rn(x[3], x[7])));
      }
      float o = __fadd_rn(sum[0], sum[1]);
      o = __fadd_rn(o, __shfl_down_sync(0xFFFFFFFFu, o, 16));
      const uint32_t gr = row0 + row, gt = t0 + 8u * n + tok;
      if (part == 0u && gr < a.rows && gt < a.T) {
        if (a.bias) o = __fadd_rn(o, a.bias[gr]);
        if (a.res) o = __fadd_rn(reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.res) + (size_t)gt * a.rs)[gr], o);
        reinterpret_cast<float *>(reinterpret_cast<char *>(a.y) + (size_t)gt * a.ys)[gr] = o;
      }
    }
  }
}

// Shared memory of the rings and the reduction, of a block's activations, and blocks whose activations fit beside the former.
template <int KIND, int NT>
struct GtFit {
  static constexpr uint32_t fixed = 2u * (8u * GT_STAGES<KIND, NT> * RS_BYTES<KIND> + GT_RED), per = NT * (256u + GtKind<KIND>::DS);
  static constexpr uint32_t cap = (GT_SMEM - fixed) / per / 32u * 32u;
  static_assert(cap >= 32u, "a phase is at least 32 blocks");
};
template <int KIND, int NT>
static uint32_t gt_phases(uint32_t nb) {
  return (((nb + 31u) & ~31u) + GtFit<KIND, NT>::cap - 1u) / GtFit<KIND, NT>::cap;
}
// Phases over the columns of a pass of sixteen tokens (5120 columns fit for Q4_0 and Q4_K, 3072 for Q6_K, 2048 for Q8_0): with more
// than one, every 16-row tile stages its activations anew.
uint32_t gemv_tokens_phases(int kind, uint32_t cols) {
  const uint32_t nb = cols / 32u;
  switch (kind) {
    case IE_B200_MAT_Q4: return gt_phases<IE_B200_MAT_Q4, 2>(nb);
    case IE_B200_MAT_Q8: return gt_phases<IE_B200_MAT_Q8, 2>(nb);
    case IE_B200_MAT_Q4K: return gt_phases<IE_B200_MAT_Q4K, 2>(nb);
    default: return gt_phases<IE_B200_MAT_Q6K, 2>(nb);
  }
}

template <int KIND, int NT>
static int launch_tokens(GtArgs a, cudaStream_t st) {
  constexpr uint32_t fixed = GtFit<KIND, NT>::fixed, per = GtFit<KIND, NT>::per;
  // the fewest phases whose activations fit beside the rings, all of about the same length
  const uint32_t up = (a.nb + 31u) & ~31u, phases = gt_phases<KIND, NT>(a.nb);
  a.P = (up / 32u + phases - 1u) / phases * 32u;
  const size_t smem = fixed + (size_t)a.P * per;
  auto k = gemv_tokens_kernel<KIND, NT>;
  if (int r = ensure_dynamic_smem(reinterpret_cast<const void *>(k), smem)) return r;
  const uint32_t tiles = (a.rows + 15u) / 16u;
  const dim3 grid(std::min(tiles, (uint32_t)sm_count()), (a.T + 8u * NT - 1u) / (8u * NT));
  IEB_LAUNCH_PDL("gemv_tokens_kernel", k, grid, dim3(GT_THREADS), smem, st, a);
  return IE_B200_OK;
}

// Sixteen tokens per pass, the last eight or fewer with one token tile.
template <int KIND>
static int pick_tokens(GtArgs a, cudaStream_t st) {
  const uint32_t tail = a.T % 16u, two = tail > 8u ? a.T : a.T - tail;  // tokens worked sixteen at a time
  const uint32_t all = a.T;
  if (two) {
    a.T = two;
    if (int r = launch_tokens<KIND, 2>(a, st)) return r;
  }
  if (two == all) return IE_B200_OK;
  a.T = all - two;
  a.xq += (size_t)two * a.xs;
  a.y = reinterpret_cast<float *>(reinterpret_cast<char *>(a.y) + (size_t)two * a.ys);
  if (a.res) a.res = reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.res) + (size_t)two * a.rs);
  return launch_tokens<KIND, 1>(a, st);
}

// y[t] = W x[t] (+ bias) (+ res[t]) for T >= 2 tokens; the checks are ie_b200_gemv's.
int gemv_tokens(int kind, const void *d_w, uint32_t rows, uint32_t cols, const void *d_x, float *d_y, const float *d_bias, const float *d_res, uint32_t T,
                size_t xs, size_t ys, size_t rs, cudaStream_t st) {
  GtArgs a = {};
  a.w = static_cast<const uint8_t *>(d_w), a.rowb = row_bytes_of(kind, cols), a.rows = rows, a.nb = cols / 32u, a.T = T;
  a.xq = static_cast<const uint8_t *>(d_x), a.y = d_y, a.bias = d_bias, a.res = d_res, a.xs = xs, a.ys = ys, a.rs = rs;
  switch (kind) {
    case IE_B200_MAT_Q4: return pick_tokens<IE_B200_MAT_Q4>(a, st);
    case IE_B200_MAT_Q8: return pick_tokens<IE_B200_MAT_Q8>(a, st);
    case IE_B200_MAT_Q4K: return pick_tokens<IE_B200_MAT_Q4K>(a, st);
    case IE_B200_MAT_Q6K: return pick_tokens<IE_B200_MAT_Q6K>(a, st);
    default: return fail(IE_B200_E_ARG, "ie_b200_gemv: unknown matrix kind %d", kind);
  }
}

}  // namespace ieb
