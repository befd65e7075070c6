// attn_prefill_tc.cu -- causal attention of a prompt chunk on the 5th-generation tensor cores (tcgen05 + tensor memory):
// T tokens at positions *pos .. *pos + T - 1 whose K / V rows are already in the half-precision cache; the role of
// ie_attn_pfg / ie_attn_fa (kernels/ie_kernels.c:3471-3693; dispatch src/hip.c:1432-1463).
//
// The rows of one KV head are its (token, query head) pairs, token-major: T x G of them. A CTA takes 128 or 256 rows (tiles of
// 128 = the rows of one MMA) of one KV head and one split of the positions, and walks the split's cache rows in blocks of
// 128: S = Q K^T into tensor memory, softmax by one thread per row, P back into the columns of S, O += P V. Q and P are
// carried as two f16 terms (22 significant bits, as everywhere on the half cache), K and V are exact, sums are fp32:
//   MMAs per block and tile: (q_hi + q_lo) K and (p_hi + p_lo) V, 128 x 128 x hd each.
// Bound: the tensor pipe (4 x 128 x 128 x hd multiply-adds per block and tile, about 2000 cycles at hd 128); the softmax of
// one tile (some 900 issue slots per warp) runs under the MMAs of the other. The kernel it replaced (mma.sync, 16 rows per
// CTA: the cache re-read from L2 for every 16 rows, 84 TFLOP/s) took 2048 us for 256 tokens x 40 heads at 32.5 k positions
// and 192 us for 256 x 28 at 4 k. It is kept for small chunks (attn_decode.cu; the rule is at attn_prefill_tc).
//
// Tensor memory (512 columns): S / P of the two tiles (128 each; 32 keys' S columns become 16 columns of p_hi and 16 of p_lo
// in place, so a thread never holds more than 32 scores), O of the two tiles (hd each).
// Shared memory: Q as MMA core matrices (hd x 256 B per term and tile), a ring of three K or V blocks (128 rows) brought by
// TMA in the 128-byte swizzle (boxes of 64 columns), one thread issuing. (cp.async in 16-byte pieces needed some 3500 cycles
// to issue a block from three warps and left the tensor pipe half idle.) V rows past the last position are zeroed in shared
// memory after they have landed: the cache may hold anything there, and 0 x NaN is not 0. For the same reason the blocks that
// some row of the CTA does not see whole are looked through for infinities and NaN (a value that overflowed the half cache must
// not reach the tokens before it): they are replaced by zeros, and added at the end to the rows that do see them.
// O is rescaled lazily: only when a row's maximum has grown by more than 2^8 (p stays far inside f16).
//
// Error. The tensor cores cut off what an accumulation loses (2^-25.7 of the accumulator per MMA, measured), so what counts is how
// many MMAs one accumulation takes. Low terms go first, into an accumulator that is still small: they cost next to nothing for S
// and at the start of O. An accumulation of O ends after a quarter of a row's blocks (pt_segment) and joins the row's sums, kept in
// fp32 by the softmax threads: in shared memory, or, for two tiles of heads of 128, which leave no room there, in the row's own
// memory. With four splits and more nothing joins (the merge adds the splits). Relative error against 64 bits (2-norm, random
// normal q, k, v, 32 x 8 heads of 128, 256 tokens, at 0 / 256 / 1000 / 8000 / 32000 positions, one split): 2.6e-7 / 4.0e-7 / 9.5e-7 /
// 4.9e-6 / 1.9e-5; high and low terms in turn and one accumulation: 5.2e-7 / 1.3e-6 / 3.0e-6 / 2.0e-5 / 7.5e-5; the mma.sync form
// (attn_decode.cu's scheme): 4.5e-7 / 7.3e-7 / 1.1e-6 / 5.2e-6 / 1.9e-5. With the splits that the launcher picks: 2.6e-7 / 4.0e-7 /
// 8.9e-7 / 4.9e-6 / 8.4e-6; 16 tokens at 4000 and 32000 positions 6.8e-7 and 4.8e-6. Exponentials by ex2.approx (2 units in the
// last place) in place of expf do not show in these figures.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math.h>

#include <algorithm>

#include "attn_prefill_tc.cuh"
#include "tc_common.cuh"

namespace ieb {

constexpr int PT_RING = 3, PT_KEYS = 128;

struct PtArgs {
  const float *q;
  float *out;
  uint8_t *oq;
  const uint32_t *pos;
  uint32_t n_head, n_kv, kv_len, T, G;
  size_t q_stride, out_stride, oq_stride;
  float scale_log2;  // log2(e) / sqrt(hd)
  float *part;       // [split][T x n_head rows][hd] unnormalised outputs, NULL: one split, final rows written here
  float *ml;         // [split][T x n_head][2] (max in log2 units, sum)
  uint32_t *err;
  uint32_t wide;     // bit 0: the rows written are 16-byte aligned, bit 1: the q rows are, bit 2: the rows written (or the records) are 32-byte aligned
  float inv_g;       // 1 / G
  const __half *vc;  // the V cache (read here only for rows that hold an infinity or a NaN)
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Eight neighbouring floats of a row: one 32-byte access (whole sectors, however far apart the lanes' rows lie) where aligned.
__device__ __forceinline__ void ld8(const float *p, float (&x)[8], bool wide) {
  if (wide) {
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]) : "l"(p) : "memory");
  } else {
#pragma unroll
    for (int e = 0; e < 8; e++) x[e] = p[e];
  }
}
__device__ __forceinline__ void st8(float *p, const uint32_t *v, bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
  } else {
#pragma unroll
    for (int e = 0; e < 8; e++) p[e] = __uint_as_float(v[e]);
  }
}

// Four neighbouring outputs of a (token, head) row per lane, eight lanes per block of 32: the row's floats and its Q8 copy.
template <int HD>
__device__ __forceinline__ void store_row4(float *out, size_t out_stride, uint8_t *oq, size_t oq_stride, uint32_t wide, uint32_t nbq, uint32_t tok, uint32_t head,
                                           uint32_t col, const float4 &o, bool in) {
  float *dst = reinterpret_cast<float *>(reinterpret_cast<char *>(out) + out_stride * tok) + (size_t)head * HD + col;
  if (in) {
    if (wide) *reinterpret_cast<float4 *>(dst) = o;
    else dst[0] = o.x, dst[1] = o.y, dst[2] = o.z, dst[3] = o.w;
  }
  if (!oq) return;
  float amax = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fmaxf(fabsf(o.z), fabsf(o.w)));
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, s));
  const float d = __fdiv_rn(amax, 127.0f), v[4] = {o.x, o.y, o.z, o.w};
  const Q8Div qd = q8_div(d);
  int sum = 0;
  uint32_t w = 0u;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int q = q8_round(v[e], qd);
    sum += q, w |= (uint32_t)(q & 255) << (8 * e);
  }
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, s);
  if (!in) return;
  uint8_t *qrow = oq + oq_stride * tok;
  const uint32_t at = head * HD + col;
  *reinterpret_cast<uint32_t *>(qrow + at) = w;
  if ((at & 31u) == 0u) reinterpret_cast<float *>(qrow + 32u * (size_t)nbq)[at / 32u] = d, reinterpret_cast<int *>(qrow + 36u * (size_t)nbq)[at / 32u] = sum;
}


// r / G for r below 2^22 (exact: r + 0.5 is at least 0.5 / G away from a multiple of G, the product's error below 2^-23 of it)
__device__ __forceinline__ uint32_t row_token(uint32_t r, float inv_g) { return (uint32_t)(((float)r + 0.5f) * inv_g); }

template <int HD>
struct PtSmem {
  static constexpr uint32_t QTERM = 128u * HD * 2u, BLOCK = PT_KEYS * HD * 2u;
  static constexpr uint32_t Q_OFF = 0u, KV_OFF = 4u * QTERM, BAR_OFF = KV_OFF + PT_RING * BLOCK, PAIR_OFF = BAR_OFF + 256u,
                            // rows' sums of the segments before: behind everything (heads of 64), in the second tile's Q (heads of 128, one tile)
                            SUM_OFF = HD == 64 ? PAIR_OFF + 2048u : Q_OFF + 2u * QTERM, TOTAL = PAIR_OFF + 2048u + (HD == 64 ? 2u * 128u * HD * 4u : 0u);
};

// Blocks of positions that one accumulation in tensor memory takes, of the n that a row tile has in all splits together; f: blocks
// that every row sees whole. A quarter of them; two (heads of 128: three) blocks that are mostly a diagonal stay together, most of
// their products are zeros (77 tokens x 32 heads of 128 at 200 positions: 5.3e-7, the mma.sync form 6.9e-7).
template <int HD>
__host__ __device__ constexpr uint32_t pt_segment(uint32_t n, uint32_t f) {
  return n <= (HD == 64 ? 2u : 3u) && f + 1u < n ? n : (n + 3u) / 4u;
}

// TILES: 128-row tiles of a CTA, eight softmax warps each.
template <int HD, int TILES>
__global__ void __launch_bounds__((8 * TILES + 2) * 32, 1) attn_prefill_tc_kernel(const PtArgs a, const __grid_constant__ CUtensorMap k_map,
                                                                                  const __grid_constant__ CUtensorMap v_map) {
  using L = PtSmem<HD>;
  constexpr int SOFT_WARPS = 8 * TILES, THREADS = (SOFT_WARPS + 2) * 32;
  constexpr bool SUM_SMEM = HD == 64 || TILES == 1;
  extern __shared__ __align__(1024) uint8_t smem_pt[];
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem_pt + L::BAR_OFF);
  uint64_t *kv_full = bars, *kv_empty = bars + PT_RING, *s_full = bars + 2 * PT_RING, *p_full = s_full + 2, *q_full = p_full + 2, *drained = q_full + 1,
           *tail = drained + 1, *pair_bar = tail + 1;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(pair_bar + 8);
  volatile uint32_t &s_abort = *(tmem_slot + 1), &s_bad = *(tmem_slot + 2);  // s_bad: zeros stand for infinities or NaN in V
  float *s_pair = reinterpret_cast<float *>(smem_pt + L::PAIR_OFF);  // [tile][half][row]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t g = blockIdx.y, split = blockIdx.z, rows_total = a.T * a.G, row0 = blockIdx.x * 128u * TILES;
  const uint32_t n_tiles = TILES == 2 && rows_total - row0 > 128u ? 2u : 1u;

  if (threadIdx.x == 0) {
    s_abort = 0u, s_bad = 0u;
    for (int i = 0; i < PT_RING; i++) mbar_init(&kv_full[i], 1u), mbar_init(&kv_empty[i], 1u);
    for (int t = 0; t < TILES; t++) mbar_init(&s_full[t], 1u), mbar_init(&p_full[t], 8u);
    mbar_init(q_full, 8u * n_tiles), mbar_init(drained, 1u), mbar_init(tail, 1u);
    for (int i = 0; i < 4 * TILES; i++) mbar_init(&pair_bar[i], 2u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == SOFT_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_prologue();

  // positions of this split: whole blocks of 128, dealt evenly (read by each role where it first needs them: the Q rows do not)
  uint32_t pos0 = 0u, first_lim = 0u, p_hi = 0u, b0 = 0u, n = 0u, seg = 1u;  // first_lim, p_hi: the fewest / most that a row of the CTA sees
  uint32_t issued = 0u;  // blocks asked for by the loader
  auto positions = [&] {
    pos0 = *a.pos, first_lim = pos0 + row_token(row0, a.inv_g) + 1u, p_hi = pos0 + row_token(min(rows_total, row0 + 128u * TILES) - 1u, a.inv_g) + 1u;
    const uint32_t blocks = (p_hi + PT_KEYS - 1u) / PT_KEYS, per = (blocks + gridDim.z - 1u) / gridDim.z;
    b0 = min(blocks, split * per), n = min(blocks, b0 + per) - b0, seg = pt_segment<HD>(blocks, first_lim / PT_KEYS);
  };

  if (warp < SOFT_WARPS) {
    // ---------------- softmax: eight warps per tile; warp w & 3 of them has 32 rows, one per lane, the two warps of a quarter half the columns each
    const uint32_t t = (uint32_t)warp >> 3, half = ((uint32_t)warp >> 2) & 1u, wq = (uint32_t)warp & 3u, rl = wq * 32u + lane, r = row0 + t * 128u + rl;
    const bool real = r < rows_total;
    const uint32_t tok = real ? row_token(r, a.inv_g) : 0u, head = g * a.G + (real ? r - tok * a.G : 0u);
    if (t < n_tiles) {
      const uint32_t lane_base = (wq * 32u) << 16, s_row = tmem + lane_base + t * 128u, o_col = tmem + lane_base + 256u + t * HD + half * (HD / 2u);
      uint64_t *pair = &pair_bar[t * 4u + wq];
      // Q rows -> two f16 terms as core matrices of 8 rows x 16 bytes: chunk c at 2048 c, row group at 128 (r / 8). A warp takes
      // 16 of the tile's rows; 8 rows x 4 chunks per step: 128 contiguous bytes of each row, and of shared memory per 8 lanes.
      {
        const uint32_t w8 = (uint32_t)warp & 7u;
        uint8_t *dst = smem_pt + L::Q_OFF + t * 2u * L::QTERM;
        float4 v[2][HD / 32][2];  // all of the rows' loads at once: one round trip
#pragma unroll
        for (uint32_t rg = 0; rg < 2; rg++) {
          const uint32_t gr = row0 + t * 128u + w8 * 16u + rg * 8u + (lane & 7u);
          const bool in = gr < rows_total;
          const uint32_t qt = in ? row_token(gr, a.inv_g) : 0u;
          const float *qp = reinterpret_cast<const float *>(reinterpret_cast<const char *>(a.q) + a.q_stride * qt) + (size_t)(g * a.G + (in ? gr - qt * a.G : 0u)) * HD +
                            8u * ((uint32_t)lane >> 3);
#pragma unroll
          for (uint32_t i = 0; i < HD / 32; i++)
#pragma unroll
            for (int p = 0; p < 2; p++) {
              v[rg][i][p] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (in) {
                if (a.wide & 2u) {
                  v[rg][i][p] = *reinterpret_cast<const float4 *>(qp + 32u * i + 4 * p);
                } else {
                  const float2 x = *reinterpret_cast<const float2 *>(qp + 32u * i + 4 * p), y = *reinterpret_cast<const float2 *>(qp + 32u * i + 4 * p + 2);
                  v[rg][i][p] = make_float4(x.x, x.y, y.x, y.y);
                }
              }
            }
        }
#pragma unroll
        for (uint32_t rg = 0; rg < 2; rg++) {
          const uint32_t qr = w8 * 16u + rg * 8u + (lane & 7u);
#pragma unroll
          for (uint32_t i = 0; i < HD / 32; i++) {
            uint32_t h[4], l[4];
#pragma unroll
            for (int p = 0; p < 2; p++)
              tc_split2(v[rg][i][p].x, v[rg][i][p].y, h[2 * p], l[2 * p]), tc_split2(v[rg][i][p].z, v[rg][i][p].w, h[2 * p + 1], l[2 * p + 1]);
            uint8_t *at = dst + (4u * i + ((uint32_t)lane >> 3)) * 2048u + qr * 16u;
            *reinterpret_cast<uint4 *>(at) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4 *>(at + L::QTERM) = make_uint4(l[0], l[1], l[2], l[3]);
          }
        }
        fence_async_shared();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_full);
      }
      positions();
      const uint32_t lim = real ? pos0 + tok + 1u : 0xFFFFFFFFu;  // positions this row sees (rows past the last are never stored)
      float m = -INFINITY, l = 0.0f;  // maximum the row's terms are taken against (log2 units), sum of this thread's terms
      float m_sum = -INFINITY;        // the maximum that the sums of the segments before are taken against
      // Those sums, of this thread's half of the row: in shared memory, columns apart by 128 rows, or (two tiles of heads of 128: no
      // room) where the row itself goes.
      float *sum_s = reinterpret_cast<float *>(smem_pt + L::SUM_OFF) + (HD == 64 ? t * HD * 128u : 0u) + half * (HD / 2u) * 128u + rl;
      auto sum_g = [&] {
        return (a.part ? a.part + (split * (size_t)a.T * a.n_head + (size_t)tok * a.n_head + head) * HD
                       : reinterpret_cast<float *>(reinterpret_cast<char *>(a.out) + a.out_stride * tok) + (size_t)head * HD) + half * (HD / 2u);
      };
      auto add_sums = [&](uint32_t (&v)[32], int c) {  // to columns 32 c .. of the running segment
        const float f = m_sum == -INFINITY ? 0.0f : ex2(m_sum - m);
        if (SUM_SMEM) {
#pragma unroll
          for (int i = 0; i < 32; i++) v[i] = __float_as_uint(fmaf(sum_s[(32 * c + i) * 128], f, __uint_as_float(v[i])));
        } else if (real) {
          const float *row = sum_g() + 32 * c;
#pragma unroll
          for (int u = 0; u < 4; u++) {
            float x[8];
            ld8(row + 8 * u, x, a.wide & 4u);
#pragma unroll
            for (int e = 0; e < 8; e++) v[8 * u + e] = __float_as_uint(fmaf(x[e], f, __uint_as_float(v[8 * u + e])));
          }
        }
      };
      bool ok = true;
      uint32_t at = 0;  // blocks of the running segment
      for (uint32_t j = 0; j < n; j++, at++) {
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(&s_full[t], j & 1u, &s_abort));  // the warp goes on or gives up as one
        if (!ok) break;
        tc_fence_after();
        const uint32_t k0 = (b0 + j) * PT_KEYS;
        const bool masked = __any_sync(0xFFFFFFFFu, k0 + PT_KEYS > lim);  // a block on the diagonal: positions that the row does not see
        auto scores = [&](uint32_t (&v)[32], uint32_t c) {  // 32 scores of the row from column 32 c (twice from tensor memory: they do not stay in 96 registers)
          tc_ld32(s_row + 32u * c, v);
          tc_wait_ld();
          if (masked) {
#pragma unroll
            for (int i = 0; i < 32; i++)
              if (k0 + 32u * c + i >= lim) v[i] = __float_as_uint(-INFINITY);
          }
        };
        // The maximum over all 128 columns, in both threads of the row: the second half costs less than an exchange would
        float mx = -INFINITY;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          uint32_t v[32];
          scores(v, c);
          float m4[4];
#pragma unroll
          for (int e = 0; e < 4; e++) m4[e] = fmaxf(__uint_as_float(v[e]), __uint_as_float(v[28 + e]));
#pragma unroll
          for (int i = 4; i < 28; i += 8)
#pragma unroll
            for (int e = 0; e < 4; e++) m4[e] = fmaxf(m4[e], fmaxf(__uint_as_float(v[i + e]), __uint_as_float(v[i + 4 + e])));
          mx = fmaxf(fmaxf(mx, fmaxf(m4[0], m4[1])), fmaxf(m4[2], m4[3]));
        }
        mx *= a.scale_log2;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pair);  // this warp has read all of S: the other may put P into it (waited for below, under the exponentials)
        if (j == 0) {
          m = mx;
        } else if (at == seg) {  // the segment's O (complete: s_full says so) joins the sums, and O starts anew
#pragma unroll 1
          for (int c = 0; c < HD / 64; c++) {
            uint32_t v[32];
            tc_ld32(o_col + 32u * c, v);
            tc_wait_ld();
            if (j != seg) add_sums(v, c);
            if (SUM_SMEM) {
#pragma unroll
              for (int i = 0; i < 32; i++) sum_s[(32 * c + i) * 128] = __uint_as_float(v[i]);
            } else if (real) {
              float *row = sum_g() + 32 * c;
#pragma unroll
              for (int u = 0; u < 4; u++) st8(row + 8 * u, v + 8 * u, a.wide & 4u);
            }
          }
          m_sum = m, at = 0;
          if (mx > m) l = m == -INFINITY ? l : l * ex2(m - mx), m = mx;
        } else {
          const bool grow = mx > m + 8.0f || (m == -INFINITY && mx > m);
          if (__any_sync(0xFFFFFFFFu, grow)) {  // rescale what the row has (PV of the block before has completed: s_full says so)
            const float f = grow ? (m == -INFINITY ? 0.0f : ex2(m - mx)) : 1.0f;
            if (grow) m = mx;
            l *= f;
#pragma unroll 1
            for (int c = 0; c < HD / 16; c++) {
              uint32_t o[8];
              tc_ld8(o_col + 8u * c, o);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
              tc_st8(o_col + 8u * c, o);
            }
          }
        }
        const float nm = m == -INFINITY ? 0.0f : -m;
        const f32x2 sc2 = pk2(a.scale_log2, a.scale_log2), nm2 = pk2(nm, nm);
        f32x2 sum2 = pk2(0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < 2; c++) {
          uint32_t v[32], p[32];
          scores(v, 2u * half + c);
#pragma unroll
          for (int i = 0; i < 16; i++) {
            float x, y;
            unpk2(fma2(pk2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sc2, nm2), x, y);
            x = ex2(x), y = ex2(y);
            const f32x2 xy = pk2(x, y);
            sum2 = add2(sum2, xy);
            const __half2 h = __floats2half2_rn(x, y);
            const float2 hf = __half22float2(h);
            unpk2(add2(xy, pk2(-hf.x, -hf.y)), x, y);
            const __half2 lo = __floats2half2_rn(x, y);
            p[i] = *reinterpret_cast<const uint32_t *>(&h), p[16 + i] = *reinterpret_cast<const uint32_t *>(&lo);
          }
          if (c == 0) {
            ok = __all_sync(0xFFFFFFFFu, mbar_wait(pair, j & 1u, &s_abort));
            tc_fence_after();  // (the other warp's loads of S come before these stores, in tensor memory's order too)
          }
          tc_st32(s_row + 32u * (2u * half + c), p);
        }
        {
          float x, y;
          unpk2(sum2, x, y);
          l += x + y;
        }
        if (t == 0u && k0 + PT_KEYS > first_lim) {  // the first tile's warps, ahead of every product with this block of V
          const uint32_t u = 2u * j + 1u;
          ok = ok && __all_sync(0xFFFFFFFFu, mbar_wait(&kv_full[u % PT_RING], (u / PT_RING) & 1u, &s_abort));
          if (ok) {
            uint4 *vb = reinterpret_cast<uint4 *>(smem_pt + L::KV_OFF + (u % PT_RING) * L::BLOCK) + threadIdx.x;
            __half2 top = __float2half2_rn(0.0f);
#pragma unroll
            for (int i = 0; i < (int)(L::BLOCK / 4096u); i++) {
              const uint4 x = vb[i * 256];
              top = __hmax2_nan(__hmax2_nan(top, __habs2(as_half2(x.x))), __habs2(as_half2(x.y)));
              top = __hmax2_nan(__hmax2_nan(top, __habs2(as_half2(x.z))), __habs2(as_half2(x.w)));
            }
            if (half_bad(*reinterpret_cast<const uint32_t *>(&top))) {
#pragma unroll 1
              for (int i = 0; i < (int)(L::BLOCK / 4096u); i++) {
                uint4 x = vb[i * 256];
                x.x &= ~half_bad(x.x), x.y &= ~half_bad(x.y), x.z &= ~half_bad(x.z), x.w &= ~half_bad(x.w);
                vb[i * 256] = x;
              }
              s_bad = 1u;
              fence_async_shared();
            }
          }
        }
        if (!ok) break;
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[t]);
      }
      // ---------------- the rows' outputs: through shared memory (the tile's Q is no longer needed) to whole row pieces ----------------
      if (ok && n > 0u) ok = __all_sync(0xFFFFFFFFu, mbar_wait(&s_full[t], n & 1u, &s_abort));
      if (ok && n > 0u) {  // the sum of the row's other half of the columns
        float *x = s_pair + t * 256u;
        x[half * 128u + rl] = l;
        __syncwarp();
        if (lane == 0) mbar_arrive(pair);
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(pair, n & 1u, &s_abort));
        l += x[(half ^ 1u) * 128u + rl];
      }
      if (ok && n == 0u) {
        // A split without blocks for this tile (the splits are dealt for the whole chunk's positions): an empty record, whose row the
        // merge does not read. Nothing is staged: no wait of this path says that the other warps have stored their part of Q.
        if (real && half == 0u)
          *reinterpret_cast<float2 *>(a.ml + (split * (size_t)a.T * a.n_head + (size_t)tok * a.n_head + head) * 2u) = make_float2(-INFINITY, 0.0f);
      } else if (ok) {
        tc_fence_after();
        constexpr uint32_t UN = HD / 8;  // 16-byte units of the half row that a warp writes
        const uint32_t nbq = a.n_head * HD / 32u;
        const size_t all = (size_t)a.T * a.n_head;
        const float inv = a.part ? 1.0f : (l > 0.0f ? 1.0f / l : 0.0f);
        uint8_t *stage = smem_pt + L::Q_OFF + t * 2u * L::QTERM + ((uint32_t)warp & 7u) * (32u * UN * 16u);
#pragma unroll 1
        for (int c = 0; c < HD / 64; c++) {
          uint32_t v[32];
          tc_ld32(o_col + 32u * c, v);
          tc_wait_ld();
          if (n > seg) add_sums(v, c);
          if (s_bad && real) {  // what the zeros in V stand for, for the positions that this row sees (every such p is positive)
            const uint32_t k1 = min(lim, (b0 + n) * PT_KEYS);
#pragma unroll 1
            for (uint32_t k = max(b0 * PT_KEYS, first_lim / PT_KEYS * PT_KEYS); k < k1; k++) {
              const uint32_t *vr = reinterpret_cast<const uint32_t *>(a.vc + ((size_t)g * a.kv_len + k) * HD + half * (HD / 2u) + 32u * c);
#pragma unroll
              for (int i = 0; i < 16; i++) {
                const uint32_t w = vr[i], bad = half_bad(w);
                if (bad) {
                  const float2 f = __half22float2(as_half2(w & bad));  // (0 where the half is finite)
                  v[2 * i] = __float_as_uint(__uint_as_float(v[2 * i]) + f.x), v[2 * i + 1] = __float_as_uint(__uint_as_float(v[2 * i + 1]) + f.y);
                }
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * inv);
#pragma unroll
          for (uint32_t u = 0; u < 8; u++)
            *reinterpret_cast<uint4 *>(stage + lane * UN * 16u + (((8u * c + u) ^ ((uint32_t)lane & (UN - 1u))) * 16u)) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
          if (!a.part && a.oq && real) {  // these 32 columns are one Q8 block, all of it in this thread
            float amax = 0.0f;
#pragma unroll
            for (int i = 0; i < 32; i++) amax = fmaxf(amax, fabsf(__uint_as_float(v[i])));
            const float d = __fdiv_rn(amax, 127.0f);
            const Q8Div qd = q8_div(d);
            uint8_t *qrow = a.oq + a.oq_stride * tok;
            const uint32_t b = (head * HD + half * (HD / 2u)) / 32u + c;
            int sum = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) {
              uint32_t w = 0u;
#pragma unroll
              for (int e = 0; e < 4; e++) {
                const int q = q8_round(__uint_as_float(v[4 * i + e]), qd);
                sum += q, w |= (uint32_t)(q & 255) << (8 * e);
              }
              reinterpret_cast<uint32_t *>(qrow + 32u * (size_t)b)[i] = w;
            }
            reinterpret_cast<float *>(qrow + 32u * (size_t)nbq)[b] = d;
            reinterpret_cast<int *>(qrow + 36u * (size_t)nbq)[b] = sum;
          }
        }
        if (a.part && real && half == 0u) {
          float *ml = a.ml + (split * all + (size_t)tok * a.n_head + head) * 2u;
          ml[0] = m, ml[1] = l;
        }
        __syncwarp();
        const uint32_t u = (uint32_t)lane % UN;
#pragma unroll 4
        for (uint32_t i = 0; i < 32u; i += 32u / UN) {
          const uint32_t sr = i + (uint32_t)lane / UN, gr = row0 + t * 128u + wq * 32u + sr;
          const float4 o = *reinterpret_cast<const float4 *>(stage + sr * UN * 16u + ((u ^ (sr & (UN - 1u))) * 16u));
          const bool in = gr < rows_total;
          const uint32_t otok = in ? row_token(gr, a.inv_g) : 0u, ohead = g * a.G + (in ? gr - otok * a.G : 0u), col = half * (HD / 2u) + 4u * u;
          float *to = a.part ? a.part + (split * all + (size_t)otok * a.n_head + ohead) * HD + col
                             : reinterpret_cast<float *>(reinterpret_cast<char *>(a.out) + a.out_stride * otok) + (size_t)ohead * HD + col;
          if (in) {
            if (a.part || (a.wide & 1u)) *reinterpret_cast<float4 *>(to) = o;
            else to[0] = o.x, to[1] = o.y, to[2] = o.z, to[3] = o.w;
          }
        }
      }
    }
  } else if (warp == SOFT_WARPS) {
    // ---------------- MMA issue: one thread ----------------
    positions();
    if (lane == 0 && n > 0u) {
      const uint32_t id_qk = (1u << 4) | ((PT_KEYS >> 3) << 17) | ((128u >> 4) << 24);                // S: K rows are K-major
      const uint32_t id_pv = (1u << 4) | (1u << 16) | (((uint32_t)HD >> 3) << 17) | ((128u >> 4) << 24);  // O: V is N-major (transposed B)
      const uint32_t q_base = smem_u32(smem_pt + L::Q_OFF), kv_base = smem_u32(smem_pt + L::KV_OFF);
      auto qk = [&](uint32_t t, uint32_t buf) {
        const uint32_t qa = q_base + t * 2u * L::QTERM, kb = kv_base + buf * L::BLOCK;
#pragma unroll
        for (uint32_t i = 0; i < HD / 8; i++) {  // the low terms first: see above
          const uint32_t s = i % (HD / 16), lo = i < HD / 16 ? L::QTERM : 0u;
          const uint64_t b = tc_desc128(kb + (s >> 2) * 16384u + (s & 3u) * 32u, 16u, 1024u);  // 64-column boxes; 8-row groups 1024 bytes apart
          tc_mma(tmem + t * 128u, tc_desc(qa + lo + s * 4096u, 2048u, 128u), b, id_qk, i ? 1u : 0u);
        }
        tc_commit(&s_full[t]);
      };
      auto pv = [&](uint32_t t, uint32_t buf, uint32_t acc) {
        const uint32_t vb = kv_base + buf * L::BLOCK;
#pragma unroll
        for (uint32_t i = 0; i < PT_KEYS / 8; i++) {  // 16 keys: two groups of 8 rows (1024 bytes apart); 64-column boxes 16 KB apart
          const uint32_t s = i % (PT_KEYS / 16), lo = i < PT_KEYS / 16 ? 16u : 0u;
          const uint64_t b = tc_desc128(vb + s * 2048u, 16384u, 1024u);
          tc_mma_ta(tmem + 256u + t * HD, tmem + t * 128u + (s >> 1) * 32u + (s & 1u) * 8u + lo, b, id_pv, (acc | i) ? 1u : 0u);
        }
      };
      // Blocks in ring order K0 V0 K1 V1 ...: number u sits in buffer u % 3. Issue order QK0 QK1 | PV0 QK0' PV1 QK1' | ...:
      // between a tile's QK and its PV lie the other tile's two products, under which its softmax runs. A tile's next QK
      // overwrites the P its PV reads: MMAs of one thread execute in issue order. (Two issuing threads, one per tile, fall
      // into step on the shared K blocks: both softmaxes at once, then both tiles' products; 4.5 us a block instead of 3.5.)
      auto full = [&](uint32_t u) { return mbar_wait(&kv_full[u % PT_RING], (u / PT_RING) & 1u, &s_abort); };
      bool ok = mbar_wait(q_full, 0u, &s_abort) && full(0u);
      if (ok) {
        tc_fence_after();
        for (uint32_t t = 0; t < n_tiles; t++) qk(t, 0u);
        tc_commit(&kv_empty[0]);
      }
      uint32_t at = 0;  // blocks of the running segment
      for (uint32_t j = 0; j < n && ok; j++, at++) {
        if (at == seg) at = 0;
        const uint32_t uv = 2u * j + 1u, uk = 2u * j + 2u;
        ok = full(uv) && (j + 1u == n || full(uk));
        for (uint32_t t = 0; t < n_tiles && ok; t++) {
          ok = mbar_wait(&p_full[t], j & 1u, &s_abort);
          if (!ok) break;
          tc_fence_after();
          pv(t, uv % PT_RING, at);
          if (t + 1u == n_tiles) tc_commit(&kv_empty[uv % PT_RING]);
          if (j + 1u < n) {
            qk(t, uk % PT_RING);
            if (t + 1u == n_tiles) tc_commit(&kv_empty[uk % PT_RING]);
          } else {
            tc_commit(&s_full[t]);
          }
        }
      }
    }
  } else {
    // ---------------- loader: K and V blocks into the ring ----------------
    positions();
    const uint32_t total = 2u * n, head_row = g * a.kv_len;
    for (uint32_t u = 0; u < total; u++) {
      const uint32_t round = u / PT_RING, buf = u % PT_RING, k0 = (b0 + (u >> 1)) * PT_KEYS, rows = min((uint32_t)PT_KEYS, p_hi - k0);
      if (!__all_sync(0xFFFFFFFFu, round == 0u || mbar_wait(&kv_empty[buf], (round - 1u) & 1u, &s_abort))) break;
      const bool ragged = (u & 1u) && rows < PT_KEYS;  // only the very last block
      uint8_t *dst = smem_pt + L::KV_OFF + buf * L::BLOCK;
      if (lane == 0) {
        uint64_t *bar = ragged ? tail : &kv_full[buf];
        mbar_expect_tx(bar, L::BLOCK);
#pragma unroll
        for (uint32_t x = 0; x < (uint32_t)HD; x += 64u) {
          if (u & 1u) tma_2d(dst + (x >> 6) * 16384u, &v_map, x, head_row + k0, bar);
          else tma_2d(dst + (x >> 6) * 16384u, &k_map, x, head_row + k0, bar);
        }
      }
      issued = u + 1u;
      if (ragged) {
        if (!__all_sync(0xFFFFFFFFu, mbar_wait(tail, 0u, &s_abort))) break;
        for (uint32_t i = lane; i < (PT_KEYS - rows) * (HD / 8u); i += 32u) {
          const uint32_t r = rows + i / (HD / 8u), c = i % (HD / 8u);
          *reinterpret_cast<uint4 *>(dst + (c >> 3) * 16384u + r * 128u + (c & 7u) * 16u) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_async_shared();
        __syncwarp();
        if (lane == 0) mbar_arrive(&kv_full[buf]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (s_abort) {  // (nobody sets it any more) do not leave while MMAs or copies still use this CTA's memory
    if (warp == SOFT_WARPS && lane == 0) tc_commit(drained), mbar_drain(drained, 0u);
    if (warp == SOFT_WARPS + 1 && lane == 0) {
      for (uint32_t u = issued > PT_RING ? issued - PT_RING : 0u; u < issued; u++) {
        const bool ragged = (u & 1u) && p_hi - (b0 + (u >> 1)) * PT_KEYS < PT_KEYS;
        mbar_drain(ragged ? tail : &kv_full[u % PT_RING], ragged ? 0u : (u / PT_RING) & 1u);
      }
    }
    // The rows say so too (a caller may have given no error word): NaN, in the outputs or in the records that the merge reads.
    const float nan = __int_as_float(0x7FFFFFFF);
    const uint32_t n_rows = min(rows_total - row0, 128u * TILES), nbq = a.n_head * HD / 32u;
    for (uint32_t i = threadIdx.x; i < n_rows * (HD / 32u); i += THREADS) {
      const uint32_t r = row0 + i / (HD / 32u), tok = row_token(r, a.inv_g), head = g * a.G + (r - tok * a.G), b = i % (HD / 32u);
      if (a.part) {
        if (b < 2u) a.ml[(split * (size_t)a.T * a.n_head + (size_t)tok * a.n_head + head) * 2u + b] = nan;
      } else {
        float *row = reinterpret_cast<float *>(reinterpret_cast<char *>(a.out) + a.out_stride * tok) + (size_t)head * HD + 32u * b;
        for (int e = 0; e < 32; e++) row[e] = nan;
        if (a.oq) reinterpret_cast<float *>(a.oq + a.oq_stride * tok + 32u * (size_t)nbq)[head * (HD / 32u) + b] = nan;
      }
    }
    if (threadIdx.x == 0 && a.err) atomicExch(a.err, 5u);
    __syncthreads();
  }
  __syncwarp();
  if (warp == SOFT_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// The splits' records of a (token, head) row -> its output and Q8 copy: hd / 4 lanes per row, four floats each. A record (-inf, 0)
// is of a split that holds nothing the row sees: its row is not read (it may never have been written).
template <int HD>
__global__ void __launch_bounds__(256) attn_prefill_merge_kernel(const float *part, const float *ml, uint32_t splits, uint32_t T, uint32_t n_head, float *out,
                                                                 uint8_t *oq, size_t out_stride, size_t oq_stride, uint32_t wide) {
  pdl_prologue();
  constexpr uint32_t LPR = HD / 4;
  const uint32_t all = T * n_head, at = blockIdx.x * (256u / LPR) + threadIdx.x / LPR, col = (threadIdx.x % LPR) * 4u;
  const bool in = at < all;
  const uint32_t row = in ? at : 0u;
  float M = -INFINITY, L = 0.0f;
  for (uint32_t s = 0; s < splits; s++) M = fmaxf(M, ml[2u * ((size_t)s * all + row)]);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (uint32_t s = 0; s < splits; s++) {
    const float2 e = *reinterpret_cast<const float2 *>(ml + 2u * ((size_t)s * all + row));
    if (e.x == -INFINITY && e.y == 0.0f) continue;
    const float4 v = *reinterpret_cast<const float4 *>(part + ((size_t)s * all + row) * HD + col);
    const float w = ex2(e.x - M);
    L = fmaf(w, e.y, L);
    acc.x = fmaf(w, v.x, acc.x), acc.y = fmaf(w, v.y, acc.y), acc.z = fmaf(w, v.z, acc.z), acc.w = fmaf(w, v.w, acc.w);
  }
  const float inv = L > 0.0f ? 1.0f / L : 0.0f;
  acc.x *= inv, acc.y *= inv, acc.z *= inv, acc.w *= inv;
  store_row4<HD>(out, out_stride, oq, oq_stride, wide, n_head * HD / 32u, row / n_head, row % n_head, col, acc, in);
}

// A row-major f16 matrix [rows][cols] as a tensor map of box_rows x box_cols boxes in the 128-byte swizzle (box_cols = 64).
static int tc_map_2d_f16(CUtensorMap *map, const void *base, uint64_t cols, uint64_t rows, uint32_t box_cols, uint32_t box_rows) {
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }();
  if (!encode) return fail(IE_B200_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t dims[2] = {cols, rows}, strides[1] = {cols * 2u};
  const cuuint32_t box[2] = {box_cols, box_rows}, step[2] = {1u, 1u};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? IE_B200_OK : fail(IE_B200_E_CUDA, "cuTensorMapEncodeTiled: error %d", (int)r);
}

// Tiles per CTA and splits of the positions. A CTA occupies an SM, so the CTAs run in whole waves of the SM count; the time of
// a choice in microseconds: waves x (blocks per split x what a block takes + start and end of a CTA + accumulations that join the
// rows' sums), plus, with splits, the merge launch and the partial rows' way through memory. Two tiles hide each other's softmax,
// one tile spreads a short chunk over more SMs and has half the rows to load and store. The figures are fitted to 2 .. 256
// tokens, 2 .. 8 KV heads of 2 .. 7 query heads at 0 .. 16000 positions with one to sixteen splits (900 timings, 6 % off on
// average; the choice made by them 1 % behind the best one): us per block, per CTA, less per CTA of few rows, per accumulation.
struct PtTime {
  float block, cta, few_rows, sum;
};
static float pick_shape(uint32_t rows, uint32_t n_kv, uint32_t blocks, uint32_t all_rows, uint32_t hd, bool may_split, uint32_t *tiles, uint32_t *splits) {
  static const PtTime time[2][2] = {{{2.12f, 5.4f, 1.24f, 0.56f}, {2.4f, 8.7f, 0.0f, 1.1f}}, {{2.52f, 7.8f, 2.5f, 0.75f}, {2.95f, 13.0f, 0.0f, 6.5f}}};  // [head size][tiles]
  const uint32_t sms = (uint32_t)sm_count(), seg = hd == 64 ? pt_segment<64>(blocks, 0u) : pt_segment<128>(blocks, 0u);
  float best = 1e30f;
  for (uint32_t t = 1; t <= 2u; t++) {
    const PtTime &c = time[hd == 64 ? 0 : 1][t - 1u];
    const uint32_t ctas = (rows + 128u * t - 1u) / (128u * t) * n_kv;
    const float cta = c.cta - c.few_rows * (rows < 128u ? 1.0f - (float)rows / 128.0f : 0.0f);
    for (uint32_t s = 1; s <= (may_split ? PT_MAX_SPLITS : 1u) && s <= blocks && (s == 1u || s * all_rows <= PT_MAX_RECORDS); s++) {
      const uint32_t per = (blocks + s - 1u) / s, waves = (ctas * s + sms - 1u) / sms, joins = (per + seg - 1u) / seg - 1u;
      float cost = (float)waves * ((float)per * c.block + cta + (float)joins * c.sum);
      if (s > 1u) cost += 2.3f + (float)s * (float)all_rows * (float)hd * 8.0f / 8.5e6f;
      if (cost < best) best = cost, *tiles = t, *splits = s;
    }
  }
  return best;
}

// Microseconds of the mma.sync form, fitted the same way (1100 timings at up to 16000 positions, 5 % off on average): its CTAs are
// up to 16 rows each, so there are many; a walk in tiles of 64 positions slows down with the CTAs that read the cache at once, and
// above what the SMs hold together comes in waves (heads of 128) or shares the SMs further (heads of 64).
static float mma_time(uint32_t ctas, uint32_t positions, uint32_t hd) {
  const float sms = (float)sm_count(), n = (float)ctas, busy = std::min(n, sms);
  const float tile = (hd == 64 ? 0.57f : 0.94f) + 0.0036f * std::max(0.0f, busy - 32.0f);
  const float waves = hd == 64 ? std::max(1.0f, n / 300.0f) : ceilf(n / (2.0f * sms));
  return (hd == 64 ? 3.0f : 5.0f) + 2.0f * busy / sms + (float)((positions + 63u) / 64u) * tile * waves;
}

size_t attn_prefill_scratch_bytes(uint32_t n_head, uint32_t hd, uint32_t T) {
  return std::min((size_t)PT_MAX_SPLITS * T * n_head, (size_t)PT_MAX_RECORDS) * (hd + 2u) * sizeof(float) + 256u;
}

template <int HD, int TILES>
static int launch_pt(const PtArgs &a, const void *kc, const void *vc, uint32_t splits, cudaStream_t st) {
  CUtensorMap km, vm;
  if (int r = tc_map_2d_f16(&km, kc, HD, (uint64_t)a.n_kv * a.kv_len, 64u, PT_KEYS)) return r;
  if (int r = tc_map_2d_f16(&vm, vc, HD, (uint64_t)a.n_kv * a.kv_len, 64u, PT_KEYS)) return r;
  auto k = attn_prefill_tc_kernel<HD, TILES>;
  if (int r = ensure_dynamic_smem(reinterpret_cast<const void *>(k), PtSmem<HD>::TOTAL)) return r;
  IEB_LAUNCH_PDL("attn_prefill_tc_kernel", k, dim3((a.T * a.G + 128u * TILES - 1u) / (128u * TILES), a.n_kv, splits), dim3((8 * TILES + 2) * 32), PtSmem<HD>::TOTAL,
                 st, a, km, vm);
  if (splits > 1u)
    IEB_LAUNCH_PDL("attn_prefill_merge_kernel", attn_prefill_merge_kernel<HD>, dim3((a.T * a.n_head + 1024u / HD - 1u) / (1024u / HD)), dim3(256), 0, st,
                   static_cast<const float *>(a.part), static_cast<const float *>(a.ml), splits, a.T, a.n_head, a.out, a.oq, a.out_stride, a.oq_stride, a.wide & 1u);
  return IE_B200_OK;
}

int attn_prefill_tc(const float *d_q, const void *d_kc, const void *d_vc, float *d_out, void *d_oq, const uint32_t *d_pos, uint32_t n_head, uint32_t n_kv,
                    uint32_t hd, uint32_t kv_len, uint32_t T, size_t q_stride, size_t out_stride, size_t oq_stride, uint32_t positions, float *d_scratch,
                    uint32_t *d_err, cudaStream_t st) {
  if (!d_q || !d_kc || !d_vc || !d_out || !d_pos) return fail(IE_B200_E_ARG, "ie_b200_attn_prefill: NULL pointer");
  if (n_kv == 0 || n_head % n_kv) return fail(IE_B200_E_SIZE, "ie_b200_attn_prefill: %u heads over %u KV heads", n_head, n_kv);
  if (hd != 64 && hd != 128) return fail(IE_B200_E_SIZE, "ie_b200_attn_prefill: head dim %u (64, 128; half-precision cache)", hd);
  if (!aligned16(d_kc) || !aligned16(d_vc) || ((uintptr_t)d_q & 7u) || (q_stride & 7u) || (d_scratch && !aligned16(d_scratch)))
    return fail(IE_B200_E_ARG, "ie_b200_attn_prefill: alignment");
  if (T == 0) return IE_B200_OK;
  if (n_head / n_kv > 8u) return fail(IE_B200_E_SIZE, "ie_b200_attn_prefill: %u query heads per KV head unsupported (1 .. 8)", n_head / n_kv);
  PtArgs a = {};
  a.q = d_q, a.out = d_out, a.oq = static_cast<uint8_t *>(d_oq), a.pos = d_pos;
  a.n_head = n_head, a.n_kv = n_kv, a.kv_len = kv_len, a.T = T, a.G = n_head / n_kv;
  a.q_stride = q_stride, a.out_stride = out_stride, a.oq_stride = oq_stride;
  a.scale_log2 = 1.44269504088896340736f / sqrtf((float)hd);
  a.err = d_err;
  a.vc = static_cast<const __half *>(d_vc);
  uint32_t splits = 1u, tiles = 1u;
  a.wide = ((((uintptr_t)d_out | out_stride) & 15u) == 0u ? 1u : 0u) | ((((uintptr_t)d_q | q_stride) & 15u) == 0u ? 2u : 0u);
  a.inv_g = 1.0f / (float)a.G;
  // Where the start and end of this kernel's CTAs, or one walk over many positions by few of them, take longer than the mma.sync form
  // does, that one runs (48 tokens of 28 x 4 heads of 128 at position 100: 9.5 against 13.5 us; 2 at 0: 5.8 / 7.8; 16 at 16000 without
  // scratch 240 / 310). A caller who has not said how many positions there are: while its CTAs fill one wave (two per SM), where the
  // cache may be long one per SM (77 tokens of 32 x 8 heads of 128, 160 CTAs: 9.6 / 10.5 us at 0, 51 / 50 at 2000, 347 / 313 at 16000).
  const uint32_t mma_ctas = (T + 16u / a.G - 1u) / (16u / a.G) * n_kv, sms = (uint32_t)sm_count();
  const float tc_time = pick_shape(T * a.G, n_kv, (std::max(positions, T) + PT_KEYS - 1u) / PT_KEYS, T * n_head, hd, d_scratch != nullptr, &tiles, &splits);
  if (positions ? mma_time(mma_ctas, positions, hd) <= tc_time : mma_ctas <= (kv_len <= 4096u ? 2u : 1u) * sms)
    return attn_prefill_mma(d_q, d_kc, d_vc, d_out, d_oq, d_pos, n_head, n_kv, hd, kv_len, T, q_stride, out_stride, oq_stride, st);
  if (splits > 1u) a.part = d_scratch, a.ml = d_scratch + (size_t)splits * T * n_head * hd;
  if (((uintptr_t)(a.part ? a.part : d_out) & 31u) == 0u && (a.part || (out_stride & 31u) == 0u)) a.wide |= 4u;
  if (hd == 64) return tiles == 1u ? launch_pt<64, 1>(a, d_kc, d_vc, splits, st) : launch_pt<64, 2>(a, d_kc, d_vc, splits, st);
  return tiles == 1u ? launch_pt<128, 1>(a, d_kc, d_vc, splits, st) : launch_pt<128, 2>(a, d_kc, d_vc, splits, st);
}

}  // namespace ieb

using namespace ieb;

extern "C" size_t ie_b200_attn_prefill_scratch_bytes(uint32_t n_head, uint32_t hd, uint32_t T) { return attn_prefill_scratch_bytes(n_head, hd, T); }

extern "C" int ie_b200_attn_prefill_split(const float *d_q, const void *d_kc, const void *d_vc, float *d_out, void *d_oq, const uint32_t *d_pos,
                                          uint32_t n_head, uint32_t n_kv, uint32_t hd, uint32_t kv_len, uint32_t T, size_t q_stride, size_t out_stride,
                                          size_t oq_stride, uint32_t positions, void *d_scratch, uint32_t *d_err, void *stream) {
  return attn_prefill_tc(d_q, d_kc, d_vc, d_out, d_oq, d_pos, n_head, n_kv, hd, kv_len, T, q_stride, out_stride, oq_stride, positions,
                         static_cast<float *>(d_scratch), d_err, static_cast<cudaStream_t>(stream));
}

extern "C" int ie_b200_attn_prefill(const float *d_q, const void *d_kc, const void *d_vc, float *d_out, void *d_oq, const uint32_t *d_pos,
                                    uint32_t n_head, uint32_t n_kv, uint32_t hd, uint32_t kv_len, uint32_t T, size_t q_stride, size_t out_stride,
                                    size_t oq_stride, void *stream) {
  return ie_b200_attn_prefill_split(d_q, d_kc, d_vc, d_out, d_oq, d_pos, n_head, n_kv, hd, kv_len, T, q_stride, out_stride, oq_stride, 0u, nullptr, nullptr,
                                    stream);
}
