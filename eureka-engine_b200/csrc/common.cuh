// common.cuh -- shared device helpers of the B200 speculative-decoding library.
//
// Weight formats are the reference's (host/llb_formats.h:4-15).  In device memory a quantised matrix is made of
// TILES of 16 rows x 256 columns (one super-block of 16 rows), [row tile][super-block], each tile contiguous, so that
// one bulk copy brings a warp's next piece of work.  Inside a tile a row's block stays together:
//   Q4_K  row r at 144 r, as stored: f16 d, f16 dmin, 12 B scales / mins, 128 B nibbles   (tools/qwen35_engine.c:258-272)
//   Q5_K  row r at 176 r, as stored: Q4_K plus 32 B of fifth bits before the nibbles       (tools/qwen35_engine.c:273-289)
//   Q6_K  row r at 208 r: ql 128 | qh 64 | scales 16; the sixteen f16 d follow at 3328 + 2 r (210 bytes a row, as stored)
//   Q8_0  row r at 272 r: 256 codes as q + 128 | 8 f16 scales                              (tools/q8_pack.py:7-10)
// Rows past the matrix (up to the next multiple of 16) and columns past it (Q8_0, up to the next multiple of 256) are zero
// weights.  F32 matrices are row-major.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define LLB_FM_F32 0
#define LLB_FM_Q8_0 1
#define LLB_FM_Q4_K 3
#define LLB_FM_Q6_K 4
#define LLB_FM_Q5_K 9

// bytes of one 16 x 256 tile, and of one row inside it
__host__ __device__ constexpr int tile_bytes(int fmt) {
  return fmt == LLB_FM_Q4_K ? 2304 : fmt == LLB_FM_Q5_K ? 2816 : fmt == LLB_FM_Q6_K ? 3360 : fmt == LLB_FM_Q8_0 ? 4352 : 0;
}
__host__ __device__ constexpr int tile_row(int fmt) {
  return fmt == LLB_FM_Q4_K ? 144 : fmt == LLB_FM_Q5_K ? 176 : fmt == LLB_FM_Q6_K ? 208 : 272;
}
// bytes of a matrix in the DEVICE layout (0: no such format)
__host__ __device__ inline size_t dev_bytes(int fmt, int rows, int cols) {
  if (fmt == LLB_FM_F32) return (size_t)rows * cols * 4;
  return (size_t)((rows + 15) >> 4) * ((cols + 255) >> 8) * tile_bytes(fmt);
}
// bytes of one row as stored in a pack (host/llb_formats.h:17)
__host__ __device__ inline size_t pack_row_bytes(int fmt, int cols) {
  switch (fmt) {
    case LLB_FM_F32: return (size_t)cols * 4;
    case LLB_FM_Q8_0: return (size_t)cols / 32 * 34;
    case LLB_FM_Q4_K: return (size_t)cols / 256 * 144;
    case LLB_FM_Q5_K: return (size_t)cols / 256 * 176;
    case LLB_FM_Q6_K: return (size_t)cols / 256 * 210;
  }
  return 0;
}

// ---- activation planes -------------------------------------------------------------------------
// A GEMM reads its T <= 16 activation rows as fp16 "planes": column t (< NH) holds hi = fp16(x),
// column NH + t holds lo = fp16((x - hi) * 2048), NH = NC / 2, so hi + lo/2048 carries about 22
// bits of x.  NC is 8 (T <= 4), 16 (T <= 8) or 32 (T <= 16).  With planes == 1 all NC columns are independent
// rows (bf16/fp16 inputs that need no second plane).
//   xh   [NC][K]    fp16, K-index permuted inside every aligned group of 8: stored order
//                   0 2 1 3 4 6 5 7, which is the order the tensor-core B fragments consume
//   xsf  [K/256][NC][16] fp16: the eight 32-column MEANS of a super-block as hi/lo pairs (hi = fp16(m),
//                   lo = fp16((m - hi) * 2048), like the planes), in the order the min-term MMA's B fragment
//                   reads them: for j = 0..3: hi(2j) hi(2j+1) lo(2j) lo(2j+1)
struct XPlanes {
  __half *xh;
  __half *xsf;
  int K;
  int NC;
};
__host__ __device__ inline size_t xp_bytes(int K, int NC) {
  return (size_t)NC * K * 2 + (size_t)(K / 256) * NC * 32;
}
__host__ __device__ inline XPlanes xp_carve(void *base, int K, int NC) {
  char *b = (char *)base;
  XPlanes xp;
  xp.xh = (__half *)b; b += (size_t)NC * K * 2;
  xp.xsf = (__half *)b;
  xp.K = K; xp.NC = NC;
  return xp;
}
#define XP_LO_SCALE 2048.0f
#define XP_LO_INV (1.0f / 2048.0f)

__host__ __device__ inline int xp_perm(int c) { return (c & ~7) | ((c & 4) | ((c & 1) << 1) | ((c & 2) >> 1)); }

// Four consecutive columns c .. c+3 (c a multiple of 4) of row t into the planes and the sub-block means; the eight lanes
// 8 j .. 8 j + 7 of a warp hold one aligned group of 32 columns.  `on` is false for a thread past the row's end (it still
// takes part in the shuffles).  Stored order inside the four: 0 2 1 3.  (Kept short: the kernels that end with it run for a
// microsecond or two, and instructions that the SM does not hold come from L2.)
__device__ __forceinline__ void xp_store4(const XPlanes &xp, int t, int planes, int c, const float (&v)[4], int lane, bool on) {
  const __half2 a = __floats2half2_rn(on ? v[0] : 0.0f, on ? v[2] : 0.0f), b = __floats2half2_rn(on ? v[1] : 0.0f, on ? v[3] : 0.0f);
  const float2 af = __half22float2(a), bf = __half22float2(b);
  float hs = ((af.x + bf.x) + af.y) + bf.y, ls = 0.0f;
  __half *x = xp.xh + (size_t)t * xp.K + c;
  if (on) *(uint2 *)x = make_uint2(*(const uint32_t *)&a, *(const uint32_t *)&b);
  if (planes == 2) {
    const __half2 e = __floats2half2_rn(on ? (v[0] - af.x) * XP_LO_SCALE : 0.0f, on ? (v[2] - af.y) * XP_LO_SCALE : 0.0f);
    const __half2 f = __floats2half2_rn(on ? (v[1] - bf.x) * XP_LO_SCALE : 0.0f, on ? (v[3] - bf.y) * XP_LO_SCALE : 0.0f);
    const float2 ef = __half22float2(e), ff = __half22float2(f);
    ls = ((ef.x + ff.x) + ef.y) + ff.y;
    if (on) *(uint2 *)(x + (size_t)(xp.NC >> 1) * xp.K) = make_uint2(*(const uint32_t *)&e, *(const uint32_t *)&f);
  }
#pragma unroll
  for (int m = 1; m < 8; m <<= 1) { hs += __shfl_xor_sync(0xffffffffu, hs, m); ls += __shfl_xor_sync(0xffffffffu, ls, m); }
  // lane 0 of the eight writes the hi plane's mean, lane 1 the lo plane's: each as an fp16 hi / rest pair
  if (on && (lane & 7) < planes) {
    const bool second = lane & 1;
    const int b32 = (c >> 5) & 7;
    const float m = (second ? ls : hs) * 0.03125f;
    const __half h1 = __float2half_rn(m);
    __half *p = xp.xsf + ((size_t)(c >> 8) * xp.NC + t + (second ? xp.NC >> 1 : 0)) * 16 + 4 * (b32 >> 1) + (b32 & 1);
    p[0] = h1; p[2] = __float2half_rn((m - __half2float(h1)) * XP_LO_SCALE);
  }
}

// ---- activations of a prompt chunk ----------------------------------------------------------------
#define PF_R 128              // most rows of a unit of a prompt chunk: the half of the dense GEMM's N = 256 that one CTA of a pair holds (pfmm.cuh)
#define PF_RMAX 256           // rows of a chunk, PF_RMAX / PF_R units
// Activations of a chunk for the dense GEMMs, "k-group major": one or two units of ru = 32, 64 or 128 rows (pf_unit_rows), each as two
// fp16 planes like the T-row planes: hi = fp16(x), lo = fp16((x - hi) * 2048), about 22 bits of x.  Element (row r, column k) of a
// unit sits at half index ((k >> 3) * ru + r) * 8 + xp_perm(k & 7) of its plane, the lo plane K * ru halves further on: eight
// consecutive columns of a row are one 16-byte core-matrix row in the order the unpacked codes have, the rows of a k-group are
// contiguous, and so is a plane's 64-column stage.  Behind the planes of a unit the means of every 32 columns, hi and then lo
// likewise: the eight of a super-block are a core-matrix row, stored twice (the two k-groups of a K = 16 step): [super-block][2][row][8].
__host__ __device__ inline int pf_unit_rows(int R) { return R > 64 ? 128 : R > 32 ? 64 : 32; }
__host__ __device__ inline size_t pf_sum_halves(int K, int ru) { return (size_t)K / 16 * ru; }               // of one plane's means
__host__ __device__ inline size_t pf_kg_halves(int K, int ru) { return (size_t)2 * K * ru + 2 * pf_sum_halves(K, ru); }
// Four consecutive columns k .. k+3 (k a multiple of 4) of row r into both planes, and the mean of the 32 that lanes 8 j .. 8 j + 7 of the warp hold
__device__ __forceinline__ void pf_kg_store4(__half *x, int K, int ru, int r, int k, float v0, float v1, float v2, float v3) {
  if (r >= ru) { x += pf_kg_halves(K, ru); r -= ru; }   // a second unit of a chunk follows the first
  const size_t i = ((size_t)(k >> 3) * ru + r) * 8 + (k & 4);
  const __half2 a = __floats2half2_rn(v0, v2), b = __floats2half2_rn(v1, v3);
  const float2 af = __half22float2(a), bf = __half22float2(b);
  const __half2 c = __floats2half2_rn((v0 - af.x) * XP_LO_SCALE, (v2 - af.y) * XP_LO_SCALE), d = __floats2half2_rn((v1 - bf.x) * XP_LO_SCALE, (v3 - bf.y) * XP_LO_SCALE);
  *(uint2 *)(x + i) = make_uint2(*(const uint32_t *)&a, *(const uint32_t *)&b);
  *(uint2 *)(x + (size_t)K * ru + i) = make_uint2(*(const uint32_t *)&c, *(const uint32_t *)&d);
  float m = ((v0 + v1) + v2) + v3;
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) m += __shfl_xor_sync(0xffffffffu, m, s);
  m *= 0.03125f;
  const int l = threadIdx.x & 7;
  if (l < 4) {   // (plane, k-group)
    const __half h = __float2half_rn(m);
    x[(size_t)2 * K * ru + (l >> 1) * pf_sum_halves(K, ru) + ((size_t)(k >> 8) * 2 + (l & 1)) * ru * 8 + r * 8 + ((k >> 5) & 7)] = l >> 1 ? __float2half_rn((m - __half2float(h)) * XP_LO_SCALE) : h;
  }
}
// ---- programmatic dependent launch --------------------------------------------------------------
// Every kernel of a pass is launched with the programmatic-serialization attribute: the next kernel's
// CTAs may become resident while this one still runs, do whatever does not depend on it (a GEMM
// prefetches its first weight chunks), and park in pdl_wait() until this grid has completed and its
// writes are visible.  Each kernel calls pdl_trigger() first and pdl_wait() before its first
// dependent read or any global write, so completion order stays the launch order.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---- small PTX wrappers ------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
// D += A(16x16, row) * B(16x8, col), fp16 inputs, fp32 accumulate
__device__ __forceinline__ void mma16816(float c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ldg128(const void *p) { return __ldg((const uint4 *)p); }
__device__ __forceinline__ uint2 ldg64(const void *p) { return __ldg((const uint2 *)p); }
__device__ __forceinline__ float2 ldg_f2(const void *p) { return __ldg((const float2 *)p); }

__device__ __forceinline__ float h2f_bits(uint32_t h16) { return __half2float(__ushort_as_half((unsigned short)h16)); }

// ---- per-format scalar dequantisers (bit-exact with tools/qwen35_engine.c:233-307) -------------
// Each returns weight (row, c) of a matrix in DEVICE layout.  __fmul_rn/__fsub_rn keep the
// reference's one-rounding-per-operation arithmetic (no FMA contraction).
__device__ __forceinline__ void q4k_scale_min(const uint8_t *s, int j, int &sc, int &mn) {
  if (j < 4) { sc = s[j] & 63; mn = s[j + 4] & 63; }
  else { sc = (s[j + 4] & 15) | ((s[j - 4] >> 6) << 4); mn = (s[j + 4] >> 4) | ((s[j] >> 6) << 4); }
}
__device__ __forceinline__ float deq_elem(int fmt, const uint8_t *W, int cols, int row, int c) {
  if (fmt == LLB_FM_F32) return ((const float *)W)[(size_t)row * cols + c];
  const int r = row & 15, i = c & 255;
  const uint8_t *tile = W + ((size_t)(row >> 4) * ((cols + 255) >> 8) + (c >> 8)) * tile_bytes(fmt), *blk = tile + r * tile_row(fmt);
  if (fmt == LLB_FM_Q8_0) {
    const uint8_t *s = blk + 256 + 2 * (i >> 5);
    float d = h2f_bits(s[0] | (s[1] << 8));
    return __fmul_rn((float)((int)blk[i] - 128), d);
  }
  if (fmt == LLB_FM_Q4_K || fmt == LLB_FM_Q5_K) {
    float d = h2f_bits(blk[0] | (blk[1] << 8)), dm = h2f_bits(blk[2] | (blk[3] << 8));
    int g = i >> 6, hi = (i >> 5) & 1, l = i & 31, sc, mn;
    q4k_scale_min(blk + 4, 2 * g + hi, sc, mn);
    const uint8_t *qs = blk + (fmt == LLB_FM_Q4_K ? 16 : 48);
    int q = hi ? (qs[32 * g + l] >> 4) : (qs[32 * g + l] & 15);
    if (fmt == LLB_FM_Q5_K) q += ((blk[16 + l] >> (2 * g + hi)) & 1) * 16;
    return __fsub_rn(__fmul_rn(__fmul_rn(d, (float)sc), (float)q), __fmul_rn(dm, (float)mn));
  }
  if (fmt == LLB_FM_Q6_K) {
    int hf = i >> 7, qd = (i >> 5) & 3, l = i & 31;
    uint8_t lq = blk[64 * hf + 32 * (qd & 1) + l];
    int nib = qd < 2 ? (lq & 15) : (lq >> 4);
    int code = (nib | (((blk[128 + 32 * hf + l] >> (2 * qd)) & 3) << 4)) - 32;
    float d = h2f_bits(tile[3328 + 2 * r] | (tile[3329 + 2 * r] << 8));
    float sc = (float)((const int8_t *)(blk + 192))[8 * hf + 2 * qd + (l >> 4)];
    return __fmul_rn(__fmul_rn(d, sc), (float)code);
  }
  return 0.0f;
}
