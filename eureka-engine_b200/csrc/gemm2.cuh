// gemm2.cuh -- the skinny GEMM: Y[t][r] = sum_c W[r][c] x[t][c], T <= 16 rows against Q4_K / Q5_K / Q6_K / Q8_0 weights.
// Integer codes go to the tensor cores as fp16 numbers (mma.m16n8k16, fp32 sums); scales never round a weight.
//
//  * a CTA owns ONE K-slice and stages that slice of the activation planes in shared memory once;
//  * a warp's piece of work is one tile of 16 rows x 256 columns (common.cuh), which one bulk copy brings into the warp's
//    private ring of two or three stages (an mbarrier a stage, no copy instructions in the other lanes).  Per-lane
//    16-byte copies took 30 of the loop's 397 instructions, most of them integer adds;
//  * Q4_K / Q5_K: a code in the low bits of an fp16 lane is the subnormal code * 2^-24, so two MMAs sum
//    code * x of a 32-column sub-block exactly; the six-bit scale multiplies that fp32 sum, d the super-block's;
//  * Q4_K, 16 rows (four n-tiles), large launches that the tcgen05 kernel (gemm3.cuh) cannot take or is kept from (a matrix of
//    one super-block's columns; LLB_GEMM3=0, llb_b200_use_tcgen05(0)): the scale is multiplied into the codes instead (FOLD), since sc * q <=
//    63 * 15 is an exact fp16 integer: one HMUL2 a fragment register, shared by the n-tiles, and the MMAs of a whole super-block
//    accumulate into one fragment.  Lane j of a row's four lanes then holds the k indices of column group j (64 columns, two
//    sub-blocks) and needs that group's scales only.  The chain of MMAs into one fragment is longer, so it takes enough
//    tiles an SM to hide it: gate|up of the 27B shape (43520 tiles) 62 us against 69, 12288 x 2048 (6144 tiles) 22.5
//    against 17.4; with one n-tile the HMUL2s (half rate) cost more than the scales save, 31 us against 26;
//  * the "min" term  dmin * sum_b m_b * sum(x in sub-block b)  is ONE extra MMA per tile: A = the eight mins as fp16 numbers
//    (m against the means' hi halves, m / 2048 against their lo halves), B = the sub-block activation means;
//  * Q6_K / Q8_0: a scale times a code does not fit fp16 exactly, so the scale multiplies the fp32 partial sum of its 16 or
//    32 columns; the code's offset is taken off in fp16 (0x6400 | c is 1024 + c; one HADD2, exact).
#pragma once
#include "gemm.cuh"
#include "tc5.cuh"

#define G2_SMEM_MAX 226304   // 227 KB less the 6 KB that a phase may use beside the ring and the activation slice
#define G2_MAXWARPS 16
#define G2_WAIT_LIMIT (1u << 19)   // tries of a bounded wait (up to 4 us each)
#define G2_DRAIN_LIMIT (1u << 13)
#define G2_BAR_BYTES 512     // one mbarrier per warp and stage (at most four)

// XPAD: padding of a plane column in shared memory (column stride = 64 mod 128 bytes for the 16-byte B reads of Q4_K / Q5_K /
// Q8_0, 32 mod 128 for the 8-byte ones of Q6_K), AUX: bytes per (super-block, column) of the sub-block means
// Ring depth: 104 to 161 KB an SM (44 KB in flight cover HBM's latency at full rate), 55 to 104 KB beside 32 plane columns,
// whose whole d = 2048 slice must fit.
// Super-blocks a copy brings.  A bulk copy costs about 85 cycles of the SM's copy engine on top of its bytes (copies alone, no
// arithmetic, gate|up of the 27B shape: 19.6 us at 2304 bytes, 11.8 us at 4608), so Q4_K takes two at a time.
// ring 1: a shorter ring for K-slices that do not fit beside the usual one (ring 0): matrices of more than GEMM_MAXSPLIT of the
// usual slices.
__host__ __device__ constexpr int g2_chunk(int fmt, int ring = 0) { return fmt == LLB_FM_Q4_K && !ring ? 2 : 1; }
__host__ __device__ constexpr int g2_stages(int fmt, int NC, int ring = 0) {
  if (ring == 2) return 2;
  if (ring) return fmt == LLB_FM_Q4_K ? 3 : NC >= 32 ? 1 : 2;
  return fmt == LLB_FM_Q4_K ? (NC >= 32 ? 1 : 2) : NC >= 32 || fmt == LLB_FM_Q8_0 ? 2 : 3;
}
// ring 2: Q4_K at 32 columns with the bytes of ring 0 as two stages of one super-block: a warp with few tiles then has the next one
// on its way while it multiplies (3072 x 8192 at sixteen rows 21.7 -> 20.3 us).  Large launches have other warps' copies for
// that and want the larger ones (FOLD).
__host__ __device__ constexpr int g2_small_ring(int fmt, int NC) { return fmt == LLB_FM_Q4_K && NC >= 32 ? 2 : 0; }
__host__ __device__ constexpr bool g2_has_short(int fmt, int NC) { return NC < 32 ? fmt == LLB_FM_Q4_K : fmt == LLB_FM_Q6_K; }
// Warps of a CTA: sixteen (128 registers a thread), fewer where the rings of sixteen would leave the activation slice less than
// the widths in use need: Q8_0's tiles are twice the size, and 32 plane columns take half of the memory.
__host__ __device__ constexpr int g2_warps(int fmt, int NC) {
  return fmt == LLB_FM_Q8_0 ? 12 : NC < 32 ? 16 : 12;
}
__host__ __device__ constexpr int g2_ring_bytes(int fmt, int NC, int ring = 0) { return g2_warps(fmt, NC) * g2_stages(fmt, NC, ring) * g2_chunk(fmt, ring) * tile_bytes(fmt); }
__host__ __device__ constexpr int g2_aux(int fmt) { return fmt == LLB_FM_Q4_K || fmt == LLB_FM_Q5_K ? 32 : 0; }
__host__ __device__ constexpr int g2_xpad(int fmt) { return fmt == LLB_FM_Q6_K ? 32 : 64; }
// bytes of shared memory of a launch whose K-slices have nsl super-blocks in `parts` parts, for NC activation columns
__host__ __device__ inline size_t g2_smem(int fmt, int nsl, int NC, int parts = 1, int ring = 0) {
  return (size_t)(parts > 1 ? g2_warps(fmt, NC) * (NC / 8) * 512 : 0) + G2_BAR_BYTES + NC * (nsl * 512 + g2_xpad(fmt)) + nsl * NC * g2_aux(fmt) + g2_ring_bytes(fmt, NC, ring);
}
inline int g2_max_slice_sb(int fmt, int NC, int ring = 0) {
  const int left = G2_SMEM_MAX - G2_BAR_BYTES - g2_ring_bytes(fmt, NC, ring) - NC * g2_xpad(fmt);
  return left / (NC * (512 + g2_aux(fmt)));
}
// the ring that a K-slice of nsl super-blocks is launched with, and the longest slice of either
inline int g2_ring_of(int fmt, int NC, int nsl) { return g2_has_short(fmt, NC) && nsl > g2_max_slice_sb(fmt, NC); }
inline int g2_longest_slice(int fmt, int NC) { return g2_max_slice_sb(fmt, NC, g2_has_short(fmt, NC)); }

// whether a launch of `work` 16 x 256 tiles has the scales folded into the codes: measured at 16 rows, the line lies between
// 10000 tiles (25.4 us folded, 21.2 not) and 12800 (29.8 folded, 31.2 not); Q5_K, whose codes take more to assemble, gains
// nothing at 12800 (30.9 against 30.5) and 3 % at 43520
__host__ __device__ constexpr bool g2_folds(int fmt, int NT) { return NT == 4 && fmt == LLB_FM_Q4_K; }
#define G2_FOLD_TILES 12000

// Where the 16-byte piece of columns c .. c+7 of a slice sits in a plane column (bytes).  Folded: lane j reads column group
// j, so the pieces of the four groups that are read together lie side by side; the others keep their order.
template <int FMT, bool FOLD> __device__ __forceinline__ int g2_xpos(int piece) {
  if constexpr (FOLD) return ((piece & ~31) | ((piece & 7) << 2) | ((piece >> 3) & 3)) * 16;
  else return piece * 16;
}

// D = A*B with a zero C operand
__device__ __forceinline__ void mma16816_z(float d[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ uint32_t g2_hmul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t g2_hadd2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ void mbar_expect(uint32_t bar_s, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_s), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst_s, const void *src, uint32_t bytes, uint32_t bar_s) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_s), "l"(src), "r"(bytes), "r"(bar_s)
               : "memory");
}

// Fragment row gid (and gid + 8) of a tile is tile row g2_row(gid) (+ 8).  Q8_0 reads eight bytes a lane: even rows and odd
// rows fall on different banks, consecutive rows do not.
template <int FMT, bool FOLD> __device__ __forceinline__ int g2_row(int gid) {
  if constexpr (FMT != LLB_FM_Q6_K && !FOLD) return ((gid & 3) << 1) | (gid >> 2);
  else return gid;
}

// The two scales and mins of column group j of a Q4_K / Q5_K row from its header words (bytes 4..15), as byte pairs:
// sc = [sc(2j), sc(2j+1)], mn likewise (tools/qwen35_engine.c:66-72)
__device__ __forceinline__ void g2_group_scales(uint32_t u0, uint32_t u1, uint32_t u2, int j, uint32_t &sc, uint32_t &mn) {
  const int s = 16 * (j & 1);
  const uint32_t a = u0 >> s, b = u1 >> s, c = u2 >> s;
  sc = j < 2 ? a & 0x3f3fu : (c & 0x0f0fu) | ((a >> 2) & 0x3030u);
  mn = j < 2 ? b & 0x3f3fu : ((c >> 4) & 0x0f0fu) | ((b >> 2) & 0x3030u);
}

// One staged tile times the staged planes of super-block c_c of the slice: acc[nt] += the tile's contribution to n-tile nt.
//   st     the tile (shared memory);  xh_s, xsf_s, CS  the staged planes, means and column stride
template <int FMT, int NT, bool FOLD>
__device__ __forceinline__ void g2_tile(const uint8_t *st, const uint8_t *xh_s, const uint8_t *xsf_s, const int CS, const int c_c, const int lane, float (&acc)[NT][4]) {
  constexpr int NC = 8 * NT;
  const int gid = lane >> 2, j = lane & 3, r0 = g2_row<FMT, FOLD>(gid);
  const uint8_t *b0 = st + r0 * tile_row(FMT), *b1 = b0 + 8 * tile_row(FMT);
  const uint8_t *xb = xh_s + gid * CS + (size_t)c_c * 512;
  if constexpr (FMT == LLB_FM_Q8_0) {
    // eight blocks of 32 codes, two MMAs each; lane j holds columns 8 j .. 8 j + 7 of a block
    const uint4 sw0 = *(const uint4 *)(b0 + 256), sw1 = *(const uint4 *)(b1 + 256);
    const uint32_t d0w[4] = {sw0.x, sw0.y, sw0.z, sw0.w}, d1w[4] = {sw1.x, sw1.y, sw1.z, sw1.w};
    xb += 16 * j;
#pragma unroll
    for (int blk = 0; blk < 8; blk++) {
      const uint2 w0 = *(const uint2 *)(b0 + 32 * blk + 8 * j), w1 = *(const uint2 *)(b1 + 32 * blk + 8 * j);
      uint32_t A[2][4];
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const uint32_t p0 = u ? w0.y : w0.x, p1 = u ? w1.y : w1.x;
        A[u][0] = g2_hadd2(__byte_perm(p0, 0x64646464u, 0x4240), 0xe480e480u);   // (1024 + byte) - 1152
        A[u][1] = g2_hadd2(__byte_perm(p1, 0x64646464u, 0x4240), 0xe480e480u);
        A[u][2] = g2_hadd2(__byte_perm(p0, 0x64646464u, 0x4341), 0xe480e480u);
        A[u][3] = g2_hadd2(__byte_perm(p1, 0x64646464u, 0x4341), 0xe480e480u);
      }
      const float2 f0 = __half22float2(*(const __half2 *)&d0w[blk >> 1]), f1 = __half22float2(*(const __half2 *)&d1w[blk >> 1]);
      const float d0 = (blk & 1) ? f0.y : f0.x, d1 = (blk & 1) ? f1.y : f1.x;
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        const uint4 bx = *(const uint4 *)(xb + (size_t)nt * 8 * CS + 64 * blk);
        float p[4];
        mma16816_z(p, A[0][0], A[0][1], A[0][2], A[0][3], bx.x, bx.y);
        mma16816(p, A[1][0], A[1][1], A[1][2], A[1][3], bx.z, bx.w);
        acc[nt][0] += d0 * p[0]; acc[nt][1] += d0 * p[1]; acc[nt][2] += d1 * p[2]; acc[nt][3] += d1 * p[3];
      }
    }
  } else if constexpr (FMT == LLB_FM_Q6_K) {
    // 16 scale groups of 16 columns, one MMA each; codes of quarters 2, 3 stay shifted left by four (16 q <= 1008)
    const float d0 = h2f_bits(*(const unsigned short *)(st + 3328 + 2 * r0)), d1 = h2f_bits(*(const unsigned short *)(st + 3328 + 2 * (r0 + 8)));
    const uint4 sw0 = *(const uint4 *)(b0 + 192), sw1 = *(const uint4 *)(b1 + 192);
    const uint32_t sc0w[4] = {sw0.x ^ 0x80808080u, sw0.y ^ 0x80808080u, sw0.z ^ 0x80808080u, sw0.w ^ 0x80808080u};
    const uint32_t sc1w[4] = {sw1.x ^ 0x80808080u, sw1.y ^ 0x80808080u, sw1.z ^ 0x80808080u, sw1.w ^ 0x80808080u};
    xb += 8 * j;
    float sS[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) sS[nt][0] = sS[nt][1] = sS[nt][2] = sS[nt][3] = 0.0f;
#pragma unroll
    for (int hf = 0; hf < 2; hf++) {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        const int o = 16 * u + 4 * j;
        const uint32_t la0 = *(const uint32_t *)(b0 + 64 * hf + o), lb0 = *(const uint32_t *)(b0 + 64 * hf + 32 + o);
        const uint32_t la1 = *(const uint32_t *)(b1 + 64 * hf + o), lb1 = *(const uint32_t *)(b1 + 64 * hf + 32 + o);
        const uint32_t hq0 = *(const uint32_t *)(b0 + 128 + 32 * hf + o), hq1 = *(const uint32_t *)(b1 + 128 + 32 * hf + o);
        const uint32_t h0s4 = hq0 << 4, h0s2 = hq0 << 2, h1s4 = hq1 << 4, h1s2 = hq1 << 2;
        const uint32_t h0o4 = (hq0 >> 8) << 4, h0o2 = (hq0 >> 8) << 2, h1o4 = (hq1 >> 8) << 4, h1o2 = (hq1 >> 8) << 2;
#pragma unroll
        for (int qd = 0; qd < 4; qd++) {
          const uint32_t l0 = (qd & 1) ? lb0 : la0, l1 = (qd & 1) ? lb1 : la1;
          const uint32_t nm = qd < 2 ? 0x000f000fu : 0x00f000f0u, hm = qd < 2 ? 0x00300030u : 0x03000300u;
          const uint32_t off = qd < 2 ? 0xe420e420u : 0xe600e600u;   // -(1024 + 32), -(1024 + 512)
          // the two high bits of quarter 0 / 2 sit four bits up, those of 1 / 3 two bits up; quarters 2, 3 in the byte's upper half
          const uint32_t e0 = g2_hadd2((l0 & nm) | ((((qd & 1) ? h0s2 : h0s4) & hm) | 0x64006400u), off);
          const uint32_t e1 = g2_hadd2((l1 & nm) | ((((qd & 1) ? h1s2 : h1s4) & hm) | 0x64006400u), off);
          const uint32_t o0 = g2_hadd2(((l0 >> 8) & nm) | ((((qd & 1) ? h0o2 : h0o4) & hm) | 0x64006400u), off);
          const uint32_t o1 = g2_hadd2(((l1 >> 8) & nm) | ((((qd & 1) ? h1o2 : h1o4) & hm) | 0x64006400u), off);
          const int gi = 8 * hf + 2 * qd + u;
          // signed scale: (sc ^ 0x80) is sc + 128 as an unsigned byte
          float s0 = __uint_as_float(__byte_perm(sc0w[gi >> 2], 0x4B000000u, 0x7650u | (gi & 3))) - 8388736.0f;
          float s1 = __uint_as_float(__byte_perm(sc1w[gi >> 2], 0x4B000000u, 0x7650u | (gi & 3))) - 8388736.0f;
          if (qd >= 2) { s0 *= 0.0625f; s1 *= 0.0625f; }
          const int kl = 128 * hf + 32 * qd + 16 * u;
#pragma unroll
          for (int nt = 0; nt < NT; nt++) {
            const uint2 bx = *(const uint2 *)(xb + (size_t)nt * 8 * CS + kl * 2);
            float p[4];
            mma16816_z(p, e0, e1, o0, o1, bx.x, bx.y);
            sS[nt][0] += s0 * p[0]; sS[nt][1] += s0 * p[1]; sS[nt][2] += s1 * p[2]; sS[nt][3] += s1 * p[3];
          }
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < NT; nt++) { acc[nt][0] += d0 * sS[nt][0]; acc[nt][1] += d0 * sS[nt][1]; acc[nt][2] += d1 * sS[nt][2]; acc[nt][3] += d1 * sS[nt][3]; }
  } else {
    constexpr int QOFF = FMT == LLB_FM_Q4_K ? 16 : 48;
    const uint4 h0 = *(const uint4 *)b0, h1 = *(const uint4 *)b1;
    if constexpr (!FOLD) {
      uint32_t scA0, scB0, mnA0, mnB0, scA1, scB1, mnA1, mnB1;
      k4_scales(h0.y, h0.z, h0.w, scA0, scB0, mnA0, mnB0);
      k4_scales(h1.y, h1.z, h1.w, scA1, scB1, mnA1, mnB1);
      const uint32_t ms = (j & 1) ? 0x4342u : 0x4140u;
      const uint32_t at0 = __byte_perm(j < 2 ? mnA0 : mnB0, 0x64646464u, ms), at1 = __byte_perm(j < 2 ? mnA1 : mnB1, 0x64646464u, ms);
      const uint32_t am0 = g2_hfma2(at0, 0x3c003c00u, 0xe400e400u), am1 = g2_hfma2(at1, 0x3c003c00u, 0xe400e400u);       // * 1 - 1024
      const uint32_t al0 = g2_hfma2(at0, 0x10001000u, 0xb800b800u), al1 = g2_hfma2(at1, 0x10001000u, 0xb800b800u);       // * 2^-11 - 0.5
      float sS[NT][4], pm[NT][4];
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        const uint2 xf = *(const uint2 *)(xsf_s + ((size_t)c_c * NC + nt * 8 + gid) * 32 + 8 * j);
        mma16816_z(pm[nt], am0, am1, al0, al1, xf.x, xf.y);
        sS[nt][0] = sS[nt][1] = sS[nt][2] = sS[nt][3] = 0.0f;
      }
      xb += 16 * j;
#pragma unroll
      for (int g = 0; g < 4; g++) {
        const uint2 a0 = *(const uint2 *)(b0 + QOFF + 32 * g + 8 * j), a1 = *(const uint2 *)(b1 + QOFF + 32 * g + 8 * j);
        uint2 f0 = make_uint2(0u, 0u), f1 = f0;
        if constexpr (FMT == LLB_FM_Q5_K) { f0 = *(const uint2 *)(b0 + 16 + 8 * j); f1 = *(const uint2 *)(b1 + 16 + 8 * j); }
        uint32_t A[2][2][4];               // [word][low / high nibbles]
#pragma unroll
        for (int w = 0; w < 2; w++) {
          const uint32_t x0 = w ? a0.y : a0.x, x1 = w ? a1.y : a1.x, y0 = x0 >> 8, y1 = x1 >> 8;
          A[w][0][0] = x0 & 0x000f000fu; A[w][0][1] = x1 & 0x000f000fu; A[w][0][2] = y0 & 0x000f000fu; A[w][0][3] = y1 & 0x000f000fu;
          A[w][1][0] = x0 & 0x00f000f0u; A[w][1][1] = x1 & 0x00f000f0u; A[w][1][2] = y0 & 0x00f000f0u; A[w][1][3] = y1 & 0x00f000f0u;
          if constexpr (FMT == LLB_FM_Q5_K) {
            const uint32_t z0 = w ? f0.y : f0.x, z1 = w ? f1.y : f1.x;
            // fifth bits 2 g (low) and 2 g + 1 (high) of every byte to bits 4 and 8
            const int sl = 4 - 2 * g, sh = 7 - 2 * g;
            const uint32_t l0 = sl >= 0 ? z0 << sl : z0 >> -sl, l1 = sl >= 0 ? z1 << sl : z1 >> -sl;
            const uint32_t u0 = z0 << sh, u1 = z1 << sh;
            A[w][0][0] |= l0 & 0x00100010u; A[w][0][1] |= l1 & 0x00100010u; A[w][0][2] |= (l0 >> 8) & 0x00100010u; A[w][0][3] |= (l1 >> 8) & 0x00100010u;
            A[w][1][0] |= u0 & 0x01000100u; A[w][1][1] |= u1 & 0x01000100u; A[w][1][2] |= (z0 >> (8 - sh)) & 0x01000100u; A[w][1][3] |= (z1 >> (8 - sh)) & 0x01000100u;
          }
        }
        const uint32_t s0 = g < 2 ? scA0 : scB0, s1 = g < 2 ? scA1 : scB1;
        const float sc0l = byte_f(s0, (2 * g) & 3), sc0h = byte_f_scaled(s0, (2 * g + 1) & 3, 0.0625f);
        const float sc1l = byte_f(s1, (2 * g) & 3), sc1h = byte_f_scaled(s1, (2 * g + 1) & 3, 0.0625f);
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
          const uint8_t *xr = xb + (size_t)nt * 8 * CS + 128 * g;
          const uint4 bl = *(const uint4 *)xr, bh = *(const uint4 *)(xr + 64);
          float pl[4], ph[4];
          mma16816_z(pl, A[0][0][0], A[0][0][1], A[0][0][2], A[0][0][3], bl.x, bl.y);
          mma16816_z(ph, A[0][1][0], A[0][1][1], A[0][1][2], A[0][1][3], bh.x, bh.y);
          mma16816(pl, A[1][0][0], A[1][0][1], A[1][0][2], A[1][0][3], bl.z, bl.w);
          mma16816(ph, A[1][1][0], A[1][1][1], A[1][1][2], A[1][1][3], bh.z, bh.w);
          sS[nt][0] += sc0l * pl[0] + sc0h * ph[0];
          sS[nt][1] += sc0l * pl[1] + sc0h * ph[1];
          sS[nt][2] += sc1l * pl[2] + sc1h * ph[2];
          sS[nt][3] += sc1l * pl[3] + sc1h * ph[3];
        }
      }
      const float d0 = h2f_bits(h0.x & 0xffffu) * TWO24, dm0 = h2f_bits(h0.x >> 16) * 32.0f;
      const float d1 = h2f_bits(h1.x & 0xffffu) * TWO24, dm1 = h2f_bits(h1.x >> 16) * 32.0f;
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        acc[nt][0] += d0 * sS[nt][0] - dm0 * pm[nt][0];
        acc[nt][1] += d0 * sS[nt][1] - dm0 * pm[nt][1];
        acc[nt][2] += d1 * sS[nt][2] - dm1 * pm[nt][2];
        acc[nt][3] += d1 * sS[nt][3] - dm1 * pm[nt][3];
      }
      return;
    }
    uint32_t sc0, mn0, sc1, mn1;
    g2_group_scales(h0.y, h0.z, h0.w, j, sc0, mn0);
    g2_group_scales(h1.y, h1.z, h1.w, j, sc1, mn1);
    // the scales as fp16 (0x6400 | s is 1024 + s), times 2^10 for the low nibbles and 2^6 for the high ones, which stay four
    // bits up: q 2^-24 * s 2^10 = 16 q 2^-24 * s 2^6 = s q 2^-14, exact
    const uint32_t L0 = g2_hmul2(g2_hadd2(__byte_perm(sc0, 0x64646464u, 0x4040), 0xe400e400u), 0x64006400u);
    const uint32_t L1 = g2_hmul2(g2_hadd2(__byte_perm(sc1, 0x64646464u, 0x4040), 0xe400e400u), 0x64006400u);
    const uint32_t H0 = g2_hmul2(g2_hadd2(__byte_perm(sc0, 0x64646464u, 0x4141), 0xe400e400u), 0x54005400u);
    const uint32_t H1 = g2_hmul2(g2_hadd2(__byte_perm(sc1, 0x64646464u, 0x4141), 0xe400e400u), 0x54005400u);
    // this lane's two mins: 1024 + m exactly; one FMA each gives m for the means' hi halves and m / 2048 for their lo halves
    const uint32_t at0 = __byte_perm(mn0, 0x64646464u, 0x4140), at1 = __byte_perm(mn1, 0x64646464u, 0x4140);
    const uint32_t am0 = g2_hfma2(at0, 0x3c003c00u, 0xe400e400u), am1 = g2_hfma2(at1, 0x3c003c00u, 0xe400e400u);       // * 1 - 1024
    const uint32_t al0 = g2_hfma2(at0, 0x10001000u, 0xb800b800u), al1 = g2_hfma2(at1, 0x10001000u, 0xb800b800u);       // * 2^-11 - 0.5
    float pl[NT][4], ph[NT][4], pm[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      const uint2 xf = *(const uint2 *)(xsf_s + ((size_t)c_c * NC + nt * 8 + gid) * 32 + 8 * j);
      mma16816_z(pm[nt], am0, am1, al0, al1, xf.x, xf.y);
    }
    xb += 16 * j;
#pragma unroll
    for (int q = 0; q < 4; q++) {        // words 2 q and 2 q + 1 of the group's 32 bytes: columns 8 q .. 8 q + 7 of both sub-blocks
      const uint2 a0 = *(const uint2 *)(b0 + QOFF + 32 * j + 8 * q), a1 = *(const uint2 *)(b1 + QOFF + 32 * j + 8 * q);
      uint32_t A[2][2][4];               // [word][low / high nibbles]
#pragma unroll
      for (int w = 0; w < 2; w++) {
        const uint32_t x0 = w ? a0.y : a0.x, x1 = w ? a1.y : a1.x, y0 = x0 >> 8, y1 = x1 >> 8;
        A[w][0][0] = g2_hmul2(x0 & 0x000f000fu, L0); A[w][0][1] = g2_hmul2(x1 & 0x000f000fu, L1);
        A[w][0][2] = g2_hmul2(y0 & 0x000f000fu, L0); A[w][0][3] = g2_hmul2(y1 & 0x000f000fu, L1);
        A[w][1][0] = g2_hmul2(x0 & 0x00f000f0u, H0); A[w][1][1] = g2_hmul2(x1 & 0x00f000f0u, H1);
        A[w][1][2] = g2_hmul2(y0 & 0x00f000f0u, H0); A[w][1][3] = g2_hmul2(y1 & 0x00f000f0u, H1);
      }
#pragma unroll
      for (int nt = 0; nt < NT; nt++) {
        const uint8_t *xr = xb + (size_t)nt * 8 * CS + 64 * q;
        const uint4 bl = *(const uint4 *)xr, bh = *(const uint4 *)(xr + 256);
        if (q == 0) {
          mma16816_z(pl[nt], A[0][0][0], A[0][0][1], A[0][0][2], A[0][0][3], bl.x, bl.y);
          mma16816_z(ph[nt], A[0][1][0], A[0][1][1], A[0][1][2], A[0][1][3], bh.x, bh.y);
        } else {
          mma16816(pl[nt], A[0][0][0], A[0][0][1], A[0][0][2], A[0][0][3], bl.x, bl.y);
          mma16816(ph[nt], A[0][1][0], A[0][1][1], A[0][1][2], A[0][1][3], bh.x, bh.y);
        }
        mma16816(pl[nt], A[1][0][0], A[1][0][1], A[1][0][2], A[1][0][3], bl.z, bl.w);
        mma16816(ph[nt], A[1][1][0], A[1][1][1], A[1][1][2], A[1][1][3], bh.z, bh.w);
      }
    }
    const float d0 = h2f_bits(h0.x & 0xffffu) * 16384.0f, dm0 = h2f_bits(h0.x >> 16) * 32.0f;
    const float d1 = h2f_bits(h1.x & 0xffffu) * 16384.0f, dm1 = h2f_bits(h1.x >> 16) * 32.0f;
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      acc[nt][0] += d0 * (pl[nt][0] + ph[nt][0]) - dm0 * pm[nt][0];
      acc[nt][1] += d0 * (pl[nt][1] + ph[nt][1]) - dm0 * pm[nt][1];
      acc[nt][2] += d1 * (pl[nt][2] + ph[nt][2]) - dm1 * pm[nt][2];
      acc[nt][3] += d1 * (pl[nt][3] + ph[nt][3]) - dm1 * pm[nt][3];
    }
  }
}

// The warp's ring as it passes from one GEMM phase to the next: barriers (one a stage), stage memory, and the parity that
// each stage's next wait looks for.
struct G2Ring { uint32_t bar_s, ring_s; const uint8_t *ring; uint32_t par; bool dead; };   // dead: a wait ran out, nothing more is requested
// smem: G2_BAR_BYTES of barriers and then the rings, `per_warp` bytes each.  Private to a warp: no block barrier needed.
__device__ __forceinline__ G2Ring g2_ring_init(uint8_t *smem, int per_warp) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  G2Ring r;
  r.bar_s = smem_u32(smem) + warp * 32;
  r.ring = smem + G2_BAR_BYTES + warp * per_warp;
  r.ring_s = smem_u32(r.ring);
  r.par = 0; r.dead = false;
  if (warp < G2_MAXWARPS && lane == 0) {
    for (int s = 0; s < 4; s++) mbar_init(r.bar_s + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  return r;
}

// The next wait on stage s.  Where one runs out, nothing is requested or waited for after it, and bits 8 .. of par keep the
// parities as they are then: those of the phases that requests in flight will complete.
__device__ __forceinline__ void g2_wait(G2Ring &r, int s, uint32_t limit, unsigned int *err) {
  if (!r.dead && !mbar_wait(r.bar_s + 8 * s, (r.par >> s) & 1u, limit)) { r.dead = true; r.par |= (r.par & 7u) << 8; if (err) atomicExch(err, 1u); }
  r.par ^= 1u << s;
}
// After a wait ran out: what is still in flight lands before the block leaves.  (A stage with no request has nothing to wait for
// and costs the limit, some milliseconds.)
__device__ __forceinline__ void g2_drain(const G2Ring &r) {
  if (r.dead) for (int s = 0; s < 3; s++) mbar_wait(r.bar_s + 8 * s, (r.par >> (8 + s)) & 1u, G2_DRAIN_LIMIT);
}

// Where a launch's row tiles live.  A policy says how many 16-row tiles there are, where tile i's 16 x 256 tiles in the
// CTA's K-slice are, and what to do with a finished row tile.  G2MatsPlain is the launch of up to four matrices that
// GemmArgs describes.
//   Cur     cursor of the row tile being copied;  locate  row tile -> cursor;  src  tile of super-block sb0 + c of the slice
template <int FMT, bool FOLD = false> struct G2MatsPlain {
  const GemmArgs &a;
  struct Cur { const uint8_t *W; };
  __device__ __forceinline__ int ntiles() const { return a.tile0[a.nmat]; }
  __device__ __forceinline__ void locate(int tile, int sb0, Cur &c) const {
    int m = 0;
    while (m + 1 < a.nmat && tile >= a.tile0[m + 1]) m++;
    c.W = a.m[m].W + ((size_t)(tile - a.tile0[m]) * a.nsb + sb0) * tile_bytes(FMT);
  }
  __device__ __forceinline__ const uint8_t *src(const Cur &c, int pc) const { return c.W + (size_t)pc * tile_bytes(FMT); }
  template <int NT> __device__ __forceinline__ void epilogue(int ks, int tile, float (&acc)[NT][4], int lane) const {
    int m = 0;
    while (m + 1 < a.nmat && tile >= a.tile0[m + 1]) m++;
    gemm_epilogue<NT>(a, a.m[m], ks, (tile - a.tile0[m]) * 16 + g2_row<FMT, FOLD>(lane >> 2), acc, lane);
  }
};

// One launch's work of a CTA (bid of cps * ksplit): fill the rings, call stage(xh_s, xsf_s, CS, sb0, nsl) -- which waits for
// whatever produces the activations, puts the CTA's slice of the planes and its side array into shared memory and ends with
// a block-wide barrier --, then stream the CTA's row tiles.  CTAs and warps beyond the launch's only take part in staging.
//
// a.parts = P warps share a row tile: its super-blocks of the slice are P parts, a warp each, and the first warp of the
// group adds in order what the others leave in shared memory.  A small launch leaves most warps of an SM without a tile of
// their own and the others with a chain of 1200 cycles a super-block (0.8B shape: four tiles an SM), which is what sharing a
// tile shortens; it also needs fewer K-slices, whose partial sums the next kernel has to add.  P depends on the launch's
// shape only, not on which of its rows are in use, so that a row's sums do not depend on its neighbours.
//
// Tile of (CTA ci, warp group w, round n) = (n * groups + w) * cps + ci: consecutive tiles go to different SMs, so the SMs'
// tile counts differ by one at most.
template <int FMT, int NT, class Stage, class Mats, bool FOLD = false, int RING = 0>
__device__ __forceinline__ void g2_phase(const GemmArgs &a, const int cps, const int bid, G2Ring &rg, uint8_t *planes, Stage stage, const Mats mats) {
  constexpr int NC = 8 * NT, WARPS = g2_warps(FMT, NC), TB = tile_bytes(FMT), ST = g2_stages(FMT, NC, RING), CH = g2_chunk(FMT, RING);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool live = bid < cps * a.ksplit && warp < WARPS;
  const int ks = bid % a.ksplit, ci = bid / a.ksplit;
  const int sb0 = (int)(((long long)ks * a.nsb) / a.ksplit), nsl = (int)(((long long)(ks + 1) * a.nsb) / a.ksplit) - sb0;
  const int CS = nsl * 512 + g2_xpad(FMT);
  uint8_t *xh_s = planes, *xsf_s = planes + NC * CS;
  const int P = a.parts, lp = 31 - __clz(P), grp = warp >> lp, mine = warp & (P - 1), nws = (WARPS >> lp) * cps;
  const int tile0 = grp * cps + ci, c0 = (mine * nsl) >> lp, c1 = ((mine + 1) * nsl) >> lp;   // this warp's tiles; its part
  const int ntiles = live ? mats.ntiles() : 0;                    // a warp that is not live sees no tiles
  int p_tile = tile0, p_c = c0;                                   // producer: (tile, super-block) of the next copy
  typename Mats::Cur p_cur;
  if (p_tile < ntiles) mats.locate(p_tile, sb0, p_cur);
  auto issue = [&](int s) {
    if (p_tile >= ntiles || rg.dead) return;
    const int n = min(CH, c1 - p_c);
    if (lane == 0) {
      const uint32_t bar = rg.bar_s + 8 * s, dst = rg.ring_s + s * CH * TB;
      mbar_expect(bar, n * TB);
      bulk_load(dst, mats.src(p_cur, p_c), n * TB, bar);
    }
    p_c += n;
    if (p_c == c1) {
      p_c = c0; p_tile += nws;
      if (p_tile < ntiles) mats.locate(p_tile, sb0, p_cur);
    }
  };
  // weights first where their addresses depend on no kernel: the ring is in flight while the producer of the activations
  // still runs, and while the activation slice is staged
#pragma unroll 1
  for (int s = 0; s < ST; s++) issue(s);
  stage(xh_s, xsf_s, CS, sb0, nsl);
  float4 *red = (float4 *)(planes + NC * (((a.nsb + a.ksplit - 1) / a.ksplit) * (512 + g2_aux(FMT)) + g2_xpad(FMT))) + warp * NT * 32 + lane;
  int s = 0;
#pragma unroll 1
  for (int tile = tile0; tile < ntiles; tile += nws) {
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; nt++) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.0f;
#pragma unroll 1
    for (int c = c0; c < c1; c += CH) {
      g2_wait(rg, s, G2_WAIT_LIMIT, a.err);
#pragma unroll 1
      for (int u = 0; u < CH && c + u < c1; u++) g2_tile<FMT, NT, FOLD>(rg.ring + (s * CH + u) * TB, xh_s, xsf_s, CS, c + u, lane, acc);
      __syncwarp();                                        // every lane has read the stage
      issue(s);
      s = s + 1 == ST ? 0 : s + 1;
    }
    if (P > 1) {
      if (mine) {
#pragma unroll
        for (int nt = 0; nt < NT; nt++) red[nt * 32] = make_float4(acc[nt][0], acc[nt][1], acc[nt][2], acc[nt][3]);
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * P) : "memory");
      if (!mine) {
#pragma unroll 1
        for (int q = 1; q < P; q++)
#pragma unroll
          for (int nt = 0; nt < NT; nt++) {
            const float4 v = red[(q * NT + nt) * 32];
            acc[nt][0] += v.x; acc[nt][1] += v.y; acc[nt][2] += v.z; acc[nt][3] += v.w;
          }
      }
      if (tile + nws < ntiles) asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * P) : "memory");   // read before it is written again
    }
    if (!mine) mats.template epilogue<NT>(ks, tile, acc, lane);
  }
}

// The activation slice from the planes in global memory: the columns of the launch's rows only (a one-row pass uses two of
// eight; an MMA's columns do not see one another, so what the others hold does not matter).  Sixteen-byte cp.async by all
// warps; one bulk copy a column took 0.5 us longer a launch.
template <int FMT, int NT, bool FOLD = false> struct G2StagePlanes {
  const GemmArgs &a;
  __device__ __forceinline__ void operator()(uint8_t *xh_s, uint8_t *xsf_s, int CS, int sb0, int nsl) const {
    constexpr int NC = 8 * NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5, ntask = a.planes * a.T * nsl;
    const uint8_t *xh = (const uint8_t *)(a.xp.xh + (size_t)sb0 * 256), *xf = (const uint8_t *)(a.xp.xsf + (size_t)sb0 * NC * 16);
    pdl_wait();
#pragma unroll 2
    for (int task = warp; task < ntask; task += nw) {   // (live column, super-block): 32 pieces, a lane each
      const int i = task / nsl, sb = task - i * nsl, c = i < a.T ? i : NC / 2 + i - a.T, p = sb * 32 + lane;
      cp_async16(smem_u32(xh_s + c * CS) + g2_xpos<FMT, FOLD>(p), xh + (size_t)c * a.K * 2 + p * 16);
    }
    if constexpr (g2_aux(FMT) != 0)         // the means of the slice: contiguous in global memory
      for (int i = threadIdx.x; i < nsl * NC * 2; i += blockDim.x) cp_async16(smem_u32(xsf_s + i * 16), xf + i * 16);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  }
};

template <int FMT, int NT, bool FOLD, int RING>
__global__ void __launch_bounds__(g2_warps(FMT, 8 * NT) * 32, 1) k_gemm2(const GemmArgs a, const int cps) {
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  constexpr int RB = g2_ring_bytes(FMT, 8 * NT, RING);
  G2Ring rg = g2_ring_init(smem, RB / g2_warps(FMT, 8 * NT));
  g2_phase<FMT, NT, G2StagePlanes<FMT, NT, FOLD>, G2MatsPlain<FMT, FOLD>, FOLD, RING>(a, cps, (int)blockIdx.x, rg, smem + G2_BAR_BYTES + RB, G2StagePlanes<FMT, NT, FOLD>{a},
                                                                                         G2MatsPlain<FMT, FOLD>{a});
  g2_drain(rg);
}
