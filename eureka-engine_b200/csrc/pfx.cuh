// pfx.cuh -- the prompt path's dense GEMM with the integer codes themselves as the tensor core's operand: Y[r][n] = sum_k W[n][k] X[r][k]
// for up to 256 prompt rows.  The other dense kernel (pfmm.cuh) dequantises every weight into two fp16 planes and pays three MMAs a
// step; here a weight of a super-block is an exact fp16 integer (times a power of two) in ONE plane, the super-block's scale comes in afterwards:
//
//   Q4_K, Q5_K  sc (q - 8) and sc (q - 16), at most 504 and 1008.  What the centring took and the mins are one more K = 16 step of a
//               super-block, 32 (8 sc - (dmin / d) m) as two fp16 halves against the means of the activations' 32-column groups
//   Q6_K        sc (q - 32), at most 4096: fp16 product and its exact remainder, two planes.  (Planes of the code's low four and high two bits are exact too and cheaper to
//               unpack, 5120 x 17408 and 20 / 50 / 120 rows 40 / 60 / 70 us where this takes 46 / 66 / 70, but they are large and cancel where codes are small: with weights of N^3 and activations of one sign, 17408 columns, what is truncated off
//               their sums came to 2.9e-6 of the result)
//   Q8_0        d q with the eight d's of the super-block scaled by a common power of two: fp16 product and its exact remainder, two planes
//
// and the activations are their two fp16 planes, so the products are exact but for the activations' 22 bits.  The accumulators of a
// super-block are read out of tensor memory and scaled by d into registers while the tensor core goes on with the next:
// chains of 17 (33) truncating additions instead of thousands.
//
// A PAIR of CTAs (cta_group::2) has 256 weight rows, 128 a CTA.  Two kernels:
//   k_pfx2  two units of 128 prompt rows, one in each CTA's shared memory, N = 256, two MMAs a step.  A super-block's codes . lo come first,
//           then, on top of that sum divided by 2048 (the MMA's own scaling of D), its codes . hi: one accumulator of 256
//           columns, so that two fit tensor memory and one is read while the other fills.  128 sums a thread in the 256 threads that read
//           them (setmaxnreg).
//   k_pfx1  RU = 64 or 128 prompt rows: the first CTA stages the hi plane, the second the lo plane, N = 2 RU, one MMA a step and
//           plane of codes; two accumulators take turns, a stage each.
//   k_pft   the same for up to 32 rows with the codes in tensor memory.
// Weights come as bulk copies of whole super-blocks of a 16-row tile into a ring of their own.
//
// gate|up of the 27B shape, 256 rows: 194 GFLOP of products in 136 us = 1.43 PFLOP/s, 87 % of cuBLAS's measured burst; the kernel of three products took 185 us.  What bounds
// k_pfx2 is the tensor pipe, 83 % active at the 1.57 GHz that the power limit leaves it (a loop of nothing but these MMAs on random operands runs at 1.37 to 1.44 GHz and 1.65
// to 1.74 PFLOP/s, on zeros at 1.82 GHz), and how the tiles fill the chip: 136 units on 74 pairs of SMs are 92 % of two rounds.  A 3011-token prompt on that shape 515 -> 432 ms.  Error against 64 bits, N(0, 1) activations,
// 5120 / 17408 columns in a prompt's K-slices: k_pfx2 Q4_K 3.1e-7 / 3.4e-7, Q5_K 3.5e-7 / 3.7e-7 (k_pfmm 6.1e-6 / 2.0e-5); k_pfx1 and k_pft beside the passes of eight rows
// whose place they take: Q4_K 1.9e-7 / 2.2e-7 (10e-7 / 3.2e-7 there), Q5_K 2.1e-7 / 2.3e-7 (4.1e-7 / 3.8e-7), Q6_K 1.07e-7 / 1.29e-7 (1.08e-7 / 1.20e-7), Q8_0 1.11e-7 /
// 1.34e-7 (1.27e-7 / 2.0e-7); 1024 columns of Q8_0 1.00e-7 (0.90e-7); with silu(g) u Q6_K 1.10e-7 / 1.32e-7 (1.12e-7 / 1.22e-7), Q8_0 1.14e-7 / 1.36e-7 (1.33e-7 / 2.05e-7).
// Every wait is bounded; one that runs out sets *err, all roles then run through, tensor memory is freed and the kernel returns.
#pragma once
#include "pfmm.cuh"
#include "gemm2.cuh"

#define PX_THREADS 512      // k_pfx2: warps 0-3 unpack, 4 loads weights, 5 activations, 6 issues MMAs, 7 forwards, 8-15 read accumulators
#define PX_HDR 1024
#define PX_SC (4 * 128 * 4)                    // scales of the last four super-blocks, a word a weight row
#define PX_OA (2 * 128 * 16)                   // the offsets' step: weight rows' side
#define PX_SMEM_MAX 231424
__host__ __device__ constexpr int px_planes(int fmt) { return fmt == LLB_FM_Q6_K || fmt == LLB_FM_Q8_0 ? 2 : 1; }
__host__ __device__ constexpr bool px_offs(int fmt) { return px_planes(fmt) == 1; }
__host__ __device__ constexpr int px_a_bytes(int fmt) { return px_planes(fmt) * PF_A_BYTES; }
__host__ __device__ constexpr int px_b_bytes(int RU) { return RU * PF_KS * 2; }          // one plane of a stage's activations
__host__ __device__ constexpr int px_ob_bytes(int RU) { return RU * 32; }                // ... and of the offsets' step
// 64-column parts after which k_pfx1's accumulators are read, a stage's: the tensor core truncates where it adds to one, so that a sum loses about 2e-8 of itself an
// MMA.  Its prompts take the place of verify rows, so it is read as often as that hides behind the MMAs.
__host__ __device__ constexpr int px_drain(int fmt) { return px_planes(fmt) == 2 ? 1 : 2; }
// The part of a sum of two planes that the truncations of its four additions with the larger plane take off, always towards zero: measured 8.9e-8 for Q8_0 and 8.2e-8 for
// Q6_K, whatever the columns, and for activations of either sign or one, with short or long tails (8.8e-8 for silu(g) u).  The sums are given it back at the end, which is
// one unit of the last place.  Where the sums are exact without it they lose by that: 1 + 0.1 N 1.02e-7 both ways, activations of which 2 % are not zero 0.8 -> 1.1e-7.
constexpr float PX_LOST = 8.5e-8f;
// k_pfx1's rings: codes in stages of eight MMAs, 128 columns of one plane or 64 of two (a stage costs the issuing warp and the unpacking ones
// some 400 cycles whatever is in it); not more than a super-block, because the offsets' step has one buffer on the weight rows' side, which a
// super-block's last stage fills and the same stage of the next fills again, when the MMAs of the stage `px_na` before that one are done;
// activations in slots of 16 KB and, where there is such a step, the means of a super-block behind them; weights in chunks of whole
// super-blocks (a copy costs the SM's copy engine about 85 cycles, gemm2.cuh).
#define PX_SLOT 16384
#define PT_RU 32              // rows of k_pft, the kernel of the fewest
#define PT_NB 4               // its slots: its two groups have two each
#define PT_THREADS 640        // warps 0-7 unpack, 8 loads weights, 9 activations, 10 and 11 issue MMAs (in the second CTA 11 forwards), 12-19 read accumulators
__host__ __device__ constexpr int px_sub(int fmt) { return 3 - px_planes(fmt); }     // 64-column parts of a stage
__host__ __device__ constexpr int px_na(int fmt) { return px_planes(fmt) == 2 ? 3 : 2; }
__host__ __device__ constexpr int px_slot_stages(int RU) { return PX_SLOT / px_b_bytes(RU); }
__host__ __device__ constexpr int px_slot_bytes(int fmt, int RU) { return PX_SLOT + (px_offs(fmt) ? px_ob_bytes(RU) : 0); }
__host__ __device__ constexpr int px_nb(int fmt) { return fmt == LLB_FM_Q8_0 ? 3 : 4; }
__host__ __device__ constexpr int px_chunk(int fmt) { return fmt == LLB_FM_Q4_K ? 2 : 1; }
__host__ __device__ constexpr int px_raw_bytes(int fmt) { return 8 * px_chunk(fmt) * tile_bytes(fmt); }
__host__ __device__ constexpr int px_fixed(int fmt, int RU) { return PX_HDR + PX_SC + (px_offs(fmt) ? PX_OA : 0) + px_na(fmt) * px_sub(fmt) * px_a_bytes(fmt) + px_nb(fmt) * px_slot_bytes(fmt, RU); }
__host__ __device__ constexpr int px_raws(int fmt, int RU) {
  const int n = (PX_SMEM_MAX - px_fixed(fmt, RU)) / px_raw_bytes(fmt);
  return n > 4 ? 4 : n;
}
__host__ __device__ constexpr int px_smem(int fmt, int RU) { return px_fixed(fmt, RU) + px_raws(fmt, RU) * px_raw_bytes(fmt); }
static_assert(px_na(LLB_FM_Q4_K) * px_sub(LLB_FM_Q4_K) <= 4 && px_drain(LLB_FM_Q4_K) == px_sub(LLB_FM_Q4_K) && px_drain(LLB_FM_Q6_K) == px_sub(LLB_FM_Q6_K), "one buffer of the offsets' step; an accumulator a stage");
// k_pfx2's rings: 64 columns of codes (a super-block's four stay until its hi products are done), 64 columns of one plane of the activations
#define PX2_NA 6
#define PX2_NB 4
#define PX2_NRAW 2
static_assert(PX2_NB >= 4 && PX2_NA >= 4 && PX2_NA <= 8, "buffers of the offsets' step: the weight rows' side two, the prompt rows' one a plane");
__host__ __device__ constexpr int px2_smem(int fmt) {
  return PX_HDR + PX_SC + 2 * PX_OA + 2 * px_ob_bytes(128) + PX2_NA * PF_A_BYTES + PX2_NB * PF_B_BYTES + PX2_NRAW * 8 * tile_bytes(fmt);
}
static_assert(px2_smem(LLB_FM_Q5_K) <= PX_SMEM_MAX, "k_pfx2's rings");
// registers a thread of k_pfx2's four warpgroups (unpack, loads and issue, two that read): together what the block is launched with
#define PX_REG_UNPACK 80
#define PX_REG_ISSUE 48
#define PX_REG_READ 192
#define PX_REG_LAUNCH 128
static_assert(PX_REG_UNPACK + PX_REG_ISSUE + 2 * PX_REG_READ == 4 * PX_REG_LAUNCH, "setmaxnreg.inc waits for ever where the shares are more than the launch's registers");
// k_pfx1: eight warps unpack (four where a thread that reads has 128 sums, below: the registers are needed there, and the MMAs of 128 rows and two planes take longer
// than four warps' unpacking), then one that loads weights, one activations, one issues MMAs, one forwards, eight read accumulators
__host__ __device__ constexpr int px1_unpack(int fmt, int RU) { return px_planes(fmt) == 2 && RU == 128 ? 4 : 8; }
__host__ __device__ constexpr int px1_threads(int fmt, int RU) { return 32 * (px1_unpack(fmt, RU) + 12); }
#define PX1_REG_UNPACK 80
__host__ __device__ constexpr int px1_reg_issue(int fmt, int RU) { return px1_unpack(fmt, RU) == 4 ? 48 : 64; }
__host__ __device__ constexpr int px1_reg_read(int fmt, int RU) { return px1_unpack(fmt, RU) == 4 ? 192 : 128; }
__host__ __device__ constexpr int px1_reg_launch(int fmt, int RU) { return px1_unpack(fmt, RU) == 4 ? 128 : 96; }
constexpr bool px1_split(int fmt, int RU) {
  return px1_unpack(fmt, RU) / 4 * PX1_REG_UNPACK + px1_reg_issue(fmt, RU) + 2 * px1_reg_read(fmt, RU) == px1_threads(fmt, RU) / 128 * px1_reg_launch(fmt, RU);
}
static_assert(px1_split(LLB_FM_Q4_K, 64) && px1_split(LLB_FM_Q4_K, 128) && px1_split(LLB_FM_Q6_K, 64) && px1_split(LLB_FM_Q6_K, 128), "as above");
__host__ __device__ constexpr uint32_t px_idesc(int N) { return 0x10000010u | ((uint32_t)(N >> 3) << 17); }   // kind::f16: D f32, A / B f16 K-major, M = 256 over the pair

// ---- one 64-column stage s of a weight row's super-block into core-matrix rows of the code planes ----
// What a super-block's row needs besides its codes.
struct PxRow { uint32_t w[4]; uint32_t kap; };
// Reads the row's header; scale = what the accumulators of the super-block are multiplied with; off: the offsets' step of the row
template <int FMT> __device__ __forceinline__ void px_head(const uint8_t *row, const uint8_t *tile, int r16, bool with_off, PxRow &h, float &scale, uint4 (&off)[2]) {
  if constexpr (px_offs(FMT)) {
    const uint4 hd = *(const uint4 *)row;
    k4_scales(hd.y, hd.z, hd.w, h.w[0], h.w[1], h.w[2], h.w[3]);
    const float d0 = h2f_bits(hd.x & 0xffffu), dm = h2f_bits(hd.x >> 16);
    float d = d0, kap = 1.0f;
    // (dmin / d) m 2^-9 has to stay an fp16 number.  Where dmin is more than 2^18 d the codes are taken 2^-j of themselves and d 2^j: what
    // that costs a code is below the mins' own rounding.
    if (!(fabsf(dm) <= 262144.0f * fabsf(d0)) && (h.w[2] | h.w[3]) != 0) {
      if (d0 == 0.0f) { d = fabsf(dm) * (1.0f / 262144.0f); kap = 0.0f; }
      else {
        const int j = min(60, (int)(__float_as_uint(fabsf(dm)) >> 23) - (int)(__float_as_uint(fabsf(d0)) >> 23) - 17);
        d = d0 * __uint_as_float((uint32_t)(127 + j) << 23); kap = __uint_as_float((uint32_t)(127 - j) << 23);
      }
    }
    const float rho = d != 0.0f && (h.w[2] | h.w[3]) != 0 ? __fdiv_rn(dm, d) : 0.0f;
    const __half2 k2 = __floats2half2_rn(kap, kap);
    h.kap = *(const uint32_t *)&k2;
    scale = d * 16384.0f;
    if (!with_off) return;
    constexpr float C = FMT == LLB_FM_Q4_K ? 8.0f : 16.0f;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t s = i < 2 ? h.w[0] : h.w[1], m = i < 2 ? h.w[2] : h.w[3];
      const float a = (C * kap * byte_f(s, (2 * i) & 3) - rho * byte_f(m, (2 * i) & 3)) * 0.001953125f;           // * 32 2^-14
      const float b = (C * kap * byte_f(s, (2 * i + 1) & 3) - rho * byte_f(m, (2 * i + 1) & 3)) * 0.001953125f;
      const __half2 hh = __floats2half2_rn(a, b);
      const float2 hf = __half22float2(hh);
      const __half2 ll = __floats2half2_rn(a - hf.x, b - hf.y);
      hi[i] = *(const uint32_t *)&hh; lo[i] = *(const uint32_t *)&ll;
    }
    off[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]); off[1] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  } else if constexpr (FMT == LLB_FM_Q6_K) {
    const uint4 sc = *(const uint4 *)(row + 192);
    h.w[0] = sc.x ^ 0x80808080u; h.w[1] = sc.y ^ 0x80808080u; h.w[2] = sc.z ^ 0x80808080u; h.w[3] = sc.w ^ 0x80808080u;
    scale = h2f_bits(*(const unsigned short *)(tile + 3328 + 2 * r16)) * 65536.0f;
  } else {
    const uint4 d = *(const uint4 *)(row + 256);
    const uint32_t w[4] = {d.x, d.y, d.z, d.w};
    uint32_t mx = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) mx = max(mx, max(w[i] & 0x7fffu, (w[i] >> 16) & 0x7fffu));
    const int e = max(1, (int)(mx >> 10));             // the largest |d| as a number from 16 to 32
    const float up = __uint_as_float((uint32_t)(146 - e) << 23);
    scale = __uint_as_float((uint32_t)(108 + e) << 23);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float2 f = __half22float2(*(const __half2 *)&w[i]);
      const __half2 n = __floats2half2_rn(f.x * up, f.y * up);
      h.w[i] = *(const uint32_t *)&n;
    }
  }
}
// k-group g of the stage, plane p: o[8 p + g].  (s is not unrolled over: with the super-block's four stages, and the eight of the MMAs, as
// straight-line code the kernel's roles threw each other out of the instruction cache; gate|up of the 27B shape 182 us.)
__device__ __forceinline__ uint32_t px_pick(const uint32_t (&w)[4], int s) { return s & 2 ? (s & 1 ? w[3] : w[2]) : (s & 1 ? w[1] : w[0]); }
// P = 2: a thread has half of the stage's columns, part `part`: columns 16 part .. of both groups of 32 (Q8_0: 32 part ..)
template <int FMT, int P = 1> __device__ __forceinline__ void px_stage(const uint8_t *row, int s, int part, const PxRow &h, uint4 (&o)[8 * px_planes(FMT) / P]) {
  if constexpr (px_offs(FMT)) {
    constexpr int QOFF = FMT == LLB_FM_Q4_K ? 16 : 48;
    const uint32_t sw = s < 2 ? h.w[0] : h.w[1];
    // the scales as fp16 (0x6400 | s is 1024 + s) times 2^10 for the low nibbles and 2^6 for the high ones, which stay four bits up;
    // codes are subnormals q 2^-24: q 2^-24 * s 2^10 - 8 s 2^-14 = 16 q 2^-24 * s 2^6 - 8 s 2^-14 = s (q - 8) 2^-14, exact
    const uint32_t sl = g2_hmul2(g2_hadd2(__byte_perm(sw, 0x64646464u, s & 1 ? 0x4242u : 0x4040u), 0xe400e400u), h.kap);
    const uint32_t sh = g2_hmul2(g2_hadd2(__byte_perm(sw, 0x64646464u, s & 1 ? 0x4343u : 0x4141u), 0xe400e400u), h.kap);
    const uint32_t L = g2_hmul2(sl, 0x64006400u), H = g2_hmul2(sh, 0x54005400u);
    constexpr uint32_t CL = FMT == LLB_FM_Q4_K ? 0x80088008u : 0x80108010u, CH = FMT == LLB_FM_Q4_K ? 0x80808080u : 0x81008100u;
    const uint32_t L8 = g2_hmul2(L, CL), H8 = g2_hmul2(H, CH);
#pragma unroll
    for (int i2 = 0; i2 < 2 / P; i2++) {
      const int g2 = P == 2 ? part : i2;
      const uint4 q = *(const uint4 *)(row + QOFF + 32 * s + 16 * g2);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      uint32_t z[4] = {0, 0, 0, 0};
      if constexpr (FMT == LLB_FM_Q5_K) { const uint4 f = *(const uint4 *)(row + 16 + 16 * g2); z[0] = f.x; z[1] = f.y; z[2] = f.z; z[3] = f.w; }
      uint32_t lo[8], hi[8];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const uint32_t y = w[i] >> 8;
        uint32_t a0 = w[i] & 0x000f000fu, a1 = y & 0x000f000fu, b0 = w[i] & 0x00f000f0u, b1 = y & 0x00f000f0u;
        if constexpr (FMT == LLB_FM_Q5_K) {   // fifth bits 2 s (low) and 2 s + 1 (high) of every byte to bits 4 and 8
          const uint32_t t = z[i] >> (2 * s);
          a0 |= (t << 4) & 0x00100010u; a1 |= (t >> 4) & 0x00100010u;
          b0 |= (t << 7) & 0x01000100u; b1 |= (t >> 1) & 0x01000100u;
        }
        lo[2 * i] = g2_hfma2(a0, L, L8); lo[2 * i + 1] = g2_hfma2(a1, L, L8);
        hi[2 * i] = g2_hfma2(b0, H, H8); hi[2 * i + 1] = g2_hfma2(b1, H, H8);
      }
      o[2 * i2] = make_uint4(lo[0], lo[1], lo[2], lo[3]); o[2 * i2 + 1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
      o[4 / P + 2 * i2] = make_uint4(hi[0], hi[1], hi[2], hi[3]); o[4 / P + 2 * i2 + 1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
    }
  } else if constexpr (FMT == LLB_FM_Q6_K) {
    const int hf = s >> 1, odd = s & 1;
    // codes as fp16 subnormals q 2^-24, those of high nibbles four bits up, then (q - 32) 2^-9 times sc 2^-7
    const uint32_t scw = px_pick(h.w, s), nm = odd ? 0x00f000f0u : 0x000f000fu, hm = odd ? 0x03000300u : 0x00300030u, up = odd ? 0x68006800u : 0x78007800u;
#pragma unroll
    for (int i2 = 0; i2 < 2 / P; i2++) {       // sixteen columns 16 c .. of both quarters
      const int c = P == 2 ? part : i2;
      const uint4 hq4 = *(const uint4 *)(row + 128 + 32 * hf + 16 * c);
      const uint32_t hw[4] = {hq4.x, hq4.y, hq4.z, hq4.w};
#pragma unroll
      for (int qq = 0; qq < 2; qq++) {
        const uint32_t sv = g2_hadd2(__byte_perm(scw, 0x64646464u, 0x4040u + 0x0101u * (2 * qq + c)), 0xe480e480u);   // (1024 + 128 + sc) - 1152
        const uint32_t S = g2_hmul2(sv, 0x20002000u);
        const uint4 l4 = *(const uint4 *)(row + 64 * hf + 32 * qq + 16 * c);
        const uint32_t lw[4] = {l4.x, l4.y, l4.z, l4.w};
        uint32_t P1[8], P2[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint32_t a0 = (lw[i] & nm) | (hw[i] << (4 - 2 * qq) & hm), a1 = ((lw[i] >> 8) & nm) | (hw[i] >> (4 + 2 * qq) & hm);
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const uint32_t x = g2_hfma2(e ? a1 : a0, up, 0xac00ac00u), p = g2_hmul2(x, S);
            P1[2 * i + e] = p; P2[2 * i + e] = g2_hfma2(x, S, p ^ 0x80008000u);
          }
        }
        const int g = 4 / P * qq + 2 * i2;
        o[g] = make_uint4(P1[0], P1[1], P1[2], P1[3]); o[g + 1] = make_uint4(P1[4], P1[5], P1[6], P1[7]);
        o[8 / P + g] = make_uint4(P2[0], P2[1], P2[2], P2[3]); o[8 / P + g + 1] = make_uint4(P2[4], P2[5], P2[6], P2[7]);
      }
    }
  } else {
    const uint32_t dw = px_pick(h.w, s);
#pragma unroll
    for (int i2 = 0; i2 < 4 / P; i2++) {       // sixteen columns of block 2 s + c / 2
      const int c = P == 2 ? 2 * part + i2 : i2;
      const uint32_t dn = __byte_perm(dw, 0, c < 2 ? 0x1010u : 0x3232u);
      const uint4 q = *(const uint4 *)(row + 64 * s + 16 * c);
      const uint32_t w[4] = {q.x, q.y, q.z, q.w};
      uint32_t P1[8], P2[8];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const uint32_t x = g2_hadd2(__byte_perm(w[i], 0x64646464u, e ? 0x4341 : 0x4240), 0xe480e480u), p = g2_hmul2(x, dn);
          P1[2 * i + e] = p; P2[2 * i + e] = g2_hfma2(x, dn, p ^ 0x80008000u);   // what the product's rounding left out
        }
      o[2 * i2] = make_uint4(P1[0], P1[1], P1[2], P1[3]); o[2 * i2 + 1] = make_uint4(P1[4], P1[5], P1[6], P1[7]);
      o[8 / P + 2 * i2] = make_uint4(P2[0], P2[1], P2[2], P2[3]); o[8 / P + 2 * i2 + 1] = make_uint4(P2[4], P2[5], P2[6], P2[7]);
    }
  }
}

// D = A B + D 2^-11
__device__ __forceinline__ void px_mma_scaled(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p, 11;\n\t}\n" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc)
      : "memory");
}
// the k-group of the stage that o[i] of a plane is (i < 8 / P)
template <int FMT, int P> __device__ __forceinline__ int px_group(int i, int part) {
  if (P == 1) return i;
  if constexpr (FMT == LLB_FM_Q8_0) return 4 * part + i;
  else return 4 * (i >> 1) + 2 * part + (i & 1);
}
// Sums of two planes: a super-block's four stages first, then the super-blocks.  One sum over all stages lost 2.5e-8 sqrt(stages / 2) of the result by its own rounding: 17408
// columns in three slices 2.1e-7, so 1.5e-7, 5120 columns 1.46e-7, so 1.33e-7.  (Two super-blocks together, where a slice has many: 1.4e-7, but 2 to 4 % of a prompt's time.)
template <int N> __device__ __forceinline__ void px_reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void px_reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// ---- the kernels: work units, tiles and slices as in pfmm.cuh.  Up to 128 prompt rows: ----
template <int FMT, int RU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(px1_threads(FMT, RU), 1) k_pfx1(const PfArgs a) {
  constexpr int NA = px_na(FMT), NB = px_nb(FMT), BS = px_slot_stages(RU), NPL = px_planes(FMT), N = 2 * RU, TB = tile_bytes(FMT), CH = px_chunk(FMT), NRAW = px_raws(FMT, RU), SS = px_sub(FMT);
  constexpr int RAWB = px_raw_bytes(FMT), AB = px_a_bytes(FMT), STB = SS * AB, SLB = px_slot_bytes(FMT, RU), PLB = px_b_bytes(RU), OPB = px_ob_bytes(RU), UW = px1_unpack(FMT, RU);
  static_assert(NRAW >= 2 && px_smem(FMT, RU) <= PX_SMEM_MAX, "a form that does not fit");
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t bar_s = smem_u32(smem);
  const uint32_t lead = t5_map_rank(bar_s, 0);     // the leader's (the pair's first CTA's) barriers, as both CTAs name them
  auto a_full = [&](int s) { return bar_s + 8u * (uint32_t)s; };               // leader: both CTAs' unpacking warps
  auto a_empty = [&](int s) { return bar_s + 32u + 8u * (uint32_t)s; };
  auto b_full = [&](int s) { return bar_s + 64u + 8u * (uint32_t)s; };         // leader: its own copy and the other CTA's, passed on from that one's b_here
  auto b_empty = [&](int s) { return bar_s + 96u + 8u * (uint32_t)s; };
  auto b_here = [&](int s) { return bar_s + 128u + 8u * (uint32_t)s; };
  auto d_full = [&](int b) { return bar_s + 160u + 8u * (uint32_t)b; };
  auto d_empty = [&](int b) { return bar_s + 176u + 8u * (uint32_t)b; };       // leader: the reading warps of both CTAs
  auto sc_full = [&](int i) { return bar_s + 192u + 8u * (uint32_t)i; };
  auto raw_full = [&](int i) { return bar_s + 224u + 8u * (uint32_t)i; };
  auto raw_empty = [&](int i) { return bar_s + 256u + 8u * (uint32_t)i; };
  uint32_t *tmem_slot = (uint32_t *)(smem + 320);
  volatile uint32_t *dead = (volatile uint32_t *)(smem + 324);
  float *scr = (float *)(smem + PX_HDR);
  uint8_t *oa = smem + PX_HDR + PX_SC, *ra = oa + (px_offs(FMT) ? PX_OA : 0), *rb = ra + NA * STB, *raw = rb + NB * SLB;
  const uint32_t oa_s = smem_u32(oa), ra_s = smem_u32(ra), rb_s = smem_u32(rb), raw_s = smem_u32(raw);
  const int ntiles = a.t128[a.nmat], npairs = (ntiles + 1) >> 1, nunits = npairs * a.ksplit;
  const int rank = blockIdx.x & 1, unit0 = blockIdx.x >> 1, ustep = gridDim.x >> 1;
  auto tile_of = [&](int u) { return 2 * (u % npairs) + rank; };

  pdl_trigger();
  if (tid == 0) {
    for (int s = 0; s < NA; s++) { mbar_init(a_full(s), 2 * UW); mbar_init(a_empty(s), 1); }
    for (int s = 0; s < NB; s++) { mbar_init(b_full(s), 2); mbar_init(b_empty(s), 1); mbar_init(b_here(s), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(d_full(b), 1); mbar_init(d_empty(b), 16); }
    for (int i = 0; i < 4; i++) mbar_init(sc_full(i), 4);
    for (int i = 0; i < NRAW; i++) { mbar_init(raw_full(i), 1); mbar_init(raw_empty(i), UW); }
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == UW + 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // both CTAs' barriers exist
  t5_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint32_t bar, uint32_t parity) {   // gives up for the whole CTA
    for (uint32_t n = 0; !mbar_wait(bar, parity, 4); n += 4) {
      if (*dead) return;
      if (n >= T5_WAIT_LIMIT) { *dead = 1; if (a.err) atomicExch(a.err, 1u); return; }
    }
  };

  if (warp < UW) {
    // ---- codes: two threads a weight row (with one the unpacking of a super-block took 3250 cycles and paced the kernel), or one ----
    px_reg_dec<PX1_REG_UNPACK>();
    const int r = tid & 127, part0 = tid >> 7, r16 = r & 15;
    const uint32_t roff = (uint32_t)(r >> 4) * (CH * TB);
    int slot = 0, rs = 0, jj = 0;
    uint32_t par = 1, rpar = 0;             // (the first round's waits on empty barriers pass)
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst;
      pf_slice(a, u, npairs, kbase, nst);
      const int nsl = nst >> 2;
#pragma unroll 1
      for (int c = 0; c < nsl; c++, jj++) {
        if (c % CH == 0) wait(raw_full(rs), rpar);
        const uint8_t *tile = raw + rs * RAWB + roff + c % CH * TB, *row = tile + r16 * tile_row(FMT);
        PxRow h;
        float scale;
        uint4 off[2];
        px_head<FMT>(row, tile, r16, part0 == 0, h, scale, off);
#pragma unroll 1
        for (int s = 0; s < 4; s += SS) {
          uint4 o[4 * NPL];
          px_stage<FMT, 2>(row, s, part0, h, o);
          wait(a_empty(slot), par);
          uint8_t *A = ra + slot * STB + r * 16;
#pragma unroll
          for (int i = 0; i < 4 * NPL; i++) *(uint4 *)(A + (i >> 2) * PF_A_BYTES + px_group<FMT, 2>(i & 3, part0) * 2048) = o[i];
          if constexpr (UW == 4) {
            px_stage<FMT, 2>(row, s, 1, h, o);
#pragma unroll
            for (int i = 0; i < 4 * NPL; i++) *(uint4 *)(A + (i >> 2) * PF_A_BYTES + px_group<FMT, 2>(i & 3, 1) * 2048) = o[i];
          }
          if constexpr (SS == 2) {
            px_stage<FMT, 2>(row, s + 1, part0, h, o);
#pragma unroll
            for (int i = 0; i < 4; i++) *(uint4 *)(A + AB + px_group<FMT, 2>(i, part0) * 2048) = o[i];
          }
          if (s == 0 && part0 == 0) {   // (the scales of the super-block four back have been read: its accumulators were, before the stages that were waited for here)
            scr[(jj & 3) * 128 + r] = scale;
            __syncwarp();
            if (lane == 0) mbar_arrive(sc_full(jj & 3));
          }
          if (s + SS == 4 && part0 == 0 && px_offs(FMT)) { *(uint4 *)(oa + r * 16) = off[0]; *(uint4 *)(oa + (128 + r) * 16) = off[1]; }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads these bytes through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(lead + (a_full(slot) - bar_s));
          if (++slot == NA) { slot = 0; par ^= 1u; }
        }
        if (c % CH == CH - 1 || c == nsl - 1) {
          if (lane == 0) mbar_arrive(raw_empty(rs));
          if (++rs == NRAW) { rs = 0; rpar ^= 1u; }
        }
      }
    }
  } else if (warp < UW + 4) {
    px_reg_dec<px1_reg_issue(FMT, RU)>();
    if (warp == UW) {
      // ---- weights: lane t requests the t-th 16-row tile of every chunk of the CTA's 128 rows ----
      int rs = 0;
      uint32_t rpar = 1;
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst, m, row0;
        pf_slice(a, u, npairs, kbase, nst);
        pf_locate(a, min(tile_of(u), ntiles - 1), m, row0);
        const int nsl = nst >> 2, nsb = a.K >> 8, have = min(8, ((a.m[m].rows + 15) >> 4) - (row0 >> 4));
        const uint8_t *src = a.m[m].W + ((size_t)((row0 >> 4) + min(lane, have - 1)) * nsb + (kbase >> 8)) * TB;
        for (int c = 0; c < nsl; c += CH) {
          const int n = min(CH, nsl - c);
          wait(raw_empty(rs), rpar);
          // (one answer for the warp: lanes that saw the word differently would leave bytes expected that nobody requests)
          if (!__any_sync(0xffffffffu, *dead != 0)) {
            if (lane == 0) mbar_expect(raw_full(rs), (uint32_t)(have * n * TB));
            __syncwarp();
            if (lane < have) bulk_load(raw_s + rs * RAWB + lane * (CH * TB), src + (size_t)c * TB, (uint32_t)(n * TB), raw_full(rs));
          }
          __syncwarp();
          if (++rs == NRAW) { rs = 0; rpar ^= 1u; }
        }
      }
    } else if (warp == UW + 1) {
      // ---- activations: the CTA's plane ----
      if (lane == 0) {
        int slot = 0;
        uint32_t par = 1;
        pdl_wait();
        const __half *x = a.x + (size_t)rank * a.K * RU, *xs = a.x + (size_t)2 * a.K * RU + (size_t)rank * pf_sum_halves(a.K, RU);
        for (int u = unit0; u < nunits; u += ustep) {
          int kbase, nst;
          pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
          for (int s = 0; s < nst; s += BS) {
            wait(b_empty(slot), par);
            if (!*dead) {
              const bool last = px_offs(FMT) && ((s + BS) & 3) == 0;
              const uint32_t bar = rank ? b_here(slot) : b_full(slot), dst = rb_s + slot * SLB;
              mbar_expect(bar, (uint32_t)(PX_SLOT + (last ? OPB : 0)));
              pf_bulk_copy(dst, x + (size_t)(kbase + s * PF_KS) * RU, PX_SLOT, bar);
              if (last) pf_bulk_copy(dst + PX_SLOT, xs + (size_t)((kbase >> 8) + (s >> 2)) * 16 * RU, OPB, bar);
            }
            if (++slot == NB) { slot = 0; par ^= 1u; }
          }
        }
      }
    } else if (warp == UW + 3) {
      // ---- tells the leader that the other CTA's activations are there ----
      if (lane == 0 && rank == 1) {
        int slot = 0;
        uint32_t par = 0;
        for (int u = unit0; u < nunits; u += ustep) {
          int kbase, nst;
          pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
          for (int s = 0; s < nst; s += BS) {
            wait(b_here(slot), par);
            mbar_arrive_cluster(lead + (b_full(slot) - bar_s));
            if (++slot == NB) { slot = 0; par ^= 1u; }
          }
        }
      }
    } else if (rank == 0) {
      // ---- the tensor cores of the pair, from the leader: the warp walks, an elected lane issues (descriptors stay in uniform registers) ----
      const bool el = t5_elect();
      const uint64_t oad = g3_desc(oa_s, 2048, 128);
      int as = 0, bs = 0, dd = 0;   // (dd: accumulators handed over)
      uint32_t apar = 0, bpar = 0;
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
        for (int s = 0; s < nst; s += SS, dd++) {
          const uint32_t D = tmem + (uint32_t)((dd & 1) * 256);
          if (dd > 1) wait(d_empty(dd & 1), (uint32_t)((dd >> 1) - 1) & 1u);
          wait(a_full(as), apar);
          const uint64_t ad = g3_desc(ra_s + as * STB, 2048, 128);
#pragma unroll
          for (int q = 0; q < SS; q++) {
            const int in = (s + q) % BS;          // part of the slot of activations
            if (in == 0) wait(b_full(bs), bpar);
            t5_fence_after();
            const uint64_t bd = g3_desc(rb_s + bs * SLB + in * PLB, RU * 16, 128);
            if (el) {
              // (two planes: the smaller one first, while there is little for the additions to truncate)
#pragma unroll
              for (int pl = NPL - 1; pl >= 0; pl--)
#pragma unroll
                for (int k = 0; k < 4; k++)
                  pf_mma_ss(D, ad + (uint64_t)(q * (AB / 16) + pl * (PF_A_BYTES / 16) + k * 256), bd + (uint64_t)(k * 2 * RU), px_idesc(N), k != 0 || pl != NPL - 1 || q != 0);
              if (q == SS - 1) {
                if (px_offs(FMT) && (s & 3) + SS == 4) pf_mma_ss(D, oad, g3_desc(rb_s + bs * SLB + PX_SLOT, RU * 16, 128), px_idesc(N), 1u);
                t5_commit_pair(a_empty(as));
                t5_commit_pair(d_full(dd & 1));
              }
              if (in == BS - 1) t5_commit_pair(b_empty(bs));
            }
            __syncwarp();
            if (in == BS - 1 && ++bs == NB) { bs = 0; bpar ^= 1u; }
          }
          if (++as == NA) { as = 0; apar ^= 1u; }
        }
      }
    }
  } else {
    // ---- accumulators into sums: lane quarter q, a weight row a thread; the two warps of a quarter have half of the prompt rows each ----
    px_reg_inc<px1_reg_read(FMT, RU)>();
    constexpr int RH = RU / 2;
    const int q = warp & 3, half = (warp - UW - 4) >> 2, R = a.R;
    const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(half * RH);
    f32x2 acc[RH / 2], sum[NPL == 2 ? RH / 2 : 1];
    const f32x2 inv = x2_pack(XP_LO_INV, XP_LO_INV);
    int jj = 0, dd = 0;
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst, m, row0;
      pf_slice(a, u, npairs, kbase, nst);
#pragma unroll
      for (int j = 0; j < RH / 2; j++) acc[j] = 0;
#pragma unroll 1
      for (int c = 0; c < nst >> 2; c++, jj++) {
        wait(sc_full(jj & 3), (uint32_t)(jj >> 2) & 1u);
        const float scf = scr[(jj & 3) * 128 + 32 * q + lane];
        const f32x2 sc = x2_pack(scf, scf);
        if constexpr (NPL == 2) {
#pragma unroll
          for (int j = 0; j < RH / 2; j++) sum[j] = 0;
        }
#pragma unroll 1
        for (int p = 0; p < 4 / SS; p++, dd++) {
          const uint32_t t1 = t0 + (uint32_t)((dd & 1) * 256);
          wait(d_full(dd & 1), (uint32_t)(dd >> 1) & 1u);
          t5_fence_after();
#pragma unroll
          for (int j0 = 0; j0 < RH; j0 += 16) {
            f32x2 v[8], w[8];
            t5_ld16x2(t1 + j0, v);
            t5_ld16x2(t1 + RU + j0, w);
            t5_wait_ld();
            if (j0 + 16 == RH) {   // given back before the last of it are added up
              t5_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(lead + (d_empty(dd & 1) - bar_s));
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const f32x2 x = x2_fma(w[j], inv, v[j]);
              if constexpr (NPL == 2) sum[j0 / 2 + j] = x2_add(sum[j0 / 2 + j], x);
              else acc[j0 / 2 + j] = x2_fma(sc, x, acc[j0 / 2 + j]);
            }
          }
        }
        if constexpr (NPL == 2) {
#pragma unroll
          for (int j = 0; j < RH / 2; j++) acc[j] = x2_fma(sc, sum[j], acc[j]);
        }
      }
      const int tile = tile_of(u);
      pf_locate(a, min(tile, ntiles - 1), m, row0);
      const int row = row0 + 32 * q + lane, n = R - half * RH;   // this warp's prompt rows in use
      if (tile < ntiles && row < a.m[m].rows) {
        const size_t os = a.m[m].ostride;
        float *out = a.m[m].out + (size_t)(u / npairs) * a.m[m].split_stride + (size_t)(half * RH) * os + row;
#pragma unroll
        for (int j = 0; j < RH; j += 2) {
          float y0, y1;
          x2_unpack(acc[j / 2], y0, y1);
          if (NPL == 2) { y0 = fmaf(y0, PX_LOST, y0); y1 = fmaf(y1, PX_LOST, y1); }
          if (j < n) *out = y0;
          out += os;
          if (j + 1 < n) *out = y1;
          out += os;
        }
      }
    }
  }
  // after a wait ran out nothing is requested any more, but copies may be on their way into this CTA's rings
  if (*dead) for (int i = 0; i < 64; i++) __nanosleep(1000);
  __syncwarp();
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // no CTA leaves while the other still arrives here or reads its memory
  if (warp == UW + 2) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- up to 32 prompt rows: the codes as the MMAs' operand in TENSOR MEMORY ----
// Two groups of four unpacking warps, a thread a weight row, take the super-blocks in turn, each with an issuing warp and accumulators of its own:
// what one group waits for the other fills.  An ITEM is what 64 columns of tensor memory hold, 128 columns of one plane of codes or 64 of two; a
// group has two such buffers and two accumulators, so that it unpacks one item while the other is multiplied, and multiplies one while the other
// is read.  Sums are added in the columns' order, as k_pfx1 adds them: the same bits.  What bounds it is a group's chain, 4000 cycles a super-block, of
// which unpacking is half.  Twenty rows, k_pfx1 with 32 / this: Q4_K 34816 x 5120 59.5 / 44 us, 5120 x 6144 17.8 / 15, Q6_K 5120 x 17408 (planes of bits) 56 / 43,
// Q8_0 24576 x 4096 61 / 47, Q5_K 8192 x 4096 19 / 17.  With 64 rows only one accumulator a group fits: Q4_K 70 / 63, Q6_K 65 / 73, Q8_0 70 / 80, not kept.
// A barrier is only ever waited for by one group, which sees every phase of it (a phase's parity tells nothing to one that missed the phase before).
__host__ __device__ constexpr int pt_items(int fmt) { return 2 * px_planes(fmt); }       // of a super-block
__host__ __device__ constexpr int pt_fixed(int fmt) { return PX_HDR + 2 * PX_SC + (px_offs(fmt) ? 2 * PX_OA : 0) + PT_NB * px_slot_bytes(fmt, PT_RU); }
__host__ __device__ constexpr int pt_raws(int fmt) {
  const int n = (PX_SMEM_MAX - pt_fixed(fmt)) / px_raw_bytes(fmt);
  return n > 4 ? 4 : n;
}
__host__ __device__ constexpr int pt_smem(int fmt) { return pt_fixed(fmt) + pt_raws(fmt) * px_raw_bytes(fmt); }
__device__ __forceinline__ void pt_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
template <int FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PT_THREADS, 1) k_pft(const PfArgs a) {
  constexpr int RU = PT_RU, NB = PT_NB, SPB = 4 / px_slot_stages(RU), NPL = px_planes(FMT), NP = pt_items(FMT), SI = 4 / NP, N = 2 * RU, TB = tile_bytes(FMT), CH = px_chunk(FMT), NRAW = pt_raws(FMT);
  constexpr int RAWB = px_raw_bytes(FMT), SLB = px_slot_bytes(FMT, RU), PLB = px_b_bytes(RU), OPB = px_ob_bytes(RU), ND = 128 / N;   // SPB: slots of activations a super-block (SI: 64-column parts an item); ND: accumulators a group
  static_assert(NRAW >= 2 && pt_smem(FMT) <= PX_SMEM_MAX && NB % (2 * SPB) == 0 && ND >= 1, "a form that does not fit");
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t bar_s = smem_u32(smem), lead = t5_map_rank(bar_s, 0);   // the leader's (the pair's first CTA's) barriers, as both CTAs name them
  auto a_full = [&](int i) { return bar_s + 8u * (uint32_t)i; };               // [group][buffer]; leader: both CTAs' unpacking warps of the group
  auto a_empty = [&](int i) { return bar_s + 32u + 8u * (uint32_t)i; };
  auto b_full = [&](int s) { return bar_s + 64u + 8u * (uint32_t)s; };         // leader: its own copy and the other CTA's, passed on from that one's b_here
  auto b_empty = [&](int s) { return bar_s + 96u + 8u * (uint32_t)s; };
  auto b_here = [&](int s) { return bar_s + 128u + 8u * (uint32_t)s; };
  auto d_full = [&](int i) { return bar_s + 160u + 8u * (uint32_t)i; };        // [group][accumulator]
  auto d_empty = [&](int i) { return bar_s + 192u + 8u * (uint32_t)i; };       // leader: the reading warps of both CTAs
  auto sc_full = [&](int i) { return bar_s + 224u + 8u * (uint32_t)i; };
  auto raw_full = [&](int i) { return bar_s + 256u + 8u * (uint32_t)i; };
  auto raw_empty = [&](int i) { return bar_s + 288u + 8u * (uint32_t)i; };
  uint32_t *tmem_slot = (uint32_t *)(smem + 320);
  volatile uint32_t *dead = (volatile uint32_t *)(smem + 324);
  float *scr = (float *)(smem + PX_HDR);
  uint8_t *oa = smem + PX_HDR + 2 * PX_SC, *rb = oa + (px_offs(FMT) ? 2 * PX_OA : 0), *raw = rb + NB * SLB;
  const uint32_t oa_s = smem_u32(oa), rb_s = smem_u32(rb), raw_s = smem_u32(raw);
  const int ntiles = a.t128[a.nmat], npairs = (ntiles + 1) >> 1, nunits = npairs * a.ksplit;
  const int rank = blockIdx.x & 1, unit0 = blockIdx.x >> 1, ustep = gridDim.x >> 1;
  auto tile_of = [&](int u) { return 2 * (u % npairs) + rank; };

  pdl_trigger();
  if (tid == 0) {
    for (int i = 0; i < 4; i++) { mbar_init(a_full(i), 8); mbar_init(a_empty(i), 1); mbar_init(d_full(i), 1); mbar_init(d_empty(i), 16); mbar_init(sc_full(i), 4); }
    for (int s = 0; s < NB; s++) { mbar_init(b_full(s), 2); mbar_init(b_empty(s), 1); mbar_init(b_here(s), 1); }
    for (int i = 0; i < NRAW; i++) { mbar_init(raw_full(i), 1); mbar_init(raw_empty(i), 8); }
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 10) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // both CTAs' barriers exist
  t5_fence_after();
  const uint32_t tmem = *tmem_slot;                    // codes: 64 columns a buffer, [group][buffer]; behind them the accumulators, 128 columns a group
  auto wait = [&](uint32_t bar, uint32_t parity) {   // gives up for the whole CTA
    for (uint32_t n = 0; !mbar_wait(bar, parity, 4); n += 4) {
      if (*dead) return;
      if (n >= T5_WAIT_LIMIT) { *dead = 1; if (a.err) atomicExch(a.err, 1u); return; }
    }
  };

  if (warp < 8) {
    // ---- codes: group g, a thread a weight row ----
    const int g = warp >> 2, r = tid & 127, r16 = r & 15;
    const uint32_t abuf = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(128 * g);
    const uint32_t roff = (uint32_t)(r >> 4) * (CH * TB);
    int rs = 0, jj = 0, it = 0;             // super-blocks of the CTA, items of the group so far
    uint32_t rpar = 0;
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst;
      pf_slice(a, u, npairs, kbase, nst);
      const int nsl = nst >> 2;
#pragma unroll 1
      for (int c = 0; c < nsl; c++, jj++) {
        if (c % CH == 0) wait(raw_full(rs), rpar);     // (by both groups, whichever has the super-block)
        if ((jj & 1) == g) {
          const uint8_t *tile = raw + rs * RAWB + roff + c % CH * TB, *row = tile + r16 * tile_row(FMT);
          PxRow h;
          float scale;
          uint4 off[2];
          px_head<FMT>(row, tile, r16, true, h, scale, off);
#pragma unroll 1
          for (int p = 0; p < NP; p++, it++) {
            uint4 o[8 * NPL];
            px_stage<FMT>(row, p * SI, 0, h, o);
            wait(a_empty(2 * g + (it & 1)), (uint32_t)((it >> 1) & 1) ^ 1u);     // (the first round passes)
            t5_fence_after();
            const uint32_t A = abuf + 64u * (uint32_t)(it & 1);
            auto put = [&](uint32_t at, const uint4 *q) {
              const uint32_t v[32] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w, q[2].x, q[2].y, q[2].z, q[2].w, q[3].x, q[3].y, q[3].z, q[3].w,
                                      q[4].x, q[4].y, q[4].z, q[4].w, q[5].x, q[5].y, q[5].z, q[5].w, q[6].x, q[6].y, q[6].z, q[6].w, q[7].x, q[7].y, q[7].z, q[7].w};
              t5_st32(at, v);
            };
            put(A, o);
            if constexpr (NPL == 2) put(A + 32, o + 8);
            else {
              px_stage<FMT>(row, p * SI + 1, 0, h, o);
              put(A + 32, o);
            }
            if (p == 0) {   // (the scales of the super-block eight back: with the group's buffer free again, the one four back is being read at the earliest)
              scr[(jj & 7) * 128 + r] = scale;
              __syncwarp();
              if (lane == 0) mbar_arrive(sc_full(jj & 3));
            }
            if (p == NP - 1 && px_offs(FMT)) {
              uint8_t *O = oa + g * PX_OA + r * 16;
              *(uint4 *)O = off[0]; *(uint4 *)(O + 2048) = off[1];
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads these bytes through the async proxy
            }
            t5_wait_st();
            t5_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead + (a_full(2 * g + (it & 1)) - bar_s));
          }
        }
        if (c % CH == CH - 1 || c == nsl - 1) {
          __syncwarp();
          if (lane == 0) mbar_arrive(raw_empty(rs));
          if (++rs == NRAW) { rs = 0; rpar ^= 1u; }
        }
      }
    }
  } else if (warp == 8) {
    // ---- weights: lane t requests the t-th 16-row tile of every chunk of the CTA's 128 rows ----
    int rs = 0;
    uint32_t rpar = 1;
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst, m, row0;
      pf_slice(a, u, npairs, kbase, nst);
      pf_locate(a, min(tile_of(u), ntiles - 1), m, row0);
      const int nsl = nst >> 2, nsb = a.K >> 8, have = min(8, ((a.m[m].rows + 15) >> 4) - (row0 >> 4));
      const uint8_t *src = a.m[m].W + ((size_t)((row0 >> 4) + min(lane, have - 1)) * nsb + (kbase >> 8)) * TB;
#pragma unroll 1
      for (int c = 0; c < nsl; c += CH) {
        const int n = min(CH, nsl - c);
        wait(raw_empty(rs), rpar);
        // (one answer for the warp: lanes that saw the word differently would leave bytes expected that nobody requests)
        if (!__any_sync(0xffffffffu, *dead != 0)) {
          if (lane == 0) mbar_expect(raw_full(rs), (uint32_t)(have * n * TB));
          __syncwarp();
          if (lane < have) bulk_load(raw_s + rs * RAWB + lane * (CH * TB), src + (size_t)c * TB, (uint32_t)(n * TB), raw_full(rs));
        }
        __syncwarp();
        if (++rs == NRAW) { rs = 0; rpar ^= 1u; }
      }
    }
  } else if (warp == 9) {
    // ---- activations: the CTA's plane; the other CTA's warp then tells the leader that they are there ----
    if (lane == 0) {
      int slot = 0;
      uint32_t par = 1;
      pdl_wait();
      const __half *x = a.x + (size_t)rank * a.K * RU, *xs = a.x + (size_t)2 * a.K * RU + (size_t)rank * pf_sum_halves(a.K, RU);
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
        for (int i = 0; i < (nst >> 2) * SPB; i++) {
          wait(b_empty(slot), par);
          if (!*dead) {
            const bool last = px_offs(FMT) && i % SPB == SPB - 1;
            const uint32_t bar = rank ? b_here(slot) : b_full(slot), dst = rb_s + slot * SLB;
            mbar_expect(bar, (uint32_t)(PX_SLOT + (last ? OPB : 0)));
            pf_bulk_copy(dst, x + (size_t)kbase * RU + (size_t)i * (PX_SLOT / 2), PX_SLOT, bar);
            if (last) pf_bulk_copy(dst + PX_SLOT, xs + (size_t)((kbase >> 8) + i / SPB) * 16 * RU, OPB, bar);
          }
          if (++slot == NB) { slot = 0; par ^= 1u; }
        }
      }
    }
  } else if (warp < 12) {
    if (rank == 1) {
      if (warp == 11 && lane == 0) {
        int slot = 0;
        uint32_t par = 0;
        for (int u = unit0; u < nunits; u += ustep) {
          int kbase, nst;
          pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
          for (int i = 0; i < (nst >> 2) * SPB; i++) {
            wait(b_here(slot), par);
            mbar_arrive_cluster(lead + (b_full(slot) - bar_s));
            if (++slot == NB) { slot = 0; par ^= 1u; }
          }
        }
      }
    } else {
      // ---- the tensor cores of the pair, from the leader: a warp a group; the whole warp walks, an elected lane issues ----
      const int g = __shfl_sync(0xffffffffu, warp - 10, 0);
      const bool el = t5_elect();
      const uint64_t oad = g3_desc(oa_s + g * PX_OA, 2048, 128);
      const uint32_t ab = tmem + (uint32_t)(128 * g), db = tmem + 256u + (uint32_t)(128 * g);
      int jj = 0, it = 0;
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
        for (int c = 0; c < nst >> 2; c++, jj++) {
          if ((jj & 1) != g) continue;
#pragma unroll 1
          for (int p = 0; p < NP; p++, it++) {
            const int buf = 2 * g + (it & 1), di = it % ND, dbar = 2 * g + di;
            const uint32_t D = db + (uint32_t)(di * N), A = ab + 64u * (uint32_t)(it & 1);
            const int sl = (jj * SPB + p * SPB / NP) % NB, in = p * SI - (p * SPB / NP) * (4 / SPB);   // the item's slot of activations, its first 64-column part there
            if (it >= ND) wait(d_empty(dbar), (uint32_t)((it / ND) - 1) & 1u);
            if (in == 0) wait(b_full(sl), (uint32_t)(jj * SPB / NB) & 1u);
            wait(a_full(buf), (uint32_t)(it >> 1) & 1u);
            t5_fence_after();
            const uint64_t bd = g3_desc(rb_s + sl * SLB + in * PLB, RU * 16, 128);
            if (el) {
              // (two planes: the smaller one first, while there is little for the additions to truncate)
#pragma unroll
              for (int pl = NPL - 1; pl >= 0; pl--)
#pragma unroll
                for (int k = 0; k < 4 * SI; k++)
                  pt_mma(D, A + (uint32_t)(32 * pl + 8 * k), bd + (uint64_t)(k / 4 * (PLB / 16) + k % 4 * 2 * RU), px_idesc(N), k != 0 || pl != NPL - 1);
              if (px_offs(FMT) && p == NP - 1) pf_mma_ss(D, oad, g3_desc(rb_s + sl * SLB + PX_SLOT, RU * 16, 128), px_idesc(N), 1u);
              t5_commit_pair(a_empty(buf));
              if (in + SI == 4 / SPB) t5_commit_pair(b_empty(sl));
              t5_commit_pair(d_full(dbar));
            }
            __syncwarp();
          }
        }
      }
    }
  } else {
    // ---- accumulators into sums: lane quarter q, a weight row a thread; the two warps of a quarter have half of the prompt rows each ----
    constexpr int RH = RU / 2;
    const int q = warp & 3, half = (warp - 12) >> 2, R = a.R;
    const uint32_t t0 = tmem + 256u + ((uint32_t)(32 * q) << 16) + (uint32_t)(half * RH);
    f32x2 acc[RH / 2], sum[NPL == 2 ? RH / 2 : 1];
    const f32x2 inv = x2_pack(XP_LO_INV, XP_LO_INV);
    int j0 = 0;
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst, m, row0;
      pf_slice(a, u, npairs, kbase, nst);
      const int nsl = nst >> 2;
#pragma unroll
      for (int j = 0; j < RH / 2; j++) acc[j] = 0;
#pragma unroll 1
      for (int c = 0; c < nsl; c++) {
        const int jj = j0 + c, g = jj & 1;
        wait(sc_full(jj & 3), (uint32_t)(jj >> 2) & 1u);
        const float scf = scr[(jj & 7) * 128 + 32 * q + lane];
        const f32x2 sc = x2_pack(scf, scf);
        if constexpr (NPL == 2) {
#pragma unroll
          for (int j = 0; j < RH / 2; j++) sum[j] = 0;
        }
#pragma unroll (NPL == 2 ? NP : 1)   // (not unrolled, the sums of two planes cost 20 rows of the 9B shape 6 %)
        for (int p = 0; p < NP; p++) {   // in the columns' order, as k_pfx1 adds them
          const int it = (jj >> 1) * NP + p, di = it % ND, dbar = 2 * g + di;
          const uint32_t t1 = t0 + (uint32_t)(128 * g + di * N);
          wait(d_full(dbar), (uint32_t)(it / ND) & 1u);
          t5_fence_after();
#pragma unroll
          for (int i0 = 0; i0 < RH; i0 += 16) {
            f32x2 v[8], w[8];
            t5_ld16x2(t1 + i0, v);
            t5_ld16x2(t1 + RU + i0, w);
            t5_wait_ld();
            if (i0 + 16 == RH) {   // given back before the last of it are added up
              t5_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive_cluster(lead + (d_empty(dbar) - bar_s));
            }
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const f32x2 x = x2_fma(w[j], inv, v[j]);
              if constexpr (NPL == 2) sum[i0 / 2 + j] = x2_add(sum[i0 / 2 + j], x);
              else acc[i0 / 2 + j] = x2_fma(sc, x, acc[i0 / 2 + j]);
            }
          }
        }
        if constexpr (NPL == 2) {
#pragma unroll
          for (int j = 0; j < RH / 2; j++) acc[j] = x2_fma(sc, sum[j], acc[j]);
        }
      }
      j0 += nsl;
      const int tile = tile_of(u);
      pf_locate(a, min(tile, ntiles - 1), m, row0);
      const int row = row0 + 32 * q + lane, n = R - half * RH;   // this warp's prompt rows in use
      if (tile < ntiles && row < a.m[m].rows) {
        const size_t os = a.m[m].ostride;
        float *out = a.m[m].out + (size_t)(u / npairs) * a.m[m].split_stride + (size_t)(half * RH) * os + row;
#pragma unroll
        for (int j = 0; j < RH; j += 2) {
          float y0, y1;
          x2_unpack(acc[j / 2], y0, y1);
          if (NPL == 2) { y0 = fmaf(y0, PX_LOST, y0); y1 = fmaf(y1, PX_LOST, y1); }
          if (j < n) *out = y0;
          out += os;
          if (j + 1 < n) *out = y1;
          out += os;
        }
      }
    }
  }
  // after a wait ran out nothing is requested any more, but copies may be on their way into this CTA's rings
  if (*dead) for (int i = 0; i < 64; i++) __nanosleep(1000);
  __syncwarp();
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // no CTA leaves while the other still arrives here or reads its memory
  if (warp == 10) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- more than 128 prompt rows: Q4_K and Q5_K ----
template <int FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PX_THREADS, 1) k_pfx2(const PfArgs a) {
  static_assert(px_planes(FMT) == 1 && PX2_NB == 4, "one plane of codes, its four stages once round the ring");
  constexpr int TB = tile_bytes(FMT), OPB = px_ob_bytes(PF_R), N = PF_RMAX, RH = 128;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t bar_s = smem_u32(smem), lead = t5_map_rank(bar_s, 0);   // the leader's barriers, as both CTAs name them
  auto a_full = [&](int i) { return bar_s + 8u * (uint32_t)i; };          // leader: both CTAs' unpacking warps
  auto a_empty = [&](int i) { return bar_s + 64u + 8u * (uint32_t)i; };
  auto b_full = [&](int i) { return bar_s + 128u + 8u * (uint32_t)i; };   // leader: its own copy and the other CTA's, passed on from that one's b_here
  auto b_empty = [&](int i) { return bar_s + 160u + 8u * (uint32_t)i; };
  auto b_here = [&](int i) { return bar_s + 192u + 8u * (uint32_t)i; };
  auto d_full = [&](int b) { return bar_s + 224u + 8u * (uint32_t)b; };
  auto d_empty = [&](int b) { return bar_s + 240u + 8u * (uint32_t)b; };  // leader: the reading warps of both CTAs
  auto sc_full = [&](int i) { return bar_s + 256u + 8u * (uint32_t)i; };
  auto raw_full = [&](int i) { return bar_s + 288u + 8u * (uint32_t)i; };
  auto raw_empty = [&](int i) { return bar_s + 304u + 8u * (uint32_t)i; };
  uint32_t *tmem_slot = (uint32_t *)(smem + 320);
  volatile uint32_t *dead = (volatile uint32_t *)(smem + 324);
  float *scr = (float *)(smem + PX_HDR);
  uint8_t *oa = smem + PX_HDR + PX_SC, *ob = oa + 2 * PX_OA, *ra = ob + 2 * OPB, *rb = ra + PX2_NA * PF_A_BYTES, *raw = rb + PX2_NB * PF_B_BYTES;   // ob: lo, hi
  const uint32_t oa_s = smem_u32(oa), ob_s = smem_u32(ob), ra_s = smem_u32(ra), rb_s = smem_u32(rb), raw_s = smem_u32(raw);
  const int ntiles = a.t128[a.nmat], npairs = (ntiles + 1) >> 1, nunits = npairs * a.ksplit;
  const int rank = blockIdx.x & 1, unit0 = blockIdx.x >> 1, ustep = gridDim.x >> 1;
  auto tile_of = [&](int u) { return 2 * (u % npairs) + rank; };
  // pairs start at different super-blocks of a slice: all of them reading the same activations at the same time is what L2 is slow at
  auto turned = [&](int c, int nsl) { c += unit0 * nsl / ustep; return c < nsl ? c : c - nsl; };

  pdl_trigger();
  if (tid == 0) {
    for (int i = 0; i < PX2_NA; i++) { mbar_init(a_full(i), 8); mbar_init(a_empty(i), 1); }
    for (int i = 0; i < PX2_NB; i++) { mbar_init(b_full(i), 2); mbar_init(b_empty(i), 1); mbar_init(b_here(i), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(d_full(b), 1); mbar_init(d_empty(b), 16); }
    for (int i = 0; i < 4; i++) mbar_init(sc_full(i), 4);
    for (int i = 0; i < PX2_NRAW; i++) { mbar_init(raw_full(i), 1); mbar_init(raw_empty(i), 4); }
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 6) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // both CTAs' barriers exist
  t5_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint32_t bar, uint32_t parity) {   // gives up for the whole CTA
    for (uint32_t n = 0; !mbar_wait(bar, parity, 4); n += 4) {
      if (*dead) return;
      if (n >= T5_WAIT_LIMIT) { *dead = 1; if (a.err) atomicExch(a.err, 1u); return; }
    }
  };

  if (warp < 4) {
    // ---- codes: a thread a weight row ----
    px_reg_dec<PX_REG_UNPACK>();
    const int r = tid, r16 = r & 15;
    int slot = 0, rs = 0, jj = 0;
    uint32_t par = 1, rpar = 0;             // (the first round's waits on empty barriers pass)
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst;
      pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
      for (int c = 0; c < nst >> 2; c++, jj++) {
        wait(raw_full(rs), rpar);
        const uint8_t *tile = raw + rs * (8 * TB) + (r >> 4) * TB, *row = tile + r16 * tile_row(FMT);
        PxRow h;
        float scale;
        uint4 off[2];
        px_head<FMT>(row, tile, r16, true, h, scale, off);
#pragma unroll 1
        for (int s = 0; s < 4; s++) {
          uint4 o[8];
          px_stage<FMT>(row, s, 0, h, o);
          wait(a_empty(slot), par);
          uint8_t *A = ra + slot * PF_A_BYTES + r * 16;
#pragma unroll
          for (int g = 0; g < 8; g++) *(uint4 *)(A + (size_t)g * 2048) = o[g];
          // what the super-blocks two and four back left here has been used: slots that were waited for hold stages of the one before this
          if (s == 0) {
            scr[(jj & 3) * 128 + r] = scale;
            __syncwarp();
            if (lane == 0) mbar_arrive(sc_full(jj & 3));
          }
          if (s == 3) { uint8_t *O = oa + (jj & 1) * PX_OA + r * 16; *(uint4 *)O = off[0]; *(uint4 *)(O + 2048) = off[1]; }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads these bytes through the async proxy
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(lead + (a_full(slot) - bar_s));
          if (++slot == PX2_NA) { slot = 0; par ^= 1u; }
        }
        if (lane == 0) mbar_arrive(raw_empty(rs));
        if (++rs == PX2_NRAW) { rs = 0; rpar ^= 1u; }
      }
    }
  } else if (warp < 8) {
    px_reg_dec<PX_REG_ISSUE>();
    if (warp == 4) {
      // ---- weights: lane t requests the t-th 16-row tile of a super-block of the CTA's 128 rows ----
      int rs = 0;
      uint32_t rpar = 1;
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst, m, row0;
        pf_slice(a, u, npairs, kbase, nst);
        pf_locate(a, min(tile_of(u), ntiles - 1), m, row0);
        const int nsb = a.K >> 8, have = min(8, ((a.m[m].rows + 15) >> 4) - (row0 >> 4));
        const uint8_t *src = a.m[m].W + ((size_t)((row0 >> 4) + min(lane, have - 1)) * nsb + (kbase >> 8)) * TB;
        const int rot = turned(0, nst >> 2);
        for (int c = 0; c < nst >> 2; c++) {
          wait(raw_empty(rs), rpar);
          const int sb = c + rot < nst >> 2 ? c + rot : c + rot - (nst >> 2);
          // (one answer for the warp: lanes that saw the word differently would leave bytes expected that nobody requests)
          if (!__any_sync(0xffffffffu, *dead != 0)) {
            if (lane == 0) mbar_expect(raw_full(rs), (uint32_t)(have * TB));
            __syncwarp();
            if (lane < have) bulk_load(raw_s + rs * (8 * TB) + lane * TB, src + (size_t)sb * TB, TB, raw_full(rs));
          }
          __syncwarp();
          if (++rs == PX2_NRAW) { rs = 0; rpar ^= 1u; }
        }
      }
    } else if (warp == 5) {
      // ---- activations of the CTA's unit: a super-block's four stages of the lo plane, then of the hi plane ----
      if (lane == 0) {
        pdl_wait();
        // (this loop's own length is part of a stage's way round: addresses are counted on, not made anew)
        const size_t lo = (size_t)a.K * PF_R, sum = pf_sum_halves(a.K, PF_R);
        const __half *x = a.x + (size_t)rank * pf_kg_halves(a.K, PF_R), *xs = x + 2 * lo;
        const uint32_t mine = rank ? b_here(0) : b_full(0);
        for (int u = unit0; u < nunits; u += ustep) {
          int kbase, nst;
          pf_slice(a, u, npairs, kbase, nst);
          const int nsl = nst >> 2;
          int c = turned(0, nsl);
#pragma unroll 1
          for (int i = 0; i < nsl; i++) {
            const __half *xc = x + (size_t)(kbase + c * 256) * PF_R, *sc = xs + (size_t)((kbase >> 8) + c) * 16 * PF_R;
#pragma unroll 1
            for (int i = 0; i < 8; i++) {
              const int s = i & 3;
              wait(b_empty(s), (uint32_t)(i >> 2) ^ 1u);
              if (!*dead) {
                mbar_expect(mine + 8 * s, (uint32_t)(PF_B_BYTES + (s == 3 ? OPB : 0)));
                pf_bulk_copy(rb_s + s * PF_B_BYTES, xc + (i < 4 ? lo : 0) + s * (PF_KS * PF_R), PF_B_BYTES, mine + 8 * s);
                if (s == 3) pf_bulk_copy(ob_s + (i >> 2) * OPB, sc + (i < 4 ? sum : 0), OPB, mine + 8 * s);
              }
            }
            if (++c == nsl) c = 0;
          }
        }
      }
    } else if (warp == 7) {
      // ---- tells the leader that the other CTA's activations are there ----
      if (lane == 0 && rank == 1) {
        for (int u = unit0; u < nunits; u += ustep) {
          int kbase, nst;
          pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
          for (int s = 0; s < 2 * nst; s++) {
            wait(b_here(s & 3), (uint32_t)(s >> 2) & 1u);
            mbar_arrive_cluster(lead + (b_full(s & 3) - bar_s));
          }
        }
      }
    } else if (rank == 0) {
      // ---- the tensor cores of the pair, from the leader: the warp walks, an elected lane issues (descriptors stay in uniform registers) ----
      const bool el = t5_elect();
      const uint64_t obd = g3_desc(ob_s, 2048, 128);
      int as0 = 0, jj = 0;
      uint32_t apar0 = 0;
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
#pragma unroll 1
        for (int c = 0; c < nst >> 2; c++, jj++) {
          const uint32_t D = tmem + (uint32_t)((jj & 1) * 256);
          const uint64_t oad = g3_desc(oa_s + (jj & 1) * PX_OA, 2048, 128);
          if (jj > 1) wait(d_empty(jj & 1), (uint32_t)((jj >> 1) - 1) & 1u);
#pragma unroll 1
          for (int i = 0; i < 8; i++) {     // (eight stages of activations: twice round their ring)
            const int s = i & 3;
            int as = as0 + s;
            uint32_t ap = apar0;
            if (as >= PX2_NA) { as -= PX2_NA; ap ^= 1u; }
            if (i < 4) wait(a_full(as), ap);
            wait(b_full(s), (uint32_t)(i >> 2));
            t5_fence_after();
            const uint64_t ad = g3_desc(ra_s + as * PF_A_BYTES, 2048, 128), bd = g3_desc(rb_s + s * PF_B_BYTES, 2048, 128);
            if (el) {
              if (i == 4) px_mma_scaled(D, ad, bd, px_idesc(N));
              else pf_mma_ss(D, ad, bd, px_idesc(N), i != 0);
#pragma unroll
              for (int k = 1; k < 4; k++) pf_mma_ss(D, ad + (uint64_t)(k * 256), bd + (uint64_t)(k * 256), px_idesc(N), 1u);
              if (s == 3) pf_mma_ss(D, oad, obd + (uint64_t)((i >> 2) * (OPB / 16)), px_idesc(N), 1u);
              t5_commit_pair(b_empty(s));
              if (i >= 4) t5_commit_pair(a_empty(as));
              if (i == 7) t5_commit_pair(d_full(jj & 1));
            }
            __syncwarp();
          }
          as0 += 4;
          if (as0 >= PX2_NA) { as0 -= PX2_NA; apar0 ^= 1u; }
        }
      }
    }
  } else {
    // ---- accumulators into sums: lane quarter q, a weight row a thread; the two warps of a quarter have a unit each ----
    px_reg_inc<PX_REG_READ>();
    const int q = warp & 3, half = (warp - 8) >> 2, R = a.R;
    const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(half * RH);
    f32x2 acc[RH / 2];
    int jj = 0;
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst, m, row0;
      pf_slice(a, u, npairs, kbase, nst);
#pragma unroll
      for (int j = 0; j < RH / 2; j++) acc[j] = 0;
#pragma unroll 1
      for (int c = 0; c < nst >> 2; c++, jj++) {
        wait(sc_full(jj & 3), (uint32_t)(jj >> 2) & 1u);
        const float scf = scr[(jj & 3) * 128 + 32 * q + lane];
        const f32x2 sc = x2_pack(scf, scf);
        const uint32_t t1 = t0 + (uint32_t)((jj & 1) * 256);
        wait(d_full(jj & 1), (uint32_t)(jj >> 1) & 1u);
        t5_fence_after();
#pragma unroll
        for (int j0 = 0; j0 < RH; j0 += 32) {
          f32x2 v[8], w[8];
          t5_ld16x2(t1 + j0, v);
          t5_ld16x2(t1 + j0 + 16, w);
          t5_wait_ld();
          if (j0 + 32 == RH) {
            t5_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead + (d_empty(jj & 1) - bar_s));
          }
#pragma unroll
          for (int j = 0; j < 8; j++) { acc[j0 / 2 + j] = x2_fma(sc, v[j], acc[j0 / 2 + j]); acc[j0 / 2 + 8 + j] = x2_fma(sc, w[j], acc[j0 / 2 + 8 + j]); }
        }
      }
      const int tile = tile_of(u);
      pf_locate(a, min(tile, ntiles - 1), m, row0);
      const int row = row0 + 32 * q + lane, n = R - half * RH;   // this warp's prompt rows in use
      if (tile < ntiles && row < a.m[m].rows) {
        const size_t os = a.m[m].ostride;
        float *out = a.m[m].out + (size_t)(u / npairs) * a.m[m].split_stride + (size_t)(half * RH) * os + row;
#pragma unroll
        for (int j = 0; j < RH; j += 2) {
          float y0, y1;
          x2_unpack(acc[j / 2], y0, y1);
          if (j < n) *out = y0;
          out += os;
          if (j + 1 < n) *out = y1;
          out += os;
        }
      }
    }
  }
  // after a wait ran out nothing is requested any more, but copies may be on their way into this CTA's rings
  if (*dead) for (int i = 0; i < 64; i++) __nanosleep(1000);
  __syncwarp();
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // no CTA leaves while the other still arrives here or reads its memory
  if (warp == 6) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}
