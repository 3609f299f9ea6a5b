// pfatt.cuh -- attention of a prompt piece's rows over the KV cache on tcgen05 (full_attn of the CPU engine, tools/qwen35_engine.c:667-726;
// the passes of a few rows have attention.cu).  A block has 128 queries of one kv head -- query r G + g is row r of the piece, head g of the
// kv head's G -- and one slice of the positions, 32 at a time:
//   scores  S[q][pos] = Q_hi K_hi + (Q_lo K_hi + Q_hi K_lo) / 2048      M = 128, N = 32; A: Q_hi in tensor memory, Q_lo in shared memory
//   softmax online per query, a thread a query; P as two fp16 planes into tensor memory
//   output  O[q][d]   = (P_hi + P_lo) V_hi + P_hi V_lo / 2048           N = head dimension; A: P in tensor memory
// The small products come first and are divided by 2048 by the first MMA on top of them (its scaling of D).  O starts anew with every 32
// positions and is added to fp32 registers, where a query's earlier sum takes the factor of its new maximum: the tensor core truncates
// where it adds, so that one accumulator over a slice would lose 2e-8 of itself an MMA.
// K comes as it lies in the cache (K-major), V likewise, which is MN-major for the second product: both by TMA in rows of 128 swizzled
// bytes, without a transposition.  (By cp.async of two warps a tile took 5300 cycles, the loads' issue; by TMA 3300.)
//
// Warps: 0-3 softmax, 4 loads K and V, 6 issues the MMAs, 8-15 read O.  A tile's scores are a tile ahead of its softmax, so the tensor core
// has S(i + 2) to do while the registers take O(i).  Per (query, slice) a maximum, a sum and an unnormalised row of O for k_pf_attn_comb.
//
// What bounds it is the MMAs of 32 positions, 16 x 41 + 32 x 21 + 6 x 129 = 2100 cycles of about 2800 a tile at head dimension 256: an operand
// A from shared memory costs 32 cycles an MMA however few columns there are (both of Q's planes there: 3300 a tile), and there is no room
// for more than 32 positions a slot, nor in tensor memory for Q_lo.  256 rows of the 27B shape (24 heads of 256, 4 kv heads), the merge with
// it: 245 -> 47 us behind 1280 positions, 1062 -> 154 behind 8000; 128 rows from the start 36 -> 20, five rows 16 -> 13.5.  Error against
// 64 bits, N(0, 1) keys and queries of 2: 4.8e-6 -> 5.2e-7, 3.4e-6 -> 4.2e-7, 5.0e-7 -> 4.2e-7, 1.9e-7 both.
// Every wait is bounded, as in pfx.cuh.
#pragma once
#include "pfx.cuh"
#include "model.cuh"
#include <cuda.h>

#define PA_THREADS 512
#define PA_BOX (2 * 32 * 128)                    // 64 dims of 32 positions, both planes
#define PA_HDR 2048                              // barriers; the factors of two tiles, a float a query
__host__ __device__ constexpr int pa_slots(int HD) { return HD > 128 ? 5 : 8; }
__host__ __device__ constexpr int pa_slot_bytes(int HD) { return 2 * 32 * HD * 2; }     // 32 positions, both planes
__host__ __device__ constexpr int pa_smem(int HD) { return PA_HDR + 128 * HD * 2 + pa_slots(HD) * pa_slot_bytes(HD); }
static_assert(pa_smem(256) <= PX_SMEM_MAX, "the queries' lo plane and five slots");
// registers a thread: softmax, loads and issue, two warpgroups that read
#define PA_REG_SOFT 96
#define PA_REG_ISSUE 48
#define PA_REG_READ 184
#define PA_REG_LAUNCH 128
static_assert(PA_REG_SOFT + PA_REG_ISSUE + 2 * PA_REG_READ == 4 * PA_REG_LAUNCH, "setmaxnreg.inc waits for ever where the shares are more than the launch's registers");
struct PaArgs {
  const float *q;            // [R][H][HD]
  int H, KV, p0, R, per;     // rows are positions p0 .. p0 + R - 1; positions of a slice, a multiple of 32
  float *pm, *pl, *po;       // [head][row][slice](, [HD])
  unsigned int *err;
};
__host__ __device__ constexpr uint32_t pa_idesc(int N, bool mn) { return 0x08000010u | (mn ? 1u << 16 : 0u) | ((uint32_t)(N >> 3) << 17); }   // D f32, A / B f16, M = 128; mn: B MN-major
__device__ __forceinline__ void pa_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D = A B + D 2^-11
__device__ __forceinline__ void pa_ts_scaled(uint32_t d, uint32_t a_tmem, uint64_t b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, 11;\n\t}\n" ::"r"(d), "r"(a_tmem), "l"(b), "r"(idesc)
      : "memory");
}

// rows of 128 swizzled bytes, eight of them 1024 bytes on from the next eight; mn_step: from 64 columns of an MN-major operand to the next 64
__device__ __forceinline__ uint64_t pa_desc(uint32_t addr_s, uint32_t mn_step) { return g3_desc(addr_s, mn_step, 1024) | (2ull << 61); }

template <int HD>
__global__ void __launch_bounds__(PA_THREADS, 1) k_pf_attn(const PaArgs a, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
  constexpr int NS = pa_slots(HD), SLB = pa_slot_bytes(HD), QPB = 128 * HD * 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t bar_s = smem_u32(smem);
  auto full = [&](int s) { return bar_s + 8u * (uint32_t)s; };
  auto empty = [&](int s) { return bar_s + 64u + 8u * (uint32_t)s; };
  auto s_full = [&](int b) { return bar_s + 128u + 8u * (uint32_t)b; };
  auto p_full = [&](int b) { return bar_s + 144u + 8u * (uint32_t)b; };
  auto pv_done = [&](int b) { return bar_s + 160u + 8u * (uint32_t)b; };
  const uint32_t o_empty = bar_s + 176u, q_full = bar_s + 184u;
  uint32_t *tmem_slot = (uint32_t *)(smem + 192);
  volatile uint32_t *dead = (volatile uint32_t *)(smem + 196);
  float *corr = (float *)(smem + 1024);           // [tile & 1][query]
  uint8_t *qs = smem + PA_HDR, *ring = qs + QPB, *qt = ring + (NS - 2) * SLB;   // qt: the hi plane on its way to tensor memory, the last two slots
  const uint32_t qs_s = smem_u32(qs), ring_s = smem_u32(ring);
  const int G = a.H / a.KV, NQ = a.R * G, kvh = blockIdx.z, split = blockIdx.y, nsplit = gridDim.y, q0 = blockIdx.x * 128, total = a.p0 + a.R;
  const int s0 = split * a.per, s1 = min(min(total, s0 + a.per), a.p0 + (min(q0 + 127, NQ - 1)) / G + 1);   // (no further than the block's last row sees)
  const int n = s1 > s0 ? (s1 - s0 + 31) >> 5 : 0;
  auto out_of = [&](int qi) { return ((size_t)(kvh * G + qi % G) * a.R + qi / G) * nsplit + split; };
  if (n == 0) {                                  // nothing of the slice is before these rows
    pdl_trigger();
    pdl_wait();
    if (tid < 128 && q0 + tid < NQ) { const size_t o = out_of(q0 + tid); a.pm[o] = -INFINITY; a.pl[o] = 0.0f; }
    return;
  }
  if (tid == 0) {
    for (int s = 0; s < NS; s++) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
    for (int b = 0; b < 2; b++) { mbar_init(s_full(b), 1); mbar_init(p_full(b), 4); mbar_init(pv_done(b), 1); }
    mbar_init(o_empty, 8); mbar_init(q_full, 4);
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 6) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  __syncthreads();
  t5_fence_after();
  pdl_trigger();                                 // (tensor memory is taken: a later kernel's block cannot sit on it while it waits for this one)
  pdl_wait();
  const uint32_t tmem = *tmem_slot;              // O: HD columns; from 256 on S: 2 x 32, P: 2 x (hi 16, lo 16), the queries' hi plane
  auto wait = [&](uint32_t bar, uint32_t parity) {   // gives up for the whole block
    for (uint32_t k = 0; !mbar_wait(bar, parity, 4); k += 4) {
      if (*dead) return;
      if (k >= T5_WAIT_LIMIT) { *dead = 1; if (a.err) atomicExch(a.err, 1u); return; }
    }
  };
  if (warp < 4 || warp >= 8) {
    // ---- the queries' planes: [8 dims][query][8], eight queries x four groups of dims a warp ----
    const int r8 = lane & 7, gq = lane >> 3;
    constexpr int UN = 16 * (HD / 32), NB = 6;   // units; a warp's loads in flight together
#pragma unroll 1
    for (int u0 = warp < 4 ? warp : warp - 4; u0 < UN; u0 += 12 * NB) {
      float4 x[NB][2];
#pragma unroll
      for (int j = 0; j < NB; j++) {
        const int u = u0 + 12 * j, qi = q0 + 8 * (u & 15) + r8, gd = 4 * (u >> 4) + gq;
        x[j][0] = x[j][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (u < UN && qi < NQ) {
          const float4 *src = (const float4 *)(a.q + ((size_t)(qi / G) * a.H + kvh * G + qi % G) * HD + 8 * gd);
          x[j][0] = __ldcg(src); x[j][1] = __ldcg(src + 1);
        }
      }
#pragma unroll
      for (int j = 0; j < NB; j++) {
        const int u = u0 + 12 * j, at = (4 * (u >> 4) + gq) * 2048 + (8 * (u & 15) + r8) * 16;
        if (u >= UN) break;
        const float v[8] = {x[j][0].x, x[j][0].y, x[j][0].z, x[j][0].w, x[j][1].x, x[j][1].y, x[j][1].z, x[j][1].w};
        uint32_t h[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const __half2 hh = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
          const float2 hf = __half22float2(hh);
          const __half2 ll = __floats2half2_rn((v[2 * i] - hf.x) * XP_LO_SCALE, (v[2 * i + 1] - hf.y) * XP_LO_SCALE);
          h[i] = *(const uint32_t *)&hh; l[i] = *(const uint32_t *)&ll;
        }
        *(uint4 *)(qt + at) = make_uint4(h[0], h[1], h[2], h[3]);
        *(uint4 *)(qs + at) = make_uint4(l[0], l[1], l[2], l[3]);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads the lo plane through the async proxy
    asm volatile("bar.sync 1, 384;" ::: "memory");
    if (warp < 4) {
#pragma unroll
      for (int c = 0; c < HD / 64; c++) {
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint4 w = *(const uint4 *)(qt + (8 * c + i) * 2048 + tid * 16);
          v[4 * i] = w.x; v[4 * i + 1] = w.y; v[4 * i + 2] = w.z; v[4 * i + 3] = w.w;
        }
        t5_st32(tmem + ((uint32_t)(32 * warp) << 16) + 384u + 32u * (uint32_t)c, v);
      }
      t5_wait_st();
      t5_fence_before();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // (the slots are the loads' from here on)
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
  }

  if (warp < 4) {
    // ---- softmax ----
    px_reg_dec<PA_REG_SOFT>();
    const int qi = q0 + tid, lim = qi < NQ ? min(s1 - 1, a.p0 + qi / G) : -1;   // the last position that the query sees here
    const uint32_t lq = tmem + ((uint32_t)(32 * warp) << 16);
    const float scale = 1.0f / sqrtf((float)HD);
    float m = -INFINITY, l = 0.0f;
#pragma unroll 1
    for (int it = 0; it < n; it++) {
      const int b = it & 1, left = lim - (s0 + 32 * it);   // positions of the tile that it sees: 0 .. left
      float s[32];
      wait(s_full(b), (uint32_t)(it >> 1) & 1u);
      t5_fence_after();
      {
        float x[16], y[16];
        t5_ld16(lq + 256u + 32u * (uint32_t)b, x);
        t5_ld16(lq + 272u + 32u * (uint32_t)b, y);
        t5_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; i++) { s[i] = x[i] * scale; s[16 + i] = y[i] * scale; }
      }
      if (left < 31) {
#pragma unroll
        for (int i = 0; i < 32; i++)
          if (i > left) s[i] = -INFINITY;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int i = 4; i < 32; i++) mx[i & 3] = fmaxf(mx[i & 3], s[i]);
      const float mn = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]))), ref = mn == -INFINITY ? 0.0f : mn;   // (nothing seen yet: every e is 0)
      const float cf = expf(m - ref);
      m = mn;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t P[32];                            // hi, lo
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const float e0 = expf(s[2 * i] - ref), e1 = expf(s[2 * i + 1] - ref);
        sum[i & 3] += e0 + e1;
        const __half2 hh = __floats2half2_rn(e0, e1);
        const float2 hf = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(e0 - hf.x, e1 - hf.y);
        P[i] = *(const uint32_t *)&hh; P[16 + i] = *(const uint32_t *)&ll;
      }
      l = l * cf + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      if (it >= 2) wait(pv_done(b), (uint32_t)((it >> 1) - 1) & 1u);   // P and the factors of two tiles back have been read
      __syncwarp();
      t5_fence_after();
      t5_st32(lq + 320u + 32u * (uint32_t)b, P);
      corr[b * 128 + tid] = cf;
      t5_wait_st();
      t5_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full(b));
    }
    if (qi < NQ) { const size_t o = out_of(qi); a.pm[o] = m; a.pl[o] = l; }
  } else if (warp < 8) {
    px_reg_dec<PA_REG_ISSUE>();
    if (warp == 4) {
      // ---- K and V: [64 dims][plane][position][128 bytes, swizzled] ----
      if (lane == 0) {
        int t = 0;
        auto load = [&](const CUtensorMap *map, int tile) {
          const int slot = t % NS;
          if (t >= NS) wait(empty(slot), (uint32_t)(t / NS - 1) & 1u);
          else if (t == NS - 2) wait(q_full, 0);
          if (!*dead) {
            mbar_expect(full(slot), SLB);
#pragma unroll
            for (int c = 0; c < HD / 64; c++)
              asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(ring_s + slot * SLB + c * PA_BOX),
                           "l"(map), "r"(kvh * HD + 64 * c), "r"(s0 + 32 * tile), "r"(0), "r"(full(slot))
                           : "memory");
          }
          t++;
        };
#pragma unroll 1
        for (int i = -2; i < n; i++) {
          if (i >= 0) load(&vmap, i);
          if (i + 2 < n) load(&kmap, i + 2);
        }
      }
    } else if (warp == 6) {
      // ---- the tensor core: the whole warp walks, an elected lane issues ----
      const bool el = t5_elect();
      constexpr uint32_t ids = pa_idesc(32, false), ido = pa_idesc(HD, true);
      const uint32_t qh = tmem + 384u;
      uint64_t ql = g3_desc(qs_s, 2048, 128);
      int t = 0;
      wait(q_full, 0);
#pragma unroll 1
      for (int i = -2; i < n; i++) {
        if (i >= 0) {
          const int b = i & 1, slot = t % NS;
          wait(p_full(b), (uint32_t)(i >> 1) & 1u);
          wait(o_empty, (uint32_t)i & 1u);       // P(i) has been seen, O(i - 1) has been read
          wait(full(slot), (uint32_t)(t / NS) & 1u);
          t5_fence_after();
          const uint64_t vh = pa_desc(ring_s + slot * SLB, PA_BOX), vl = vh + PA_BOX / 32;
          const uint32_t ph = tmem + 320u + 32u * (uint32_t)b, pl = ph + 16u;
          constexpr uint64_t K16 = 128;          // 16 positions further on, in 16-byte units
          if (el) {
            t5_mma_f16_ts(tmem, ph, vl, ido, 0);
            t5_mma_f16_ts(tmem, ph + 8, vl + K16, ido, 1);
            pa_ts_scaled(tmem, pl, vh, ido);
            t5_mma_f16_ts(tmem, pl + 8, vh + K16, ido, 1);
            t5_mma_f16_ts(tmem, ph, vh, ido, 1);
            t5_mma_f16_ts(tmem, ph + 8, vh + K16, ido, 1);
            t5_commit(pv_done(b));
            t5_commit(empty(slot));
          }
          __syncwarp();
          t++;
        }
        if (i + 2 < n) {
          const int b = i & 1, slot = t % NS;
          wait(full(slot), (uint32_t)(t / NS) & 1u);
          t5_fence_after();
          const uint64_t kh = pa_desc(ring_s + slot * SLB, 16), kl = kh + PA_BOX / 32;
          constexpr uint64_t K64 = PA_BOX / 16;  // 64 dims further on; 16 are two 16-byte units of a row
          const uint32_t D = tmem + 256u + 32u * (uint32_t)b;
          asm volatile("" : "+l"(ql));   // (the steps' descriptors are sums made on the spot: kept over the loop they would be 32 registers)
          if (el) {
#pragma unroll
            for (int k = 0; k < HD / 16; k++) pa_ss(D, ql + 256 * k, kh + (k >> 2) * K64 + 2 * (k & 3), ids, k != 0);
#pragma unroll
            for (int k = 0; k < HD / 16; k++) t5_mma_f16_ts(D, qh + 8 * k, kl + (k >> 2) * K64 + 2 * (k & 3), ids, 1);
            pa_ts_scaled(D, qh, kh, ids);
#pragma unroll
            for (int k = 1; k < HD / 16; k++) t5_mma_f16_ts(D, qh + 8 * k, kh + (k >> 2) * K64 + 2 * (k & 3), ids, 1);
            t5_commit(s_full(b));
            t5_commit(empty(slot));
          }
          __syncwarp();
          t++;
        }
      }
    }
  } else {
    // ---- O into registers: lane quarter q, a query a thread; the two warps of a quarter have half of the dims each ----
    px_reg_inc<PA_REG_READ>();
    constexpr int NH = HD / 2;
    const int q = warp & 3, half = (warp - 8) >> 2;
    const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(half * NH);
    f32x2 acc[NH / 2];
#pragma unroll
    for (int j = 0; j < NH / 2; j++) acc[j] = 0;
#pragma unroll 1
    for (int it = 0; it < n; it++) {
      const int b = it & 1;
      // (the products of a tile, the first one's too, wait until its P and factors have been seen here and the tile before has been read: until
      // then P and the factors two tiles on cannot come, so that a phase of p_full is never missed)
      wait(p_full(b), (uint32_t)(it >> 1) & 1u);
      const float c = corr[b * 128 + 32 * q + lane];
      const f32x2 c2 = x2_pack(c, c);
      __syncwarp();
      if (lane == 0) mbar_arrive(o_empty);
      wait(pv_done(b), (uint32_t)(it >> 1) & 1u);
      t5_fence_after();
#pragma unroll
      for (int i0 = 0; i0 < NH; i0 += 16) {
        f32x2 v[8];
        t5_ld16x2(t0 + i0, v);
        t5_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i0 / 2 + j] = x2_fma(acc[i0 / 2 + j], c2, v[j]);
      }
      t5_fence_before();
    }
    // whole 128-byte pieces of rows, turned in the queries' shared memory: every MMA is done
    float *st = (float *)qs + (warp - 8) * 1024;
    uint32_t at[8];                              // rows 32 q + 4 i + (lane >> 3) of po
#pragma unroll
    for (int i = 0; i < 8; i++) at[i] = (uint32_t)out_of(q0 + 32 * q + 4 * i + (lane >> 3));
#pragma unroll
    for (int c0 = 0; c0 < NH; c0 += 32) {
#pragma unroll
      for (int k = 0; k < 8; k++) {
        float4 v;
        x2_unpack(acc[c0 / 2 + 2 * k], v.x, v.y);
        x2_unpack(acc[c0 / 2 + 2 * k + 1], v.z, v.w);
        *(float4 *)(st + lane * 32 + ((k ^ (lane & 7)) << 2)) = v;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int rr = 4 * i + (lane >> 3), k = lane & 7;
        if (q0 + 32 * q + rr < NQ) *(float4 *)(a.po + (size_t)at[i] * HD + half * NH + c0 + 4 * k) = *(const float4 *)(st + rr * 32 + ((k ^ (rr & 7)) << 2));
      }
      __syncwarp();
    }
  }
  // after a wait ran out nothing is requested any more, but copies may be on their way
  if (*dead) for (int i = 0; i < 64; i++) __nanosleep(1000);
  __syncwarp();
  t5_fence_before();
  __syncthreads();
  if (warp == 6) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// The slices merged and normalised, the sigmoid output gate, into the activations of attn_output (k_attn_comb's arithmetic): a warp a (row, head)
__global__ void __launch_bounds__(256) k_pf_attn_comb(const float *__restrict__ pm, const float *__restrict__ pl, const float *__restrict__ po, PartIn qg, int H, int hd,
                                                      int R, int ns, __half *__restrict__ kg, int row0, int ru) {
  pdl_trigger();
  pdl_wait();
  const int u = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (u >= R * H) return;
  const int h = u % H, t = u / H;
  const size_t qb = ((size_t)h * R + t) * ns;
  float M = -INFINITY;
  for (int s = lane; s < ns; s += 32) M = fmaxf(M, __ldcg(pm + qb + s));
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, i));
  float4 o[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  float L = 0.0f;
#pragma unroll 1
  for (int s0 = 0; s0 < ns; s0 += 32) {          // a lane a slice's weight, then the slices' rows two at a time
    const float m = s0 + lane < ns ? __ldcg(pm + qb + s0 + lane) : -INFINITY, w = m == -INFINITY ? 0.0f : expf(m - M);
    if (w != 0.0f) L += __ldcg(pl + qb + s0 + lane) * w;
#pragma unroll 1
    for (int j = 0; j < 32 && s0 + j < ns; j += 2) {
      float ws[2];
      float4 v[2][2];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        ws[q] = __shfl_sync(0xffffffffu, w, j + q);
#pragma unroll
        for (int i = 0; i < 2; i++)              // (a slice that the row sees nothing of has no sums)
          v[q][i] = ws[q] != 0.0f && 128 * i < hd ? __ldcg((const float4 *)(po + (qb + s0 + j + q) * hd + 128 * i + 4 * lane)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < 2; q++)
#pragma unroll
        for (int i = 0; i < 2; i++) { o[i].x += v[q][i].x * ws[q]; o[i].y += v[q][i].y * ws[q]; o[i].z += v[q][i].z * ws[q]; o[i].w += v[q][i].w * ws[q]; }
    }
  }
#pragma unroll
  for (int i = 16; i > 0; i >>= 1) L += __shfl_xor_sync(0xffffffffu, L, i);
#pragma unroll
  for (int i = 0; i < 2; i++)
    if (128 * i < hd) {
      const int c = 128 * i + 4 * lane;
      const float4 g = part_get4(qg, (size_t)t * 2 * H * hd + (size_t)h * 2 * hd + hd + c);
      pf_kg_store4(kg, H * hd, ru, row0 + t, h * hd + c, (o[i].x / L) / (1.0f + expf(-g.x)), (o[i].y / L) / (1.0f + expf(-g.y)), (o[i].z / L) / (1.0f + expf(-g.z)),
                   (o[i].w / L) / (1.0f + expf(-g.w)));
    }
}
