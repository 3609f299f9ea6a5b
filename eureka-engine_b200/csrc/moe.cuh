// moe.cuh -- the routed-expert FFN's two GEMMs (llb_moe_gu, llb_moe_dn of tools/payload-moeany.patch;
// host side host/llb_host.c:622-724) for the T <= 16 rows of a verify pass (the rows of several streams), on the
// K-quant tiles of gemm2.cuh.
//
// Device layout of a layer's experts: two stacks of ne + 1 blocks, the shared expert being block ne,
//   GU  block e = [ef gate rows][ef up rows] of d columns      (es_gu bytes per block)
//   D   block e = d rows of ef columns                         (es_d bytes per block)
// A token's slots are its k chosen experts in rank order and then the shared expert: ids[live row][0..k],
// wt[t][0..k] (the shared slot carries sigmoid(shared gate)).
//
// The work is grouped by expert.  A UNIT is an expert with up to four (row, slot) pairs that chose it: their hi and lo
// halves are the eight columns of one n-tile, so a weight tile is loaded and unpacked once for four rows.  The pairs of
// a pass in (row, slot) order are dealt out to units in that order; the units' tiles are one list, of which a CTA takes a
// consecutive piece, so that it stages the activations of two units or so and not of the whole pass.
//
//   k_moe_gu   routes first: every CTA makes the same choice from the router's logits (the rows side by side, a warp
//              each) and the same list of units, and the first one leaves them in global memory.  That is
//              shorter than a choice made by the last block of the router's launch: its counter, fence and second trip
//              to L2 were half of the 7.4 us that launch took at four rows.  Then gate|up of every unit; g, u [T][(k+1) ef]
//   k_moe_dn   planes of wt * silu(g) * u of its units in shared memory, then d rows of ef columns; the sum of a
//              (row, slot) goes out as K-slice `slot` of the row, which the consumer adds in slot order: the
//              rank-order weighted sum plus the gated shared expert
// With a virtual matrix per (row, slot), the columns of all rows staged and a tile multiplied with the n-tiles of its
// row's group of eight, the two launches of a layer of the 35B-A3B shape took 18 us at four rows, 54 at eight and 93 at sixteen;
// eight streams of that model with 40 tokens of prompt and 16 of output 193 ms, now 147.
// Column t of a tile is computed by the same instructions wherever it stands in its unit and whatever the other columns
// hold, so a row's result does not depend on which rows share its pass.
#pragma once
#include "gemm2.cuh"
#include "ffn_fused.cuh"
#include "rowops.cuh"

#define MOE_WARPS G2_MAXWARPS
// shared memory that the choice takes: units, chosen ids, per 32 pairs those that open a unit, the rows in use
__host__ __device__ inline int moe_sel_bytes(int pairs) { return pairs * 16 + ((pairs * 4 + 15) & ~15) + 96 + 64; }
// bytes of a unit's staged activations: eight plane columns of nsl super-blocks and their means
__host__ __device__ inline int moe_unit_bytes(int fmt, int nsl) { return 8 * (nsl * 512 + g2_xpad(fmt)) + nsl * 8 * g2_aux(fmt); }

// a unit as stored: x expert, y pairs, z / w pairs 0, 1 / 2, 3 as row | slot << 8 (16 bits each)
__device__ __forceinline__ int moe_member(const int4 &u, int i) { return ((i < 2 ? u.z : u.w) >> (16 * (i & 1))) & 0xffff; }

// The choice of a pass.  sel: moe_sel_bytes of shared memory; units at its front.  Returns how many units there are.
// Every thread of the block; ends with a barrier.
template <int NQ> __device__ __forceinline__ int moe_select(const MoeArgs &m, uint8_t *sel) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pairs_max = m.T * m.nslot, nk = m.nslot - 1;
  int4 *units = (int4 *)sel;
  int *ids = (int *)(sel + pairs_max * 16);
  unsigned int *lead = (unsigned int *)(sel + pairs_max * 16 + ((pairs_max * 4 + 15) & ~15));
  int *rows = (int *)(lead + 24);
  // which rows are in use: the first n of a pass of one stream, of every stream's rows else
  bool on = false;
  if (lane < m.T) {
    const int z = lane / m.per;
    on = lane - z * m.per < __ldcg(&((const RowSet *)((const char *)((uintptr_t)m.rs & ~(uintptr_t)1) + (size_t)z * m.stride))->n);
  }
  const unsigned int mask = __ballot_sync(0xffffffffu, on);
  const int np = __popc(mask) * m.nslot;
  for (int t = warp; t < m.T; t += MOE_WARPS)
    if ((mask >> t) & 1) {
      const int ri = __popc(mask & ((1u << t) - 1));
      if (lane == 0) rows[ri] = t;
      moe_route_row<NQ>(m.lg + (size_t)t * (m.ne + 1), m.ne, nk, ids + ri * m.nslot, blockIdx.x == 0 ? m.wt + (size_t)t * m.nslot : nullptr, lane);
    }
  for (int i = threadIdx.x; i < pairs_max; i += blockDim.x) units[i] = make_int4(0, 0, 0, 0);
  __syncthreads();
  // Pair p = (live row, slot) is number cnt of its expert's pairs; every fourth one opens a unit.  lp: the pair that opened its unit.
  // (a block of 512 threads takes the 528 pairs of sixteen rows of 32 experts in two trips)
  int lp[2], cn[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int p = threadIdx.x + q * MOE_WARPS * 32;
    lp[q] = p; cn[q] = 0;
    if (p < np) {
      const int e = ids[p];
      int cnt = 0, lpos = p;
#pragma unroll 4
      for (int o = 0; o < p; o++)
        if (ids[o] == e) { if (!(cnt & 3)) lpos = o; cnt++; }
      if (!(cnt & 3)) lpos = p;
      lp[q] = lpos; cn[q] = cnt & 3;
    }
    const unsigned int b = __ballot_sync(0xffffffffu, p < np && lp[q] == p);
    if (lane == 0 && p < pairs_max + 31) lead[p >> 5] = b;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const int p = threadIdx.x + q * MOE_WARPS * 32;
    if (p >= np) continue;
    const int l = lp[q];
    int u = __popc(lead[l >> 5] & ((1u << (l & 31)) - 1));
    for (int w = 0; w < (l >> 5); w++) u += __popc(lead[w]);
    const int ri = p / m.nslot, slot = p - ri * m.nslot, t = rows[ri];
    ((unsigned short *)&units[u].z)[cn[q]] = (unsigned short)(t | slot << 8);
    if (l == p) units[u].x = min(max(ids[p], 0), m.ne);
    atomicMax(&units[u].y, cn[q] + 1);
  }
  int nu = 0;
  for (int w = 0; w < (np + 31) >> 5; w++) nu += __popc(lead[w]);
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int i = threadIdx.x; i < np; i += blockDim.x) m.ids[i] = ids[i];
    for (int i = threadIdx.x; i < nu; i += blockDim.x) m.units[1 + i] = units[i];
    if (threadIdx.x == 0) m.units[0] = make_int4(nu, 0, 0, 0);
  }
  return nu;
}

// The tiles [lo, hi) of a launch (tpu tiles to a unit), by all warps: rings of st stages of ch super-blocks, staged in batches of ub
// units.  src(unit, tile) is the first 16 x 256 tile of row tile `tile` of unit `unit`, stage(first, n) puts units first ..
// into shared memory and ends with a barrier, epi(unit, tile, acc) takes a finished row tile (8 columns).
// P = a.parts warps share a row tile, as in g2_phase.
template <int FMT, class Src, class Stage, class Epi>
__device__ __forceinline__ void moe_phase(const GemmArgs &a, G2Ring &rg, const int st, const int ch, const int ub, const int tpu, const int lo, const int hi, const int nsl, uint8_t *planes, float4 *red0,
                                          Src src, Stage stage, Epi epi) {
  constexpr int TB = tile_bytes(FMT);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int P = a.parts, lp = 31 - __clz(P), grp = warp >> lp, mine = warp & (P - 1), step = MOE_WARPS >> lp;
  const int c0 = (mine * nsl) >> lp, c1 = ((mine + 1) * nsl) >> lp;
  const int CS = nsl * 512 + g2_xpad(FMT), UB = moe_unit_bytes(FMT, nsl);
  int p_t = lo + grp, p_c = c0;                       // producer: (tile, super-block) of the next copy
  const uint8_t *p_w = nullptr;
  auto locate = [&]() { if (p_t < hi) { const int u = p_t / tpu; p_w = src(u, p_t - u * tpu); } };
  locate();
  auto issue = [&](int s) {
    if (p_t >= hi || rg.dead) return;
    const int n = min(ch, c1 - p_c);
    if (lane == 0) {
      const uint32_t bar = rg.bar_s + 8 * s;
      mbar_expect(bar, n * TB);
      bulk_load(rg.ring_s + s * ch * TB, p_w + (size_t)p_c * TB, n * TB, bar);
    }
    p_c += n;
    if (p_c == c1) { p_c = c0; p_t += step; locate(); }
  };
#pragma unroll 1
  for (int s = 0; s < st; s++) issue(s);
  float4 *red = red0 + warp * 32 + lane;
  int s = 0, tile = lo + grp;
#pragma unroll 1
  for (int ub0 = lo / tpu; ub0 * tpu < hi; ub0 += ub) {
    if (ub0 * tpu > lo) __syncthreads();              // the units in shared memory are done with
    const int un = min(ub, (hi - 1) / tpu - ub0 + 1), end = min(hi, (ub0 + un) * tpu);
    stage(ub0, un);
#pragma unroll 1
    for (; tile < end; tile += step) {
      const int u = tile / tpu;
      const uint8_t *xh = planes + (size_t)(u - ub0) * UB, *xf = xh + 8 * CS;
      float acc[1][4] = {{0.f, 0.f, 0.f, 0.f}};
#pragma unroll 1
      for (int c = c0; c < c1; c += ch) {
        g2_wait(rg, s, G2_WAIT_LIMIT, a.err);
#pragma unroll 1
        for (int k = 0; k < ch && c + k < c1; k++) g2_tile<FMT, 1, false>(rg.ring + (s * ch + k) * TB, xh, xf, CS, c + k, lane, acc);
        __syncwarp();                                 // every lane has read the stage
        issue(s);
        s = s + 1 == st ? 0 : s + 1;
      }
      if (P > 1) {
        if (mine) *red = make_float4(acc[0][0], acc[0][1], acc[0][2], acc[0][3]);
        asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * P) : "memory");
        if (!mine) {
#pragma unroll 1
          for (int q = 1; q < P; q++) { const float4 v = red[q * 32]; acc[0][0] += v.x; acc[0][1] += v.y; acc[0][2] += v.z; acc[0][3] += v.w; }
        }
        if (tile + step < hi) asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(32 * P) : "memory");   // read before it is written again
      }
      if (!mine) {
        // columns 0 .. 3 the hi halves of the unit's pairs, columns 4 .. 7 their lo halves (held by lane j ^ 2)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[0][i] += __shfl_xor_sync(0xffffffffu, acc[0][i], 2) * XP_LO_INV;
        if ((lane & 3) < 2) epi(u, tile - u * tpu, acc[0]);
      }
    }
  }
}

template <int FMT, int NQ>
__global__ void __launch_bounds__(MOE_WARPS * 32, 1) k_moe_gu(const GemmArgs a, const MoeArgs m, const int st, const int ch, const int ub) {
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  const int per_warp = st * ch * tile_bytes(FMT), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  G2Ring rg = g2_ring_init(smem, per_warp);
  uint8_t *sel = smem + G2_BAR_BYTES + MOE_WARPS * per_warp, *planes = sel + moe_sel_bytes(m.T * m.nslot);
  const int4 *units = (const int4 *)sel;
  const int nsl = a.nsb, tpu = m.ef >> 3;             // 2 ef / 16 tiles a unit
  pdl_wait();
  const int nu = moe_select<NQ>(m, sel), nt = nu * tpu;
  const int lo = (int)((long long)nt * blockIdx.x / gridDim.x), hi = (int)((long long)nt * (blockIdx.x + 1) / gridDim.x);
  const int CS = nsl * 512 + g2_xpad(FMT), UB = moe_unit_bytes(FMT, nsl);
  auto src = [&](int u, int tile) { return m.W + (size_t)units[u].x * m.es + (size_t)tile * nsl * tile_bytes(FMT); };
  // the rows' plane columns from global memory: (unit, pair, hi or lo, super-block), 32 pieces a warp and a lane's piece of the means
  auto stage = [&](int u0, int un) {
    const int NC = a.xp.NC, ntask = un * 8 * nsl;
#pragma unroll 2
    for (int i = warp; i < ntask; i += MOE_WARPS) {
      const int ul = i / (8 * nsl), r = i - ul * 8 * nsl, col = r / nsl, sb = r - col * nsl, p = sb * 32 + lane;
      const int4 u = units[u0 + ul];
      if ((col & 3) >= u.y) continue;
      const int gc = (moe_member(u, col & 3) & 0xff) + (col < 4 ? 0 : NC / 2);
      const uint32_t dst = smem_u32(planes + (size_t)ul * UB);
      cp_async16(dst + col * CS + p * 16, (const uint8_t *)(a.xp.xh + (size_t)gc * a.K) + p * 16);
      if (g2_aux(FMT) != 0 && lane < 2) cp_async16(dst + 8 * CS + (sb * 8 + col) * 32 + lane * 16, (const uint8_t *)(a.xp.xsf + ((size_t)sb * NC + gc) * 16) + lane * 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  };
  auto epi = [&](int u, int tile, const float (&v)[4]) {
    const int4 un = units[u];
    const int r = tile * 16 + g2_row<FMT, false>(lane >> 2);   // rows r and r + 8 of [gate | up]; a tile is all gate or all up
    float *base = r < m.ef ? m.g + r : m.u + (r - m.ef);
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int q = 2 * (lane & 3) + i;
      if (q < un.y) {
        const int mb = moe_member(un, q);
        float *dst = base + ((size_t)(mb & 0xff) * m.nslot + (mb >> 8)) * m.ef;
        dst[0] = v[i]; dst[8] = v[i + 2];
      }
    }
  };
  if (lo < hi) moe_phase<FMT>(a, rg, st, ch, ub, tpu, lo, hi, nsl, planes, (float4 *)(planes + (size_t)ub * UB), src, stage, epi);
  g2_drain(rg);
}

template <int FMT>
__global__ void __launch_bounds__(MOE_WARPS * 32, 1) k_moe_dn(const GemmArgs a, const MoeArgs m, const int st, const int ch, const int ub) {
  extern __shared__ __align__(128) uint8_t smem[];
  pdl_trigger();
  const int per_warp = st * ch * tile_bytes(FMT), lane = threadIdx.x & 31;
  G2Ring rg = g2_ring_init(smem, per_warp);
  int4 *units = (int4 *)(smem + G2_BAR_BYTES + MOE_WARPS * per_warp);   // this CTA's (ks of them to an expert's unit)
  const int ks = a.ksplit, tpu = m.d >> 4, eb = m.ef >> 8, umax = m.T * m.nslot;
  pdl_wait();
  const int nu = min(__ldcg((const int *)m.units), umax), nt = nu * ks * tpu;
  const int lo = (int)((long long)nt * blockIdx.x / gridDim.x), hi = (int)((long long)nt * (blockIdx.x + 1) / gridDim.x);
  if (lo >= hi) return;
  const int u0 = lo / tpu / ks, u1 = (hi - 1) / tpu / ks;
  for (int i = threadIdx.x; i <= u1 - u0; i += blockDim.x) units[i] = __ldcg(m.units + 1 + u0 + i);
  __syncthreads();
  uint8_t *planes = (uint8_t *)units + umax * 16;
  const int nsl = eb / ks, CS = nsl * 512 + g2_xpad(FMT), UB = moe_unit_bytes(FMT, nsl);
  auto first = [&](int k) { return k * nsl; };   // first super-block of K-slice k of an expert's columns
  auto src = [&](int u, int tile) { return m.W + (size_t)units[u / ks - u0].x * m.es + ((size_t)tile * eb + first(u % ks)) * tile_bytes(FMT); };
  auto stage = [&](int v0, int vn) {
    const int ngrp = nsl * 64, ntask = vn * 4 * ngrp;   // (unit, pair, group of four columns)
    for (int t0 = threadIdx.x; t0 < ntask; t0 += 4 * blockDim.x) {
      float4 gv[4], uv[4];
      float w[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int task = t0 + q * blockDim.x, vp = task / ngrp, c = 4 * (task - vp * ngrp);
        gv[q] = make_float4(0.f, 0.f, 0.f, 0.f); uv[q] = gv[q]; w[q] = 0.0f;
        if (task < ntask) {
          const int v = v0 + (vp >> 2);
          const int4 un = units[v / ks - u0];
          const int cg = first(v % ks) * 256 + c;
          if ((vp & 3) < un.y) {
            const int mb = moe_member(un, vp & 3);
            const size_t i = (size_t)(mb & 0xff) * m.nslot + (mb >> 8);
            gv[q] = __ldcg((const float4 *)(m.g + i * m.ef + cg)); uv[q] = __ldcg((const float4 *)(m.u + i * m.ef + cg));
            w[q] = __ldcg(m.wt + i);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int task = t0 + q * blockDim.x, vp = task / ngrp, c = 4 * (task - vp * ngrp);
        if (task < ntask) {   // whole warps: ngrp and blockDim are multiples of 32
          const float h[4] = {(gv[q].x / (1.0f + expf(-gv[q].x))) * uv[q].x * w[q], (gv[q].y / (1.0f + expf(-gv[q].y))) * uv[q].y * w[q],
                              (gv[q].z / (1.0f + expf(-gv[q].z))) * uv[q].z * w[q], (gv[q].w / (1.0f + expf(-gv[q].w))) * uv[q].w * w[q]};
          uint8_t *xh = planes + (size_t)(vp >> 2) * UB;
          ffn_store4<FMT>(xh, xh + 8 * CS, CS, vp & 3, c, h, lane);
        }
      }
    }
    __syncthreads();
  };
  auto epi = [&](int u, int tile, const float (&v)[4]) {
    const int4 un = units[u / ks - u0];
    float *base = m.out + tile * 16 + g2_row<FMT, false>(lane >> 2);
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int q = 2 * (lane & 3) + i;
      if (q < un.y) {
        const int mb = moe_member(un, q);
        float *dst = base + (size_t)((mb >> 8) * ks + u % ks) * m.split_stride + (size_t)(mb & 0xff) * m.d;
        dst[0] = v[i]; dst[8] = v[i + 2];
      }
    }
  };
  moe_phase<FMT>(a, rg, st, ch, ub, tpu, lo, hi, nsl, planes, (float4 *)(planes + (size_t)ub * UB), src, stage, epi);
  g2_drain(rg);
}
