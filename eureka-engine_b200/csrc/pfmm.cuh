// pfmm.cuh -- the prompt path's dense GEMM on the fifth-generation tensor cores: Y[r][n] = sum_k W[n][k] X[r][k] for a
// chunk of 129 to 256 prompt rows against Q6_K / Q8_0 weights (the others, and fewer rows: pfx.cuh).  It replaces, for this library, the
// reference's chunked tensor-core prefill GEMM (tools/pf27/pfmm.cuh:311-384: int8 mma.sync + cp.async on sm_86; its
// caller host/llb_pf.h:551 pf_take) with a design for sm_100a:
//
//   * the multiply is tcgen05.mma over a PAIR of CTAs (kind::f16, cta_group::2: M = 256 weight rows, 128 a CTA, N = 256 prompt
//     rows, K = 16 per instruction), both operands in shared memory, fp32 accumulators in TENSOR MEMORY;
//   * BOTH operands are two fp16 planes, hi = fp16(v) and lo = fp16((v - hi) * 2048) (about 22 bits of v, as the T-row
//     path's activation planes): a 16-column step is three MMAs, hi.hi into one accumulator of 256 columns and the
//     two cross terms hi.lo and lo.hi into another (together all 512 columns of tensor memory); the epilogue adds the
//     cross terms divided by 2048 (lo.lo is below fp32 resolution).  With one fp16 plane per operand every GEMM output carried a relative error of 4e-4, which a
//     random 8-layer model amplified past the path's 2e-2 bar;
//   * a pair because each CTA then stages half of the chunk's rows only: a step of 16 columns moves 40 KB through its shared
//     memory (60 KB alone), and a third stage fits.  N = 256 because a dequantised weight (14.5 thread instructions)
//     then serves all rows of a chunk.  What bounds it is the tensor pipe, 384 cycles a step of 433.  gate|up of the 27B shape,
//     256 rows: 270 us with two units of N = 128 a stage, 232 us with one CTA and N = 256, 185 us so (single CTAs took
//     528 cycles a step: the issuing threads' three barriers a stage and MMAs out of vector registers were their chain);
//   * the activation planes arrive by TMA: the chunk's activations are kept in global memory in the order the operand
//     wants (two units of 128 rows, k-group major, common.cuh), so a CTA's 64-column stage of one plane is ONE contiguous
//     16 KB cp.async.bulk that completes on an mbarrier (plain bulk copies of this GPU's own memory, no multicast);
//   * the weight planes are made on the fly: eight warps read the packed super-blocks (each thread one row's 32 weights
//     of a stage), dequantise in fp32 (the formulas of tools/qwen35_engine.c:233-307, one FMA per weight), split
//     each weight into its two planes and store 16-byte core-matrix rows; stores of a warp are conflict-free;
//   * a three-stage ring of (32 KB weights, 32 KB activations) with full / empty mbarriers decouples the roles, so
//     loads and dequantisation run ahead of the MMAs; four more warps read a finished tile out with tcgen05.ld.  One full
//     barrier a stage, the leader's: the other CTA's warps arrive on it through the cluster;
//   * every wait is bounded: a wait that runs out sets *err, and all roles then run through without waiting, so the
//     kernel returns, frees its tensor memory and leaves the context usable (llb_b200_wait_errors() reports it).
#pragma once
#include "gemm.cuh"
#include "tc5.cuh"
#include "pf.cuh"

#define PF_KS 64              // columns per ring stage
#define PF_STAGES 3
#define PF_A_BYTES (128 * PF_KS * 2)     // one plane of a CTA's 128 weight rows
#define PF_B_BYTES (PF_R * PF_KS * 2)    // one plane of a CTA's half of the chunk's rows
#define PF_STAGE_BYTES (2 * PF_A_BYTES + 2 * PF_B_BYTES)   // [A hi | A lo | B hi | B lo]
#define PF_SMEM (1024 + PF_STAGES * PF_STAGE_BYTES)
#define PF_THREADS 512        // warps 0-7 dequantise, 8 loads activations, 9-10 issue MMAs, 11 forwards, 12-15 write results
#define PF_IDESC (0x10000010u | ((uint32_t)(PF_RMAX >> 3) << 17))  // kind::f16: D f32, A / B f16 K-major, N = 256, M = 256 over the pair


__device__ __forceinline__ void pf_mma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void pf_bulk_copy(uint32_t dst_s, const void *src, uint32_t bytes, uint32_t bar_s) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_s), "l"(src), "r"(bytes), "r"(bar_s)
               : "memory");
}

// ---- weights: packed super-blocks -> fp16 core-matrix rows ------------------------------------------
// A thread takes the 32 weights of one row that start at column c0 (a multiple of 32): raw words with pf_load, fp32
// values with pf_deq, then pf_split8 turns every eight of them into a 16-byte row of each plane (k-groups c0/8 .. + 3).
struct PfRaw { uint32_t w[8], x[8], h[2]; };

// row: the row's block in the first super-block of its row tile;  doff: from there to the row's d (Q6_K)
template <int FMT> __device__ __forceinline__ void pf_load(const uint8_t *row, int doff, int c0, PfRaw &r) {
  const uint8_t *blk = row + (size_t)(c0 >> 8) * tile_bytes(FMT);
  if constexpr (FMT == LLB_FM_Q8_0) {
    const int i = c0 & 255;
    const uint4 a = ldg128(blk + i), b = ldg128(blk + i + 16);
    r.w[0] = a.x; r.w[1] = a.y; r.w[2] = a.z; r.w[3] = a.w; r.w[4] = b.x; r.w[5] = b.y; r.w[6] = b.z; r.w[7] = b.w;
    r.h[0] = *(const unsigned short *)(blk + 256 + 2 * (i >> 5));
  } else {
    const int j8 = (c0 >> 5) & 7, hf = j8 >> 2, qd = j8 & 3;
    const uint4 a = ldg128(blk + 64 * hf + 32 * (qd & 1)), b = ldg128(blk + 64 * hf + 32 * (qd & 1) + 16);
    const uint4 c = ldg128(blk + 128 + 32 * hf), d = ldg128(blk + 128 + 32 * hf + 16);
    r.w[0] = a.x; r.w[1] = a.y; r.w[2] = a.z; r.w[3] = a.w; r.w[4] = b.x; r.w[5] = b.y; r.w[6] = b.z; r.w[7] = b.w;
    r.x[0] = c.x; r.x[1] = c.y; r.x[2] = c.z; r.x[3] = c.w; r.x[4] = d.x; r.x[5] = d.y; r.x[6] = d.z; r.x[7] = d.w;
    r.h[0] = *(const unsigned short *)(blk + 192 + 8 * hf + 2 * qd);   // the two int8 scales of this quarter
    r.h[1] = *(const unsigned short *)(blk + doff);
  }
}

// An integer code c < 128 sitting in bits 16.. of a word becomes the float 128 + c by OR-ing 0x43000000 (no conversion
// instruction); one FMA then gives scale * c - offset: fmaf(128 + c, scale, -(128 scale + offset)).  The constant is rounded
// once per sub-block (about 1e-6 of a weight); both planes together still carry the result to about 22 bits.
__device__ __forceinline__ float pf_code_f(uint32_t x, int j, uint32_t mask) {
  // byte j of x, masked, moved to bits 16..: shifts by 16, 8, 0, -8
  const uint32_t v = j == 0 ? x << 16 : j == 1 ? x << 8 : j == 2 ? x : x >> 8;
  return __uint_as_float((v & (mask << 16)) | 0x43000000u);
}

// the 32 weights as fp32
template <int FMT> __device__ __forceinline__ void pf_deq(const PfRaw &r, int c0, float (&w)[32]) {
  if constexpr (FMT == LLB_FM_Q8_0) {
    const float d = h2f_bits(r.h[0]), c = -384.0f * d;     // byte = q + 128, float = 256 + byte
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t x = r.w[i];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t v = j == 0 ? x << 15 : j == 1 ? x << 7 : j == 2 ? x >> 1 : x >> 9;
        w[4 * i + j] = fmaf(__uint_as_float((v & (0xffu << 15)) | 0x43800000u), d, c);
      }
    }
  } else {
    const int qd = (c0 >> 5) & 3;
    const float d = h2f_bits(r.h[1]);
    const float s0 = __fmul_rn(d, (float)(int8_t)(r.h[0] & 0xff)), s1 = __fmul_rn(d, (float)(int8_t)(r.h[0] >> 8));
    const float k0 = -160.0f * s0, k1 = -160.0f * s1;      // (128 + code) - 160 = code - 32
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const uint32_t x = qd < 2 ? r.w[i] : r.w[i] >> 4, hb = (r.x[i] >> (2 * qd)) & 0x03030303u;
      const uint32_t c6 = (x & 0x0f0f0f0fu) | (hb << 4);   // four six-bit codes, one a byte
#pragma unroll
      for (int j = 0; j < 4; j++) w[4 * i + j] = fmaf(pf_code_f(c6, j, 0x3fu), i < 4 ? s0 : s1, i < 4 ? k0 : k1);
    }
  }
}
// eight weights -> one 16-byte row of the hi plane and one of the lo plane, in the activations' order of columns (xp_perm).  hi is the weight with its low 13 mantissa
// bits cleared (exactly an fp16 number for normal magnitudes), lo the exact remainder times 2048.
__device__ __forceinline__ void pf_split8(const float *w, uint4 &hi, uint4 &lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = (i >> 1) * 4 + (i & 1);
    const float a = w[c], b = w[c + 2];
    const float ah = __uint_as_float(__float_as_uint(a) & 0xffffe000u), bh = __uint_as_float(__float_as_uint(b) & 0xffffe000u);
    const __half2 hh = __floats2half2_rn(ah, bh), ll = __floats2half2_rn((a - ah) * XP_LO_SCALE, (b - bh) * XP_LO_SCALE);
    h[i] = *(const uint32_t *)&hh; l[i] = *(const uint32_t *)&ll;
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// ---- the kernel ------------------------------------------------------------------------------------------------
// Work unit = (pair of 128-row tiles, K-slice); CTA pair b takes units b, b + pairs, ..., its CTA r tile 2 i + r of pair i.  Every
// role walks the same unit sequence.  The last pair's second tile may not exist: its CTA repeats the last one and stores nothing.
__device__ __forceinline__ void pf_locate(const PfArgs &a, int tile, int &m, int &row0) {
  m = 0;
  while (m + 1 < a.nmat && tile >= a.t128[m + 1]) m++;
  row0 = (tile - a.t128[m]) * 128;
}
// K-slices are whole super-blocks, as equal as they come: first column and 64-column stages of unit u
__device__ __forceinline__ void pf_slice(const PfArgs &a, int u, int npairs, int &kbase, int &nst) {
  const int ks = u / npairs, nsb = a.K >> 8;
  const int sb0 = (int)(((long long)ks * nsb) / a.ksplit), sb1 = (int)(((long long)(ks + 1) * nsb) / a.ksplit);
  kbase = sb0 << 8; nst = (sb1 - sb0) << 2;
}

template <int FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PF_THREADS, 1) k_pfmm(const PfArgs a) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // header: full[4] +0, full_b[4] +32, empty[4] +64, acc_full +128, acc_empty +136, tensor-memory address +144, dead +148.
  // The pair's first CTA (the leader) issues the MMAs: its full counts the dequantising warps of both CTAs, its own activations and
  // the other CTA's (which land on that CTA's full_b and are passed on), its acc_empty the result warps of both; the MMAs'
  // commits arrive in both CTAs.
  const uint32_t bar_s = smem_u32(smem);
  auto full = [&](int s) { return bar_s + 8u * (uint32_t)s; };
  auto full_b = [&](int s) { return bar_s + 32u + 8u * (uint32_t)s; };
  auto empty = [&](int s) { return bar_s + 64u + 8u * (uint32_t)s; };
  const uint32_t acc_full = bar_s + 128u, acc_empty = bar_s + 136u;
  uint32_t *tmem_slot = (uint32_t *)(smem + 144);
  volatile uint32_t *dead = (volatile uint32_t *)(smem + 148);
  uint8_t *ring = smem + 1024;
  const uint32_t ring_s = smem_u32(ring);
  const int ntiles = a.t128[a.nmat], npairs = (ntiles + 1) >> 1, nunits = npairs * a.ksplit;
  const int rank = blockIdx.x & 1, unit0 = blockIdx.x >> 1, ustep = gridDim.x >> 1;
  auto tile_of = [&](int u) { return 2 * (u % npairs) + rank; };

  pdl_trigger();
  if (tid == 0) {
    for (int s = 0; s < PF_STAGES; s++) { mbar_init(full(s), 18); mbar_init(full_b(s), 1); mbar_init(empty(s), 2); }
    mbar_init(acc_full, 2); mbar_init(acc_empty, 8);
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
  const uint32_t tmem_base = *tmem_slot;
  // a bounded wait that gives up for the whole CTA
  // (a phase that is complete costs one try: the issuing warps' waits are part of the chain that paces the MMAs)
  auto wait = [&](uint32_t bar, uint32_t parity) {
    for (uint32_t n = 0; !mbar_wait(bar, parity, 4); n += 4) {
      if (*dead) return;
      if (n >= T5_WAIT_LIMIT) { *dead = 1; if (a.err) atomicExch(a.err, 1u); return; }
    }
  };

  if (warp < 8) {
    // ---- weights: thread = (row r of the tile, half h of the stage's 64 columns) ----
    const int r = tid & 127, h = tid >> 7;
    PfRaw raw0, raw1;                                  // two stages of raw words in flight (never indexed: they stay in registers)
    int it = 0;                                        // stages produced so far by this CTA
    // the loads run two stages ahead of the conversion: cursor (lu, ls) is the stage to load next
    int lu = unit0, ls = 0, lkbase = 0, lnst = 0, lm = 0, lrow0 = 0;
    const uint8_t *lrow = nullptr;
    int ldoff = 0;
    auto lplan = [&]() {
      if (lu < nunits) {
        pf_locate(a, min(tile_of(lu), ntiles - 1), lm, lrow0);
        pf_slice(a, lu, npairs, lkbase, lnst);
        const int row = min(lrow0 + r, a.m[lm].rows - 1);
        lrow = a.m[lm].W + (size_t)(row >> 4) * (a.K >> 8) * tile_bytes(FMT) + (row & 15) * tile_row(FMT);
        ldoff = 3328 + 2 * (row & 15) - (row & 15) * 208;
      }
    };
    auto lnext = [&](PfRaw &dst) {
      if (lu < nunits) {
        pf_load<FMT>(lrow, ldoff, lkbase + ls * PF_KS + 32 * h, dst);
        if (++ls == lnst) { ls = 0; lu += ustep; lplan(); }
      }
    };
    // converts the stage held in rw (columns c0 ..), refills rw with the stage two ahead, publishes the stage
    auto one = [&](PfRaw &rw, int c0) {
      const int slot = it % PF_STAGES;
      float w[32];
      pf_deq<FMT>(rw, c0, w);
      lnext(rw);
      if (it >= PF_STAGES) wait(empty(slot), (uint32_t)((it / PF_STAGES) + 1) & 1u);
      uint8_t *A = ring + (size_t)slot * PF_STAGE_BYTES;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint4 hi, lo;
        pf_split8(w + 8 * j, hi, lo);
        *(uint4 *)(A + ((size_t)(4 * h + j) * 128 + r) * 16) = hi;
        *(uint4 *)(A + PF_A_BYTES + ((size_t)(4 * h + j) * 128 + r) * 16) = lo;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMA reads these bytes through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(t5_map_rank(full(slot), 0));
      it++;
    };
    lplan();
    lnext(raw0);
    lnext(raw1);
    for (int u = unit0; u < nunits; u += ustep) {
      int kbase, nst;
      pf_slice(a, u, npairs, kbase, nst);
      for (int s = 0; s < nst; s += 2) {               // nst is a multiple of four: a K-slice is whole super-blocks
        one(raw0, kbase + 32 * h + s * PF_KS);
        one(raw1, kbase + 32 * h + (s + 1) * PF_KS);
      }
    }
  } else if (warp == 8) {
    // ---- activations of this CTA's half of the chunk's rows: one 16 KB bulk copy per plane and stage ----
    if (lane == 0) {
      int it = 0;
      pdl_wait();   // the activations come from the kernel in front; the weights do not, and nothing is written before MMAs have read activations
      const __half *x = a.x + (size_t)rank * pf_kg_halves(a.K, PF_R);   // a unit's planes follow the previous unit's (common.cuh)
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
        for (int s = 0; s < nst; s++, it++) {
          const int slot = it % PF_STAGES;
          if (it >= PF_STAGES) wait(empty(slot), (uint32_t)((it / PF_STAGES) + 1) & 1u);
          if (*dead) continue;
          const __half *src = x + (size_t)((kbase + s * PF_KS) >> 3) * PF_R * 8;
          const uint32_t dst = ring_s + slot * PF_STAGE_BYTES + 2 * PF_A_BYTES, bar = rank ? full_b(slot) : full(slot);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(2 * PF_B_BYTES)) : "memory");
          pf_bulk_copy(dst, src, PF_B_BYTES, bar);
          pf_bulk_copy(dst + PF_B_BYTES, src + (size_t)a.K * PF_R, PF_B_BYTES, bar);
        }
      }
    }
  } else if (warp == 11) {
    // ---- tells the leader that the other CTA's activations are there ----
    if (lane == 0 && rank == 1) {
      int it = 0;
      for (int u = unit0; u < nunits; u += ustep) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
        for (int s = 0; s < nst; s++, it++) {
          const int slot = it % PF_STAGES;
          wait(full_b(slot), (uint32_t)(it / PF_STAGES) & 1u);
          mbar_arrive_cluster(t5_map_rank(full(slot), 0));
        }
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ---- the tensor cores of the pair, from the leader.  The products of a step are spread over two warps; MMAs into one
    // accumulator come from one thread (a thread's MMAs execute in its issue order, MMAs of different threads would not be
    // ordered):
    //   warp 9: hi.hi -> D1     warp 10: hi.lo and lo.hi -> D23     result = D1 + D23 / 2048
    //   (tensor-memory columns of each CTA: D1 at 0, D23 at 256)
    // The whole warp walks the stages and one elected lane issues, so that descriptors stay in uniform registers: inside a
    // single lane's branch an MMA cost 100 to 200 cycles to issue, more than it takes to execute.
    if (rank == 0) {
      const int which = __shfl_sync(0xffffffffu, warp - 9, 0);
      const bool el = t5_elect();
      int it = 0, i = 0, slot = 0;
      uint32_t par = 0;
      for (int u = unit0; u < nunits; u += ustep, i++) {
        int kbase, nst;
        pf_slice(a, u, npairs, kbase, nst);
        if (i >= 1) wait(acc_empty, (uint32_t)(i - 1) & 1u);   // the previous tiles have been read out of tensor memory
        t5_fence_after();
        for (int s = 0; s < nst; s++, it++) {
          wait(full(slot), par);
          t5_fence_after();
          const uint32_t st = ring_s + slot * PF_STAGE_BYTES, b0 = st + 2 * PF_A_BYTES;
          const uint64_t a_hi = g3_desc(st, 2048, 128), a_lo = g3_desc(st + PF_A_BYTES, 2048, 128);
          const uint64_t b_hi = g3_desc(b0, 2048, 128), b_lo = g3_desc(b0 + PF_B_BYTES, 2048, 128);
          if (el) {
#pragma unroll
            for (int k = 0; k < PF_KS / 16; k++) {   // a step is two k-groups further on: the address field counts 16-byte units
              const uint64_t kk = (uint64_t)(k * 2 * 2048 / 16);
              const uint32_t first = (s | k) != 0;
              if (which == 0) pf_mma_ss(tmem_base, a_hi + kk, b_hi + kk, PF_IDESC, first);
              else {
                pf_mma_ss(tmem_base + PF_RMAX, a_hi + kk, b_lo + kk, PF_IDESC, first);
                pf_mma_ss(tmem_base + PF_RMAX, a_lo + kk, b_hi + kk, PF_IDESC, 1u);
              }
            }
            t5_commit_pair(empty(slot));   // arrives in both CTAs when this thread's MMAs have read the stage
            if (s + 1 == nst) t5_commit_pair(acc_full);   // ... and when this thread's share of the tiles is in tensor memory
          }
          __syncwarp();
          if (++slot == PF_STAGES) { slot = 0; par ^= 1u; }
        }
      }
      // nothing of the pair may still run on the tensor cores when its tensor memory is freed
      if (i > 0) mbar_wait(acc_full, (uint32_t)(i - 1) & 1u);   // (bounded; after a wait that gave up too: the commits above always arrive)
    }
  } else if (warp >= 12) {
    // ---- results: lane quarter q of the accumulators, one weight row per thread ----
    // The tensor core waits for this (both accumulators fill tensor memory), so the loop holds nothing but loads, sums and
    // stores: with the matrix's fields read and the row count tested at every store a tile took 20000 cycles here, a tenth to a
    // fifth of its life; now 2000.
    const int q = warp - 12, R = a.R;
    int i = 0;
    for (int u = unit0; u < nunits; u += ustep, i++) {
      int m, row0;
      const int tile = tile_of(u);
      pf_locate(a, min(tile, ntiles - 1), m, row0);
      const int row = row0 + 32 * q + lane;
      const bool on = tile < ntiles && row < a.m[m].rows;
      const size_t os = a.m[m].ostride;
      float *out = a.m[m].out + (size_t)(u / npairs) * a.m[m].split_stride + row;
      wait(acc_full, (uint32_t)i & 1u);
      t5_fence_after();
      const uint32_t t0 = tmem_base + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
      for (int c = 0; c < R; c += 16) {       // chunk rows c .. c + 15 are columns c .. of both accumulators
        float v[16], v2[16];
        t5_ld16(t0 + c, v);
        t5_ld16(t0 + c + PF_RMAX, v2);
        t5_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] += v2[j] * XP_LO_INV;
        if (on && c + 16 <= R) {
#pragma unroll
          for (int j = 0; j < 16; j++) { *out = v[j]; out += os; }
        } else if (on) {
#pragma unroll
          for (int j = 0; j < 16; j++) { if (c + j < R) *out = v[j]; out += os; }
        }
      }
      t5_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(t5_map_rank(acc_empty, 0));
    }
  }
  // after a wait ran out nothing is requested any more, but copies may be on their way into this CTA's ring: they land within
  // microseconds, and their barriers count others too, so the CTA gives them 64
  if (*dead) for (int i = 0; i < 64; i++) __nanosleep(1000);
  __syncwarp();
  t5_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");   // no CTA leaves while the other still arrives here or reads its memory
  if (warp == 10) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}
