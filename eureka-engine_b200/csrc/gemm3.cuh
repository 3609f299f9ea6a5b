// gemm3.cuh -- the skinny GEMM of large Q4_K launches on the fifth-generation tensor cores (tcgen05), T <= 16.
//
// The mma.sync kernel (gemm2.cuh) is bound by its instructions, not by the weights' bytes: gate|up of the 27B shape takes as
// long when its weights come from L2 as from HBM (23 us; 15.4 at the measured copy rate), and the work around its
// MMAs grows with the rows (60 us at sixteen).  Here
//   * the multiply is tcgen05.mma (M = 128 weight rows, N = 16 or 32 plane columns, K = 16) with the weight operand in TENSOR
//     MEMORY, which costs the SM's issue slots nothing and does not grow with the rows;
//   * the six-bit scale is multiplied into the code: sc * (q - 8) is an exact fp16 number, so a whole super-block of 256
//     columns accumulates into ONE fp32 accumulator and d comes in once per super-block.  A row of a super-block is 32 words,
//     nine instructions each for eight products: about 210 warp instructions a 16 x 256 tile against 351;
//   * what the 8 took, and the "min" term, are an MMA each against the means of the sub-blocks, the second into an accumulator of its
//     own, as in gemm2.cuh.  The tensor core truncates where it adds to an accumulator.  With q from 0 to 15 the sixteen MMAs of a
//     super-block climb, for activations with a mean, to a sum that the min term then all but cancels, and sixteen truncations of one
//     sign are left: x = 1 + 0.1 N against quantised Gaussian weights, 5120 columns, 6.5e-5 of the result's norm off 64 bits (k_gemm2 3.5e-6).
//     Centred, the climb is one MMA, the chain's last: 2.3e-6; N(0, 1) 7e-7 -> 3.1e-7 (3.4e-7 to 1.2e-6), silu(g) u 7e-7 -> 3.8e-7 (4e-7 to
//     5e-6); |N| 2.3e-6 at 5120 columns and 3.7e-6 at 17408 (1.7e-6 and 2.1e-6; at sixteen rows 2.3e-5 and 4.2e-5).
// gate|up of the 27B shape, launches of a graph over cold weights: 27.0 -> 25.4 us at one row, 27.5 -> 27.4 at four, 36.4 -> 33.3 at eight, 58.8 ->
// 46.5 at sixteen; centring cost 0.4 us at one and four rows, 1.5 at eight.  What is left: the activations, which every SM reads before its first
// MMA (about 4 us for four rows of 5120 columns; cp.async or plain loads, in one order or a different one in every CTA, take the same),
// the groups' chains of waits, 16 warps an SM deep at most (half of the issue slots are in use), and tiles of 128 rows that do not divide evenly.
//
// Roles of a CTA (one an SM): GROUPS of four warps, a thread a weight row, take the super-blocks of the CTA's tiles in turn:
// unpack into the group's operand buffer, and before the next one read the accumulators of the last and scale them into the
// row's sums.  A group has its own operand and accumulators, so groups wait for nothing but their own MMAs; a warp a group issues
// them (all lanes walk, an elected one issues: descriptors stay in uniform registers; one warp for all groups paced the
// kernel, 990 cycles a super-block, a third of them in waits that find their phase complete), one requests the weights (two
// super-blocks of eight 16-row tiles a stage, a bulk copy a tile).  At the end of a tile the other groups leave their sums in shared memory
// and the group that came last adds them in order and writes.
//   Tensor memory: see g3_reuse.  Three groups at N = 16, two at N = 32.
//   Shared memory: activation planes of the K-slice as K-major core matrices [k / 8][column][8 halves] (their k-order 0 2 1 3 4 6
//   5 7 is the one the unpack produces), the sub-block means likewise, the groups' sums, the ring.
//   N is 16 at least, and with 8 plane columns half of an accumulator is whatever a neighbouring k-group's columns give; nobody
//   reads it.
// Every wait is bounded; one that runs out sets *err, all roles then run through without waiting, copies in flight get time to
// land, tensor memory is freed and the kernel returns.
#pragma once
#include "gemm2.cuh"
static_assert(GEMM_MAXMAT == 4, "k_gemm3 finds a tile's matrix with three compares");

#define G3_HDR 256
#define G3_SMEM_MAX 231424
#define G3_CH 2                // super-blocks a copy brings
#define G3_STAGE (8 * G3_CH * tile_bytes(LLB_FM_Q4_K))
__host__ __device__ constexpr int g3_groups(int NC) { return NC <= 16 ? 3 : 2; }
__host__ __device__ constexpr int g3_n(int NC) { return NC <= 16 ? 16 : 32; }
// Tensor memory: the groups' operands -- 128 columns of products, behind them 16 of scales and mins --, then the groups' accumulators, D of
// the products and the scales' part, P of the mins.  Three groups are short of room:
//   8 plane columns: half of each N = 16 is nothing anybody reads.  D's is the upper half; P's B operand starts a column group
//     early, so that its own is the lower one, and the two lie over one another: 24 columns.
//   16: scales and mins take the place of the first half of the products once that half's MMAs are done (a wait more an item: 4 % of
//     the operator's time where it was measured, at 8).
__host__ __device__ constexpr bool g3_reuse(int NC) { return NC == 16; }
__host__ __device__ constexpr int g3_a_cols(int NC) { return g3_reuse(NC) ? 128 : 144; }
__host__ __device__ constexpr int g3_p_col(int NC) { return NC == 8 ? 8 : g3_n(NC); }    // P behind D
__host__ __device__ constexpr int g3_d_cols(int NC) { return g3_p_col(NC) + g3_n(NC); }
static_assert(3 * (g3_a_cols(8) + g3_d_cols(8)) <= 512 && 3 * (g3_a_cols(16) + g3_d_cols(16)) <= 512 && 2 * (g3_a_cols(32) + g3_d_cols(32)) <= 512, "tensor memory");
__host__ __device__ constexpr int g3_threads(int NC) { return g3_groups(NC) * 160 + 32; }
__host__ __device__ constexpr int g3_red_bytes(int NC) { return (NC <= 16 ? 2 : 1) * (g3_groups(NC) - 1) * 128 * NC * 4; }
// planes and means of a K-slice of nsl super-blocks (and what the MMAs read beyond the last column)
__host__ __device__ inline int g3_xp_bytes(int NC, int nsl) { return nsl * NC * (512 + 32) + 512; }
__host__ __device__ inline int g3_stages(int NC, int nsl) {
  const int left = G3_SMEM_MAX - G3_HDR - g3_red_bytes(NC) - g3_xp_bytes(NC, nsl), st = left / G3_STAGE;
  return st > 4 ? 4 : st;
}
// A CTA's barriers by number, eight bytes each from the front of its shared memory, and the arrivals that complete a phase.
// A stage has two raw_full barriers that its uses take in turn: a group passes over chunks, and bulk copies land in any order, so
// it comes to use u of a stage without having seen use u - 1 land; with one barrier the parity of a phase that is still
// pending reads as use u complete.  Use u - 2 of the stage it knows to have landed (g3_walk below).
enum { G3_RAW_FULL = 0 /* [2][4] */, G3_RAW_EMPTY = 8, G3_A_FULL = 12 /* [3][2] */, G3_D_FULL = 18, G3_RED_FULL = 21, G3_RED_EMPTY = 23, G3_XP_FULL = 25, G3_HALF = 26 /* [3] */, G3_BARS = 29 };
__host__ __device__ constexpr int g3_bar_count(int NC, int b) {
  return b < G3_RAW_EMPTY ? 1 : b < G3_A_FULL ? 4 * G3_CH : b < G3_D_FULL ? 4 : b < G3_RED_FULL ? 1 : b < G3_RED_EMPTY ? 4 * (g3_groups(NC) - 1) : b < G3_XP_FULL ? 4 : b < G3_HALF ? g3_groups(NC) * 128 : 1;
}
// A group's walk: the item (tile of the CTA, super-block of the slice), the stage it lies in and which use of that stage.  nsl >= NG,
// so that every group has an item in every tile; st >= 2.  NG super-blocks on are two chunks on at most (a tile's last chunk may hold
// one): the chunk a group comes from was requested behind use u - 1 of the stage it goes to or is that use, which was requested when
// every group had read use u - 2.
struct G3Walk {
  int ti, c, slot, use;
  __host__ __device__ __forceinline__ void start(int g, int st) { ti = 0; c = g; slot = (g / G3_CH) % st; use = (g / G3_CH) / st; }
  __host__ __device__ __forceinline__ void next(int NG, int nsl, int st) {
    int step = -(c / G3_CH);            // as many stages as chunk boundaries lie between
    c += NG;
    if (c >= nsl) { c -= nsl; ti++; step += (nsl + G3_CH - 1) / G3_CH; }
    slot += step + c / G3_CH;
    if (slot >= st) { slot -= st; use++; }
  }
  __host__ __device__ __forceinline__ int full() const { return G3_RAW_FULL + 4 * (use & 1) + slot; }   // its barrier and the phase of that
  __host__ __device__ __forceinline__ int phase() const { return use >> 1; }
  // arrivals a warp owes its stage for the item (a stage with one super-block stands for two)
  __host__ __device__ __forceinline__ int owed(int nsl) const { return c + 1 == nsl && c % G3_CH == 0 ? G3_CH : 1; }
};
// The sums of a tile: the buffer where the other groups leave theirs, which use of the buffer that is, and the group that adds them up
// (it has the tile's last super-block).  From the second use on EVERY group waits until the use before has been read, the adding group
// too: it may have been a writer then and not know that the other writer had arrived, and the parity of that phase of red_full, still
// pending, would read as this one's.
struct G3Sum { int p, n, owner; };
__host__ __device__ __forceinline__ G3Sum g3_sum(int NC, int nsl, int t) {
  return G3Sum{NC <= 16 ? t & 1 : 0, NC <= 16 ? t >> 1 : t, ((t + 1) * nsl - 1) % g3_groups(NC)};
}
__host__ __device__ constexpr uint32_t g3_idesc(int N) { return 0x08000010u | ((uint32_t)(N >> 3) << 17); }   // kind::f16: D f32, A / B f16 K-major, M = 128

template <int NC>
__global__ void __launch_bounds__(g3_threads(NC), 1) k_gemm3(const GemmArgs a, const int cps, const int st) {
  constexpr int NG = g3_groups(NC), N = g3_n(NC), TB = tile_bytes(LLB_FM_Q4_K);
  extern __shared__ __align__(128) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ks = blockIdx.x % a.ksplit, ci = blockIdx.x / a.ksplit;
  const int sb0 = (int)(((long long)ks * a.nsb) / a.ksplit), nsl = (int)(((long long)(ks + 1) * a.nsb) / a.ksplit) - sb0;
  // header: the barriers, tmem, dead
  const uint32_t bar_s = smem_u32(smem);
  auto bar = [&](int b) { return bar_s + 8u * b; };
  auto raw_empty = [&](int i) { return bar(G3_RAW_EMPTY + i); };
  auto a_full = [&](int g, int h) { return bar(G3_A_FULL + 2 * g + h); };
  auto half_done = [&](int g) { return bar(G3_HALF + g); };
  auto d_full = [&](int g) { return bar(G3_D_FULL + g); };
  auto red_full = [&](int p) { return bar(G3_RED_FULL + p); };
  auto red_empty = [&](int p) { return bar(G3_RED_EMPTY + p); };
  const uint32_t xp_full = bar(G3_XP_FULL);
  uint32_t *tmem_slot = (uint32_t *)(smem + 8 * G3_BARS);
  volatile uint32_t *dead = (volatile uint32_t *)(smem + 8 * G3_BARS + 4);
  uint8_t *Bp = smem + G3_HDR, *Bm = Bp + (size_t)nsl * NC * 512 + 256;
  float *red = (float *)(smem + G3_HDR + g3_xp_bytes(NC, (a.nsb + a.ksplit - 1) / a.ksplit));
  uint8_t *ring = (uint8_t *)red + g3_red_bytes(NC);
  const uint32_t Bp_s = smem_u32(Bp), Bm_s = smem_u32(Bm), ring_s = smem_u32(ring);
  int t128[GEMM_MAXMAT + 1];
  t128[0] = 0;
#pragma unroll
  for (int m = 0; m < GEMM_MAXMAT; m++) t128[m + 1] = t128[m] + (m < a.nmat ? (a.m[m].rows + 127) >> 7 : 0);
  const int ntiles = t128[GEMM_MAXMAT], my_tiles = ci < ntiles ? (ntiles - ci + cps - 1) / cps : 0, nch = (nsl + G3_CH - 1) / G3_CH;
  // first row of tile t in its matrix m
  auto locate = [&](int t, int &m) {
    m = (t >= t128[1]) + (t >= t128[2]) + (t >= t128[3]);   // t128[k] = ntiles beyond the last matrix
    return (t - (m == 0 ? 0 : m == 1 ? t128[1] : m == 2 ? t128[2] : t128[3])) * 128;
  };
  pdl_trigger();
  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < G3_BARS; b++) mbar_init(bar(b), g3_bar_count(NC, b));
    *dead = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  t5_fence_before();
  __syncthreads();
  t5_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint32_t bar, uint32_t parity) {   // gives up for the whole CTA
    for (uint32_t n = 0; !mbar_wait(bar, parity, 4); n += 4) {
      if (*dead) return;
      if (n >= T5_WAIT_LIMIT) { *dead = 1; if (a.err) atomicExch(a.err, 1u); return; }
    }
  };

  if (warp < 4 * NG) {
    // ---- workers: group g, row r of the tile ----
    const int g = warp >> 2, q = warp & 3, r = 32 * q + lane;
    const uint32_t lane_off = (uint32_t)(32 * q) << 16;
    const uint32_t abuf = tmem + lane_off + (uint32_t)(g * g3_a_cols(NC)), dbuf = tmem + lane_off + (uint32_t)(NG * g3_a_cols(NC) + g * g3_d_cols(NC));
    const uint32_t roff = (uint32_t)(r >> 4) * (G3_CH * TB) + (r & 15) * tile_row(LLB_FM_Q4_K);
    float acc[NC];
#pragma unroll
    for (int j = 0; j < NC; j++) acc[j] = 0.0f;
    float d_p = 0.0f, dm_p = 0.0f;      // scales of the super-block whose accumulators are read next
    G3Walk wk;
    wk.start(g, st);
    int it = 0, ti_p = 0;               // items so far; the tile of the last one
    // What stands against the means of the activations' sub-blocks (hi halves, and lo halves, which are stored times 2048), as fp16:
    // 8 s 32 2^-19 = s / 2048 and that over 2048, the products' offset; m and m / 2048
    auto store_means = [&](uint32_t at, uint32_t scA, uint32_t scB, uint32_t mnA, uint32_t mnB) {
      uint32_t s8[8], mm[8];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t sel = (j & 1) ? 0x4342u : 0x4140u, s = __byte_perm(j < 2 ? scA : scB, 0x64646464u, sel), m = __byte_perm(j < 2 ? mnA : mnB, 0x64646464u, sel);
        s8[2 * j] = g2_hfma2(s, 0x10001000u, 0xb800b800u); s8[2 * j + 1] = g2_hfma2(s, 0x00040004u, 0x8c008c00u);
        mm[2 * j] = g2_hfma2(m, 0x3c003c00u, 0xe400e400u); mm[2 * j + 1] = g2_hfma2(m, 0x10001000u, 0xb800b800u);
      }
      t5_st8(at, s8);
      t5_st8(at + 8, mm);
    };
    // the accumulators of the last item into the row's sums
    auto drain = [&]() {
      wait(d_full(g), (uint32_t)(it - 1) & 1u);
      t5_fence_after();
#pragma unroll
      for (int j0 = 0; j0 < NC; j0 += 8) {
        float v[8], p[8];
        t5_ld8(dbuf + j0, v);
        t5_ld8(dbuf + g3_p_col(NC) + (NC == 8 ? 8 : 0) + j0, p);
        t5_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; j++) acc[j0 + j] += d_p * v[j] - dm_p * p[j];
      }
      t5_fence_before();
    };
    // A finished tile: the group that has its last super-block (which comes here last) adds the others' sums to its own in group
    // order, then hi + lo / 2048.  (Nothing but loads, sums and stores: with the matrix's fields read at every store a tile of
    // sixteen rows took 4700 cycles.)
    auto flush = [&](int t) {
      const G3Sum sm = g3_sum(NC, nsl, t);
      const int p = sm.p, n = sm.n, og = sm.owner;
      if (n > 0) wait(red_empty(p), (uint32_t)(n - 1) & 1u);
      if (g != og) {
        float *w = red + (size_t)(p * (NG - 1) + (g > og ? g - 1 : g)) * 128 * NC + r;
#pragma unroll
        for (int j = 0; j < NC; j++) w[j * 128] = acc[j];
        __syncwarp();
        if (lane == 0) mbar_arrive(red_full(p));
      } else {
        int m;
        const int row = locate(ci + t * cps, m) + r, T = a.T, os = a.m[m].ostride, rows = a.m[m].rows, per = a.m[m].tok_per, tst = a.m[m].tok_stride, tadd = a.m[m].tok_add;
        float *out = a.m[m].out + (size_t)ks * a.m[m].split_stride + row;
        const int *ts = a.m[m].tok_slot;
        wait(red_full(p), (uint32_t)n & 1u);
#pragma unroll
        for (int k = 0; k < NG - 1; k++) {
          const float *w = red + (size_t)(p * (NG - 1) + k) * 128 * NC + r;
#pragma unroll
          for (int j = 0; j < NC; j++) acc[j] += w[j * 128];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(red_empty(p));
        if (a.planes == 2) {
#pragma unroll
          for (int j = 0; j < NC / 2; j++) acc[j] += acc[j + NC / 2] * XP_LO_INV;
        }
        if (row < rows) {
          if (!ts) {
#pragma unroll
            for (int j = 0; j < NC; j++) {
              if (j < T) *out = acc[j];
              out += os;
            }
          } else {
            // every slot's load in flight at once, row j of stream z counted along: a division a column took longer than all the rest of a
            // tile (the DeltaNet inputs of the 35B-A3B shape, sixteen rows of four streams, 31 us a launch where the mma.sync kernel takes 20)
            int blk[NC / 2], z = 0, tl = 0;     // (passes only: two planes, T <= NC / 2)
#pragma unroll
            for (int j = 0; j < NC / 2; j++) {
              blk[j] = j < T ? __ldcg(ts + z * tst + tl) + z * tadd : 0;
              if (++tl == per) { tl = 0; z++; }
            }
#pragma unroll
            for (int j = 0; j < NC / 2; j++) if (j < T) out[(size_t)blk[j] * os] = acc[j];
          }
        }
      }
#pragma unroll
      for (int j = 0; j < NC; j++) acc[j] = 0.0f;
    };
    // the activation slice: eight pieces of sixteen bytes in flight a thread
    auto stage = [&]() {
      pdl_wait();
      const int half = NC / 2, T = a.T, np = nsl * 32 * NC, nm = nsl * 2 * NC;
      const bool two = a.planes == 2;
      const uint8_t *xh = (const uint8_t *)(a.xp.xh + (size_t)sb0 * 256), *xf = (const uint8_t *)(a.xp.xsf + (size_t)sb0 * NC * 16);
      const size_t cs = (size_t)a.K * 2;
      auto live = [&](int col) { return (two && col >= half ? col - half : col) < T; };
      // (four k-groups of eight columns a warp: whole sectors of the source, whole rows of core matrices at the destination)
#pragma unroll 1
      for (int i0 = tid; i0 < np; i0 += 8 * NG * 128) {
        uint4 x[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int i = i0 + u * NG * 128, blk = i >> 5, col = blk % (NC / 8) * 8 + (i & 7), kg = blk / (NC / 8) * 4 + ((i >> 3) & 3);
          x[u] = i < np && live(col) ? __ldcg((const uint4 *)(xh + col * cs + kg * 16)) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int i = i0 + u * NG * 128, blk = i >> 5, col = blk % (NC / 8) * 8 + (i & 7), kg = blk / (NC / 8) * 4 + ((i >> 3) & 3);
          if (i < np) *(uint4 *)(Bp + (kg * NC + col) * 16) = x[u];
        }
      }
#pragma unroll 1
      for (int i = tid; i < nm; i += NG * 128) {   // (super-block, column, half of its means)
        const int sb = i / (2 * NC), col = (i >> 1) % NC, h = i & 1;
        if (live(col)) *(uint4 *)(Bm + ((sb * 2 + h) * NC + col) * 16) = __ldcg((const uint4 *)(xf + ((size_t)sb * NC + col) * 32 + h * 16));
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the MMAs read these bytes through the async proxy
      mbar_arrive(xp_full);
    };
#pragma unroll 1
    while (wk.ti < my_tiles) {
      wait(bar(wk.full()), (uint32_t)wk.phase() & 1u);
      const uint8_t *row = ring + (size_t)wk.slot * G3_STAGE + roff + wk.c % G3_CH * TB;
      const uint4 hd = *(const uint4 *)row;
      uint32_t scA, scB, mnA, mnB;
      k4_scales(hd.y, hd.z, hd.w, scA, scB, mnA, mnB);
#pragma unroll
      for (int gq = 0; gq < 4; gq++) {            // 64 columns: sub-block 2 gq in the low nibbles, 2 gq + 1 in the high ones
        const uint8_t *qs = row + 16 + 32 * gq;
        const uint4 qa = *(const uint4 *)qs, qb = *(const uint4 *)(qs + 16);
        const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
        // the scales as fp16 (0x6400 | s is 1024 + s) times 2^5 for the low nibbles and 2 for the high ones, which stay four bits
        // up: q 2^-24 * s 2^5 - 8 s 2^-19 = 16 q 2^-24 * s 2 - 8 s 2^-19 = s (q - 8) 2^-19, exact
        const uint32_t sw = gq < 2 ? scA : scB;
        const uint32_t L = g2_hfma2(__byte_perm(sw, 0x64646464u, gq & 1 ? 0x4242 : 0x4040), 0x50005000u, 0xf800f800u);
        const uint32_t H = g2_hfma2(__byte_perm(sw, 0x64646464u, gq & 1 ? 0x4343 : 0x4141), 0x40004000u, 0xe800e800u);
        const uint32_t L8 = g2_hmul2(L, 0x80088008u), H8 = g2_hmul2(H, 0x80808080u);   // * -2^-21, * -2^-17
        uint32_t v[32];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const uint32_t y = w[i] >> 8;
          v[2 * i] = g2_hfma2(w[i] & 0x000f000fu, L, L8); v[2 * i + 1] = g2_hfma2(y & 0x000f000fu, L, L8);
          v[16 + 2 * i] = g2_hfma2(w[i] & 0x00f000f0u, H, H8); v[17 + 2 * i] = g2_hfma2(y & 0x00f000f0u, H, H8);
        }
        if (gq == 0) {
          // the operand buffer and the accumulators are free once the last item's MMAs are done and its sums are read
          if (it > 0) {
            drain();
            if (wk.ti != ti_p) flush(ti_p);
          }
          if (!g3_reuse(NC)) store_means(abuf + 128, scA, scB, mnA, mnB);
        }
        t5_st32(abuf + 32 * gq, v);
        if (g3_reuse(NC) && gq == 3) {
          if (it == 0) stage();
          wait(half_done(g), (uint32_t)it & 1u);
          t5_fence_after();
          store_means(abuf, scA, scB, mnA, mnB);
        }
        if (gq & 1) {
          t5_wait_st();
          t5_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(a_full(g, gq >> 1));
        }
      }
      if (lane == 0) mbar_arrive_n(raw_empty(wk.slot), wk.owed(nsl));
      d_p = h2f_bits(hd.x & 0xffffu) * 524288.0f; dm_p = h2f_bits(hd.x >> 16) * 32.0f;
      ti_p = wk.ti;
      it++;
      wk.next(NG, nsl, st);
      if (!g3_reuse(NC) && it == 1) stage();
    }
    if (it > 0) { drain(); flush(ti_p); }
  } else if (warp == 4 * NG) {
    // ---- weights: lane t requests the t-th 16-row tile of every chunk ----
    int slot = 0, use = 0;
    for (int t = 0; t < my_tiles; t++) {
      int m;
      const int row0 = locate(ci + t * cps, m), have = min(8, ((a.m[m].rows + 15) >> 4) - (row0 >> 4));
      const uint8_t *src = a.m[m].W + ((size_t)((row0 >> 4) + lane) * a.nsb + sb0) * TB;
      for (int k = 0; k < nch; k++) {
        const int n = min(G3_CH, nsl - k * G3_CH);
        const uint32_t full = bar(G3_RAW_FULL + 4 * (use & 1) + slot);
        if (use > 0) wait(raw_empty(slot), (uint32_t)(use - 1) & 1u);
        // (one answer for the warp: lanes that saw the word differently would leave bytes expected that nobody requests)
        if (!__any_sync(0xffffffffu, *dead != 0)) {
          if (lane == 0) mbar_expect(full, (uint32_t)(have * n * TB));
          __syncwarp();
          if (lane < have) bulk_load(ring_s + slot * G3_STAGE + lane * (G3_CH * TB), src + (size_t)k * G3_CH * TB, (uint32_t)(n * TB), full);
        }
        __syncwarp();
        if (++slot == st) { slot = 0; use++; }
      }
    }
  } else {
    // ---- the tensor core: a warp issues a group's MMAs ----
    const int g = __shfl_sync(0xffffffffu, warp - 4 * NG - 1, 0);
    const bool el = t5_elect();
    const uint32_t ab = tmem + (uint32_t)(g * g3_a_cols(NC)), db = tmem + (uint32_t)(NG * g3_a_cols(NC) + g * g3_d_cols(NC)), mb = ab + (g3_reuse(NC) ? 0u : 128u);
    const int items = my_tiles * nsl;
    int c = g;
    uint32_t par = 0;
    for (int s = g; s < items; s += NG) {
      if (s == g) wait(xp_full, 0);
      const uint64_t bd = g3_desc(Bp_s + c * NC * 512, NC * 16, 128), md = g3_desc(Bm_s + c * NC * 32, NC * 16, 128);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        wait(a_full(g, h), par);
        t5_fence_after();
        if (el) {
#pragma unroll
          for (int k = 0; k < 8; k++) t5_mma_f16_ts(db, ab + 64 * h + 8 * k, bd + (uint64_t)((8 * h + k) * 2 * NC), g3_idesc(N), (h | k) != 0);
          if (h == 1) {
            t5_mma_f16_ts(db, mb, md, g3_idesc(N), 1);
            t5_mma_f16_ts(db + g3_p_col(NC), mb + 8, NC == 8 ? md - 8 : md, g3_idesc(N), 0);   // (128 bytes early)
            t5_commit(d_full(g));
          } else if (g3_reuse(NC)) t5_commit(half_done(g));
        }
        __syncwarp();
      }
      c += NG;
      if (c >= nsl) c -= nsl;
      par ^= 1u;
    }
  }
  // After a wait ran out: copies in flight land, and nothing of this CTA may still run on the tensor core when its tensor memory
  // is freed.  (Otherwise the workers have waited for all of both.)
  if (*dead) for (int i = 0; i < 64; i++) __nanosleep(1000);
  t5_fence_before();
  __syncthreads();
  if (warp == 0) {
    t5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}
