// gemm.cu -- host side of the dequant-fused skinny GEMMs (kernel in gemm2.cuh, its arithmetic in gemm.cuh).
#include "gemm2.cuh"
#include "gemm3.cuh"
#include "ffn_fused.cuh"
#include "moe.cuh"
#include "host.cuh"

// Can the tcgen05 kernel take this K-split?  (a super-block of every tile for each of its groups, two stages beside the planes)
// At 8 plane columns it is for launches on their own: between the small kernels of a pass, where the mma.sync kernel's ring and first
// tiles are ready when the activations come, it is the slower one (27B shape, 24 cycles of four rows 143.6 ms without it, 151 with
// it; 24 passes of one row 121.7 and 123.4), alone the faster (gate|up at four rows 27.5 and 27.4 us, at one 27.0 and 25.4).
static bool g3_fits(int fmt, int NC, int nsb, int ks, bool alone) {
  if (g_llb.gemm3 == 0 || fmt != LLB_FM_Q4_K || (NC == 8 && !alone && g_llb.gemm3 == 2)) return false;
  return ks >= 1 && nsb / ks >= g3_groups(NC) && g3_stages(NC, (nsb + ks - 1) / ks) >= 2;
}
static unsigned int *g_ffn_sync = nullptr;   // the fused FFN's grid barrier: two counters
static unsigned int *g_g3_err = nullptr;   // device word: set when a bounded wait of a kernel ran out
unsigned int *gemm_err_word(void) { return g_g3_err; }
// Cost model of a launch, in cycles of one SM.  The work of its tiles is about 45 + 6.3 cycles a plane column and
// 16 x 256 tile, 65 + for Q5_K with its fifth bits (measured with the copies left out on the 27B shape's gate|up launch at 4, 8 and 16 rows); a warp's own
// chain, where that is longer, about 1200 cycles a tile (two stages of copies in flight), with 350 for adding up the parts of
// a row tile that warps share (each of them where per_tile is the operator's).  nc: plane columns that are multiplied
static double gemm_stream_cost(int fmt, int warps, int nc, int tiles, int slice, int parts, double per_tile = 1200.0) {
  const int rounds = (tiles * parts + warps - 1) / warps;
  const double work = (double)tiles * slice * ((fmt == LLB_FM_Q5_K ? 65.0 : 45.0) + 6.3 * nc), chain = rounds * ((slice + parts - 1) / parts * per_tile + (per_tile > 1200.0 ? 350.0 * (parts - 1) : parts > 1 ? 350.0 : 0.0));
  return work > chain ? work : chain;
}
// Parts of a row tile's K-slice (g2_phase): the power of two with the lowest cost that divides the warps, leaves every part a
// super-block and whose sums fit beside the activation slice.  tiles: row tiles of a CTA, nsb in ks slices
static int gemm_pick_parts(int fmt, int NC, int tiles, int nsb, int ks) {
  const int warps = g2_warps(fmt, NC), slice = (nsb + ks - 1) / ks, ring = g2_ring_of(fmt, NC, slice);
  int best = 1;
  for (int p = 2; p <= 16 && p <= nsb / ks && warps % p == 0; p *= 2)
    if (g2_smem(fmt, slice, NC, p, ring) <= G2_SMEM_MAX && gemm_stream_cost(fmt, warps, NC, tiles, slice, p) < gemm_stream_cost(fmt, warps, NC, tiles, slice, best)) best = p;
  return best;
}
template <int FMT, int NT> static int launch_two(cudaStream_t s, GemmArgs &a) {
  const int NC = 8 * NT, nsl = (a.nsb + a.ksplit - 1) / a.ksplit;
  int cps = g_llb.sms / a.ksplit;
  if (cps < 1) cps = 1;
  // every SM takes part as long as there is a tile for it: the tiles are dealt out one per CTA in turn
  if (cps > a.tile0[a.nmat]) cps = a.tile0[a.nmat];
  a.parts = gemm_pick_parts(FMT, NC, (a.tile0[a.nmat] + cps - 1) / cps, a.nsb, a.ksplit);
  const int ring = g2_ring_of(FMT, NC, nsl);
  const size_t smem = g2_smem(FMT, nsl, NC, a.parts, ring);
  if (smem > G2_SMEM_MAX) return llb_fail("k_gemm2: a K-slice of %d super-blocks needs %zu bytes of shared memory", nsl, smem);
  const bool fold = (long long)a.tile0[a.nmat] * a.nsb >= G2_FOLD_TILES;
  constexpr int RS = g2_small_ring(FMT, 8 * NT);
  cudaError_t e = llb_launch(ring ? k_gemm2<FMT, NT, false, RS ? RS : g2_has_short(FMT, 8 * NT)> : fold && g2_folds(FMT, NT) ? k_gemm2<FMT, NT, g2_folds(FMT, NT), 0> : k_gemm2<FMT, NT, false, RS>,
                             dim3(cps * a.ksplit), dim3(g2_warps(FMT, NC) * 32), smem, s, a, cps);
  if (e != cudaSuccess) return llb_fail("k_gemm2 launch: %s", cudaGetErrorString(e));
  return 0;
}

template <int NC> static int launch_three(cudaStream_t s, const GemmArgs &a) {
  const int nsl = (a.nsb + a.ksplit - 1) / a.ksplit, st = g3_stages(NC, nsl);
  int ntiles = 0;
  for (int i = 0; i < a.nmat; i++) ntiles += (a.m[i].rows + 127) / 128;
  int cps = g_llb.sms / a.ksplit;
  if (cps < 1) cps = 1;
  if (cps > ntiles) cps = ntiles;
  const size_t smem = (size_t)G3_HDR + g3_xp_bytes(NC, nsl) + g3_red_bytes(NC) + (size_t)st * G3_STAGE;
  cudaError_t e = llb_launch(k_gemm3<NC>, dim3(cps * a.ksplit), dim3(g3_threads(NC)), smem, s, a, cps, st);
  if (e != cudaSuccess) return llb_fail("k_gemm3 launch: %s", cudaGetErrorString(e));
  return 0;
}
// What one agent of a CTA of k_gemm3 does with the CTA's barriers, in its order: a warp of group `agent`, behind the groups the warp
// that requests the weights, then a group's issuing warp.  ops: {0 wait, barrier, phase}, {1 arrive, barrier, times}, {2 arrive, barrier,
// once a copy requested here has landed or an MMA issued here is done}.  Returns their number, -1 where the kernel takes no such slice.
int gemm3_trace(int NC, int nsl, int tiles, int agent, int *ops, int cap) {
  const int NG = g3_groups(NC), st = g3_stages(NC, nsl);
  if ((NC != 8 && NC != 16 && NC != 32) || nsl < NG || st < 2 || tiles < 1 || agent < 0 || agent > 2 * NG) return -1;
  int n = 0;
  auto op = [&](int kind, int b, int v) { if (3 * n + 2 < cap) { ops[3 * n] = kind; ops[3 * n + 1] = b; ops[3 * n + 2] = v; } n++; };
  if (agent < NG) {
    G3Walk wk;
    int it = 0, ti_p = 0;
    auto flush = [&](int t) {
      const G3Sum sm = g3_sum(NC, nsl, t);
      if (sm.n > 0) op(0, G3_RED_EMPTY + sm.p, sm.n - 1);
      if (agent != sm.owner) op(1, G3_RED_FULL + sm.p, 1);
      else { op(0, G3_RED_FULL + sm.p, sm.n); op(1, G3_RED_EMPTY + sm.p, 1); }
    };
    for (wk.start(agent, st); wk.ti < tiles; wk.next(NG, nsl, st)) {
      op(0, wk.full(), wk.phase());
      if (it > 0) { op(0, G3_D_FULL + agent, it - 1); if (wk.ti != ti_p) flush(ti_p); }
      ti_p = wk.ti;
      op(1, G3_A_FULL + 2 * agent, 1);
      if (g3_reuse(NC)) { if (it == 0) op(1, G3_XP_FULL, 32); op(0, G3_HALF + agent, it); }
      op(1, G3_A_FULL + 2 * agent + 1, 1);
      op(1, G3_RAW_EMPTY + wk.slot, wk.owed(nsl));
      if (it++ == 0 && !g3_reuse(NC)) op(1, G3_XP_FULL, 32);
    }
    op(0, G3_D_FULL + agent, it - 1);
    flush(ti_p);
  } else if (agent == NG) {
    const int nch = (nsl + G3_CH - 1) / G3_CH;
    for (int k = 0; k < tiles * nch; k++) {
      const int slot = k % st, use = k / st;
      if (use > 0) op(0, G3_RAW_EMPTY + slot, use - 1);
      op(2, G3_RAW_FULL + 4 * (use & 1) + slot, 1);
    }
  } else {
    const int g = agent - NG - 1;
    for (int s = g, k = 0; s < tiles * nsl; s += NG, k++) {
      if (k == 0) op(0, G3_XP_FULL, 0);
      op(0, G3_A_FULL + 2 * g, k);
      if (g3_reuse(NC)) op(2, G3_HALF + g, 1);
      op(0, G3_A_FULL + 2 * g + 1, k);
      op(2, G3_D_FULL + g, 1);
    }
  }
  return n;
}
int gemm3_bar_count(int NC, int b) { return (NC != 8 && NC != 16 && NC != 32) || b < 0 || b >= G3_BARS ? -1 : g3_bar_count(NC, b); }

// 1 when a bounded wait of the tcgen05 kernel or of the fused FFN's barrier has run out since the library was
// initialised (or since the word was last cleared)
int gemm_wait_errors(void) {
  unsigned int v = 0;
  if (g_g3_err && cudaMemcpy(&v, g_g3_err, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return (int)v;
}
int gemm_wait_errors_clear(void) {
  if (g_g3_err) CU_OK(cudaMemset(g_g3_err, 0, 4));
  return 0;
}

// The two device-side waits of this file, each made to run out on purpose with a small limit: an mbarrier nobody
// arrives on (the wait of k_gemm3 and k_pfmm, tc5.cuh) and the fused FFN's grid barrier told to expect one block more
// than the launch has.  One block, one waiting thread; the wait gives up after `limit` tries, sets the error word
// exactly as in the real kernels and the kernel returns.  which = 2: the skinny GEMM's ring with a stage that was never
// requested and two that were.  The wait for the first runs out; the drain must leave nothing in flight, or the word reads 2.
__global__ void k_wait_selftest(int which, unsigned int limit, unsigned int *sync, unsigned int *err) {
  __shared__ __align__(8) uint64_t bar;
  if (which == 2) {
    __shared__ __align__(128) uint8_t mem[G2_BAR_BYTES + 3 * 4096];
    G2Ring r = g2_ring_init(mem, 3 * 4096);
    if (threadIdx.x == 0)
      for (int s = 1; s < 3; s++) { mbar_expect(r.bar_s + 8 * s, 4096); bulk_load(r.ring_s + s * 4096, sync, 4096, r.bar_s + 8 * s); }
    __syncwarp();
    for (int s = 0; s < 3; s++) g2_wait(r, s, limit, err);
    g2_drain(r);
    if (!r.dead || !mbar_wait(r.bar_s + 8, 0, 1) || !mbar_wait(r.bar_s + 16, 0, 1)) atomicExch(err, 2u);
    return;
  }
  if (which == 0) {
    const uint32_t bar_s = smem_u32(&bar);
    if (threadIdx.x == 0) {
      mbar_init(bar_s, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(bar_s, 0, limit)) atomicExch(err, 1u);
  } else {
    ffn_grid_sync(sync, 2u, err, limit);
    if (threadIdx.x == 0) { sync[0] = 0; sync[1] = 0; }   // the block that never came would have reset them
  }
}
int gemm_wait_selftest(cudaStream_t s, int which, int limit) {
  if (which < 0 || which > 2 || limit < 1 || limit > 100000) return llb_fail("wait selftest: which 0..2, limit 1..100000");
  unsigned int *sync = nullptr;
  CU_OK(cudaMalloc(&sync, 4096));        // a private pair of counters: the barrier of real launches is not touched; 4 KB to copy from
  CU_OK(cudaMemsetAsync(sync, 0, 4096, s));
  k_wait_selftest<<<1, 32, 0, s>>>(which, (unsigned int)limit, sync, g_g3_err);
  CU_OK(cudaGetLastError());
  CU_OK(cudaStreamSynchronize(s));
  CU_OK(cudaFree(sync));
  return 0;
}

template <typename K> static int setup_smem(K k) {
  CU_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, G2_SMEM_MAX));
  return 0;
}
template <int FMT, int NT> static int setup_fmt2() {
  constexpr int RS = g2_small_ring(FMT, 8 * NT);
  return setup_smem(k_gemm2<FMT, NT, false, RS>) || setup_smem(k_gemm2<FMT, NT, g2_folds(FMT, NT), 0>) || setup_smem(k_gemm2<FMT, NT, false, RS ? RS : g2_has_short(FMT, 8 * NT)>);
}
template <int FMT> static int setup_fmt() { return setup_fmt2<FMT, 1>() || setup_fmt2<FMT, 2>() || setup_fmt2<FMT, 4>(); }
template <int FMT> static int setup_experts() { return setup_smem(k_moe_gu<FMT, 8>) || setup_smem(k_moe_gu<FMT, 32>) || setup_smem(k_moe_dn<FMT>); }

template <int NC> static int setup_three() {
  CU_OK(cudaFuncSetAttribute(k_gemm3<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, G3_SMEM_MAX));
  return 0;
}

int gemm_setup(void) {
  if (setup_fmt<LLB_FM_Q4_K>() || setup_fmt<LLB_FM_Q5_K>() || setup_fmt<LLB_FM_Q6_K>() || setup_fmt<LLB_FM_Q8_0>()) return -1;
  if (setup_three<8>() || setup_three<16>() || setup_three<32>()) return -1;
  if (setup_experts<LLB_FM_Q4_K>() || setup_experts<LLB_FM_Q5_K>() || setup_experts<LLB_FM_Q6_K>()) return -1;
  CU_OK(cudaFuncSetAttribute(k_ffn<LLB_FM_Q4_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, G2_SMEM_MAX));
  CU_OK(cudaFuncSetAttribute(k_ffn<LLB_FM_Q5_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, G2_SMEM_MAX));
  CU_OK(cudaFuncSetAttribute(k_ffn<LLB_FM_Q6_K>, cudaFuncAttributeMaxDynamicSharedMemorySize, G2_SMEM_MAX));
  if (!g_ffn_sync) {
    CU_OK(cudaMalloc(&g_ffn_sync, 8));
    CU_OK(cudaMemset(g_ffn_sync, 0, 8));
  }
  if (!g_g3_err) {
    CU_OK(cudaMalloc(&g_g3_err, 4));
    CU_OK(cudaMemset(g_g3_err, 0, 4));
  }
  return 0;
}

// the fewest K-slices that the mma.sync kernel can take: the activation slice of a CTA has to fit in shared memory, beside the usual
// ring, or where that would take too many slices, beside the shorter one
static int g2_least_ksplit(int fmt, int NC, int nsb) {
  const int mx = g2_max_slice_sb(fmt, NC), most = g2_longest_slice(fmt, NC), lo = (nsb + mx - 1) / mx;
  return lo <= GEMM_MAXSPLIT ? lo : (nsb + most - 1) / most;
}
int gemm_fix_ksplit(int fmt, int NC, int nsb, int ks, bool alone) {
  if (ks < 1) ks = 1;
  if (!g3_fits(fmt, NC, nsb, ks, alone)) {
    const int least = g2_least_ksplit(fmt, NC, nsb);
    if (ks < least) ks = least;
  }
  if (ks > GEMM_MAXSPLIT) ks = GEMM_MAXSPLIT;
  if (ks > nsb) ks = nsb;
  return ks;
}

// (the fewest slices that either kernel takes, held against the room of the kernel that takes them)
bool gemm_fits(int fmt, int NC, int nsb, int cap) {
  const int ks = gemm_fix_ksplit(fmt, NC, nsb, 1);
  return ks <= cap && (g3_fits(fmt, NC, nsb, ks, false) || (nsb + ks - 1) / ks <= g2_longest_slice(fmt, NC));
}

// K-slices per row tile: streaming, the staging of the slice (24 cycles a plane column of a super-block), and a charge per slice for the partial sums that the consumer
// has to add (direct: a launch of its own adds them, 1.5 us).  At 32 plane columns a warp's chain is nearer 3000 cycles a tile
// (fitted on fifteen shapes, four formats, one to eight slices; with 1200 the operator's choices were 4.5 % off the best of those,
// now 1 %: Q4_K 8192 x 3072 at sixteen rows 18.0 -> 15.8 us, 5120 x 5120 18.5 -> 15.9).  The operator alone goes by it: a
// split decides the order of a model's sums, and the passes were timed with the splits they have.
static double gemm_split_cost(int fmt, int NC, int ntiles, int nsb, int ks, int sms, bool direct) {
  const int cps = sms / ks > 0 ? sms / ks : 1, slice = (nsb + ks - 1) / ks, tiles = (ntiles + cps - 1) / cps;
  const double stream = gemm_stream_cost(fmt, g2_warps(fmt, NC), NC, tiles, slice, gemm_pick_parts(fmt, NC, tiles, nsb, ks), direct && NC >= 32 ? 3000.0 : 1200.0);
  return (stream + 24.0 * NC * slice) * (1.0 + 0.02 * (ks - 1)) + 25.0 * NC * (ks - 1) + (direct && ks > 1 ? 3000.0 : 0.0);
}
// The tcgen05 kernel's cost on the same scale, in a pass: a super-block of 128 rows in a CTA, a tile's way out, the slice's activations, the
// pipeline's fill -- times 0.7, because that scale flatters the other kernel (27B shape, a prompt of 48 tokens in passes of eight rows
// 51.7 ms without the kernel, 49.2 with this factor 1, 48.5 with 0.7; ten cycles of sixteen rows 125.2, 114.6, 114.2).
// 4000 cycles more: its first MMA waits for all activations, and what the mma.sync kernel has ready by then is worth that much.
static double g3_cost(int NC, int ntiles, int nsb, int ks, int sms) {
  const int cps = sms / ks > 0 ? sms / ks : 1, slice = (nsb + ks - 1) / ks, tiles = ((ntiles + 7) / 8 + cps - 1) / cps;
  const double sb = NC >= 32 ? 970.0 : 820.0;
  return 0.7 * (tiles * (slice * sb + 900.0) * (1.0 + 0.02 * (ks - 1)) + 4000.0 + 12.0 * NC * slice) + 25.0 * NC * (ks - 1) + 4000.0;
}
// Microseconds of the operator's launch and its sums with either kernel, for a width's most rows (the choice may not depend on the
// rows: a row's bits do not).  Fitted on 56 shapes of 4 to 68 super-blocks and 512 to 40000 rows, 148 SMs, weights cold, every K-split: half
// of the launches within 5 %, nine in ten within 12 %.  The scale of gemm_split_cost, whose costs the passes go by, is too kind to the
// tcgen05 kernel here by up to a third: 6144 x 5120 at eight rows went there and took 12.9 us for 10.7, 17408 x 5120 at four 17.6 for 15.6.
static double g3_us(int NC, int ntiles, int nsb, int ks, int sms) {
  static const double c[3][6] = {{2.24, 0.0324, 0.1108, 0.87, 1.94, 0.1536}, {2.38, 0.0327, 0.1378, 0.86, 1.27, 0.1711}, {3.16, 0.0225, 0.1268, 1.10, 0.86, 0.2106}};
  const double *k = c[NC / 16];
  const int cps = sms / ks > 0 ? sms / ks : 1, slice = (nsb + ks - 1) / ks, tiles = ((ntiles + 7) / 8 + cps - 1) / cps;
  return k[0] + k[1] * NC * slice + k[2] * tiles * slice + (ks > 1 ? k[3] + k[4] * 32e-6 * NC * ks * ntiles : 0.0) + k[5] * 2304e-6 * ntiles * nsb;
}
static double g2_us(int NC, int ntiles, int nsb, int ks, int sms) {
  static const double c[3][9] = {{1.76, 0.0089, 0.0319, 0.0406, 0.196, 0.87, 0.75, 0.1295, 0.4115}, {1.75, 0.0169, 0.0474, 0.1672, 0.0, 1.27, 0.86, 0.1168, 0.2108}, {2.59, 0.0122, 0.0451, 0.8476, 0.0, 0.97, 1.02, 0.0930, 0.0}};
  const double *k = c[NC / 16];
  int cps = sms / ks > 0 ? sms / ks : 1;
  if (cps > ntiles) cps = ntiles > 0 ? ntiles : 1;
  const int slice = (nsb + ks - 1) / ks, tiles = (ntiles + cps - 1) / cps, p = gemm_pick_parts(LLB_FM_Q4_K, NC, tiles, nsb, ks), w = g2_warps(LLB_FM_Q4_K, NC);
  const int rounds = (tiles * p + w - 1) / w;
  return k[0] + k[1] * NC * slice + k[2] * tiles * slice + k[3] * rounds * ((slice + p - 1) / p) + (p > 1 ? k[4] * rounds : 0.0) + (ks > 1 ? k[5] + k[6] * 32e-6 * NC * ks * ntiles : 0.0) +
         k[7] * 2304e-6 * ntiles * nsb + k[8] * rounds;
}
// Whether the tcgen05 kernel in k3 slices is the operator's choice over the other in k2: where it is faster by more than the fit is off at
// shapes that are near.  At 8 plane columns, where the two are, a slice more counts 0.3 us.  Of the 56 shapes eleven, sixteen and forty-six
// change kernels at 8, 16 and 32 columns; none is more than 3.7 % slower for it, on average they are 1.6, 3.3 and 16 % faster.
static bool g3_better(int NC, int ntiles, int nsb, int k3, int k2, int sms) {
  const double slice = NC == 8 ? 0.3 : 0.0, margin = NC == 8 ? 0.97 : NC == 16 ? 0.95 : 0.96;
  return g3_us(NC, ntiles, nsb, k3, sms) + slice * k3 < margin * (g2_us(NC, ntiles, nsb, k2, sms) + slice * k2);
}
// Which kernel a launch takes at this K-split: the tcgen05 one where it can and costs less (or has been asked for).
static bool g3_use(int fmt, int NC, int ntiles, int nsb, int ks, int sms, bool alone) {
  if (!g3_fits(fmt, NC, nsb, ks, alone)) return false;
  if (g_llb.gemm3 == 1 || ks < g2_least_ksplit(fmt, NC, nsb)) return true;
  if (alone) return g3_better(NC, ntiles, nsb, ks, ks, sms);
  return g3_cost(NC, ntiles, nsb, ks, sms) < gemm_split_cost(fmt, NC, ntiles, nsb, ks, sms, false);
}
// The operator's K-slices where the caller names none, and in *g3 its kernel: each kernel's own best, then the better of the two.
static int gemm_pick_alone(int fmt, int NC, int ntiles, int nsb, int sms, bool *g3) {
  const int least = g2_least_ksplit(fmt, NC, nsb);
  int k2 = 0, k3 = 0;
  double c2 = 0.0, c3 = 0.0;
  for (int ks = 1; ks <= GEMM_MAXSPLIT && ks <= nsb; ks++) {
    if (ks >= least) {
      const double c = gemm_split_cost(fmt, NC, ntiles, nsb, ks, sms, true);
      if (!k2 || c < c2 - 1e-9) { k2 = ks; c2 = c; }
    }
    if (g3_fits(fmt, NC, nsb, ks, true)) {
      const double c = g3_us(NC, ntiles, nsb, ks, sms) + (NC == 8 ? 0.3 : 0.0) * ks;
      if (!k3 || c < c3) { k3 = ks; c3 = c; }
    }
  }
  *g3 = k3 && (!k2 || g_llb.gemm3 == 1 || g3_better(NC, ntiles, nsb, k3, k2, sms));
  return *g3 ? k3 : k2 ? k2 : gemm_fix_ksplit(fmt, NC, nsb, 1, true);
}
int gemm_pick_ksplit(int fmt, int NC, int ntiles, int nsb, int sms) {
  int best = 1;
  double best_cost = 1e30;
  for (int ks = 1; ks <= GEMM_MAXSPLIT && ks <= nsb; ks++) {
    if (gemm_fix_ksplit(fmt, NC, nsb, ks) != ks) continue;
    if (g_llb.gemm3 == 1 && best_cost < 1e30 && !g3_fits(fmt, NC, nsb, ks, false) && g3_fits(fmt, NC, nsb, best, false)) continue;
    const double cost = g3_use(fmt, NC, ntiles, nsb, ks, sms, false) ? g3_cost(NC, ntiles, nsb, ks, sms) : gemm_split_cost(fmt, NC, ntiles, nsb, ks, sms, false);
    // (the tcgen05 kernel asked for: before any split that it cannot take comes one that it can)
    const bool asked = g_llb.gemm3 == 1 && g3_fits(fmt, NC, nsb, ks, false) && !g3_fits(fmt, NC, nsb, best, false);
    if (cost < best_cost - 1e-9 || asked) { best_cost = cost; best = ks; }
  }
  return gemm_fix_ksplit(fmt, NC, nsb, best);
}

int gemm_which(int fmt, int NC, int ntiles, int nsb, int sms, bool alone, int *ksplit) {
  bool g3 = false;
  if (alone && *ksplit <= 0) {
    // (the choice costs 1.5 us of a call of 9, and depends on nothing but these: a thread keeps its last ones)
    struct Kept { int fmt, NC, ntiles, nsb, sms, mode, ks; bool g3; };
    static thread_local Kept kept[64];
    const int mode = g_llb.gemm3;
    Kept &e = kept[((unsigned)ntiles * 31u + (unsigned)nsb * 7u + (unsigned)fmt * 3u + (unsigned)NC) & 63u];
    if (e.ks < 1 || e.fmt != fmt || e.NC != NC || e.ntiles != ntiles || e.nsb != nsb || e.sms != sms || e.mode != mode) {
      e = Kept{fmt, NC, ntiles, nsb, sms, mode, 0, false};
      e.ks = gemm_pick_alone(fmt, NC, ntiles, nsb, sms, &e.g3);
    }
    *ksplit = e.ks; g3 = e.g3;
  } else {
    *ksplit = gemm_fix_ksplit(fmt, NC, nsb, *ksplit > 0 ? *ksplit : gemm_pick_ksplit(fmt, NC, ntiles, nsb, sms), alone);
    g3 = g3_use(fmt, NC, ntiles, nsb, *ksplit, sms, alone);
  }
  return g3 ? 3 : 2;
}

// One K-split for a launch whose partial sums outlive the pass (attn_qkv into the conv ring): valid at both
// plane widths in use, the cost model's choice at the speculative width where that fits, at most `cap`.
// Returns 0 when no split up to `cap` fits both widths.
int gemm_ring_ksplit(int fmt, int nsb, int ntiles, int nc_spec, int nc_pf, int sms, int cap) {
  const int lo_a = gemm_fix_ksplit(fmt, nc_spec, nsb, 1), lo_b = gemm_fix_ksplit(fmt, nc_pf, nsb, 1);
  const int lo = lo_a > lo_b ? lo_a : lo_b;
  if (cap > nsb) cap = nsb;
  if (lo > cap) return 0;
  int ks = gemm_pick_ksplit(fmt, nc_spec, ntiles, nsb, sms);
  if (ks < lo) ks = lo;
  if (ks > cap) ks = cap;
  return ks;
}

// fills nsb and the tile table of a launch and checks its shape
static int gemm_prepare(int fmt, GemmArgs &a, bool fused = false) {
  if (a.nmat < 1 || a.nmat > GEMM_MAXMAT) return llb_fail("gemm: nmat %d", a.nmat);
  if (a.K % 256) return llb_fail("gemm: K %d is not a multiple of 256", a.K);
  if (a.xp.NC != 8 && a.xp.NC != 16 && a.xp.NC != 32) return llb_fail("gemm: NC %d", a.xp.NC);
  if (a.xp.K != a.K) return llb_fail("gemm: planes hold %d columns, K is %d", a.xp.K, a.K);
  a.err = g_g3_err;
  a.nsb = a.K / 256;
  a.tile0[0] = 0;
  for (int i = 0; i < a.nmat; i++) a.tile0[i + 1] = a.tile0[i] + (a.m[i].rows + 15) / 16;
  for (int i = a.nmat; i < GEMM_MAXMAT; i++) a.tile0[i + 1] = a.tile0[a.nmat];
  if (!fused && a.ksplit != gemm_fix_ksplit(fmt, a.xp.NC, a.nsb, a.ksplit, a.alone)) return llb_fail("gemm: ksplit %d is not valid for this shape", a.ksplit);
  return 0;
}

// ---- the fused FFN launch (ffn_fused.cuh) ------------------------------------------------------
// shared memory of the launch: the ring, and the larger of gate|up's planes (nsb1 super-blocks) and a down slice's (nsl2)
static size_t ffn_smem(int fmt2, int nsb1, int nsl2) {
  const size_t s1 = g2_smem(LLB_FM_Q4_K, nsb1, 8, 1, 1), s2 = g2_smem(fmt2, nsl2, 8, 1, 1) - g2_ring_bytes(fmt2, 8, 1) + FFN_RING;
  return s1 > s2 ? s1 : s2;
}
template <int FMT2> static int launch_ffn(cudaStream_t s, const GemmArgs &a1, const GemmArgs &a2) {
  int cps1 = g_llb.sms, cps2 = g_llb.sms / a2.ksplit;
  if (cps1 > a1.tile0[a1.nmat]) cps1 = a1.tile0[a1.nmat];
  if (cps2 < 1) cps2 = 1;
  if (cps2 > a2.tile0[a2.nmat]) cps2 = a2.tile0[a2.nmat];
  const int grid = cps1 > cps2 * a2.ksplit ? cps1 : cps2 * a2.ksplit;
  if (grid > g_llb.sms) return llb_fail("k_ffn: %d CTAs do not fit %d SMs", grid, g_llb.sms);   // the barrier needs them all resident
  const size_t smem = ffn_smem(FMT2, a1.nsb, (a2.nsb + a2.ksplit - 1) / a2.ksplit);
  if (smem > G2_SMEM_MAX) return llb_fail("k_ffn: %zu bytes of shared memory", smem);
  cudaError_t e = llb_launch(k_ffn<FMT2>, dim3(grid), dim3(512), smem, s, a1, a2, cps1, cps2, g_ffn_sync, g_g3_err);
  if (e != cudaSuccess) return llb_fail("k_ffn launch: %s", cudaGetErrorString(e));
  return 0;
}
// Can the FFN of these formats and widths run as one launch?  (gate|up in one K-slice, T <= 4.)  ks2: the down phase's K-split
bool gemm_ffn_fusable(int fmt_gu, int fmt_dn, int NC, int d, int f, int *ks2) {
  if (!g_llb.ffn_fused || !g_ffn_sync || NC != 8 || fmt_gu != LLB_FM_Q4_K || d % 256 || f % 256) return false;
  if (fmt_dn != LLB_FM_Q4_K && fmt_dn != LLB_FM_Q5_K && fmt_dn != LLB_FM_Q6_K) return false;
  *ks2 = gemm_fix_ksplit(fmt_dn, NC, f / 256, gemm_pick_ksplit(fmt_dn, NC, d / 16, f / 256, g_llb.sms));
  return ffn_smem(fmt_dn, d / 256, (f / 256 + *ks2 - 1) / *ks2) <= G2_SMEM_MAX;
}
// a1: gate and up (two matrices, Q4_K, ksplit 1, outputs complete); a2: down in format fmt2 with its own K-split
int gemm_launch_ffn(cudaStream_t s, GemmArgs &a1, int fmt2, GemmArgs &a2) {
  if (a1.nmat != 2 || a1.ksplit != 1 || a2.nmat != 1 || a1.xp.NC != 8 || a2.xp.NC != 8) return llb_fail("k_ffn: unsupported launch shape");
  if (gemm_prepare(LLB_FM_Q4_K, a1, true) || gemm_prepare(fmt2, a2, true)) return -1;
  a1.parts = a2.parts = 1;
  if (a2.K != a1.m[0].rows || a1.m[1].rows != a1.m[0].rows) return llb_fail("k_ffn: down takes %d columns, gate/up have %d/%d rows", a2.K, a1.m[0].rows, a1.m[1].rows);
  if (fmt2 == LLB_FM_Q4_K) return launch_ffn<LLB_FM_Q4_K>(s, a1, a2);
  if (fmt2 == LLB_FM_Q5_K) return launch_ffn<LLB_FM_Q5_K>(s, a1, a2);
  if (fmt2 == LLB_FM_Q6_K) return launch_ffn<LLB_FM_Q6_K>(s, a1, a2);
  return llb_fail("k_ffn: down format %d", fmt2);
}

// ---- the routed experts' GEMMs (moe.cuh) ---------------------------------------------------------
// Shape of a launch of `units` units at most (tpu tiles of nsl super-blocks each), with `sel` bytes in front of the planes: CTAs,
// parts of a row tile, the rings, and how many units are staged at a time -- all that a CTA meets where they fit.  It depends on the
// pass's capacity, not on the rows in use or their experts: a row's sums do not depend on its neighbours.
struct MoeShape { int cps, parts, st, ch, ub; size_t smem; };
static bool moe_shape(int fmt, int units, int tpu, int nsl, int sel, MoeShape &o) {
  const long long tiles = (long long)units * tpu;
  o.cps = tiles < g_llb.sms ? (int)tiles : g_llb.sms;
  const int mine = (int)((tiles + o.cps - 1) / o.cps), need = mine / tpu + 2 < units ? mine / tpu + 2 : units;
  o.parts = 1;
  for (int p = 2; p <= MOE_WARPS && p <= nsl; p *= 2)
    if (gemm_stream_cost(fmt, MOE_WARPS, 8, mine, nsl, p) < gemm_stream_cost(fmt, MOE_WARPS, 8, mine, nsl, o.parts)) o.parts = p;
  static const int rings[4][2] = {{2, 2}, {3, 1}, {2, 1}, {1, 1}};
  for (o.ub = need < 4 ? need : 4; o.ub >= 1; o.ub--)
    for (int r = fmt == LLB_FM_Q4_K ? 0 : 1; r < (o.ub > 1 ? 3 : 4); r++) {
      o.st = rings[r][0]; o.ch = rings[r][1];
      o.smem = G2_BAR_BYTES + (size_t)MOE_WARPS * o.st * o.ch * tile_bytes(fmt) + sel + (size_t)o.ub * moe_unit_bytes(fmt, nsl) + (o.parts > 1 ? MOE_WARPS * 512 : 0);
      if (o.smem <= G2_SMEM_MAX) return true;
    }
  return false;
}
static int moe_check(int fmt, const MoeArgs &m) {
  if (fmt != LLB_FM_Q4_K && fmt != LLB_FM_Q5_K && fmt != LLB_FM_Q6_K) return llb_fail("moe gemm: expert stacks of format %d have no kernel", fmt);
  if (m.ef % 256 || m.d % 256) return llb_fail("moe gemm: widths %d, %d are not multiples of 256", m.ef, m.d);
  if (m.T < 1 || m.T > MOE_MAXROWS || m.ne < 1 || m.ne > 1024 || m.nslot < 2 || m.nslot > 33 || m.nslot - 1 > m.ne) return llb_fail("moe gemm: %d rows, %d experts, top %d", m.T, m.ne, m.nslot - 1);
  return 0;
}
static void moe_gemm_args(GemmArgs &a, int K, int ks, const MoeArgs &m, const MoeShape &o) {
  memset(&a, 0, sizeof a);
  a.K = K; a.nsb = K / 256; a.ksplit = ks; a.parts = o.parts; a.planes = 2; a.T = m.T; a.err = g_g3_err;
}
// the choice, then gate|up of every unit on planes of d columns (whole sums: one K-slice)
int gemm_launch_moe_gu(cudaStream_t s, int fmt, const XPlanes &xp, const MoeArgs &m) {
  if (moe_check(fmt, m)) return -1;
  if (xp.K != m.d) return llb_fail("moe gemm: planes of %d columns, the experts take %d", xp.K, m.d);
  MoeShape o;
  if (!moe_shape(fmt, m.T * m.nslot, m.ef / 8, m.d / 256, moe_sel_bytes(m.T * m.nslot), o)) return llb_fail("moe gemm: %d columns do not fit one K-slice", m.d);
  GemmArgs a;
  moe_gemm_args(a, m.d, 1, m, o);
  a.xp = xp;
  const bool wide = m.ne > 256;
#define MOE_GO(F) CU_OK(llb_launch(wide ? k_moe_gu<F, 32> : k_moe_gu<F, 8>, dim3(o.cps), dim3(MOE_WARPS * 32), o.smem, s, a, m, o.st, o.ch, o.ub))
  if (fmt == LLB_FM_Q4_K) MOE_GO(LLB_FM_Q4_K);
  else if (fmt == LLB_FM_Q5_K) MOE_GO(LLB_FM_Q5_K);
  else MOE_GO(LLB_FM_Q6_K);
#undef MOE_GO
  return 0;
}
// K-slices of an expert's ef columns in the down launch: one, or where a unit's activations do not fit the fewest equal ones that do
int gemm_moe_dn_ksplit(int fmt, const MoeArgs &m) {
  MoeShape o;
  for (int ks = 1; ks <= m.ef / 256; ks++)
    if (m.ef / 256 % ks == 0 && moe_shape(fmt, m.T * m.nslot * ks, m.d / 16, m.ef / 256 / ks, m.T * m.nslot * 16, o)) return ks;
  return 0;
}
// the units' down matrices on wt * silu(g) * u; slice slot * ks + k of m.out is K-slice k of that slot
int gemm_launch_moe_dn(cudaStream_t s, int fmt, const MoeArgs &m, int ks) {
  if (moe_check(fmt, m)) return -1;
  MoeShape o;
  if (ks < 1 || m.ef / 256 % ks || !moe_shape(fmt, m.T * m.nslot * ks, m.d / 16, m.ef / 256 / ks, m.T * m.nslot * 16, o)) return llb_fail("moe gemm: %d K-slices of %d columns", ks, m.ef);
  GemmArgs a;
  moe_gemm_args(a, m.ef, ks, m, o);
#define MOE_GO(F) CU_OK(llb_launch(k_moe_dn<F>, dim3(o.cps), dim3(MOE_WARPS * 32), o.smem, s, a, m, o.st, o.ch, o.ub))
  if (fmt == LLB_FM_Q4_K) MOE_GO(LLB_FM_Q4_K);
  else if (fmt == LLB_FM_Q5_K) MOE_GO(LLB_FM_Q5_K);
  else MOE_GO(LLB_FM_Q6_K);
#undef MOE_GO
  return 0;
}

int gemm_launch(cudaStream_t s, int fmt, GemmArgs &a) {
  if (gemm_prepare(fmt, a)) return -1;
  if (a.tile0[a.nmat] < 1) return 0;
  const int NT = a.xp.NC / 8;
  if (a.alone ? a.g3 : g3_use(fmt, a.xp.NC, a.tile0[a.nmat], a.nsb, a.ksplit, g_llb.sms, false)) return NT == 1 ? launch_three<8>(s, a) : NT == 2 ? launch_three<16>(s, a) : launch_three<32>(s, a);
  if (fmt == LLB_FM_Q4_K) return NT == 1 ? launch_two<LLB_FM_Q4_K, 1>(s, a) : NT == 2 ? launch_two<LLB_FM_Q4_K, 2>(s, a) : launch_two<LLB_FM_Q4_K, 4>(s, a);
  if (fmt == LLB_FM_Q5_K) return NT == 1 ? launch_two<LLB_FM_Q5_K, 1>(s, a) : NT == 2 ? launch_two<LLB_FM_Q5_K, 2>(s, a) : launch_two<LLB_FM_Q5_K, 4>(s, a);
  if (fmt == LLB_FM_Q6_K) return NT == 1 ? launch_two<LLB_FM_Q6_K, 1>(s, a) : NT == 2 ? launch_two<LLB_FM_Q6_K, 2>(s, a) : launch_two<LLB_FM_Q6_K, 4>(s, a);
  if (fmt == LLB_FM_Q8_0) return NT == 1 ? launch_two<LLB_FM_Q8_0, 1>(s, a) : NT == 2 ? launch_two<LLB_FM_Q8_0, 2>(s, a) : launch_two<LLB_FM_Q8_0, 4>(s, a);
  return llb_fail("gemm: format %d has no kernel", fmt);
}
