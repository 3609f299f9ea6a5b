// pf.cu -- the prompt path: a chunk of up to PF_RMAX = 256 prompt rows per pass, dense GEMMs (pfx.cuh, pfmm.cuh) and attention (pfatt.cuh) on tcgen05,
// row-batched small ops.  It stands where the reference has its fast prefill tier (host/llb_pf.h:551 pf_take; kernels
// tools/pf27/pfmm.cuh, host/llb_pf.cuh; hand-off into the speculative state host/llb_host.c:1831-1899 spec_pf /
// spec_take): the trunk's K/V rows, conv history and DeltaNet state after the chunk, the drafter's K/V rows for the
// chunk's positions (k and v only: no drafter attention, FFN or head), and the normed hidden row it continues from.
// The arithmetic follows the CPU engine (tools/qwen35_engine.c:510-761) like the T-row kernels of ops_model.cu; what
// differs is the order of the GEMMs' sums (pfx.cuh, pfmm.cuh) and that a DeltaNet layer scans the chunk's rows in one
// kernel with the state in registers, writing the state once.
#include <mutex>

#include "pfmm.cuh"
#include "pfx.cuh"
#include "pfatt.cuh"
#include "model.cuh"
#include "pf.cuh"

static unsigned int *g_pf_err = nullptr;   // device word: a bounded wait of one of the tcgen05 kernels here ran out

static decltype(&cuTensorMapEncodeTiled) g_tensor_map = nullptr;

template <int FMT> static int pf_attr() {
  CU_OK(cudaFuncSetAttribute(k_pfmm<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SMEM));
  return 0;
}
// (their warpgroups trade registers: a launch with fewer than they were counted with would wait for ever)
template <typename K> static int px_attr(K k, int smem, int regs) {
  CU_OK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cudaFuncAttributes at;
  CU_OK(cudaFuncGetAttributes(&at, k));
  if (at.numRegs != regs) return llb_fail("pfx: built with %d registers a thread, its register split needs %d", at.numRegs, regs);
  return 0;
}
template <int FMT> static int px_attr1() {
  CU_OK(cudaFuncSetAttribute(k_pft<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, pt_smem(FMT)));
  return px_attr(k_pfx1<FMT, 64>, px_smem(FMT, 64), px1_reg_launch(FMT, 64)) || px_attr(k_pfx1<FMT, 128>, px_smem(FMT, 128), px1_reg_launch(FMT, 128));
}
template <int FMT> static int px_attr2() { return px_attr(k_pfx2<FMT>, px2_smem(FMT), PX_REG_LAUNCH); }
#define PF_SCAN_NW 4                            // warps of a scan block, 8 state rows each
#define PF_SCAN_BLOCKS (128 / (8 * PF_SCAN_NW)) // blocks of a head
#define PF_SCAN_SMEM (220 * 1024)
__global__ void k_pf_scan(const PfSegs sg, const float *__restrict__ y, const float *__restrict__ gram, const float *__restrict__ beta, const float *__restrict__ decay, DeltaShape sh,
                          float *__restrict__ o);
static int setup(void) {
  if (pf_attr<LLB_FM_Q6_K>() || pf_attr<LLB_FM_Q8_0>()) return -1;
  if (px_attr1<LLB_FM_Q4_K>() || px_attr1<LLB_FM_Q5_K>() || px_attr1<LLB_FM_Q6_K>() || px_attr1<LLB_FM_Q8_0>() || px_attr2<LLB_FM_Q4_K>() || px_attr2<LLB_FM_Q5_K>()) return -1;
  if (px_attr(k_pf_attn<128>, pa_smem(128), PA_REG_LAUNCH) || px_attr(k_pf_attn<256>, pa_smem(256), PA_REG_LAUNCH)) return -1;
  CU_OK(cudaFuncSetAttribute(k_pf_scan, cudaFuncAttributeMaxDynamicSharedMemorySize, PF_SCAN_SMEM - 24 * 1024));
  if (!g_tensor_map) {
    cudaDriverEntryPointQueryResult found;
    CU_OK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", (void **)&g_tensor_map, 12000, cudaEnableDefault, &found));
    if (!g_tensor_map) return llb_fail("the driver has no cuTensorMapEncodeTiled");
  }
  if (!g_pf_err) {
    CU_OK(cudaMalloc(&g_pf_err, 4));
    CU_OK(cudaMemset(g_pf_err, 0, 4));
  }
  return 0;
}
// 1 where the device has no room for the kernels
int pf_setup(void) {
  static std::mutex one;
  std::lock_guard<std::mutex> hold(one);
  cudaGetLastError();
  const int rc = setup();
  return rc && cudaGetLastError() == cudaErrorMemoryAllocation ? 1 : rc;
}
int pf_wait_errors(void) {
  unsigned int v = 0;
  if (g_pf_err && cudaMemcpy(&v, g_pf_err, 4, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return (int)v;
}
int pf_wait_errors_clear(void) {
  if (g_pf_err) CU_OK(cudaMemset(g_pf_err, 0, 4));
  return 0;
}

// K-slices of a dense launch: whole waves of (pair of tiles, slice) units over the pairs of SMs, each unit costing its slice's
// super-blocks plus about two super-blocks' worth of pipeline fill and epilogue; slices are whole super-blocks.
int pf_pick_ksplit(int ntiles, int nsb, int sms) {
  int best = 1;
  double best_cost = 1e30;
  for (int ks = 1; ks <= 8 && ks <= nsb; ks++) {
    const long long units = (long long)((ntiles + 1) / 2) * ks, waves = (units + sms / 2 - 1) / (sms / 2);
    const double cost = (double)waves * ((nsb + ks - 1) / ks + 2.0) * (1.0 + 0.03 * (ks - 1));   // the longest slice sets the pace
    if (cost < best_cost - 1e-9) { best_cost = cost; best = ks; }
  }
  return best;
}

// fills the tile table; K-slices are whole super-blocks, as equal as they come
int pf_gemm(cudaStream_t s, int fmt, PfArgs &a) {
  if (a.nmat < 1 || a.nmat > PF_MAXMAT) return llb_fail("pf gemm: nmat %d", a.nmat);
  if (a.K % 256 || a.ksplit < 1 || a.ksplit > a.K / 256) return llb_fail("pf gemm: K %d in %d slices", a.K, a.ksplit);
  if (a.R < 1 || a.R > PF_RMAX) return llb_fail("pf gemm: %d rows", a.R);
  a.t128[0] = 0;
  for (int i = 0; i < PF_MAXMAT; i++) a.t128[i + 1] = a.t128[i] + (i < a.nmat ? (a.m[i].rows + 127) / 128 : 0);
  a.err = g_pf_err;
  const int units = (a.t128[a.nmat] + 1) / 2 * a.ksplit;   // pairs of tiles
  if (units < 1) return 0;
  const int grid = 2 * (units < g_llb.sms / 2 ? units : g_llb.sms / 2);
  cudaError_t e = cudaErrorInvalidValue;
  const int ru = pf_unit_rows(a.R);
#define PT_GO(F) e = llb_launch(k_pft<F>, dim3(grid), dim3(PT_THREADS), (size_t)pt_smem(F), s, a)
#define PX_GO(F, RU) e = llb_launch(k_pfx1<F, RU>, dim3(grid), dim3(px1_threads(F, RU)), (size_t)px_smem(F, RU), s, a)
#define PX_ONE(F) do { if (ru == 32) PT_GO(F); else if (ru == 64) PX_GO(F, 64); else PX_GO(F, 128); } while (0)
#define PX_TWO(F) e = llb_launch(k_pfx2<F>, dim3(grid), dim3(PX_THREADS), (size_t)px2_smem(F), s, a)
  switch (fmt) {
    case LLB_FM_Q4_K: if (a.R > PF_R) PX_TWO(LLB_FM_Q4_K); else PX_ONE(LLB_FM_Q4_K); break;
    case LLB_FM_Q5_K: if (a.R > PF_R) PX_TWO(LLB_FM_Q5_K); else PX_ONE(LLB_FM_Q5_K); break;
    case LLB_FM_Q6_K: if (a.R > PF_R) e = llb_launch(k_pfmm<LLB_FM_Q6_K>, dim3(grid), dim3(PF_THREADS), (size_t)PF_SMEM, s, a); else PX_ONE(LLB_FM_Q6_K); break;
    case LLB_FM_Q8_0: if (a.R > PF_R) e = llb_launch(k_pfmm<LLB_FM_Q8_0>, dim3(grid), dim3(PF_THREADS), (size_t)PF_SMEM, s, a); else PX_ONE(LLB_FM_Q8_0); break;
    default: return llb_fail("pf gemm: format %d has no kernel", fmt);
  }
#undef PX_TWO
#undef PX_ONE
#undef PT_GO
#undef PX_GO
  if (e != cudaSuccess) return llb_fail("dense GEMM launch: %s", cudaGetErrorString(e));
  return 0;
}

// ---- row-batched small ops: one launch covers the R rows of the chunk --------------------------------
// Every kernel triggers its dependents first and waits for its producer before it touches a buffer another kernel writes.
// Those buffers are reused by every layer and the chain of resident, waiting kernels can be a dozen launches deep (the scan
// of a chunk is long), so loads of them bypass L1 (__ldcg / part_get): an SM's L1 may still hold what an earlier layer put
// in the same buffer.  Found the hard way: with plain loads the third DeltaNet layer of a chunk read the second one's rows.
__device__ __forceinline__ float pf_warp_sum(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}
__device__ __forceinline__ float pf_block_sum(float v, float *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = pf_warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = 0.0f;
  for (int i = 0; i < nw; i++) t += red[i];
  return t;
}
__device__ __forceinline__ float pf_silu(float x) { return x / (1.0f + expf(-x)); }

// embedding rows of the chunk's tokens (llb_embedk; bit-exact dequantisation)
__global__ void k_pf_embed(int fmt, const uint8_t *__restrict__ W, int d, const int *__restrict__ ids, float *__restrict__ x) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.y;
  const int row = ids[t];
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d; c += gridDim.x * blockDim.x) x[(size_t)t * d + c] = deq_elem(fmt, W, d, row, c);
}
int op_pf_embed(cudaStream_t s, int fmt, const uint8_t *W, int d, const int *ids, int R, float *x) {
  CU_OK(llb_launch(k_pf_embed, dim3((d + 255) / 256, R), dim3(256), (size_t)0, s, fmt, W, d, ids, x));
  return 0;
}

// v = xin + sum(partials); xout = v (optional); h = (v * s) * w with s = 1 / sqrt(mean(v^2) + eps) (rms_norm,
// tools/qwen35_engine.c:510-515); h goes to the k-group-major fp16 activations at column kg_col0 and, optionally,
// to hn_out as f32.  One block per row, as k_norm_xp.
#define PF_NORM_MAXT 1024
template <int NI>
__global__ void __launch_bounds__(PF_NORM_MAXT) k_pf_norm(const float *__restrict__ xin, PartIn add, const float *__restrict__ w, float eps, int d,
                                                          float *__restrict__ xout, __half *__restrict__ kg, int kg_K, int kg_col0, int ru, int row0, float *__restrict__ hn_out) {
  float4 wv[NI];
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    wv[i] = c < d ? *(const float4 *)(w + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  pdl_trigger();
  pdl_wait();
  __shared__ float red[32];
  const int t = blockIdx.x;
  const size_t row = (size_t)t * d;
  float4 v[NI];
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    v[i] = (c < d && xin) ? __ldcg((const float4 *)(xin + row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < d && add.p) { const float4 p = part_get4(add, row + c); v[i].x += p.x; v[i].y += p.y; v[i].z += p.z; v[i].w += p.w; }
  }
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    if (c < d) {
      if (xout) *(float4 *)(xout + row + c) = v[i];
      ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    }
  }
  ss = pf_block_sum(ss, red);
  const float sc = 1.0f / sqrtf(ss / (float)d + eps);
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    if (c >= d) continue;   // whole warps: d is a multiple of 128
    const float h0 = v[i].x * sc * wv[i].x, h1 = v[i].y * sc * wv[i].y, h2 = v[i].z * sc * wv[i].z, h3 = v[i].w * sc * wv[i].w;
    if (hn_out) *(float4 *)(hn_out + row + c) = make_float4(h0, h1, h2, h3);
    if (kg) pf_kg_store4(kg, kg_K, ru, row0 + t, kg_col0 + c, h0, h1, h2, h3);
  }
}
int op_pf_norm(cudaStream_t s, const float *xin, PartIn add, const float *w, float eps, int d, float *xout, __half *kg, int kg_K, int kg_col0, float *hn_out, int R, int ru, int row0) {
  if (d % 128 || kg_col0 % 128 || d > 4 * 4 * PF_NORM_MAXT) return llb_fail("pf norm: d %d at column %d", d, kg_col0);
  const int d4 = d / 4, ni = (d4 + PF_NORM_MAXT - 1) / PF_NORM_MAXT;
  const int threads = (((d4 + ni - 1) / ni) + 31) & ~31;
#define PF_NORM_GO(NI) CU_OK(llb_launch(k_pf_norm<NI>, dim3(R), dim3(threads), (size_t)0, s, xin, add, w, eps, d, xout, kg, kg_K, kg_col0, ru, row0, hn_out))
  switch (ni) {
    case 1: PF_NORM_GO(1); break;
    case 2: PF_NORM_GO(2); break;
    case 3: PF_NORM_GO(3); break;
    default: PF_NORM_GO(4); break;
  }
#undef PF_NORM_GO
  return 0;
}

// silu(gate) * up -> activations of ffn_down (llb_t_siluq)
__global__ void __launch_bounds__(256) k_pf_silu(PartIn g, PartIn u, int f, int ru, __half *__restrict__ kg) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.y, c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c >= f) return;   // whole warps
  const size_t i = (size_t)t * f + c;
  const float4 gv = part_get4(g, i), uv = part_get4(u, i);
  pf_kg_store4(kg, f, ru, t, c, pf_silu(gv.x) * uv.x, pf_silu(gv.y) * uv.y, pf_silu(gv.z) * uv.z, pf_silu(gv.w) * uv.w);
}
int op_pf_silu(cudaStream_t s, PartIn g, PartIn u, int f, __half *kg, int R, int ru) {
  CU_OK(llb_launch(k_pf_silu, dim3((f / 4 + 255) / 256, R), dim3(256), (size_t)0, s, g, u, f, ru, kg));
  return 0;
}

// ---- per-head QK RMSNorm, partial NEOX RoPE, K and V rows into the cache (tools/qwen35_engine.c:523-533, 667-690) ----
// A warp a (row, head), eight heads of a row a block: the query heads, then the key heads, then the value heads, from u0 on.  A row's angles are
// computed once a block (in 64 bits, as the CPU engine does): with a block a head, as the passes of a few rows have it, they were most of a
// launch, 36 us for 256 rows of 32 heads of 256.
__global__ void __launch_bounds__(256) k_pf_qkrope(PartIn q, PartIn k, PartIn v, const float *__restrict__ qn_w, const float *__restrict__ kn_w, const double *__restrict__ invfreq,
                                                   AttnShape sh, int p0, int u0, float *__restrict__ qout, __half *__restrict__ Kc, __half *__restrict__ Vc) {
  __shared__ float cs[128], sn[128];
  __shared__ __align__(16) float hv[8][256];
  const int t = blockIdx.y, pos = p0 + t, wp = threadIdx.x >> 5, lane = threadIdx.x & 31, u = u0 + blockIdx.x * 8 + wp, hd = sh.hd, half = sh.rope_dim >> 1, kvd = sh.KV * hd;
  pdl_trigger();
  if (u0 + (int)blockIdx.x * 8 < sh.H + sh.KV) {   // (some head of the block turns)
    const int i = threadIdx.x >> 1;
    if (i < half) {
      const double th = (double)(float)((double)pos * invfreq[i]);
      if (threadIdx.x & 1) sn[i] = (float)sin(th);
      else cs[i] = (float)cos(th);
    }
  }
  __syncthreads();
  pdl_wait();
  if (u >= sh.H + 2 * sh.KV) return;
  const int kind = u < sh.H ? 0 : u < sh.H + sh.KV ? 1 : 2, g = u - (kind == 0 ? 0 : kind == 1 ? sh.H : sh.H + sh.KV);
  const PartIn &in = kind == 0 ? q : kind == 1 ? k : v;
  const size_t at = kind == 0 ? (size_t)t * 2 * sh.H * hd + (size_t)g * 2 * hd : (size_t)t * kvd + g * hd;
  float4 x[2];
  float ss = 0.0f;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    x[j] = 128 * j < hd ? part_get4(in, at + 128 * j + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    ss += x[j].x * x[j].x + x[j].y * x[j].y + x[j].z * x[j].z + x[j].w * x[j].w;
  }
  if (kind < 2) {
    const float *w = kind ? kn_w : qn_w;
    const float sc = 1.0f / sqrtf(pf_warp_sum(ss) / (float)hd + sh.eps);
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (128 * j < hd) {
        const float4 n = *(const float4 *)(w + 128 * j + 4 * lane);
        x[j].x = x[j].x * sc * n.x; x[j].y = x[j].y * sc * n.y; x[j].z = x[j].z * sc * n.z; x[j].w = x[j].w * sc * n.w;
        *(float4 *)&hv[wp][128 * j + 4 * lane] = x[j];
      }
    __syncwarp();
    for (int i = lane; i < half; i += 32) {
      const float a = hv[wp][i], b = hv[wp][i + half], c = cs[i], s = sn[i];
      hv[wp][i] = __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s));
      hv[wp][i + half] = __fadd_rn(__fmul_rn(a, s), __fmul_rn(b, c));
    }
    __syncwarp();
  }
#pragma unroll
  for (int j = 0; j < 2; j++)
    if (128 * j < hd) {
      const int c = 128 * j + 4 * lane;
      if (kind < 2) x[j] = *(const float4 *)&hv[wp][c];
      if (kind == 0) { *(float4 *)(qout + ((size_t)t * sh.H + g) * hd + c) = x[j]; continue; }
      __half *dst = (kind == 1 ? Kc : Vc) + (size_t)pos * kvd + g * hd + c;
      const __half2 a = __floats2half2_rn(x[j].x, x[j].y), b = __floats2half2_rn(x[j].z, x[j].w);
      const float2 af = __half22float2(a), bf = __half22float2(b);
      const __half2 al = __floats2half2_rn((x[j].x - af.x) * XP_LO_SCALE, (x[j].y - af.y) * XP_LO_SCALE), bl = __floats2half2_rn((x[j].z - bf.x) * XP_LO_SCALE, (x[j].w - bf.y) * XP_LO_SCALE);
      *(uint2 *)dst = make_uint2(*(const uint32_t *)&a, *(const uint32_t *)&b);
      *(uint2 *)(dst + sh.kv_plane) = make_uint2(*(const uint32_t *)&al, *(const uint32_t *)&bl);
    }
}
// kv_only: only the K and V rows (the drafter's cache fill: no query rows)
int op_pf_qkrope(cudaStream_t s, PartIn q, PartIn k, PartIn v, const float *qn_w, const float *kn_w, const double *invfreq, AttnShape sh, int p0, int R, float *qout, float *Kc, float *Vc, bool kv_only) {
  if (sh.hd != 128 && sh.hd != 256) return llb_fail("attention: head_dim %d", sh.hd);
  const int u0 = kv_only ? sh.H : 0;
  CU_OK(llb_launch(k_pf_qkrope, dim3((sh.H + 2 * sh.KV - u0 + 7) / 8, R), dim3(256), (size_t)0, s, q, k, v, qn_w, kn_w, invfreq, sh, p0, u0, qout, (__half *)Kc, (__half *)Vc));
  return 0;
}

// ---- attention of a piece (pfatt.cuh) ---------------------------------------------------------------
// Slices of the positions: the fewest rounds of blocks, each as long as its slice's tiles plus about five for the queries going in and the sums coming out, and a
// quarter of a tile a slice for the merge.  Measured, with the merge: 256 rows of 24 heads of 256 over 4 behind 1280 positions 90 us with one slice, 58 with two, 48 with three
// (144 blocks), 70 with four; 9 rows behind 8000 positions 61 with 8, 38 with 24, 35 with 32, 40 with 63; 128 rows of 8 heads over 2 behind 384 27 with two, 21 with 8, 24 with 16.
static int pa_pick(int blocks, int total) {
  const int tiles = (total + 31) >> 5, sms = g_llb.sms;
  int best = 1;
  double best_cost = 1e30;
  for (int ns = 1; ns <= tiles && (ns == 1 || blocks * ns <= 2 * sms); ns++) {
    const double cost = (double)((blocks * ns + sms - 1) / sms) * ((tiles + ns - 1) / ns + 5.0) + 0.25 * ns;
    if (cost < best_cost) { best_cost = cost; best = ns; }
  }
  return best;
}
// (head, row, slice) triples of the largest piece
size_t op_pf_attn_parts(int H, int KV) {
  const int most = KV * ((PF_RMAX * (H / KV) + 127) / 128);
  return (size_t)128 * (most > 2 * g_llb.sms ? most : 2 * g_llb.sms);
}
// a layer's K or V rows of positions 0 .. total - 1, both planes: a box is 64 dims of 32 positions; what lies past the last is read as zeros
static int pa_map(CUtensorMap *map, const float *base, AttnShape sh, int total) {
  const cuuint64_t kvd = (cuuint64_t)sh.KV * sh.hd, dim[3] = {kvd, (cuuint64_t)total, 2}, step[2] = {kvd * 2, (cuuint64_t)sh.kv_plane * 2};
  const cuuint32_t box[3] = {64, 32, 2}, one[3] = {1, 1, 1};
  const CUresult r = g_tensor_map(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void *)base, dim, step, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : llb_fail("attention: tensor map of %d positions: error %d", total, (int)r);
}
int op_pf_attn(cudaStream_t s, const float *q, const float *Kc, const float *Vc, PartIn qg, AttnShape sh, int p0, int R, float *pm, float *pl, float *po, __half *kg, int row0, int ru) {
  const int tiles = (R * (sh.H / sh.KV) + 127) / 128, total = p0 + R;
  const int want = pa_pick(sh.KV * tiles, total), per = ((total + 31) / 32 + want - 1) / want * 32, ns = (total + per - 1) / per;
  const PaArgs a{q, sh.H, sh.KV, p0, R, per, pm, pl, po, g_pf_err};
  CUtensorMap km, vm;
  if (pa_map(&km, Kc, sh, total) || pa_map(&vm, Vc, sh, total)) return -1;
  const dim3 grid(tiles, ns, sh.KV);
  if (sh.hd == 128) CU_OK(llb_launch(k_pf_attn<128>, grid, dim3(PA_THREADS), (size_t)pa_smem(128), s, a, km, vm));
  else if (sh.hd == 256) CU_OK(llb_launch(k_pf_attn<256>, grid, dim3(PA_THREADS), (size_t)pa_smem(256), s, a, km, vm));
  else return llb_fail("attention: head_dim %d", sh.hd);
  CU_OK(llb_launch(k_pf_attn_comb, dim3((R * sh.H + 7) / 8), dim3(256), (size_t)0, s, pm, pl, po, qg, sh.H, sh.hd, R, ns, kg, row0, ru));
  return 0;
}

// ---- gated DeltaNet over a chunk (tools/qwen35_engine.c:581-662) -----------------------------------
// A chunk's sequences go through together, a step of eight rows of one of them at a time (four prompts of 25 to 40 tokens, 48 layers of 48
// heads: 5.7 ms in turn, 2.6 together).
// What the scan needs, one launch: a warp takes one unit of eight rows.
//   q or k group   conv1d + SiLU of its columns, then q / max(|q|, eps) / sqrt(128) or k / max(|k|, eps) (no eps inside the root,
//                  :613-620).  A group's two warps share a block: k passes through shared memory, the k warp makes the rows'
//                  products k_s . k_t (s < t), the q warp k_s . q_t (s <= t): 28 + 36 values, gram
//   value head     conv1d + SiLU of its v columns
//   32 gates       beta = sigmoid(b), decay = exp(softplus(a + dt) * ssm_a), head-major; transcendentals through double as
//                  k_delta and the CPU engine do
// conv1d: row t of the chunk (position p0 + t) reads its KC - 1 predecessors from the chunk's own raw rows or, before the
// chunk's first row, from the position-indexed ring (tap KC - 1 is the current token, :599-600).  A lane has four channels of
// the eight rows: a raw row is loaded 11 / 8 times instead of KC times, all rows of a K-slice in flight together.
// MT: taps kept (the first MT - KC are zero and add exactly zero).
#define PF_CH 8                 // rows of a scan step
#define PF_GRAM 64
__host__ __device__ __forceinline__ constexpr int pf_kk(int t, int s) { return t * (t - 1) / 2 + s; }          // k_s . k_t, s < t
__host__ __device__ __forceinline__ constexpr int pf_kq(int t, int s) { return 28 + t * (t + 1) / 2 + s; }     // k_s . q_t, s <= t
__device__ __forceinline__ float dot4(float4 a, float4 b) { return (a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w); }
template <int MT>
__device__ __forceinline__ void pf_conv_rows(const PartIn &qkv, const PartIn &ring, const float *__restrict__ cw, int convd, int KC, int p0, int R, int t0, int c, float4 (&out)[PF_CH]) {
  constexpr int NR = PF_CH + MT - 1;
  float4 x[NR];
#pragma unroll
  for (int r = 0; r < NR; r++) x[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int k = 0; k < qkv.ns; k++) {
    const float *p = qkv.p + k * qkv.stride + c;
#pragma unroll
    for (int r = 0; r < NR; r++) {
      const int t = t0 + r - (MT - 1);
      if (t >= 0 && t < R) { const float4 l = __ldcg((const float4 *)(p + (size_t)t * convd)); x[r].x += l.x; x[r].y += l.y; x[r].z += l.z; x[r].w += l.w; }
    }
  }
  if (t0 == 0) {
#pragma unroll
    for (int r = 0; r < MT - 1; r++)
      if (r >= MT - KC) p_parts4(ring, (size_t)((p0 + r - (MT - 1)) & (CONV_RING - 1)) * convd + c, x[r]);
  }
  float w[4][MT];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int k = 0; k < MT; k++) w[i][k] = k >= MT - KC ? __ldg(cw + (size_t)(c + i) * KC + k - (MT - KC)) : 0.0f;
#pragma unroll
  for (int q = 0; q < PF_CH; q++) {
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < MT; k++) {
      a[0] = __fadd_rn(a[0], __fmul_rn(x[q + k].x, w[0][k])); a[1] = __fadd_rn(a[1], __fmul_rn(x[q + k].y, w[1][k]));
      a[2] = __fadd_rn(a[2], __fmul_rn(x[q + k].z, w[2][k])); a[3] = __fadd_rn(a[3], __fmul_rn(x[q + k].w, w[3][k]));
    }
    out[q] = make_float4(pf_silu(a[0]), pf_silu(a[1]), pf_silu(a[2]), pf_silu(a[3]));
  }
}
// Sums over the lanes of 32 values each: an exchange halves the values a lane holds, lane l ends with the sum of value l.
__device__ __forceinline__ float pf_lane_sums(float (&v)[32], int lane) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1)
#pragma unroll
    for (int i = 0; i < m; i++) {
      const float keep = lane & m ? v[i + m] : v[i], send = lane & m ? v[i] : v[i + m];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
  return v[0];
}
template <int MT>
__global__ void __launch_bounds__(128) k_pf_conv(const PfSegs sg, PartIn qkv, int ring_ks, const float *__restrict__ cw, PartIn bp, PartIn ap, const float *__restrict__ dt,
                                                 const float *__restrict__ sa, DeltaShape sh, float *__restrict__ y, float *__restrict__ gram,
                                                 float *__restrict__ beta, float *__restrict__ decay) {
  __shared__ __align__(16) float kx[2][PF_CH][128];
  int si = 0, t0 = blockIdx.y * PF_CH;   // the sequence whose step this is, and the step's first row of it
  for (; t0 >= sg.s[si].R; si++) t0 -= (sg.s[si].R + PF_CH - 1) / PF_CH * PF_CH;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, p0 = sg.s[si].p0, R = sg.s[si].R, nqk = (sh.GK + 1) / 2, nv = (sh.TR + 3) / 4;
  const PartIn ring{sg.s[si].ring, ring_ks, (long long)CONV_RING * sh.convd};
  const size_t off = sg.s[si].off;
  qkv.p += off * sh.convd; y += off * sh.convd; bp.p += off * sh.TR; ap.p += off * sh.TR;
  int bx = blockIdx.x;
  pdl_trigger();
  pdl_wait();
  if (bx < nqk) {
    const int g = 2 * bx + (wp & 1), isk = wp >> 1;
    const bool on = g < sh.GK;
    float4 x[PF_CH];
    const int c = min(g, sh.GK - 1) * 128 + 4 * lane + isk * sh.kdc;
    pf_conv_rows<MT>(qkv, ring, cw, sh.convd, sh.KC, p0, R, t0, c, x);
#pragma unroll
    for (int t = 0; t < PF_CH; t++) {
      const float nx = sqrtf(pf_warp_sum(dot4(x[t], x[t])));
      const float ix = (isk ? 1.0f : 0.08838834764831845f) / (nx > sh.eps ? nx : sh.eps);   // 1 / sqrt(128)
      x[t].x *= ix; x[t].y *= ix; x[t].z *= ix; x[t].w *= ix;
      if (on && t0 + t < R) *(float4 *)(y + (size_t)(t0 + t) * sh.convd + c) = x[t];
      if (isk) *(float4 *)&kx[wp & 1][t][4 * lane] = x[t];
    }
    __syncthreads();
    float *G = gram + ((size_t)g * PF_STEPS + blockIdx.y) * PF_GRAM;
    float v[32];
    if (isk) {
#pragma unroll
      for (int t = 0; t < PF_CH; t++)
#pragma unroll
        for (int s = 0; s < t; s++) v[pf_kk(t, s)] = dot4(x[s], x[t]);
#pragma unroll
      for (int i = 28; i < 32; i++) v[i] = 0.0f;
      const float r = pf_lane_sums(v, lane);
      if (on && lane < 28) G[lane] = r;
    } else {
      float last[4];
#pragma unroll
      for (int s = 0; s < PF_CH; s++) {
        const float4 k = *(const float4 *)&kx[wp & 1][s][4 * lane];
#pragma unroll
        for (int t = s; t < PF_CH; t++) {
          const float d = dot4(k, x[t]);
          if (pf_kq(t, s) - 28 < 32) v[pf_kq(t, s) - 28] = d;
          else last[pf_kq(t, s) - 60] = d;
        }
      }
      const float r = pf_lane_sums(v, lane);
#pragma unroll
      for (int i = 0; i < 4; i++) last[i] = pf_warp_sum(last[i]);
      if (on) {
        G[28 + lane] = r;
        if (lane == 0) *(float4 *)(G + 60) = make_float4(last[0], last[1], last[2], last[3]);
      }
    }
    return;
  }
  bx -= nqk;
  if (bx < nv) {
    const int h = bx * 4 + wp, c = 2 * sh.kdc + h * 128 + 4 * lane;
    if (h >= sh.TR) return;
    float4 v[PF_CH];
    pf_conv_rows<MT>(qkv, ring, cw, sh.convd, sh.KC, p0, R, t0, c, v);
#pragma unroll
    for (int t = 0; t < PF_CH; t++)
      if (t0 + t < R) *(float4 *)(y + (size_t)(t0 + t) * sh.convd + c) = v[t];
    return;
  }
  const int i = (bx - nv) * 128 + threadIdx.x, t = t0 + i / sh.TR, h = i % sh.TR, at = h * (PF_STEPS * PF_CH) + blockIdx.y * PF_CH + i / sh.TR;
  if (i >= PF_CH * sh.TR || t >= R) return;
  const float b = part_get(bp, (size_t)t * sh.TR + h), a = part_get(ap, (size_t)t * sh.TR + h);
  beta[at] = 1.0f / (1.0f + (float)exp((double)-b));
  const float x = a + dt[h];
  const float sp = x > 20.0f ? x : (float)log1p((double)(float)exp((double)(x < 88.0f ? x : 88.0f)));
  decay[at] = (float)exp((double)(sp * sa[h]));
}
// The recurrence over the chunk's R rows.  Block (hh, y) keeps 32 state rows of value head hh in registers from the first
// row of the chunk to the last and writes them back once (a lane: four state rows, columns 4 cq .. and 64 + 4 cq ..).
// Per row t and state row j: S_j *= decay; delta = (v_j - S_j . k) * beta; S_j += k * delta; o_j = S_j . q (:630-646).
//
// Row by row that is a chain: a dot product, its shuffles, the update, 0.4 to 0.6 us a row.  Here a step takes eight rows.  With
// S the state before them and d(s, t] the product of decays of rows s + 1 .. t,
//     delta_t = beta_t (v_t - d[0, t] S . k_t - sum_{s < t} d(s, t] (k_s . k_t) delta_s)
//     o_t     = d[0, t] S . q_t + sum_{s <= t} d(s, t] (k_s . q_t) delta_s
//     S      <- d[0, 7] S + sum_s d(s, 7] delta_s k_s
// so the sixteen dot products of a state row with S run side by side, their sums over the sixteen lanes are one exchange
// tree (64 values, 60 shuffles) that leaves row t's sums of two state rows in a lane, and the chain is the substitution: eight
// steps of a shuffle and a multiply-add; the update's deltas come by shuffles that wait for nothing.  The decays' products never
// divide, so a decay of nearly zero does no harm.  Multiply-adds: three a state element and row instead of four, two an
// instruction.  Sixteen lanes a state row, not eight: the loads of q and k, which every state row repeats, were the longer
// part of a step with eight (shared memory: 66 us a chunk of the 48-head shape against 48).  What bounds it now is one warp's
// chain: 960 instructions a step in 2300 cycles.  A lane takes its state rows and the step's rows in the order of its own lane bits (row
// t ^ tq for t), which spares the exchange its selections, 150 instructions a step, and lets the update's k stay in registers: 45 -> 40 us a
// chunk of 256 rows.  The ops between a DeltaNet layer's GEMMs, before and now: 84.5 -> 55 ms of a
// 3011-token prompt (48 layers, 48 heads), 47 -> 28 ms of 4096 tokens (24 layers, 32 heads), 23 -> 9.7 ms of 2000 tokens (18
// layers, 8 heads).
// Rows come through double-buffered shared memory, the next eight requested before the present ones are computed.
__global__ void __launch_bounds__(32 * PF_SCAN_NW, 2) k_pf_scan(const PfSegs sg, const float *__restrict__ y, const float *__restrict__ gram, const float *__restrict__ beta, const float *__restrict__ decay, DeltaShape sh,
                                                     float *__restrict__ o) {
  constexpr int NT = 32 * PF_SCAN_NW, NJ = 8 * PF_SCAN_NW, VS = NJ + 4;   // a block's threads and state rows; v rows padded so that eight lanes' reads miss one another's banks
  __shared__ __align__(16) float qs[2][PF_CH][128], ks[2][PF_CH][128], vs[2][PF_CH][VS], gs[2][PF_GRAM], bs[2][PF_CH], ds[2][PF_CH];
  const int hh = blockIdx.x, jq = blockIdx.y, tid = threadIdx.x, g = hh % sh.GK, jg = tid >> 4, cq = tid & 15, tq = tid & 7, rh = (tid >> 3) & 1;
  const PfSeg &me = sg.s[blockIdx.z];
  const int R = me.R;
  int step0 = 0;                          // its first step of the chunk's
  for (int i = 0; i < (int)blockIdx.z; i++) step0 += (sg.s[i].R + PF_CH - 1) / PF_CH;
  y += (size_t)me.off * sh.convd; o += (size_t)me.off * sh.vdc;
  pdl_trigger();
  const size_t head_sz = 128 * 128, slot_sz = (size_t)sh.TR * head_sz;
  float4 *Sp = (float4 *)(me.S + (size_t)(*(const volatile int *)&me.ctl->sc) * slot_sz + (size_t)hh * head_sz + (size_t)(NJ * jq + 4 * jg) * 128 + 4 * cq);   // the committed slot: stable during the pass
  f32x2 st[4][4];
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int i = 0; i < 2; i++) { const float4 v = __ldcg(Sp + 32 * (r ^ 2 * rh) + 16 * i); st[r][2 * i] = x2_pack(v.x, v.y); st[r][2 * i + 1] = x2_pack(v.z, v.w); }
  pdl_wait();
  const int nb = (R + PF_CH - 1) / PF_CH;
  auto stage = [&](int b) {   // rows past the chunk repeat its last one; their beta counts as zero and their decay as one
    const int buf = b & 1;
#pragma unroll
    for (int i = tid; i < PF_CH * 32; i += NT) {
      const int r = i >> 5, c = 4 * (i & 31);
      const float *row = y + (size_t)min(b * PF_CH + r, R - 1) * sh.convd + g * 128 + c;
      cp_async16(smem_u32(&qs[buf][r][c]), row);
      cp_async16(smem_u32(&ks[buf][r][c]), row + sh.kdc);
    }
    for (int i = tid; i < PF_CH * NJ / 4; i += NT) {
      const int r = i / (NJ / 4), c = 4 * (i % (NJ / 4));
      cp_async16(smem_u32(&vs[buf][r][c]), y + (size_t)min(b * PF_CH + r, R - 1) * sh.convd + 2 * sh.kdc + hh * 128 + NJ * jq + c);
    }
    if (tid < PF_GRAM / 4) cp_async16(smem_u32(&gs[buf][4 * tid]), gram + ((size_t)g * PF_STEPS + step0 + b) * PF_GRAM + 4 * tid);
    else if (tid < PF_GRAM / 4 + 2) cp_async16(smem_u32(&bs[buf][4 * (tid & 1)]), beta + (hh * PF_STEPS + step0 + b) * PF_CH + 4 * (tid & 1));
    else if (tid < PF_GRAM / 4 + 4) cp_async16(smem_u32(&ds[buf][4 * (tid & 1)]), decay + (hh * PF_STEPS + step0 + b) * PF_CH + 4 * (tid & 1));
  };
  stage(0);
  cp_async_commit();
  float *op = o + hh * 128 + NJ * jq + 4 * jg + 2 * rh;
  for (int b = 0; b < nb; b++) {
    const int buf = b & 1, n = min(PF_CH, R - b * PF_CH);
    cp_async_wait<0>();
    __syncthreads();   // the present rows are there, and nobody reads the buffer of the next ones any more
    if (b + 1 < nb) stage(b + 1);
    cp_async_commit();
    f32x2 kk[PF_CH][4];
    float kv[4][PF_CH], qv[4][PF_CH];
#pragma unroll
    for (int t = 0; t < PF_CH; t++) {   // row t ^ tq
      f32x2 (&k)[4] = kk[t], q[4];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const ulonglong2 a = *(const ulonglong2 *)&ks[buf][t ^ tq][64 * i + 4 * cq], c = *(const ulonglong2 *)&qs[buf][t ^ tq][64 * i + 4 * cq];
        k[2 * i] = a.x; k[2 * i + 1] = a.y; q[2 * i] = c.x; q[2 * i + 1] = c.y;
      }
#pragma unroll
      for (int r = 0; r < 4; r++) {
        f32x2 a = x2_mul(st[r][0], k[0]), c = x2_mul(st[r][0], q[0]);
#pragma unroll
        for (int i = 1; i < 4; i++) { a = x2_fma(st[r][i], k[i], a); c = x2_fma(st[r][i], q[i], c); }
        float lo, hi;
        x2_unpack(a, lo, hi); kv[r][t] = lo + hi;
        x2_unpack(c, lo, hi); qv[r][t] = lo + hi;
      }
    }
    // the exchange over lane bit 3 keeps two of the four state rows, those over bits 2 .. 0 row tq of the eight: with a lane's state rows and
    // rows of the step in the order of its own bits it keeps the first half of its values each time, and its partner's second half is the same rows'
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int t = 0; t < PF_CH; t++) {
        kv[r][t] += __shfl_xor_sync(0xffffffffu, kv[r + 2][t], 8);
        qv[r][t] += __shfl_xor_sync(0xffffffffu, qv[r + 2][t], 8);
      }
#pragma unroll
    for (int m = 4; m > 0; m >>= 1)
#pragma unroll
      for (int i = 0; i < m; i++)
#pragma unroll
        for (int r = 0; r < 2; r++) {
          kv[r][i] += __shfl_xor_sync(0xffffffffu, kv[r][i + m], m);
          qv[r][i] += __shfl_xor_sync(0xffffffffu, qv[r][i + m], m);
        }
    // lane tq is row t = tq from here on
    float dec[PF_CH], M[PF_CH], N[PF_CH], e[PF_CH];
#pragma unroll
    for (int s = 0; s < PF_CH; s++) dec[s] = s < n ? ds[buf][s] : 1.0f;
    const float bt = tq < n ? bs[buf][tq] : 0.0f;
    float w = 1.0f;
#pragma unroll
    for (int s = PF_CH - 1; s >= 0; s--) {
      if (s + 1 < PF_CH) w = s < tq ? w * dec[s + 1] : 1.0f;
      M[s] = s < tq ? bt * w * gs[buf][pf_kk(tq, 0) + s] : 0.0f;
      N[s] = s <= tq ? w * gs[buf][pf_kq(tq, 0) + s] : 0.0f;
    }
    const float P = w * dec[0];
    e[PF_CH - 1] = 1.0f;
#pragma unroll
    for (int s = PF_CH - 2; s >= 0; s--) e[s] = e[s + 1] * dec[s + 1];
    const float P7 = e[0] * dec[0];
    const float2 vv = *(const float2 *)&vs[buf][tq][4 * jg + 2 * rh];
    float x[2] = {bt * (vv.x - P * kv[0][0]), bt * (vv.y - P * kv[1][0])}, ov[2] = {P * qv[0][0], P * qv[1][0]};
    const f32x2 pp = x2_pack(P7, P7);
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
      for (int i = 0; i < 4; i++) st[r][i] = x2_mul(st[r][i], pp);
#pragma unroll
    for (int s = 0; s < PF_CH; s++) {
      float d[2];
#pragma unroll
      for (int r = 0; r < 2; r++) {
        d[r] = __shfl_sync(0xffffffffu, x[r], s, 8);
        x[r] -= M[s] * d[r];
        ov[r] += N[s] * d[r];
      }
    }
    float et = 1.0f;
#pragma unroll
    for (int s = 0; s < PF_CH; s++) et = s == tq ? e[s] : et;
    x[0] *= et; x[1] *= et;
#pragma unroll
    for (int s = 0; s < PF_CH; s++) {   // row s ^ tq
#pragma unroll
      for (int r = 0; r < 4; r++) {
        const float d = s == 0 && r < 2 ? x[r] : __shfl_xor_sync(0xffffffffu, x[r & 1], s + 8 * (r >> 1));
        const f32x2 d2 = x2_pack(d, d);
#pragma unroll
        for (int i = 0; i < 4; i++) st[r][i] = x2_fma(kk[s][i], d2, st[r][i]);
      }
    }
    if (tq < n) *(float2 *)(op + (size_t)(b * PF_CH + tq) * sh.vdc) = make_float2(ov[0], ov[1]);
  }
#pragma unroll
  for (int r = 0; r < 4; r++)
#pragma unroll
    for (int i = 0; i < 2; i++) {
      float4 v;
      x2_unpack(st[r][2 * i], v.x, v.y); x2_unpack(st[r][2 * i + 1], v.z, v.w);
      Sp[32 * (r ^ 2 * rh) + 16 * i] = v;
    }
}
// gated RMSNorm of each head's output -> activations of ssm_out (:648-654); a warp per (head, row), eight rows a block.  One more
// block a head copies the chunk's last raw rows into the conv history: whole values into K-slice 0, zeros into the rest
// (here, because the conv kernel's first rows still read the old history).
__global__ void __launch_bounds__(256) k_pf_gnorm(const float *__restrict__ o, PartIn z, const float *__restrict__ nw, DeltaShape sh, __half *__restrict__ kg,
                                                  PartIn qkv, int ring_ks, const PfSegs sg, int ru) {
  const int p0 = sg.s[blockIdx.z].p0, R = sg.s[blockIdx.z].R, row0 = sg.s[blockIdx.z].off;
  float *ring = sg.s[blockIdx.z].ring;
  const int hh = blockIdx.x, t = blockIdx.y * 8 + (threadIdx.x >> 5), i = threadIdx.x & 31;
  const float4 w = __ldg((const float4 *)(nw + 4 * i));
  pdl_trigger();
  pdl_wait();
  if (8 * (int)blockIdx.y >= R) {
    if (8 * (int)blockIdx.y >= R + 8) return;   // (another sequence has more rows)
    const int nr = min(R, CONV_RING), nc = sh.convd / 4;
    for (int j = hh * 256 + threadIdx.x; j < nr * nc; j += sh.TR * 256) {
      const int tr = R - nr + j / nc, c = 4 * (j % nc);
      const size_t dst = (size_t)((p0 + tr) & (CONV_RING - 1)) * sh.convd + c;
      *(float4 *)(ring + dst) = part_get4(qkv, (size_t)(row0 + tr) * sh.convd + c);
      for (int k = 1; k < ring_ks; k++) *(float4 *)(ring + (size_t)k * CONV_RING * sh.convd + dst) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  if (t >= R) return;
  const size_t idx = (size_t)(row0 + t) * sh.vdc + hh * 128 + 4 * i;
  const float4 v = __ldcg((const float4 *)(o + idx)), zz = part_get4(z, idx);
  const float r = 1.0f / sqrtf(pf_warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) / 128.0f + sh.eps);
  pf_kg_store4(kg, sh.vdc, ru, row0 + t, hh * 128 + 4 * i, v.x * r * w.x * pf_silu(zz.x), v.y * r * w.y * pf_silu(zz.y), v.z * r * w.z * pf_silu(zz.z), v.w * r * w.w * pf_silu(zz.w));
}

// One DeltaNet layer's ops between its input GEMM (qkv | z | beta | alpha) and its output GEMM, for R rows at p0 ...
int op_pf_delta(cudaStream_t s, PartIn qkv, PartIn z, PartIn bp, PartIn ap, int ring_ks, const float *cw, const float *dt, const float *sa,
                const float *nw, DeltaShape sh, const PfSegs &sg, float *y, float *gram, float *beta, float *decay, float *o, __half *kg, int ru) {
  if (sh.SZ != 128 || sh.KC > CONV_RING / 2) return llb_fail("pf delta: state size %d, conv kernel %d", sh.SZ, sh.KC);
  int steps = 0, most = 0;
  for (int i = 0; i < sg.n; i++) { const int n = (sg.s[i].R + PF_CH - 1) / PF_CH; steps += n; most = n > most ? n : most; }
  const dim3 cgrid((sh.GK + 1) / 2 + (sh.TR + 3) / 4 + (PF_CH * sh.TR + 127) / 128, steps);
  if (sh.KC <= 4) CU_OK(llb_launch(k_pf_conv<4>, cgrid, dim3(128), (size_t)0, s, sg, qkv, ring_ks, cw, bp, ap, dt, sa, sh, y, gram, beta, decay));
  else CU_OK(llb_launch(k_pf_conv<CONV_RING / 2>, cgrid, dim3(128), (size_t)0, s, sg, qkv, ring_ks, cw, bp, ap, dt, sa, sh, y, gram, beta, decay));
  // A block's chain takes as long alone as with others on its SM, but the scheduler stacks blocks on few SMs while others idle
  // (32-head shape: 38 ms of a 4096-token prompt so, 28 ms spread): a block asks for the shared memory of its even share of an SM.
  const int blocks = sh.TR * PF_SCAN_BLOCKS * sg.n, per = (blocks + g_llb.sms - 1) / g_llb.sms;
  const size_t pad = per < 6 ? (size_t)(PF_SCAN_SMEM / per - 24 * 1024) : 0;
  CU_OK(llb_launch(k_pf_scan, dim3(sh.TR, PF_SCAN_BLOCKS, sg.n), dim3(32 * PF_SCAN_NW), pad, s, sg, (const float *)y, (const float *)gram, (const float *)beta, (const float *)decay, sh, o));
  CU_OK(llb_launch(k_pf_gnorm, dim3(sh.TR, most + 1, sg.n), dim3(256), (size_t)0, s, (const float *)o, z, nw, sh, kg, qkv, ring_ks, sg, ru));
  return 0;
}

// ---- operator entry point: the dense GEMM alone ------------------------------------------------------
// f32 rows [R][K] -> fp16, k-group major
__global__ void __launch_bounds__(256) k_pf_pack(const float *__restrict__ x, int K, int ru, __half *__restrict__ kg) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.y, c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c >= K) return;   // whole warps: K is a multiple of 128
  const float4 v = __ldcg((const float4 *)(x + (size_t)t * K + c));
  pf_kg_store4(kg, K, ru, t, c, v.x, v.y, v.z, v.w);
}
int op_pf_pack(cudaStream_t s, const float *x, int K, int R, __half *kg) {
  CU_OK(llb_launch(k_pf_pack, dim3((K / 4 + 255) / 256, R), dim3(256), (size_t)0, s, x, K, pf_unit_rows(R), kg));
  return 0;
}

extern "C" __attribute__((visibility("default")))
int llb_b200_pf_gemm(int fmt, unsigned long long w, int rows, int K, unsigned long long x_f32, int R, unsigned long long out_f32, int ksplit) {
  if (!g_llb.stream) return llb_fail("llb_b200_init has not been called");
  if (K < 256 || K % 256 || rows < 1 || R < 1 || R > PF_RMAX) return llb_fail("pf_gemm: rows %d, K %d, R %d (K a multiple of 256, R up to %d)", rows, K, R, PF_RMAX);
  if (!tile_bytes(fmt)) return llb_fail("pf_gemm: format %d has no kernel", fmt);
  if (pf_setup()) return -1;
  const int nsb = K / 256;
  if (ksplit <= 0) ksplit = pf_pick_ksplit((rows + 127) / 128, nsb, g_llb.sms);
  if (ksplit > nsb) return llb_fail("pf_gemm: %d K-slices of %d super-blocks", ksplit, nsb);
  __half *kg = nullptr;
  float *parts = nullptr;
  CU_OK(cudaMalloc(&kg, 2 * pf_kg_halves(K, PF_R) * 2));      // two units of 128 rows
  CU_OK(cudaMemsetAsync(kg, 0, 2 * pf_kg_halves(K, PF_R) * 2, g_llb.stream));
  if (ksplit > 1) CU_OK(cudaMalloc(&parts, (size_t)ksplit * R * rows * 4));
  int rc = op_pf_pack(g_llb.stream, (const float *)(uintptr_t)x_f32, K, R, kg);
  PfArgs a;
  memset(&a, 0, sizeof a);
  a.nmat = 1; a.K = K; a.ksplit = ksplit; a.R = R; a.x = kg;
  a.m[0].W = (const uint8_t *)(uintptr_t)w; a.m[0].rows = rows; a.m[0].ostride = rows;
  a.m[0].out = ksplit > 1 ? parts : (float *)(uintptr_t)out_f32; a.m[0].split_stride = (long long)R * rows;
  if (!rc) rc = pf_gemm(g_llb.stream, fmt, a);
  if (!rc && ksplit > 1) rc = ops_sum_parts(g_llb.stream, parts, ksplit, (long long)R * rows, R * rows, (float *)(uintptr_t)out_f32);
  cudaStreamSynchronize(g_llb.stream);
  cudaFree(kg);
  if (parts) cudaFree(parts);
  if (!rc && cudaGetLastError() != cudaSuccess) rc = llb_fail("pf_gemm: a kernel failed");
  return rc;
}

// ---- what the agents of the kernels here do with their barriers --------------------------------------
// For a check without a GPU: every warp's waits and arrivals in its order, with the kernels' own rings and numbering.  ops: {0 wait, barrier, phase},
// {1 arrive, barrier, times}, {2 arrive, barrier, once a copy requested or an MMA issued here is done}; a pair's second CTA has the same
// barriers from PT_BARS on.  Returns the operations' number, 0 for an agent that has none, -1 past the last agent.
struct PfTrace {
  int *ops, cap, n = 0;
  void put(int kind, int b, int v) { if (3 * n + 2 < cap) { ops[3 * n] = kind; ops[3 * n + 1] = b; ops[3 * n + 2] = v; } n++; }
  void wait(int b, int phase) { put(0, b, phase); }
  void free_again(int b, int use) { if (use > 0) put(0, b, use - 1); }     // a ring's buffer at its use-th use
  void arrive(int b) { put(1, b, 1); }
  void later(int b) { put(2, b, 1); }
};
#define PT_BARS 64
static int pa_trace(PfTrace &t, int NS, int n, int agent) {
  const int full = 0, empty = 8, s_full = 16, p_full = 18, pv_done = 20, o_empty = 22, q_full = 23;
  if (agent < 4) {            // softmax
    t.arrive(q_full);
    for (int it = 0; it < n; it++) {
      t.wait(s_full + (it & 1), it >> 1);
      if (it >= 2) t.wait(pv_done + (it & 1), (it >> 1) - 1);
      t.arrive(p_full + (it & 1));
    }
  } else if (agent == 4) {    // loads
    int k = 0;
    auto load = [&] {
      const int slot = k % NS;
      if (k >= NS) t.wait(empty + slot, k / NS - 1);
      else if (k == NS - 2) t.wait(q_full, 0);
      t.later(full + slot);
      k++;
    };
    for (int i = -2; i < n; i++) {
      if (i >= 0) load();
      if (i + 2 < n) load();
    }
  } else if (agent == 5) {    // issues the MMAs
    int k = 0;
    t.wait(q_full, 0);
    for (int i = -2; i < n; i++) {
      if (i >= 0) {
        t.wait(p_full + (i & 1), i >> 1);
        t.wait(o_empty, i);
        t.wait(full + k % NS, k / NS);
        t.later(pv_done + (i & 1)); t.later(empty + k % NS);
        k++;
      }
      if (i + 2 < n) {
        t.wait(full + k % NS, k / NS);
        t.later(s_full + (i & 1)); t.later(empty + k % NS);
        k++;
      }
    }
  } else if (agent < 14) {    // O
    for (int it = 0; it < n; it++) {
      t.wait(p_full + (it & 1), it >> 1);
      t.arrive(o_empty);
      t.wait(pv_done + (it & 1), it >> 1);
    }
  } else return -1;
  return t.n;
}
static int pa_count(int b) { return b == 22 ? 8 : b == 18 || b == 19 || b == 23 ? 4 : 1; }

enum { PT_A_FULL = 0, PT_A_EMPTY = 8, PT_B_FULL = 16, PT_B_EMPTY = 20, PT_B_HERE = 24, PT_D_FULL = 28, PT_D_EMPTY = 32, PT_SC = 36, PT_RAW_FULL = 40, PT_RAW_EMPTY = 44 };
// the roles that the GEMM kernels have alike; me: the CTA's barriers
static void pt_weights(PfTrace &t, int me, int NRAW, int CH, int units, int nsl) {
  int k = 0;
  for (int u = 0; u < units; u++)
    for (int c = 0; c < nsl; c += CH, k++) { t.free_again(me + PT_RAW_EMPTY + k % NRAW, k / NRAW); t.later(me + PT_RAW_FULL + k % NRAW); }
}
static void pt_activations(PfTrace &t, int rank, int NB, int slots) {
  for (int i = 0; i < slots; i++) { t.free_again(rank * PT_BARS + PT_B_EMPTY + i % NB, i / NB); t.later((rank ? PT_BARS + PT_B_HERE : PT_B_FULL) + i % NB); }
}
static void pt_forward(PfTrace &t, int NB, int slots) {
  for (int i = 0; i < slots; i++) { t.wait(PT_BARS + PT_B_HERE + i % NB, i / NB); t.arrive(PT_B_FULL + i % NB); }
}
static void pt_both(PfTrace &t, int b) { t.later(b); t.later(PT_BARS + b); }
template <int FMT, int RU> static int px1_trace(PfTrace &t, int units, int nsl, int agent) {
  constexpr int NA = px_na(FMT), NB = px_nb(FMT), BS = px_slot_stages(RU), CH = px_chunk(FMT), NRAW = px_raws(FMT, RU), SS = px_sub(FMT);
  constexpr int UW = px1_unpack(FMT, RU), AG = UW + 12;
  const int rank = agent / AG, w = agent % AG, me = rank * PT_BARS;
  if (agent >= 2 * AG) return -1;
  if (w < UW) {
    int k = 0, rk = 0, jj = 0;
    for (int u = 0; u < units; u++)
      for (int c = 0; c < nsl; c++, jj++) {
        if (c % CH == 0) t.wait(me + PT_RAW_FULL + rk % NRAW, rk / NRAW);
        for (int s = 0; s < 4; s += SS, k++) {
          t.free_again(me + PT_A_EMPTY + k % NA, k / NA);
          if (s == 0 && w < 4) t.arrive(me + PT_SC + (jj & 3));
          t.arrive(PT_A_FULL + k % NA);
        }
        if (c % CH == CH - 1 || c == nsl - 1) { t.arrive(me + PT_RAW_EMPTY + rk % NRAW); rk++; }
      }
  } else if (w == UW) pt_weights(t, me, NRAW, CH, units, nsl);
  else if (w == UW + 1) pt_activations(t, rank, NB, units * (4 * nsl / BS));
  else if (w == UW + 2 && rank == 0) {
    int k = 0, bk = 0;
    for (int i = 0; i < units * nsl * 4; i += SS, k++) {
      if (k > 1) t.wait(PT_D_EMPTY + (k & 1), (k >> 1) - 1);
      t.wait(PT_A_FULL + k % NA, k / NA);
      for (int q = 0; q < SS; q++) {
        const int in = (i + q) % BS;
        if (in == 0) t.wait(PT_B_FULL + bk % NB, bk / NB);
        if (q == SS - 1) { pt_both(t, PT_A_EMPTY + k % NA); pt_both(t, PT_D_FULL + (k & 1)); }
        if (in == BS - 1) { pt_both(t, PT_B_EMPTY + bk % NB); bk++; }
      }
    }
  } else if (w == UW + 3 && rank == 1) pt_forward(t, NB, units * (4 * nsl / BS));
  else if (w >= UW + 4) {
    for (int jj = 0, k = 0; jj < units * nsl; jj++) {
      t.wait(me + PT_SC + (jj & 3), jj >> 2);
      for (int p = 0; p < 4 / SS; p++, k++) { t.wait(me + PT_D_FULL + (k & 1), k >> 1); t.arrive(PT_D_EMPTY + (k & 1)); }
    }
  }
  return t.n;
}
static int px1_count(int b, int UW) { return b < 8 ? 2 * UW : b >= 32 && b < 36 ? 16 : b >= 16 && b < 20 ? 2 : b >= 36 && b < 40 ? 4 : b >= 44 ? UW : 1; }
template <int FMT> static int pt_trace(PfTrace &t, int units, int nsl, int agent) {
  constexpr int NB = PT_NB, SPB = 4 / px_slot_stages(PT_RU), NP = pt_items(FMT), SI = 4 / NP, ND = 128 / (2 * PT_RU), CH = px_chunk(FMT), NRAW = pt_raws(FMT);
  const int rank = agent / 20, w = agent % 20, me = rank * PT_BARS;
  if (agent >= 40) return -1;
  if (w < 8) {
    const int g = w >> 2;
    int it = 0, rk = 0, jj = 0;
    for (int u = 0; u < units; u++)
      for (int c = 0; c < nsl; c++, jj++) {
        if (c % CH == 0) t.wait(me + PT_RAW_FULL + rk % NRAW, rk / NRAW);
        if ((jj & 1) == g)
          for (int p = 0; p < NP; p++, it++) {
            t.free_again(me + PT_A_EMPTY + 2 * g + (it & 1), it >> 1);
            if (p == 0) t.arrive(me + PT_SC + (jj & 3));
            t.arrive(PT_A_FULL + 2 * g + (it & 1));
          }
        if (c % CH == CH - 1 || c == nsl - 1) { t.arrive(me + PT_RAW_EMPTY + rk % NRAW); rk++; }
      }
  } else if (w == 8) pt_weights(t, me, NRAW, CH, units, nsl);
  else if (w == 9) pt_activations(t, rank, NB, units * nsl * SPB);
  else if (w < 12) {
    if (rank == 1) { if (w == 11) pt_forward(t, NB, units * nsl * SPB); }
    else {
      const int g = w - 10;
      for (int jj = g, it = 0; jj < units * nsl; jj += 2)
        for (int p = 0; p < NP; p++, it++) {
          const int buf = 2 * g + (it & 1), dbar = 2 * g + it % ND, sl = (jj * SPB + p * SPB / NP) % NB, in = p * SI - (p * SPB / NP) * (4 / SPB);
          if (it >= ND) t.wait(PT_D_EMPTY + dbar, it / ND - 1);
          if (in == 0) t.wait(PT_B_FULL + sl, jj * SPB / NB);
          t.wait(PT_A_FULL + buf, it >> 1);
          pt_both(t, PT_A_EMPTY + buf);
          if (in + SI == 4 / SPB) pt_both(t, PT_B_EMPTY + sl);
          pt_both(t, PT_D_FULL + dbar);
        }
    }
  } else {
    for (int jj = 0; jj < units * nsl; jj++)
      for (int p = 0; p < NP; p++) {
        const int g = jj & 1, it = (jj >> 1) * NP + p, dbar = 2 * g + it % ND;
        if (p == 0) t.wait(me + PT_SC + (jj & 3), jj >> 2);
        t.wait(me + PT_D_FULL + dbar, it / ND);
        t.arrive(PT_D_EMPTY + dbar);
      }
  }
  return t.n;
}
static int pt_count(int b) { return b < 8 || b >= 44 ? 8 : b >= 32 && b < 36 ? 16 : b >= 16 && b < 20 ? 2 : b >= 36 && b < 40 ? 4 : 1; }
static int px2_trace(PfTrace &t, int units, int nsl, int agent) {
  const int rank = agent / 16, w = agent % 16, me = rank * PT_BARS, NA = PX2_NA, NB = PX2_NB;
  if (agent >= 32) return -1;
  if (w < 4) {
    for (int jj = 0, k = 0; jj < units * nsl; jj++) {
      t.wait(me + PT_RAW_FULL + jj % PX2_NRAW, jj / PX2_NRAW);
      for (int s = 0; s < 4; s++, k++) {
        t.free_again(me + PT_A_EMPTY + k % NA, k / NA);
        if (s == 0) t.arrive(me + PT_SC + (jj & 3));
        t.arrive(PT_A_FULL + k % NA);
      }
      t.arrive(me + PT_RAW_EMPTY + jj % PX2_NRAW);
    }
  } else if (w == 4) pt_weights(t, me, PX2_NRAW, 1, units, nsl);
  else if (w == 5) pt_activations(t, rank, NB, units * nsl * 8);
  else if (w == 6 && rank == 0) {
    for (int jj = 0; jj < units * nsl; jj++) {
      if (jj > 1) t.wait(PT_D_EMPTY + (jj & 1), (jj >> 1) - 1);
      for (int i = 0; i < 8; i++) {
        const int s = i & 3, k = 4 * jj + s, as = k % NA;
        if (i < 4) t.wait(PT_A_FULL + as, k / NA);
        t.wait(PT_B_FULL + s, 2 * jj + (i >> 2));
        pt_both(t, PT_B_EMPTY + s);
        if (i >= 4) pt_both(t, PT_A_EMPTY + as);
        if (i == 7) pt_both(t, PT_D_FULL + (jj & 1));
      }
    }
  } else if (w == 7 && rank == 1) pt_forward(t, NB, units * nsl * 8);
  else if (w >= 8) {
    for (int jj = 0; jj < units * nsl; jj++) { t.wait(me + PT_SC + (jj & 3), jj >> 2); t.wait(me + PT_D_FULL + (jj & 1), jj >> 1); t.arrive(PT_D_EMPTY + (jj & 1)); }
  }
  return t.n;
}
static int px2_count(int b) { return b < 8 ? 8 : b >= 32 && b < 36 ? 16 : b >= 16 && b < 20 ? 2 : b >= 36 && b < 40 || b >= 44 ? 4 : 1; }
// kernel: 0 k_pf_attn (form: head dimension; units x nsl tiles of positions), 1 k_pfx1 / k_pft of `form` rows, 2 k_pfx2
extern "C" __attribute__((visibility("default")))
int llb_b200_pf_trace(int kernel, int form, int fmt, int units, int nsl, int agent, int *ops, int cap) {
  PfTrace t{ops, cap};
  if (kernel == 0) return form == 128 || form == 256 ? pa_trace(t, pa_slots(form), units * nsl, agent) : -1;
#define PT_ALL(F) (form == 32 ? pt_trace<F>(t, units, nsl, agent) : form == 64 ? px1_trace<F, 64>(t, units, nsl, agent) : px1_trace<F, 128>(t, units, nsl, agent))
  if (kernel == 1)
    switch (fmt) {
      case LLB_FM_Q4_K: return PT_ALL(LLB_FM_Q4_K);
      case LLB_FM_Q5_K: return PT_ALL(LLB_FM_Q5_K);
      case LLB_FM_Q6_K: return PT_ALL(LLB_FM_Q6_K);
      case LLB_FM_Q8_0: return PT_ALL(LLB_FM_Q8_0);
      default: return -1;
    }
#undef PT_ALL
  return kernel == 2 ? px2_trace(t, units, nsl, agent) : -1;
}
// arrivals that complete a phase of barrier `bar`
extern "C" __attribute__((visibility("default")))
int llb_b200_pf_bar_count(int kernel, int form, int fmt, int bar) {
  bar %= PT_BARS;
  return kernel == 0 ? pa_count(bar) : kernel == 2 ? px2_count(bar) : form == 32 ? pt_count(bar) : px1_count(bar, px1_unpack(fmt, form));
}
