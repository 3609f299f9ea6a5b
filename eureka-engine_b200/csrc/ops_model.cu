// ops_model.cu -- the non-GEMM device ops of the verify / draft passes, T rows per launch.
// Each kernel restates one or more of the reference's llb_t_* row kernels
// (tools/payload-spec2.patch:35-483); the arithmetic follows the CPU engine
// (tools/qwen35_engine.c:510-778), which is what parity is judged against.
#include <cooperative_groups.h>

#include "model.cuh"
#include "rowops.cuh"
#include "tc5.cuh"
namespace cg = cooperative_groups;

// sum over the block; every thread gets the result (red: >= 32 floats of shared memory)
__device__ __forceinline__ float block_sum(float v, float *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  float t = 0.0f;
  for (int i = 0; i < nw; i++) t += red[i];
  return t;
}
static Streams g_streams = {1 << 30, 0};
void ops_set_streams(int per, int stride) { g_streams.per = per > 0 ? per : 1 << 30; g_streams.stride = stride; }
Streams ops_streams(void) { return g_streams; }

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// ---- embedding rows (llb_embedk, tools/payload-kpair.patch:526) ---------------------------------
__global__ void k_embed(int fmt, const uint8_t *__restrict__ W, int d, const RowSet *rs, Streams sg, float *__restrict__ x) {
  int rs_n, rs_p0, tl;
  const int t = blockIdx.y;
  rs = rs_begin_row(rs, sg, t, rs_n, rs_p0, tl);
  if (tl >= rs_n) return;
  const int row = __ldcg(&rs->tok[tl]);   // (a draft's token was written by the kernel two launches in front)
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d; c += gridDim.x * blockDim.x) x[(size_t)t * d + c] = deq_elem(fmt, W, d, row, c);
}
int op_embed(cudaStream_t s, int fmt, const uint8_t *W, int d, const RowSet *rs, int Tmax, float *x) {
  CU_OK(llb_launch(k_embed, dim3((d + 255) / 256, Tmax), dim3(256), (size_t)(0), s, fmt, W, d, rs, g_streams, x));
  CU_OK(cudaGetLastError());
  return 0;
}

// ---- residual add + RMSNorm -> activation planes (llb_t_rnaddq / llb_t_rnormq,
// tools/payload-spec2.patch:35-112; rms_norm tools/qwen35_engine.c:510-515) ----------------------
// v = xin + sum(partials); xout = v (optional); h = (v * s) * w, s = 1/sqrt(mean(v^2) + eps);
// h goes to the planes at column offset xp_col0 and, optionally, to hn_out as f32.
// A row is a cluster of CL blocks (one, where the row is short), each with its part of the columns, four consecutive ones a
// thread (float4 loads and stores).  What bounds it is one SM's way to L2: a row of 5120 columns in eleven K-slices is 245 KB, 1.9 us
// through one SM's port; in four it and the blocks' sums, pushed to the peers with st.async, take less.  The 27B shape's passes took
// 1.2 % longer with a block a row, the 35B-A3B shape's (2048 columns) 1.3 %.
#define NORM_MAXT 1024
#define NORM_CL 4
template <int NI, int CL>
__global__ void __launch_bounds__(NORM_MAXT) k_norm_xp(const float *__restrict__ xin, PartIn add, const float *__restrict__ w, float eps, int d,
                                                       float *__restrict__ xout, XPlanes xp, int xp_col0, float *__restrict__ hn_out,
                                                       const RowSet *rs, Streams sg, int zero_if_pos0, unsigned int *err) {
  __shared__ float red[32], part[CL];
  __shared__ __align__(8) uint64_t bar;
  const uint32_t bar_s = smem_u32(&bar);
  const int rank = CL > 1 ? blockIdx.x % CL : 0, dc = CL > 1 ? d / CL : d, cb = rank * dc;   // this block's columns cb .. cb + dc - 1
  if constexpr (CL > 1) {
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_s) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_s), "r"(4u * CL) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  // the norm weights depend on no kernel: their trip to DRAM overlaps the wait on the producer
  float4 wv[NI], v[NI];
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    wv[i] = c < dc ? __ldg((const float4 *)(w + cb + c)) : v[i];
  }
  int rs_n, rs_p0, tl;
  const int t = blockIdx.x / CL;
  rs = rs_begin_row(rs, sg, t, rs_n, rs_p0, tl);
  if constexpr (CL > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every peer's barrier is there
  if (tl >= rs_n) return;   // every block of the row takes this exit
  const bool zero = zero_if_pos0 && (rs_p0 + tl == 0);
  const size_t row = (size_t)t * d + cb;
  if (xin && !zero) {
#pragma unroll
    for (int i = 0; i < NI; i++) {
      const int c = 4 * (threadIdx.x + i * blockDim.x);
      if (c < dc) v[i] = __ldcg((const float4 *)(xin + row + c));
    }
  }
  if (add.p && !zero) {
    // four slices of every group in flight a trip, added in slice order
    const float *pk = add.p + row;
#pragma unroll 1
    for (int k = 0; k < add.ns; k += 4, pk += 4 * add.stride) {
      float4 l[4][NI];
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < NI; i++) {
          const int c = 4 * (threadIdx.x + i * blockDim.x);
          l[q][i] = (c < dc && k + q < add.ns) ? __ldcg((const float4 *)(pk + (size_t)q * add.stride + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < NI; i++) { v[i].x += l[q][i].x; v[i].y += l[q][i].y; v[i].z += l[q][i].z; v[i].w += l[q][i].w; }
    }
  }
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);
    if (xout && c < dc) *(float4 *)(xout + row + c) = v[i];
    ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;   // (zeros past the row's end)
  }
  const int lane = threadIdx.x & 31, nwp = blockDim.x >> 5;
  ss = warp_sum(ss);
  if (lane == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = warp_sum(lane < nwp ? red[lane] : 0.0f);
  if constexpr (CL > 1) {
    if (threadIdx.x < CL) cl_push(smem_u32(&part[rank]), ss, bar_s, lane);
    if (!cl_wait(bar_s) && threadIdx.x == 0) atomicExch(err, 1u);   // (a block leaves when every push to it is there)
    ss = part[0];
#pragma unroll
    for (int i = 1; i < CL; i++) ss += part[i];
  }
  const float sc = 1.0f / sqrtf(ss / (float)d + eps);
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const int c = 4 * (threadIdx.x + i * blockDim.x);   // eight lanes hold 32 consecutive columns
    const float h[4] = {v[i].x * sc * wv[i].x, v[i].y * sc * wv[i].y, v[i].z * sc * wv[i].z, v[i].w * sc * wv[i].w};
    if (c < dc && hn_out) *(float4 *)(hn_out + row + c) = make_float4(h[0], h[1], h[2], h[3]);
    xp_store4(xp, t, 2, xp_col0 + cb + c, h, lane, c < dc);
  }
}
// Four blocks a row from NORM_SPLIT columns on (whole groups of 32 columns to each), one below: 1024 columns are one trip of one block.
#define NORM_SPLIT 2048
int op_norm_xp(cudaStream_t s, const float *xin, PartIn add, const float *w, float eps, int d, float *xout, XPlanes xp,
               int xp_col0, float *hn_out, const RowSet *rs, int Tmax, int zero_if_pos0) {
  if (d % 32 || xp_col0 % 32 || d > 4 * 4 * NORM_MAXT) return llb_fail("norm: d %d at column %d", d, xp_col0);
  const bool split = d >= NORM_SPLIT && d % (32 * NORM_CL) == 0;
  const int d4 = d / 4 / (split ? NORM_CL : 1), ni = (d4 + NORM_MAXT - 1) / NORM_MAXT;
  const int threads = (((d4 + ni - 1) / ni) + 31) & ~31;
  if (split) {   // (d / 4 / NORM_CL <= NORM_MAXT)
    CU_OK(llb_launch_cluster(k_norm_xp<1, NORM_CL>, dim3(Tmax * NORM_CL), dim3(threads), NORM_CL, s, xin, add, w, eps, d, xout, xp, xp_col0, hn_out, rs, g_streams, zero_if_pos0, gemm_err_word()));
    return 0;
  }
#define NORM_GO(NI) CU_OK(llb_launch(k_norm_xp<NI, 1>, dim3(Tmax), dim3(threads), (size_t)(0), s, xin, add, w, eps, d, xout, xp, xp_col0, hn_out, rs, g_streams, zero_if_pos0, gemm_err_word()))
  switch (ni) {
    case 1: NORM_GO(1); break;
    case 2: NORM_GO(2); break;
    case 3: NORM_GO(3); break;
    default: NORM_GO(4); break;
  }
#undef NORM_GO
  return 0;
}

// ---- silu(gate) * up -> planes (llb_t_siluq, tools/payload-spec2.patch:114-124) -----------------
__global__ void __launch_bounds__(256) k_silu_xp(PartIn g, PartIn u, int f, XPlanes xp, const RowSet *rs, Streams sg) {
  int rs_n, rs_p0, tl;
  const int t = blockIdx.y, lane = threadIdx.x & 31;
  rs = rs_begin_row(rs, sg, t, rs_n, rs_p0, tl);
  if (tl >= rs_n) return;
  const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);   // four columns per thread, eight lanes per 32-column group
  const bool on = c < f;
  float h[4] = {0.f, 0.f, 0.f, 0.f};
  if (on) {
    const size_t i = (size_t)t * f + c;
    float4 gv = make_float4(0.f, 0.f, 0.f, 0.f), uv = gv;
    const float *pg = g.p + i, *pu = u.p + i;
    const int ns = max(g.ns, u.ns);
#pragma unroll 1
    for (int k = 0; k < ns; k += 2, pg += 2 * g.stride, pu += 2 * u.stride) {   // both matrices' slices in flight together
      float4 l[2], m[2];
#pragma unroll
      for (int q = 0; q < 2; q++) {
        l[q] = k + q < g.ns ? __ldcg((const float4 *)(pg + q * g.stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
        m[q] = k + q < u.ns ? __ldcg((const float4 *)(pu + q * u.stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < 2; q++) {
        gv.x += l[q].x; gv.y += l[q].y; gv.z += l[q].z; gv.w += l[q].w;
        uv.x += m[q].x; uv.y += m[q].y; uv.z += m[q].z; uv.w += m[q].w;
      }
    }
    h[0] = silu_f(gv.x) * uv.x; h[1] = silu_f(gv.y) * uv.y; h[2] = silu_f(gv.z) * uv.z; h[3] = silu_f(gv.w) * uv.w;
  }
  xp_store4(xp, t, 2, c, h, lane, on);
}
int op_silu_xp(cudaStream_t s, PartIn g, PartIn u, int f, XPlanes xp, const RowSet *rs, int Tmax) {
  if (f % 32) return llb_fail("silu: f %d", f);
  CU_OK(llb_launch(k_silu_xp, dim3((f / 4 + 255) / 256, Tmax), dim3(256), (size_t)(0), s, g, u, f, xp, rs, g_streams));
  CU_OK(cudaGetLastError());
  return 0;
}

// ---- the router of a routed-expert layer (host/llb_host.c:622-724; llb_moe_topk of tools/payload-moeany.patch) ----
// Router logits lg[t][r] = W[r] . h[t] for the ne router rows and the shared expert's gate row (row ne): F32
// weights, a block per row, all rows of the pass; the gate|up launch makes the choice from them (moe.cuh).  Bound by the one trip
// to L2 for the rows of h, so four rows are in flight at a time: row by row, each trip behind the last, sixteen rows
// took 21 us.
__global__ void __launch_bounds__(256, 2) k_moe_router(const float *__restrict__ W, const float *__restrict__ h, int d, int ne, float *__restrict__ lg, const RowSet *rs, int n_all) {
  int rs_n, rs_p0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = blockIdx.x, nrows = ne + 1;
  __shared__ float red[8][MOE_MAXROWS];
  // the row's weights depend on no kernel: fetched before the wait (two float4 per thread cover d <= 2048)
  const float4 *wr = (const float4 *)(W + (size_t)r * d);
  const int c0 = threadIdx.x, c1 = threadIdx.x + 256, nc = d / 4;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 w0 = c0 < nc ? __ldg(wr + c0) : z4, w1 = c1 < nc ? __ldg(wr + c1) : z4;
  rs = rs_begin(rs, rs_n, rs_p0);
  if (n_all > 0) rs_n = n_all;   // a pass over several streams: every row of the pass (a stream's idle rows cost nothing that matters)
#pragma unroll 1
  for (int t0 = 0; t0 < rs_n; t0 += 4) {
    float4 a[4], b[4];
    float acc[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float4 *x = (const float4 *)(h + (size_t)min(t0 + q, rs_n - 1) * d);
      a[q] = c0 < nc ? __ldcg(x + c0) : z4;
      b[q] = c1 < nc ? __ldcg(x + c1) : z4;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      acc[q] = (w0.x * a[q].x + w0.y * a[q].y) + (w0.z * a[q].z + w0.w * a[q].w);
      acc[q] += (w1.x * b[q].x + w1.y * b[q].y) + (w1.z * b[q].z + w1.w * b[q].w);
    }
    for (int c = threadIdx.x + 512; c < nc; c += 256) {
      const float4 w = __ldg(wr + c);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float4 v = __ldcg((const float4 *)(h + (size_t)min(t0 + q, rs_n - 1) * d) + c);
        acc[q] += (w.x * v.x + w.y * v.y) + (w.z * v.z + w.w * v.w);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float v = warp_sum(acc[q]);
      if (lane == 0) red[warp][t0 + q] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < rs_n) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; w++) v += red[w][threadIdx.x];
    lg[(size_t)threadIdx.x * nrows + r] = v;
  }
}
int op_moe_logits(cudaStream_t s, const float *Wr, const float *h, int d, int ne, float *lg, const RowSet *rs, int Tmax) {
  if (Tmax > MOE_MAXROWS) return llb_fail("moe route: %d rows in a pass (at most %d)", Tmax, MOE_MAXROWS);
  if (ne < 1 || ne > 1024 || d % 4) return llb_fail("moe route: %d experts, d %d", ne, d);
  CU_OK(llb_launch(k_moe_router, dim3(ne + 1), dim3(256), (size_t)(0), s, Wr, h, d, ne, lg, rs, g_streams.stride ? Tmax : 0));
  return 0;
}

// ---- per-head QK RMSNorm + partial NEOX RoPE; K and V rows straight into their cache slots
// (llb_t_qkr, tools/payload-spec2.patch:159-204; tools/qwen35_engine.c:523-533, 667-690) ----------
// grid (H + 2 KV, Tmax), block hd.  q input rows are [H][q(hd) | gate(hd)].  The cache keeps a value as two
// fp16 numbers in two planes kv_plane halves apart, hi = fp16(x) and lo = fp16((x - hi) * 2048): the bytes
// of the f32, in the form the attention kernel's tensor-core operands take.
__global__ void k_qkrope(PartIn q, PartIn k, PartIn v, const float *__restrict__ qn_w, const float *__restrict__ kn_w,
                         const double *__restrict__ invfreq, AttnShape sh, float *__restrict__ qout, __half *__restrict__ Kc,
                         __half *__restrict__ Vc, const RowSet *rs, Streams sg, int blk0) {
  int rs_n, rs_p0, tl;
  const int t = blockIdx.y, b = blockIdx.x + blk0, i = threadIdx.x, hd = sh.hd;
  rs = rs_begin_row(rs, sg, t, rs_n, rs_p0, tl);
  extern __shared__ float hv[];
  __shared__ float red[32];
  if (tl >= rs_n) return;
  const int pos = rs_p0 + tl, kvd = sh.KV * hd;
  Kc += (size_t)(t / sg.per) * sh.kv_group; Vc += (size_t)(t / sg.per) * sh.kv_group;   // the row's stream has its own cache
  if (b >= sh.H + sh.KV) {  // V row: copied
    const int g = b - sh.H - sh.KV;
    kv_put(Vc, sh.kv_plane, (size_t)pos * kvd + g * hd + i, part_get(v, (size_t)t * kvd + g * hd + i));
    return;
  }
  float x;
  const float *nw;
  float *dst = nullptr;
  size_t kdst = 0;
  if (b < sh.H) {
    x = part_get(q, (size_t)t * 2 * sh.H * hd + (size_t)b * 2 * hd + i);
    nw = qn_w;
    dst = qout + ((size_t)t * sh.H + b) * hd;
  } else {
    const int g = b - sh.H;
    x = part_get(k, (size_t)t * kvd + g * hd + i);
    nw = kn_w;
    kdst = (size_t)pos * kvd + g * hd;
  }
  const float ss = block_sum(x * x, red);
  const float sc = 1.0f / sqrtf(ss / (float)hd + sh.eps);
  const float y = x * sc * nw[i];
  hv[i] = y;
  __syncthreads();
  float out = y;
  const int half = sh.rope_dim >> 1;
  if (i < sh.rope_dim) {
    const int pi = i < half ? i : i - half;
    const float th = (float)((double)pos * invfreq[pi]);
    const float c = (float)cos((double)th), sn = (float)sin((double)th);
    const float a = hv[pi], bb = hv[pi + half];
    out = i < half ? __fsub_rn(__fmul_rn(a, c), __fmul_rn(bb, sn)) : __fadd_rn(__fmul_rn(a, sn), __fmul_rn(bb, c));
  }
  if (dst) dst[i] = out;
  else kv_put(Kc, sh.kv_plane, kdst + i, out);
}
int op_qkrope(cudaStream_t s, PartIn q, PartIn k, PartIn v, const float *qn_w, const float *kn_w, const double *invfreq,
              AttnShape sh, float *qout, float *Kc, float *Vc, const RowSet *rs, int Tmax, bool kv_only) {
  // blocks 0 .. H-1 are the query heads, then KV key heads, then KV value heads
  const int blk0 = kv_only ? sh.H : 0;
  CU_OK(llb_launch(k_qkrope, dim3(sh.H + 2 * sh.KV - blk0, Tmax), dim3(sh.hd), (size_t)((size_t)sh.hd * 4), s, q, k, v, qn_w, kn_w, invfreq, sh, qout,
                   (__half *)Kc, (__half *)Vc, rs, g_streams, blk0));
  CU_OK(cudaGetLastError());
  return 0;
}

// ---- gated DeltaNet ------------------------------------------------------------------------------
// conv1d + SiLU over the position-indexed ring, gates, the recurrent scan over the T rows with per-row state checkpoints,
// then the gated RMSNorm of each head's output into the planes of ssm_out's input: one kernel
// (llb_t_midconv, llb_t_l2qk + llb_t_gdl, llb_t_grn, tools/payload-spec2.patch:319-447; tools/qwen35_engine.c:589-654).
// grid (TR, 4) in clusters of four blocks = one value head, 256 threads: block (hh, jq) owns state rows j = 32 jq .. + 31 of
// head hh, 16 registers of state per thread (thread = row jr, column eighth cq).  The state is read from ring slot sc and
// the state after row r is written to slot (sc + r + 1) % R, so rejecting rows costs nothing: the next cycle simply starts
// from the slot of the last served row.
//
// What bounds it is a chain of latencies, not bytes (a 27B layer moves 16 MB of state in 2.4 us; conv and scan as two kernels
// took 3 + 13 us of a four-row pass).  What keeps the chain short: the conv is part of the kernel (every block redoes the 256
// q and k channels of its group; with all rows x slices of the ring in flight as float4 loads that is one trip to L2 and one
// launch less, where row by row and slice by slice the trips took 20 us); inputs are requested long before their use; the gates' double-precision functions run in the last warp while its loads and the other warps' conv do; and the
// sums of squares of the gated norm are pushed into the peers' shared memory and cost one cluster barrier, behind which
// the gate factors are made.
#define DL_THREADS 256
#define DL_ALONE (104 * 1024)   // dynamic shared memory of a block that wants its SM for itself
#define DL_MAXR (SPEC_MAXT + CONV_RING / 2 - 1)   // history rows of a pass: n + KC - 1
__device__ __forceinline__ float4 dl_slice(const PartIn &a, size_t i, int k) {
  return k < a.ns ? __ldcg((const float4 *)(a.p + i + k * a.stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void add4(float4 &v, const float4 l) { v.x += l.x; v.y += l.y; v.z += l.z; v.w += l.w; }
__global__ void __cluster_dims__(1, 4, 1) __launch_bounds__(DL_THREADS, 2)
k_delta(float *__restrict__ S, const SpecCtl *__restrict__ ctl, PartIn ring, const float *__restrict__ cw, PartIn bp, PartIn ap,
        const float *__restrict__ dt, const float *__restrict__ sa, PartIn z, const float *__restrict__ nw, DeltaShape sh, XPlanes xp,
        const RowSet *rs, Streams sg, long long s_group) {
  __shared__ __align__(16) float raw[DL_MAXR][288];          // channels: q 128 | k 128 | v 32 (this block's)
  __shared__ __align__(16) float ys[SPEC_MAXT][288], os[SPEC_MAXT][32];
  __shared__ float db[SPEC_MAXT][2], tot[SPEC_MAXT][4];
  cg::cluster_group cl = cg::this_cluster();
  const int hh = blockIdx.x, jq = blockIdx.y, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int g = hh % sh.GK, jr = tid >> 3, cq = tid & 7, KC = sh.KC;
  const size_t slot_sz = (size_t)sh.TR * 128 * 128;
  // The committed state (ring slot sc) was written by an earlier pass and sc by that pass's accept kernel, and the row set
  // likewise (rs_stable): neither depends on the kernel in front, so the 16 KB of state that a block reads from HBM, and the
  // conv's taps, are requested before the dependency wait.
  pdl_trigger();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // waited for before the first push: every peer runs
  // blockIdx.z: the stream -- its control block, its state ring, its rows of the pass
  ctl = (const SpecCtl *)((const char *)ctl + (size_t)blockIdx.z * sg.stride);
  const bool early = (uintptr_t)rs & 1u;
  rs = (const RowSet *)(((uintptr_t)rs & ~(uintptr_t)1) + (size_t)blockIdx.z * sg.stride);
  const int row0 = sg.stride ? blockIdx.z * sg.per : 0;
  const int R = *(const volatile int *)&ctl->R, sc = *(const volatile int *)&ctl->sc;
  int n = 0, pos0 = 0;
  if (early) { n = *(const volatile int *)&rs->n; pos0 = *(const volatile int *)&rs->pos0; }
  float *St = S + blockIdx.z * s_group + (size_t)hh * 128 * 128 + (size_t)(32 * jq + jr) * 128 + 4 * cq;   // columns 4 cq + 32 i ..
  float st[16];
#pragma unroll
  for (int i = 0; i < 4; i++) { const float4 v = __ldcg((const float4 *)(St + (size_t)sc * slot_sz) + 8 * i); st[4 * i] = v.x; st[4 * i + 1] = v.y; st[4 * i + 2] = v.z; st[4 * i + 3] = v.w; }
  // the conv's channels: tid and, in the first two warps, tid + 224, of the first seven warps; up to four taps kept in registers
  float tap[2][4];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int c = tid + 224 * j, cc = c < 128 ? g * 128 + c : c < 256 ? sh.kdc + g * 128 + c - 128 : 2 * sh.kdc + hh * 128 + 32 * jq + c - 256;
    const float *w = cw + (size_t)cc * KC + KC - 1;
#pragma unroll
    for (int k = 0; k < 4; k++) tap[j][k] = wp < (j ? 2 : 7) && k < KC ? __ldg(w - k) : 0.0f;
  }
  const float dtv = __ldg(dt + hh), sav = __ldg(sa + hh);
  // rows this thread writes at the end: row zt, columns zc .. of the block's 32 (the first two warps)
  const int zt = 4 * wp + (lane >> 3), zc = 4 * (lane & 7), col = hh * 128 + 32 * jq + zc;
  const size_t zi = (size_t)(row0 + zt) * sh.vdc + col;
  pdl_wait();
  if (!early) { n = __ldcg(&rs->n); pos0 = __ldcg(&rs->pos0); }
  const int nr = n + KC - 1;
  if (n < 1) { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); return; }   // every block of the cluster takes the same exit
  // the gates' inputs, then the ring rows, then (behind them, for the end) z: four slices of each in flight
  float gl[4], hl[4];
  const size_t gi = (size_t)(row0 + lane) * sh.TR + hh;
  const bool gon = wp == 7 && lane < n, zon = zt < n;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    gl[k] = gon && k < bp.ns ? __ldcg(bp.p + gi + k * bp.stride) : 0.0f;
    hl[k] = gon && k < ap.ns ? __ldcg(ap.p + gi + k * ap.stride) : 0.0f;
  }
  // history row r is position pos0 - (KC - 1) + r.  Item = (row, four channels); a stream's ring is [K-slice][CONV_RING slots].
  // (Every thread makes one trip at least: the last warp's gates are in it, however few items a short conv kernel leaves.)
  const float *rp = ring.p + (size_t)blockIdx.z * ring.ns * CONV_RING * sh.convd;
  const int items = KC > 3 ? nr * 72 : max(nr * 72, DL_THREADS);
#pragma unroll 1
  for (int i0 = tid; i0 < items; i0 += 2 * DL_THREADS) {
    float4 v[2], l[4][2];
    const float *p[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = min(i0 + DL_THREADS * q, nr * 72 - 1), r = i / 72, c4 = i - r * 72;
      const int c = c4 < 32 ? g * 128 + 4 * c4 : c4 < 64 ? sh.kdc + g * 128 + 4 * (c4 - 32) : 2 * sh.kdc + hh * 128 + 32 * jq + 4 * (c4 - 64);
      p[q] = rp + (size_t)((pos0 - (KC - 1) + r) & (CONV_RING - 1)) * sh.convd + c;
      v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int q = 0; q < 2; q++) l[u][q] = u < ring.ns ? __ldcg((const float4 *)(p[q] + u * ring.stride)) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (gon && i0 < DL_THREADS) {
      // gates, while the rows are on their way: decay = exp(softplus(a + dt) ssm_a), beta = sigmoid(b)
      float b = 0.0f, x = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; k++) { b += gl[k]; x += hl[k]; }
      for (int k = 4; k < bp.ns; k++) b += __ldcg(bp.p + gi + k * bp.stride);
      for (int k = 4; k < ap.ns; k++) x += __ldcg(ap.p + gi + k * ap.stride);
      x += dtv;
      float sp = x;
      if (x <= 20.0f) sp = (float)log1p((double)(float)exp((double)x));
      db[lane][0] = (float)exp((double)(sp * sav));
      db[lane][1] = 1.0f / (1.0f + (float)exp((double)-b));
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int q = 0; q < 2; q++) add4(v[q], l[u][q]);
#pragma unroll 1
    for (int k = 4; k < ring.ns; k++) { add4(v[0], __ldcg((const float4 *)(p[0] + k * ring.stride))); add4(v[1], __ldcg((const float4 *)(p[1] + k * ring.stride))); }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int i = i0 + DL_THREADS * q, r = i / 72;
      if (i < nr * 72) *(float4 *)&raw[r][4 * (i - r * 72)] = v[q];
    }
  }
  float4 zl[4];
#pragma unroll
  for (int k = 0; k < 4; k++) zl[k] = zon ? dl_slice(z, zi, k) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 nwv = __ldg((const float4 *)(nw + 32 * jq + zc));
  __syncthreads();
  // conv: tap KC-1 is the current token (tools/qwen35_engine.c:599-600); thread = channel
  if (KC <= 4) {
#pragma unroll
    for (int j = 0; j < 2; j++) {
      if (wp >= (j ? 2 : 7)) break;
      const int c = tid + 224 * j;
      // the history slides through h; a tap that is not used adds exactly zero to the sum
      float h1 = KC > 3 ? raw[KC - 4][c] : 0.0f, h2 = KC > 2 ? raw[KC - 3][c] : 0.0f, h3 = raw[KC - 2][c];
#pragma unroll 2
      for (int t = 0; t < n; t++) {
        const float h = raw[t + KC - 1][c];
        float a = __fadd_rn(0.0f, __fmul_rn(h1, tap[j][3]));
        a = __fadd_rn(a, __fmul_rn(h2, tap[j][2]));
        a = __fadd_rn(a, __fmul_rn(h3, tap[j][1]));
        a = __fadd_rn(a, __fmul_rn(h, tap[j][0]));
        ys[t][c] = silu_f(a);
        h1 = h2; h2 = h3; h3 = h;
      }
    }
  } else {
#pragma unroll 1
    for (int c = tid; c < 288; c += DL_THREADS) {
      const int cc = c < 128 ? g * 128 + c : c < 256 ? sh.kdc + g * 128 + c - 128 : 2 * sh.kdc + hh * 128 + 32 * jq + c - 256;
#pragma unroll 1
      for (int t = 0; t < n; t++) {
        float a = 0.0f;
        for (int k = 0; k < KC; k++) a = __fadd_rn(a, __fmul_rn(raw[t + k][c], __ldg(cw + (size_t)cc * KC + k)));
        ys[t][c] = silu_f(a);
      }
    }
  }
  __syncthreads();
  // L2 norms of q and k: a warp a row
#pragma unroll 1
  for (int i = wp; i < 2 * n; i += DL_THREADS / 32) {
    float4 *p = (float4 *)&ys[i >> 1][128 * (i & 1)] + lane;
    const float4 v = *p;
    const float nq = sqrtf(warp_sum((v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w)));
    float s = 1.0f / (nq > sh.eps ? nq : sh.eps);
    if (!(i & 1)) s *= 0.08838834764831845f;   // 1 / sqrt(128)
    *p = make_float4(v.x * s, v.y * s, v.z * s, v.w * s);
  }
  __syncthreads();
  int slot = sc;
#pragma unroll 1
  for (int t = 0; t < n; t++) {
    const float dec = db[t][0], bt = db[t][1];
    float kq[16], ka[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; i++) { const float4 v = *(const float4 *)&ys[t][128 + 32 * i + 4 * cq]; kq[4 * i] = v.x; kq[4 * i + 1] = v.y; kq[4 * i + 2] = v.z; kq[4 * i + 3] = v.w; }
#pragma unroll
    for (int i = 0; i < 16; i++) { st[i] *= dec; ka[i & 3] += st[i] * kq[i]; }
    float kvacc = (ka[0] + ka[1]) + (ka[2] + ka[3]);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) kvacc += __shfl_xor_sync(0xffffffffu, kvacc, m);
    const float delta = (ys[t][256 + jr] - kvacc) * bt;
    float oa[4] = {0.f, 0.f, 0.f, 0.f};
    slot = slot + 1 == R ? 0 : slot + 1;
    float4 *dst = (float4 *)(St + (size_t)slot * slot_sz);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float4 q = *(const float4 *)&ys[t][32 * i + 4 * cq];
      st[4 * i] += kq[4 * i] * delta; st[4 * i + 1] += kq[4 * i + 1] * delta; st[4 * i + 2] += kq[4 * i + 2] * delta; st[4 * i + 3] += kq[4 * i + 3] * delta;
      oa[0] += st[4 * i] * q.x; oa[1] += st[4 * i + 1] * q.y; oa[2] += st[4 * i + 2] * q.z; oa[3] += st[4 * i + 3] * q.w;
      dst[8 * i] = make_float4(st[4 * i], st[4 * i + 1], st[4 * i + 2], st[4 * i + 3]);
    }
    float oacc = (oa[0] + oa[1]) + (oa[2] + oa[3]);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1) oacc += __shfl_xor_sync(0xffffffffu, oacc, m);
    if (cq == 0) os[t][jr] = oacc;
  }
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  if (wp < n) {
    const float v = os[wp][lane], s2 = warp_sum(v * v);
    if (lane < 4) *cl.map_shared_rank(&tot[wp][jq], lane) = s2;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  float h[4] = {0.f, 0.f, 0.f, 0.f};
  if (zon) {   // rows 4 wp .. 4 wp + 3, eight lanes a row
    float4 zz = zl[0];
    add4(zz, zl[1]); add4(zz, zl[2]); add4(zz, zl[3]);
    for (int k = 4; k < z.ns; k++) add4(zz, dl_slice(z, zi, k));
    const float4 o = *(const float4 *)&os[zt][zc];
    h[0] = o.x * nwv.x * silu_f(zz.x); h[1] = o.y * nwv.y * silu_f(zz.y); h[2] = o.z * nwv.z * silu_f(zz.z); h[3] = o.w * nwv.w * silu_f(zz.w);
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // every block's sums of squares are here; nothing remote is touched after this
  if (wp < 2) {
    const float *tt = tot[zon ? zt : 0];
    const float r = 1.0f / sqrtf((((tt[0] + tt[1]) + tt[2]) + tt[3]) / 128.0f + sh.eps);   // rank order
#pragma unroll
    for (int i = 0; i < 4; i++) h[i] *= r;
    xp_store4(xp, row0 + zt, 2, col, h, lane, zon);
  }
}
int delta_setup(void) {
  CU_OK(cudaFuncSetAttribute(k_delta, cudaFuncAttributeMaxDynamicSharedMemorySize, DL_ALONE));
  return 0;
}
int op_delta(cudaStream_t s, float *S, const SpecCtl *ctl, PartIn ring, const float *cw, PartIn bp, PartIn ap, const float *dt, const float *sa,
             PartIn z, const float *nw, DeltaShape sh, XPlanes xp, const RowSet *rs, int nz, long long s_group) {
  if (sh.SZ != 128) return llb_fail("DeltaNet state size %d (only 128, as host/llb_host.c:1608)", sh.SZ);
  if (sh.KC > CONV_RING / 2) return llb_fail("conv kernel %d", sh.KC);
  // An SM's stores leave it at about 32 bytes a cycle, and two of a cluster's blocks on one SM share them (a row of the scan 0.64 us
  // there): where every block can have an SM, each asks for nearly half of the shared memory. 0.8B shape (32 blocks) 26.6 -> 25.7 and
  // 23.5 -> 22.7 ms a chat turn, both sides in turn on two machines, 35B-A3B shape (128 blocks) 109.2 -> 107.8 and 104.4 -> 102.5; with
  // more blocks than SMs there is nothing to spread.
  const size_t alone = 4 * sh.TR * nz <= g_llb.sms ? DL_ALONE : 0;
  CU_OK(llb_launch(k_delta, dim3(sh.TR, 4, nz), dim3(DL_THREADS), alone, s, S, ctl, ring, cw, bp, ap, dt, sa, z, nw, sh, xp, rs, g_streams, s_group));
  return 0;
}

// ---- top-2 over the logits (llb_t_amaxp / llb_t_amax, tools/payload-spec2.patch:450-483) ---------
// Order: larger value first, lower id on equal values (tools/qwen35_engine.c:763-778).
__global__ void __launch_bounds__(256) k_top2_part(PartIn logits, int V, long long row_stride,
                                                   float *__restrict__ part, const RowSet *rs, Streams sg) {
  int rs_n, rs_p0, tl;
  const int t = blockIdx.y;
  rs = rs_begin_row(rs, sg, t, rs_n, rs_p0, tl);
  __shared__ Top2 sh[8];
  if (tl >= rs_n) return;
  const size_t z0 = (size_t)t * row_stride;
  const int per = (V + gridDim.x - 1) / gridDim.x, i0 = blockIdx.x * per, i1 = min(V, i0 + per);
  Top2 a = {0.f, -1, 0.f, -1};
  // (four values of a thread in flight at a time: one by one, a vocabulary of 151936 took nine trips to L2)
#pragma unroll 1
  for (int i = i0 + threadIdx.x; i < i1; i += 4 * blockDim.x) {
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] = i + q * blockDim.x < i1 ? __ldcg(logits.p + z0 + i + q * blockDim.x) : 0.0f;
#pragma unroll 1
    for (int k = 1; k < logits.ns; k++) {
      const float *pk = logits.p + (size_t)k * logits.stride + z0 + i;
      float l[4];
#pragma unroll
      for (int q = 0; q < 4; q++) l[q] = i + q * blockDim.x < i1 ? __ldcg(pk + q * blockDim.x) : 0.0f;
#pragma unroll
      for (int q = 0; q < 4; q++) v[q] += l[q];
    }
#pragma unroll
    for (int q = 0; q < 4; q++) t2_push(a, v[q], i + q * blockDim.x < i1 ? i + q * (int)blockDim.x : -1);
  }
  a = t2_warp(a);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x < 32) {
    Top2 b = threadIdx.x < 8 ? sh[threadIdx.x] : Top2{0.f, -1, 0.f, -1};
    b = t2_warp(b);
    if (threadIdx.x == 0) {
      float *p = part + ((size_t)t * gridDim.x + blockIdx.x) * 4;
      p[0] = b.v1; p[1] = __int_as_float(b.i1); p[2] = b.v2; p[3] = __int_as_float(b.i2);
    }
  }
}
int op_top2_part(cudaStream_t s, PartIn logits, int V, long long row_stride, float *part, const RowSet *rs, int Tmax) {
  CU_OK(llb_launch(k_top2_part, dim3(TOP2_NB, Tmax), dim3(256), (size_t)(0), s, logits, V, row_stride, part, rs, g_streams));
  CU_OK(cudaGetLastError());
  return 0;
}
__device__ __forceinline__ Top2 t2_final(const float *part, int t, int lane) {
  Top2 a = {0.f, -1, 0.f, -1};
  float4 p[TOP2_NB / 32];
#pragma unroll
  for (int q = 0; q < TOP2_NB / 32; q++) p[q] = __ldcg((const float4 *)part + (size_t)t * TOP2_NB + lane + 32 * q);   // (to L2: every drafter step writes the same partials)
#pragma unroll
  for (int q = 0; q < TOP2_NB / 32; q++) { t2_push(a, p[q].x, __float_as_int(p[q].y)); t2_push(a, p[q].z, __float_as_int(p[q].w)); }
  return t2_warp(a);
}

// ---- fused argmax + accept/reject + commit -------------------------------------------------------
// The reference serves row r while the caller's next token equals the row's input
// (host/llb_host.c:1911) and advances the state ring by the rows served (:1932); under greedy
// sampling that is "accept while argmax(row j) == draft j+1" (host/llb_sampler_impl.h:400-405).
// Here the whole decision runs on the device and also prepares the next cycle: new p0, ring slot,
// committed token, and the drafter's catch-up rows (host/llb_host.c:1815).
__global__ void k_accept(const float *__restrict__ part, SpecCtl *__restrict__ ctl, SpecResult *__restrict__ ring, int ring_n, int per,
                         const int *__restrict__ smp_tok, const float *__restrict__ smp_val) {
  pdl_trigger();
  pdl_wait();
  __shared__ Top2 rows[SPEC_MAXT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // one block per stream: its control block, its result ring, its rows of the pass
  ctl += blockIdx.x; ring += (size_t)blockIdx.x * ring_n;
  const int row0 = blockIdx.x * per;
  const int T = __ldcg(&ctl->verify.n);
  if (T < 1) return;   // an empty pass (the sizing run at open, a stream that is not running) decides nothing
  if (warp < T) {
    Top2 a = t2_final(part, row0 + warp, lane);
    // sampling mode: the row's emitted token is the sampler's (llb_smp_verify / llb_smp_sample), not the argmax; the
    // argmax's runner-up stays in the record's third and fourth words
    if (smp_tok) { const int st = __ldcg(smp_tok + row0 + warp); if (a.i1 != st) { a.i2 = a.i1; a.v2 = a.v1; } a.i1 = st; a.v1 = __ldcg(smp_val + row0 + warp); }
    if (lane == 0) rows[warp] = a;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  const int p0 = __ldcg(&ctl->verify.pos0);
  int tin[SPEC_MAXT];   // the drafts were written by this cycle's earlier kernels
#pragma unroll
  for (int r = 0; r < SPEC_MAXT; r++) tin[r] = __ldcg(&ctl->verify.tok[r]);
  SpecResult *res = ring + (ctl->seq % (unsigned long long)ring_n);
  int served = 1;
  if (ctl->forced > 0) served = T;
  else {
#pragma unroll
    for (int r = 1; r < SPEC_MAXT; r++) if (served == r && r < T && rows[r - 1].i1 == tin[r]) served++;
  }
  res->p0 = p0; res->T = T; res->served = served;
  res->pad = (ctl->chk_on && (ctl->chk_pos != p0 || ctl->chk_tok != tin[0])) ? 1 : 0;
  ctl->chk_on = 0;
#pragma unroll
  for (int r = 0; r < SPEC_MAXT; r++) {
    res->tin[r] = r < T ? tin[r] : -1;
    res->ids[r] = r < T ? rows[r].i1 : -1;
    res->top2[r][0] = r < T ? (unsigned)rows[r].i1 : 0u;
    res->top2[r][1] = r < T ? __float_as_uint(rows[r].v1) : 0u;
    res->top2[r][2] = r < T ? (unsigned)rows[r].i2 : 0u;
    res->top2[r][3] = r < T ? __float_as_uint(rows[r].v2) : 0u;
  }
  // commit: the state after the last served row becomes the committed state
  ctl->sc = (ctl->sc + served) % ctl->R;
  const int np0 = p0 + served;
  // the drafter catches up over the served positions p0+1 .. p0+served, whose tokens are the
  // emitted ids (or the given prompt tokens), paired with the trunk's normed hidden rows 0..served-1
  ctl->catchup.n = served;
  ctl->catchup.pos0 = p0 + 1;
  for (int r = 0; r < served; r++) ctl->catchup.tok[r] = ctl->forced > 0 ? ctl->next_tok[r] : rows[r].i1;
  const int tok0 = ctl->catchup.tok[served - 1];
  if (ctl->hist)   // the prompt-lookup drafter searches the whole token history
    for (int r = 0; r < served; r++) ctl->hist[p0 + 1 + r] = ctl->catchup.tok[r];
  int Tn = ctl->k + 1;
  if (np0 + Tn > ctl->max_pos) Tn = ctl->max_pos - np0 > 0 ? ctl->max_pos - np0 : 1;
  ctl->verify.n = Tn;
  ctl->verify.pos0 = np0;
  ctl->verify.tok[0] = tok0;
  for (int r = 0; r < SPEC_MAXT; r++) ctl->verify.slot[r] = (np0 + r) & (CONV_RING - 1);
  ctl->forced = 0;
  __threadfence_system();
  res->seq = ctl->seq + 1;   // written last: the host polls it
  ctl->seq += 1;
}
int op_accept(cudaStream_t s, const float *part, SpecCtl *ctl, SpecResult *ring, int ring_n, int Tmax, int nz, int per, const int *smp_tok,
              const float *smp_val) {
  CU_OK(llb_launch(k_accept, dim3(nz), dim3(32 * (nz > 1 ? per : Tmax)), (size_t)(0), s, part, ctl, ring, ring_n, per, smp_tok, smp_val));
  CU_OK(cudaGetLastError());
  return 0;
}

// ---- prompt-lookup drafter (spec_draft, host/llb_host.c:1655-1676) --------------------------------
// The reference scans the token history on the host every cycle: the LATEST earlier position j whose last
// L = 3, 2, 1 tokens equal the history's last L, longest L first; the up-to-k tokens after j are the drafts.
// Here one block scans the device copy of the history right after the accept kernel, so the next cycle's
// rows are complete before its graph is launched.  Each thread keeps the latest match per L of its stride.
__global__ void __launch_bounds__(256) k_lookup_draft(SpecCtl *__restrict__ ctl) {
  pdl_trigger();
  pdl_wait();
  __shared__ int best[3];
  ctl += blockIdx.x;   // one block per stream
  const int *hist = ctl->hist;
  const int pos = __ldcg(&ctl->verify.pos0);   // (this block, the row count and the history's end: just written by k_accept)
  const int rows = __ldcg(&ctl->verify.n);
  if (!hist || rows < 1) return;
  if (threadIdx.x < 3) best[threadIdx.x] = -1;
  __syncthreads();
  const int t0 = __ldcg(hist + pos), t1 = pos >= 1 ? __ldcg(hist + pos - 1) : -1, t2 = pos >= 2 ? __ldcg(hist + pos - 2) : -1;
  int b1 = -1, b2 = -1, b3 = -1;
  for (int j = pos - 1 - (int)threadIdx.x; j >= 0; j -= blockDim.x) {
    if (__ldcg(hist + j) != t0) continue;
    if (b1 < 0) b1 = j;
    if (j >= 1 && pos >= 2 && __ldcg(hist + j - 1) == t1) {
      if (b2 < 0) b2 = j;
      if (j >= 2 && pos >= 3 && __ldcg(hist + j - 2) == t2) { if (b3 < 0) b3 = j; }
    }
    if (b3 >= 0) break;   // later iterations only see smaller j
  }
  if (b1 >= 0) atomicMax(&best[0], b1);
  if (b2 >= 0) atomicMax(&best[1], b2);
  if (b3 >= 0) atomicMax(&best[2], b3);
  __syncthreads();
  if (threadIdx.x != 0) return;
  const int j = best[2] >= 0 ? best[2] : best[1] >= 0 ? best[1] : best[0];
  int n = 0;
  if (j >= 0) {
    const int room = rows - 1;   // the accept kernel already clipped the rows to the context
    while (n < ctl->k && n < room && j + 1 + n <= pos) { ctl->verify.tok[1 + n] = __ldcg(hist + j + 1 + n); n++; }
  }
  ctl->verify.n = 1 + n;
}
int op_lookup_draft(cudaStream_t s, SpecCtl *ctl, int nz) {
  CU_OK(llb_launch(k_lookup_draft, dim3(nz), dim3(256), (size_t)(0), s, ctl));
  CU_OK(cudaGetLastError());
  return 0;
}

// After a drafter pass: the head argmax of its last row is draft j (mapped through the draft-vocab ids,
// host/llb_host.c:1800-1807); it becomes verify input j and the token of the next chained row, whose hidden
// is the drafter's own normed hidden of that last row (host/llb_host.c:1824-1827).
#define PICK_THREADS 512
__global__ void __launch_bounds__(PICK_THREADS) k_draft_pick(const float *__restrict__ part, const int *__restrict__ ids, SpecCtl *__restrict__ ctl,
                             int from_chain, int j, const float *__restrict__ mt_hn, float *__restrict__ chain_h, int d, int per) {
  pdl_trigger();
  pdl_wait();
  // one block per stream: its control block and its rows of the drafter pass; the chained row is the stream's row 0
  ctl += blockIdx.x;
  const size_t row0 = (size_t)blockIdx.x * per;
  part += row0 * TOP2_NB * 4; mt_hn += row0 * d; chain_h += row0 * d;
  const RowSet *rs = from_chain ? &ctl->chain : &ctl->catchup;
  const int last = __ldcg(&rs->n) - 1, p = __ldcg(&ctl->verify.pos0), n = __ldcg(&ctl->verify.n);
  // (every thread has read the row count before the first one writes it: in the drafter's later steps the chain is the row set)
  __syncthreads();
  if (last < 0) return;
  if (threadIdx.x >= 32) {   // the first warp picks while the others copy (d is a multiple of 32)
    const float4 *src = (const float4 *)(mt_hn + (size_t)last * d);
#pragma unroll 4
    for (int c = threadIdx.x - 32; c < d / 4; c += PICK_THREADS - 32) ((float4 *)chain_h)[c] = __ldcg(src + c);
    return;
  }
  const Top2 a = t2_final(part, last, threadIdx.x);
  if (threadIdx.x == 0) {
    const int tok = a.i1 < 0 ? 0 : ids ? ids[a.i1] : a.i1;
    if (j < n) ctl->verify.tok[j] = tok;
    ctl->chain.n = 1;
    ctl->chain.pos0 = p + j;
    ctl->chain.tok[0] = tok;
    ctl->chain.slot[0] = 0;
  }
}
int op_draft_pick(cudaStream_t s, const float *part, const int *ids, SpecCtl *ctl, int from_chain, int j, const float *mt_hn,
                  float *chain_h, int d, int nz, int per) {
  CU_OK(llb_launch(k_draft_pick, dim3(nz), dim3(PICK_THREADS), (size_t)(0), s, part, ids, ctl, from_chain, j, mt_hn, chain_h, d, per));
  CU_OK(cudaGetLastError());
  return 0;
}
