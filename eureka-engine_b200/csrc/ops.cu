// ops.cu -- format and activation-plane utility kernels.
#include <vector>

#include "host.cuh"

// ---- activations -> fp16 planes ----------------------------------------------------------------
// a thread takes four consecutive columns; a warp may be partly past the row's end (K is a multiple of 32)
__global__ void __launch_bounds__(256) k_xp_from_f32(const float *__restrict__ x, int K, int planes, XPlanes xp) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.y, c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < K) {
    const float *r = x + (size_t)t * K + c;
    if (!((uintptr_t)x & 15)) { const float4 f = __ldcg((const float4 *)r); v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w; }
    else for (int i = 0; i < 4; i++) v[i] = __ldcg(r + i);
  }
  xp_store4(xp, t, planes, c, v, threadIdx.x & 31, c < K);
}
__global__ void __launch_bounds__(256) k_xp_from_bf16(const unsigned short *__restrict__ x, int K, XPlanes xp) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.y, c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < K) {
    const unsigned short *r = x + (size_t)t * K + c;
    uint2 w;
    if (!((uintptr_t)x & 7)) w = __ldcg((const uint2 *)r);
    else w = make_uint2(__ldcg(r) | ((uint32_t)__ldcg(r + 1) << 16), __ldcg(r + 2) | ((uint32_t)__ldcg(r + 3) << 16));
    v[0] = __uint_as_float(w.x << 16); v[1] = __uint_as_float(w.x & 0xffff0000u); v[2] = __uint_as_float(w.y << 16); v[3] = __uint_as_float(w.y & 0xffff0000u);
  }
  xp_store4(xp, t, 1, c, v, threadIdx.x & 31, c < K);
}
int ops_xp_from_f32(cudaStream_t s, const float *x, int T, int planes, XPlanes xp) {
  if (xp.K % 32) return llb_fail("xp: K %d", xp.K);
  if (T * planes > xp.NC) return llb_fail("xp: %d rows x %d planes do not fit %d columns", T, planes, xp.NC);
  CU_OK(llb_launch(k_xp_from_f32, dim3((xp.K + 1023) / 1024, T), dim3(256), (size_t)(0), s, x, xp.K, planes, xp));
  CU_OK(cudaGetLastError());
  return 0;
}
int ops_xp_from_bf16(cudaStream_t s, const void *x, int T, XPlanes xp) {
  if (xp.K % 32) return llb_fail("xp: K %d", xp.K);
  if (T > xp.NC) return llb_fail("xp: %d rows do not fit %d columns", T, xp.NC);
  CU_OK(llb_launch(k_xp_from_bf16, dim3((xp.K + 1023) / 1024, T), dim3(256), (size_t)(0), s, (const unsigned short *)x, xp.K, xp));
  CU_OK(cudaGetLastError());
  return 0;
}

// ---- bit-exact row dequantisation (embedding rows; the dequant parity check) -------------------
__global__ void k_dequant_rows(int fmt, const uint8_t *__restrict__ W, int cols, const int *__restrict__ row_ids,
                               float *__restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.y;
  const int row = row_ids ? row_ids[r] : r;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x)
    out[(size_t)r * cols + c] = deq_elem(fmt, W, cols, row, c);
}
int ops_dequant_rows(cudaStream_t s, int fmt, const uint8_t *W, int rows, int cols, const int *row_ids, int nrows,
                     float *out) {
  (void)rows;
  if (nrows < 1) return 0;
  int gx = (cols + 255) / 256;
  if (gx > 64) gx = 64;
  // gridDim.y is limited to 65535 rows per launch; whole row tiles a launch, so that its first row starts one
  for (int r0 = 0; r0 < nrows; r0 += 65520) {
    int n = nrows - r0 < 65520 ? nrows - r0 : 65520;
    CU_OK(llb_launch(k_dequant_rows, dim3(gx, n), dim3(256), (size_t)(0), s, fmt, row_ids ? W : W + dev_bytes(fmt, r0, cols), cols,
                                              row_ids ? row_ids + r0 : nullptr, out + (size_t)r0 * cols));
    CU_OK(cudaGetLastError());
  }
  return 0;
}

// A GEMM's first weight copies do not wait for the kernel in front of it (programmatic launch), so weights that a kernel has
// just written need something between the two that is no kernel: what comes behind it starts when it is done.
static unsigned int *g_fence = nullptr;
int ops_setup(void) {
  if (!g_fence) CU_OK(cudaMalloc(&g_fence, 4));
  return 0;
}
static bool g_fence_held = false;
static int ops_fence(cudaStream_t s) {
  if (!g_fence_held) CU_OK(cudaMemsetAsync(g_fence, 0, 4, s));
  return 0;
}
// while a model is loaded: no launch reads weights before the last of them is uploaded, one fence behind all of them is enough
int ops_fence_hold(bool on) {
  g_fence_held = on;
  return on ? 0 : ops_fence(g_llb.stream);
}

// ---- pack rows -> device tiles (common.cuh) ------------------------------------------------------
// A block per tile; a thread moves two bytes at a time (a stored Q6_K block is only 2-byte aligned), or one where an address is
// odd.  Bytes past the stored row (columns that are not whole blocks) read as zero.  Runs once per matrix, at load.
template <typename U>
__global__ void __launch_bounds__(256) k_to_tiles(int fmt, const uint8_t *__restrict__ src, int rows, int cols, uint8_t *__restrict__ dst) {
  const int nsb = (cols + 255) >> 8, tb = tile_bytes(fmt), tr = tile_row(fmt), sz = sizeof(U);
  const size_t prb = pack_row_bytes(fmt, cols), blk = pack_row_bytes(fmt, 256);
  for (size_t tile = blockIdx.x; tile < (size_t)((rows + 15) >> 4) * nsb; tile += gridDim.x) {
    const int row0 = (int)(tile / nsb) * 16, sb = (int)(tile % nsb);
    for (int o = threadIdx.x * sz; o < tb; o += blockDim.x * sz) {
      int r = o / tr, b = o - r * tr;                      // row of the tile, byte of its block
      if (fmt == LLB_FM_Q6_K && o >= 3328) { r = (o - 3328) >> 1; b = 208 + (o & 1); }
      const bool codes = fmt == LLB_FM_Q8_0 && b < 256;
      size_t at = sb * blk + b;                            // byte of the stored row
      bool in = row0 + r < rows;
      if (fmt == LLB_FM_Q8_0) {
        at = codes ? (size_t)sb * 256 + b : (size_t)cols + sb * 16 + b - 256;
        in = in && (codes ? sb * 256 + b : sb * 256 + 16 * ((b - 256) & ~1)) < cols;
      }
      U v = 0;
      if (in && at + sz <= prb) v = *(const U *)(src + (size_t)(row0 + r) * prb + at);
      if (codes) v ^= (U)0x8080;
      *(U *)(dst + tile * tb + o) = v;
    }
  }
}
int ops_to_tiles(cudaStream_t s, int fmt, const uint8_t *src, int rows, int cols, uint8_t *dst) {
  const size_t n = (size_t)((rows + 15) >> 4) * ((cols + 255) >> 8);
  if (!n) return 0;
  const bool odd = (((uintptr_t)src | (uintptr_t)dst | pack_row_bytes(fmt, cols) | (fmt == LLB_FM_Q8_0 ? cols : 0)) & 1) != 0;
  const unsigned grid = (unsigned)(n < 16384 ? n : 16384);
  if (odd) k_to_tiles<uint8_t><<<grid, 256, 0, s>>>(fmt, src, rows, cols, dst);
  else k_to_tiles<unsigned short><<<grid, 256, 0, s>>>(fmt, src, rows, cols, dst);
  CU_OK(cudaGetLastError());
  return ops_fence(s);
}
// A range of rows and columns of one tiled matrix into another (a tensor-parallel rank's share): `n` rows from srow to
// drow, `nc` columns from scol to dcol, in blocks of 256 columns (Q8_0: 32).  Called at load only.
__global__ void __launch_bounds__(128) k_tile_slice(int fmt, const uint8_t *__restrict__ src, int scols, uint8_t *__restrict__ dst, int dcols, int srow, int drow,
                                                    int scol, int dcol, int nc) {
  const int tb = tile_bytes(fmt), tr = tile_row(fmt), unit = fmt == LLB_FM_Q8_0 ? 32 : 256;
  const int rs = srow + blockIdx.x, rd = drow + blockIdx.x;
  for (int u = 0; u < nc / unit; u++) {
    const int cs = scol + u * unit, cd = dcol + u * unit;
    const uint8_t *st = src + ((size_t)(rs >> 4) * ((scols + 255) >> 8) + (cs >> 8)) * tb;
    uint8_t *dt = dst + ((size_t)(rd >> 4) * ((dcols + 255) >> 8) + (cd >> 8)) * tb;
    const uint8_t *sr = st + (rs & 15) * tr;
    uint8_t *dr = dt + (rd & 15) * tr;
    if (fmt == LLB_FM_Q8_0) {
      const int is = cs & 255, id = cd & 255;
      if (threadIdx.x < 32) dr[id + threadIdx.x] = sr[is + threadIdx.x];
      else if (threadIdx.x < 34) dr[256 + 2 * (id >> 5) + threadIdx.x - 32] = sr[256 + 2 * (is >> 5) + threadIdx.x - 32];
    } else {
      for (int i = threadIdx.x; i < tr; i += blockDim.x) dr[i] = sr[i];
      if (fmt == LLB_FM_Q6_K && threadIdx.x < 2) dt[3328 + 2 * (rd & 15) + threadIdx.x] = st[3328 + 2 * (rs & 15) + threadIdx.x];
    }
  }
}
int ops_tile_slice(cudaStream_t s, int fmt, const uint8_t *src, int scols, uint8_t *dst, int dcols, int srow, int drow, int n, int scol, int dcol, int nc) {
  if (n < 1 || nc < 1) return 0;
  k_tile_slice<<<n, 128, 0, s>>>(fmt, src, scols, dst, dcols, srow, drow, scol, dcol, nc);
  CU_OK(cudaGetLastError());
  return ops_fence(s);
}

// ---- fixed-order sum of K-slice partials --------------------------------------------------------
// All slices of a value in one trip to L2 (NS of them; 0: any number, four a trip).  Loads to L2: the GEMM in front wrote the
// partial sums, and the buffer is used by one call after another.
template <int NS> __device__ __forceinline__ float sum_parts(const float *p, int nsplit, long long stride) {
  float v;
  if constexpr (NS > 0) {
    float l[NS];
#pragma unroll
    for (int k = 0; k < NS; k++) l[k] = __ldcg(p + k * stride);
    v = l[0];
#pragma unroll
    for (int k = 1; k < NS; k++) v += l[k];
  } else {
    v = __ldcg(p);
#pragma unroll 4
    for (int k = 1; k < nsplit; k++) v += __ldcg(p + k * stride);
  }
  return v;
}
__global__ void k_sum_parts(const float *__restrict__ parts, int nsplit, long long stride, int n, float *__restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = sum_parts<0>(parts + i, nsplit, stride);
}
template <int NS> __global__ void __launch_bounds__(256) k_sum_slices(const float *__restrict__ parts, long long stride, int n, float *__restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = sum_parts<NS>(parts + i, NS, stride);
}
// outputs of two to four matrices, one after the other in a slice: output m's first value is value at[m]
struct SumOut { float *p[GEMM_MAXMAT]; int at[GEMM_MAXMAT]; };
template <int NS> __global__ void __launch_bounds__(256) k_sum_slices_of(const float *__restrict__ parts, long long stride, int n, const SumOut o) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int m = 0;
#pragma unroll
  for (int k = 1; k < GEMM_MAXMAT; k++) if (i >= o.at[k]) m = k;
  o.p[m][i - o.at[m]] = sum_parts<NS>(parts + i, NS, stride);
}
int ops_sum_parts(cudaStream_t s, const float *parts, int nsplit, long long split_stride, int n, float *out) {
  const dim3 grid((n + 255) / 256);
  switch (nsplit) {
#define SUM_GO(NS) case NS: CU_OK(llb_launch(k_sum_slices<NS>, grid, dim3(256), (size_t)(0), s, parts, split_stride, n, out)); break;
    SUM_GO(2) SUM_GO(3) SUM_GO(4) SUM_GO(5) SUM_GO(6) SUM_GO(7) SUM_GO(8) SUM_GO(9) SUM_GO(10) SUM_GO(11) SUM_GO(12) SUM_GO(13) SUM_GO(14) SUM_GO(15) SUM_GO(16)
#undef SUM_GO
    default: CU_OK(llb_launch(k_sum_parts, grid, dim3(256), (size_t)(0), s, parts, nsplit, split_stride, n, out));
  }
  CU_OK(cudaGetLastError());
  return 0;
}
// ... of nmat outputs of n[i] values each, one after the other in a slice (2 <= nsplit <= GEMM_MAXSPLIT): a launch costs the host 1.4 us of a call's 10
int ops_sum_parts_of(cudaStream_t s, const float *parts, int nsplit, long long split_stride, int nmat, const int *n, float *const *out) {
  if (nmat == 1) return ops_sum_parts(s, parts, nsplit, split_stride, n[0], out[0]);
  SumOut o;
  int total = 0;
  for (int i = 0; i < GEMM_MAXMAT; i++) {
    o.p[i] = i < nmat ? out[i] : nullptr; o.at[i] = i < nmat ? total : 0x7fffffff;
    if (i < nmat) total += n[i];
  }
  const dim3 grid((total + 255) / 256);
  switch (nsplit) {
#define SUM_GO(NS) case NS: CU_OK(llb_launch(k_sum_slices_of<NS>, grid, dim3(256), (size_t)(0), s, parts, split_stride, total, o)); break;
    SUM_GO(2) SUM_GO(3) SUM_GO(4) SUM_GO(5) SUM_GO(6) SUM_GO(7) SUM_GO(8) SUM_GO(9) SUM_GO(10) SUM_GO(11) SUM_GO(12) SUM_GO(13) SUM_GO(14) SUM_GO(15) SUM_GO(16)
#undef SUM_GO
    default: return llb_fail("sum of %d slices", nsplit);
  }
  CU_OK(cudaGetLastError());
  return 0;
}

// ---- the launch half of the backend contract ----------------------------------------------------
// host/llb_backend.h:9-24 asks a backend for LLB_LAUNCH(k, gx, gy, bx, &a0, ...) / LLB_LAUNCH_SM: kernels are fetched
// by name (cuModuleGetFunction in the reference, tools/payload-spec.patch:9-23), every argument is the address of a
// host variable copied at the call, launches run in call order on one stream.  host/llb_backend_cuda.h:125-184 adds a
// recorder: between llb_graph_begin and llb_graph_end the launches are kept and then run as one CUDA graph, a repeated
// kernel sequence re-uses its graph, and any other device call ends the recording first ("bail").
//
// The kernels reachable by name are the library's own leaves with plain argument lists; the reference's kernel names
// (llb_spec_gu3, ...) are not among them: their argument lists carry its two-plane int8 activation format, so an
// unknown name returns NULL and the caller fails cleanly.
struct llb_b200_kernel { const char *name; const void *fn; int nparams; };
static const llb_b200_kernel g_kernels[] = {
    {"llb_b200_k_dequant_rows", (const void *)k_dequant_rows, 5},   // (int fmt, const u8 *W, int cols, const int *row_ids, float *out), grid (x, rows)
    {"llb_b200_k_sum_parts", (const void *)k_sum_parts, 5},         // (const float *parts, int nsplit, long long stride, int n, float *out)
    {"llb_b200_k_to_tiles", (const void *)k_to_tiles<uint8_t>, 5},  // (int fmt, const u8 *pack rows, int rows, int cols, u8 *device layout), any grid x
    {"llb_b200_k_xp_from_f32", (const void *)k_xp_from_f32, 4},     // (const float *x, int K, int planes, XPlanes xp), grid ((K + 1023) / 1024, T)
};

#define GRAPH_SLOTS 16      // cached kernel sequences (LLB_GSLOT of the reference)
#define GRAPH_MAXNODES 2048 // launches per recorded step (LLB_GMAX)
struct GraphSig { const void *fn; unsigned gx, gy, bx, sm; };
static bool g_rec = false;
static std::vector<GraphSig> g_rec_sig;
static struct { std::vector<const void *> fns; cudaGraphExec_t exec = nullptr; } g_slot[GRAPH_SLOTS];
static int g_victim = 0;
static unsigned long long g_gstat[4];   // graphs built, steps replayed, steps that re-used a cached graph, bails

// ends a recording by running what was recorded once, outside any cache
static int graph_flush(bool count_bail) {
  if (!g_rec) return 0;
  g_rec = false;
  cudaGraph_t g = nullptr;
  CU_OK(cudaStreamEndCapture(g_llb.stream, &g));
  if (count_bail) g_gstat[3] += 1;
  if (!g) return 0;
  cudaGraphExec_t ex = nullptr;
  cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
  if (e == cudaSuccess) e = cudaGraphLaunch(ex, g_llb.stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g_llb.stream);
  if (ex) cudaGraphExecDestroy(ex);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return llb_fail("graph recorder: %s", cudaGetErrorString(e));
  return 0;
}
int backend_graph_bail(void) { return graph_flush(true); }

extern "C" {
__attribute__((visibility("default"))) const llb_b200_kernel *llb_b200_kernel_by_name(const char *name) {
  if (name)
    for (const llb_b200_kernel &k : g_kernels)
      if (!strcmp(k.name, name)) return &k;
  llb_fail("kernel_by_name: the library has no kernel called %s", name ? name : "(null)");
  return nullptr;
}

__attribute__((visibility("default"))) int llb_b200_launch(const llb_b200_kernel *k, unsigned gx, unsigned gy, unsigned bx, unsigned sm, void **args, unsigned na) {
  if (!g_llb.stream) return llb_fail("llb_b200_init has not been called");
  if (!k) return llb_fail("launch: no kernel (an unknown name?)");
  if ((int)na != k->nparams) return llb_fail("launch: %s takes %d arguments, %u given", k->name, k->nparams, na);
  if (!gx || !gy || !bx || bx > 1024) return llb_fail("launch: %s with grid %u x %u, block %u", k->name, gx, gy, bx);
  if (g_rec) {
    if (g_rec_sig.size() >= GRAPH_MAXNODES) return llb_fail("graph recorder: more than %d launches in one step", GRAPH_MAXNODES);
    g_rec_sig.push_back({k->fn, gx, gy, bx, sm});
  }
  const cudaError_t e = cudaLaunchKernel(k->fn, dim3(gx, gy, 1), dim3(bx, 1, 1), args, sm, g_llb.stream);
  if (e != cudaSuccess) return llb_fail("launch of %s: %s", k->name, cudaGetErrorString(e));
  return k->fn == (const void *)k_to_tiles<uint8_t> ? ops_fence(g_llb.stream) : 0;
}

__attribute__((visibility("default"))) int llb_b200_graph_begin(void) {
  if (!g_llb.stream) return llb_fail("llb_b200_init has not been called");
  if (g_rec) return 0;
  CU_OK(cudaStreamBeginCapture(g_llb.stream, cudaStreamCaptureModeThreadLocal));
  g_rec = true;
  g_rec_sig.clear();
  return 0;
}

__attribute__((visibility("default"))) int llb_b200_graph_end(void) {
  if (!g_rec) return 0;
  g_rec = false;
  cudaGraph_t g = nullptr;
  CU_OK(cudaStreamEndCapture(g_llb.stream, &g));
  if (!g || g_rec_sig.empty()) { if (g) cudaGraphDestroy(g); return 0; }
  // a step with the kernel sequence of a cached graph only updates that graph's nodes
  int sl = -1;
  for (int i = 0; i < GRAPH_SLOTS && sl < 0; i++) {
    if (!g_slot[i].exec || g_slot[i].fns.size() != g_rec_sig.size()) continue;
    bool same = true;
    for (size_t j = 0; same && j < g_rec_sig.size(); j++) same = g_slot[i].fns[j] == g_rec_sig[j].fn;
    if (same) sl = i;
  }
  cudaError_t e = cudaSuccess;
  if (sl >= 0) {
    cudaGraphExecUpdateResultInfo info;
    if (cudaGraphExecUpdate(g_slot[sl].exec, g, &info) == cudaSuccess) g_gstat[2] += 1;
    else { cudaGetLastError(); cudaGraphExecDestroy(g_slot[sl].exec); g_slot[sl].exec = nullptr; sl = -1; }
  }
  if (sl < 0) {
    sl = g_victim; g_victim = (g_victim + 1) % GRAPH_SLOTS;
    if (g_slot[sl].exec) cudaGraphExecDestroy(g_slot[sl].exec);
    g_slot[sl].exec = nullptr;
    e = cudaGraphInstantiate(&g_slot[sl].exec, g, 0);
    g_slot[sl].fns.clear();
    for (const GraphSig &q : g_rec_sig) g_slot[sl].fns.push_back(q.fn);
    g_gstat[0] += 1;
  }
  cudaGraphDestroy(g);
  if (e == cudaSuccess) e = cudaGraphLaunch(g_slot[sl].exec, g_llb.stream);
  if (e != cudaSuccess) return llb_fail("graph recorder: %s", cudaGetErrorString(e));
  g_gstat[1] += 1;
  return 0;
}

__attribute__((visibility("default"))) int llb_b200_graph_bail(void) { return backend_graph_bail(); }
__attribute__((visibility("default"))) void llb_b200_graph_stats(unsigned long long out[4]) { for (int i = 0; i < 4; i++) out[i] = g_gstat[i]; }
}  // extern "C"
