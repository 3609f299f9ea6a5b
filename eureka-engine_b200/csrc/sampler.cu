// sampler.cu -- sampling-mode verify on the device: for every row of a verify pass, the token the reference's sampler
// pack would emit from that row's logits -- llb_smp_verify for a row that has a draft (accept with probability
// min(1, p / q), q one-hot because both drafters are deterministic; on a reject a draw from the residual
// max(0, p - q)), llb_smp_sample for the row that has none (host/llb_sampler_impl.h:384-444).  The reference reads V
// logits back per served row and decides on the host (smp_pick, host/llb_host.c:1407-1470); here the rows of a pass
// are decided by one kernel inside the cycle's graph and k_accept takes the emitted tokens from it instead of the
// argmax, so a sampled cycle is still one graph launch and one result record.
//
// The chain (host/llb_sampler_impl.h:322-358): logit bias -> repeat / frequency / presence penalties over the last
// repeat_last_n tokens -> top_k -> top_p -> min_p -> temperature -> probabilities expf(l - max) with their sum in
// double.  The reference keeps llama.cpp's float arithmetic on purpose; where the order of float operations decides
// a result (the float running sums of top_p, the penalty expression) one thread does them in the reference's order
// with no fused multiply-add.  exp is taken in double and rounded (the host's expf is within half an ulp of that).
//   top_k in 1..256, and argmax (temp <= 0: the list of one): the k largest under the order "logit descending, id
//     ascending" (the reference's partial selection, ties to the earlier candidate) in two launches -- k_smp_cand keeps
//     the k largest of every 2048 ids, k_smp_pick the k largest of what is left --, then the short sorted list goes
//     through top_p, min_p, temperature and the draw in the reference's own arithmetic, operation for operation: what is
//     independent per entry (exp, divisions) a thread each, the running sums by one thread in order.
//   top_k off: the whole vocabulary in id order; min_p is a mask, the probabilities' sum and the walk's running sums
//     are block-wide reductions and scans in double (they differ from the sequential double sums in the last bits only).
//   top_p without top_k needs the reference's float sum over the whole vocabulary in id order and is refused by
//     llb_spec_set_sampler, as are top_k > 256 and a penalty window longer than 256.
// Random numbers: the reference's counter RNG, splitmix64 of (seed, 4 pos + k + 1) (host/llb_sampler_impl.h:142-155):
// draw 1 decides accept, draw 2 the residual, draw 0 a plain sample; pos = the position the token will occupy.
#include "model.cuh"
#include "sampler.cuh"

#define SMP_THREADS 1024

__device__ __forceinline__ double smp_draw(unsigned long long seed, unsigned long long pos, unsigned int k) {
  unsigned long long z = seed ^ 0x6A09E667F3BCC909ull;
  z += (pos * 4ull + k + 1ull) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}
__device__ __forceinline__ float smp_expf(float x) { return (float)exp((double)x); }
// a comes before b: logit descending, then id ascending
__device__ __forceinline__ bool smp_before(float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); }

struct SmpShared {
  int win[SMP_MAX_WIN];
  float rv[32];
  int ri[32];
  double rd[32];
  float bv;
  int bi;
  double bd;
  int hit_lo, hit_hi;
};

// block-wide best (v, i) under smp_before; every thread gets it.  i < 0: no candidate.
__device__ __forceinline__ void smp_block_best(float &v, int &i, SmpShared &sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, m);
    const int oi = __shfl_xor_sync(0xffffffffu, i, m);
    if (oi >= 0 && (i < 0 || smp_before(ov, oi, v, i))) { v = ov; i = oi; }
  }
  __syncthreads();
  if (lane == 0) { sh.rv[w] = v; sh.ri[w] = i; }
  __syncthreads();
  if (w == 0) {
    v = sh.rv[lane]; i = sh.ri[lane];
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, m);
      const int oi = __shfl_xor_sync(0xffffffffu, i, m);
      if (oi >= 0 && (i < 0 || smp_before(ov, oi, v, i))) { v = ov; i = oi; }
    }
    if (lane == 0) { sh.bv = v; sh.bi = i; }
  }
  __syncthreads();
  v = sh.bv; i = sh.bi;
}
// block-wide sum in double; every thread gets it
__device__ __forceinline__ double smp_block_sum(double x, SmpShared &sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
  __syncthreads();
  if (lane == 0) sh.rd[w] = x;
  __syncthreads();
  if (w == 0) {
    x = sh.rd[lane];
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) x += __shfl_xor_sync(0xffffffffu, x, m);
    if (lane == 0) sh.bd = x;
  }
  __syncthreads();
  return sh.bd;
}
// exclusive prefix over the threads of the block (thread order), in double
__device__ __forceinline__ double smp_block_excl(double x, SmpShared &sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double inc = x;
#pragma unroll
  for (int m = 1; m < 32; m <<= 1) { const double o = __shfl_up_sync(0xffffffffu, inc, m); if (lane >= m) inc += o; }
  __syncthreads();
  if (lane == 31) sh.rd[w] = inc;
  __syncthreads();
  if (w == 0) {
    double t = sh.rd[lane], ti = t;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) { const double o = __shfl_up_sync(0xffffffffu, ti, m); if (lane >= m) ti += o; }
    sh.rd[lane] = ti - t;
  }
  __syncthreads();
  return sh.rd[w] + inc - x;
}

// The walk over the whole vocabulary in id order: the first id whose running sum of val(i) reaches tgt, else the last id
// with val > 0.  Every thread owns a run of consecutive ids.
template <class F> __device__ __forceinline__ int smp_walk_all(int V, double tgt, F val, SmpShared &sh) {
  const int per = (V + SMP_THREADS - 1) / SMP_THREADS, i0 = threadIdx.x * per, i1 = min(V, i0 + per);
  double mine = 0.0;
  int last = -1;
  for (int i = i0; i < i1; i++) { const float p = val(i); if (p > 0.0f) { mine += (double)p; last = i; } }
  const double before = smp_block_excl(mine, sh);
  if (threadIdx.x == 0) { sh.hit_lo = 0x7fffffff; sh.hit_hi = -1; }
  __syncthreads();
  if (last >= 0) atomicMax(&sh.hit_hi, last);
  if (mine > 0.0 && before + mine >= tgt) {
    double run = before;
    for (int i = i0; i < i1; i++) {
      const float p = val(i);
      if (p <= 0.0f) continue;
      run += (double)p;
      if (run >= tgt) { atomicMin(&sh.hit_lo, i); break; }
    }
  }
  __syncthreads();
  return sh.hit_lo != 0x7fffffff ? sh.hit_lo : sh.hit_hi;
}

// What a row's decision starts from.  Engine mode (ctl != null): the row's stream, position, draft and penalty window come
// from the control block; test mode: from the explicit arrays.  The window's tokens go to win (every thread of the block takes
// part; the caller synchronises).  False: the row is not in use.
struct SmpTest { const int *draft; const long long *pos; const int *win, *nwin; };
__device__ __forceinline__ bool smp_row_in(const SmpDev &P, const SpecCtl *ctl, Streams sg, const SmpTest &ts, int t, int *win, int &draft, int &nwin, unsigned long long &pos) {
  nwin = 0;
  if (ctl) {
    const int z = t / sg.per, tl = t - z * sg.per;
    const SpecCtl *c = (const SpecCtl *)((const char *)ctl + (size_t)z * sg.stride);
    const RowSet &rs = c->verify;
    const int n = __ldcg(&rs.n), pos0 = __ldcg(&rs.pos0);   // (to L2: earlier kernels of this cycle wrote the drafts)
    if (tl >= n) return false;
    const int prow = pos0 + tl;
    pos = (unsigned long long)prow + 1ull;   // the position the emitted token will occupy
    draft = tl + 1 < n ? __ldcg(&rs.tok[tl + 1]) : -1;
    if (P.pen_on && win) {
      // the tokens at positions prow + 1 - N .. prow: history up to the pass's first row, then the pass's own inputs
      const int N = P.repeat_last_n, q0 = prow + 1 - N > 0 ? prow + 1 - N : 0;
      nwin = prow + 1 - q0;
      for (int a = threadIdx.x; a < nwin; a += blockDim.x) { const int q = q0 + a; win[a] = q >= pos0 ? __ldcg(&rs.tok[q - pos0]) : c->hist ? __ldcg(c->hist + q) : -1; }
    }
  } else {
    draft = ts.draft[t]; pos = (unsigned long long)ts.pos[t];
    if (P.pen_on && win) { nwin = ts.nwin[t]; for (int a = threadIdx.x; a < nwin; a += blockDim.x) win[a] = ts.win[(size_t)t * SMP_MAX_WIN + a]; }
  }
  return true;
}
// Whether place a of the window is its token's first; cnt: the token's occurrences in it
__device__ __forceinline__ bool smp_first_of(const int *win, int nwin, int a, int &cnt) {
  const int tk = win[a];
  bool first = true;
  cnt = 0;
  for (int b = 0; b < nwin; b++) { if (win[b] == tk) { cnt++; if (b < a) first = false; } }
  return first;
}
__device__ __forceinline__ float smp_penalise(const SmpDev &P, float x, int cnt) {
  x = x <= 0.0f ? __fmul_rn(x, P.repeat_penalty) : __fdiv_rn(x, P.repeat_penalty);
  return __fsub_rn(x, __fadd_rn(__fmul_rn((float)cnt, P.frequency), P.presence));
}

// ---- the k largest ------------------------------------------------------------------------------------------------
// A candidate as one word that sorts as smp_before does: the logit's bits made monotonic, then the complement of the id.
// 0 is no candidate (and what a NaN becomes: it is never drawn); -0 sorts as +0.
__device__ __forceinline__ unsigned long long smp_key(float v, int id) {
  if (v != v) return 0ull;
  const unsigned int u = __float_as_uint(v + 0.0f);
  return (unsigned long long)((u & 0x80000000u) ? ~u : u | 0x80000000u) << 32 | (0xffffffffu - (unsigned int)id);
}
__device__ __forceinline__ float smp_key_val(unsigned long long k) {
  const unsigned int u = (unsigned int)(k >> 32);
  return __uint_as_float((u & 0x80000000u) ? u & 0x7fffffffu : ~u);
}
__device__ __forceinline__ int smp_key_id(unsigned long long k) { return (int)(0xffffffffu - (unsigned int)k); }
// block-wide sum of c, every thread gets it; one barrier a call (part: two rows that take turns)
__device__ __forceinline__ int smp_count(int c, unsigned int (*part)[32], int &ph) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0) part[ph][w] = (unsigned int)c;
  __syncthreads();
  c = __reduce_add_sync(0xffffffffu, lane < nw ? (int)part[ph][lane] : 0);
  ph ^= 1;
  return c;
}
// The word that exactly K keys of the block reach (K of them at least are not 0; no two that are not 0 are equal): its upper half
// bit by bit, which ends as soon as the count fits, and where equal logits straddle the line the lower half among those.
template <int N> __device__ __forceinline__ unsigned long long smp_kth(const unsigned long long (&key)[N], int K, unsigned int (*part)[32], int &ph) {
  unsigned int hi = 0, lo = 0;
#pragma unroll 1
  for (int bit = 31; bit >= 0; bit--) {
    const unsigned int c = hi | (1u << bit);
    int n = 0;
#pragma unroll
    for (int j = 0; j < N; j++) n += (unsigned int)(key[j] >> 32) >= c;
    n = smp_count(n, part, ph);
    if (n >= K) { hi = c; if (n == K) return (unsigned long long)hi << 32; }
  }
  int gt = 0;
#pragma unroll
  for (int j = 0; j < N; j++) gt += (unsigned int)(key[j] >> 32) > hi;
  const int need = K - smp_count(gt, part, ph);
#pragma unroll 1
  for (int bit = 31; bit >= 0; bit--) {
    const unsigned int c = lo | (1u << bit);
    int n = 0;
#pragma unroll
    for (int j = 0; j < N; j++) n += (unsigned int)(key[j] >> 32) == hi && (unsigned int)key[j] >= c;
    if (smp_count(n, part, ph) >= need) lo = c;
  }
  return (unsigned long long)hi << 32 | lo;
}

// Block (chunk, row): biases and penalties on VPT x 256 consecutive ids, and the K largest of them, in any order, into
// cand[row][chunk][K] (zeros behind the last).  One block a row, with the K picks as K rounds of a block-wide argmax over the
// whole vocabulary, took 765 us for two rows of 151936 logits and top_k 40, a quarter of a cycle of the 9B shape; the two launches
// take about 30.
#define SMP_CAND_THREADS 256
template <int VPT>
__global__ void __launch_bounds__(SMP_CAND_THREADS) k_smp_cand(SmpDev P, PartIn lg, int V, int K, unsigned long long *__restrict__ cand, size_t cand_row,
                                                                const SpecCtl *__restrict__ ctl, Streams sg, SmpTest ts) {
  constexpr int CHUNK = VPT * SMP_CAND_THREADS;
  __shared__ float val[CHUNK];
  __shared__ int win[SMP_MAX_WIN];
  __shared__ unsigned int part[2][32];
  __shared__ int fill;
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.y, tid = threadIdx.x, i0 = blockIdx.x * CHUNK, n = min(CHUNK, V - i0);
  int draft, nwin, ph = 0;
  unsigned long long pos;
  if (!smp_row_in(P, ctl, sg, ts, t, win, draft, nwin, pos)) return;
  const size_t l0 = (size_t)t * V + i0;
#pragma unroll
  for (int j = 0; j < VPT; j++) { const int i = tid + j * SMP_CAND_THREADS; if (i < n) val[i] = part_get(lg, l0 + i); }
  if (tid == 0) fill = 0;
  __syncthreads();
  if (P.n_bias) {
    if (tid < P.n_bias) {                              // several biases of one id are added in their order, by the first of them
      const int id = P.bias_ids[tid];
      bool first = id >= i0 && id < i0 + n;
      for (int j = 0; j < tid && first; j++) first = P.bias_ids[j] != id;
      if (first) for (int j = tid; j < P.n_bias; j++) if (P.bias_ids[j] == id) val[id - i0] = __fadd_rn(val[id - i0], P.bias_vals[j]);
    }
    __syncthreads();
  }
  if (nwin > 0) {
    if (tid < nwin) {
      const int id = win[tid];
      int cnt;
      if (id >= i0 && id < i0 + n && smp_first_of(win, nwin, tid, cnt)) val[id - i0] = smp_penalise(P, val[id - i0], cnt);
    }
    __syncthreads();
  }
  unsigned long long key[VPT];
  int valid = 0;
#pragma unroll
  for (int j = 0; j < VPT; j++) { const int i = tid + j * SMP_CAND_THREADS; key[j] = i < n ? smp_key(val[i], i0 + i) : 0ull; valid += key[j] != 0; }
  valid = smp_count(valid, part, ph);
  const unsigned long long least = valid > K ? smp_kth(key, K, part, ph) : 1ull;
  unsigned long long *out = cand + (size_t)t * cand_row + (size_t)blockIdx.x * K;
#pragma unroll
  for (int j = 0; j < VPT; j++) if (key[j] >= least) out[atomicAdd(&fill, 1)] = key[j];
  for (int i = tid; i < K; i += SMP_CAND_THREADS) if (i >= valid) out[i] = 0ull;
}

// One block a row: the K largest of the nc candidates, sorted, then the list's stages and the draw.
#define SMP_PICK_VPT 16     // candidates a thread holds at a time: 16384 of them, all there are up to V = 524288 at K = 256
__global__ void __launch_bounds__(SMP_THREADS) k_smp_pick(SmpDev P, PartIn lg, int V, int K, const unsigned long long *__restrict__ cand, size_t cand_row, int nc,
                                                           const SpecCtl *__restrict__ ctl, Streams sg, SmpTest ts, int *__restrict__ tok_out,
                                                           float *__restrict__ val_out, int *__restrict__ acc_out, unsigned int *__restrict__ err) {
  __shared__ unsigned long long sel[SMP_MAX_TOPK];
  __shared__ float l[SMP_MAX_TOPK], p[SMP_MAX_TOPK], e[SMP_MAX_TOPK];
  __shared__ double r[SMP_MAX_TOPK];
  __shared__ int id[SMP_MAX_TOPK];
  __shared__ unsigned int part[2][32];
  __shared__ int fill, s_n, s_go;
  __shared__ float s_sum;
  __shared__ double s_dsum;
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, tid = threadIdx.x;
  int draft, nwin, ph = 0, have = 0;
  unsigned long long pos;
  if (!smp_row_in(P, ctl, sg, ts, t, nullptr, draft, nwin, pos)) return;
  const unsigned long long *c = cand + (size_t)t * cand_row;
  // batches of candidates, each together with the best so far (one batch in all but extreme vocabularies)
#pragma unroll 1
  for (int base = 0; base < nc; base += SMP_PICK_VPT * SMP_THREADS) {
    unsigned long long key[SMP_PICK_VPT + 1];
    int valid = 0;
#pragma unroll
    for (int j = 0; j < SMP_PICK_VPT; j++) { const int i = base + tid + j * SMP_THREADS; key[j] = i < nc ? __ldcg(c + i) : 0ull; valid += key[j] != 0; }
    key[SMP_PICK_VPT] = tid < have ? sel[tid] : 0ull;
    valid = smp_count(valid + (tid < have), part, ph);
    const unsigned long long least = valid > K ? smp_kth(key, K, part, ph) : 1ull;
    if (tid == 0) fill = 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j <= SMP_PICK_VPT; j++) if (key[j] >= least) sel[atomicAdd(&fill, 1)] = key[j];
    __syncthreads();
    have = valid > K ? K : valid;
  }
  if (have == 0) {   // nothing but NaN in the row
    if (tid == 0) { tok_out[t] = 0; val_out[t] = part_get(lg, (size_t)t * V); if (acc_out) acc_out[t] = 0; atomicExch(err, 3u); }
    return;
  }
  if (tid < have) {
    const unsigned long long k = sel[tid];
    int rank = 0;
    for (int i = 0; i < have; i++) rank += sel[i] > k;
    l[rank] = smp_key_val(k); id[rank] = smp_key_id(k);
  }
  __syncthreads();
  int tok = id[0], accepted = 0, n = have;
  if (P.temp <= 0.0f) accepted = draft >= 0 && tok == draft;
  else {
    if (P.top_p < 1.0f) {                                  // llama's top_p over a sorted list: float softmax, float running sum
      if (tid < n) e[tid] = smp_expf(__fsub_rn(l[tid], l[0]));
      __syncthreads();
      if (tid == 0) { float sum = 0.0f; for (int i = 0; i < n; i++) sum = __fadd_rn(sum, e[i]); s_sum = sum; }
      __syncthreads();
      if (tid < n) e[tid] = __fdiv_rn(e[tid], s_sum);
      __syncthreads();
      if (tid == 0) {
        float cum = 0.0f;
        int last = n;
        for (int i = 0; i < n; i++) {
          cum = __fadd_rn(cum, e[i]);
          if (cum >= P.top_p && i + 1 >= P.min_keep) { last = i + 1; break; }
        }
        s_n = last;
      }
      __syncthreads();
      n = s_n;
    }
    if (P.min_p > 0.0f && n > 0) {                          // sorted min_p
      const float floor_l = __fadd_rn(l[0], P.log_min_p);
      int i = 1;
      for (; i < n; i++) if (l[i] < floor_l && i >= P.min_keep) break;
      n = i;
    }
    const float mx = P.temp != 1.0f ? __fdiv_rn(l[0], P.temp) : l[0];
    if (tid < n) p[tid] = smp_expf(__fsub_rn(P.temp != 1.0f ? __fdiv_rn(l[tid], P.temp) : l[tid], mx));
    __syncthreads();
    if (tid == 0) {
      double sum = 0.0, pd = 0.0;
      for (int i = 0; i < n; i++) sum += (double)p[i];
      int sel_i = -1;
      s_go = 0;
      if (draft < 0) {                                      // a plain draw: walk the unnormalised p against sum * u
        if (n == 1) sel_i = 0;
        else {
          const double tgt = sum * smp_draw(P.seed, pos, 0);
          double run = 0.0;
          for (int i = 0; i < n && sel_i < 0; i++) { run += (double)p[i]; if (run >= tgt) sel_i = i; }
          if (sel_i < 0) sel_i = n - 1;
        }
      } else {
        for (int i = 0; i < n; i++) if (id[i] == draft) pd = (double)p[i] / sum;
        s_go = !(smp_draw(P.seed, pos, 1) < pd);
      }
      s_dsum = sum; s_n = sel_i;
    }
    __syncthreads();
    if (draft < 0) tok = id[s_n];
    else if (!s_go) { tok = draft; accepted = 1; }
    else {                                                  // the residual max(0, p - q)
      if (tid < n) {
        const double pi = (double)p[tid] / s_dsum, qi = id[tid] == draft ? 1.0 : 0.0;
        r[tid] = pi > qi ? pi - qi : 0.0;
      }
      __syncthreads();
      if (tid == 0) {
        double rs = 0.0;
        for (int i = 0; i < n; i++) rs += r[i];
        const bool same = !(rs > 0.0);                      // p == q exactly: the reference falls back to a draw from p
        const double tgt = (same ? s_dsum : rs) * smp_draw(P.seed, pos, 2);
        double run = 0.0;
        int at = -1, last = same ? n - 1 : -1;
        for (int i = 0; i < n && at < 0; i++) {
          const float w = same ? p[i] : (float)r[i];
          if (!same) { if (w <= 0.0f) continue; last = i; }
          run += (double)w;
          if (run >= tgt) at = i;
        }
        s_n = at < 0 ? last : at;
      }
      __syncthreads();
      tok = s_n < 0 ? -1 : id[s_n];
    }
  }
  if (tid == 0) {
    if (tok < 0 || tok >= V) { tok = id[0]; atomicExch(err, 3u); }
    tok_out[t] = tok;
    val_out[t] = part_get(lg, (size_t)t * V + tok);   // the raw logit of the emitted token (host/llb_host.c:1455-1456)
    if (acc_out) acc_out[t] = accepted;
  }
}

// The whole vocabulary (top_k off): one block per row of the pass.
__global__ void __launch_bounds__(SMP_THREADS) k_smp_rows(SmpDev P, PartIn lg, int V, float *__restrict__ adj, const SpecCtl *__restrict__ ctl, Streams sg,
                                                           SmpTest ts, int *__restrict__ tok_out, float *__restrict__ val_out,
                                                           int *__restrict__ acc_out, unsigned int *__restrict__ err) {
  __shared__ SmpShared sh;
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, tid = threadIdx.x;
  int draft, nwin;
  unsigned long long pos;
  if (!smp_row_in(P, ctl, sg, ts, t, sh.win, draft, nwin, pos)) return;
  float *row = adj + (size_t)t * V;
  const size_t l0 = (size_t)t * V;
  // ---- bias, then penalties -------------------------------------------------------------------------------------
  for (int i = tid; i < V; i += SMP_THREADS) {
    float v = part_get(lg, l0 + i);
    for (int j = 0; j < P.n_bias; j++) if (P.bias_ids[j] == i) v = __fadd_rn(v, P.bias_vals[j]);
    row[i] = v;
  }
  __syncthreads();
  if (tid < nwin) {
    const int tk = sh.win[tid];
    int cnt;
    if (tk >= 0 && tk < V && smp_first_of(sh.win, nwin, tid, cnt)) row[tk] = smp_penalise(P, row[tk], cnt);
  }
  __syncthreads();
  int tok = 0, accepted = 0;
  // ---- the block-wide first maximum ------------------------------------------------------------------------------
  float bv = -INFINITY;
  int bi = -1;
  for (int i = tid; i < V; i += SMP_THREADS) { const float v = row[i]; if (bi < 0 || v > bv) { bv = v; bi = i; } }
  smp_block_best(bv, bi, sh);
  const float top_v = bv;
  const int top_i = bi;
  {
    // ---- the whole vocabulary in id order: min_p as a mask, sums and walks as block-wide reductions ----------------
    const float floor_l = P.min_p > 0.0f ? __fadd_rn(top_v, P.log_min_p) : -INFINITY;
    const float T = P.temp, mx = T != 1.0f ? __fdiv_rn(top_v, T) : top_v;
    auto e_of = [&](int i) -> float {
      const float v = row[i];
      if (!(v >= floor_l)) return 0.0f;
      return smp_expf(__fsub_rn(T != 1.0f ? __fdiv_rn(v, T) : v, mx));
    };
    double part = 0.0;
    int kept = 0;
    {
      const int per = (V + SMP_THREADS - 1) / SMP_THREADS, i0 = tid * per, i1 = min(V, i0 + per);
      for (int i = i0; i < i1; i++) { const float e = e_of(i); part += (double)e; kept += row[i] >= floor_l; }
    }
    const double sum = smp_block_sum(part, sh);
    if (P.min_p > 0.0f && P.min_keep > 1) {
      const int w = (int)(smp_block_sum((double)kept, sh) + 0.5);
      if (w < P.min_keep && tid == 0) atomicExch(err, 2u);   // the reference sorts and keeps min_keep here: not built
    }
    if (draft < 0) {
      tok = smp_walk_all(V, sum * smp_draw(P.seed, pos, 0), e_of, sh);
    } else {
      const double pd = (draft >= 0 && draft < V) ? (double)e_of(draft) / sum : 0.0;
      if (smp_draw(P.seed, pos, 1) < pd) { tok = draft; accepted = 1; }
      else {
        auto r_of = [&](int i) -> float {
          if (i == draft) return 0.0f;                        // max(0, p - 1)
          return (float)((double)e_of(i) / sum);
        };
        double rpart = 0.0;
        {
          const int per = (V + SMP_THREADS - 1) / SMP_THREADS, i0 = tid * per, i1 = min(V, i0 + per);
          for (int i = i0; i < i1; i++) if (i != draft) rpart += (double)e_of(i) / sum;
        }
        const double rs = smp_block_sum(rpart, sh);
        const double u2 = smp_draw(P.seed, pos, 2);
        if (!(rs > 0.0)) tok = smp_walk_all(V, sum * u2, e_of, sh);
        else tok = smp_walk_all(V, rs * u2, r_of, sh);
      }
    }
  }
  if (tid == 0) {
    if (tok < 0 || tok >= V) { tok = top_i; atomicExch(err, 3u); }
    tok_out[t] = tok;
    val_out[t] = part_get(lg, l0 + tok);   // the raw logit of the emitted token (host/llb_host.c:1455-1456)
    if (acc_out) acc_out[t] = accepted;
  }
}

// Ids a block of k_smp_cand takes: 2048, and four times that where the candidates of a row would fill more than half of
// what k_smp_pick holds at a time
static int smp_chunk(int V, int K) { return (long long)((V + 2047) / 2048) * K > SMP_PICK_VPT * SMP_THREADS / 2 ? 8192 : 2048; }
static int smp_list(const SmpDev &P, int V) { const int k = P.temp <= 0.0f ? 1 : P.top_k; return k < V ? k : V; }   // 0: the whole vocabulary
// floats of scratch a row needs, whatever the parameters: the adjusted logits, or K = 256 candidates of eight bytes a chunk
size_t smp_row_floats(int V) {
  const size_t a = (size_t)V, b = (size_t)((V + 2047) / 2048) * SMP_MAX_TOPK * 2;
  return ((a > b ? a : b) + 1) & ~(size_t)1;
}
int op_smp_rows(cudaStream_t s, const SmpDev &P, PartIn lg, int V, float *adj, const SpecCtl *ctl, int rows, const int *t_draft, const long long *t_pos,
                const int *t_win, const int *t_nwin, int *tok_out, float *val_out, int *acc_out, unsigned int *err) {
  const int K = smp_list(P, V);
  const SmpTest ts{t_draft, t_pos, t_win, t_nwin};
  if (K <= 0) {
    CU_OK(llb_launch(k_smp_rows, dim3(rows), dim3(SMP_THREADS), (size_t)0, s, P, lg, V, adj, ctl, ops_streams(), ts, tok_out, val_out, acc_out, err));
    return 0;
  }
  const int chunk = smp_chunk(V, K), nb = (V + chunk - 1) / chunk;
  unsigned long long *cand = (unsigned long long *)adj;
  const size_t cand_row = smp_row_floats(V) / 2;
  CU_OK(llb_launch(chunk == 2048 ? k_smp_cand<8> : k_smp_cand<32>, dim3(nb, rows), dim3(SMP_CAND_THREADS), (size_t)0, s, P, lg, V, K, cand, cand_row, ctl, ops_streams(), ts));
  CU_OK(llb_launch(k_smp_pick, dim3(rows), dim3(SMP_THREADS), (size_t)0, s, P, lg, V, K, (const unsigned long long *)cand, cand_row, nb * K, ctl, ops_streams(), ts, tok_out,
                   val_out, acc_out, err));
  return 0;
}

// host side: the parameters as the kernel takes them; -1 (and a message) for what has no device path
int smp_prepare(const llb_smp_params *p, SmpDev *d, bool *argmax_only) {
  memset(d, 0, sizeof *d);
  if (p->n_bias < 0 || p->n_bias > SMP_MAX_BIAS) return llb_fail("sampler: %d logit biases (at most %d)", p->n_bias, SMP_MAX_BIAS);
  const bool pen_on = !(p->repeat_last_n <= 0 || (p->repeat_penalty == 1.0f && p->frequency == 0.0f && p->presence == 0.0f));
  *argmax_only = p->temp <= 0.0f && p->n_bias == 0 && !pen_on;   // llb_smp_is_argmax (host/llb_sampler_impl.h:81-83)
  if (pen_on && p->repeat_last_n > SMP_MAX_WIN) return llb_fail("sampler: a penalty window of %d tokens (at most %d)", p->repeat_last_n, SMP_MAX_WIN);
  if (p->temp > 0.0f) {
    if (p->top_k > SMP_MAX_TOPK) return llb_fail("sampler: top_k %d (at most %d on the device)", p->top_k, SMP_MAX_TOPK);
    if (p->top_p < 1.0f && p->top_k <= 0) return llb_fail("sampler: top_p < 1 needs top_k in 1..%d (the reference's float sum over the whole vocabulary in id order has no device path)", SMP_MAX_TOPK);
  }
  d->temp = p->temp; d->top_p = p->top_p; d->min_p = p->min_p; d->top_k = p->top_k; d->repeat_penalty = p->repeat_penalty;
  d->repeat_last_n = p->repeat_last_n; d->presence = p->presence; d->frequency = p->frequency; d->seed = p->seed; d->min_keep = p->min_keep;
  d->pen_on = pen_on ? 1 : 0;
  d->log_min_p = p->min_p > 0.0f ? logf(p->min_p) : 0.0f;   // the host's logf, as the reference takes it
  d->n_bias = p->n_bias;
  for (int j = 0; j < p->n_bias; j++) { d->bias_ids[j] = p->bias_ids[j]; d->bias_vals[j] = p->bias_vals[j]; }
  return 0;
}
