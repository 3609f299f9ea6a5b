// rowops.cuh -- device helpers of the row-wise and attention kernels (ops_model.cu, attention.cu).
#pragma once
#include "model.cuh"

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, m));
  return v;
}

// ---- top k of a routed-expert layer's router (host/llb_host.c:651-667; llb_moe_topk of tools/payload-moeany.patch) ----
#define MOE_MAXROWS 16   // rows of a pass (several streams of k + 1 rows)
// One warp per row of the pass: softmax over the ne logits, the k largest probabilities in descending order with
// ties to the lower index, their weights divided by their sum clamped at 6.103515625e-5; slot k is the shared
// expert (id ne) with weight sigmoid(its gate logit).
// (wt null: the weights are not wanted.)  A round of the selection is two warp-wide reductions of integers: the probabilities are not
// negative, so their bits order as they do.
template <int NQ> __device__ __forceinline__ void moe_route_row(const float *l, int ne, int nk, int *ids, float *wt, int lane) {
  float p[NQ];   // experts lane, lane + 32, ...: ne <= 32 NQ
  float mx = -INFINITY;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int e = lane + 32 * q;
    p[q] = e < ne ? __ldcg(l + e) : -INFINITY;
    mx = fmaxf(mx, p[q]);
  }
  const float gate = __ldcg(l + ne);
  mx = warp_max(mx);
  float sm = 0.0f;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const int e = lane + 32 * q;
    if (e < ne) { p[q] = expf(p[q] - mx); sm += p[q]; }
  }
  sm = warp_sum(sm);
  const float inv = 1.0f / sm;
  unsigned int key[NQ];   // the probability's bits + 1; 0: none, taken, or not a number
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    const float v = p[q] * inv;
    key[q] = lane + 32 * q < ne && v >= 0.0f ? __float_as_uint(v) + 1u : 0u;
  }
  float s = 0.0f, mine_w = 0.0f;   // lane j keeps the weight of rank j
  int mine_id = 0;
  for (int j = 0; j < nk; j++) {
    unsigned int bk = 0, bi = 0x7fffffffu;
#pragma unroll
    for (int q = 0; q < NQ; q++)
      if (key[q] > bk) { bk = key[q]; bi = lane + 32 * q; }   // ascending q: the lane's lowest index among equals
    const unsigned int k = __reduce_max_sync(0xffffffffu, bk);
    const unsigned int i = __reduce_min_sync(0xffffffffu, bk == k && k > 0 ? bi : 0x7fffffffu);
#pragma unroll
    for (int q = 0; q < NQ; q++)
      if (i == (unsigned int)(lane + 32 * q)) key[q] = 0;
    const float bv = k > 0 ? __uint_as_float(k - 1u) : -1.0f;
    s += bv;
    if (j == lane) { mine_w = bv; mine_id = (int)i; }
  }
  s = s < 6.103515625e-5f ? 6.103515625e-5f : s;
  if (lane < nk) { ids[lane] = mine_id; if (wt) wt[lane] = mine_w / s; }
  if (lane == 0) {
    ids[nk] = ne;
    if (wt) wt[nk] = 1.0f / (1.0f + expf(-gate));
  }
}

// ---- top-2: larger value first, lower id on equal values (tools/qwen35_engine.c:763-778) ----
struct Top2 { float v1; int i1; float v2; int i2; };
__device__ __forceinline__ bool t2_before(float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); }
__device__ __forceinline__ void t2_push(Top2 &a, float v, int i) {
  if (i < 0) return;
  if (a.i1 < 0 || t2_before(v, i, a.v1, a.i1)) { a.v2 = a.v1; a.i2 = a.i1; a.v1 = v; a.i1 = i; }
  else if (a.i2 < 0 || t2_before(v, i, a.v2, a.i2)) { a.v2 = v; a.i2 = i; }
}
__device__ __forceinline__ Top2 t2_warp(Top2 a) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    float v1 = __shfl_xor_sync(0xffffffffu, a.v1, m), v2 = __shfl_xor_sync(0xffffffffu, a.v2, m);
    int i1 = __shfl_xor_sync(0xffffffffu, a.i1, m), i2 = __shfl_xor_sync(0xffffffffu, a.i2, m);
    t2_push(a, v1, i1);
    t2_push(a, v2, i2);
  }
  return a;
}

// a K or V value into its cache: two fp16 numbers in two planes
__device__ __forceinline__ void kv_put(__half *c, long long plane, size_t i, float x) {
  const __half h = __float2half_rn(x);
  c[i] = h;
  c[plane + i] = __float2half_rn((x - __half2float(h)) * XP_LO_SCALE);
}

// ---- tensor-core operands of the attention kernels ----
#define ATT_PT 32
#define ATT_PS 40   // halves per row of the probability tiles: 80-byte rows keep ldmatrix conflict-free
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

