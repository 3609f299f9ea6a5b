// pf.cuh -- host interface of the prompt path (pf.cu): the dense tcgen05 GEMM and the row-batched ops of a chunk.
#pragma once
#include "model.cuh"

#define PF_MAXMAT 4
struct PfMat {
  const uint8_t *W;     // device layout (common.cuh)
  float *out;           // [ksplit][PF rows][ostride]
  int rows, ostride;
  long long split_stride;
};
struct PfArgs {
  PfMat m[PF_MAXMAT];
  int nmat;
  int t128[PF_MAXMAT + 1];   // prefix sums of 128-row tiles
  int K, ksplit, R;          // columns, K-slices, rows of the chunk in use (<= PF_RMAX)
  const __half *x;           // activations, k-group major
  unsigned int *err;
};


int pf_setup(void);                               // -1, or 1: no room on the device
int pf_wait_errors_clear(void);
int pf_wait_errors(void);                         // 1 when a bounded wait of the dense GEMM ran out
int pf_pick_ksplit(int ntiles, int nsb, int sms);
int pf_gemm(cudaStream_t s, int fmt, PfArgs &a);  // fills the tile table; a.ksplit <= K / 256
int op_pf_embed(cudaStream_t s, int fmt, const uint8_t *W, int d, const int *ids, int R, float *x);
int op_pf_norm(cudaStream_t s, const float *xin, PartIn add, const float *w, float eps, int d, float *xout, __half *kg, int kg_K, int kg_col0, float *hn_out, int R, int ru, int row0 = 0);   // rows row0 .. of kg, whose units have ru rows
int op_pf_silu(cudaStream_t s, PartIn g, PartIn u, int f, __half *kg, int R, int ru);
int op_pf_qkrope(cudaStream_t s, PartIn q, PartIn k, PartIn v, const float *qn_w, const float *kn_w, const double *invfreq, AttnShape sh, int p0, int R, float *qout, float *Kc, float *Vc, bool kv_only = false);
size_t op_pf_attn_parts(int H, int KV);           // values of pm and pl; po has head_dim as many
int op_pf_attn(cudaStream_t s, const float *q, const float *Kc, const float *Vc, PartIn qg, AttnShape sh, int p0, int R, float *pm, float *pl, float *po, __half *kg, int row0, int ru);
// the sequences of a chunk: rows off .. off + R - 1 of it are positions p0 .. of one; its conv history, state and control block
#define PF_PIECES 16                                 // most of them
#define PF_STEPS (PF_RMAX / 8 + PF_PIECES)           // most steps of eight rows, each of one sequence
struct PfSeg { int p0, R, off; float *ring, *S; const SpecCtl *ctl; };
struct PfSegs { int n; PfSeg s[PF_PIECES]; };
int op_pf_delta(cudaStream_t s, PartIn qkv, PartIn z, PartIn bp, PartIn ap, int ring_ks, const float *cw, const float *dt, const float *sa,
                const float *nw, DeltaShape sh, const PfSegs &sg, float *y, float *gram, float *beta, float *decay, float *o, __half *kg, int ru);   // gram: GK x PF_STEPS x 64; beta, decay: TR x 8 PF_STEPS
