// The GPT's decode step as one resident kernel (decode_step.cu): what it is given and what a cache keeps for it.
#pragma once
#include <cuda.h>

#include <type_traits>
#include <vector>

#include "model.cuh"

// What a block of the model needs beside its matrices
struct DecodeBlock { bf16 *K, *V; const bf16* ve; long long lam_b, lam_x0, ve_gate; int window; };

struct DecodeStepState {
  int blocks_n = 0, columns = 0;     // blocks of the kernel, and the columns it takes; 0: this model takes the chain of kernels
  CUtensorMap* maps = nullptr;       // four a block (QKV, wo, fc, proj), then the head
  DecodeBlock* blocks = nullptr;
  unsigned int* counters = nullptr;
  // [columns][width], fp32 unless noted: embedding, mixed stream, stream after the attention, stream for the backout,
  // four partial sums of the MLP, projections, reciprocal norms, MLP inner (bf16), attention partials and their (max, sum)
  float *x0 = nullptr, *xm = nullptr, *xa = nullptr, *xb = nullptr, *part = nullptr, *qkv = nullptr, *inv = nullptr, *att = nullptr;
  float2* att_ml = nullptr;
  bf16* up = nullptr;
};

struct DecodeStepArgs {
  const CUtensorMap* maps; const DecodeBlock* blocks; unsigned int* counters;
  float *x0, *xm, *xa, *xb, *part, *qkv, *inv, *att;
  float2* att_ml;
  bf16* up;
  const float* theta;
  const bf16* wte; bf16* xe_prev;
  const float *sin_t, *cos_t;
  int *tok0, *pos, *doc_start, *lastpos;
  float* logits;
  unsigned int* status;
  long long off_smear, off_lam_s, off_lam_y;
  int d, dq, kv, H, Hkv, V, Vp, L, backout, B, t, maxT, docs, splits, n_counters, red_bytes;
  float eps;
};

void decode_step_plan(const femto_handle* h, int max_batch, DecodeStepState& st);
size_t decode_step_bytes(const femto_handle* h, DecodeStepState st);
void decode_step_carve(const femto_handle* h, char*& p, DecodeStepState& st);
int decode_step_setup(const femto_handle* h, DecodeStepState& st, const std::vector<void*>& K, const std::vector<void*>& V);
int decode_step_run(const femto_handle* h, const DecodeStepState& st, DecodeStepArgs a, const int* tokens, const int* positions, cudaStream_t s);
