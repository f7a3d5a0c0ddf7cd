// The GPT's decode step as one resident kernel (decode_step.cu): what it is given and what a cache keeps for it.
#pragma once
#include <cuda.h>

#include <type_traits>
#include <vector>

#include "model.cuh"

// What a block of the model needs beside its matrices
struct DecodeBlock { bf16 *K, *V; const bf16* ve; long long lam_b, lam_x0, ve_gate; int window; };

struct DecodeStepState {
  int ring[2] = {0, 0};              // slots of its ring for up to 8 and up to 16 columns
  int blocks_n = 0, columns = 0;     // blocks of the kernel, and the columns it takes; 0: this model takes the chain of kernels
  CUtensorMap* maps = nullptr;       // four a block (QKV, wo, fc, proj), then the head
  DecodeBlock* blocks = nullptr;
  unsigned int *launches = nullptr, *hints = nullptr;      // hints: finished items by kind, 128 bytes apart
  // Named words.  One fp32 in 8 bytes, [columns][width]: the mixed stream, the stream after the attention, the stream for the backout, four
  // partial sums of the MLP, projections, the first 16 of the normalised row, ranges of the attention (max, sum, channels)
  uint2 *xm = nullptr, *xa = nullptr, *xb = nullptr, *part = nullptr, *qkv = nullptr, *h16 = nullptr, *att_part = nullptr;
  // Rows of bf16, three words of 16 bytes for 16 columns: what the QKV and the head read, what the MLP reads, its inside by quarters, attention
  uint4 *xn = nullptr, *xa2 = nullptr, *up = nullptr, *att = nullptr;
  size_t named_bytes = 0, hint_bytes = 0;
  float* x0 = nullptr;               // embedding
};

struct DecodeStepArgs {
  const CUtensorMap* maps; const DecodeBlock* blocks; unsigned int *launches, *hints;
  uint2 *xm, *xa, *xb, *part, *qkv, *h16, *att_part;
  uint4 *xn, *xa2, *up, *att;
  float* x0;
  const float* theta;
  const bf16* wte; bf16 *xe_prev, *xe_new;
  const float *sin_t, *cos_t;
  int *tok0, *pos, *doc_start, *lastpos;
  float* logits;
  unsigned int* status;
  long long off_smear, off_lam_s, off_lam_y;
  int d, dq, kv, H, Hkv, V, Vp, L, backout, B, t, maxT, docs, splits, red_bytes, ring;
  float eps;
};

void decode_step_plan(const femto_handle* h, int max_batch, DecodeStepState& st);
size_t decode_step_bytes(const femto_handle* h, DecodeStepState st);
void decode_step_carve(const femto_handle* h, char*& p, DecodeStepState& st);
int decode_step_setup(const femto_handle* h, DecodeStepState& st, const std::vector<void*>& K, const std::vector<void*>& V);
int decode_step_run(const femto_handle* h, const DecodeStepState& st, DecodeStepArgs a, const int* tokens, const int* positions, cudaStream_t s,
                    bool* ran);      // false: the launch was refused and nothing of the cache has changed
// (tokens NULL: the step alone, waiting for what k_step_begin would have left; see femto_selftest_decode_wait)
