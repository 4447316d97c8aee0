// The decode step as one resident kernel (step_resident.cu).
#pragma once
#include "kernels.h"

namespace nfai {

struct ResidentArgs {
  const void* w[5] = {};              // QKV, O, gate/up and down of layer 0, the head
  const float *attn_norm = nullptr, *ffn_norm = nullptr;  // of layer 0
  uint64_t layer_stride = 0;          // bytes from a layer's weights and gains to the next one's
  void *kc = nullptr, *vc = nullptr;  // [L][ctx][kvH*d] float16
  uint32_t L = 0, H = 0, qH = 0, kvH = 0, d = 0, F = 0, V = 0, ctx = 0, ropeDim = 0;
  float eps = 0.f;
  const void* embd = nullptr;
  const float* out_norm = nullptr;
  const float2* rope_cs = nullptr;
  StepState* state = nullptr;
  const uint32_t* prompt = nullptr;   // non-null: the token comes from here (StepState::prompt_idx)
  float* xbuf = nullptr;              // [2L + 1][H] residual streams
  float* logits = nullptr;
  float* part_val = nullptr;          // [CTAs]
  uint32_t* part_idx = nullptr;
  uint32_t* history = nullptr;
  uint32_t history_cap = 0;
  unsigned long long* words = nullptr;  // [L + 1][words_per_layer] (value, tag), zero before the first step
  uint32_t* epoch = nullptr;            // steps so far
  uint32_t* ticket = nullptr;           // zero between steps
  uint32_t with_head = 1;
  unsigned long long wait_ns = 1000000000ull;  // budget of a poll
  // filled in by resident_plan
  uint32_t words_per_layer = 0, splits = 1;
};
struct ResidentStep : ResidentArgs {
  alignas(64) unsigned char maps[5][4][128] = {};  // of w: boxes of 16, 8, 4 and 2 rows
};

size_t resident_words_per_layer(uint32_t H, uint32_t qH, uint32_t kvH, uint32_t d, uint32_t F);
// Steps from this position on are a sequence of launches (p as resident_plan left it).
uint32_t resident_positions(const ResidentArgs& p);
// Fills in the launch's layout; false where the sizes, types or the device do not fit (the step is then a sequence of launches).
bool resident_plan(int wdtype, int kvdtype, ResidentStep* p);
cudaError_t launch_step_resident(cudaStream_t s, const ResidentStep& p);

}  // namespace nfai
