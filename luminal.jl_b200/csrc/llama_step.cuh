// One launch for a small float32 Llama's step.
#pragma once
#include "common.cuh"

namespace lmb {

constexpr int kLlamaStepBatch = 4;

struct LlamaStepLayer {
  const float *wqkv, *wo, *wgu, *wdown;      // Layout<float>
  const float *gain_attn, *gain_ffn;
  float* kv;                                 // this layer's cache
  float* capture;                            // [B][hidden] copy of the residual rows, or NULL
};

struct LlamaStepParams {
  int n_layers = 0, B = 0, Hl = 0, KVl = 0, G = 0, hidden = 0, ffn = 0, vocab = 0, logits_pitch = 0;
  bool with_head = false;
  float eps = 0.f, scale = 1.f;
  int64_t kv_b = 0, kv_h = 0;
  int *tokens = nullptr, *pos = nullptr, *hist = nullptr, *step_ctr = nullptr, *stop = nullptr;
  const int* limit = nullptr;
  const float *embed = nullptr, *gain_final = nullptr, *head = nullptr, *inv_freq = nullptr;
  float *x = nullptr, *q = nullptr, *attn = nullptr, *act = nullptr, *logits = nullptr;     // [B][..], rows as wide as they are
  const LlamaStepLayer* layers = nullptr;
  unsigned* done = nullptr;
  float2* best = nullptr;
  int* err = nullptr;
};

// Whether the kernel runs this decoder at this batch and cache capacity, and its scratch
bool llama_step_fits(int B, int D, int hidden, int ffn, int vocab, int n_layers, int capacity);
int64_t llama_step_scratch_bytes(int n_layers, int sms);
// Copies the layers' table to the scratch; waits for it.  Before the launches that read it are recorded.
int32_t llama_step_layers(const LlamaStepLayer* layers, int n_layers, void* scratch, cudaStream_t stream);
int32_t llama_step_launch(Ctx* ctx, LlamaStepParams p, int D, void* scratch, cudaStream_t stream);

}  // namespace lmb
