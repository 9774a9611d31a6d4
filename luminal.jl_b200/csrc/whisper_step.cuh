// A bf16 Whisper decoder's step in two launches.
#pragma once
#include "common.cuh"

namespace lmb {

constexpr int kWhisperStepLayers = 32, kWhisperStepBatch = 16, kWhisperStepSplits = 4;

struct WhisperStepLayer {
  const __nv_bfloat16 *wqkv, *wo, *wqc, *woc, *wfc1, *wfc2;
  const float *wg_qkv, *bf_qkv, *b_o, *gain_cross, *wg_qc, *bf_qc, *b_oc, *gain_ffn, *wg_fc1, *bf_fc1, *b_fc2, *gain_next;
  __nv_bfloat16* kv;                   // this layer's cache
  const __nv_bfloat16* cross;          // and cross-attention cache
  float* capture;                      // [B][hidden] copy of the residual rows, or NULL
};

struct WhisperStepParams {
  int n_layers = 0, B = 0, Bp = 0, H = 0, hidden = 0, ffn = 0, vocab = 0, q_pitch = 0, cross_len = 0, splits = 0;
  float eps = 0.f, qk_scale = 1.f;
  int64_t kv_b = 0, kv_h = 0, cross_b = 0, cross_h = 0;
  int *tokens = nullptr, *pos = nullptr;
  const __nv_bfloat16* embed = nullptr;
  const float *pos_emb = nullptr, *gain_first = nullptr;
  float *x = nullptr, *ssq = nullptr, *sum = nullptr;                       // in the launched step's layouts
  __nv_bfloat16 *xn = nullptr, *q = nullptr, *attn = nullptr, *act = nullptr;
  bool with_head = false;              // logits, greedy tokens and positions too
  const __nv_bfloat16* head = nullptr;
  const float *wg_head = nullptr, *bf_head = nullptr;
  float* logits = nullptr;
  int logits_pitch = 0;
  int *hist = nullptr, *step_ctr = nullptr, *stop = nullptr;
  const int* limit = nullptr;
  float *part_o = nullptr, *part_ml = nullptr;
  float2* best = nullptr;
  unsigned *done = nullptr, *head_done = nullptr;
  int* err = nullptr;
  const WhisperStepLayer* layers = nullptr;
};

// Whether the kernel runs this decoder at this batch, and its scratch: counters, then the cross attention's partial results.
bool whisper_step_fits(int B, int D, int heads, int kv_heads, int hidden, int ffn, int n_layers);
int64_t whisper_step_scratch_bytes(int B, int heads, int n_layers, int sms);
// Copies the layers' table to the scratch; waits for it.  Before the launches that read it are recorded.
int32_t whisper_step_layers(const WhisperStepLayer* layers, int n_layers, void* scratch, cudaStream_t stream);
int32_t whisper_step_launch(Ctx* ctx, WhisperStepParams p, void* scratch, cudaStream_t stream);

}  // namespace lmb
