// Steps of a recorded graph (lmb200_capture_begin .. lmb200_capture_end) and the kernel that runs many of them in one launch.
#pragma once
#include <vector>

#include "common.cuh"

namespace lmb {

constexpr int kMaxRank = 8;
constexpr float kInvLn2 = 1.4426950408889634f;

// postfix programs of lmb200_fused_ew
constexpr int kFusedMaxInputs = 8, kFusedMaxInstr = 64, kFusedMaxStack = 16;
enum FusedOp { F_PUSH_IN = 0, F_PUSH_CONST = 1, F_ADD = 2, F_MUL = 3, F_MOD = 4, F_LT = 5, F_MAX = 6, F_LOG2 = 7, F_EXP2 = 8,
               F_SIN = 9, F_COS = 10, F_SQRT = 11, F_RECIP = 12, F_RELU = 13, F_FMA = 14, F_ADD_RELU = 15 };

#ifdef __CUDACC__
__device__ __forceinline__ float apply_op(int op, float a, float b, float c) {
  switch (op) {
    case LMB200_OP_ADD: return a + b;
    case LMB200_OP_MUL: return a * b;
    case LMB200_OP_MOD: return fmodf(a, b);
    case LMB200_OP_LESSTHAN: return a < b ? 1.0f : 0.0f;
    case LMB200_OP_MAX: return fmaxf(a, b);
    case LMB200_OP_LOG2: return log2f(a);
    case LMB200_OP_EXP2: return exp2f(a);
    case LMB200_OP_SIN: return sinf(a);
    case LMB200_OP_COS: return cosf(a);
    case LMB200_OP_SQRT: return sqrtf(a);
    case LMB200_OP_RECIP: return 1.0f / a;
    case LMB200_OP_RELU: return fmaxf(a, 0.0f);
    case LMB200_OP_COPY: return a;
    case LMB200_OP_FUSED_MUL_ADD: return __fadd_rn(__fmul_rn(a, b), c);   // (a .* b) .+ c, two roundings
    case LMB200_OP_FUSED_ADD_RELU: return fmaxf(a + b, 0.0f);
  }
  return 0.f;
}

__device__ __forceinline__ float fused_unary(int op, float a) {
  switch (op) {
    case F_LOG2: return log2f(a);
    case F_EXP2: return exp2f(a);
    case F_SIN: return sinf(a);
    case F_COS: return cosf(a);
    case F_SQRT: return sqrtf(a);
    case F_RECIP: return 1.0f / a;
    case F_RELU: return fmaxf(a, 0.0f);
  }
  return a;
}

__device__ __forceinline__ float fused_binary(int op, float a, float b) {
  switch (op) {
    case F_ADD: return __fadd_rn(a, b);
    case F_MUL: return __fmul_rn(a, b);
    case F_MOD: return fmodf(a, b);
    case F_LT: return a < b ? 1.0f : 0.0f;
    case F_MAX: return fmaxf(a, b);
    case F_ADD_RELU: return fmaxf(__fadd_rn(a, b), 0.0f);
  }
  return 0.f;
}

__device__ __forceinline__ float silu_gate(float a, float up) {
  const float e = exp2f((a * -1.0f) * kInvLn2);
  const float sg = 1.0f / (1.0f + e);
  return (a * sg) * up;
}
#endif

enum StepKind { STEP_EW, STEP_FUSED, STEP_SILU, STEP_COPY, STEP_RESHAPE, STEP_PAD, STEP_REDUCE, STEP_MATMUL, STEP_GATHER, STEP_CUMSUM, STEP_NORM };

// element [i0, i1, ..] of a tensor as base[offset + sum i_k st_k]; `elems` elements from base on belong to it
struct StepView {
  const float* base = nullptr;
  int64_t elems = 0, offset = 0;
  int rank = 0;
  int64_t d[kMaxRank] = {}, st[kMaxRank] = {};
};

struct RecordedStep {
  StepKind kind = STEP_EW;
  int op = 0;                          // EW: opcode; REDUCE: kind; NORM: 1 = centred
  float* out = nullptr;
  int rank = 0;
  int64_t d[kMaxRank] = {};            // the output
  std::vector<StepView> in;            // row-major tensors as the call named them (NORM: x, gain, bias; a missing one has no base)
  std::vector<int> arg;                // PAD: left margins; COPY: per output axis the source axis + 1 (0: none), from kMaxRank on per source axis its start;
                                       // FUSED: opcodes
  std::vector<float> val;              // FUSED: arguments; NORM: epsilon
  int64_t n = 0, inner = 0;            // REDUCE: axis length and elements behind it; NORM, CUMSUM: row length; GATHER: table rows
  cudaGraphNode_t node = nullptr;      // the kernel this step was recorded as
};

// a row-major tensor
StepView step_tensor(const float* p, int rank, const int64_t* d);

// Between capture_begin and capture_end: notes the step whose kernel was just launched into the capture.
void record_step(Ctx* ctx, RecordedStep&& s);
void record_begin(Ctx* ctx);

// After capture: replaces runs of recorded steps in `graph` by kernels that run them.  *programs receives the device memory these read
// (the caller frees it with the graph); *kernels the number of kernels the graph now launches.  The graph is left as it was where nothing is gained.
void record_finish(Ctx* ctx, cudaGraph_t* graph, std::vector<void*>* programs, int64_t* kernels);
void record_drop(Ctx* ctx);

}  // namespace lmb
