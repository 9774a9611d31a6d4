// What the kernels that run a whole decode step (llama_step.cu, whisper_step.cu) share, and the end of a greedy step wherever it is launched.
#pragma once
#include <math_constants.h>

#include "common.cuh"

namespace lmb {

constexpr long long kStepWaitCycles = 4000000000ll;        // about 2 s

// Waits until `need` units of the piece before have been counted; false if that took too long (*err says so to the host, *given_up, in shared memory and zero
// at the start, to this block).  All threads call it.
__device__ __forceinline__ bool wait_units(const unsigned* counter, unsigned need, int* err, int* given_up) {
  if (threadIdx.x == 0) {
    const long long t0 = clock64();
    unsigned spins = 0, v;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
      if (v >= need) break;
      if ((++spins & 255u) == 0u && (clock64() - t0 > kStepWaitCycles || *reinterpret_cast<volatile int*>(err) != 0)) {
        *reinterpret_cast<volatile int*>(err) = 1;
        *given_up = 1;
        break;
      }
    }
  }
  __syncthreads();
  return *given_up == 0;
}
__device__ __forceinline__ void count_unit(unsigned* counter) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
}

// Whether this is the last block of the grid to come here; all threads call it once.  *flag, in shared memory, is this block's.
__device__ __forceinline__ bool last_block(unsigned* gone, int* flag) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *flag = atomicAdd(gone, 1u) == gridDim.x - 1u ? 2 : 0;
    __threadfence();
  }
  __syncthreads();
  return *flag == 2;
}

// The id of the largest of the blocks' best logits (the lowest id of equals), by a warp; pairs: (logit, id) of a sequence, `pitch` apart.
__device__ __forceinline__ int best_of_blocks(const float2* pairs, int pitch, int lane) {
  float v = -CUDART_INF_F;
  int i = 0x7fffffff;
  for (int k = lane; k < (int)gridDim.x; k += 32) {
    const float2 o = __ldcg(pairs + (int64_t)k * pitch);
    const int oi = __float_as_int(o.y);
    if (o.x > v || (o.x == v && oi < i)) { v = o.x; i = oi; }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float o = __shfl_xor_sync(0xffffffffu, v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, i, off);
    if (o > v || (o == v && oi < i)) { v = o; i = oi; }
  }
  return i;
}

// Sequence b's greedy token, by one thread.  stop (or NULL): the end-of-text id or -1, how many sequences have produced it, [2 + b] whether sequence b has: it then
// keeps emitting it, the batch form of the reference's `break` at EOT (src/Decoding.jl:126-129).  hist may be NULL.
__device__ __forceinline__ void keep_token(int id, int b, int B, int* tokens, int* hist, const int* step_ctr, int* stop) {
  const int eot = stop ? stop[0] : -1;
  if (eot >= 0) {
    if (stop[2 + b]) id = eot;
    else if (id == eot) { stop[2 + b] = 1; atomicAdd(&stop[1], 1); }
  }
  tokens[b] = id;
  if (hist) hist[(int64_t)(*step_ctr) * B + b] = id;
}

}  // namespace lmb
