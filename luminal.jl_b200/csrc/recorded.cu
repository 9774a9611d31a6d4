// Recorded graphs of primitive ops as few launches.
//
// A traced graph of the reference is a chain of hundreds of steps of a microsecond's work or less.  As one graph node per step a replay is bound by
// the time from one node to the next (404 nodes of a small Llama's 32-token graph: 2.4 us each, 985 us), and most of these nodes only move
// elements.  At capture_end the runs of such steps become ONE kernel each (vm_kernel) where that is estimated to be faster (own_us, plan_run): a CTA per SM walks through its own list of (step, tile)
// entries and waits for the steps its entry reads by their tile counters, so what counts is the dependency chain, not the number of steps.  Two things
// shorten that chain:
//   * a movement step (permute, expand, slice, most reshapes) is an affine view of what it reads.  A step that reads such a step's output reads the
//     source through the view instead (plan_steps), so movements are still written out -- every buffer holds what it held -- but nobody waits for them;
//   * a product whose tiles of 32 x 32 would leave SMs idle takes tiles of 32 x 8.
// The arithmetic of every step is that of its own kernel in prims.cu, sums in the same order: a replay gives the bits of the calls it records.
// Measured: the comment at vm_kernel.
#include "recorded.cuh"

#include <algorithm>
#include <stdlib.h>
#include <string.h>

namespace lmb {

StepView step_tensor(const float* p, int rank, const int64_t* d) {
  StepView v;
  v.base = p; v.rank = rank;
  int64_t mul = 1;
  for (int k = rank - 1; k >= 0; --k) { v.d[k] = d[k]; v.st[k] = mul; mul *= d[k]; }
  v.elems = mul;
  return v;
}

namespace {

constexpr int kVmThreads = 256, kMaxDeps = 31, kPitchNarrow = 260, kPitchWide = 132;
constexpr int kBufFloats = 48 * kPitchNarrow;            // a 32 x 16 product's operands, 256 k at a time: the largest user
constexpr long long kVmWaitCycles = 4000000000ll;        // about 2 s

// One step as the kernel reads it.  Strides in elements; every index fits 32 bits (checked where it is built).
struct __align__(16) VmOp {
  float* out;
  const float* in[8];
  int kind, op, rank, n_in;
  int total, per, n_instr, n_dep;
  uint32_t d[8], mul[8];               // output axes; quotients by d as (umulhi(n, mul) + n) >> shift for n < 2^31
  int st[8][8];                        // [input][axis]
  int p[8];
  float f;
  uint8_t shift[8], code[kFusedMaxInstr];
  float arg[kFusedMaxInstr];
  uint32_t dep[kMaxDeps];              // step | tiles << 16
};
constexpr int kOpWords = sizeof(VmOp) / 4;
static_assert(sizeof(VmOp) % 16 == 0 && kOpWords <= kVmThreads, "one word of a step per thread");

struct VmParams {
  const VmOp* ops;
  const uint32_t* entries;             // step | tile << 16, in the order a CTA takes them
  const int* first;                    // [grid + 1]
  unsigned* done;                      // [steps] finished tiles, then the CTAs that have left
  int n_ops;
  int* err;
};

struct FastDiv { uint32_t mul; int shift; };
FastDiv fast_div(uint32_t d) {
  int l = 0;
  while ((1ull << l) < d) ++l;
  return {(uint32_t)(((1ull << 32) * ((1ull << l) - d)) / d + 1), l};
}

__device__ __forceinline__ uint32_t quotient(uint32_t n, uint32_t mul, int shift) { return (__umulhi(n, mul) + n) >> shift; }

// offsets of up to N inputs for output element o
template <int N>
__device__ __forceinline__ void offsets(const VmOp& q, uint32_t o, int (&off)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) off[i] = 0;
  uint32_t rem = o;
  for (int k = q.rank - 1; k >= 0; --k) {
    const uint32_t nx = k ? quotient(rem, q.mul[k], q.shift[k]) : 0u, idx = rem - nx * q.d[k];
    rem = nx;
#pragma unroll
    for (int i = 0; i < N; ++i) off[i] += (int)idx * q.st[i][k];
  }
}

template <int N>
__device__ __forceinline__ void vm_fused(const VmOp& q, int tile, float* buf) {
  float* leaf = buf + threadIdx.x;                       // [input][thread]
  float* stack = buf + kFusedMaxInputs * kVmThreads + threadIdx.x;
  for (int j = 0; j < q.per; ++j) {
    const uint32_t o = (uint32_t)(tile * q.per + j) * kVmThreads + threadIdx.x;
    if (o >= (uint32_t)q.total) return;
    int off[N];
    offsets(q, o, off);
    float v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = i < q.n_in ? q.in[i][off[i]] : 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) leaf[i * kVmThreads] = v[i];
    float top = 0.f;                                     // the stack's last value; those below it from stack[0] on
    int below = -1;
    for (int pc = 0; pc < q.n_instr; ++pc) {
      const int op = q.code[pc];
      if (op <= F_PUSH_CONST) {
        if (below >= 0) stack[below * kVmThreads] = top;
        ++below;
        top = op == F_PUSH_CONST ? q.arg[pc] : leaf[(int)q.arg[pc] * kVmThreads];
      } else if (op >= F_LOG2 && op <= F_RELU) {
        top = fused_unary(op, top);
      } else if (op == F_FMA) {
        const float b = stack[(below - 1) * kVmThreads], a = stack[(below - 2) * kVmThreads];
        top = __fadd_rn(__fmul_rn(a, b), top);
        below -= 2;
      } else {
        top = fused_binary(op, stack[(below - 1) * kVmThreads], top);
        --below;
      }
    }
    q.out[o] = top;
  }
}

__device__ __forceinline__ void vm_copy(const VmOp& q, int tile) {
  uint32_t rem[8];
  int off[8];
  const uint32_t o0 = (uint32_t)tile * q.per * kVmThreads + threadIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) { rem[j] = o0 + j * kVmThreads; off[j] = 0; }
  for (int k = q.rank - 1; k >= 0; --k) {
    const uint32_t mul = q.mul[k], d = q.d[k];
    const int sh = q.shift[k], st = q.st[0][k];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t nx = k ? quotient(rem[j], mul, sh) : 0u;
      off[j] += (int)(rem[j] - nx * d) * st;
      rem[j] = nx;
    }
  }
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < q.per && o0 + j * kVmThreads < (uint32_t)q.total) v[j] = q.in[0][off[j]];
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < q.per && o0 + j * kVmThreads < (uint32_t)q.total) q.out[o0 + j * kVmThreads] = v[j];
}

// a column-major reshape that is no affine view: st[0] the input's strides, st[1] its axes, st[2] and st[3] their quotients, st[4] the output axes'
// places in column-major order; p[0] the input's rank
__device__ __forceinline__ void vm_reshape(const VmOp& q, int tile) {
  for (int j = 0; j < q.per; ++j) {
    const uint32_t o = (uint32_t)(tile * q.per + j) * kVmThreads + threadIdx.x;
    if (o >= (uint32_t)q.total) return;
    uint32_t rem = o, lin = 0;
    for (int k = q.rank - 1; k >= 0; --k) {
      const uint32_t nx = k ? quotient(rem, q.mul[k], q.shift[k]) : 0u;
      lin += (rem - nx * q.d[k]) * (uint32_t)q.st[4][k];
      rem = nx;
    }
    int src = 0;
    for (int k = 0; k < q.p[0]; ++k) {
      const uint32_t nx = quotient(lin, (uint32_t)q.st[2][k], q.st[3][k]);
      src += (int)(lin - nx * (uint32_t)q.st[1][k]) * q.st[0][k];
      lin = nx;
    }
    q.out[o] = q.in[0][src];
  }
}

// st[1] left margins, st[2] the input's axes
__device__ __forceinline__ void vm_pad(const VmOp& q, int tile) {
  for (int j = 0; j < q.per; ++j) {
    const uint32_t o = (uint32_t)(tile * q.per + j) * kVmThreads + threadIdx.x;
    if (o >= (uint32_t)q.total) return;
    uint32_t rem = o;
    int src = 0;
    bool inside = true;
    for (int k = q.rank - 1; k >= 0; --k) {
      const uint32_t nx = k ? quotient(rem, q.mul[k], q.shift[k]) : 0u;
      const int i = (int)(rem - nx * q.d[k]) - q.st[1][k];
      rem = nx;
      if (i < 0 || i >= q.st[2][k]) inside = false;
      src += i * q.st[0][k];
    }
    q.out[o] = inside ? q.in[0][src] : 0.f;
  }
}

// p: axis length, elements behind the axis.  Rows of at most 256 values come through shared memory: reading them by one thread each is uncoalesced.
__device__ __forceinline__ void vm_reduce(const VmOp& q, int tile, float* buf) {
  const int n = q.p[0], inner = q.p[1];
  if (q.per == 32) {
    const int row0 = tile * 32, rows = min(32, q.total - row0), pitch = n + 1 - (n & 1);
    const float* src = q.in[0] + (int64_t)row0 * n;
    for (int r = threadIdx.x >> 5; r < rows; r += kVmThreads / 32)
      for (int i = threadIdx.x & 31; i < n; i += 32) buf[r * pitch + i] = src[r * n + i];
    __syncthreads();
    if ((int)threadIdx.x < rows) {
      const float* p = buf + threadIdx.x * pitch;
      float acc = q.op == LMB200_REDUCE_SUM ? 0.f : -INFINITY;
#pragma unroll 16
      for (int i = 0; i < n; ++i) acc = q.op == LMB200_REDUCE_SUM ? acc + p[i] : fmaxf(acc, p[i]);
      q.out[row0 + threadIdx.x] = acc;
    }
    return;
  }
  const uint32_t o = (uint32_t)tile * kVmThreads + threadIdx.x;
  if (o >= (uint32_t)q.total) return;
  const uint32_t a = o / (uint32_t)inner, c = o - a * inner;
  const float* p = q.in[0] + (int64_t)a * n * inner + c;
  float acc = q.op == LMB200_REDUCE_SUM ? 0.f : -INFINITY;
  int i = 0;
  for (; i + 16 <= n; i += 16) {
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = p[(int64_t)(i + j) * inner];
#pragma unroll
    for (int j = 0; j < 16; ++j) acc = q.op == LMB200_REDUCE_SUM ? acc + v[j] : fmaxf(acc, v[j]);
  }
  for (; i < n; ++i) {
    const float v = p[(int64_t)i * inner];
    acc = q.op == LMB200_REDUCE_SUM ? acc + v : fmaxf(acc, v);
  }
  q.out[o] = acc;
}

// 32 rows x COLS columns of a product; st[0] = A's strides (batch, batch, row, k), st[1] = B's (batch, batch, k, column); p: M, N, K, column tiles,
// row tiles, inner batch, A and B in vectors of four k.  Warp w multiplies k = 16 w .. 16 w + 15 of every 128, as matmul_kernel does, a lane one
// column and COLS rows; both operands lie k-contiguous in shared memory (pitch = 4 mod 32 words: rows 4 banks apart), four k per read.
template <int COLS, int KC, int PITCH>
__device__ __forceinline__ void vm_matmul(const VmOp& q, int tile, float* buf) {
  constexpr int kA = 32 * KC / kVmThreads, kB = COLS * KC / kVmThreads, kLanesK = KC / 32, kLanesK4 = KC / 128, kGroups = 32 / COLS;
  float* As = buf;                                       // [row][k]
  float* Bs = buf + 32 * PITCH;                          // [column][k]
  const int M = q.p[0], N = q.p[1], K = q.p[2];
  const int tn = tile % q.p[3], tmb = tile / q.p[3], tm = tmb % q.p[4], bt = tmb / q.p[4], b1 = bt % q.p[5], b0 = bt / q.p[5];
  const float* a = q.in[0] + b0 * q.st[0][0] + b1 * q.st[0][1];
  const float* b = q.in[1] + b0 * q.st[1][0] + b1 * q.st[1][1];
  float* c = q.out + (int64_t)bt * M * N;
  const int sam = q.st[0][2], sak = q.st[0][3], sbk = q.st[1][2], sbn = q.st[1][3];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, row0 = tm * 32, col0 = tn * COLS;
  const int lc = lane % COLS, lg = lane / COLS;
  const bool b_cols = sbk != 1;                          // lanes along the axis that is contiguous in memory
  float an[kA], bn[kB], acc[COLS];
#pragma unroll
  for (int r = 0; r < COLS; ++r) acc[r] = 0.f;
  // rows or columns and k of this thread's elements of a chunk: lanes along the axis that is contiguous in memory
  const bool a4 = q.p[6] & 1, b4 = q.p[6] & 2;
  auto fetch = [&](int k0) {
    if (a4) {
#pragma unroll
      for (int j = 0; j < kA / 4; ++j) {
        const int r = w + 8 * (j / kLanesK4), k = 4 * (lane + 32 * (j % kLanesK4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row0 + r < M && k0 + k < K) v = *reinterpret_cast<const float4*>(a + (row0 + r) * sam + k0 + k);
        an[4 * j] = v.x; an[4 * j + 1] = v.y; an[4 * j + 2] = v.z; an[4 * j + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kA; ++j) {
        const int r = w + 8 * (j / kLanesK), k = lane + 32 * (j % kLanesK);
        an[j] = (row0 + r < M && k0 + k < K) ? a[(row0 + r) * sam + (k0 + k) * sak] : 0.f;
      }
    }
    if (b4) {
#pragma unroll
      for (int j = 0; j < kB / 4; ++j) {
        const int n = w + 8 * (j / kLanesK4), k = 4 * (lane + 32 * (j % kLanesK4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (col0 + n < N && k0 + k < K) v = *reinterpret_cast<const float4*>(b + (col0 + n) * sbn + k0 + k);
        bn[4 * j] = v.x; bn[4 * j + 1] = v.y; bn[4 * j + 2] = v.z; bn[4 * j + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int n = b_cols ? lc : w + 8 * (j / kLanesK), k = b_cols ? lg + kGroups * (w + 8 * j) : lane + 32 * (j % kLanesK);
        bn[j] = (col0 + n < N && k0 + k < K) ? b[(k0 + k) * sbk + (col0 + n) * sbn] : 0.f;
      }
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += KC) {
    if (a4) {
#pragma unroll
      for (int j = 0; j < kA / 4; ++j)
        *reinterpret_cast<float4*>(&As[(w + 8 * (j / kLanesK4)) * PITCH + 4 * (lane + 32 * (j % kLanesK4))]) = make_float4(an[4 * j], an[4 * j + 1], an[4 * j + 2], an[4 * j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < kA; ++j) As[(w + 8 * (j / kLanesK)) * PITCH + lane + 32 * (j % kLanesK)] = an[j];
    }
    if (b4) {
#pragma unroll
      for (int j = 0; j < kB / 4; ++j)
        *reinterpret_cast<float4*>(&Bs[(w + 8 * (j / kLanesK4)) * PITCH + 4 * (lane + 32 * (j % kLanesK4))]) = make_float4(bn[4 * j], bn[4 * j + 1], bn[4 * j + 2], bn[4 * j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < kB; ++j) {
        const int n = b_cols ? lc : w + 8 * (j / kLanesK), k = b_cols ? lg + kGroups * (w + 8 * j) : lane + 32 * (j % kLanesK);
        Bs[n * PITCH + k] = bn[j];
      }
    }
    __syncthreads();
    if (k0 + KC < K) fetch(k0 + KC);
#pragma unroll
    for (int h = 0; h < KC; h += 128) {
      if (k0 + h + 16 * w >= K) break;
#pragma unroll
      for (int k = h + 16 * w; k < h + 16 * w + 16; k += 4) {
        const float4 bv = *reinterpret_cast<const float4*>(&Bs[lc * PITCH + k]);
#pragma unroll
        for (int r = 0; r < COLS; ++r) {
          const float4 av = *reinterpret_cast<const float4*>(&As[(lg + kGroups * r) * PITCH + k]);
          acc[r] = fmaf(av.x, bv.x, acc[r]);
          acc[r] = fmaf(av.y, bv.y, acc[r]);
          acc[r] = fmaf(av.z, bv.z, acc[r]);
          acc[r] = fmaf(av.w, bv.w, acc[r]);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < COLS; ++r) buf[(w * 32 + lg + kGroups * r) * COLS + lc] = acc[r];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < COLS / 8; ++j) {
    const int e = (int)threadIdx.x + kVmThreads * j, r = e / COLS, n = e % COLS;
    float t = 0.f;
#pragma unroll
    for (int v = 0; v < 8; ++v) t += buf[(v * 32 + r) * COLS + n];
    if (row0 + r < M && col0 + n < N) c[(row0 + r) * N + col0 + n] = t;
  }
}

// a row per tile: in = x, gain, bias; p[0] its length, op 1 = centred
__device__ __forceinline__ void vm_norm(const VmOp& q, int row, float* buf) {
  const int n = q.p[0], tid = threadIdx.x;
  const float* xr = q.in[0] + (int64_t)row * n;
  float* yr = q.out + (int64_t)row * n;
  auto block_sum = [&](float v) -> float {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((tid & 31) == 0) buf[tid >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += buf[i];
    return t;
  };
  float mean = 0.f;
  if (q.op) {
    float s = 0.f;
    for (int i = tid; i < n; i += kVmThreads) s += xr[i];
    mean = block_sum(s) * (1.0f / (float)n);
  }
  float ss = 0.f;
  for (int i = tid; i < n; i += kVmThreads) { const float v = xr[i] + mean * -1.0f; ss += v * v; }
  const float var = block_sum(ss) * (1.0f / (float)n);
  const float inv = 1.0f / sqrtf(var + q.f);
  for (int i = tid; i < n; i += kVmThreads) {
    float v = (xr[i] + mean * -1.0f) * inv;
    if (q.in[1]) v = v * q.in[1][i];
    if (q.in[2]) v = v + q.in[2][i];
    yr[i] = v;
  }
}

__device__ __forceinline__ void vm_run(const VmOp& q, int tile, float* buf) {
  switch (q.kind) {
    case STEP_EW:
    case STEP_SILU:
      for (int j = 0; j < q.per; ++j) {
        const uint32_t o = (uint32_t)(tile * q.per + j) * kVmThreads + threadIdx.x;
        if (o >= (uint32_t)q.total) return;
        int off[3];
        offsets(q, o, off);
        const float a = q.in[0][off[0]], b = q.n_in > 1 ? q.in[1][off[1]] : 0.f, c = q.n_in > 2 ? q.in[2][off[2]] : 0.f;
        q.out[o] = q.kind == STEP_SILU ? silu_gate(a, b) : apply_op(q.op, a, b, c);
      }
      return;
    case STEP_FUSED:
      if (q.n_in <= 2) vm_fused<2>(q, tile, buf);
      else if (q.n_in <= 4) vm_fused<4>(q, tile, buf);
      else vm_fused<kFusedMaxInputs>(q, tile, buf);
      return;
    case STEP_COPY: vm_copy(q, tile); return;
    case STEP_RESHAPE: vm_reshape(q, tile); return;
    case STEP_PAD: vm_pad(q, tile); return;
    case STEP_REDUCE: vm_reduce(q, tile, buf); return;
    case STEP_MATMUL:
      if (q.op == 8) vm_matmul<8, 256, kPitchNarrow>(q, tile, buf);
      else if (q.op == 16) vm_matmul<16, 256, kPitchNarrow>(q, tile, buf);
      else vm_matmul<32, 128, kPitchWide>(q, tile, buf);
      return;
    case STEP_GATHER:                                    // in = table, ids; p: row length, table rows
      for (int j = 0; j < q.per; ++j) {
        const uint32_t o = (uint32_t)(tile * q.per + j) * kVmThreads + threadIdx.x;
        if (o >= (uint32_t)q.total) return;
        const uint32_t r = o / (uint32_t)q.p[0], col = o - r * q.p[0];
        const int64_t id = (int64_t)q.in[1][r];
        q.out[o] = (id >= 0 && id < q.p[1]) ? q.in[0][id * q.p[0] + col] : 0.f;
      }
      return;
    case STEP_CUMSUM: {                                  // p[0]: row length
      const uint32_t r = (uint32_t)tile * kVmThreads + threadIdx.x;
      if (r >= (uint32_t)q.total) return;
      const int n = q.p[0];
      const float* x = q.in[0] + (int64_t)r * n;
      float* y = q.out + (int64_t)r * n;
      float acc = 0.f;
      int i = 0;
      for (; i + 16 <= n; i += 16) {
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = x[i + j];
#pragma unroll
        for (int j = 0; j < 16; ++j) { acc += v[j]; y[i + j] = acc; }
      }
      for (; i < n; ++i) { acc += x[i]; y[i] = acc; }
      return;
    }
    case STEP_NORM: vm_norm(q, tile, buf); return;
  }
}

// One CTA per SM (launched cooperatively: they wait for one another).  Bound by the dependency chain: per link one counter through L2 (release, acquire),
// the operands' trip from L2 and the step itself.  The next entry's step is fetched while the present one waits and runs.
// The small Llama's 32-token graph (404 steps, a longest chain of 90): 237 us a replay, 2.0 us per element-wise link and 2.2 to 4 us per product, 950 us
// as 404 nodes.  Of an element-wise link 1.1 us is the step with its release; a second fence in front of the release made that 1.4.
__global__ void __launch_bounds__(kVmThreads, 1) vm_kernel(const VmParams P) {
  extern __shared__ __align__(16) float buf[];
  __shared__ VmOp ops[2];
  __shared__ int dead;
  const int tid = threadIdx.x, lane = tid & 31;
  const int first = P.first[blockIdx.x], last = P.first[blockIdx.x + 1];
  if (tid == 0) dead = 0;
  auto word = [&](uint32_t entry) -> uint32_t {
    return tid < kOpWords ? reinterpret_cast<const uint32_t*>(P.ops + (entry & 0xffffu))[tid] : 0u;
  };
  uint32_t entry = first < last ? P.entries[first] : 0u, next = first + 1 < last ? P.entries[first + 1] : 0u;
  if (first < last && tid < kOpWords) reinterpret_cast<uint32_t*>(&ops[0])[tid] = word(entry);
  __syncthreads();
  for (int e = first; e < last; ++e) {
    const VmOp& q = ops[(e - first) & 1];
    const uint32_t ahead = e + 1 < last ? word(next) : 0u, after = e + 2 < last ? P.entries[e + 2] : 0u;
    if (tid < 32) {
      const unsigned need = lane < q.n_dep ? q.dep[lane < kMaxDeps ? lane : 0] : 0u;
      const unsigned* flag = P.done + (need & 0xffffu);
      bool ready = lane >= q.n_dep;
      const long long t0 = clock64();
      unsigned spins = 0;
      for (;;) {
        if (!ready) {
          unsigned v;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
          ready = v >= (need >> 16);
        }
        if (__all_sync(0xffffffffu, ready)) break;
        // Not at full rate for long: beside 146 CTAs that ask on, the loads of the two that sum 512 rows of 1000 take three times as long (228 us, 87 so)
        if (spins > 8u) __nanosleep(spins > 64u ? 200 : 40);
        if ((++spins & 255u) == 0u) {
          const bool over = clock64() - t0 > kVmWaitCycles || *reinterpret_cast<volatile int*>(P.err) != 0;
          if (__any_sync(0xffffffffu, over)) {
            if (lane == 0) { *reinterpret_cast<volatile int*>(P.err) = 1; dead = 1; }
            break;
          }
        }
      }
    }
    __syncthreads();
    if (dead) break;
    vm_run(q, (int)(entry >> 16), buf);
    if (tid < kOpWords) reinterpret_cast<uint32_t*>(&ops[(e + 1 - first) & 1])[tid] = ahead;
    __syncthreads();
    if (tid == 0) {
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.done + (entry & 0xffffu)) : "memory");
    }
    entry = next;
    next = after;
  }
  // the last CTA out empties the counters for the next replay
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    dead = atomicAdd(P.done + P.n_ops, 1u) == gridDim.x - 1 ? 2 : 0;
    __threadfence();
  }
  __syncthreads();
  if (dead == 2)
    for (int i = tid; i <= P.n_ops; i += kVmThreads) P.done[i] = 0u;
}

// ---------------------------------------------------------------------------------------------
// planning
// ---------------------------------------------------------------------------------------------
struct Range { uintptr_t lo, hi; };                       // bytes

// what a view reaches, or nothing if that lies outside its tensor or a 32-bit index
bool view_range(const StepView& v, Range* r) {
  int64_t far = v.offset;
  for (int k = 0; k < v.rank; ++k) {
    if (v.d[k] < 1 || v.st[k] < 0) return false;
    far += (v.d[k] - 1) * v.st[k];
  }
  if (!v.base || v.offset < 0 || far >= v.elems || far > 0x7fffffff) return false;
  r->lo = reinterpret_cast<uintptr_t>(v.base + v.offset);
  r->hi = reinterpret_cast<uintptr_t>(v.base + far + 1);
  return true;
}

bool same_axes(const StepView& v, int rank, const int64_t* d) {
  int k = 0;
  for (int j = 0; j < rank; ++j) {
    if (d[j] == 1) continue;
    while (k < v.rank && v.d[k] == 1) ++k;
    if (k >= v.rank || v.d[k] != d[j]) return false;
    ++k;
  }
  while (k < v.rank && v.d[k] == 1) ++k;
  return k == v.rank;
}

// the view `in` of a tensor that is itself the view `src` (axes alike but for those of one element): strides taken over axis by axis
StepView through(const StepView& in, const StepView& src) {
  StepView v = in;
  v.base = src.base; v.elems = src.elems; v.offset = src.offset;
  int k = 0;
  for (int j = 0; j < in.rank; ++j) {
    v.st[j] = 0;
    if (in.d[j] == 1) continue;
    while (src.d[k] == 1) ++k;
    v.st[j] = src.st[k++];
  }
  return v;
}

// column-major reshape of a view as a view, where the new axes split or join the old ones in place
bool reshape_view(const StepView& in, int rank, const int64_t* d, StepView* out) {
  int64_t od[kMaxRank], os[kMaxRank];
  int n = 0;
  for (int k = 0; k < in.rank; ++k)
    if (in.d[k] != 1) { od[n] = in.d[k]; os[n] = in.st[k]; ++n; }
  StepView v = in;
  v.rank = rank;
  int oi = 0, ni = 0;
  for (int k = 0; k < rank; ++k) { v.d[k] = d[k]; v.st[k] = 0; }
  while (oi < n && ni < rank) {
    int oj = oi + 1, nj = ni + 1;
    int64_t op = od[oi], np = d[ni];
    while (op != np) {
      if (np < op) { if (nj >= rank) return false; np *= d[nj++]; }
      else { if (oj >= n) return false; op *= od[oj++]; }
    }
    for (int k = oi; k + 1 < oj; ++k)                     // the joined axes must run on in column-major order
      if (os[k + 1] != os[k] * od[k]) return false;
    int64_t s = os[oi];
    for (int k = ni; k < nj; ++k) { v.st[k] = s; s *= d[k]; }
    oi = oj; ni = nj;
  }
  if (oi < n) return false;
  for (; ni < rank; ++ni)
    if (d[ni] != 1) return false;
  *out = v;
  return true;
}

int64_t elements(const RecordedStep& s) {
  int64_t t = 1;
  for (int k = 0; k < s.rank; ++k) t *= s.d[k];
  return t;
}

int64_t matmul_tiles(const RecordedStep& s, int cols) {
  int64_t b = 1;
  for (int k = 0; k + 2 < s.rank; ++k) b *= s.d[k];
  return b * ceil_div(s.d[s.rank - 2], 32) * ceil_div(s.d[s.rank - 1], cols);
}

// What a step takes, in microseconds: as the kernel it was recorded as, from one such kernel to the next, and a tile of it in vm_kernel beside the
// kHandOver of an entry (release, notice, the step's description).  From chains of 8 and of 24 steps of one kind replayed both ways, 170 kinds and
// sizes: within a quarter of most; among them (own | here) element-wise steps of 4096, 131072 and 520000 elements 1.5 | 1.4, 2.4 | 2.7 and 4.0 | 8.2 us; fusion
// groups of 41 instructions 6.0 | 6.1 at 4096, 25 | 82 at 520000; products of 1 x 1024 x 1024 18 | 7.3, 128 x 1024 x 1024 18.7 | 18.7, 4096 x 128 x 128
// 10 | 17; norms of 148 and of 2000 rows of 256 1.8 | 2.2 and 4.5 | 29; sums of 512 rows of 256 35 | 8.7, of 32000 rows of 64 10 | 24.
constexpr double kHandOver = 0.8, kVmLaunch = 6.0;
double own_us(const RecordedStep& s) {
  const double total = (double)elements(s), n = (double)s.n;
  switch (s.kind) {
    case STEP_RESHAPE: return 1.9 + total / 1.4e5;
    case STEP_FUSED: {
      const double k = (double)s.arg.size();
      return 1.6 + 0.11 * k + (total > 32768 ? 2.5 + 0.1 * k + total / 520e3 * (5.0 + 0.17 * k) : 0.0);
    }
    case STEP_REDUCE:                                      // (rows that start in the same bank of L1 are slower)
      return s.inner == 1 ? 1.6 + n * (0.0136 + (s.n % 32 ? 0.06 : 0.12) * std::min(total, 256.0) / 256.0) : 1.4 + 0.0155 * n;
    case STEP_MATMUL: {
      const double tiles = (double)matmul_tiles(s, 32);
      return 2.0 + 0.0165 * (double)s.in[0].d[s.in[0].rank - 1] * std::max(1.0, tiles / 148.0) + 0.006 * tiles;
    }
    case STEP_CUMSUM: return 1.2 + n * (0.043 + 0.055 * std::min(total / n, 16.0) / 16.0 + 0.06 * std::min(total / n, 256.0) / 256.0);
    case STEP_NORM: return 1.4 + 0.0008 * n + 0.0011 * total / n + (s.op ? 0.4 : 0.0);
    default: return 1.3 + total / 2e5;
  }
}

struct Tiling { int per; int64_t tiles; };                // elements a thread takes (REDUCE: rows a tile), and the step's tiles
// cols: columns of a product's tile; spread: other steps wait for this one, which then spreads over the CTAs (a movement nobody waits for takes eight
// elements a thread)
Tiling tiling(const RecordedStep& s, int sms, int cols, bool spread) {
  const int64_t total = elements(s);
  int per = 1;
  switch (s.kind) {
    case STEP_REDUCE:
      per = s.inner == 1 && s.n <= 256 ? 32 : 1;
      return {per, ceil_div(total, per == 32 ? 32 : kVmThreads)};
    case STEP_MATMUL: return {1, matmul_tiles(s, cols)};
    case STEP_CUMSUM: return {1, ceil_div(total / s.n, kVmThreads)};
    case STEP_NORM: return {1, total / s.n};
    default:
      while (per < 8 && (!spread || ceil_div(total, kVmThreads * per) > sms)) per *= 2;
      return {per, ceil_div(total, kVmThreads * per)};
  }
}
double tile_us(const RecordedStep& s, const Tiling& t, int cols) {
  const double n = (double)s.n, per = t.per;
  switch (s.kind) {
    case STEP_COPY: return 0.4 + 0.15 * per;
    case STEP_RESHAPE: return 1.1 + 0.15 * per;
    case STEP_FUSED: return 0.5 + per * (0.2 + 0.12 * (double)s.arg.size());
    case STEP_REDUCE: return t.per == 32 ? 1.5 + 0.027 * n : 0.9 + 0.023 * n;
    case STEP_MATMUL: {
      const double K = (double)s.in[0].d[s.in[0].rank - 1];
      return cols == 8 ? 1.0 + 0.0055 * K : cols == 16 ? 1.0 + 0.009 * K : 1.8 + 0.0162 * K;
    }
    case STEP_CUMSUM: {
      const double rows = std::min((double)elements(s) / n, 256.0);
      return 1.5 + n * (0.0166 + 0.02 * std::min(rows, 16.0) / 16.0 + (rows > 64.0 ? 0.22 : 0.03) * rows / (rows > 64.0 ? 256.0 : 64.0));
    }
    case STEP_NORM: return 1.1 + 0.0009 * n + (s.op ? 0.35 : 0.0);
    default: return 0.35 + 0.4 * per;
  }
}
// columns of a product's tile: the fewest with which it takes one round of the CTAs
int product_cols(const RecordedStep& s, int sms) {
  int cols = 8;
  while (cols < 32 && matmul_tiles(s, cols) > sms) cols *= 2;
  return cols;
}

// A step that takes kOwnGain longer here than by its own kernel keeps that kernel.  That ends the vm_kernel in front of it and everything in that has to be
// done by then, and starts another behind: 30 us for each of three such steps of a 128-token graph of hidden 1024 (907 us a replay, 857 with them inside).
// Rows beyond 256 elements are summed by a thread each: as fast as the own kernel while nothing else runs, but its loads want the L1 that vm_kernel's shared
// memory takes (sums of 16 rows of 4096 with a broadcast add between them 107 us, 227 here).  Movements, which nobody waits for, are only bounded in size: half
// a million elements.
constexpr double kOwnGain = 16.0;
constexpr int64_t kOwnElements = 1 << 19;
bool own_kernel(const RecordedStep& s, int sms) {
  if (elements(s) > kOwnElements || s.n > 0x7fffffff) return true;
  for (const StepView& v : s.in)
    if (v.base && v.elems > 0x7fffffff) return true;
  if (s.kind == STEP_COPY) return false;
  const int cols = s.kind == STEP_MATMUL ? product_cols(s, sms) : 0;
  const Tiling t = tiling(s, sms, cols, true);
  if (t.tiles > 65535 || (s.kind == STEP_REDUCE && s.n > 256)) return true;
  return (double)ceil_div(t.tiles, sms) * (kHandOver + tile_us(s, t, cols)) > own_us(s) + kOwnGain;
}

struct Planned {
  RecordedStep* s;
  bool own = false;                    // runs as the kernel it was recorded as
  bool is_view = false;                // its output is `view` (of a source that others may read instead)
  bool redirected = false;             // reads a movement's source in the place of its output, which the recorded kernel names: it can only run in a vm_kernel
  StepView view;
  Range write;
  std::vector<Range> reads;
  std::vector<StepView> in;            // as it is run
  int stage = 0, level = 0;            // even stages: one vm_kernel each; odd ones: kernels in order
  std::vector<int> after;              // steps of the same stage it waits for
};

// A product's operand as (batch, batch, row, column) strides: leading axes of the view are the batches.
bool operand_strides(const StepView& v, int64_t st[4], int64_t b[2]) {
  if (v.rank < 2 || v.rank > 4) return false;
  for (int k = 0; k < 2; ++k) { st[k] = 0; b[k] = 1; }
  for (int k = 0; k + 2 < v.rank; ++k) {
    st[k + 4 - v.rank] = v.st[k];
    b[k + 4 - v.rank] = v.d[k];
  }
  st[2] = v.st[v.rank - 2];
  st[3] = v.st[v.rank - 1];
  return true;
}

// tensors the recorded calls name, cut into pieces that are written and read as wholes
struct Memory {
  std::vector<uintptr_t> cut;
  struct Piece { int writer = -1; std::vector<int> readers; };
  std::vector<Piece> piece;
  void build(const std::vector<Planned>& plan) {
    for (const Planned& p : plan) {
      cut.push_back(p.write.lo); cut.push_back(p.write.hi);
      for (const StepView& v : p.s->in)
        if (v.base) { cut.push_back(reinterpret_cast<uintptr_t>(v.base)); cut.push_back(reinterpret_cast<uintptr_t>(v.base + v.elems)); }
    }
    std::sort(cut.begin(), cut.end());
    cut.erase(std::unique(cut.begin(), cut.end()), cut.end());
    piece.assign(cut.size(), Piece());
  }
  template <typename F> void over(const Range& r, F f) {
    size_t i = std::upper_bound(cut.begin(), cut.end(), r.lo) - cut.begin() - 1;
    for (; i < cut.size() && cut[i] < r.hi; ++i) f(piece[i]);
  }
  int last_writer(const Range& r) {
    int w = -1;
    over(r, [&](Piece& p) { w = std::max(w, p.writer); });
    return w;
  }
};

// Views, stages and dependencies of a run of steps.  false: a step cannot be described.
bool plan_steps(std::vector<Planned>& plan, int sms) {
  for (Planned& p : plan) {
    const RecordedStep& s = *p.s;
    const int64_t total = elements(s);
    p.write = {reinterpret_cast<uintptr_t>(s.out), reinterpret_cast<uintptr_t>(s.out + total)};
    p.own = own_kernel(s, sms);
  }
  Memory mem;
  mem.build(plan);
  std::vector<int> dep;
  for (size_t i = 0; i < plan.size(); ++i) {
    Planned& p = plan[i];
    const RecordedStep& s = *p.s;
    p.in = s.in;
    if (!p.own && s.kind != STEP_REDUCE && s.kind != STEP_GATHER && s.kind != STEP_CUMSUM && s.kind != STEP_NORM) {
      for (StepView& v : p.in) {
        Range r;
        const StepView whole = v;
        if (!view_range(v, &r)) return false;
        const int j = mem.last_writer(r);
        if (j < 0 || !plan[j].is_view || plan[j].s->out != v.base || elements(*plan[j].s) != v.elems) continue;
        // the call sees the tensor as a row-major one (a movement's own axes come on top of it, below)
        const StepView& src = plan[j].view;
        Range rs;
        if (!same_axes(v, src.rank, src.d) || !view_range(src, &rs)) continue;
        if (mem.last_writer(rs) >= j) continue;           // the source has been written over since
        StepView t = through(whole, src);
        if (s.kind == STEP_MATMUL) {                      // a product reads one operand's axis contiguously or not at all through views
          const int64_t a = t.st[t.rank - 1], c = t.st[t.rank - 2];
          if (a != 1 && c != 1) continue;
          if (&v == &p.in[0] && a != 1) continue;
        }
        v = t;
        p.redirected = true;
      }
    }
    // a movement step is a view of what it reads
    if (s.kind == STEP_COPY) {
      StepView v;
      v.base = p.in[0].base; v.elems = p.in[0].elems; v.offset = p.in[0].offset;
      v.rank = s.rank;
      for (int k = 0; k < p.in[0].rank; ++k) v.offset += (int64_t)s.arg[kMaxRank + k] * p.in[0].st[k];
      for (int k = 0; k < s.rank; ++k) { v.d[k] = s.d[k]; v.st[k] = s.arg[k] ? p.in[0].st[s.arg[k] - 1] : 0; }
      Range r;
      if (!view_range(v, &r)) return false;
      p.view = v;
      p.is_view = true;
    } else if (s.kind == STEP_RESHAPE) {
      Range r;
      p.is_view = reshape_view(p.in[0], s.rank, s.d, &p.view) && view_range(p.view, &r);
    }
    const StepView* reads = p.is_view ? &p.view : p.in.data();
    for (const StepView* v = reads; v != reads + (p.is_view ? 1 : p.in.size()); ++v) {
      if (!v->base) continue;
      Range r;
      if (!view_range(*v, &r)) return false;
      if (r.lo < p.write.hi && p.write.lo < r.hi) return false;                   // in place: order within a step is the kernel's
      p.reads.push_back(r);
    }
    // dependencies
    dep.clear();
    for (const Range& r : p.reads)
      mem.over(r, [&](Memory::Piece& c) { if (c.writer >= 0) dep.push_back(c.writer); });
    mem.over(p.write, [&](Memory::Piece& c) {
      if (c.writer >= 0) dep.push_back(c.writer);
      dep.insert(dep.end(), c.readers.begin(), c.readers.end());
    });
    std::sort(dep.begin(), dep.end());
    dep.erase(std::unique(dep.begin(), dep.end()), dep.end());
    p.stage = p.own ? 1 : 0;
    for (int j : dep) p.stage = std::max(p.stage, plan[j].stage + ((plan[j].stage & 1) != (p.own ? 1 : 0)));
    for (int j : dep)
      if (plan[j].stage == p.stage && !p.own) { p.after.push_back(j); p.level = std::max(p.level, plan[j].level + 1); }
    // (steps of other stages are done or not begun when this stage's kernel runs)
    for (const Range& r : p.reads) mem.over(r, [&](Memory::Piece& c) { c.readers.push_back((int)i); });
    mem.over(p.write, [&](Memory::Piece& c) { c.writer = (int)i; c.readers.clear(); });
  }
  return true;
}

bool fits(int64_t v) { return v >= 0 && v <= 0x7fffffff; }

// Output axes and the inputs' strides over them with axes of one element dropped and axes that every operand runs through in one go joined.
void set_axes(VmOp* q, int rank, const int64_t* d, size_t n_in, const int64_t (*st)[kMaxRank]) {
  int64_t od[kMaxRank], os[8][kMaxRank];
  int n = 0;
  for (int k = 0; k < rank; ++k) {
    if (d[k] == 1) continue;
    bool join = n > 0;
    for (size_t i = 0; i < n_in && join; ++i) join = os[i][n - 1] == st[i][k] * d[k];
    if (join) {
      od[n - 1] *= d[k];
      for (size_t i = 0; i < n_in; ++i) os[i][n - 1] = st[i][k];
    } else {
      od[n] = d[k];
      for (size_t i = 0; i < n_in; ++i) os[i][n] = st[i][k];
      ++n;
    }
  }
  q->rank = n;
  for (int k = 0; k < n; ++k) {
    q->d[k] = (uint32_t)od[k];
    const FastDiv f = fast_div((uint32_t)od[k]);
    q->mul[k] = f.mul; q->shift[k] = (uint8_t)f.shift;
    for (size_t i = 0; i < n_in; ++i) q->st[i][k] = (int)os[i][k];
  }
}

// strides of a view broadcast against the output (1-dims prepended); checked by the call itself
void broadcast(const StepView& v, int rank, const int64_t* d, int64_t* st) {
  const int shift = rank - v.rank;
  for (int k = 0; k < rank; ++k) st[k] = k >= shift && v.d[k - shift] == d[k] && v.d[k - shift] != 1 ? v.st[k - shift] : 0;
}

// Fills the kernel's form of a step; returns its tiles, 0 if it has none.  cols: columns of a product's tile
int64_t encode(const Planned& p, const Tiling& t, int cols, VmOp* q) {
  const RecordedStep& s = *p.s;
  memset(q, 0, sizeof(*q));
  const int64_t total = elements(s);
  q->kind = s.kind; q->op = s.op; q->out = s.out;
  q->n_in = (int)p.in.size();
  q->total = (int)total;
  q->per = t.per;
  for (size_t i = 0; i < p.in.size(); ++i) q->in[i] = p.in[i].base ? p.in[i].base + p.in[i].offset : nullptr;
  switch (s.kind) {
    case STEP_EW:
    case STEP_SILU:
    case STEP_FUSED: {
      int64_t st[kFusedMaxInputs][kMaxRank];
      for (size_t i = 0; i < p.in.size(); ++i) broadcast(p.in[i], s.rank, s.d, st[i]);
      set_axes(q, s.rank, s.d, p.in.size(), st);
      if (s.kind == STEP_FUSED) {
        q->n_instr = (int)s.arg.size();
        for (size_t i = 0; i < s.arg.size(); ++i) { q->code[i] = (uint8_t)s.arg[i]; q->arg[i] = s.val[i]; }
      }
      break;
    }
    case STEP_COPY:
    case STEP_RESHAPE:
      if (p.is_view) {
        q->kind = STEP_COPY; q->n_in = 1;
        q->in[0] = p.view.base + p.view.offset;
        set_axes(q, p.view.rank, p.view.d, 1, &p.view.st);
        break;
      }
      [[fallthrough]];
    case STEP_PAD: {
      q->rank = s.rank;
      int64_t mul = 1;
      for (int k = 0; k < s.rank; ++k) {
        q->d[k] = (uint32_t)s.d[k];
        const FastDiv f = fast_div(q->d[k]);
        q->mul[k] = f.mul; q->shift[k] = (uint8_t)f.shift;
        q->st[4][k] = (int)mul;
        mul *= s.d[k];
      }
      const StepView& v = p.in[0];
      q->p[0] = v.rank;
      for (int k = 0; k < v.rank; ++k) {
        q->st[0][k] = (int)v.st[k];
        if (s.kind == STEP_PAD) { q->st[1][k] = s.arg[k]; q->st[2][k] = (int)v.d[k]; continue; }
        const FastDiv f = fast_div((uint32_t)v.d[k]);
        q->st[1][k] = (int)v.d[k]; q->st[2][k] = (int)f.mul; q->st[3][k] = f.shift;
      }
      break;
    }
    case STEP_REDUCE:
      q->p[0] = (int)s.n; q->p[1] = (int)s.inner;
      break;
    case STEP_MATMUL: {
      int64_t sa[4], sb[4], ba[2], bb[2];
      if (!operand_strides(p.in[0], sa, ba) || !operand_strides(p.in[1], sb, bb)) return 0;
      for (int k = 0; k < 4; ++k) {
        if (!fits(sa[k]) || !fits(sb[k])) return 0;
        q->st[0][k] = (int)sa[k]; q->st[1][k] = (int)sb[k];
      }
      q->op = cols;
      q->p[0] = (int)s.d[s.rank - 2]; q->p[1] = (int)s.d[s.rank - 1]; q->p[2] = (int)p.in[0].d[p.in[0].rank - 1];
      q->p[3] = (int)ceil_div(q->p[1], cols); q->p[4] = (int)ceil_div(q->p[0], 32); q->p[5] = (int)ba[1];
      // four k at a time where every row starts on 16 bytes
      const auto vec = [&](const float* base, const int64_t* st, int row) {
        return q->p[2] % 4 == 0 && reinterpret_cast<uintptr_t>(base) % 16 == 0 && (st[0] | st[1] | st[row]) % 4 == 0 && st[5 - row] == 1;
      };
      q->p[6] = (vec(q->in[0], sa, 2) ? 1 : 0) | (vec(q->in[1], sb, 3) ? 2 : 0);
      break;
    }
    case STEP_GATHER:
      q->p[0] = (int)s.inner; q->p[1] = (int)s.n;
      break;
    case STEP_CUMSUM:
      q->total = (int)(total / s.n);
      q->p[0] = (int)s.n;
      break;
    case STEP_NORM:
      q->p[0] = (int)s.n; q->f = s.val[0];
      break;
  }
  return t.tiles;
}

// One vm_kernel: the steps of a stage, their tiles dealt to the CTAs.  An entry only waits for entries of lower levels, and every CTA's list ascends in
// levels, so all waits end.  The steps on a longest chain take their earliest level and the CTAs from 0 on; the tiles of the others go, level by level, to CTAs
// that have nothing to do then and in the next level, so that they delay nobody.
struct Program {
  std::vector<VmOp> ops;
  std::vector<uint32_t> entries;
  std::vector<int> first;
  std::vector<int64_t> tiles;
  std::vector<int> limit;                                                // the last level each step may take: before the first that waits for it
  int levels = 0;
  double us = 0.0;                                                       // what a replay of it takes: own_us's measurements
};

// Everything but the entries; false: a step cannot be described.
bool describe_program(const std::vector<Planned>& plan, const std::vector<int>& steps, int sms, Program* out) {
  const int n = (int)steps.size();
  if (n > 65535) return false;
  std::vector<int> index(plan.size(), -1);
  for (int i = 0; i < n; ++i) index[steps[i]] = i;
  int levels = 0;
  for (int i : steps) levels = std::max(levels, plan[i].level + 1);
  out->levels = levels;
  std::vector<int>& limit = out->limit;
  limit.assign(n, levels - 1);
  std::vector<bool> waited_for(n, false);
  for (int i = n - 1; i >= 0; --i)
    for (int j : plan[steps[i]].after) {
      limit[index[j]] = std::min(limit[index[j]], limit[i] - 1);
      waited_for[index[j]] = true;
    }
  // columns of a level's product tiles: the fewest with which its products take one round of the CTAs
  std::vector<int64_t> product(3 * levels, 0);
  for (int i : steps)
    if (plan[i].s->kind == STEP_MATMUL)
      for (int c = 0; c < 3; ++c) product[3 * plan[i].level + c] += matmul_tiles(*plan[i].s, 8 << c);
  std::vector<int64_t>& tiles = out->tiles;
  tiles.resize(n);
  // a level takes its longest entry as often as its chain's tiles go round the CTAs; the other tiles lie beside them on all CTAs
  std::vector<int64_t> chain_tiles(levels, 0);
  std::vector<double> longest(levels, 0.0);
  double chain_us = 0.0, rest_us = 0.0;
  out->ops.resize(n);
  for (int i = 0; i < n; ++i) {
    const Planned& p = plan[steps[i]];
    int c = 0;
    while (c < 2 && product[3 * p.level + c] > sms) ++c;
    const Tiling t = tiling(*p.s, sms, 8 << c, waited_for[i]);
    tiles[i] = encode(p, t, 8 << c, &out->ops[i]);
    if (tiles[i] < 1 || tiles[i] > 65535 || (int)p.after.size() > kMaxDeps) return false;
    const double us = kHandOver + tile_us(*p.s, t, 8 << c);
    if (limit[i] == p.level) {
      chain_tiles[p.level] += t.tiles;
      longest[p.level] = std::max(longest[p.level], us);
    } else {
      rest_us += us * (double)t.tiles / sms;
    }
  }
  for (int l = 0; l < levels; ++l) chain_us += longest[l] * (double)ceil_div(chain_tiles[l], sms);
  out->us = kVmLaunch + chain_us + rest_us;
  for (int i = 0; i < n; ++i) {
    const Planned& p = plan[steps[i]];
    out->ops[i].n_dep = (int)p.after.size();
    for (size_t k = 0; k < p.after.size(); ++k) out->ops[i].dep[k] = (uint32_t)index[p.after[k]] | (uint32_t)(tiles[index[p.after[k]]] << 16);
  }
  return true;
}

// Deals the tiles to the CTAs.
void place_program(const std::vector<Planned>& plan, const std::vector<int>& steps, int sms, Program* out) {
  const int n = (int)steps.size(), levels = out->levels;
  const std::vector<int64_t>& tiles = out->tiles;
  const std::vector<int>& limit = out->limit;
  std::vector<int> index(plan.size(), -1);
  for (int i = 0; i < n; ++i) index[steps[i]] = i;
  struct Place { int cta, level; uint32_t entry; };
  std::vector<Place> places;
  std::vector<int> used(levels + 1, 0);                                  // CTAs the chain's steps take in a level
  std::vector<int> at(n, -1);
  for (int i = 0; i < n; ++i) {
    const int l = plan[steps[i]].level;
    if (limit[i] != l) continue;
    at[i] = l;
    for (int64_t t = 0; t < tiles[i]; ++t) places.push_back({(int)((used[l] + t) % sms), l, (uint32_t)i | (uint32_t)t << 16});
    used[l] += (int)std::min<int64_t>(tiles[i], 1 << 20);
  }
  // the others, those with the least slack first; a step's tiles all lie behind what it waits for and before what waits for it
  std::vector<int> rest;
  for (int i = 0; i < n; ++i)
    if (at[i] < 0) rest.push_back(i);
  std::vector<int> taken(levels, 0);                                     // tiles of such steps in a level so far, from the last CTA down
  std::stable_sort(rest.begin(), rest.end(), [&](int a, int b) { return limit[a] < limit[b]; });
  for (int i : rest) {
    int lo = plan[steps[i]].level;
    for (int j : plan[steps[i]].after) lo = std::max(lo, at[index[j]] + 1);
    int l = lo, last = lo;
    for (int64_t t = 0; t < tiles[i]; ++t) {
      const auto room = [&](int k) { return sms - std::max(std::min(used[k], sms), std::min(used[k + 1], sms)) - taken[k]; };
      while (l < limit[i] && room(l) <= 0) ++l;
      if (room(l) <= 0) l = lo + (int)(t % (limit[i] - lo + 1));         // none left: spread over them
      places.push_back({sms - 1 - taken[l] % sms, l, (uint32_t)i | (uint32_t)t << 16});
      ++taken[l];
      last = std::max(last, l);
    }
    at[i] = last;
  }
  // by CTA, then level
  std::vector<int> from((size_t)sms * levels + 1, 0);
  for (const Place& p : places) ++from[(size_t)p.cta * levels + p.level + 1];
  for (size_t k = 1; k < from.size(); ++k) from[k] += from[k - 1];
  for (int c = 0; c <= sms; ++c) out->first.push_back(from[(size_t)c * levels]);
  out->entries.resize(places.size());
  for (const Place& p : places) out->entries[from[(size_t)p.cta * levels + p.level]++] = p.entry;
}

struct Recorder {
  std::vector<RecordedStep> steps;
};

// Programs in device memory, one allocation for all of a graph's: steps | entries | first | counters of each in turn.
struct Image {
  std::vector<char> host;
  std::vector<VmParams> at;                                // pointers as offsets until place()
  void add(Ctx* ctx, const Program& pg) {
    const size_t a = pg.ops.size() * sizeof(VmOp), b = round_up(pg.entries.size() * 4, 16), c = round_up(pg.first.size() * 4, 16), d = round_up((pg.ops.size() + 1) * 4, 16);
    const size_t o = host.size();
    host.resize(o + a + b + c + d, 0);
    memcpy(host.data() + o, pg.ops.data(), a);
    memcpy(host.data() + o + a, pg.entries.data(), pg.entries.size() * 4);
    memcpy(host.data() + o + a + b, pg.first.data(), pg.first.size() * 4);
    VmParams vp;
    vp.ops = reinterpret_cast<const VmOp*>(o);
    vp.entries = reinterpret_cast<const uint32_t*>(o + a);
    vp.first = reinterpret_cast<const int*>(o + a + b);
    vp.done = reinterpret_cast<unsigned*>(o + a + b + c);
    vp.n_ops = (int)pg.ops.size();
    vp.err = ctx->dev_err;
    at.push_back(vp);
  }
  // false: no device memory; *mem is the caller's to free
  bool place(Ctx* ctx, void** mem) {
    if (cudaMalloc(mem, host.size()) != cudaSuccess) { *mem = nullptr; return false; }
    if (cudaMemcpyAsync(*mem, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->own_stream) != cudaSuccess || cudaStreamSynchronize(ctx->own_stream) != cudaSuccess) return false;
    const uintptr_t base = reinterpret_cast<uintptr_t>(*mem);
    for (VmParams& v : at) {
      v.ops = reinterpret_cast<const VmOp*>(base + reinterpret_cast<uintptr_t>(v.ops));
      v.entries = reinterpret_cast<const uint32_t*>(base + reinterpret_cast<uintptr_t>(v.entries));
      v.first = reinterpret_cast<const int*>(base + reinterpret_cast<uintptr_t>(v.first));
      v.done = reinterpret_cast<unsigned*>(base + reinterpret_cast<uintptr_t>(v.done));
    }
    return true;
  }
};

// A run shorter than this is not looked at: the kernel's launch alone takes as long as four of the shortest steps.
constexpr size_t kShortestRun = 6;

// a recorded kernel as it is, behind *prev (the attributes' copy takes the destination first, whatever the header calls its arguments: read back on both nodes)
bool append_kernel(cudaGraph_t graph, cudaGraphNode_t* prev, cudaGraphNode_t recorded, int64_t* kernels) {
  cudaKernelNodeParams kp{};
  cudaGraphNode_t node = nullptr;
  if (cudaGraphKernelNodeGetParams(recorded, &kp) != cudaSuccess) return false;
  if (cudaGraphAddKernelNode(&node, graph, *prev ? prev : nullptr, *prev ? 1 : 0, &kp) != cudaSuccess) return false;
  if (cudaGraphKernelNodeCopyAttributes(node, recorded) != cudaSuccess) return false;
  *prev = node;
  ++*kernels;
  return true;
}

// A new graph is planned, uploaded and rebuilt once: 0.1 to 0.3 ms of its first call, and the estimates are a tenth off.
constexpr double kWorthIt = 0.92;

// A run of steps as stages: a program of vm_kernel each, or (programs without steps) the recorded kernels.
struct Run {
  std::vector<Planned> plan;
  std::vector<std::vector<int>> of;    // a stage's steps
  std::vector<Program> pg;
};

// false: the run gains nothing from being replaced.
bool plan_run(Ctx* ctx, RecordedStep* steps, size_t n, Run* run) {
  const char* e = getenv("LMB200_GRAPH_KERNEL");           // 0: recorded kernels only, 1: vm_kernel wherever it can be (A/B runs)
  if (e && atoi(e) == 0) return false;
  std::vector<Planned>& plan = run->plan;
  plan.resize(n);
  for (size_t i = 0; i < n; ++i) plan[i].s = &steps[i];
  if (!plan_steps(plan, ctx->sm_count)) return false;
  int stages = 0;
  for (const Planned& p : plan) stages = std::max(stages, p.stage + 1);
  run->of.resize(stages);
  for (size_t i = 0; i < n; ++i) run->of[plan[i].stage].push_back((int)i);
  run->pg.resize(stages);
  double recorded = 0.0, planned = 0.0;
  bool any = false;
  for (int s = 0; s < stages; ++s) {
    double own = 0.0;
    bool redirected = false;
    for (int i : run->of[s]) { own += own_us(steps[i]); redirected = redirected || plan[i].redirected; }
    recorded += own;
    Program& pg = run->pg[s];
    if (s % 2 == 0 && !run->of[s].empty() && !describe_program(plan, run->of[s], ctx->sm_count, &pg)) return false;
    // A stage that is faster as its own kernels runs as those, unless a step reads past a movement: it then waits for the movement's source only and may stand
    // in front of the movement, whose output its recorded kernel would read.
    if (!pg.ops.empty() && pg.us >= own && !redirected && !e) pg = Program();
    planned += pg.ops.empty() ? own : pg.us;
    any = any || !pg.ops.empty();
  }
  if (!any || (!e && planned >= kWorthIt * recorded)) return false;
  for (int s = 0; s < stages; ++s)
    if (!run->pg[s].ops.empty()) place_program(plan, run->of[s], ctx->sm_count, &run->pg[s]);
  return true;
}

// Appends it to `graph` behind *prev, *vp its first program; false: the graph is no longer usable.
bool append_run(Ctx* ctx, cudaGraph_t graph, cudaGraphNode_t* prev, const Run& run, VmParams** vp, int64_t* kernels) {
  for (size_t s = 0; s < run.of.size(); ++s) {
    if (run.pg[s].ops.empty()) {
      for (int i : run.of[s])
        if (!append_kernel(graph, prev, run.plan[i].s->node, kernels)) return false;
      continue;
    }
    cudaKernelNodeParams kp{};
    void* args[1] = {(*vp)++};
    kp.func = (void*)vm_kernel;
    kp.gridDim = dim3((unsigned)ctx->sm_count);
    kp.blockDim = dim3(kVmThreads);
    kp.sharedMemBytes = kBufFloats * 4;
    kp.kernelParams = args;
    cudaGraphNode_t node = nullptr;
    if (cudaGraphAddKernelNode(&node, graph, *prev ? prev : nullptr, *prev ? 1 : 0, &kp) != cudaSuccess) return false;
    cudaKernelNodeAttrValue coop{};
    coop.cooperative = 1;
    if (cudaGraphKernelNodeSetAttribute(node, cudaKernelNodeAttributeCooperative, &coop) != cudaSuccess) return false;
    *prev = node;
    ++*kernels;
  }
  return true;
}

// The chain's kernels in order; false if the graph is anything but a chain of kernels.
bool chain_of(cudaGraph_t graph, const std::vector<RecordedStep>& steps, std::vector<cudaGraphNode_t>* chain) {
  size_t roots = 0, total = 0;
  if (cudaGraphGetRootNodes(graph, nullptr, &roots) != cudaSuccess || roots != 1) return false;
  if (cudaGraphGetNodes(graph, nullptr, &total) != cudaSuccess) return false;
  if (total == steps.size()) {                             // one stream's launches, each recorded as the only thing the next depends on
    for (const RecordedStep& s : steps) chain->push_back(s.node);
    return true;
  }
  cudaGraphNode_t at = nullptr;
  if (cudaGraphGetRootNodes(graph, &at, &roots) != cudaSuccess) return false;
  for (;;) {
    cudaGraphNodeType type;
    if (cudaGraphNodeGetType(at, &type) != cudaSuccess || type != cudaGraphNodeTypeKernel) return false;
    chain->push_back(at);
    cudaGraphNode_t behind[2] = {};
    cudaGraphEdgeData edge[2] = {};
    size_t n = 2;
    if (cudaGraphNodeGetDependentNodes_v2(at, behind, edge, &n) != cudaSuccess) return false;
    if (n == 0) break;
    if (behind[1]) return false;
    at = behind[0];
  }
  return chain->size() == total;
}

}  // namespace

void record_begin(Ctx* ctx) { ctx->recorder = new Recorder(); }

void record_drop(Ctx* ctx) {
  delete static_cast<Recorder*>(ctx->recorder);
  ctx->recorder = nullptr;
}

void record_step(Ctx* ctx, RecordedStep&& s) {
  Recorder* r = static_cast<Recorder*>(ctx->recorder);
  if (!r) return;
  cudaStreamCaptureStatus status;
  const cudaGraphNode_t* deps = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t n = 0;
  if (cudaStreamGetCaptureInfo_v3(ctx->stream, &status, nullptr, nullptr, &deps, &edges, &n) == cudaSuccess && status == cudaStreamCaptureStatusActive && n == 1) {
    s.node = deps[0];
    r->steps.push_back(std::move(s));
  } else {
    cudaGetLastError();
  }
}

void record_finish(Ctx* ctx, cudaGraph_t* graph, std::vector<void*>* programs, int64_t* kernels) {
  Recorder* r = static_cast<Recorder*>(ctx->recorder);
  if (!r) return;
  std::vector<RecordedStep> steps = std::move(r->steps);
  record_drop(ctx);
  if (steps.size() < kShortestRun) return;
  std::vector<cudaGraphNode_t> chain;
  if (!chain_of(*graph, steps, &chain)) {
    cudaGetLastError();
    return;
  }
  struct Piece { size_t at, n; bool replaced; };           // kernels of the chain
  std::vector<Piece> pieces;
  std::vector<Run> runs;
  for (size_t c = 0, i = 0; c < chain.size();) {
    size_t n = 0;                                          // recorded steps from this node of the chain on
    while (i + n < steps.size() && c + n < chain.size() && steps[i + n].node == chain[c + n]) ++n;
    Run run;
    const bool replaced = n >= kShortestRun && plan_run(ctx, &steps[i], n, &run);
    if (replaced) runs.push_back(std::move(run));
    i += n;
    if (n == 0) n = 1;
    pieces.push_back({c, n, replaced});
    c += n;
  }
  if (runs.empty()) return;
  cudaGraph_t made = nullptr;
  cudaGraphNode_t prev = nullptr;
  void* mem = nullptr;
  int64_t count = 0;
  Image image;
  for (const Run& r : runs)
    for (const Program& pg : r.pg)
      if (!pg.ops.empty()) image.add(ctx, pg);
  bool ok = image.place(ctx, &mem) && cudaFuncSetAttribute(vm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBufFloats * 4) == cudaSuccess &&
            cudaGraphCreate(&made, 0) == cudaSuccess;
  size_t next = 0;
  VmParams* vp = image.at.data();
  for (const Piece& p : pieces) {
    if (ok && p.replaced) ok = append_run(ctx, made, &prev, runs[next++], &vp, &count);
    for (size_t k = p.at; ok && !p.replaced && k < p.at + p.n; ++k) ok = append_kernel(made, &prev, chain[k], &count);
  }
  cudaGetLastError();
  if (ok) {
    cudaGraphDestroy(*graph);
    *graph = made;
    *kernels = count;
    programs->push_back(mem);
  } else {                                                 // as recorded, then
    cudaFree(mem);
    if (made) cudaGraphDestroy(made);
  }
}

}  // namespace lmb
