// Primitive graph ops on float32 row-major device tensors: what the reference's execute_op!
// dispatches to, one call per node (src/Execution.jl:216-371, 580-618), plus the stand-alone
// forms of the fused layer ops.  These are the op-by-op path of execute() on the B200 device;
// the decode session does not go through them.
#include <math.h>

#include "common.cuh"
#include "pdl.cuh"
#include "recorded.cuh"

namespace lmb {
namespace {

// A traced graph is a chain of hundreds of these, most of a microsecond's work, so what counts is the time from one to the next.  Kernels with a
// short thread per output element are launched programmatically (each waits for its predecessor before it touches memory).  The others, whose
// CTAs work for a while -- products, reductions, scans, norms -- start in plain order: CTAs that become resident early pile up on the SMs that
// were free first, and the kernel is as slow as the fullest of them (sums of 65536 rows of 1024: 274 us in plain order, 366 otherwise; scans 700 and
// 1050).  Index arithmetic is 32-bit (I = uint32_t) wherever the element counts allow: a 64-bit division is a subroutine of about a hundred instructions.
// The small Llama's 32-token graph as 404 kernels, per call: 1431 -> 985 us with the
// matmul below (1126 with all of them programmatic); recorded graphs run such steps as one kernel (recorded.cu).
constexpr float kHalfPi = 1.5707963267948966f;

struct Idx {
  int rank;
  int64_t out_d[kMaxRank];
  int64_t sa[kMaxRank], sb[kMaxRank], sc[kMaxRank];   // operand strides (0 = broadcast)
};

template <typename I>
__global__ void ew_kernel(int op, float* out, const float* a, const float* b, const float* c, Idx ix, int64_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (I o = blockIdx.x * (I)blockDim.x + threadIdx.x; o < (I)total; o += (I)gridDim.x * blockDim.x) {
    I rem = o;
    int64_t oa = 0, ob = 0, oc = 0;
    for (int k = ix.rank - 1; k >= 0; --k) {
      const I d = (I)ix.out_d[k], nx = rem / d, i = rem - nx * d;
      rem = nx;
      oa += i * ix.sa[k]; ob += i * ix.sb[k]; oc += i * ix.sc[k];
    }
    out[o] = apply_op(op, a ? a[oa] : 0.f, b ? b[ob] : 0.f, c ? c[oc] : 0.f);
  }
}

// One element-wise fusion group per launch: a postfix program over up to 8 broadcast inputs,
// interpreted per output element with every operation rounded to float32 on its own (no
// contraction), so the result equals running the group's nodes one by one.
// Stands in for FusedElementwiseOp (src/Compiler.jl:323-357, executor src/Execution.jl:552-563).
struct FusedProgram {
  int n_in, n_instr, rank;
  int64_t out_d[kMaxRank];
  int64_t st[kFusedMaxInputs][kMaxRank];      // input strides over the output's axes (0 = broadcast)
  const float* in[kFusedMaxInputs];
  int op[kFusedMaxInstr];
  float arg[kFusedMaxInstr];                  // PUSH_IN: input index; PUSH_CONST: the value
};
template <typename I>
__global__ void fused_ew_kernel(float* out, const FusedProgram pg, int64_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (I o = blockIdx.x * (I)blockDim.x + threadIdx.x; o < (I)total; o += (I)gridDim.x * blockDim.x) {
    int64_t off[kFusedMaxInputs];
#pragma unroll
    for (int i = 0; i < kFusedMaxInputs; ++i) off[i] = 0;
    I rem = o;
    for (int k = pg.rank - 1; k >= 0; --k) {
      const I d = (I)pg.out_d[k], nx = rem / d, idx = rem - nx * d;
      rem = nx;
#pragma unroll
      for (int i = 0; i < kFusedMaxInputs; ++i)
        if (i < pg.n_in) off[i] += idx * pg.st[i][k];
    }
    float stack[kFusedMaxStack];
    int sp = 0;
    for (int pc = 0; pc < pg.n_instr; ++pc) {
      const int op = pg.op[pc];
      if (op == F_PUSH_IN) { const int i = (int)pg.arg[pc]; stack[sp++] = pg.in[i][off[i]]; continue; }
      if (op == F_PUSH_CONST) { stack[sp++] = pg.arg[pc]; continue; }
      if (op == F_FMA) {
        const float c = stack[--sp], b = stack[--sp], a = stack[sp - 1];
        stack[sp - 1] = __fadd_rn(__fmul_rn(a, b), c);
        continue;
      }
      if (op >= F_LOG2 && op <= F_RELU) {
        stack[sp - 1] = fused_unary(op, stack[sp - 1]);
        continue;
      }
      const float b = stack[--sp], a = stack[sp - 1];
      stack[sp - 1] = fused_binary(op, a, b);
    }
    out[o] = stack[0];
  }
}

// out[o] = in[offset + sum idx_k * stride_k] over the OUT shape: permute / expand / slice
struct Gather {
  int rank;
  int64_t out_d[kMaxRank];
  int64_t st[kMaxRank];
  int64_t offset;
};
template <typename I>
__global__ void strided_copy_kernel(float* out, const float* in, Gather gt, int64_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (I o = blockIdx.x * (I)blockDim.x + threadIdx.x; o < (I)total; o += (I)gridDim.x * blockDim.x) {
    I rem = o;
    int64_t src = gt.offset;
    for (int k = gt.rank - 1; k >= 0; --k) {
      const I d = (I)gt.out_d[k], nx = rem / d, i = rem - nx * d;
      rem = nx;
      src += i * gt.st[k];
    }
    out[o] = in[src];
  }
}

struct Pad {
  int rank;
  int64_t out_d[kMaxRank], in_d[kMaxRank], left[kMaxRank];
};
template <typename I>
__global__ void pad_kernel(float* out, const float* in, Pad pd, int64_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (I o = blockIdx.x * (I)blockDim.x + threadIdx.x; o < (I)total; o += (I)gridDim.x * blockDim.x) {
    I rem = o;
    int64_t src = 0, mul = 1;
    bool inside = true;
    for (int k = pd.rank - 1; k >= 0; --k) {
      const I d = (I)pd.out_d[k], nx = rem / d;
      const int64_t i = (int64_t)(rem - nx * d) - pd.left[k];
      rem = nx;
      if (i < 0 || i >= pd.in_d[k]) inside = false;
      src += i * mul;
      mul *= pd.in_d[k];
    }
    out[o] = inside ? in[src] : 0.f;
  }
}

// column-major-order-preserving reshape between two row-major tensors
struct Reshape {
  int in_rank, out_rank;
  int64_t in_d[kMaxRank], out_d[kMaxRank];
};
template <typename I>
__global__ void reshape_cm_kernel(float* out, const float* in, Reshape rs, int64_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (I o = blockIdx.x * (I)blockDim.x + threadIdx.x; o < (I)total; o += (I)gridDim.x * blockDim.x) {
    // row-major index of out -> multi-index -> column-major linear index
    I rem = o, lin = 0;
    I idx[kMaxRank];
    for (int k = rs.out_rank - 1; k >= 0; --k) { const I d = (I)rs.out_d[k], nx = rem / d; idx[k] = rem - nx * d; rem = nx; }
    I mul = 1;
    for (int k = 0; k < rs.out_rank; ++k) { lin += idx[k] * mul; mul *= (I)rs.out_d[k]; }
    // column-major linear index -> multi-index of in -> row-major offset
    I src = 0;
    for (int k = 0; k < rs.in_rank; ++k) { const I d = (I)rs.in_d[k], nx = lin / d; idx[k] = lin - nx * d; lin = nx; }
    for (int k = 0; k < rs.in_rank; ++k) src = src * (I)rs.in_d[k] + idx[k];
    out[o] = in[src];
  }
}

// reduce over one axis: in viewed as [outer, n, inner]
__global__ void reduce_kernel(int kind, float* out, const float* in, int64_t outer, int64_t n, int64_t inner) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t total = outer * inner;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < total; o += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = o / inner, c = o - a * inner;
    const float* p = in + a * n * inner + c;
    float acc = kind == LMB200_REDUCE_SUM ? 0.f : -INFINITY;
    int64_t i = 0;
    for (; i + 16 <= n; i += 16) {                  // same order, 16 loads in flight
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = p[(i + j) * inner];
#pragma unroll
      for (int j = 0; j < 16; ++j) acc = kind == LMB200_REDUCE_SUM ? acc + v[j] : fmaxf(acc, v[j]);
    }
    for (; i < n; ++i) {
      const float v = p[i * inner];
      acc = kind == LMB200_REDUCE_SUM ? acc + v : fmaxf(acc, v);
    }
    out[o] = acc;
  }
}

// C[bt] = A[bt] (MxK) * B[bt] (KxN), 32x32 tiles, plain fp32 FMAs.  A traced graph's products are a few tiles with K of a few hundred:
// a chain of k steps, each a trip to L2, which 32 k at a time took 13 to 18 us for 32 x 256 x 256.  Now a step is 128 k, of
// which every warp multiplies 16 for the whole tile (a column and 32 rows per thread: 9 shared-memory reads for 32 FMAs), the next step
// is on its way meanwhile, and the eight warps' sums are added in warp order at the end.
constexpr int kMatmulThreads = 256, kMatmulK = 128, kMatmulPitch = 36;
__global__ void __launch_bounds__(kMatmulThreads) matmul_kernel(float* C, const float* A, const float* Bm, int M, int N, int K,
                                                                int64_t sA, int64_t sB, int64_t sC) {
  __shared__ __align__(16) float buf[kMatmulK * (kMatmulPitch + 32)];
  float* As = buf;                                       // [k][row], rows padded to 36
  float* Bs = buf + kMatmulK * kMatmulPitch;             // [k][column]
  pdl_launch_dependents();
  pdl_wait();
  const int bt = blockIdx.z;
  const float* a = A + bt * sA;
  const float* b = Bm + bt * sB;
  float* c = C + bt * sC;
  const int tx = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row0 = blockIdx.y * 32, col = blockIdx.x * 32 + tx;
  float an[16], bn[16], acc[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) acc[r] = 0.f;
  auto fetch = [&](int k0) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int r = row0 + w + 8 * (j >> 2), ka = k0 + tx + 32 * (j & 3), kb = k0 + w + 8 * j;
      an[j] = (r < M && ka < K) ? a[(int64_t)r * K + ka] : 0.f;
      bn[j] = (kb < K && col < N) ? b[(int64_t)kb * N + col] : 0.f;
    }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += kMatmulK) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      As[(tx + 32 * (j & 3)) * kMatmulPitch + w + 8 * (j >> 2)] = an[j];
      Bs[(w + 8 * j) * 32 + tx] = bn[j];
    }
    __syncthreads();
    if (k0 + kMatmulK < K) fetch(k0 + kMatmulK);
    if (k0 + 16 * w < K) {
#pragma unroll 4
      for (int k = 16 * w; k < 16 * w + 16; ++k) {
        const float bv = Bs[k * 32 + tx];
#pragma unroll
        for (int r = 0; r < 32; r += 4) {
          const float4 av = *reinterpret_cast<const float4*>(&As[k * kMatmulPitch + r]);
          acc[r] = fmaf(av.x, bv, acc[r]);
          acc[r + 1] = fmaf(av.y, bv, acc[r + 1]);
          acc[r + 2] = fmaf(av.z, bv, acc[r + 2]);
          acc[r + 3] = fmaf(av.w, bv, acc[r + 3]);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < 32; ++r) buf[(w * 32 + r) * 32 + tx] = acc[r];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = 4 * w + j;
    float t = 0.f;
#pragma unroll
    for (int v = 0; v < 8; ++v) t += buf[(v * 32 + r) * 32 + tx];
    if (row0 + r < M && col < N) c[(int64_t)(row0 + r) * N + col] = t;
  }
}

__global__ void gather_kernel(float* out, const float* table, int64_t vocab, int64_t dim, const float* ids, int64_t n_ids) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t total = n_ids * dim;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < total; o += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = o / dim, c = o - r * dim;
    const int64_t id = (int64_t)ids[r];
    out[o] = (id >= 0 && id < vocab) ? table[id * dim + c] : 0.f;
  }
}

// im2col of the last axis: out[bc, o, k] = a[bc, o*stride + k*dilation]   (src/Execution.jl:481-504)
__global__ void unfold1d_kernel(float* out, const float* a, int64_t BC, int64_t Lin, int64_t O, int64_t K, int64_t stride,
                                int64_t dilation) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t total = BC * O * K;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = i % K, o = (i / K) % O, bc = i / (K * O);
    out[i] = a[bc * Lin + o * stride + k * dilation];
  }
}

__global__ void cumsum_kernel(float* out, const float* in, int64_t rows, int64_t n) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= rows) return;
  float acc = 0.f;
  for (int64_t i = 0; i < n; ++i) { acc += in[r * n + i]; out[r * n + i] = acc; }
}

// mode 0: RMSNorm(+scale); mode 1: LayerNorm (mean-centred, optional w and bias)
__global__ void __launch_bounds__(256) norm_kernel(float* y, const float* x, const float* w, const float* bias,
                                                   int64_t n, float eps, int mean_centre) {
  __shared__ float red[8];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  const float* xr = x + blockIdx.x * n;
  float* yr = y + blockIdx.x * n;
  auto block_sum = [&](float v) -> float {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((tid & 31) == 0) red[tid >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[i];
    return t;
  };
  float mean = 0.f;
  if (mean_centre) {
    float s = 0.f;
    for (int64_t i = tid; i < n; i += 256) s += xr[i];
    mean = block_sum(s) * (1.0f / (float)n);
  }
  float ss = 0.f;
  for (int64_t i = tid; i < n; i += 256) { const float v = xr[i] + mean * -1.0f; ss += v * v; }
  const float var = block_sum(ss) * (1.0f / (float)n);
  const float inv = 1.0f / sqrtf(var + eps);
  for (int64_t i = tid; i < n; i += 256) {
    float v = (xr[i] + mean * -1.0f) * inv;
    if (w) v = v * w[i];
    if (bias) v = v + bias[i];
    yr[i] = v;
  }
}

__global__ void silu_gate_kernel(float* out, const float* gate, const float* up, int64_t n) {
  pdl_launch_dependents();
  pdl_wait();
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < n; o += (int64_t)gridDim.x * blockDim.x) {
    out[o] = silu_gate(gate[o], up[o]);
  }
}

__global__ void rope_kernel(float* out, const float* x, int64_t BH, int64_t S, int64_t D, int64_t prev_seq, float l2base) {
  pdl_launch_dependents();
  pdl_wait();
  const int64_t half = D / 2;
  const int64_t total = BH * S * half;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < total; o += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = o % half, s = (o / half) % S, bh = o / (half * S);
    // inv_freq = recip(exp2((i*2*(1/D)) * log2(base)));  angle = (s + prev) * inv_freq
    const float fr = __fmul_rn(__fmul_rn(__fmul_rn((float)i, 2.0f), 1.0f / (float)D), l2base);
    const float inv = 1.0f / exp2f(fr);
    const float ang = __fmul_rn((float)s + (float)prev_seq, inv);
    const float sn = sinf(ang), cs = sinf(kHalfPi + ang * -1.0f);
    const float* xr = x + (bh * S + s) * D;
    float* yr = out + (bh * S + s) * D;
    const float x0 = xr[i], x1 = xr[i + half];
    yr[i] = x0 * cs + (x1 * sn) * -1.0f;
    yr[i + half] = x0 * sn + x1 * cs;
  }
}

__global__ void __launch_bounds__(256) argmax_kernel(int32_t* out, const float* x, int64_t n) {
  __shared__ float sv[256];
  __shared__ int si[256];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  const float* row = x + blockIdx.x * n;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int64_t i = tid; i < n; i += 256) {
    const float v = row[i];
    if (v > best || (v == best && (int)i < bi)) { best = v; bi = (int)i; }
  }
  sv[tid] = best; si[tid] = bi;
  __syncthreads();
  for (int off = 128; off > 0; off >>= 1) {
    if (tid < off) {
      const float v = sv[tid + off];
      const int i = si[tid + off];
      if (v > sv[tid] || (v == sv[tid] && i < si[tid])) { sv[tid] = v; si[tid] = i; }
    }
    __syncthreads();
  }
  if (tid == 0) out[blockIdx.x] = si[0];
}

int grid_for(int64_t total) {
  int64_t g = ceil_div(total, 256);
  if (g > 148 * 16) g = 148 * 16;
  if (g < 1) g = 1;
  return (int)g;
}

// element counts (an operand is never larger than what a 32-bit index of the output reaches through its strides, which stay 64-bit)
bool fits32(int64_t total) { return total <= 0x7fffffff; }

int32_t check_dims(int32_t rank, const int64_t* dims, int64_t* total) {
  LMB_REQUIRE(rank >= 0 && rank <= kMaxRank, "rank %d outside 0..%d", rank, kMaxRank);
  LMB_REQUIRE(rank == 0 || dims, "null dims");
  int64_t t = 1;
  for (int i = 0; i < rank; ++i) {
    LMB_REQUIRE(dims[i] >= 1, "dimension %d is %lld", i, (long long)dims[i]);
    t *= dims[i];
  }
  *total = t;
  return LMB200_OK;
}

// strides of an operand broadcast against out (1-dims prepended, src/Execution.jl:207-214)
int32_t bcast_strides(int out_rank, const int64_t* out_d, int rank, const int64_t* d, int64_t* st, const char* what) {
  LMB_REQUIRE(rank <= out_rank, "%s: operand rank %d above output rank %d", what, rank, out_rank);
  const int shift = out_rank - rank;
  int64_t mul = 1;
  for (int k = out_rank - 1; k >= 0; --k) {
    const int j = k - shift;
    if (j < 0) { st[k] = 0; continue; }
    if (d[j] == out_d[k]) { st[k] = d[j] == 1 ? 0 : mul; }
    else if (d[j] == 1) st[k] = 0;
    else return fail(LMB200_EINVAL, "%s: dimension mismatch in broadcasting: %lld vs %lld", what, (long long)d[j],
                     (long long)out_d[k]);
    mul *= d[j];
  }
  return LMB200_OK;
}

}  // namespace
}  // namespace lmb

using namespace lmb;

#define CTX_OR_FAIL()                  \
  Ctx* ctx = ctx_from(h);              \
  if (!ctx) return LMB200_EINVAL;      \
  LMB_CUDA(cudaSetDevice(ctx->device))

#define LAUNCHED()          \
  ctx->launches++;          \
  LMB_CUDA(cudaGetLastError())

namespace {

// between capture_begin and capture_end: what was just launched, for record_finish()
RecordedStep step_of(StepKind kind, float* out, int rank, const int64_t* d, std::vector<StepView> in) {
  RecordedStep s;
  s.kind = kind; s.out = out; s.rank = rank; s.in = std::move(in);
  for (int k = 0; k < rank; ++k) s.d[k] = d[k];
  return s;
}

// a movement: per output axis the source axis + 1 (0: none), then per source axis where it starts
RecordedStep movement(float* out, int rank, const int64_t* d, const StepView& in, const int* axis, const int64_t* start) {
  RecordedStep s = step_of(STEP_COPY, out, rank, d, {in});
  s.arg.assign(2 * kMaxRank, 0);
  for (int k = 0; k < rank; ++k) s.arg[k] = axis[k];
  if (start)
    for (int k = 0; k < in.rank; ++k) s.arg[kMaxRank + k] = (int)start[k];
  return s;
}

}  // namespace

extern "C" int32_t lmb200_ew(lmb200_ctx h, int32_t opcode, float* out, int32_t out_rank, const int64_t* out_dims,
                             const float* a, int32_t a_rank, const int64_t* a_dims, const float* b, int32_t b_rank,
                             const int64_t* b_dims, const float* c, int32_t c_rank, const int64_t* c_dims) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && a, "ew: null pointer");
  const bool binary = opcode <= LMB200_OP_MAX || opcode >= LMB200_OP_FUSED_MUL_ADD;
  const bool ternary = opcode == LMB200_OP_FUSED_MUL_ADD;
  LMB_REQUIRE((opcode >= 0 && opcode <= LMB200_OP_MAX) || (opcode >= LMB200_OP_LOG2 && opcode <= LMB200_OP_FUSED_ADD_RELU),
              "ew: opcode %d", opcode);
  LMB_REQUIRE(!binary || b, "ew: opcode %d needs operand b", opcode);
  LMB_REQUIRE(!ternary || c, "ew: opcode %d needs operand c", opcode);
  Idx ix{};
  int64_t total, tmp;
  LMB_TRY(check_dims(out_rank, out_dims, &total));
  ix.rank = out_rank;
  for (int i = 0; i < out_rank; ++i) ix.out_d[i] = out_dims[i];
  LMB_TRY(check_dims(a_rank, a_dims, &tmp));
  LMB_TRY(bcast_strides(out_rank, out_dims, a_rank, a_dims, ix.sa, "ew a"));
  if (binary) {
    LMB_TRY(check_dims(b_rank, b_dims, &tmp));
    LMB_TRY(bcast_strides(out_rank, out_dims, b_rank, b_dims, ix.sb, "ew b"));
  }
  if (ternary) {
    LMB_TRY(check_dims(c_rank, c_dims, &tmp));
    LMB_TRY(bcast_strides(out_rank, out_dims, c_rank, c_dims, ix.sc, "ew c"));
  }
  LMB_CUDA(launch_k(fits32(total) ? ew_kernel<uint32_t> : ew_kernel<int64_t>, dim3((unsigned)(grid_for(total))), dim3(256), 0, ctx->stream, opcode, out, a, binary ? b : nullptr, ternary ? c : nullptr, ix, total));
  LAUNCHED();
  if (ctx->recorder) {
    RecordedStep r = step_of(STEP_EW, out, out_rank, out_dims, {step_tensor(a, a_rank, a_dims)});
    if (binary) r.in.push_back(step_tensor(b, b_rank, b_dims));
    if (ternary) r.in.push_back(step_tensor(c, c_rank, c_dims));
    r.op = opcode;
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_fused_ew(lmb200_ctx h, float* out, int32_t out_rank, const int64_t* out_dims, int32_t n_inputs,
                                   const float* const* inputs, const int32_t* in_ranks, const int64_t* in_dims,
                                   int32_t n_instr, const int32_t* ops, const float* args) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && ops && args && in_ranks && n_inputs >= 0 && (n_inputs == 0 || (inputs && in_dims)), "fused_ew: null pointer");
  LMB_REQUIRE(n_inputs <= kFusedMaxInputs, "fused_ew: %d inputs (at most %d)", n_inputs, kFusedMaxInputs);
  LMB_REQUIRE(n_instr >= 1 && n_instr <= kFusedMaxInstr, "fused_ew: %d instructions (1..%d)", n_instr, kFusedMaxInstr);
  FusedProgram pg{};
  int64_t total, tmp;
  LMB_TRY(check_dims(out_rank, out_dims, &total));
  pg.rank = out_rank; pg.n_in = n_inputs; pg.n_instr = n_instr;
  for (int i = 0; i < out_rank; ++i) pg.out_d[i] = out_dims[i];
  const int64_t* d = in_dims;
  for (int i = 0; i < n_inputs; ++i) {
    LMB_REQUIRE(inputs[i], "fused_ew: input %d is null", i);
    LMB_TRY(check_dims(in_ranks[i], d, &tmp));
    LMB_TRY(bcast_strides(out_rank, out_dims, in_ranks[i], d, pg.st[i], "fused_ew input"));
    pg.in[i] = inputs[i];
    d += in_ranks[i];
  }
  int depth = 0;                                   // the program must be well-formed postfix: checked here, not on the device
  for (int pc = 0; pc < n_instr; ++pc) {
    const int op = ops[pc];
    LMB_REQUIRE(op >= F_PUSH_IN && op <= F_ADD_RELU, "fused_ew: opcode %d at %d", op, pc);
    int need = 0, push = 1;
    if (op == F_PUSH_IN) LMB_REQUIRE(args[pc] >= 0 && (int)args[pc] < n_inputs && (float)(int)args[pc] == args[pc], "fused_ew: input index at %d", pc);
    if (op == F_FMA) need = 3;
    else if (op >= F_LOG2 && op <= F_RELU) need = 1;
    else if (op >= F_ADD) need = 2;
    LMB_REQUIRE(depth >= need, "fused_ew: stack underflow at instruction %d", pc);
    depth += push - need;
    LMB_REQUIRE(depth <= kFusedMaxStack, "fused_ew: stack deeper than %d at instruction %d", kFusedMaxStack, pc);
    pg.op[pc] = op; pg.arg[pc] = args[pc];
  }
  LMB_REQUIRE(depth == 1, "fused_ew: the program leaves %d values", depth);
  if (total == 0) return LMB200_OK;
  LMB_CUDA(launch_k(fits32(total) ? fused_ew_kernel<uint32_t> : fused_ew_kernel<int64_t>, dim3((unsigned)(grid_for(total))), dim3(256), 0, ctx->stream, out, pg, total));
  LAUNCHED();
  if (ctx->recorder) {
    RecordedStep r = step_of(STEP_FUSED, out, out_rank, out_dims, {});
    const int64_t* id = in_dims;
    for (int i = 0; i < n_inputs; id += in_ranks[i], ++i) r.in.push_back(step_tensor(inputs[i], in_ranks[i], id));
    r.arg.assign(ops, ops + n_instr);
    r.val.assign(args, args + n_instr);
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_reduce(lmb200_ctx h, int32_t kind, float* out, const float* in, int32_t rank,
                                 const int64_t* dims, int32_t axis) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in, "reduce: null pointer");
  LMB_REQUIRE(kind == LMB200_REDUCE_SUM || kind == LMB200_REDUCE_MAX, "reduce: kind %d", kind);
  int64_t total;
  LMB_TRY(check_dims(rank, dims, &total));
  LMB_REQUIRE(axis >= 0 && axis < rank, "reduce: axis %d of rank %d", axis, rank);
  int64_t outer = 1, inner = 1;
  for (int i = 0; i < axis; ++i) outer *= dims[i];
  for (int i = axis + 1; i < rank; ++i) inner *= dims[i];
  LMB_CUDA(launch_k_opt(false, reduce_kernel, dim3((unsigned)(grid_for(outer * inner))), dim3(256), 0, ctx->stream, kind, out, in, outer, dims[axis], inner));
  LAUNCHED();
  if (ctx->recorder) {
    int64_t od[kMaxRank];
    int n = 0;
    for (int i = 0; i < rank; ++i)
      if (i != axis) od[n++] = dims[i];
    RecordedStep r = step_of(STEP_REDUCE, out, n, od, {step_tensor(in, rank, dims)});
    r.op = kind; r.n = dims[axis]; r.inner = inner;
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_matmul(lmb200_ctx h, float* out, const float* a, int32_t a_rank, const int64_t* a_dims,
                                 const float* b, int32_t b_rank, const int64_t* b_dims) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && a && b, "matmul: null pointer");
  int64_t ta, tb;
  LMB_TRY(check_dims(a_rank, a_dims, &ta));
  LMB_TRY(check_dims(b_rank, b_dims, &tb));
  // the four cases of batch_matmul (src/Execution.jl:12-54); anything else is the reference's error
  const bool ok = (a_rank == 2 && b_rank == 2) || (a_rank == 3 && b_rank == 2) || (a_rank == 3 && b_rank == 3) ||
                  (a_rank == 4 && b_rank == 4);
  LMB_REQUIRE(ok, "Batch matmul not implemented for %dD and %dD", a_rank, b_rank);
  const int64_t M = a_dims[a_rank - 2], K = a_dims[a_rank - 1], N = b_dims[b_rank - 1];
  LMB_REQUIRE(b_dims[b_rank - 2] == K, "matmul: inner dimensions %lld vs %lld", (long long)K, (long long)b_dims[b_rank - 2]);
  int64_t batch = 1;
  for (int i = 0; i < a_rank - 2; ++i) batch *= a_dims[i];
  if (b_rank > 2)
    for (int i = 0; i < b_rank - 2; ++i)
      LMB_REQUIRE(a_dims[i] == b_dims[i], "Batch dimensions must match: %lld vs %lld", (long long)a_dims[i], (long long)b_dims[i]);
  LMB_REQUIRE(batch <= 65535, "matmul: batch %lld too large", (long long)batch);
  dim3 grid((unsigned)ceil_div(N, 32), (unsigned)ceil_div(M, 32), (unsigned)batch);
  LMB_CUDA(launch_k_opt(false, matmul_kernel, grid, dim3(kMatmulThreads), 0, ctx->stream, out, a, b, (int)M, (int)N, (int)K, M * K, b_rank > 2 ? K * N : 0, M * N));
  LAUNCHED();
  if (ctx->recorder) {
    int64_t od[kMaxRank];
    for (int i = 0; i < a_rank; ++i) od[i] = i == a_rank - 1 ? N : a_dims[i];
    record_step(ctx, step_of(STEP_MATMUL, out, a_rank, od, {step_tensor(a, a_rank, a_dims), step_tensor(b, b_rank, b_dims)}));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_permute(lmb200_ctx h, float* out, const float* in, int32_t rank, const int64_t* in_dims,
                                  const int32_t* perm) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in && perm, "permute: null pointer");
  int64_t total;
  LMB_TRY(check_dims(rank, in_dims, &total));
  int64_t in_st[kMaxRank];
  int64_t mul = 1;
  for (int k = rank - 1; k >= 0; --k) { in_st[k] = mul; mul *= in_dims[k]; }
  Gather gt{};
  gt.rank = rank;
  bool seen[kMaxRank] = {false};
  for (int k = 0; k < rank; ++k) {
    LMB_REQUIRE(perm[k] >= 0 && perm[k] < rank && !seen[perm[k]], "permute: bad permutation");
    seen[perm[k]] = true;
    gt.out_d[k] = in_dims[perm[k]];
    gt.st[k] = in_st[perm[k]];
  }
  // A warp that reads 32 places more than 1 MB apart, of a tensor larger than L2, waits for address translation: the 64-bit kernel, which has fewer
  // reads in flight, is the faster one ([128, 128, 128, 32] turned round 1136 us, 1360 with 32-bit indices; [32, 2048, 1024] 1524 and 1814).
  // Everywhere else it is the other way round ([8192, 8192] 377 and 284; [16, 2048, 2048] with the 16 last 451 and 325).
  const bool far = rank > 0 && total > (1 << 25) && gt.out_d[rank - 1] >= 32 && gt.st[rank - 1] * 4 > (1 << 20);
  LMB_CUDA(launch_k(fits32(total) && !far ? strided_copy_kernel<uint32_t> : strided_copy_kernel<int64_t>, dim3((unsigned)(grid_for(total))), dim3(256), 0, ctx->stream, out, in, gt, total));
  LAUNCHED();
  if (ctx->recorder) {
    int axis[kMaxRank];
    for (int k = 0; k < rank; ++k) axis[k] = perm[k] + 1;
    record_step(ctx, movement(out, rank, gt.out_d, step_tensor(in, rank, in_dims), axis, nullptr));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_reshape_colmajor(lmb200_ctx h, float* out, const float* in, int32_t in_rank,
                                           const int64_t* in_dims, int32_t out_rank, const int64_t* out_dims) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in, "reshape: null pointer");
  int64_t ti, to;
  LMB_TRY(check_dims(in_rank, in_dims, &ti));
  LMB_TRY(check_dims(out_rank, out_dims, &to));
  LMB_REQUIRE(ti == to, "Length mismatch in Reshape!: %lld vs %lld", (long long)to, (long long)ti);
  Reshape rs{};
  rs.in_rank = in_rank; rs.out_rank = out_rank;
  for (int i = 0; i < in_rank; ++i) rs.in_d[i] = in_dims[i];
  for (int i = 0; i < out_rank; ++i) rs.out_d[i] = out_dims[i];
  LMB_CUDA(launch_k(fits32(to) ? reshape_cm_kernel<uint32_t> : reshape_cm_kernel<int64_t>, dim3((unsigned)(grid_for(to))), dim3(256), 0, ctx->stream, out, in, rs, to));
  LAUNCHED();
  if (ctx->recorder) {
    record_step(ctx, step_of(STEP_RESHAPE, out, out_rank, out_dims, {step_tensor(in, in_rank, in_dims)}));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_expand(lmb200_ctx h, float* out, const float* in, int32_t in_rank, const int64_t* in_dims,
                                 int32_t axis, int64_t size) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in, "expand: null pointer");
  int64_t ti;
  LMB_TRY(check_dims(in_rank, in_dims, &ti));
  LMB_REQUIRE(in_rank < kMaxRank && axis >= 0 && axis <= in_rank && size >= 1, "expand: axis %d size %lld", axis, (long long)size);
  Gather gt{};
  gt.rank = in_rank + 1;
  int64_t mul = 1;
  int64_t in_st[kMaxRank];
  for (int k = in_rank - 1; k >= 0; --k) { in_st[k] = mul; mul *= in_dims[k]; }
  for (int k = 0, j = 0; k < gt.rank; ++k) {
    if (k == axis) { gt.out_d[k] = size; gt.st[k] = 0; }
    else { gt.out_d[k] = in_dims[j]; gt.st[k] = in_st[j]; ++j; }
  }
  const int64_t total = ti * size;
  LMB_CUDA(launch_k(fits32(total) ? strided_copy_kernel<uint32_t> : strided_copy_kernel<int64_t>, dim3((unsigned)(grid_for(total))), dim3(256), 0, ctx->stream, out, in, gt, total));
  LAUNCHED();
  if (ctx->recorder) {
    int source[kMaxRank];
    for (int k = 0, j = 0; k < gt.rank; ++k) source[k] = k == axis ? 0 : ++j;
    record_step(ctx, movement(out, gt.rank, gt.out_d, step_tensor(in, in_rank, in_dims), source, nullptr));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_slice(lmb200_ctx h, float* out, const float* in, int32_t rank, const int64_t* in_dims,
                                const int64_t* starts, const int64_t* stops) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in && starts && stops, "slice: null pointer");
  int64_t ti;
  LMB_TRY(check_dims(rank, in_dims, &ti));
  Gather gt{};
  gt.rank = rank;
  int64_t mul = 1, total = 1;
  for (int k = rank - 1; k >= 0; --k) {
    const int64_t s = starts[k] < 0 ? 0 : starts[k];
    const int64_t e = stops[k] > in_dims[k] ? in_dims[k] : stops[k];
    LMB_REQUIRE(e > s, "slice: empty range on axis %d", k);
    gt.out_d[k] = e - s;
    gt.st[k] = mul;
    gt.offset += s * mul;
    mul *= in_dims[k];
    total *= e - s;
  }
  LMB_CUDA(launch_k(fits32(total) ? strided_copy_kernel<uint32_t> : strided_copy_kernel<int64_t>, dim3((unsigned)(grid_for(total))), dim3(256), 0, ctx->stream, out, in, gt, total));
  LAUNCHED();
  if (ctx->recorder) {
    int source[kMaxRank];
    int64_t from[kMaxRank];
    for (int k = 0; k < rank; ++k) { source[k] = k + 1; from[k] = starts[k] < 0 ? 0 : starts[k]; }
    if (fits32(ti)) record_step(ctx, movement(out, rank, gt.out_d, step_tensor(in, rank, in_dims), source, from));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_pad(lmb200_ctx h, float* out, const float* in, int32_t rank, const int64_t* in_dims,
                              const int64_t* left, const int64_t* right) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in && left && right, "pad: null pointer");
  int64_t ti;
  LMB_TRY(check_dims(rank, in_dims, &ti));
  Pad pd{};
  pd.rank = rank;
  int64_t total = 1;
  for (int k = 0; k < rank; ++k) {
    LMB_REQUIRE(left[k] >= 0 && right[k] >= 0, "pad: negative padding");
    pd.in_d[k] = in_dims[k]; pd.left[k] = left[k];
    pd.out_d[k] = in_dims[k] + left[k] + right[k];
    total *= pd.out_d[k];
  }
  LMB_CUDA(launch_k(fits32(total) ? pad_kernel<uint32_t> : pad_kernel<int64_t>, dim3((unsigned)(grid_for(total))), dim3(256), 0, ctx->stream, out, in, pd, total));
  LAUNCHED();
  if (ctx->recorder) {
    RecordedStep r = step_of(STEP_PAD, out, rank, pd.out_d, {step_tensor(in, rank, in_dims)});
    for (int k = 0; k < rank; ++k) r.arg.push_back((int)left[k]);
    if (fits32(total)) record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_gather(lmb200_ctx h, float* out, const float* table, int64_t vocab, int64_t dim,
                                 const float* ids, int64_t n_ids) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && table && ids && vocab >= 1 && dim >= 1 && n_ids >= 1, "gather: bad argument");
  LMB_CUDA(launch_k(gather_kernel, dim3((unsigned)(grid_for(n_ids * dim))), dim3(256), 0, ctx->stream, out, table, vocab, dim, ids, n_ids));
  LAUNCHED();
  if (ctx->recorder) {
    const int64_t od[2] = {n_ids, dim}, td[2] = {vocab, dim};
    RecordedStep r = step_of(STEP_GATHER, out, 2, od, {step_tensor(table, 2, td), step_tensor(ids, 1, &n_ids)});
    r.n = vocab; r.inner = dim;
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_unfold1d(lmb200_ctx h, float* out, const float* in, int64_t rows, int64_t length, int64_t kernel,
                                   int64_t stride, int64_t dilation) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in && rows >= 1 && kernel >= 1 && stride >= 1 && dilation >= 1, "unfold: bad argument");
  const int64_t O = (length - dilation * (kernel - 1) - 1) / stride + 1;
  LMB_REQUIRE(O >= 1, "unfold: length %lld too short for kernel %lld", (long long)length, (long long)kernel);
  LMB_CUDA(launch_k(unfold1d_kernel, dim3((unsigned)(grid_for(rows * O * kernel))), dim3(256), 0, ctx->stream, out, in, rows, length, O, kernel, stride, dilation));
  LAUNCHED();
  return LMB200_OK;
}

extern "C" int32_t lmb200_cumsum_last(lmb200_ctx h, float* out, const float* in, int64_t rows, int64_t n) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && in && rows >= 1 && n >= 1, "cumsum: bad argument");
  LMB_CUDA(launch_k_opt(false, cumsum_kernel, dim3((unsigned)(ceil_div(rows, 128))), dim3(128), 0, ctx->stream, out, in, rows, n));
  LAUNCHED();
  if (ctx->recorder) {
    const int64_t od[2] = {rows, n};
    RecordedStep r = step_of(STEP_CUMSUM, out, 2, od, {step_tensor(in, 2, od)});
    r.n = n;
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_rmsnorm_scale(lmb200_ctx h, float* y, const float* x, const float* w, int64_t rows,
                                        int64_t n, float eps) {
  CTX_OR_FAIL();
  LMB_REQUIRE(y && x && rows >= 1 && n >= 1, "rmsnorm: bad argument");
  LMB_CUDA(launch_k_opt(false, norm_kernel, dim3((unsigned)(rows)), dim3(256), 0, ctx->stream, y, x, w, nullptr, n, eps, 0));
  LAUNCHED();
  if (ctx->recorder) {
    const int64_t od[2] = {rows, n};
    RecordedStep r = step_of(STEP_NORM, y, 2, od, {step_tensor(x, 2, od), step_tensor(w, 1, &n), step_tensor(nullptr, 1, &n)});
    r.op = 0; r.n = n;
    r.val = {eps};
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_layernorm(lmb200_ctx h, float* y, const float* x, const float* w, const float* bias,
                                    int64_t rows, int64_t n, float eps) {
  CTX_OR_FAIL();
  LMB_REQUIRE(y && x && rows >= 1 && n >= 1, "layernorm: bad argument");
  LMB_CUDA(launch_k_opt(false, norm_kernel, dim3((unsigned)(rows)), dim3(256), 0, ctx->stream, y, x, w, bias, n, eps, 1));
  LAUNCHED();
  if (ctx->recorder) {
    const int64_t od[2] = {rows, n};
    RecordedStep r = step_of(STEP_NORM, y, 2, od, {step_tensor(x, 2, od), step_tensor(w, 1, &n), step_tensor(bias, 1, &n)});
    r.op = 1; r.n = n;
    r.val = {eps};
    record_step(ctx, std::move(r));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_silu_gate(lmb200_ctx h, float* out, const float* gate, const float* up, int64_t n) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && gate && up && n >= 1, "silu_gate: bad argument");
  LMB_CUDA(launch_k(silu_gate_kernel, dim3((unsigned)(grid_for(n))), dim3(256), 0, ctx->stream, out, gate, up, n));
  LAUNCHED();
  if (ctx->recorder) {
    record_step(ctx, step_of(STEP_SILU, out, 1, &n, {step_tensor(gate, 1, &n), step_tensor(up, 1, &n)}));
  }
  return LMB200_OK;
}

extern "C" int32_t lmb200_rope(lmb200_ctx h, float* out, const float* x, int64_t B, int64_t H, int64_t S, int64_t D,
                               int64_t prev_seq, float base) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && x && B >= 1 && H >= 1 && S >= 1 && D >= 2 && D % 2 == 0, "rope: bad argument");
  LMB_CUDA(launch_k(rope_kernel, dim3((unsigned)(grid_for(B * H * S * (D / 2)))), dim3(256), 0, ctx->stream, out, x, B * H, S, D, prev_seq, log2f(base)));
  LAUNCHED();
  return LMB200_OK;
}

extern "C" int32_t lmb200_argmax(lmb200_ctx h, int32_t* out, const float* x, int64_t rows, int64_t n) {
  CTX_OR_FAIL();
  LMB_REQUIRE(out && x && rows >= 1 && n >= 1, "argmax: bad argument");
  LMB_CUDA(launch_k_opt(false, argmax_kernel, dim3((unsigned)(rows)), dim3(256), 0, ctx->stream, out, x, n));
  LAUNCHED();
  return LMB200_OK;
}
