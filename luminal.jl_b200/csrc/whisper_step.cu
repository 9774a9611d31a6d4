// A bf16 Whisper decoder's step as two launches: embedding and layers; head, greedy tokens and positions.
//
// The step of a small decoder is a chain: eight dependent pieces per layer -- q/k/v, self attention, out_proj, cross q, cross attention, out_proj, fc1,
// fc2 -- each a microsecond of work.  As launches they cost 6.8 us each (Whisper-base, batch 8, 1500 cross-attention keys: 328 us a step; in a chain of the
// large GEMV kernels, whose tiles of 128 rows leave most SMs idle here, 350).  Here one CTA per SM takes a fixed share of every piece's units (16 rows of
// a matrix; one sequence's head, or a part of its keys) and counts finished units through L2; a consumer has its weights or its first cross-attention
// keys in registers before it starts to wait.  189 us a step: 2.0 to 2.6 us a piece -- a microsecond of it the release of the results and the notice of it,
// another the trip of the next piece's input -- 4.0 for the cross attention (25 MB) and 2.8 for fc2, whose second half of the weights does not fit the registers.
// Products are mma.sync m16n8k16 with the batch as N = 8 or 16: at this width a tcgen05 tile of 128 rows would occupy 4 to 16 SMs.  k is split over a
// CTA's eight warps and added in warp order.
// Registers are what this kernel is short of: a spilled word comes back from L2, since every wait empties L1 (four units of weights ahead instead of two,
// at 650 bytes of spills: 238 us).
#include "whisper_step.cuh"

#include "pdl.cuh"
#include "step.cuh"

#include <stdlib.h>

#include <algorithm>

namespace lmb {
namespace {

constexpr int kThreads = 256, kWarps = 8, kD = 64, kMaxHidden = 1024;
constexpr float kLog2e = 1.4426950408889634f;

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// weights and cross-attention keys: written before the launch, read once
__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 ld_data(const void* p) { return *reinterpret_cast<const uint4*>(p); }

__device__ __forceinline__ float gelu_ref(float a) {       // src/HighLevelOps.jl:153-168, as the launched step's epilogue
  const float inner = (0.7978845608f * a) * (1.0f + (0.044715f * a) * a);
  const float z = inner * 2.0f;
  const float sg = 1.0f / (1.0f + exp2f((z * -1.0f) * kLog2e));
  const float th = sg * 2.0f + -1.0f;
  return (a * 0.5f) * (1.0f + th);
}

// threadIdx.x anew in every unit: what eight pieces derive from it would otherwise be kept across all of them, in spilled registers
__device__ __forceinline__ int thread_index() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

struct Shared {
  float red[kWarps * 16 * 16];         // [warp][row][column]; attention: [warp][d]
  float stat[2][kWarps][16];           // the input norm's sums, per warp; attention: maxima and sums; head: best logits and their ids
  float inv[16], mu[16];               // head: the norm's scale and, times it, the mean
  __align__(16) bf16 x[kMaxHidden * kWhisperStepBatch];    // out_proj of the cross attention: its input, [k / 8][column][k % 8]
  WhisperStepLayer layer[2];           // the present layer's matrices and the next one's
  int dead;
};

// The input norm's sums of x^2 and x, per warp: four slots a warp at a time, columns along the lanes.
template <int NT>
__device__ __forceinline__ void input_sums(const WhisperStepParams& p, Shared& sm, int warp, int lane) {
  const int slots = p.hidden >> 4;
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    float s2 = 0.f, s1 = 0.f;
    for (int s = warp * 4 + (lane >> 3); s < slots; s += 32) {
      s2 += p.ssq[s * 32 + 8 * nt + (lane & 7)];
      s1 += p.sum[s * 32 + 8 * nt + (lane & 7)];
    }
    s2 += __shfl_xor_sync(0xffffffffu, s2, 8); s2 += __shfl_xor_sync(0xffffffffu, s2, 16);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 8); s1 += __shfl_xor_sync(0xffffffffu, s1, 16);
    if (lane < 8) { sm.stat[0][warp][8 * nt + lane] = s2; sm.stat[1][warp][8 * nt + lane] = s1; }
  }
}
// 1 / sqrt(variance + eps) of column b, and the mean times it
__device__ __forceinline__ float2 norm_scale(const WhisperStepParams& p, const Shared& sm, int b) {
  float s2 = 0.f, s1 = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) { s2 += sm.stat[0][w][b]; s1 += sm.stat[1][w][b]; }
  const float rn = 1.0f / (float)p.hidden, mu = s1 * rn;
  const float inv = 1.0f / sqrtf(fmaxf(s2 * rn - mu * mu, 0.f) + p.eps);
  return make_float2(inv, mu * inv);
}

enum Piece { QKV, SELF, OUT_SELF, Q_CROSS, CROSS, OUT_CROSS, FC1, FC2 };

// One row's value x of the residual (rows 16 rt + e / (8 NT), column e % (8 NT)): x, x * gain for the next product, and the sums of x and x^2 over
// the tile's rows for its norm (slots as the launched step's).  All threads call it; those from 128 NT on hold nothing.
template <int NT>
__device__ __forceinline__ void finish_rows(const WhisperStepParams& p, int rt, float xv, float gain, float* capture, Shared& sm) {
  constexpr int N = 8 * NT;
  const int e = threadIdx.x, row = 16 * rt + e / N, b = e % N, warp = e >> 5, lane = e & 31;
  const bool live = e < 16 * N;
  if (live) {
    p.x[(size_t)row * p.Bp + b] = xv;
    p.xn[(size_t)(row >> 3) * (p.Bp * 8) + (b >> 3) * 64 + (b & 7) * 8 + (row & 7)] = __float2bfloat16_rn(xv * gain);
    if (capture && b < p.B) capture[(size_t)b * p.hidden + row] = xv;
  }
  float s2 = live ? xv * xv : 0.f, s1 = live ? xv : 0.f;
#pragma unroll
  for (int off = N; off < 32; off <<= 1) {
    s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    s1 += __shfl_xor_sync(0xffffffffu, s1, off);
  }
  __syncthreads();                                         // (sm.stat has been read)
  if (lane < N) { sm.stat[0][warp][lane] = s2; sm.stat[1][warp][lane] = s1; }
  __syncthreads();
  if (e < N) {
    float t2 = 0.f, t1 = 0.f;
#pragma unroll
    for (int w = 0; w < 16 * N / 32; ++w) { t2 += sm.stat[0][w][e]; t1 += sm.stat[1][w][e]; }
    p.ssq[rt * 32 + e] = t2;
    p.sum[rt * 32 + e] = t1;
  }
}

// Rows 16 rt .. 16 rt + 15 of a matrix [rows, K] times the batch, and what the piece does with them.  Warp w takes k = 64 u .. 64 u + 63 for u = w, w + 8, ..;
// a lane's 16 bytes of a row are 8 consecutive k, and both operands give the same k the same place among the MMAs' sixteen.
template <int NT>
__device__ __forceinline__ bool gemv_unit(const WhisperStepParams& p, const WhisperStepLayer& L, int piece, int rt, const unsigned* before, unsigned need, Shared& sm) {
  constexpr int N = 8 * NT, kAhead = 2;
  const int tid = thread_index(), lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const bool norm = piece == QKV || piece == Q_CROSS || piece == FC1, joined = piece == OUT_CROSS && p.splits > 1;
  const int K = piece == FC2 ? p.ffn : p.hidden, units = K >> 6, KS = (K + 127) >> 7;
  const bf16 *W, *x = norm ? p.xn : piece == FC2 ? p.act : p.attn;
  const float *wg = nullptr, *bias, *gain = nullptr;
  switch (piece) {
    case QKV: W = L.wqkv; wg = L.wg_qkv; bias = L.bf_qkv; break;
    case OUT_SELF: W = L.wo; bias = L.b_o; gain = L.gain_cross; break;
    case Q_CROSS: W = L.wqc; wg = L.wg_qc; bias = L.bf_qc; break;
    case OUT_CROSS: W = L.woc; bias = L.b_oc; gain = L.gain_ffn; break;
    case FC1: W = L.wfc1; wg = L.wg_fc1; bias = L.bf_fc1; break;
    default: W = L.wfc2; bias = L.b_fc2; gain = L.gain_next; break;
  }
  const bf16* tile = W + (size_t)(rt >> 3) * KS * 16384 + (rt & 7) * 128 + t * 1024 + g * 8;
  uint4 wa[kAhead][4];
  auto fetch = [&](int u0) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int u = u0 + kWarps * i;
      if (u >= units) break;
      const bf16* w = tile + (size_t)(u >> 1) * 16384 + (u & 1) * 8192;
      wa[i][0] = ld_stream(w); wa[i][1] = ld_stream(w + 64); wa[i][2] = ld_stream(w + 4096); wa[i][3] = ld_stream(w + 4096 + 64);
    }
  };
  fetch(warp);
  // this thread's row of the epilogue
  const int row = 16 * rt + tid / N, b = tid % N, rr = tid / N;
  const bool live = tid < 16 * N;
  const float bias_row = live ? bias[row] : 0.f, other_row = live ? (norm ? wg : gain)[row] : 0.f;
  if (!wait_units(before, need, p.err, &sm.dead)) return false;
  float xv = 0.f;
  if (!norm && live) xv = p.x[(size_t)row * p.Bp + b];
  if (norm) input_sums<NT>(p, sm, warp, lane);
  if (joined) {                                            // the cross attention's parts, put together
    const int items = p.B * p.H * 8;
#pragma unroll 1
    for (int i = tid; i < items; i += kThreads) {
      const int pair = i >> 3, s0 = pair * p.splits, bb = pair / p.H, hh = pair - bb * p.H;
      float2 ml[kWhisperStepSplits];
      float4 o[kWhisperStepSplits][2];
#pragma unroll
      for (int s = 0; s < kWhisperStepSplits; ++s)
        if (s < p.splits) {
          const float4* part = reinterpret_cast<const float4*>(p.part_o + (size_t)(s0 + s) * kD + 8 * (i & 7));
          ml[s] = *reinterpret_cast<const float2*>(p.part_ml + 2 * (s0 + s));
          o[s][0] = part[0];
          o[s][1] = part[1];
        }
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, m = -CUDART_INF_F, den = 0.f;
#pragma unroll
      for (int s = 0; s < kWhisperStepSplits; ++s)
        if (s < p.splits) m = fmaxf(m, ml[s].x);
#pragma unroll
      for (int s = 0; s < kWhisperStepSplits; ++s)
        if (s < p.splits) {
          const float f = exp2f(ml[s].x - m);
          const float4 o0 = o[s][0], o1 = o[s][1];
          den += f * ml[s].y;
          v[0] += f * o0.x; v[1] += f * o0.y; v[2] += f * o0.z; v[3] += f * o0.w;
          v[4] += f * o1.x; v[5] += f * o1.y; v[6] += f * o1.z; v[7] += f * o1.w;
        }
      const float inv = 1.0f / den;
      *reinterpret_cast<uint4*>(sm.x + (hh * 8 + (i & 7)) * (8 * N) + bb * 8) =
          make_uint4(pack(v[0] * inv, v[1] * inv), pack(v[2] * inv, v[3] * inv), pack(v[4] * inv, v[5] * inv), pack(v[6] * inv, v[7] * inv));
    }
    __syncthreads();
  }
  float acc[NT][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
  for (int u0 = warp; u0 < units; u0 += kWarps * kAhead) {
    if (u0 != warp) fetch(u0);
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int u = u0 + kWarps * i;
      if (u >= units) break;
      uint4 xb[2][NT];
      if (joined) {
        const bf16* xp = sm.x + (8 * u + t) * (8 * N) + g * 8;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) { xb[0][nt] = ld_data(xp + nt * 64); xb[1][nt] = ld_data(xp + 32 * N + nt * 64); }
      } else {
        const bf16* xp = x + (size_t)(8 * u + t) * (p.Bp * 8) + g * 8;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          xb[0][nt] = ld_data(xp + nt * 64);
          xb[1][nt] = ld_data(xp + (size_t)4 * (p.Bp * 8) + nt * 64);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const uint4 a = wa[i][2 * h], c = wa[i][2 * h + 1];
          mma_bf16(acc[nt], a.x, c.x, a.y, c.y, xb[h][nt].x, xb[h][nt].y);
          mma_bf16(acc[nt], a.z, c.z, a.w, c.w, xb[h][nt].z, xb[h][nt].w);
        }
    }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
    float* r = sm.red + (warp * 16 + g) * N + 8 * nt + 2 * t;
    r[0] = acc[nt][0]; r[1] = acc[nt][1]; r[8 * N] = acc[nt][2]; r[8 * N + 1] = acc[nt][3];
  }
  __syncthreads();
  float v = 0.f;
  if (live) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) v += sm.red[(w * 16 + rr) * N + b];
    if (norm) {
      const float2 scale = norm_scale(p, sm, b);
      v = v * scale.x - scale.y * other_row;
    }
    v += bias_row;
  }
  if (!norm) {
    finish_rows<NT>(p, rt, xv + v, other_row, piece == FC2 ? L.capture : nullptr, sm);
  } else if (live && b < p.B) {
    if (piece == FC1) {
      p.act[(size_t)(row >> 3) * (p.Bp * 8) + (b >> 3) * 64 + (b & 7) * 8 + (row & 7)] = __float2bfloat16_rn(gelu_ref(v));
    } else {                                               // rows in the order of the fused q/k/v matrix: 16 of one head, for q and k d and d + 32 in pairs
      const int hs = rt >> 2, jj = rt & 3, d = 8 * jj + (rr & 7) + (rr >> 3) * (kD / 2);
      if (piece == Q_CROSS || hs < p.H) {
        p.q[(size_t)b * p.q_pitch + hs * kD + d] = __float2bfloat16_rn(v * p.qk_scale);
      } else {
        const int pos = p.pos[b];
        if (hs < 2 * p.H) L.kv[b * p.kv_b + (hs - p.H) * p.kv_h + kcache_offset(pos, d, kD)] = __float2bfloat16_rn(v * p.qk_scale);
        else L.kv[b * p.kv_b + (hs - 2 * p.H) * p.kv_h + vcache_offset(pos, 16 * jj + rr, kD)] = __float2bfloat16_rn(v);
      }
    }
  }
  return true;
}

// One sequence's head, or one of `splits` parts of its keys.  Warp w takes every eighth block of 16 keys, two of them in flight; the cross-attention
// cache does not change during the step, so its first two are on their way before the wait.
template <bool CROSS>
__device__ __forceinline__ bool attention_unit(const WhisperStepParams& p, const WhisperStepLayer& L, int unit, const unsigned* before, unsigned need, Shared& sm) {
  const int tid = thread_index(), lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int splits = CROSS ? p.splits : 1, pair = unit / splits, part = unit - pair * splits, b = pair / p.H, h = pair - b * p.H;
  const int T = CROSS ? p.cross_len : p.pos[b] + 1, blocks = (T + 15) >> 4, per = (blocks + splits - 1) / splits;
  const int end = min(blocks, (part + 1) * per);
  const uint4* base = reinterpret_cast<const uint4*>(CROSS ? L.cross + b * p.cross_b + h * p.cross_h : L.kv + b * p.kv_b + h * p.kv_h) + lane;
  uint4 kf[2][4], vf[2][4];
  auto load = [&](int i, int kb) {
    const uint4* blk = base + (size_t)kb * (4 * kD);
#pragma unroll
    for (int k = 0; k < 4; ++k) kf[i][k] = CROSS ? ld_stream(blk + 32 * k) : blk[32 * k];
#pragma unroll
    for (int k = 0; k < 4; ++k) vf[i][k] = CROSS ? ld_stream(blk + 128 + 32 * k) : blk[128 + 32 * k];
  };
  const int kb0 = part * per + warp;
  if (CROSS) {
    if (kb0 < end) load(0, kb0);
    if (kb0 + kWarps < end) load(1, kb0 + kWarps);
  }
  if (!wait_units(before, need, p.err, &sm.dead)) return false;
  if (!CROSS) {
    if (kb0 < end) load(0, kb0);
    if (kb0 + kWarps < end) load(1, kb0 + kWarps);
  }
  uint32_t qf[4][2];                                       // column 0 of the eight is this head
  const bf16* q = p.q + (size_t)b * p.q_pitch + h * kD;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    qf[k][0] = g == 0 ? *reinterpret_cast<const uint32_t*>(q + 16 * k + 2 * t) : 0u;
    qf[k][1] = g == 0 ? *reinterpret_cast<const uint32_t*>(q + 16 * k + 2 * t + 8) : 0u;
  }
  float m = -CUDART_INF_F, l = 0.f, o[4][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) o[k][0] = o[k][1] = o[k][2] = o[k][3] = 0.f;
  auto process = [&](int i, int kb) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 4; ++k) mma_bf16(s, kf[i][k].x, kf[i][k].y, kf[i][k].z, kf[i][k].w, qf[k][0], qf[k][1]);
    const int key = kb * 16 + g;
    if (key >= T) s[0] = -CUDART_INF_F;
    if (key + 8 >= T) s[2] = -CUDART_INF_F;
    float bm = fmaxf(s[0], s[2]);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, off));
    const float mn = fmaxf(m, bm), a = exp2f((m - mn) * kLog2e), p0 = exp2f((s[0] - mn) * kLog2e), p1 = exp2f((s[2] - mn) * kLog2e);
    l = l * a + (p0 + p1);
    m = mn;
    const uint32_t pb0 = movmatrix_trans(pack(p0, 0.f)), pb1 = movmatrix_trans(pack(p1, 0.f));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      o[k][0] *= a; o[k][2] *= a;
      mma_bf16(o[k], vf[i][k].x, vf[i][k].y, vf[i][k].z, vf[i][k].w, pb0, pb1);
    }
  };
  for (int kb = kb0; kb < end; kb += 2 * kWarps) {
    process(0, kb);
    if (kb + 2 * kWarps < end) load(0, kb + 2 * kWarps);
    if (kb + kWarps < end) {
      process(1, kb + kWarps);
      if (kb + 3 * kWarps < end) load(1, kb + 3 * kWarps);
    }
  }
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
  if (t == 0) {
    if (g == 0) { sm.stat[0][warp][0] = m; sm.stat[1][warp][0] = l; }
#pragma unroll
    for (int k = 0; k < 4; ++k) { sm.red[warp * kD + 16 * k + g] = o[k][0]; sm.red[warp * kD + 16 * k + g + 8] = o[k][2]; }
  }
  __syncthreads();
  if (tid < kD) {
    float M = sm.stat[0][0][0], acc = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, sm.stat[0][w][0]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = exp2f((sm.stat[0][w][0] - M) * kLog2e);
      acc += f * sm.red[w * kD + tid];
      sum += f * sm.stat[1][w][0];
    }
    if (splits == 1) {
      const int k = h * kD + tid;
      p.attn[(size_t)(k >> 3) * (p.Bp * 8) + (b >> 3) * 64 + (b & 7) * 8 + (k & 7)] = __float2bfloat16_rn(acc * (1.0f / sum));
    } else {
      p.part_o[(size_t)unit * kD + tid] = acc;
      if (tid == 0) { p.part_ml[2 * unit] = M * kLog2e; p.part_ml[2 * unit + 1] = sum; }
    }
  }
  return true;
}

template <int NT>
__global__ void __launch_bounds__(kThreads, 1) whisper_step_kernel(const __grid_constant__ WhisperStepParams p) {
  __shared__ Shared sm;
  const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x;
  if (tid == 0) sm.dead = 0;
  __syncthreads();
  // units of the pieces, and the CTA that takes a piece's first unit: the short pieces go to CTAs that the one before leaves free, which then have
  // their weights at hand
  const int rows = p.hidden >> 4, n_qkv = 3 * rows, n_self = p.B * p.H, n_cross = n_self * p.splits, n_fc1 = p.ffn >> 4;
  const int at_out = n_self % G, at_qc = (n_self + rows) % G, at_last = (G - rows % G) % G;
  unsigned* c = p.done;
  bool ok = true;
  for (int rt = cta; rt < rows; rt += G) {                 // embedding and position
    constexpr int N = 8 * NT;
    const int row = 16 * rt + tid / N, b = tid % N;
    float xv = 0.f;
    if (tid < 16 * N && b < p.B) {
      const int tok = p.tokens[b];
      xv = tok >= 0 && tok < p.vocab ? __bfloat162float(p.embed[(int64_t)tok * p.hidden + row]) : 0.f;
      xv += p.pos_emb[(int64_t)p.pos[b] * p.hidden + row];
    }
    finish_rows<NT>(p, rt, xv, tid < 16 * N ? p.gain_first[row] : 0.f, nullptr, sm);
    count_unit(c);
  }
  int before = rows;
  constexpr int kWords = sizeof(WhisperStepLayer) / 4;
  static_assert(kWords <= kThreads, "one word of a layer per thread");
  const uint32_t* table = reinterpret_cast<const uint32_t*>(p.layers);
  if (tid < kWords) reinterpret_cast<uint32_t*>(&sm.layer[0])[tid] = table[tid];
#pragma unroll 1
  for (int i = 0; i < 8 * p.n_layers && ok; ++i, ++c) {
    const int piece = i & 7, layer = i >> 3;
    const WhisperStepLayer& L = sm.layer[layer & 1];
    if (piece == 0) {                                      // the next layer's into the other half, which nobody reads any more
      __syncthreads();
      if (tid < kWords && layer + 1 < p.n_layers) reinterpret_cast<uint32_t*>(&sm.layer[(layer + 1) & 1])[tid] = table[(layer + 1) * kWords + tid];
    }
    const int n = piece == QKV ? n_qkv : piece == SELF ? n_self : piece == CROSS ? n_cross : piece == FC1 ? n_fc1 : rows;
    const int first = piece == OUT_SELF ? at_out : piece == Q_CROSS ? at_qc : piece == OUT_CROSS || piece == FC2 ? at_last : 0;
#pragma unroll 1
    for (int u = (cta - first + G) % G; u < n; u += G) {
      if (piece == SELF) ok = attention_unit<false>(p, L, u, c, before, sm);
      else if (piece == CROSS) ok = attention_unit<true>(p, L, u, c, before, sm);
      else ok = gemv_unit<NT>(p, L, piece, u, c, before, sm);
      if (!ok) break;
      count_unit(c + 1);
    }
    before = n;
  }
  // the last CTA out empties the counters for the next step
  const int n_done = 1 + 8 * p.n_layers;
  if (last_block(p.done + n_done, &sm.dead))
    for (int i = tid; i <= n_done; i += kThreads) p.done[i] = 0u;
}

// The tied head, the greedy tokens with their bookkeeping, and the positions.  A warp takes whole tiles of 16 rows, four units of 64 k on their way, so that
// the matrix streams without a barrier (the first units before the layers' kernel is waited for); every CTA leaves its best (logit, id) per sequence, and
// the last one to do so ends the step.  Instead of a launch each for the three.
template <int NT>
__global__ void __launch_bounds__(kThreads, 1) whisper_head_kernel(const __grid_constant__ WhisperStepParams p) {
  __shared__ Shared sm;
  constexpr int N = 8 * NT, kAhead = 4;
  const int tid = thread_index(), lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int tiles = (p.vocab + 15) >> 4, units = p.hidden >> 6, KS = (p.hidden + 127) >> 7, stride = gridDim.x * kWarps;
  uint4 wa[kAhead][4];
  auto fetch = [&](int i, int rt, int u) {
    if (rt >= tiles || u >= units) return;
    const bf16* w = p.head + (size_t)(rt >> 3) * KS * 16384 + (rt & 7) * 128 + t * 1024 + g * 8 + (size_t)(u >> 1) * 16384 + (u & 1) * 8192;
    wa[i][0] = ld_stream(w); wa[i][1] = ld_stream(w + 64); wa[i][2] = ld_stream(w + 4096); wa[i][3] = ld_stream(w + 4096 + 64);
  };
  int rt = blockIdx.x * kWarps + warp;
#pragma unroll
  for (int i = 0; i < kAhead; ++i) fetch(i, rt, i);
  pdl_wait();
  input_sums<NT>(p, sm, warp, lane);
  __syncthreads();
  if (tid < N) {
    const float2 scale = norm_scale(p, sm, tid);
    sm.inv[tid] = scale.x;
    sm.mu[tid] = scale.y;
  }
  __syncthreads();
  float best[NT][2], inv[NT][2], mu[NT][2];
  int id[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      best[nt][j] = -CUDART_INF_F; id[nt][j] = 0x7fffffff;
      inv[nt][j] = sm.inv[8 * nt + 2 * t + j]; mu[nt][j] = sm.mu[8 * nt + 2 * t + j];
    }
#pragma unroll 1
  for (; rt < tiles; rt += stride) {
    float acc[NT][4], wg[2], bias[2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
#pragma unroll
    for (int j = 0; j < 2; ++j) {                          // (padded to whole row groups)
      const int row = 16 * rt + g + 8 * j;
      wg[j] = row < p.vocab ? p.wg_head[row] : 0.f;
      bias[j] = row < p.vocab ? p.bf_head[row] : 0.f;
    }
#pragma unroll 1
    for (int u0 = 0; u0 < units; u0 += kAhead) {
      const bool more = u0 + kAhead < units;
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        if (u0 + i < units) {
          const bf16* xp = p.xn + (size_t)(8 * (u0 + i) + t) * (p.Bp * 8) + g * 8;
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              const uint4 xb = ld_data(xp + (size_t)h * 4 * (p.Bp * 8) + nt * 64), a = wa[i][2 * h], c = wa[i][2 * h + 1];
              mma_bf16(acc[nt], a.x, c.x, a.y, c.y, xb.x, xb.y);
              mma_bf16(acc[nt], a.z, c.z, a.w, c.w, xb.z, xb.w);
            }
        }
        fetch(i, more ? rt : rt + stride, more ? u0 + kAhead + i : i);
      }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = k & 1, r = k >> 1, b = 8 * nt + 2 * t + j, row = 16 * rt + g + 8 * r;
        const float v = acc[nt][k] * inv[nt][j] - mu[nt][j] * wg[r] + bias[r];
        if (b < p.B && row < p.vocab) {
          p.logits[(int64_t)b * p.logits_pitch + row] = v;
          if (v > best[nt][j]) { best[nt][j] = v; id[nt][j] = row; }       // (rows ascend: the first of equals stays)
        }
      }
  }
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, best[nt][j], off);
        const int i = __shfl_xor_sync(0xffffffffu, id[nt][j], off);
        if (v > best[nt][j] || (v == best[nt][j] && i < id[nt][j])) { best[nt][j] = v; id[nt][j] = i; }
      }
      if (g == 0) { sm.stat[0][warp][8 * nt + 2 * t + j] = best[nt][j]; sm.stat[1][warp][8 * nt + 2 * t + j] = __int_as_float(id[nt][j]); }
    }
  __syncthreads();
  if (tid < N) {
    float v = sm.stat[0][0][tid];
    int i = __float_as_int(sm.stat[1][0][tid]);
#pragma unroll
    for (int w = 1; w < kWarps; ++w) {
      const float o = sm.stat[0][w][tid];
      const int oi = __float_as_int(sm.stat[1][w][tid]);
      if (o > v || (o == v && oi < i)) { v = o; i = oi; }
    }
    p.best[blockIdx.x * kWhisperStepBatch + tid] = make_float2(v, __int_as_float(i));
  }
  if (!last_block(p.head_done, &sm.dead)) return;
  for (int b = warp; b < p.B; b += kWarps) {
    const int id = best_of_blocks(p.best + b, kWhisperStepBatch, lane);
    if (lane == 0) {
      keep_token(id, b, p.B, p.tokens, p.hist, p.step_ctr, p.stop);
      if (p.pos[b] < p.limit[b]) p.pos[b] += 1;
    }
  }
  __syncthreads();
  if (tid == 0) {
    *p.step_ctr += 1;
    *p.head_done = 0u;                                     // for the next step
  }
}

int64_t layer_bytes(int n_layers) { return round_up((int64_t)n_layers * sizeof(WhisperStepLayer), 256); }
int64_t counter_bytes(int n_layers) { return round_up((int64_t)(3 + 8 * n_layers) * 4, 256); }

}  // namespace

// D = 64, one key head per query head, and a batch of two MMA column tiles at most: beyond that the weights' tiles of 16 rows are multiplied with four or
// more column tiles and the launched step's tcgen05 GEMVs are used.  With two column tiles only up to a width of 768: at 1024 a sequence's heads are 1.3 to
// 1.7 rounds of the CTAs and the products outweigh the launches.  Launched -> two launches, a step at 1500 cross-attention keys: width 512, six layers, batch 1, 8, 16
// 284 -> 164, 316 -> 187, 343 -> 230 us; 768, twelve 577 -> 393, 662 -> 458, 721 -> 667; 1024, 24 1155 -> 915, 1376 -> 1080; batch 12, 16 1461 -> 1501, 1574 -> 1558
// (380 positions 1556 -> 1631, 1675 -> 1688).  LMB200_WHISPER_STEP=0: launched, 1: wherever it can be (A/B runs).
bool whisper_step_fits(int B, int D, int heads, int kv_heads, int hidden, int ffn, int n_layers) {
  const char* e = getenv("LMB200_WHISPER_STEP");
  if (e && atoi(e) == 0) return false;
  return B <= kWhisperStepBatch && D == kD && heads == kv_heads && hidden == heads * kD && ffn % 64 == 0 && hidden <= kMaxHidden && n_layers <= kWhisperStepLayers &&
         (e || B <= 8 || hidden <= 768);
}

int64_t whisper_step_scratch_bytes(int B, int heads, int n_layers, int sms) { return layer_bytes(n_layers) + counter_bytes(n_layers) + (int64_t)B * heads * kWhisperStepSplits * (kD + 2) * 4 + (int64_t)sms * kWhisperStepBatch * 8; }

int32_t whisper_step_layers(const WhisperStepLayer* layers, int n_layers, void* scratch, cudaStream_t stream) {
  LMB_CUDA(cudaMemcpyAsync(scratch, layers, n_layers * sizeof(WhisperStepLayer), cudaMemcpyHostToDevice, stream));
  LMB_CUDA(cudaStreamSynchronize(stream));
  return LMB200_OK;
}

int32_t whisper_step_launch(Ctx* ctx, WhisperStepParams p, void* scratch, cudaStream_t stream) {
  const int pairs = p.B * p.H, blocks = (p.cross_len + 15) / 16;
  // parts of the cross attention's keys: as many as the CTAs take in one round, of at least a block per warp
  int splits = std::max(1, std::min({kWhisperStepSplits, ctx->sm_count / pairs, blocks / kWarps}));
  splits = (int)ceil_div(blocks, ceil_div(blocks, splits));
  p.splits = splits;
  p.layers = static_cast<const WhisperStepLayer*>(scratch);
  char* s = static_cast<char*>(scratch) + layer_bytes(p.n_layers);
  p.done = reinterpret_cast<unsigned*>(s);
  p.head_done = p.done + 2 + 8 * p.n_layers;
  p.part_o = reinterpret_cast<float*>(s + counter_bytes(p.n_layers));
  p.part_ml = p.part_o + (int64_t)pairs * kWhisperStepSplits * kD;
  p.best = reinterpret_cast<float2*>(p.part_ml + (int64_t)pairs * kWhisperStepSplits * 2);
  p.err = ctx->dev_err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctx->sm_count);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;             // the CTAs wait for one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LMB_CUDA(cudaLaunchKernelEx(&cfg, p.B <= 8 ? whisper_step_kernel<1> : whisper_step_kernel<2>, p));
  ctx->launches++;
  if (!p.with_head) return LMB200_OK;
  LMB_CUDA(launch_k(p.B <= 8 ? whisper_head_kernel<1> : whisper_head_kernel<2>, dim3((unsigned)ctx->sm_count), dim3(kThreads), 0, stream, p));
  ctx->launches++;
  return LMB200_OK;
}

}  // namespace lmb
