// A small float32 Llama's step as one launch.
//
// Five dependent pieces per layer -- q/k/v with the norm in front, attention, o_proj, gate/up with its norm, down_proj -- each a fraction of a microsecond's
// work at a few hundred features.  As launches (two norms, four products, attention and its merge per layer, then head, token and position) a step of the
// small Llama (hidden 256, four layers, vocabulary 1024) is 36 of them, 1.5 to 4 us each.  Here one CTA per SM takes a fixed share of every piece's
// units -- 16 rows of a matrix, or one sequence's query head -- and counts finished units through L2; the weights a unit needs are in registers before it
// starts to wait: 132 -> 58 us a step at 100 keys, one step behind the other (97 us through the host with the logits; hidden 1024, 16 layers, ffn 4096, four sequences of 1000 keys
// 2946 -> 1156; of the 160 sizes measured those that llama_step_fits lets in are 1.09 to 2.8 times faster).  The norms are computed by every unit that reads their row: cheaper than another trip through L2.  Products: a lane holds 8 k of two
// rows (the layout of the launched kernel's tiles), a warp every eighth chunk of 32 k; lanes, then warps, are added in order.
#include "llama_step.cuh"

#include "step.cuh"

#include <algorithm>

namespace lmb {
namespace {

constexpr int kThreads = 256, kWarps = 8, kAhead = 3;
constexpr int kMaxHidden = 4 * kThreads, kMaxFfn = 4096;
constexpr float kLog2e = 1.4426950408889634f, kHalfPi = 1.5707963267948966f;

enum Piece { QKV, ATTEND, OUT, GATE_UP, DOWN, HEAD };

struct Shared {
  float red[kWarps * 16 * kLlamaStepBatch];    // [warp][row][column]; attention: [warp][d], 128 at most
  float attn[kWarps * 128];
  float sum[kLlamaStepBatch][kWarps];
  float best[kLlamaStepBatch][kWarps];
  int best_id[kLlamaStepBatch][kWarps];
  LlamaStepLayer layer[2];                     // the present layer's matrices and the next one's
  int flag;
};

// the residual row before the layers have written it: the token's embedding (out of range: zeros, as _gather_kernel! does, src/Execution.jl:580-595)
__device__ __forceinline__ const float* embedding(const LlamaStepParams& p, int b) {
  const int tok = p.tokens[b];
  return tok >= 0 && tok < p.vocab ? p.embed + (int64_t)tok * p.hidden : nullptr;
}

// Rows 16 rb .. 16 rb + 15 of a matrix times the batch (NB columns), and what the piece does with them.  xs: the input, [column][k].
template <int NB, int DU>
__device__ __forceinline__ bool gemv_unit(const LlamaStepParams& p, const LlamaStepLayer& L, int piece, bool first_layer, int rb, const unsigned* before,
                                          unsigned need, Shared& sm, float* xs) {
  constexpr int D = 16 * DU;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const bool norm = piece == QKV || piece == GATE_UP || piece == HEAD;
  const int K = piece == DOWN ? p.ffn : p.hidden, KC = (K + 31) >> 5;
  const float* W = piece == QKV ? L.wqkv : piece == OUT ? L.wo : piece == GATE_UP ? L.wgu : piece == DOWN ? L.wdown : p.head;
  const float* gain = piece == QKV ? L.gain_attn : piece == GATE_UP ? L.gain_ffn : p.gain_final;
  const float4* tile = reinterpret_cast<const float4*>(W + (size_t)rb * KC * 512 + lane * 16);
  float4 w[kAhead][4];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int c = c0 + kWarps * i;
      if (c >= KC) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) w[i][k] = __ldg(tile + (size_t)c * 128 + k);
    }
  };
  fetch(warp);
  float4 gn = make_float4(0.f, 0.f, 0.f, 0.f);
  if (norm && 4 * tid < K) gn = __ldg(reinterpret_cast<const float4*>(gain) + tid);
  if (need && !wait_units(before, need, p.err, &sm.flag)) return false;
  // the input, a multiple of 32 wide
  const int width = 32 * KC, n4 = K >> 2;
  if (norm) {                                              // (hidden <= 4 kThreads: a thread's four features of every row stay in registers)
    float4 v[NB];
    const bool mine = tid < n4;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      v[b] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (b >= p.B || !mine) continue;
      const float* row = piece == QKV && first_layer ? embedding(p, b) : p.x + (size_t)b * K;
      if (row) v[b] = *reinterpret_cast<const float4*>(row + 4 * tid);
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float ss = v[b].x * v[b].x + v[b].y * v[b].y + v[b].z * v[b].z + v[b].w * v[b].w;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
      if (lane == 0) sm.sum[b][warp] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (b >= p.B || !mine) continue;
      float s = 0.f;
#pragma unroll
      for (int u = 0; u < kWarps; ++u) s += sm.sum[b][u];
      const float inv = 1.0f / sqrtf(s * (1.0f / (float)K) + p.eps);
      *reinterpret_cast<float4*>(xs + b * width + 4 * tid) = make_float4((v[b].x * inv) * gn.x, (v[b].y * inv) * gn.y, (v[b].z * inv) * gn.z, (v[b].w * inv) * gn.w);
    }
  } else {
    const float* src = piece == OUT ? p.attn : p.act;
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (b < p.B)
        for (int i = tid; i < n4; i += kThreads) *reinterpret_cast<float4*>(xs + b * width + 4 * i) = *reinterpret_cast<const float4*>(src + (size_t)b * K + 4 * i);
  }
  if (width != K)                                          // (weights behind K are zero, what lies here may not be a number)
    for (int i = tid; i < NB * (width - K); i += kThreads) xs[(i / (width - K)) * width + K + i % (width - K)] = 0.f;
  __syncthreads();
  float acc[2][NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) acc[0][b] = acc[1][b] = 0.f;
  for (int c0 = warp; c0 < KC; c0 += kWarps * kAhead) {
    if (c0 != warp) fetch(c0);
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int c = c0 + kWarps * i;
      if (c >= KC) continue;
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        if (b >= p.B) continue;
        const float4* x4 = reinterpret_cast<const float4*>(xs + b * width + 32 * c + 8 * t);
        const float4 x0 = x4[0], x1 = x4[1];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 a = w[i][2 * h], e = w[i][2 * h + 1];
          float v = acc[h][b];
          v = fmaf(a.x, x0.x, v); v = fmaf(a.y, x0.y, v); v = fmaf(a.z, x0.z, v); v = fmaf(a.w, x0.w, v);
          v = fmaf(e.x, x1.x, v); v = fmaf(e.y, x1.y, v); v = fmaf(e.z, x1.z, v); v = fmaf(e.w, x1.w, v);
          acc[h][b] = v;
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      float v = acc[h][b];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (t == 0) sm.red[(warp * 16 + 8 * h + g) * NB + b] = v;
    }
  __syncthreads();
  // a thread finishes rows r and r + 8 of one column: the pairs the epilogues combine
  const int r = tid / NB, b = tid % NB;
  if (tid < 8 * NB && b < p.B) {
    float v0 = 0.f, v1 = 0.f;
#pragma unroll
    for (int v = 0; v < kWarps; ++v) { v0 += sm.red[(v * 16 + r) * NB + b]; v1 += sm.red[(v * 16 + 8 + r) * NB + b]; }
    const int row = 16 * rb + r;
    if (piece == QKV) {
      const int hs = rb / DU, jj = rb - hs * DU, pos = p.pos[b];
      if (hs < p.Hl + p.KVl) {                             // rows r and r + 8 are the rotated pair d0, d0 + D / 2; src/NN.jl:253-303
        const int d0 = 8 * jj + r;
        const float ang = (float)pos * p.inv_freq[d0];
        const float sn = sinf(ang), cs = sinf(kHalfPi + ang * -1.0f);   // cos(a) = sin(pi/2 - a)
        const float o0 = v0 * cs + (v1 * sn) * -1.0f, o1 = v0 * sn + v1 * cs;
        if (hs < p.Hl) {
          float* q = p.q + ((size_t)b * p.Hl + hs) * D;
          q[d0] = o0;
          q[d0 + D / 2] = o1;
        } else {
          float* kc = L.kv + b * p.kv_b + (hs - p.Hl) * p.kv_h;
          kc[kcache_offset(pos, d0, D)] = o0;
          kc[kcache_offset(pos, d0 + D / 2, D)] = o1;
        }
      } else {
        float* vc = L.kv + b * p.kv_b + (hs - p.Hl - p.KVl) * p.kv_h;
        vc[vcache_offset(pos, 16 * jj + r, D)] = v0;
        vc[vcache_offset(pos, 16 * jj + r + 8, D)] = v1;
      }
    } else if (piece == GATE_UP) {                         // gate and up; silu as src/HighLevelOps.jl:153-160
      const int o = 8 * rb + r;
      if (o < p.ffn) {
        const float e = exp2f((v0 * -1.0f) * kLog2e);
        const float sg = 1.0f / (1.0f + e);
        p.act[(size_t)b * p.ffn + o] = (v0 * sg) * v1;
      }
    } else if (piece == HEAD) {
      float best = -CUDART_INF_F;
      int id = 0x7fffffff;
      if (row < p.vocab) {
        p.logits[(int64_t)b * p.logits_pitch + row] = v0;
        if (v0 > best) { best = v0; id = row; }
      }
      if (row + 8 < p.vocab) {
        p.logits[(int64_t)b * p.logits_pitch + row + 8] = v1;
        if (v1 > best) { best = v1; id = row + 8; }
      }
      unsigned mask = 0;                                   // the unit's threads lie in one warp, columns are neighbours
#pragma unroll
      for (int v = 0; v < 8; ++v) mask |= ((1u << p.B) - 1u) << (v * NB);
#pragma unroll
      for (int off = NB; off < 8 * NB; off <<= 1) {
        const float o = __shfl_xor_sync(mask, best, off);
        const int oi = __shfl_xor_sync(mask, id, off);
        if (o > best || (o == best && oi < id)) { best = o; id = oi; }
      }
      if (r == 0 && (best > sm.best[b][0] || (best == sm.best[b][0] && id < sm.best_id[b][0]))) { sm.best[b][0] = best; sm.best_id[b][0] = id; }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = row + 8 * h;
        if (o >= p.hidden) continue;
        float* x = p.x + (size_t)b * p.hidden + o;
        float old = 0.f;
        if (piece == OUT && first_layer) { const float* e = embedding(p, b); if (e) old = e[o]; }
        else old = *x;
        const float nx = old + (h ? v1 : v0);
        *x = nx;
        if (piece == DOWN && L.capture) L.capture[(size_t)b * p.hidden + o] = nx;
      }
    }
  }
  return true;
}

// One sequence's query head.  Warp w takes every eighth block of 16 keys; lane (g, t) holds keys g and g + 8, dimensions 2t, 2t + 1, 2t + 8, 2t + 9 of every 16.
template <int DU>
__device__ __forceinline__ bool attention_unit(const LlamaStepParams& p, const LlamaStepLayer& L, int unit, const unsigned* before, unsigned need, Shared& sm) {
  constexpr int D = 16 * DU;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int b = unit / p.Hl, hl = unit - b * p.Hl, T = p.pos[b] + 1, blocks = (T + 15) >> 4;
  if (!wait_units(before, need, p.err, &sm.flag)) return false;
  const float* base = L.kv + b * p.kv_b + (hl / p.G) * p.kv_h + lane * 8;
  float4 qv[DU];
  const float* q = p.q + ((size_t)b * p.Hl + hl) * D;
#pragma unroll
  for (int k = 0; k < DU; ++k) {
    const float2 a = *reinterpret_cast<const float2*>(q + 16 * k + 2 * t), c = *reinterpret_cast<const float2*>(q + 16 * k + 2 * t + 8);
    qv[k] = make_float4(a.x, a.y, c.x, c.y);
  }
  float m = -CUDART_INF_F, l = 0.f, o[DU][2];
#pragma unroll
  for (int k = 0; k < DU; ++k) o[k][0] = o[k][1] = 0.f;
  for (int kb = warp; kb < blocks; kb += kWarps) {
    const float* blk = base + (size_t)kb * (32 * D);
    float4 kf[DU][2], vf[DU][2];
#pragma unroll
    for (int k = 0; k < DU; ++k) {
      kf[k][0] = *reinterpret_cast<const float4*>(blk + 256 * k);
      kf[k][1] = *reinterpret_cast<const float4*>(blk + 256 * k + 4);
    }
#pragma unroll
    for (int k = 0; k < DU; ++k) {
      vf[k][0] = *reinterpret_cast<const float4*>(blk + 256 * (DU + k));
      vf[k][1] = *reinterpret_cast<const float4*>(blk + 256 * (DU + k) + 4);
    }
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int k = 0; k < DU; ++k) {
      s0 = fmaf(qv[k].x, kf[k][0].x, s0); s0 = fmaf(qv[k].y, kf[k][0].y, s0); s0 = fmaf(qv[k].z, kf[k][1].x, s0); s0 = fmaf(qv[k].w, kf[k][1].y, s0);
      s1 = fmaf(qv[k].x, kf[k][0].z, s1); s1 = fmaf(qv[k].y, kf[k][0].w, s1); s1 = fmaf(qv[k].z, kf[k][1].z, s1); s1 = fmaf(qv[k].w, kf[k][1].w, s1);
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1); s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1); s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    s0 = 16 * kb + g < T ? s0 * p.scale : -CUDART_INF_F;             // src/NN.jl:369
    s1 = 16 * kb + g + 8 < T ? s1 * p.scale : -CUDART_INF_F;
    float bm = fmaxf(s0, s1);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, off));
    const float mn = fmaxf(m, bm), a = exp2f((m - mn) * kLog2e);     // exp(x) = exp2(x * 1/ln2), src/HighLevelOps.jl:127-129
    const float p0 = exp2f((s0 - mn) * kLog2e), p1 = exp2f((s1 - mn) * kLog2e);
    l = l * a + (p0 + p1);
    m = mn;
    if (16 * kb + 16 > T) {            // what lies behind the context may be no number (an earlier request's), which a weight of 0 would not stop
#pragma unroll
      for (int k = 0; k < DU; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int key = 16 * kb + 2 * t + 8 * h;
          if (key >= T) vf[k][h].x = vf[k][h].z = 0.f;
          if (key + 1 >= T) vf[k][h].y = vf[k][h].w = 0.f;
        }
    }
    const float pa = __shfl_sync(0xffffffffu, p0, 8 * t), pb = __shfl_sync(0xffffffffu, p0, 8 * t + 4);
    const float pc = __shfl_sync(0xffffffffu, p1, 8 * t), pd = __shfl_sync(0xffffffffu, p1, 8 * t + 4);
#pragma unroll
    for (int k = 0; k < DU; ++k) {
      float u = o[k][0] * a, v = o[k][1] * a;
      u = fmaf(pa, vf[k][0].x, u); u = fmaf(pb, vf[k][0].y, u); u = fmaf(pc, vf[k][1].x, u); u = fmaf(pd, vf[k][1].y, u);
      v = fmaf(pa, vf[k][0].z, v); v = fmaf(pb, vf[k][0].w, v); v = fmaf(pc, vf[k][1].z, v); v = fmaf(pd, vf[k][1].w, v);
      o[k][0] = u; o[k][1] = v;
    }
  }
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
#pragma unroll
  for (int k = 0; k < DU; ++k)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float v = o[k][h];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      if (t == 0) sm.attn[warp * D + 16 * k + 8 * h + g] = v;
    }
  if (lane == 0) { sm.sum[0][warp] = m; sm.sum[1][warp] = l; }
  __syncthreads();
  if (tid < D) {
    float M = sm.sum[0][0], acc = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 1; w < kWarps; ++w) M = fmaxf(M, sm.sum[0][w]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = exp2f((sm.sum[0][w] - M) * kLog2e);
      acc += f * sm.attn[w * D + tid];
      sum += f * sm.sum[1][w];
    }
    p.attn[((size_t)b * p.Hl + hl) * D + tid] = acc * (1.0f / sum);
  }
  return true;
}

template <int NB, int DU>
__global__ void __launch_bounds__(kThreads, 1) llama_step_kernel(const __grid_constant__ LlamaStepParams p) {
  extern __shared__ __align__(16) float xs[];
  __shared__ Shared sm;
  const int G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWords = sizeof(LlamaStepLayer) / 4;
  const uint32_t* table = reinterpret_cast<const uint32_t*>(p.layers);
  if (tid < kWords) reinterpret_cast<uint32_t*>(&sm.layer[0])[tid] = table[tid];
  if (tid == 0) sm.flag = 0;
  if (tid < kLlamaStepBatch) { sm.best[tid][0] = -CUDART_INF_F; sm.best_id[tid][0] = 0x7fffffff; }
  __syncthreads();
  // units of the pieces, and the CTA that takes a piece's first unit: where the piece before left room, so that the weights are at hand
  const int n_qkv = (p.Hl + 2 * p.KVl) * DU, n_att = p.B * p.Hl, n_out = (p.hidden + 15) >> 4, n_gu = (2 * p.ffn + 15) >> 4, n_head = (p.vocab + 15) >> 4;
  const int at_att = n_qkv % G, at_out = (n_qkv + n_att) % G, at_gu = (at_out + n_out) % G, at_down = (at_gu + n_gu) % G;
  unsigned* c = p.done;                                    // [pieces + 1] finished units, from the second on
  unsigned before = 0;
  bool ok = true;
  const int pieces = 5 * p.n_layers + (p.with_head ? 1 : 0);
#pragma unroll 1
  for (int i = 0; i < pieces && ok; ++i, ++c) {
    const int layer = i / 5, piece = layer < p.n_layers ? i - 5 * layer : (int)HEAD;
    if (piece == QKV) {                                    // the next layer's into the other half, which nobody reads any more
      __syncthreads();
      if (tid < kWords && layer + 1 < p.n_layers) reinterpret_cast<uint32_t*>(&sm.layer[(layer + 1) & 1])[tid] = table[(layer + 1) * kWords + tid];
    }
    const LlamaStepLayer& L = sm.layer[layer & 1];
    const int n = piece == QKV ? n_qkv : piece == ATTEND ? n_att : piece == GATE_UP ? n_gu : piece == HEAD ? n_head : n_out;
    const int first = piece == ATTEND ? at_att : piece == OUT ? at_out : piece == GATE_UP ? at_gu : piece == DOWN ? at_down : 0;
#pragma unroll 1
    for (int u = (cta - first + G) % G; u < n; u += G) {
      if (piece == ATTEND) ok = attention_unit<DU>(p, L, u, c, before, sm);
      else ok = gemv_unit<NB, DU>(p, L, piece, layer == 0, u, c, before, sm, xs);
      if (!ok) break;
      if (piece == HEAD) __syncthreads();                  // (counted once per CTA, below)
      else count_unit(c + 1);
    }
    before = (unsigned)n;
  }
  if (p.with_head) {
    __syncthreads();
    if (tid < p.B) p.best[cta * kLlamaStepBatch + tid] = make_float2(sm.best[tid][0], __int_as_float(sm.best_id[tid][0]));
  }
  // the last CTA out chooses the tokens, moves the positions and empties the counters for the next step
  if (!last_block(p.done, &sm.flag)) return;
  for (int b = warp; b < p.B; b += kWarps) {
    if (p.with_head) {
      const int id = best_of_blocks(p.best + b, kLlamaStepBatch, lane);
      if (lane == 0) keep_token(id, b, p.B, p.tokens, p.hist, p.step_ctr, p.stop);
    }
    if (lane == 0 && p.pos[b] < p.limit[b]) p.pos[b] += 1;
  }
  __syncthreads();
  if (tid == 0) *p.step_ctr += 1;
  for (int i = tid; i <= pieces; i += kThreads) p.done[i] = 0u;
}

int64_t layer_bytes(int n_layers) { return round_up((int64_t)n_layers * sizeof(LlamaStepLayer), 256); }
int64_t counter_bytes(int n_layers) { return round_up((int64_t)(2 + 5 * n_layers) * 4, 256); }

typedef void (*Kernel)(LlamaStepParams);
Kernel kernel_of(int B, int D) {
  if (B == 1) return D == 32 ? llama_step_kernel<1, 2> : D == 64 ? llama_step_kernel<1, 4> : llama_step_kernel<1, 8>;
  return D == 32 ? llama_step_kernel<4, 2> : D == 64 ? llama_step_kernel<4, 4> : llama_step_kernel<4, 8>;
}

}  // namespace

// Sizes up to which the one launch was measured to be the faster way (and what its shared memory and registers hold); a context longer than 1024 keys would be
// one CTA's work per head, which the launched attention splits.  The head is the part that loses: a CTA takes its 16-row units one after the other, 1.1 us each
// with one sequence and 2.2 with four, where the launched product streams the matrix; a layer gains 4 to 17 us at short contexts.  Launched -> one launch, 8 keys:
// hidden 64, one layer, vocabulary 32768, one and four sequences 34 -> 42, 35 -> 62 us; 256, one layer, 16384 43 -> 33, 43 -> 46; 256, four layers, 65536
// 145 -> 111, 152 -> 158; 1024 with 32 heads, 16 layers, 65536 895 -> 701, 960 -> 1054; 1024, 16 layers, 32000, four 1337 -> 958.
bool llama_step_fits(int B, int D, int hidden, int ffn, int vocab, int n_layers, int capacity) {
  return B <= kLlamaStepBatch && (D == 32 || D == 64 || D == 128) && hidden % 4 == 0 && ffn % 4 == 0 && hidden <= kMaxHidden && ffn <= kMaxFfn && capacity <= 1024 &&
         vocab <= (B <= 2 ? 65536 : 32768) && (int64_t)vocab * (1 + B) <= 32768ll * n_layers && n_layers <= 64;
}

int64_t llama_step_scratch_bytes(int n_layers, int sms) { return layer_bytes(n_layers) + counter_bytes(n_layers) + (int64_t)sms * kLlamaStepBatch * 8; }

int32_t llama_step_layers(const LlamaStepLayer* layers, int n_layers, void* scratch, cudaStream_t stream) {
  LMB_CUDA(cudaMemcpyAsync(scratch, layers, n_layers * sizeof(LlamaStepLayer), cudaMemcpyHostToDevice, stream));
  LMB_CUDA(cudaStreamSynchronize(stream));
  return LMB200_OK;
}

int32_t llama_step_launch(Ctx* ctx, LlamaStepParams p, int D, void* scratch, cudaStream_t stream) {
  p.layers = static_cast<const LlamaStepLayer*>(scratch);
  char* s = static_cast<char*>(scratch) + layer_bytes(p.n_layers);
  p.done = reinterpret_cast<unsigned*>(s);
  p.best = reinterpret_cast<float2*>(s + counter_bytes(p.n_layers));
  p.err = ctx->dev_err;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctx->sm_count);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)(p.B == 1 ? 1 : kLlamaStepBatch) * 32 * std::max(ceil_div(p.hidden, 32), ceil_div(p.ffn, 32)) * 4;
  if (cfg.dynamicSmemBytes > 40 * 1024)
    LMB_CUDA(cudaFuncSetAttribute(kernel_of(p.B, D), cudaFuncAttributeMaxDynamicSharedMemorySize, kLlamaStepBatch * kMaxFfn * 4));
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;             // the CTAs wait for one another
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LMB_CUDA(cudaLaunchKernelEx(&cfg, kernel_of(p.B, D), p));
  ctx->launches++;
  return LMB200_OK;
}

}  // namespace lmb
