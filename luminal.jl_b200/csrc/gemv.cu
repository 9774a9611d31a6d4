// Bandwidth-bound decode GEMV with fused epilogues (store / SiLU-gate / RoPE + KV append).
//
// bf16 kernels: stream-K over bulk-TMA.  Weights and activations sit in HBM in the tensor-core
// canonical K-major layout (common.cuh), cut into units of 128 rows x 128 k = one contiguous
// 32 KB block; the grid is one CTA per SM and CTA c takes the contiguous unit range
// [c*U/G, (c+1)*U/G), so every SM streams the same number of bytes in a single wave whatever the
// matrix shape.  A producer warp keeps a ring of 5 shared-memory stages full with cp.async.bulk
// copies (one 32 KB copy of weights, evict-first, + the matching activation slice) signalled
// through mbarriers.  One thread issues tcgen05.mma (M = 128 rows, N = batch padding, K = 16)
// straight from the stage through shared-memory descriptors, accumulators double-buffered in
// TMEM; tcgen05.commit hands the stage back to the producer; four epilogue warps read the
// accumulators with tcgen05.ld (one row per thread) and run the fused epilogue while the next
// row group is already being multiplied.
// When a CTA's range leaves a row group its partial result is folded: alone -> epilogue; shared
// -> global scratch + counter, the last contributor sums the parts in CTA order (deterministic).
//
// float32 ("ring") kernel: weights streamed by plain loads through a register ring, fp32 FMAs --
// the parity path.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "gemv.cuh"
#include "pdl.cuh"
#include "tc.cuh"

namespace lmb {

namespace {

constexpr float kInvLn2 = 1.4426950408889634f;      // Float32(1/log(2)) as the reference rounds it
constexpr float kHalfPi = 1.5707963267948966f;
constexpr size_t kMaxSmem = 224 * 1024;

int g_variant = GEMV_TCGEN05;

// gelu(a) = a*0.5*(1 + tanh(0.7978845608*a*(1 + 0.044715*a*a))), tanh(z) = sigmoid(2z)*2 - 1,
// sigmoid through exp2 -- the reference's decomposition, src/HighLevelOps.jl:153-168
__device__ __forceinline__ float gelu_ref(float a) {
  const float inner = (0.7978845608f * a) * (1.0f + (0.044715f * a) * a);
  const float z = inner * 2.0f;
  const float sg = 1.0f / (1.0f + exp2f((z * -1.0f) * kInvLn2));
  const float th = sg * 2.0f + -1.0f;
  return (a * 0.5f) * (1.0f + th);
}

// ---------------------------------------------------------------------------------------------
// Epilogue over a finished tile in shared memory: tile[r * RP + b], r < RPC rows of the CTA's row
// group starting at logical internal row row0.
// ---------------------------------------------------------------------------------------------
template <typename WT>
__device__ __forceinline__ void run_epilogue(const GemvParams& p, const float* tile, int RPC, int RP, int Bp,
                                             int row0, int tid, int nthreads) {
  if (p.epi == EPI_STORE_F32) {
    for (int i = tid; i < RPC * Bp; i += nthreads) {
      const int b = i / RPC, r = i - b * RPC;
      const int row = row0 + r;
      if (b < p.B && row < p.rows)
        p.out[(int64_t)b * p.out_pitch + row] = tile[r * RP + b] + (p.bias ? p.bias[row] : 0.f);
    }
  } else if (p.epi == EPI_GELU_ACT) {
    WT* act = reinterpret_cast<WT*>(p.act);
    for (int i = tid; i < RPC * Bp; i += nthreads) {
      const int b = i / RPC, r = i - b * RPC;
      const int row = row0 + r;
      if (b < p.B && row < p.n_act)
        act[Layout<WT>::x_offset(b, row, Bp)] = from_f32<WT>(gelu_ref(tile[r * RP + b] + (p.bias ? p.bias[row] : 0.f)));
    }
  } else if (p.epi == EPI_SILU_GATE) {
    WT* act = reinterpret_cast<WT*>(p.act);
    for (int i = tid; i < (RPC / 2) * Bp; i += nthreads) {
      const int b = i / (RPC / 2), j = i - b * (RPC / 2);
      const int m = j >> 3, r = j & 7;
      const int o = row0 / 2 + j;
      if (b < p.B && o < p.n_act) {
        const float a = tile[(16 * m + r) * RP + b], u = tile[(16 * m + r + 8) * RP + b];
        // silu(a) = a * (1 / (1 + exp2((a * -1) * (1/ln2))))     src/HighLevelOps.jl:153-160
        const float e = exp2f((a * -1.0f) * kInvLn2);
        const float sg = 1.0f / (1.0f + e);
        act[Layout<WT>::x_offset(b, o, Bp)] = from_f32<WT>((a * sg) * u);
      }
    }
  } else {  // EPI_QKV_ROPE
    WT* q_out = reinterpret_cast<WT*>(p.q_out);
    WT* kv = reinterpret_cast<WT*>(p.kv_layer);
    const int D = p.D, tiles_per_head = D >> 4, half = D >> 1;
    for (int i = tid; i < (RPC / 2) * Bp; i += nthreads) {
      const int b = i / (RPC / 2), j = i - b * (RPC / 2);
      const int m = j >> 3, r = j & 7;
      const int gt = row0 / 16 + m;                  // global 16-row tile
      if (b >= p.B || gt >= p.RB) continue;
      const int pos = p.pos[b];                      // every sequence has its own position
      const float fpos = (float)pos;
      const int hs = gt / tiles_per_head, jj = gt - hs * tiles_per_head;
      float v0 = tile[(16 * m + r) * RP + b], v1 = tile[(16 * m + r + 8) * RP + b];
      if (p.bias) { v0 += p.bias[gt * 16 + r]; v1 += p.bias[gt * 16 + r + 8]; }
      if (hs < p.Hl + p.KVl) {
        // rows r / r+8 of the tile are the RoPE pair (d0, d0 + D/2)      src/NN.jl:253-303
        const int d0 = 8 * jj + r;
        float o0, o1;
        if (p.rope) {
          const float ang = fpos * p.inv_freq[d0];
          const float sn = sinf(ang);
          const float cs = sinf(kHalfPi + ang * -1.0f);   // cos(a) = sin(pi/2 - a)
          o0 = v0 * cs + (v1 * sn) * -1.0f;
          o1 = v0 * sn + v1 * cs;
        } else {
          o0 = v0 * p.qk_scale;
          o1 = v1 * p.qk_scale;
        }
        if (hs < p.Hl) {
          WT* q = q_out + (int64_t)b * p.q_pitch + hs * D;
          q[d0] = from_f32<WT>(o0);
          q[d0 + half] = from_f32<WT>(o1);
        } else {
          WT* kc = kv + b * p.kv_batch_stride + (hs - p.Hl) * p.kv_head_stride;
          kc[kcache_offset(pos, d0, D)] = from_f32<WT>(o0);
          kc[kcache_offset(pos, d0 + half, D)] = from_f32<WT>(o1);
        }
      } else {
        WT* vc = kv + b * p.kv_batch_stride + (hs - p.Hl - p.KVl) * p.kv_head_stride;
        const int d = 16 * jj + r;
        vc[vcache_offset(pos, d, D)] = from_f32<WT>(v0);
        vc[vcache_offset(pos, d + 8, D)] = from_f32<WT>(v1);
      }
    }
  }
}

// sum `n` partial tiles (dense [RPC*Bp] each, `stride` floats apart) into tile[r*RP+b]
__device__ __forceinline__ void sum_partials(float* tile, const float* part, int n, int64_t stride, int RPC, int RP,
                                             int Bp, int tid, int nthreads) {
  const int total = RPC * Bp;
  for (int i0 = tid; i0 < total; i0 += nthreads * 4) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < n; ++k) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i = i0 + j * nthreads;
        if (i < total) s[j] += __ldcg(part + (int64_t)k * stride + i);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = i0 + j * nthreads;
      if (i < total) { const int r = i / Bp, b = i - r * Bp; tile[r * RP + b] = s[j]; }
    }
  }
}

// =============================================================================================
// ring kernel
// =============================================================================================
constexpr int kRingThreads = 256;

template <typename WT> struct Unit;   // 16 rows x 32 k of weights as seen by one lane
template <> struct Unit<__nv_bfloat16> { uint4 v[2]; };
template <> struct Unit<float> { uint4 v[4]; };

template <typename WT>
__device__ __forceinline__ void load_unit(Unit<WT>& u, const WT* W, int64_t rb, int KC, int kc, int lane) {
  constexpr int N = sizeof(Unit<WT>) / 16;
  const uint4* p = reinterpret_cast<const uint4*>(W + ((rb * KC + kc) * 32 + lane) * 16);
#pragma unroll
  for (int i = 0; i < N; ++i) u.v[i] = __ldcs(p + i);
}
template <typename WT>
__device__ __forceinline__ void zero_unit(Unit<WT>& u) {
  constexpr int N = sizeof(Unit<WT>) / 16;
#pragma unroll
  for (int i = 0; i < N; ++i) u.v[i] = make_uint4(0, 0, 0, 0);
}

template <typename WT, int NB, int MT, int STAGES>
__global__ void __launch_bounds__(kRingThreads, 1) gemv_ring_kernel(const GemvParams p) {
  constexpr int Bp = 8 * NB;
  constexpr int RPC = 2 * MT * 16;
  constexpr bool kBf16 = std::is_same<WT, __nv_bfloat16>::value;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WT* xs = reinterpret_cast<WT*>(smem_raw);           // [chunks][Bp][32], a copy of the global slice
  float* red = reinterpret_cast<float*>(smem_raw);
  __shared__ int s_last;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rg = warp >> 2, kw = warp & 3;
  const int kc0 = blockIdx.y * p.kc_per_split;
  const int kc1 = min(p.KC, kc0 + p.kc_per_split);
  const int64_t rb_base = (int64_t)blockIdx.x * (2 * MT) + rg * MT;
  const WT* W = reinterpret_cast<const WT*>(p.W);

  pdl_launch_dependents();
  // prefetch the first weight units before touching the activations
  Unit<WT> ring[STAGES][MT];
#pragma unroll
  for (int s = 0; s < STAGES; ++s) {
    const int kc = kc0 + kw + 4 * s;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      if (s < STAGES - 1 && kc < kc1 && rb_base + mt < p.RB) load_unit<WT>(ring[s][mt], W, rb_base + mt, p.KC, kc, lane);
      else zero_unit<WT>(ring[s][mt]);
    }
  }
  pdl_wait();      // everything below reads or writes what earlier kernels produced
  {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const WT*>(p.x) + (int64_t)kc0 * Bp * 32);
    uint4* dst = reinterpret_cast<uint4*>(xs);
    const int nvec = (kc1 - kc0) * Bp * 32 * (int)sizeof(WT) / 16;
#pragma unroll 8
    for (int i = tid; i < nvec; i += kRingThreads) dst[i] = src[i];
  }
  __syncthreads();

  float acc[MT][kBf16 ? NB : 2 * Bp][kBf16 ? 4 : 1];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < (kBf16 ? NB : 2 * Bp); ++j)
#pragma unroll
      for (int k = 0; k < (kBf16 ? 4 : 1); ++k) acc[i][j][k] = 0.f;

  for (int base = kc0 + kw; base < kc1; base += 4 * STAGES) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      const int cur = base + 4 * s;
      if (cur < kc1) {
        const int nxt = cur + 4 * (STAGES - 1);      // refill the slot freed by the previous iteration
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          if (nxt < kc1 && rb_base + mt < p.RB)
            load_unit<WT>(ring[(s + STAGES - 1) % STAGES][mt], W, rb_base + mt, p.KC, nxt, lane);
        }
        const WT* xc = xs + (cur - kc0) * (Bp * 32) + 8 * t;
        if constexpr (kBf16) {
          uint4 bx[NB];
#pragma unroll
          for (int nt = 0; nt < NB; ++nt) bx[nt] = *reinterpret_cast<const uint4*>(xc + (8 * nt + g) * 32);
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const uint4 lo = ring[s][mt].v[0], hi = ring[s][mt].v[1];
#pragma unroll
            for (int nt = 0; nt < NB; ++nt) {
              mma_bf16(acc[mt][nt], lo.x, hi.x, lo.y, hi.y, bx[nt].x, bx[nt].y);
              mma_bf16(acc[mt][nt], lo.z, hi.z, lo.w, hi.w, bx[nt].z, bx[nt].w);
            }
          }
        } else {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const float4 l0 = *reinterpret_cast<const float4*>(&ring[s][mt].v[0]);
            const float4 l1 = *reinterpret_cast<const float4*>(&ring[s][mt].v[1]);
            const float4 h0 = *reinterpret_cast<const float4*>(&ring[s][mt].v[2]);
            const float4 h1 = *reinterpret_cast<const float4*>(&ring[s][mt].v[3]);
#pragma unroll
            for (int c = 0; c < Bp; ++c) {
              const float4 x0 = *reinterpret_cast<const float4*>(xc + c * 32);
              const float4 x1 = *reinterpret_cast<const float4*>(xc + c * 32 + 4);
              float lo = acc[mt][2 * c][0], hi = acc[mt][2 * c + 1][0];
              lo = fmaf(l0.x, x0.x, lo); lo = fmaf(l0.y, x0.y, lo); lo = fmaf(l0.z, x0.z, lo); lo = fmaf(l0.w, x0.w, lo);
              lo = fmaf(l1.x, x1.x, lo); lo = fmaf(l1.y, x1.y, lo); lo = fmaf(l1.z, x1.z, lo); lo = fmaf(l1.w, x1.w, lo);
              hi = fmaf(h0.x, x0.x, hi); hi = fmaf(h0.y, x0.y, hi); hi = fmaf(h0.z, x0.z, hi); hi = fmaf(h0.w, x0.w, hi);
              hi = fmaf(h1.x, x1.x, hi); hi = fmaf(h1.y, x1.y, hi); hi = fmaf(h1.z, x1.z, hi); hi = fmaf(h1.w, x1.w, hi);
              acc[mt][2 * c][0] = lo; acc[mt][2 * c + 1][0] = hi;
            }
          }
        }
      }
    }
  }
  __syncthreads();   // everyone is done with xs; reuse the memory for the k-warp reduction

  // red[kw][r][b] (row pitch RP = Bp+1 against bank conflicts), r = row inside the CTA tile
  constexpr int RP = Bp + 1;
  constexpr int SLAB = RPC * RP;
  {
    float* mine = red + kw * SLAB;
    if constexpr (kBf16) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int r0 = (rg * MT + mt) * 16 + g;
#pragma unroll
        for (int nt = 0; nt < NB; ++nt) {
          const int c = 8 * nt + 2 * t;
          mine[r0 * RP + c] = acc[mt][nt][0];
          mine[r0 * RP + c + 1] = acc[mt][nt][1];
          mine[(r0 + 8) * RP + c] = acc[mt][nt][2];
          mine[(r0 + 8) * RP + c + 1] = acc[mt][nt][3];
        }
      }
    } else {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const int r0 = (rg * MT + mt) * 16 + g;
#pragma unroll
        for (int c = 0; c < Bp; ++c) {
          float lo = acc[mt][2 * c][0], hi = acc[mt][2 * c + 1][0];
          lo += __shfl_xor_sync(0xffffffffu, lo, 1);
          lo += __shfl_xor_sync(0xffffffffu, lo, 2);
          hi += __shfl_xor_sync(0xffffffffu, hi, 1);
          hi += __shfl_xor_sync(0xffffffffu, hi, 2);
          if (t == 0) {
            mine[r0 * RP + c] = lo;
            mine[(r0 + 8) * RP + c] = hi;
          }
        }
      }
    }
  }
  __syncthreads();
  // sum the 4 k-warp slabs into slab 0 (each thread owns its (r,b) positions: no hazard)
  for (int i = tid; i < RPC * Bp; i += kRingThreads) {
    const int r = i / Bp, b = i - r * Bp, o = r * RP + b;
    red[o] = (red[o] + red[SLAB + o]) + (red[2 * SLAB + o] + red[3 * SLAB + o]);
  }
  if (p.ksplit > 1) {
    float* my_part = p.partials + ((int64_t)blockIdx.x * p.ksplit + blockIdx.y) * (RPC * Bp);
    for (int i = tid; i < RPC * Bp; i += kRingThreads) {
      const int r = i / Bp, b = i - r * Bp;
      my_part[i] = red[r * RP + b];
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      const unsigned prev = atomicAdd(&p.counters[blockIdx.x], 1u);
      s_last = (prev == (unsigned)p.ksplit - 1u);
    }
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) p.counters[blockIdx.x] = 0u;   // ready for the next launch
    __threadfence();
    sum_partials(red, p.partials + (int64_t)blockIdx.x * p.ksplit * (RPC * Bp), p.ksplit, RPC * Bp, RPC, RP, Bp, tid,
                 kRingThreads);
  }
  __syncthreads();
  run_epilogue<WT>(p, red, RPC, RP, Bp, blockIdx.x * RPC, tid, kRingThreads);
}

// =============================================================================================
// bf16 stream-K kernels
// =============================================================================================
constexpr int kStages = 5;
constexpr int kWStage = 32768;                   // 128 rows x 128 k, bf16
constexpr long long kWaitLimit = 4000000000LL;   // clock cycles (~2 s) before a wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  After a time-out the thread stops waiting for good (`dead`), so control flow --
// and with it every barrier -- stays the same for all threads; the launch is flagged as failed.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, bool& dead, int* err) {
  if (dead) return;
  if (mbar_try_wait(bar, parity)) return;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > kWaitLimit) {
      dead = true;
      if (err) atomicExch(err, 1);
      return;
    }
  }
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}

// The producer warp's last act: one 32 KB L2 prefetch per lane and round over this CTA's share of the
// next GEMV's weight heads (see GemvParams::pf_base).
__device__ __forceinline__ void prefetch_next_weights(const GemvParams& p, int lane) {
  if (!p.pf_base) return;
  const long long total = (long long)p.pf_parts * p.pf_chunk;
  const int n0 = (int)((long long)blockIdx.x * total / gridDim.x), n1 = (int)((long long)(blockIdx.x + 1) * total / gridDim.x);
  for (int n = n0 + lane; n < n1; n += 32) {
    const int part = n / p.pf_chunk, within = n - part * p.pf_chunk;
    const long long unit = (long long)part * p.pf_units / p.pf_parts + within;
    const char* a = reinterpret_cast<const char*>(p.pf_base) + unit * 32768;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(a), "r"(32768u) : "memory");
  }
}

struct UnitRange {
  int KS, nrbg, u0, u1;
  long long U, G;
};
__device__ __forceinline__ UnitRange unit_range(const GemvParams& p) {
  UnitRange ur;
  ur.KS = (p.K + 127) >> 7;
  ur.nrbg = (p.rows + 127) >> 7;
  ur.U = (long long)ur.nrbg * ur.KS;
  ur.G = gridDim.x;
  ur.u0 = (int)((long long)blockIdx.x * ur.U / ur.G);
  ur.u1 = (int)((long long)(blockIdx.x + 1) * ur.U / ur.G);
  return ur;
}
// CTAs that share row group r: CTA of unit u is ceil((u+1)*G/U) - 1
__device__ __forceinline__ void contributors(const UnitRange& ur, int r, int* c_first, int* n) {
  const long long ua = (long long)r * ur.KS, ub = ua + ur.KS - 1;
  *c_first = (int)(((ua + 1) * ur.G + ur.U - 1) / ur.U) - 1;
  const int c_last = (int)(((ub + 1) * ur.G + ur.U - 1) / ur.U) - 1;
  *n = c_last - *c_first + 1;
}

// producer loop shared by both kernels: one 32 KB weight copy + one activation copy per unit
template <int Bp>
__device__ __forceinline__ void produce(const GemvParams& p, const UnitRange& ur, unsigned char* smem,
                                        uint64_t* full_bar, uint64_t* empty_bar, int lane, int* err) {
  constexpr int kXStage = Bp * 256;
  constexpr int kStage = kWStage + kXStage;
  uint64_t pol_w, pol_x;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol_w));
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(pol_x));
  const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(p.W);
  const __nv_bfloat16* X = reinterpret_cast<const __nv_bfloat16*>(p.x);
  bool dead = false;
  // The weights never change: the first stages' weight copies go out before this kernel waits for
  // its predecessor; the activation copies (and everything else) come after the wait.
  const int n_units = ur.u1 - ur.u0;
  const int n_pre = n_units < kStages ? n_units : kStages;
  if (lane == 0) {
    for (int it = 0; it < n_pre; ++it) {
      const int u = ur.u0 + it;
      const int r = u / ur.KS, ks = u - r * ur.KS;
      mbar_expect_tx(&full_bar[it], (uint32_t)kStage);
      bulk_g2s(smem + it * kStage, W + ((int64_t)r * ur.KS + ks) * 16384, (uint32_t)kWStage, &full_bar[it], pol_w);
    }
  }
  pdl_wait();
  if (lane == 0) {
    for (int it = 0; it < n_pre; ++it) {
      const int ks = (ur.u0 + it) % ur.KS;
      bulk_g2s(smem + it * kStage + kWStage, X + (int64_t)ks * (128 * Bp), (uint32_t)kXStage, &full_bar[it], pol_x);
    }
  }
  __syncwarp();
  int it = n_pre;
  for (int u = ur.u0 + n_pre; u < ur.u1; ++u, ++it) {
    const int s = it % kStages, k = it / kStages;
    mbar_wait(&empty_bar[s], (k & 1) ^ 1, dead, err);
    const int r = u / ur.KS, ks = u - r * ur.KS;
    if (lane == 0) {
      unsigned char* st = smem + s * kStage;
      mbar_expect_tx(&full_bar[s], (uint32_t)kStage);
      bulk_g2s(st, W + ((int64_t)r * ur.KS + ks) * 16384, (uint32_t)kWStage, &full_bar[s], pol_w);
      bulk_g2s(st + kWStage, X + (int64_t)ks * (128 * Bp), (uint32_t)kXStage, &full_bar[s], pol_x);
    }
    __syncwarp();
  }
  prefetch_next_weights(p, lane);
}

// ---------------------------------------------------------------------------------------------
// tcgen05 variant
// ---------------------------------------------------------------------------------------------
constexpr int kTcThreads = 6 * 32;    // warp 0 producer, warp 1 MMA issue + TMEM, warps 2..5 epilogue

__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  // K-major, no swizzle: start address, leading (K-direction) and stride (M/N-direction) byte
  // offsets between 8x8 core matrices, all in 16-byte units; bit 46 = descriptor version 1.
  return (uint64_t)((saddr & 0x3FFFF) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) |
         ((uint64_t)(sbo_bytes >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
using tc::elect_one;
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

template <int N> __device__ __forceinline__ void tmem_load_row(float (&v)[N], uint32_t taddr);
template <>
__device__ __forceinline__ void tmem_load_row<32>(float (&v)[32], uint32_t taddr) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
template <>
__device__ __forceinline__ void tmem_load_row<16>(float (&v)[16], uint32_t taddr) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// What a row's epilogue reads besides the accumulators; the chain kernel fetches it while the weights stream.
struct RowConst { float wg, bias, inv_freq, sn, cs; int pos; };      // sn, cs: the rotation where all sequences are at one position
__device__ __forceinline__ RowConst row_const(const GemvParams& p, int row) {
  RowConst rc = {0.f, 0.f, 0.f, 0.f, p.qk_scale, 0};               // (no rotation: q and k rows are only scaled)
  if (row < p.rows) {
    if (p.ln_wg) rc.wg = p.ln_wg[row];
    if (p.bias) rc.bias = p.bias[row];
  }
  if (p.epi == EPI_QKV_ROPE) {
    rc.pos = p.pos[0];
    const int rb = row >> 4, tiles_per_head = p.D >> 4;
    if (p.rope && rb / tiles_per_head < p.Hl + p.KVl) {
      rc.inv_freq = p.inv_freq[8 * (rb % tiles_per_head) + (row & 7)];
      if (p.pos_uniform) {
        const float ang = (float)rc.pos * rc.inv_freq;
        rc.sn = sinf(ang);
        rc.cs = sinf(kHalfPi + ang * -1.0f);        // cos(a) = sin(pi/2 - a)
      }
    }
  }
  return rc;
}

// EPI_GELU_TOKEN: the entry of sequence b's token (two dependent loads from anywhere in a table of hundreds of MB)
__device__ __forceinline__ float token_factor(const GemvParams& p, int b, int row) {
  const int tok = p.tokens[b];
  return tok >= 0 && tok < p.token_rows ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.token_table)[(int64_t)tok * p.token_pitch + row]) : 0.f;
}

// Epilogue of one accumulator row held by one thread (v[b], b < N).  Rows g and g+8 of a 16-row
// block -- the pairs the fused epilogues combine -- are 8 lanes apart in the same warp.
// The thread holds batch columns b0 .. b0+NV-1 of the row (the whole row when NV == BP); BP is the
// batch padding of the activation buffers.
// X: the epilogues of decoders described layer by layer (softcap, EPI_STORE_RELU2) are compiled in.  They have instantiations of their
// own: the other models' kernels carry no code of them.
template <int NV, int BP, bool X>
__device__ __forceinline__ void row_epilogue(const GemvParams& p, float (&v)[NV], int row, int b0, const float* s_inv, const RowConst& rc,
                                             const float* factor = nullptr) {
  typedef Layout<__nv_bfloat16> LY;
  constexpr int N = NV;
  const int rb = row >> 4, rr = row & 15, g = rr & 7, hi = rr >> 3;
  if (s_inv) {                                   // the norm scale of the input, one per sequence (InvScale)
#pragma unroll
    for (int b = 0; b < N; ++b) v[b] *= s_inv[b0 + b];
    if (p.ln_wg) {                               // LayerNorm: the mean's share, inv * mu * (W g)[row]
#pragma unroll
      for (int b = 0; b < N; ++b) v[b] -= s_inv[32 + b0 + b] * rc.wg;
    }
  }
  if (p.bias) {
#pragma unroll
    for (int b = 0; b < N; ++b) v[b] += rc.bias;
  }
  if (p.epi == EPI_STORE_F32) {
    if (row < p.rows) {
      if (X && p.softcap > 0.f) {
#pragma unroll
        for (int b = 0; b < N; ++b) v[b] = p.softcap * tanhf(v[b] / p.softcap);
      }
#pragma unroll
      for (int b = 0; b < N; ++b)
        if (b0 + b < p.B) p.out[(int64_t)(b0 + b) * p.out_pitch + row] = v[b];
    }
    return;
  }
  if (X && (p.epi == EPI_STORE_RELU2 || p.epi == EPI_STORE_ACT)) {
    if (row < p.act_row0) {
#pragma unroll
      for (int b = 0; b < N; ++b)
        if (b0 + b < p.B) p.out[(int64_t)(b0 + b) * p.out_pitch + row] = v[b];
    } else if (row - p.act_row0 < p.n_act) {
      __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(p.act);
#pragma unroll
      for (int b = 0; b < N; ++b) {
        const float u = fmaxf(v[b], 0.f);
        if (b0 + b < p.B) act[LY::x_offset(b0 + b, p.act_col0 + row - p.act_row0, BP)] = __float2bfloat16_rn(p.epi == EPI_STORE_ACT ? v[b] : u * u);
      }
    }
    return;
  }
  if (X && p.epi == EPI_GELU_TOKEN) {
    if (row < p.rows) {
      __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(p.act);
#pragma unroll
      for (int b = 0; b < N; ++b) {
        if (b0 + b >= p.B) continue;
        const float e = factor ? factor[b] : token_factor(p, b0 + b, row);
        act[LY::x_offset(b0 + b, row, BP)] = __float2bfloat16_rn(gelu_ref(v[b]) * e);
      }
    }
    return;
  }
  if (p.epi == EPI_GELU_ACT) {
    if (row < p.n_act) {
      __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(p.act);
#pragma unroll
      for (int b = 0; b < N; ++b)
        if (b0 + b < p.B) act[LY::x_offset(b0 + b, row, BP)] = __float2bfloat16_rn(gelu_ref(v[b]));
    }
    return;
  }
  float w[N];                                   // the partner row's values
#pragma unroll
  for (int b = 0; b < N; ++b) w[b] = __shfl_xor_sync(0xffffffffu, v[b], 8);
  if (row >= p.rows) return;
  if (p.epi == EPI_SILU_GATE) {
    const int o = rb * 8 + g;
    if (hi == 0 && o < p.n_act) {
      __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(p.act);
#pragma unroll
      for (int b = 0; b < N; ++b) {
        if (b0 + b < p.B) {
          const float a = v[b], u = w[b];
          // silu(a) = a * (1 / (1 + exp2((a * -1) * (1/ln2))))     src/HighLevelOps.jl:153-160
          const float ex = exp2f((a * -1.0f) * kInvLn2);
          const float sg = 1.0f / (1.0f + ex);
          act[LY::x_offset(b0 + b, o, BP)] = __float2bfloat16_rn((a * sg) * u);
        }
      }
    }
    return;
  }
  // EPI_QKV_ROPE
  __nv_bfloat16* kv = reinterpret_cast<__nv_bfloat16*>(p.kv_layer);
  const int D = p.D, tiles_per_head = D >> 4, half = D >> 1;
  // One position per sequence.  When the host knows they are all equal (pos_uniform) the rotation's sine and
  // cosine are computed once per row; otherwise once per batch column.
  int pos = rc.pos;
  const int hs = rb / tiles_per_head, jj = rb - hs * tiles_per_head;
  if (hs < p.Hl + p.KVl) {
    // rows g / g+8 of the block are the RoPE pair (d0, d0 + D/2)      src/NN.jl:253-303
    const int d0 = 8 * jj + g;
    float sn = rc.sn, cs = rc.cs;
    const float inv_f = rc.inv_freq;
    const int d = hi ? d0 + half : d0;
#pragma unroll
    for (int b = 0; b < N; ++b) {
      if (b0 + b < p.B) {
        if (!p.pos_uniform) {
          pos = p.pos[b0 + b];
          if (p.rope) {
            const float ang = (float)pos * inv_f;
            sn = sinf(ang);
            cs = sinf(kHalfPi + ang * -1.0f);
          }
        }
        // low row: x0*cos - x1*sin; high row: x0*sin + x1*cos (x0 = the low row's value)
        const float o = hi ? (w[b] * sn + v[b] * cs) : (v[b] * cs + (w[b] * sn) * -1.0f);
        if (hs < p.Hl) {
          reinterpret_cast<__nv_bfloat16*>(p.q_out)[(int64_t)(b0 + b) * p.q_pitch + hs * D + d] = __float2bfloat16_rn(o);
        } else {
          kv[(b0 + b) * p.kv_batch_stride + (hs - p.Hl) * p.kv_head_stride + kcache_offset(pos, d, D)] = __float2bfloat16_rn(o);
        }
      }
    }
  } else {
    const int d = 16 * jj + rr;
#pragma unroll
    for (int b = 0; b < N; ++b)
      if (b0 + b < p.B) {
        if (!p.pos_uniform) pos = p.pos[b0 + b];
        kv[(b0 + b) * p.kv_batch_stride + (hs - p.Hl - p.KVl) * p.kv_head_stride + vcache_offset(pos, d, D)] =
            __float2bfloat16_rn(v[b]);
      }
  }
}

// Optional per-CTA phase stamps (SM clock) for tuning; compiled in only with -DLMB_GEMV_TRACE.
#ifdef LMB_GEMV_TRACE
__device__ long long g_gemv_trace[160 * 16];
__device__ __forceinline__ long long gtime_ns() { long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }
}  // namespace
int32_t gemv_trace_copy(long long* out) {
  return cudaMemcpyFromSymbol(out, g_gemv_trace, sizeof(g_gemv_trace)) == cudaSuccess ? 0 : -3;
}
namespace {
#define LMB_TRACE(slot) (g_gemv_trace[blockIdx.x * 16 + (slot)] = clock64())
#define LMB_TRACE_NS(slot) (g_gemv_trace[blockIdx.x * 16 + (slot)] = gtime_ns())
#else
#define LMB_TRACE(slot) ((void)0)
#define LMB_TRACE_NS(slot) ((void)0)
#endif

// The epilogue group (128 threads, e = 0..127) turns the producer's per-CTA sums of squares into the
// per-sequence scale 1 / sqrt(mean(x*x) + eps) (src/HighLevelOps.jl:299-304).  Four lanes share a
// sequence; each adds every fourth slot in ascending order and the four are combined pairwise, the
// same arithmetic in every CTA and on every rank.
// Slots part, part + 4, ... added in ascending order, 16 loads in flight: one load after the other took 9 us for 128 slots.
__device__ __forceinline__ float sum_slots(const float* slots, int tiles, int part, int b) {
  float s = 0.f;
  for (int t0 = part; t0 < tiles; t0 += 64) {
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = t0 + 4 * i < tiles ? __ldcg(slots + (t0 + 4 * i) * 32 + b) : 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += v[i];
  }
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s;
}
__device__ __forceinline__ void compute_inv_scale(const InvScale& iv, float* s_inv, int e) {
  if (!iv.ssq) return;
  const int b = e >> 2, part = e & 3;
  const float s = sum_slots(iv.ssq, iv.tiles, part, b), sx = iv.sum ? sum_slots(iv.sum, iv.tiles, part, b) : 0.f;
  if (part == 0) {
    const float rn = 1.0f / (float)iv.n;
    const float mu = sx * rn;                                   // 0 for RMSNorm
    const float inv = 1.0f / sqrtf(fmaxf(s * rn - mu * mu, 0.f) + iv.eps);
    s_inv[b] = inv;
    s_inv[32 + b] = mu * inv;
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
}

__device__ __forceinline__ uint4 peer_load16(const void* p) {
  uint4 v;
  asm volatile("ld.relaxed.sys.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void peer_store16(void* p, uint4 v) {
  asm volatile("st.relaxed.sys.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// bf16 -0.0 marks "not written yet" in a push buffer: a partial that rounds to it is sent as +0.0
__device__ __forceinline__ uint32_t pack_bf16x2_sendable(float a, float b) {
  uint32_t w = pack_bf16x2(a, b);
  if ((w & 0xFFFFu) == 0x8000u) w &= 0xFFFF0000u;
  if ((w >> 16) == 0x8000u) w &= 0x0000FFFFu;
  return w;
}
__device__ __forceinline__ bool has_empty_bf16(const uint4& u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  bool any = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) any = any || (w[i] & 0xFFFFu) == 0x8000u || (w[i] >> 16) == 0x8000u;
  return any;
}
__device__ __forceinline__ void unpack_bf16x8(const uint4& u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// EPI_RESID_NORM on the tile a cluster CTA finalises (rows_per = 128 / C rows of row group r, all Bp
// batch columns), run by the 128 epilogue threads once every partial row of the cluster sits in `recv`.
// Thread e owns rows (e >> 2) + 32 j and the 8 batch columns 8 (e & 3) .. + 7, so that a warp covers
// 8 consecutive rows x Bp columns: its peer stores and its reads of x are contiguous 512-byte runs.
template <int N>
__device__ __forceinline__ void resid_norm_tile(const GemvParams& p, const unsigned char* recv_raw, int C, int c, int r,
                                                int e, float* s_red) {
  constexpr int BG = N / 8;
  const int lane = e & 31, we = e >> 5;
  const int rows_per = 128 / C;
  const int bg = e & 3, rl0 = e >> 2;
  const int row0 = r * 128 + c * rows_per;
  const int iters = (rows_per + 31) >> 5;                      // 1, 1, 2, 4 for 16, 32, 64, 128 rows
  const float4* recv = reinterpret_cast<const float4*>(recv_raw);
  const int n = p.push.n, me = p.push.rank;
  float acc[4][8];
  bool valid[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int rl = rl0 + 32 * j;
    valid[j] = j < iters && bg < BG && rl < rows_per && row0 + rl < p.rows;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[j][i] = 0.f;
    if (valid[j]) {
      for (int src = 0; src < C; ++src) {                      // the cluster's partials, in CTA order
        const float4 t0 = recv[((src * rows_per + rl) * N + 8 * bg) / 4], t1 = recv[((src * rows_per + rl) * N + 8 * bg) / 4 + 1];
        acc[j][0] += t0.x; acc[j][1] += t0.y; acc[j][2] += t0.z; acc[j][3] += t0.w;
        acc[j][4] += t1.x; acc[j][5] += t1.y; acc[j][6] += t1.z; acc[j][7] += t1.w;
      }
    }
  }
  if (n > 1) {
    const unsigned long long epoch = *p.push.step * kPeerEpochStride + p.push.phase;
    // this rank's partial, rounded to bf16 (never the "not written yet" pattern), into the same place of every peer's region
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!valid[j]) continue;
      uint4 u;
      u.x = pack_bf16x2_sendable(acc[j][0], acc[j][1]); u.y = pack_bf16x2_sendable(acc[j][2], acc[j][3]);
      u.z = pack_bf16x2_sendable(acc[j][4], acc[j][5]); u.w = pack_bf16x2_sendable(acc[j][6], acc[j][7]);
      unpack_bf16x8(u, acc[j]);                                // what this rank adds is what its peers receive
      const size_t at = ((size_t)me * p.rows + (row0 + rl0 + 32 * j)) * N + 8 * bg;
#pragma unroll
      for (int rk = 0; rk < 8; ++rk)
        if (rk < n && rk != me) peer_store16(p.push.part[rk] + at, u);
    }
    if (e < n && e != me) {                                    // validity channel, unordered with the data
      const bool poisoned = *reinterpret_cast<volatile int*>(p.push.broken) != 0;
      asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p.push.flag[e] + me * kPushMaxCtas + blockIdx.x),
                   "l"(epoch | (poisoned ? kPeerPoison : 0ull))
                   : "memory");
    }
    const uint4 empty = make_uint4(kPeerEmptyPair, kPeerEmptyPair, kPeerEmptyPair, kPeerEmptyPair);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!valid[j]) continue;
      __nv_bfloat16* mine = p.push.part[me] + ((size_t)(row0 + rl0 + 32 * j)) * N + 8 * bg;      // + rk * rows * N
      const size_t src_stride = (size_t)p.rows * N;
      uint4 got[8];
      unsigned pending = 0;
#pragma unroll
      for (int rk = 0; rk < 8; ++rk)
        if (rk < n && rk != me) pending |= 1u << rk;
      const long long t0 = clock64();
      unsigned spins = 0;
      while (pending) {
#pragma unroll
        for (int rk = 0; rk < 8; ++rk)
          if (pending & (1u << rk)) got[rk] = peer_load16(mine + rk * src_stride);
#pragma unroll
        for (int rk = 0; rk < 8; ++rk)
          if ((pending & (1u << rk)) && !has_empty_bf16(got[rk])) pending &= ~(1u << rk);
        if (pending && (++spins & 63u) == 0u) {
          if (*reinterpret_cast<volatile int*>(p.push.broken) != 0) break;       // an earlier wait of this rank already failed
          if (clock64() - t0 > p.push.wait_cycles) { peer_mark_failed(p.push.dev_err, p.push.broken, 1); break; }
        }
      }
      float tot[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) tot[i] = 0.f;
#pragma unroll
      for (int rk = 0; rk < 8; ++rk) {                         // rank order, the same on every rank
        if (rk >= n) continue;
        float pv[8];
        if (rk == me) {
#pragma unroll
          for (int i = 0; i < 8; ++i) pv[i] = acc[j][i];
        } else {
          unpack_bf16x8(got[rk], pv);
          *reinterpret_cast<uint4*>(mine + rk * src_stride) = empty;   // ready for the reduction after the next
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) tot[i] += pv[i];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[j][i] = tot[i];
    }
    if (e < n && e != me) {                                    // the senders' validity marks (normally long there)
      const unsigned long long* flag = p.push.flag[me] + e * kPushMaxCtas + blockIdx.x;
      const long long t0 = clock64();
      unsigned spins = 0;
      for (;;) {
        unsigned long long v;
        asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(flag) : "memory");
        bool bad = false;
        if (peer_signal_ok(v, epoch, &bad)) {
          if (bad) peer_mark_failed(p.push.dev_err, p.push.broken, 2);
          break;
        }
        if ((++spins & 63u) == 0u) {
          if (*reinterpret_cast<volatile int*>(p.push.broken) != 0) break;
          if (clock64() - t0 > p.push.wait_cycles) { peer_mark_failed(p.push.dev_err, p.push.broken, 1); break; }
        }
      }
    }
  }
  // residual add, the next Linear's input x * gain, this tile's share of the sum of squares (and, for a LayerNorm, of the sum)
  float ssq[8], sxv[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { ssq[i] = 0.f; sxv[i] = 0.f; }
  __nv_bfloat16* xg = reinterpret_cast<__nv_bfloat16*>(p.rn.xg);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (!valid[j]) continue;
    const int grow = row0 + rl0 + 32 * j;
    float4* xr = reinterpret_cast<float4*>(p.rn.x + (size_t)grow * N + 8 * bg);
    float4 x0 = xr[0], x1 = xr[1];
    const float bias = p.bias ? p.bias[grow] : 0.f;             // the projection's own bias (Whisper)
    x0.x += acc[j][0] + bias; x0.y += acc[j][1] + bias; x0.z += acc[j][2] + bias; x0.w += acc[j][3] + bias;
    x1.x += acc[j][4] + bias; x1.y += acc[j][5] + bias; x1.z += acc[j][6] + bias; x1.w += acc[j][7] + bias;
    xr[0] = x0; xr[1] = x1;
    const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    const float g = p.rn.gain[grow];
    __nv_bfloat16* o = xg + (size_t)(grow >> 3) * (N * 8) + bg * 64 + (grow & 7);      // Layout::x_offset(8 bg + i, grow, N) = o + 8 i
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o[8 * i] = __float2bfloat16_rn(xv[i] * g);
      ssq[i] += xv[i] * xv[i];
      sxv[i] += xv[i];
    }
    if (p.rn.capture) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * bg + i < p.B) p.rn.capture[(size_t)(8 * bg + i) * p.rows + grow] = xv[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {                                // over the 8 rows of the warp that share these batch columns
    ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], 4);
    ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], 8);
    ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], 16);
  }
  if (lane < 4) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s_red[we * 32 + 8 * lane + i] = ssq[i];
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  if (e < 32) p.rn.ssq[(size_t)blockIdx.x * 32 + e] = ((s_red[e] + s_red[32 + e]) + s_red[64 + e]) + s_red[96 + e];
  if (p.rn.sum) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      sxv[i] += __shfl_xor_sync(0xffffffffu, sxv[i], 4);
      sxv[i] += __shfl_xor_sync(0xffffffffu, sxv[i], 8);
      sxv[i] += __shfl_xor_sync(0xffffffffu, sxv[i], 16);
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");         // s_red has been read
    if (lane < 4) {
#pragma unroll
      for (int i = 0; i < 8; ++i) s_red[we * 32 + 8 * lane + i] = sxv[i];
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    if (e < 32) p.rn.sum[(size_t)blockIdx.x * 32 + e] = ((s_red[e] + s_red[32 + e]) + s_red[64 + e]) + s_red[96 + e];
  }
}

// EPI_POST_NORM on the tile a cluster CTA finalises; threads and rows as in resid_norm_tile.
template <int N>
__device__ __forceinline__ void post_norm_tile(const GemvParams& p, const unsigned char* recv_raw, int C, int c, int r, int e, float* s_red,
                                               float* s_scale, const float* s_inv, int* err) {
  constexpr int BG = N / 8;
  const int lane = e & 31, we = e >> 5;
  const int rows_per = 128 / C;
  const int bg = e & 3, rl0 = e >> 2;
  const int row0 = r * 128 + c * rows_per;
  const int iters = (rows_per + 31) >> 5;
  const float4* recv = reinterpret_cast<const float4*>(recv_raw);
  float acc[4][8], xv[4][8], ss[8];
  bool valid[4];
#pragma unroll
  for (int i = 0; i < 8; ++i) ss[i] = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int rl = rl0 + 32 * j;
    valid[j] = j < iters && bg < BG && rl < rows_per && row0 + rl < p.rows;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[j][i] = xv[j][i] = 0.f;
    if (!valid[j]) continue;
    for (int src = 0; src < C; ++src) {
      const float4 t0 = recv[((src * rows_per + rl) * N + 8 * bg) / 4], t1 = recv[((src * rows_per + rl) * N + 8 * bg) / 4 + 1];
      acc[j][0] += t0.x; acc[j][1] += t0.y; acc[j][2] += t0.z; acc[j][3] += t0.w;
      acc[j][4] += t1.x; acc[j][5] += t1.y; acc[j][6] += t1.z; acc[j][7] += t1.w;
    }
    const float4* xr = reinterpret_cast<const float4*>(p.pn.x + (size_t)(row0 + rl) * N + 8 * bg);
    const float4 x0 = xr[0], x1 = xr[1];
    xv[j][0] = x0.x; xv[j][1] = x0.y; xv[j][2] = x0.z; xv[j][3] = x0.w;
    xv[j][4] = x1.x; xv[j][5] = x1.y; xv[j][6] = x1.z; xv[j][7] = x1.w;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (s_inv) acc[j][i] *= s_inv[8 * bg + i];
      ss[i] += acc[j][i] * acc[j][i];
    }
  }
  auto publish = [&](float* slots, bool flagged) {             // per-CTA sums of ss over the rows
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 4);
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 8);
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 16);
    }
    if (lane < 4) {
#pragma unroll
      for (int i = 0; i < 8; ++i) s_red[we * 32 + 8 * lane + i] = ss[i];
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    if (e < 32) {
      const float t = ((s_red[e] + s_red[32 + e]) + s_red[64 + e]) + s_red[96 + e];
      unsigned u = __float_as_uint(t);
      if (flagged && u == kSlotEmpty) u = 0x7FC00000u;
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;\n" ::"l"(slots + (size_t)blockIdx.x * 32 + e), "r"(u) : "memory");
    }
  };
  publish(p.pn.slots, true);
  if (p.pn.clear)
    for (int i = blockIdx.x * 32 + (e & 31); i < kPushMaxCtas * 32; i += gridDim.x * 32)
      if (e < 32) p.pn.clear[i] = __uint_as_float(kSlotEmpty);
  {                                                            // four lanes per sequence, the same sums in every CTA
    const int b = e >> 2, part = e & 3, n = (int)gridDim.x;
    float s = 0.f;
    const long long t0 = clock64();
    bool late = false;
    for (int first = part; first < n; first += 32) {           // eight slots in flight
      unsigned u[8];
      bool wait = true;
      while (wait) {
        wait = false;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          u[i] = 0u;
          if (first + 4 * i < n) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(u[i]) : "l"(p.pn.slots + (first + 4 * i) * 32 + b) : "memory");
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) wait = wait || u[i] == kSlotEmpty;
        if (wait && (late || clock64() - t0 > kWaitLimit)) {
          if (!late && err) atomicExch(err, 1);
          late = true;
          wait = false;
        }
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) s += __uint_as_float(u[i]);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (part == 0) s_scale[b] = 1.0f / sqrtf(s / (float)p.rows + p.pn.eps);
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  __nv_bfloat16* xg = reinterpret_cast<__nv_bfloat16*>(p.pn.xg);
#pragma unroll
  for (int i = 0; i < 8; ++i) ss[i] = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (!valid[j]) continue;
    const int grow = row0 + rl0 + 32 * j;
    const float w = p.pn.w[grow], g = p.pn.gain ? p.pn.gain[grow] : 1.0f;
    __nv_bfloat16* o = xg + (size_t)(grow >> 3) * (N * 8) + bg * 64 + (grow & 7);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      xv[j][i] += acc[j][i] * s_scale[8 * bg + i] * w;
      o[8 * i] = __float2bfloat16_rn(xv[j][i] * g);
      ss[i] += xv[j][i] * xv[j][i];
    }
    float4* xr = reinterpret_cast<float4*>(p.pn.x + (size_t)grow * N + 8 * bg);
    xr[0] = make_float4(xv[j][0], xv[j][1], xv[j][2], xv[j][3]);
    xr[1] = make_float4(xv[j][4], xv[j][5], xv[j][6], xv[j][7]);
    if (p.pn.capture) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * bg + i < p.B) p.pn.capture[(size_t)(8 * bg + i) * p.rows + grow] = xv[j][i];
    }
  }
  if (p.pn.ssq) publish(p.pn.ssq, false);
}

template <int N, bool X>
__global__ void __launch_bounds__(kTcThreads, 1) gemv_tc_kernel(const GemvParams p, int* err) {
  constexpr int kXStage = N * 256;
  constexpr int kStage = kWStage + kXStage;
  constexpr uint32_t kTmemCols = 2 * N;       // two accumulator buffers (32 or 64 columns)
  // instruction descriptor, kind::f16: D = f32 (bit 4), A = B = bf16 (bits 7, 10), both K-major,
  // N >> 3 at bit 17, M >> 4 at bit 24
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ float s_inv_buf[64];        // [0, 32): inv per sequence, [32, 64): mean * inv (LayerNorm)
  const float* s_inv = p.inv.ssq ? s_inv_buf : nullptr;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const UnitRange ur = unit_range(p);
  if (tid == 0) {
    LMB_TRACE(0); LMB_TRACE_NS(10);
#pragma unroll
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_full[0], 1); mbar_init(&acc_full[1], 1);
    mbar_init(&acc_empty[0], 4); mbar_init(&acc_empty[1], 4);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  bool dead = false;
  pdl_launch_dependents();
  if (tid == 0) LMB_TRACE(1);

  if (warp == 0) {
    produce<N>(p, ur, smem, full_bar, empty_bar, lane, err);
  } else if (warp == 1) {
    pdl_wait();
    if (lane == 0) LMB_TRACE(2);
    // ---------------- MMA issue ----------------
    if (elect_one()) {
      int it = 0, seg = 0;
      for (int u = ur.u0; u < ur.u1; ++u, ++it) {
        const int ks = u % ur.KS;
        const bool first = (u == ur.u0) || ks == 0;
        const bool last = (u == ur.u1 - 1) || ks == ur.KS - 1;
        const int buf = seg & 1;
        if (first) mbar_wait(&acc_empty[buf], ((seg >> 1) & 1) ^ 1, dead, err);   // epilogue has drained this buffer
        const int s = it % kStages, k = it / kStages;
        mbar_wait(&full_bar[s], k & 1, dead, err);
        tc_fence_after();
        if (it == 0) LMB_TRACE(3);
        const uint32_t st = smem_u32(smem + s * kStage);
        const uint64_t adesc = smem_desc(st, 2048, 128);
        const uint64_t bdesc = smem_desc(st + kWStage, N * 16, 128);
#pragma unroll
        for (int j = 0; j < 8; ++j)     // 8 k-steps of 16: two core matrices along K each
          tc_mma_f16(tmem_base + buf * N, adesc + (uint64_t)(j * (4096 >> 4)), bdesc + (uint64_t)(j * ((2 * N * 16) >> 4)),
                     kIdesc, (first && j == 0) ? 0u : 1u);
        tc_commit(&empty_bar[s]);       // stage free once these MMAs have read it
        if (last) tc_commit(&acc_full[buf]);
        if (last) ++seg;
      }
      LMB_TRACE(4);
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: warp quarter q owns TMEM lanes / rows 32q .. 32q+31 ----------------
    // A row group whose k range is shared by n > 1 CTAs is folded by all of them together: each
    // stores its partial accumulator and counts itself in; once this CTA has finished its own
    // units it waits until every contributor of the group has arrived and then sums, in contributor
    // order, the 16-row blocks that fall to it (block j goes to contributor j mod n) and runs
    // their epilogue.  The sum order is fixed, so results do not depend on timing.
    pdl_wait();
    const int q = warp & 3;
    const int e = tid - 64;                      // 0..127 inside the epilogue group
    compute_inv_scale(p.inv, s_inv_buf, e);
    int seg = 0;
    int pend_r[2], pend_first[2], pend_n[2], n_pend = 0;
    for (int u = ur.u0; u < ur.u1; ++seg) {
      const int r = u / ur.KS;
      const int u_end = min(ur.u1, (r + 1) * ur.KS);
      u = u_end;
      const int buf = seg & 1;
      mbar_wait(&acc_full[buf], (seg >> 1) & 1, dead, err);
      tc_fence_after();
      float v[N];
      tmem_load_row<N>(v, tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(buf * N));
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      if (tid == 64) LMB_TRACE(5);
      const int row_in_group = 32 * q + lane;
      int c_first, n;
      contributors(ur, r, &c_first, &n);
      if (n == 1) {
        row_epilogue<N, N, X>(p, v, r * 128 + row_in_group, 0, s_inv, row_const(p, r * 128 + row_in_group));
        continue;
      }
      float4* part = reinterpret_cast<float4*>(p.partials) + (int64_t)r * p.ksplit * (128 * N / 4);
      float4* mine = part + (int64_t)((int)blockIdx.x - c_first) * (128 * N / 4) + row_in_group * (N / 4);
#pragma unroll
      for (int i = 0; i < N / 4; ++i) mine[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      __threadfence();
      asm volatile("bar.sync 1, 128;\n" ::: "memory");
      if (e == 0) atomicAdd(&p.counters[r * 8], 1u);
      if (tid == 64) LMB_TRACE(6);
      if (n_pend < 2) { pend_r[n_pend] = r; pend_first[n_pend] = c_first; pend_n[n_pend] = n; ++n_pend; }
    }
    // wait for every contributor of the shared row groups.  The last segment is shared with CTAs
    // that finished it long ago, the first one with a CTA that ends on it about now.
    if (e == 0) {
      const long long t0 = clock64();
      for (int ip = n_pend - 1; ip >= 0; --ip) {
        for (;;) {
          unsigned seen;
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(p.counters + pend_r[ip] * 8) : "memory");
          if (seen >= (unsigned)pend_n[ip] || dead) break;
          if (clock64() - t0 > kWaitLimit) { dead = true; if (err) atomicExch(err, 1); break; }
        }
      }
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    if (tid == 64) LMB_TRACE(7);
    const int row16 = lane & 15, cg = e >> 4;               // one float4 (4 batch columns) per thread
    if (cg < N / 4 && n_pend > 0) {                          // warp-uniform: whole warps drop out for N = 16
      // Per shared row group this contributor owns the 16-row blocks ci, ci + n, ... (at most 4) and
      // sums each over the contributors in ascending order.  A round trip to L2 at the end of a
      // kernel costs microseconds, so every partial this thread needs is fetched with one wave of
      // cp.async into the (now idle) pipeline stages, slot s of thread e at byte s * 2048 + e * 16,
      // and summed from shared memory afterwards.
      constexpr int kSlots = (kStages * kStage) / 2048;
      constexpr int64_t kPartStride = 128 * N / 4;           // float4s per contributor
      const uint32_t fs = smem_u32(smem) + (uint32_t)e * 16u;
      int n_[2], ci_[2], nj_[2];
      const float4* part_[2];
#pragma unroll
      for (int ip = 0; ip < 2; ++ip) {
        const bool on = ip < n_pend;
        n_[ip] = on ? pend_n[ip] : 1;
        ci_[ip] = on ? (int)blockIdx.x - pend_first[ip] : 8;
        nj_[ip] = ci_[ip] < 8 ? (8 - ci_[ip] + n_[ip] - 1) / n_[ip] : 0;
        part_[ip] = reinterpret_cast<const float4*>(p.partials) + (int64_t)(on ? pend_r[ip] : 0) * p.ksplit * kPartStride +
                    row16 * (N / 4) + cg;
      }
      auto issue = [&](int ip, int slot, int k0, int k1) -> int {
        for (int jj = 0; jj < nj_[ip]; ++jj) {
          const float4* src = part_[ip] + 16 * (ci_[ip] + jj * n_[ip]) * (N / 4);
          for (int k = k0; k < k1; ++k, ++slot)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(fs + (uint32_t)slot * 2048u), "l"(src + k * kPartStride) : "memory");
        }
        return slot;
      };
      auto lds4 = [&](int slot) -> float4 {
        float4 t;
        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w) : "r"(fs + (uint32_t)slot * 2048u));
        return t;
      };
      auto consume = [&](int ip, int slot) -> int {
        for (int jj = 0; jj < nj_[ip]; ++jj) {
          float v4[4] = {0.f, 0.f, 0.f, 0.f};
          for (int k = 0; k < n_[ip]; ++k, ++slot) {
            const float4 t = lds4(slot);
            v4[0] += t.x; v4[1] += t.y; v4[2] += t.z; v4[3] += t.w;
          }
          const int row = pend_r[ip] * 128 + 16 * (ci_[ip] + jj * n_[ip]) + row16;
          row_epilogue<4, N, X>(p, v4, row, 4 * cg, s_inv, row_const(p, row));
        }
        return slot;
      };
      const int cnt0 = nj_[0] * n_[0], cnt1 = nj_[1] * n_[1];
      if (cnt0 + cnt1 <= kSlots) {
        const int s1 = issue(0, 0, 0, n_[0]);
        issue(1, s1, 0, n_[1]);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        if (tid == 64) LMB_TRACE(12);
        consume(1, consume(0, 0));
      } else {
        // a row group shared by more CTAs than there are slots (tiny matrices): waves over k
#pragma unroll 1
        for (int ip = 0; ip < 2; ++ip) {
          if (nj_[ip] == 0) continue;
          if (nj_[ip] * n_[ip] <= kSlots) {
            issue(ip, 0, 0, n_[ip]);
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            consume(ip, 0);
            continue;
          }
          float v4[4] = {0.f, 0.f, 0.f, 0.f};          // n > kSlots > 8, so there is one block
          for (int k0 = 0; k0 < n_[ip]; k0 += kSlots) {
            const int k1 = min(n_[ip], k0 + kSlots);
            issue(ip, 0, k0, k1);
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            for (int sl = 0; sl < k1 - k0; ++sl) {
              const float4 t = lds4(sl);
              v4[0] += t.x; v4[1] += t.y; v4[2] += t.z; v4[3] += t.w;
            }
          }
          const int row = pend_r[ip] * 128 + 16 * ci_[ip] + row16;
          row_epilogue<4, N, X>(p, v4, row, 4 * cg, s_inv, row_const(p, row));
        }
      }
      if (tid == 64) LMB_TRACE(13);
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    if (e < n_pend) {
      const int r = pend_r[e], n = pend_n[e];
      const unsigned prev = atomicAdd(&p.counters[r * 8 + 1], 1u);
      if (prev == (unsigned)n - 1u) {                       // every contributor has read: ready for the next launch
        p.counters[r * 8] = 0u;
        p.counters[r * 8 + 1] = 0u;
      }
    }
    if (tid == 64) LMB_TRACE(8);
  }
  // all roles meet before the accumulator memory is given back
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (tid == 0) { LMB_TRACE(9); LMB_TRACE_NS(11); }
}

// =============================================================================================
// Cluster variant for small matrices.  The stream-K kernel folds a shared row group through
// global scratch: store, fence, count, wait, fetch -- about 6 us after the last MMA, more than
// the streaming itself once a matrix is a few tens of MB (tensor-parallel shards, q/k/v, o_proj).
// Here a thread-block cluster of C CTAs owns one 128-row group, CTA c streams the c-th share of
// its k range, and the partial accumulators are exchanged through distributed shared memory:
// every CTA sends each peer the rows that peer finalises (128 / C of them), one cluster barrier,
// then every CTA sums its rows over the C sources in rank order and runs their epilogue.
// =============================================================================================
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t dsmem_addr(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void dsmem_store4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <int N, bool X>
__global__ void __launch_bounds__(kTcThreads, 1) gemv_cl_kernel(const GemvParams p, int* err) {
  constexpr int kXStage = N * 256;
  constexpr int kStage = kWStage + kXStage;
  constexpr uint32_t kTmemCols = N < 32 ? 32 : N;     // an allocation is at least 32 columns
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
  extern __shared__ __align__(1024) unsigned char smem[];       // kStages stages, then recv[C][128 / C][N] floats
  __shared__ __align__(8) uint64_t full_bar[kStages];
  __shared__ __align__(8) uint64_t empty_bar[kStages];
  __shared__ __align__(8) uint64_t acc_full;
  __shared__ uint32_t tmem_base_slot;
  __shared__ float s_inv_buf[64];        // [0, 32): inv per sequence, [32, 64): mean * inv (LayerNorm)
  __shared__ float s_red[128];
  __shared__ float s_scale[X ? 32 : 1];
  const float* s_inv = p.inv.ssq ? s_inv_buf : nullptr;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = (int)cluster_nctarank(), c = (int)cluster_ctarank();
  const int r = (int)blockIdx.x / C;                              // row group of this cluster
  const int KS = (p.K + 127) >> 7;
  const int ks0 = (int)((long long)c * KS / C), ks1 = (int)((long long)(c + 1) * KS / C);
  const int n_steps = ks1 - ks0;
  if (tid == 0) {
    LMB_TRACE(0); LMB_TRACE_NS(10);
#pragma unroll
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  bool dead = false;
  pdl_launch_dependents();
  if (tid == 0) LMB_TRACE(1);

  if (warp == 0) {
    // ---------------- producer: weights before the dependency wait, activations after ----------------
    uint64_t pol_w, pol_x;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol_w));
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(pol_x));
    const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(p.W) + ((int64_t)r * KS + ks0) * 16384;
    const __nv_bfloat16* X = reinterpret_cast<const __nv_bfloat16*>(p.x) + (int64_t)ks0 * (128 * N);
    const int n_pre = n_steps < kStages ? n_steps : kStages;
    if (lane == 0) {
      for (int i = 0; i < n_pre; ++i) {
        mbar_expect_tx(&full_bar[i], (uint32_t)kStage);
        bulk_g2s(smem + i * kStage, W + (int64_t)i * 16384, (uint32_t)kWStage, &full_bar[i], pol_w);
      }
    }
    pdl_wait();
    if (lane == 0) {
      for (int i = 0; i < n_pre; ++i)
        bulk_g2s(smem + i * kStage + kWStage, X + (int64_t)i * (128 * N), (uint32_t)kXStage, &full_bar[i], pol_x);
    }
    __syncwarp();
    for (int i = n_pre; i < n_steps; ++i) {
      const int s = i % kStages, k = i / kStages;
      mbar_wait(&empty_bar[s], (k & 1) ^ 1, dead, err);
      if (lane == 0) {
        unsigned char* sp = smem + s * kStage;
        mbar_expect_tx(&full_bar[s], (uint32_t)kStage);
        bulk_g2s(sp, W + (int64_t)i * 16384, (uint32_t)kWStage, &full_bar[s], pol_w);
        bulk_g2s(sp + kWStage, X + (int64_t)i * (128 * N), (uint32_t)kXStage, &full_bar[s], pol_x);
      }
      __syncwarp();
    }
    prefetch_next_weights(p, lane);
  } else if (warp == 1) {
    // ---------------- MMA issue ----------------
    pdl_wait();
    if (lane == 0) LMB_TRACE(2);
    if (elect_one()) {
      for (int i = 0; i < n_steps; ++i) {
        const int s = i % kStages, k = i / kStages;
        mbar_wait(&full_bar[s], k & 1, dead, err);
        tc_fence_after();
        if (i == 0) LMB_TRACE(3);
        const uint32_t sa = smem_u32(smem + s * kStage);
        const uint64_t adesc = smem_desc(sa, 2048, 128);
        const uint64_t bdesc = smem_desc(sa + kWStage, N * 16, 128);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          tc_mma_f16(tmem_base, adesc + (uint64_t)(j * (4096 >> 4)), bdesc + (uint64_t)(j * ((2 * N * 16) >> 4)), kIdesc,
                     (i == 0 && j == 0) ? 0u : 1u);
        tc_commit(&empty_bar[s]);
        if (i == n_steps - 1) tc_commit(&acc_full);
      }
      LMB_TRACE(4);
    }
    __syncwarp();
  } else {
    // ---------------- epilogue warps: send every row to the CTA that finalises it ----------------
    pdl_wait();
    const int q = warp & 3;
    compute_inv_scale(p.inv, s_inv_buf, tid - 64);
    float v[N];
    if (n_steps > 0) {
      mbar_wait(&acc_full, 0, dead, err);
      tc_fence_after();
      tmem_load_row<N>(v, tmem_base + ((uint32_t)(32 * q) << 16));
      tc_fence_before();
      if (tid == 64) LMB_TRACE(5);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] = 0.f;
    }
    const int rows_per = 128 / C;
    const int row = 32 * q + lane;
    const int owner = row / rows_per, row_local = row - owner * rows_per;
    const uint32_t recv_local = smem_u32(smem + kStages * kStage) + (uint32_t)(((c * rows_per + row_local) * N) * 4);
    const uint32_t dst = dsmem_addr(recv_local, (uint32_t)owner);
#pragma unroll
    for (int i = 0; i < N / 4; ++i) dsmem_store4(dst + 16u * i, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    if (tid == 64) LMB_TRACE(6);
  }
  // every partial row is in its owner's shared memory once all CTAs of the cluster are here
  cluster_sync_all();
  if (tid == 64) LMB_TRACE(7);
  if (warp >= 2 && p.epi == EPI_RESID_NORM) {
    resid_norm_tile<N>(p, smem + kStages * kStage, C, c, r, tid - 64, s_red);
  } else if (X && warp >= 2 && p.epi == EPI_POST_NORM) {
    post_norm_tile<N>(p, smem + kStages * kStage, C, c, r, tid - 64, s_red, s_scale, s_inv, err);
  } else if (warp >= 2) {
    const int e = tid - 64;
    const int rows_per = 128 / C;
    const int row16 = lane & 15, cg = e >> 4;               // one float4 (4 batch columns) per thread
    if (cg < N / 4) {
      const float4* recv = reinterpret_cast<const float4*>(smem + kStages * kStage);
      for (int j = 0; j < rows_per / 16; ++j) {
        float v4[4] = {0.f, 0.f, 0.f, 0.f};
        for (int src = 0; src < C; ++src) {
          const float4 t = recv[((src * rows_per + 16 * j + row16) * N) / 4 + cg];
          v4[0] += t.x; v4[1] += t.y; v4[2] += t.z; v4[3] += t.w;
        }
        const int row = r * 128 + c * rows_per + 16 * j + row16;
        row_epilogue<4, N, X>(p, v4, row, 4 * cg, s_inv, row_const(p, row));
      }
    }
  }
  if (tid == 64) LMB_TRACE(8);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (tid == 0) { LMB_TRACE(9); LMB_TRACE_NS(11); }
}

// =============================================================================================
// Chain kernel: several dependent GEMVs of a step in one launch.
//
// A decode step is a chain of short GEMVs, and one launch each leaves HBM idle between the last MMA of one and the
// first bytes of the next: fold, epilogue, drain, launch, set-up and ring fill, about 8 us of which a 34 to 50 MB matrix streams
// for 5 to 8.  Here one persistent grid (clusters of 4 CTAs, one CTA per SM) runs them all.  Weights depend on nothing, so the
// weight producer walks straight through the list and has its ring full of the next GEMV's units when that one may start.
//   Work: cluster i takes row groups i, i + n, ...; CTA c of it the c-th quarter of the k range.  A warp's 32 accumulator rows
//   are exactly the rows one CTA of the cluster finalises: it sends them there with st.async (the receiver's mbarrier
//   counts the bytes; no fence, no cluster barrier), and the receiver adds the four parts in CTA order.
//   Dependency: every CTA counts itself into done[op] once its epilogues are written; the activation producer and
//   the epilogue warps of the next GEMV wait for that count.  Counting all CTAs is enough for the buffers that are written again
//   (xg, ssq, act) as well: whoever writes them has waited for all readers.
//   Clusters of 4: 33 of them fit a B200 (132 SMs, which stream at the same 7.1 TB/s as 148); of 8 only 15 fit, one short of the 16
//   row groups of a 2048-wide model, and of 2 a narrow projection would leave half the chip idle.
//   Measured (8 layers, per step, one launch per GEMV -> chained): Llama-3-8B shape at 1031 keys, batch 1 1044 -> 955 us, batch 32
//   1252 -> 1143 us; Phi-3-mini batch 16 at 2052 keys 760 -> 693 us; Kevatar width 2048 batch 16 825 -> 734 us.  gemv_chain_clusters has the rule.
//   Since then the links take less: one release and one acquire per dependency, the proxy fence on the reading side only, parameters a link
//   ahead in shared memory, and the layers' decode attention as a link (chain_attend).  Whole steps through the host, 32 layers: Llama-3-8B batch 1, 1031 keys
//   3.34 -> 3.05 ms, batch 32, 8184 keys 9.37 -> 8.82; Phi-3-mini batch 16, 2052 keys 2.69 -> 2.29.
//   LayerNorms (sums of x beside those of squares) are not built in: the Whisper decoder, which needs them, was slower chained at width 512,
//   327 -> 350 us a step, one unit of k per tile; up to 16 sequences its step is a kernel of its own instead (whisper_step.cu, 189 us).
//   warp 0 weights, 1 MMA, 2..5 epilogue (and attention), 6 activations.
// =============================================================================================
constexpr int kChainThreads = 7 * 32;
constexpr int kChainLine = 32;               // counters are a 128-byte line apart

template <int M>
struct ChainParams {
  GemvParams op[M];
  int n_ops = 0;
  unsigned* done = nullptr;                  // [kChainMaxAttend + 1] lines, zero between launches; the last one counts exits
};
// what a link's epilogue reads of its parameters: all in front of the tensor-parallel exchange, which no chain has
constexpr int kChainOpBytes = (int)(offsetof(GemvParams, push) + 15) / 16 * 16;
static_assert(kChainOpBytes <= 480, "two links' parameters beside the barriers in the 2 KB that the ring leaves");
// D > 0: the kernel with attention at that head dimension
template <int D> using ChainParamsOf = ChainParams<(D > 0 ? kChainMaxAttend : kChainMax)>;

template <int N> constexpr int kChainStages = N == 16 ? 6 : 5;
template <int N> constexpr size_t chain_smem() { return (size_t)kChainStages<N> * (kWStage + N * 256) + 128 * N * 4 + 1024; }

__device__ __forceinline__ void dsmem_store4_async(uint32_t addr, uint32_t bar, float a, float b, float c, float d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1,%2,%3,%4}, [%5];\n" ::"r"(addr), "f"(a), "f"(b),
               "f"(c), "f"(d), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity, bool& dead, int* err) {
  if (dead) return;
  const long long t0 = clock64();
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return;
    if (clock64() - t0 > kWaitLimit) {
      dead = true;
      if (err) atomicExch(err, 1);
      return;
    }
  }
}
// the CTAs that take part in a link
__device__ __forceinline__ unsigned chain_ctas(const GemvParams& p, int ncl) {
  if (p.epi == EPI_ATTEND) return (unsigned)min(ncl * kChainC, p.B * p.KVl * p.ksplit);
  return (unsigned)(min(ncl, (p.rows + 127) >> 7) * kChainC);
}
__device__ __forceinline__ void chain_wait_done(const unsigned* done, unsigned want, bool& dead, int* err) {
  if (dead) return;
  const long long t0 = clock64();
  for (;;) {
    unsigned seen;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(done) : "memory");
    if (seen >= want) return;
    if (clock64() - t0 > kWaitLimit) {
      dead = true;
      if (err) atomicExch(err, 1);
      return;
    }
  }
}

__device__ __forceinline__ void chain_wait_shared(const unsigned* count, unsigned want, bool& dead, int* err) {
  if (dead) return;
  const long long t0 = clock64();
  for (;;) {
    unsigned seen;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];\n" : "=r"(seen) : "r"(smem_u32(count)) : "memory");
    if (seen >= want) return;
    if (clock64() - t0 > kWaitLimit) {
      dead = true;
      if (err) atomicExch(err, 1);
      return;
    }
  }
}

// a row of N floats in the receive buffer: its 16-byte pieces are rotated so that a warp's rows meet different banks
template <int N>
__device__ __forceinline__ int chain_piece(int row, int piece) {
  return N == 32 ? piece ^ (row & 7) : piece ^ ((row >> 1) & 3);
}

// EPI_RESID_NORM for the 32 rows this CTA finalises, one rank; arithmetic and order as in resid_norm_tile.
// Thread e holds row e >> 2 and batch columns 8 (e & 3) .. + 7; the residual row is fetched while the weights stream.
struct ChainResid { float4 x0, x1; float gain, bias; };
template <int N>
__device__ __forceinline__ void chain_resid_load(const GemvParams& p, int row0, int e, ChainResid& h) {
  const int bg = e & 3, grow = row0 + (e >> 2);
  if (bg >= N / 8 || grow >= p.rows) return;
  const float4* xr = reinterpret_cast<const float4*>(p.rn.x + (size_t)grow * N + 8 * bg);
  h.x0 = xr[0]; h.x1 = xr[1];
  h.bias = p.bias ? p.bias[grow] : 0.f;
  h.gain = p.rn.gain[grow];
}
template <int N>
__device__ __forceinline__ void chain_resid_tile(const GemvParams& p, const ChainResid& h, const float4* recv, int row0, int slot, int e, float* s_red) {
  constexpr int BG = N / 8;
  const int lane = e & 31, we = e >> 5, bg = e & 3, rl = e >> 2, grow = row0 + rl;
  const bool valid = bg < BG && grow < p.rows;
  float ssq[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) ssq[i] = 0.f;
  if (valid) {
    float acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
    for (int src = 0; src < kChainC; ++src) {
      const float4 t0 = recv[(src * 32 + rl) * (N / 4) + chain_piece<N>(rl, 2 * bg)], t1 = recv[(src * 32 + rl) * (N / 4) + chain_piece<N>(rl, 2 * bg + 1)];
      acc[0] += t0.x; acc[1] += t0.y; acc[2] += t0.z; acc[3] += t0.w;
      acc[4] += t1.x; acc[5] += t1.y; acc[6] += t1.z; acc[7] += t1.w;
    }
    const float xv[8] = {h.x0.x + (acc[0] + h.bias), h.x0.y + (acc[1] + h.bias), h.x0.z + (acc[2] + h.bias), h.x0.w + (acc[3] + h.bias),
                         h.x1.x + (acc[4] + h.bias), h.x1.y + (acc[5] + h.bias), h.x1.z + (acc[6] + h.bias), h.x1.w + (acc[7] + h.bias)};
    float4* xr = reinterpret_cast<float4*>(p.rn.x + (size_t)grow * N + 8 * bg);
    xr[0] = make_float4(xv[0], xv[1], xv[2], xv[3]);
    xr[1] = make_float4(xv[4], xv[5], xv[6], xv[7]);
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.rn.xg) + (size_t)(grow >> 3) * (N * 8) + bg * 64 + (grow & 7);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      o[8 * i] = __float2bfloat16_rn(xv[i] * h.gain);
      ssq[i] = xv[i] * xv[i];
    }
    if (p.rn.capture) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * bg + i < p.B) p.rn.capture[(size_t)(8 * bg + i) * p.rows + grow] = xv[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {                                // over the tile's 32 rows, in a fixed order
    ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], 4);
    ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], 8);
    ssq[i] += __shfl_xor_sync(0xffffffffu, ssq[i], 16);
  }
  if (lane < 4) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s_red[we * 32 + 8 * lane + i] = ssq[i];
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  if (e < 32) p.rn.ssq[(size_t)slot * 32 + e] = ((s_red[e] + s_red[32 + e]) + s_red[64 + e]) + s_red[96 + e];
}

// EPI_POST_NORM for the 32 rows this CTA finalises; protocol, arithmetic and order as in post_norm_tile.  The op's CTAs (n of
// them, one tile each) wait for one another's sums of squares; rows and columns of a thread as in chain_resid_tile.
template <int N>
__device__ __forceinline__ void chain_post_load(const GemvParams& p, int row0, int e, ChainResid& h) {
  const int bg = e & 3, grow = row0 + (e >> 2);
  if (bg >= N / 8 || grow >= p.rows) return;
  const float4* xr = reinterpret_cast<const float4*>(p.pn.x + (size_t)grow * N + 8 * bg);
  h.x0 = xr[0]; h.x1 = xr[1];
  h.bias = p.pn.w[grow];
  h.gain = p.pn.gain ? p.pn.gain[grow] : 1.0f;
}
template <int N>
__device__ __forceinline__ void chain_post_tile(const GemvParams& p, const ChainResid& h, const float4* recv, int row0, int slot, int n, int e,
                                                float* s_red, float* s_scale, const float* s_inv, int* err) {
  constexpr int BG = N / 8;
  const int lane = e & 31, we = e >> 5, bg = e & 3, rl = e >> 2, grow = row0 + rl;
  const bool valid = bg < BG && grow < p.rows;
  float acc[8], ss[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = ss[i] = 0.f;
  if (valid) {
#pragma unroll
    for (int src = 0; src < kChainC; ++src) {
      const float4 t0 = recv[(src * 32 + rl) * (N / 4) + chain_piece<N>(rl, 2 * bg)], t1 = recv[(src * 32 + rl) * (N / 4) + chain_piece<N>(rl, 2 * bg + 1)];
      acc[0] += t0.x; acc[1] += t0.y; acc[2] += t0.z; acc[3] += t0.w;
      acc[4] += t1.x; acc[5] += t1.y; acc[6] += t1.z; acc[7] += t1.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (s_inv) acc[i] *= s_inv[8 * bg + i];
      ss[i] = acc[i] * acc[i];
    }
  }
  auto publish = [&](float* slots, bool flagged) {             // this tile's sums of ss over the rows
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 4);
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 8);
      ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], 16);
    }
    if (lane < 4) {
#pragma unroll
      for (int i = 0; i < 8; ++i) s_red[we * 32 + 8 * lane + i] = ss[i];
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    if (e < 32) {
      const float t = ((s_red[e] + s_red[32 + e]) + s_red[64 + e]) + s_red[96 + e];
      unsigned u = __float_as_uint(t);
      if (flagged && u == kSlotEmpty) u = 0x7FC00000u;
      asm volatile("st.relaxed.gpu.global.u32 [%0], %1;\n" ::"l"(slots + (size_t)slot * 32 + e), "r"(u) : "memory");
    }
  };
  publish(p.pn.slots, true);
  // the set of the next output norm: its last readers have counted themselves into done[] before this op began
  if (p.pn.clear && e < 32)
    for (int i = slot * 32 + e; i < kPushMaxCtas * 32; i += n * 32) p.pn.clear[i] = __uint_as_float(kSlotEmpty);
  {                                                            // four lanes per sequence, the same sums in every CTA
    const int b = e >> 2, part = e & 3;
    float s = 0.f;
    const long long t0 = clock64();
    bool late = false;
    for (int first = part; first < n; first += 64) {           // sixteen slots in flight
      unsigned u[16];
      bool wait = true;
      while (wait) {
        wait = false;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          u[i] = 0u;
          if (first + 4 * i < n) asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(u[i]) : "l"(p.pn.slots + (first + 4 * i) * 32 + b) : "memory");
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) wait = wait || u[i] == kSlotEmpty;
        if (wait && (late || clock64() - t0 > kWaitLimit)) {
          if (!late && err) atomicExch(err, 1);
          late = true;
          wait = false;
        }
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) s += __uint_as_float(u[i]);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (part == 0) s_scale[b] = 1.0f / sqrtf(s / (float)p.rows + p.pn.eps);
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) ss[i] = 0.f;
  if (valid) {
    float xv[8] = {h.x0.x, h.x0.y, h.x0.z, h.x0.w, h.x1.x, h.x1.y, h.x1.z, h.x1.w};
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.pn.xg) + (size_t)(grow >> 3) * (N * 8) + bg * 64 + (grow & 7);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      xv[i] += acc[i] * s_scale[8 * bg + i] * h.bias;
      o[8 * i] = __float2bfloat16_rn(xv[i] * h.gain);
      ss[i] = xv[i] * xv[i];
    }
    float4* xr = reinterpret_cast<float4*>(p.pn.x + (size_t)grow * N + 8 * bg);
    xr[0] = make_float4(xv[0], xv[1], xv[2], xv[3]);
    xr[1] = make_float4(xv[4], xv[5], xv[6], xv[7]);
    if (p.pn.capture) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * bg + i < p.B) p.pn.capture[(size_t)(8 * bg + i) * p.rows + grow] = xv[i];
    }
  }
  if (p.pn.ssq) publish(p.pn.ssq, false);
}

// Decode attention as a link (EPI_ATTEND; the launched kernel's arithmetic, attention.cu).  A unit is one of `ksplit` parts of one sequence's key head;
// CTA i takes units i, i + grid, ...  Keys and values come through the weights' ring, 64 keys (four blocks of the tiled cache) a stage: all but a sequence's
// newest are in the cache since earlier steps, so the producer fetches them while the projections before still run, and only the stage with the newest
// key waits for q/k/v.  Each epilogue warp takes one block of 16 keys of a stage.
struct ChainUnit { int bk, b, kvl, T, part, parts, begin, end; };      // keys begin .. end - 1; begin >= end: nothing
__device__ __forceinline__ ChainUnit chain_unit(const GemvParams& p, int u) {
  ChainUnit w;
  const int pairs = p.B * p.KVl;
  w.part = u / pairs;
  w.bk = u - w.part * pairs;
  w.b = w.bk / p.KVl;
  w.kvl = w.bk - w.b * p.KVl;
  w.T = p.pos[w.b] + 1;
  const int even = (((w.T + p.ksplit - 1) / p.ksplit + 63) >> 6) << 6, per = even < p.kc_per_split ? even : p.kc_per_split;
  w.parts = (w.T + per - 1) / per;
  w.begin = w.part * per;
  w.end = min(w.T, w.begin + per);
  return w;
}
// stages of a link's units that fall to this CTA
__device__ __forceinline__ int chain_attend_stages(const GemvParams& p) {
  int n = 0;
  for (int u = blockIdx.x; u < p.B * p.KVl * p.ksplit; u += gridDim.x) {
    const ChainUnit w = chain_unit(p, u);
    n += max(0, (w.end - w.begin + 63) >> 6);
  }
  return n;
}
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
  return d;
}

// One unit, by the 128 epilogue threads.  it: the ring's place, which it moves on.  scratch: 128 N floats, of which a warp's heads take G D.
template <int D, int N, int ST>
__device__ __forceinline__ void chain_attend(const GemvParams& p, const ChainUnit& u, int& it, const unsigned char* ring, uint64_t* full_bar, uint64_t* empty_bar,
                                             float* scratch, float* s_ml, int e, bool& dead, int* err) {
  constexpr int DK = D / 16, kStage = kWStage + N * 256;
  const int lane = e & 31, warp = e >> 5, g = lane >> 2, t = lane & 3, G = p.Hl / p.KVl;
  const float c = p.qk_scale * kInvLn2;
  uint32_t qf[DK][2];
  {
    const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(p.q_out) + (int64_t)u.b * p.q_pitch + (u.kvl * G + g) * D;
#pragma unroll
    for (int k = 0; k < DK; ++k) {
      qf[k][0] = g < G ? *reinterpret_cast<const uint32_t*>(q + 16 * k + 2 * t) : 0u;
      qf[k][1] = g < G ? *reinterpret_cast<const uint32_t*>(q + 16 * k + 2 * t + 8) : 0u;
    }
  }
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f, o[DK][4];
#pragma unroll
  for (int k = 0; k < DK; ++k) o[k][0] = o[k][1] = o[k][2] = o[k][3] = 0.f;
  for (int key = u.begin; key < u.end; key += 64, ++it) {
    const int s = it % ST;
    mbar_wait(&full_bar[s], (it / ST) & 1, dead, err);
    const int key0 = key + 16 * warp;
    if (key0 < u.end) {
      const uint4* blk = reinterpret_cast<const uint4*>(ring + (size_t)s * kStage) + warp * (4 * D) + lane;
      float sc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < DK; ++k) mma_bf16_16816(sc, blk[32 * k], qf[k][0], qf[k][1]);
      if (key0 + g >= u.end) sc[0] = sc[1] = -INFINITY;
      if (key0 + g + 8 >= u.end) sc[2] = sc[3] = -INFINITY;
      float b0 = fmaxf(sc[0], sc[2]), b1 = fmaxf(sc[1], sc[3]);
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) {
        b0 = fmaxf(b0, __shfl_xor_sync(0xffffffffu, b0, off));
        b1 = fmaxf(b1, __shfl_xor_sync(0xffffffffu, b1, off));
      }
      const float n0 = fmaxf(m0, b0), n1 = fmaxf(m1, b1);
      const float a0 = exp2f((m0 - n0) * c), a1 = exp2f((m1 - n1) * c);
      const float p00 = exp2f((sc[0] - n0) * c), p01 = exp2f((sc[1] - n1) * c), p10 = exp2f((sc[2] - n0) * c), p11 = exp2f((sc[3] - n1) * c);
      l0 = l0 * a0 + (p00 + p10);
      l1 = l1 * a1 + (p01 + p11);
      m0 = n0;
      m1 = n1;
      const uint32_t pb0 = movmatrix_trans(pack_bf16x2(p00, p01)), pb1 = movmatrix_trans(pack_bf16x2(p10, p11));
#pragma unroll
      for (int k = 0; k < DK; ++k) {
        o[k][0] *= a0; o[k][1] *= a1; o[k][2] *= a0; o[k][3] *= a1;
        mma_bf16_16816(o[k], blk[32 * (DK + k)], pb0, pb1);
      }
    }
    asm volatile("bar.sync 1, 128;\n" ::: "memory");             // the stage has been read
    if (e == 0) mbar_arrive(&empty_bar[s]);
  }
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, off);
    l1 += __shfl_xor_sync(0xffffffffu, l1, off);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (2 * t + h < G) {
      float* so = scratch + (warp * G + 2 * t + h) * D;
#pragma unroll
      for (int k = 0; k < DK; ++k) { so[16 * k + g] = o[k][h]; so[16 * k + g + 8] = o[k][2 + h]; }
      if (g == 0) { s_ml[warp * 8 + 2 * t + h] = h ? m1 : m0; s_ml[32 + warp * 8 + 2 * t + h] = h ? l1 : l0; }
    }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.act);
  const int64_t slot0 = (int64_t)u.bk * p.ksplit, slot = slot0 + u.part;
  for (int i = e; i < G * D; i += 128) {
    const int h = i / D, d = i - h * D;
    float M = s_ml[h], acc = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 1; w < 4; ++w) M = fmaxf(M, s_ml[w * 8 + h]);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float f = exp2f((s_ml[w * 8 + h] - M) * c);
      acc += f * scratch[(w * G + h) * D + d];
      sum += f * s_ml[32 + w * 8 + h];
    }
    if (u.parts == 1) {
      out[xcanon_offset(u.b, (u.kvl * G + h) * D + d, N)] = __float2bfloat16_rn(acc * (1.0f / sum));
    } else {
      p.partials[(slot * G + h) * D + d] = acc;
      if (d == 0) { p.out[(slot * G + h) * 2] = M * c; p.out[(slot * G + h) * 2 + 1] = sum; }        // the maximum in log2 units
    }
  }
  if (u.parts == 1) return;
  // The CTA that finishes last for this sequence's head merges the parts.  A chain of trips to L2: the counter's one release and acquire cover all
  // threads' partial results (barriers on both sides), and the first parts' values are on their way while the weights are formed.
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  if (e == 0) {
    unsigned before;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;\n" : "=r"(before) : "l"(&p.counters[u.bk]) : "memory");
    s_ml[64] = before == (unsigned)u.parts - 1u ? 1.f : 0.f;
    if (before == (unsigned)u.parts - 1u) p.counters[u.bk] = 0u;
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  if (s_ml[64] == 0.f) return;
  constexpr int kMine = N / 4;                                    // G D <= 32 N outputs, 128 threads
  float *w_m = scratch, *w_l = scratch + u.parts * G;             // [part][head]
  const float* po = p.partials + slot0 * G * D + e;
  float v[4][kMine], acc[kMine];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int j = 0; j < kMine; ++j) v[s][j] = s0 + s < u.parts && e + 128 * j < G * D ? __ldcg(po + (int64_t)(s0 + s) * G * D + 128 * j) : 0.f;
  };
  fetch(0);
  for (int i = e; i < u.parts * G; i += 128) {
    const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.out + (slot0 * G + i) * 2));
    w_m[i] = ml.x;
    w_l[i] = ml.y;
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  if (e < G) {
    float M = -INFINITY, sum = 0.f;
    for (int s = 0; s < u.parts; ++s) M = fmaxf(M, w_m[s * G + e]);
    for (int s = 0; s < u.parts; ++s) sum += exp2f(w_m[s * G + e] - M) * w_l[s * G + e];
    s_ml[e] = M;
    s_ml[8 + e] = 1.0f / sum;
  }
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
  for (int i = e; i < u.parts * G; i += 128) w_m[i] = exp2f(w_m[i] - s_ml[i % G]);
  asm volatile("bar.sync 1, 128;\n" ::: "memory");
#pragma unroll
  for (int j = 0; j < kMine; ++j) acc[j] = 0.f;
  for (int s0 = 0; s0 < u.parts; s0 += 4) {
    if (s0) fetch(s0);
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (s0 + s < u.parts) {
#pragma unroll
        for (int j = 0; j < kMine; ++j) {
          const int i = e + 128 * j;
          if (i < G * D) acc[j] += w_m[(s0 + s) * G + i / D] * v[s][j];
        }
      }
  }
#pragma unroll
  for (int j = 0; j < kMine; ++j) {
    const int i = e + 128 * j, h = i / D;
    if (i < G * D) out[xcanon_offset(u.b, (u.kvl * G + h) * D + i - h * D, N)] = __float2bfloat16_rn(acc[j] * s_ml[8 + h]);
  }
}

template <int N, bool X, int D>
__global__ void __launch_bounds__(kChainThreads, 1) gemv_chain_kernel(const __grid_constant__ ChainParamsOf<D> P, int* err) {
  constexpr int ST = kChainStages<N>;
  constexpr int kXStage = N * 256;
  constexpr int kStage = kWStage + kXStage;
  constexpr uint32_t kTmemCols = 2 * N;                          // two accumulators
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((128u >> 4) << 24);
  extern __shared__ __align__(1024) unsigned char smem[];        // ST stages, then recv[4][32][N] floats
  __shared__ __align__(8) uint64_t full_bar[ST];                 // two arrivals: weights, activations
  __shared__ __align__(8) uint64_t empty_bar[ST];
  __shared__ __align__(8) uint64_t acc_full[2];
  __shared__ __align__(8) uint64_t acc_empty[2];
  __shared__ __align__(8) uint64_t recv_full;                    // the four parts of this CTA's rows have arrived
  __shared__ __align__(8) uint64_t send_ok;                      // every CTA of the cluster has read its receive buffer
  __shared__ unsigned attended;                                  // attentions whose stages in this CTA have been read
  __shared__ uint32_t tmem_base_slot;
  __shared__ float s_inv_buf[64];
  __shared__ float s_red[128];
  __shared__ float s_scale[X ? 32 : 1];
  __shared__ __align__(16) unsigned char s_op[2][kChainOpBytes];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c = (int)cluster_ctarank(), cid = (int)blockIdx.x / kChainC, ncl = (int)gridDim.x / kChainC;
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < ST; ++s) {
      mbar_init(&full_bar[s], 2);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_full[0], 1); mbar_init(&acc_full[1], 1);
    mbar_init(&acc_empty[0], 4); mbar_init(&acc_empty[1], 4);
    mbar_init(&recv_full, 1);
    mbar_init(&send_ok, kChainC);
    attended = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  bool dead = false;
  pdl_launch_dependents();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");      // the peers' barriers are initialised: waited for before the first send

  if (warp == 0) {
    // ---------------- weights ----------------
    if (elect_one()) {
      uint64_t pol_w;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol_w));
      int it = 0;
      bool after_launch = false;
      for (int o = 0; o < P.n_ops; ++o) {
        if (D > 0 && P.op[o].epi == EPI_ATTEND) {
          const GemvParams& p = P.op[o];
          if (!after_launch) pdl_wait();                         // positions and cache, unlike weights, are the step's
          after_launch = true;
          bool fresh = o == 0;
          for (int u = blockIdx.x; u < p.B * p.KVl * p.ksplit; u += gridDim.x) {
            const ChainUnit w = chain_unit(p, u);
            const __nv_bfloat16* kv = reinterpret_cast<const __nv_bfloat16*>(p.kv_layer) + w.b * p.kv_batch_stride + w.kvl * p.kv_head_stride;
            for (int key = w.begin; key < w.end; key += 64, ++it) {
              if (!fresh && key + 64 >= w.T) {                   // the newest key and value come from the projection before
                chain_wait_done(P.done + (o - 1) * kChainLine, chain_ctas(P.op[o - 1], ncl), dead, err);
                asm volatile("fence.proxy.async;\n" ::: "memory");
                fresh = true;
              }
              const int s = it % ST, k = it / ST;
              const uint32_t bytes = (uint32_t)(min(4, (w.end - key + 15) >> 4) * 64 * D);
              mbar_wait(&empty_bar[s], (k & 1) ^ 1, dead, err);
              mbar_expect_tx(&full_bar[s], bytes);
              bulk_g2s(smem + s * kStage, kv + (int64_t)(key >> 4) * (32 * D), bytes, &full_bar[s], pol_w);
              mbar_arrive(&full_bar[s]);                         // (there are no activations)
            }
          }
          continue;
        }
        const int KS = (P.op[o].K + 127) >> 7, nrbg = (P.op[o].rows + 127) >> 7;
        const int ks0 = c * KS / kChainC, ks1 = (c + 1) * KS / kChainC;
        const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(P.op[o].W);
        for (int r = cid; r < nrbg; r += ncl)
          for (int ks = ks0; ks < ks1; ++ks, ++it) {
            const int s = it % ST, k = it / ST;
            mbar_wait(&empty_bar[s], (k & 1) ^ 1, dead, err);
            mbar_expect_tx(&full_bar[s], (uint32_t)kWStage);
            bulk_g2s(smem + s * kStage, W + ((int64_t)r * KS + ks) * 16384, (uint32_t)kWStage, &full_bar[s], pol_w);
          }
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  } else if (warp == 6) {
    // ---------------- activations ----------------
    pdl_wait();
    if (elect_one()) {
      uint64_t pol_x;
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(pol_x));
      int it = 0;
      for (int o = 0; o < P.n_ops; ++o) {
        if (D > 0 && P.op[o].epi == EPI_ATTEND) {
          it += chain_attend_stages(P.op[o]);
          continue;
        }
        const int KS = (P.op[o].K + 127) >> 7, nrbg = (P.op[o].rows + 127) >> 7;
        const int ks0 = c * KS / kChainC, ks1 = (c + 1) * KS / kChainC;
        if (cid >= nrbg || ks0 >= ks1) continue;
        if (o > 0) {
          chain_wait_done(P.done + (o - 1) * kChainLine, chain_ctas(P.op[o - 1], ncl), dead, err);
          asm volatile("fence.proxy.async;\n" ::: "memory");      // the bulk copies read what the epilogues stored
        }
        const __nv_bfloat16* xsrc = reinterpret_cast<const __nv_bfloat16*>(P.op[o].x);
        for (int r = cid; r < nrbg; r += ncl)
          for (int ks = ks0; ks < ks1; ++ks, ++it) {
            const int s = it % ST, k = it / ST;
            mbar_wait(&empty_bar[s], (k & 1) ^ 1, dead, err);
            mbar_expect_tx(&full_bar[s], (uint32_t)kXStage);
            bulk_g2s(smem + s * kStage + kWStage, xsrc + (int64_t)ks * (128 * N), (uint32_t)kXStage, &full_bar[s], pol_x);
          }
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  } else if (warp == 1) {
    // ---------------- MMA issue ----------------
    if (elect_one()) {
      int it = 0, seg = 0;
      unsigned attentions = 0;
      for (int o = 0; o < P.n_ops; ++o) {
        if (D > 0 && P.op[o].epi == EPI_ATTEND) {
          if (attentions == 0) pdl_wait();
          const int n = chain_attend_stages(P.op[o]);
          // Not before they have been read: a barrier's parity tells a stage's fills apart only from the one before, and the stages skipped here may
          // go round the ring several times.
          if (n > 0) chain_wait_shared(&attended, ++attentions, dead, err);
          it += n;
          continue;
        }
        const int KS = (P.op[o].K + 127) >> 7, nrbg = (P.op[o].rows + 127) >> 7;
        const int n_steps = (c + 1) * KS / kChainC - c * KS / kChainC;
        if (n_steps == 0) continue;
        for (int r = cid; r < nrbg; r += ncl, ++seg) {
          const int buf = seg & 1;
          mbar_wait(&acc_empty[buf], ((seg >> 1) & 1) ^ 1, dead, err);
          tc_fence_after();
          for (int i = 0; i < n_steps; ++i, ++it) {
            const int s = it % ST, k = it / ST;
            mbar_wait(&full_bar[s], k & 1, dead, err);
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + s * kStage);
            const uint64_t adesc = smem_desc(sa, 2048, 128);
            const uint64_t bdesc = smem_desc(sa + kWStage, N * 16, 128);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              tc_mma_f16(tmem_base + buf * N, adesc + (uint64_t)(j * (4096 >> 4)), bdesc + (uint64_t)(j * ((2 * N * 16) >> 4)), kIdesc,
                         (i == 0 && j == 0) ? 0u : 1u);
            tc_commit(&empty_bar[s]);
            if (i == n_steps - 1) tc_commit(&acc_full[buf]);
          }
        }
      }
    }
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  } else {
    // ---------------- epilogue ----------------
    pdl_wait();
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    const int q = warp & 3, e = tid - 64;
    const float4* recv = reinterpret_cast<const float4*>(smem + ST * kStage);
    const uint32_t to = dsmem_addr(smem_u32(recv) + (uint32_t)((c * 32 + lane) * N * 4), (uint32_t)q);
    const uint32_t to_bar = dsmem_addr(smem_u32(&recv_full), (uint32_t)q);
    int seg = 0, g = 0;                        // accumulators drained, tiles exchanged
    int it = 0;                                // the ring's stages, which only attention reads here
    // The links' parameters, a link ahead: a constant-bank line that is read for the first time takes about half a microsecond, one after the other, and
    // q/k/v's epilogue needs eight of them.
    auto fetch_op = [&](int o) {
      const uint32_t* from = reinterpret_cast<const uint32_t*>(&P.op[o]);
      for (int i = e; i < kChainOpBytes / 4; i += 128) reinterpret_cast<uint32_t*>(s_op[o & 1])[i] = from[i];
    };
    fetch_op(0);
    asm volatile("bar.sync 1, 128;\n" ::: "memory");
    for (int o = 0; o < P.n_ops; ++o) {
      const GemvParams& p = *reinterpret_cast<const GemvParams*>(s_op[o & 1]);
      if (D > 0 && p.epi == EPI_ATTEND) {
        const int units = p.B * p.KVl * p.ksplit;
        if (o > 0 && (int)blockIdx.x < units) {
          if (e == 0) chain_wait_done(P.done + (o - 1) * kChainLine, chain_ctas(P.op[o - 1], ncl), dead, err);
          asm volatile("bar.sync 1, 128;\n" ::: "memory");
        }
        if (o + 1 < P.n_ops) fetch_op(o + 1);                     // (the other half: everybody is done with the link before)
        if ((int)blockIdx.x >= units) {
          asm volatile("bar.sync 1, 128;\n" ::: "memory");
          continue;
        }
        // the receive buffer is free: what the peers send next needs this link's outputs
        const int it0 = it;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
          const ChainUnit w = chain_unit(p, u);
          if (w.begin < w.end) chain_attend<(D > 0 ? D : 64), N, ST>(p, w, it, smem, full_bar, empty_bar, const_cast<float*>(reinterpret_cast<const float*>(recv)), s_red, e, dead, err);
        }
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        if (e == 0 && it != it0) asm volatile("red.release.cta.shared.add.u32 [%0], 1;\n" ::"r"(smem_u32(&attended)) : "memory");
        if (e == 0 && o + 1 < P.n_ops) asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(P.done + o * kChainLine) : "memory");
        continue;
      }
      const int KS = (p.K + 127) >> 7, nrbg = (p.rows + 127) >> 7;
      const int n_steps = (c + 1) * KS / kChainC - c * KS / kChainC;
      if (cid >= nrbg) {
        if (o + 1 < P.n_ops) fetch_op(o + 1);
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
        continue;
      }
      if (D > 0) it += n_steps * ((nrbg - cid + ncl - 1) / ncl);
      const float* s_inv = p.inv.ssq ? s_inv_buf : nullptr;
      if (o > 0) {
        if (e == 0) chain_wait_done(P.done + (o - 1) * kChainLine, chain_ctas(P.op[o - 1], ncl), dead, err);
        asm volatile("bar.sync 1, 128;\n" ::: "memory");
      }
      compute_inv_scale(p.inv, s_inv_buf, e);
      if (o + 1 < P.n_ops) fetch_op(o + 1);
      for (int r = cid; r < nrbg; r += ncl, ++g) {
        const int row0 = r * 128 + c * 32;
        // what the epilogue reads besides the accumulators, fetched while the weights stream
        ChainResid h;
        RowConst rc[2];
        float factor[2][4];
        if (p.epi == EPI_RESID_NORM) {
          chain_resid_load<N>(p, row0, e, h);
        } else if (X && p.epi == EPI_POST_NORM) {
          chain_post_load<N>(p, row0, e, h);
        } else {
          rc[0] = row_const(p, row0 + (lane & 15));
          rc[1] = row_const(p, row0 + 16 + (lane & 15));
          if (X && p.epi == EPI_GELU_TOKEN) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int b = 4 * (e >> 4) + (i & 3), row = row0 + 16 * (i >> 2) + (lane & 15);
              factor[i >> 2][i & 3] = b < p.B && row < p.rows ? token_factor(p, b, row) : 0.f;
            }
          }
        }
        float v[N];
        if (n_steps > 0) {
          const int buf = seg & 1;
          mbar_wait(&acc_full[buf], (seg >> 1) & 1, dead, err);
          tc_fence_after();
          tmem_load_row<N>(v, tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(buf * N));
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[buf]);
          ++seg;
        } else {
#pragma unroll
          for (int i = 0; i < N; ++i) v[i] = 0.f;
        }
        if (e == 0) mbar_expect_tx(&recv_full, 128u * N * 4u);
        if (g > 0) mbar_wait_cluster(&send_ok, (g - 1) & 1, dead, err);
#pragma unroll
        for (int i = 0; i < N / 4; ++i)
          dsmem_store4_async(to + 16u * chain_piece<N>(lane, i), to_bar, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        mbar_wait_cluster(&recv_full, g & 1, dead, err);
        if (p.epi == EPI_RESID_NORM) {
          chain_resid_tile<N>(p, h, recv, row0, r * kChainC + c, e, s_red);
        } else if (X && p.epi == EPI_POST_NORM) {
          chain_post_tile<N>(p, h, recv, row0, r * kChainC + c, nrbg * kChainC, e, s_red, s_scale, s_inv, err);
        } else {
          const int row16 = lane & 15, cg = e >> 4;
          if (cg < N / 4) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              float v4[4] = {0.f, 0.f, 0.f, 0.f};
              const int rl = 16 * j + row16;
#pragma unroll
              for (int src = 0; src < kChainC; ++src) {
                const float4 t = recv[(src * 32 + rl) * (N / 4) + chain_piece<N>(rl, cg)];
                v4[0] += t.x; v4[1] += t.y; v4[2] += t.z; v4[3] += t.w;
              }
              row_epilogue<4, N, X>(p, v4, row0 + rl, 4 * cg, s_inv, rc[j], factor[j]);
            }
          }
        }
        const bool last = r + ncl >= nrbg && o + 1 < P.n_ops;
        asm volatile("bar.sync 1, 128;\n" ::: "memory");         // the receive buffer has been read
        // The barrier puts every thread's stores before thread 0's release, which covers them.  (The bulk copies that read them are behind a proxy fence
        // on the reader's side, after its acquire; another one here, by all threads, cost a microsecond per link.)
        if (last && e == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(P.done + o * kChainLine) : "memory");
        if (e < kChainC) mbar_arrive_remote(dsmem_addr(smem_u32(&send_ok), (uint32_t)e));
      }
    }
  }
  if (dead) {                                  // copies may still be on their way into this shared memory
    const long long t0 = clock64();
    while (clock64() - t0 < kWaitLimit / 100) {}
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();                          // no peer sends into a CTA that has gone
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
  }
  if (tid == 0) {                              // the last CTA out leaves the counters empty
    unsigned* gone = P.done + kChainMaxAttend * kChainLine;
    __threadfence();
    if (atomicAdd(gone, 1u) == gridDim.x - 1u) {
      for (int o = 0; o < P.n_ops; ++o) P.done[o * kChainLine] = 0u;
      *gone = 0u;
    }
  }
}

bool layered_epilogue(const GemvParams& p) {
  return p.epi == EPI_STORE_RELU2 || p.epi == EPI_STORE_ACT || p.epi == EPI_GELU_TOKEN || p.epi == EPI_POST_NORM || p.softcap > 0.f;
}

template <int Bp>
constexpr size_t cluster_smem() {
  return (size_t)kStages * (kWStage + Bp * 256) + 128 * Bp * 4 + 1024;
}

template <int Bp>
int32_t launch_cluster(Ctx* ctx, const GemvParams& p, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ceil_div(p.rows, 128) * p.cluster));
  cfg.blockDim = dim3(kTcThreads);
  cfg.dynamicSmemBytes = cluster_smem<Bp>();
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  LMB_CUDA(cudaLaunchKernelEx(&cfg, layered_epilogue(p) ? gemv_cl_kernel<Bp, true> : gemv_cl_kernel<Bp, false>, p, ctx->dev_err));
  ctx->launches++;
  return LMB200_OK;
}

// The largest cluster size (8, 4, 2) that keeps rows/128 x C CTAs on the device in one wave and
// gives every CTA at least one k step; 0: use the stream-K kernel.
template <int Bp>
int cluster_choice(const Ctx* ctx, int rows, int K) {
  const int nrbg = (int)ceil_div(rows, 128), KS = (int)ceil_div(K, 128);
  for (int C = 8; C >= 2; C >>= 1) {
    if (C > KS || (int64_t)nrbg * C > ctx->sm_count) continue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nrbg * C));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = cluster_smem<Bp>();
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n_clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&n_clusters, gemv_cl_kernel<Bp, false>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (n_clusters >= nrbg) return C;
  }
  return 0;
}

template <typename WT, int NB, int MT, int STAGES>
int32_t launch_ring(Ctx* ctx, const GemvParams& p, cudaStream_t stream) {
  constexpr int Bp = 8 * NB, RPC = 2 * MT * 16;
  const size_t xs_bytes = (size_t)p.kc_per_split * Bp * 32 * sizeof(WT);
  const size_t red_bytes = (size_t)4 * RPC * (Bp + 1) * sizeof(float);
  const size_t smem = xs_bytes > red_bytes ? xs_bytes : red_bytes;
  LMB_REQUIRE(smem <= kMaxSmem, "gemv: %zu bytes of shared memory exceed the configured %zu", smem, kMaxSmem);
  dim3 grid((unsigned)ceil_div(p.RB, 2 * MT), (unsigned)p.ksplit);
  LMB_CUDA(launch_k(gemv_ring_kernel<WT, NB, MT, STAGES>, grid, dim3(kRingThreads), smem, stream, p));
  ctx->launches++;
  return LMB200_OK;
}

template <int Bp>
constexpr size_t stream_smem() {
  return (size_t)kStages * (kWStage + Bp * 256) + 1024;
}

template <int Bp>
int32_t launch_bf16(Ctx* ctx, const GemvParams& p, cudaStream_t stream) {
  if (p.cluster >= 1) return launch_cluster<Bp>(ctx, p, stream);
  LMB_REQUIRE(p.epi != EPI_RESID_NORM && p.epi != EPI_POST_NORM, "gemv: this epilogue needs a plan of gemv_plan_resid");
  LMB_CUDA(launch_k(layered_epilogue(p) ? gemv_tc_kernel<Bp, true> : gemv_tc_kernel<Bp, false>, dim3(p.grid), dim3(kTcThreads), stream_smem<Bp>(), stream, p, ctx->dev_err));
  ctx->launches++;
  return LMB200_OK;
}

template <int N>
cudaLaunchConfig_t chain_config(cudaLaunchAttribute* attr, int clusters, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * kChainC));
  cfg.blockDim = dim3(kChainThreads);
  cfg.dynamicSmemBytes = chain_smem<N>();
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kChainC;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cfg;
}

template <int N>
int chain_clusters() {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = chain_config<N>(attr, 1, 0);
  cfg.numAttrs = 1;
  int n = 0, m = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemv_chain_kernel<N, false, 0>, &cfg) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&m, gemv_chain_kernel<N, true, 0>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return std::min(n, m);
}

template <int N, int D>
int32_t launch_chain_of(Ctx* ctx, const GemvParams* op, int n, unsigned* done, int clusters, cudaStream_t stream) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = chain_config<N>(attr, clusters, stream);
  static_assert(sizeof(ChainParamsOf<D>) <= 32 * 1024 - 64, "kernel parameters");
  ChainParamsOf<D> P;
  bool x = false;
  for (int i = 0; i < n; ++i) {
    P.op[i] = op[i];
    x = x || layered_epilogue(op[i]);
  }
  P.n_ops = n;
  P.done = done;
  if constexpr (D > 0) {
    LMB_REQUIRE(!x, "gemv chain: attention beside a layered decoder's projections");
    LMB_CUDA(cudaLaunchKernelEx(&cfg, gemv_chain_kernel<N, false, D>, P, ctx->dev_err));
  } else {
    LMB_CUDA(cudaLaunchKernelEx(&cfg, x ? gemv_chain_kernel<N, true, 0> : gemv_chain_kernel<N, false, 0>, P, ctx->dev_err));
  }
  ctx->launches++;
  return LMB200_OK;
}
template <int N>
int32_t launch_chain(Ctx* ctx, const GemvParams* op, int n, unsigned* done, int clusters, int D, cudaStream_t stream) {
  switch (D) {
    case 0: return launch_chain_of<N, 0>(ctx, op, n, done, clusters, stream);
    case 64: return launch_chain_of<N, 64>(ctx, op, n, done, clusters, stream);
    case 96: return launch_chain_of<N, 96>(ctx, op, n, done, clusters, stream);
    default: return launch_chain_of<N, 128>(ctx, op, n, done, clusters, stream);
  }
}

constexpr int kMtF32 = 1;
constexpr size_t kMaxXsBytes = 96 * 1024;

}  // namespace

void gemv_set_variant(int variant) { (void)variant; g_variant = GEMV_TCGEN05; }
int gemv_variant() { return g_variant; }

void gemv_prefetch_next(GemvParams& p, const Ctx* ctx, int dtype, const void* next_W, int next_rows, int next_K,
                        const GemvPlan& next_plan) {
  (void)ctx;
  static const int budget_mb = [] { const char* e = getenv("LMB200_L2_PREFETCH_MB"); return e ? atoi(e) : 24; }();
  if (dtype != LMB200_BF16 || g_variant != GEMV_TCGEN05 || budget_mb <= 0 || !next_W) return;
  const int KS = (int)ceil_div(next_K, 128), nrbg = (int)ceil_div(next_rows, 128);
  const int64_t U = (int64_t)nrbg * KS;
  const int parts = next_plan.cluster >= 1 ? nrbg * next_plan.cluster : next_plan.grid;
  if (parts <= 0 || U / parts < 1) return;
  int64_t chunk = ((int64_t)budget_mb * 1000000 / 32768) / parts;
  if (chunk < 1) chunk = 1;
  if (chunk > U / parts) chunk = U / parts;
  p.pf_base = next_W; p.pf_units = (int)U; p.pf_parts = parts; p.pf_chunk = (int)chunk;
}

GemvPlan gemv_plan(const Ctx* ctx, int dtype, int B, int rows, int K) {
  GemvPlan pl;
  if (dtype == LMB200_BF16) {
    const int Bp = Layout<__nv_bfloat16>::batch_pad(B);
    const int KS = (int)ceil_div(K, 128);
    const int nrbg = (int)ceil_div(rows, 128);
    const int64_t U = (int64_t)nrbg * KS;
    int G = ctx->sm_count;
    if (G > U) G = (int)U;
    pl.grid = G;
    const int64_t upc_min = U / G;                       // >= 1
    pl.ksplit = (int)ceil_div(KS, upc_min) + 1;          // contributors reserved per row group
    pl.kc_per_split = KS;
    pl.partial_floats = (int64_t)nrbg * pl.ksplit * 128 * Bp;   // [row group][contributor][128 x Bp]
    pl.n_counters = nrbg * 8;
    // small matrices: a cluster per row group, partials through distributed shared memory
    const char* ce = getenv("LMB200_GEMV_CLUSTER");             // 0: never; N (MB): size limit, default 128
    const int64_t limit_mb = ce ? atoi(ce) : 128;
    if (g_variant == GEMV_TCGEN05 && (int64_t)rows * K * 2 <= limit_mb * 1000000)
      pl.cluster = Bp == 16 ? cluster_choice<16>(ctx, rows, K) : cluster_choice<32>(ctx, rows, K);
    return pl;
  }
  const int Bp = Layout<float>::batch_pad(B);
  const int RB = (int)ceil_div(rows, 16), KC = (int)ceil_div(K, 32);
  const int MT = kMtF32;
  const int RPC = 2 * MT * 16;
  const size_t esz = 4;
  const int nrbg = (int)ceil_div(RB, 2 * MT);
  // One CTA per SM is resident (register ring).  Pick the k-split that minimises
  //   waves * (chunks per CTA + fixed cost of staging x and the epilogue, in chunk units)
  // with the activation slice fitting shared memory and at least one chunk per k-warp.
  const int per_max = (int)(kMaxXsBytes / (Bp * 32 * esz));
  const int kFixed = 6;
  int best_ks = 1, best_per = KC;
  double best_cost = 1e30;
  for (int ks_try = 1; ks_try <= KC; ++ks_try) {
    const int per_try = (int)ceil_div(KC, ks_try);
    if (per_try > per_max) continue;
    if (per_try < 4 && ks_try > 1) break;
    const int ks_eff = (int)ceil_div(KC, per_try);
    const double waves = (double)ceil_div((int64_t)nrbg * ks_eff, ctx->sm_count);
    const double cost = waves * (per_try + kFixed) + 0.02 * ks_eff;
    if (cost < best_cost) { best_cost = cost; best_ks = ks_eff; best_per = per_try; }
  }
  pl.ksplit = best_ks;
  pl.kc_per_split = best_per;
  pl.grid = nrbg * best_ks;
  pl.partial_floats = best_ks > 1 ? (int64_t)nrbg * best_ks * RPC * Bp : 0;
  pl.n_counters = nrbg;
  return pl;
}

GemvPlan gemv_plan_resid(const Ctx* ctx, int B, int rows, int K) {
  GemvPlan pl = gemv_plan(ctx, LMB200_BF16, B, rows, K);
  const int Bp = Layout<__nv_bfloat16>::batch_pad(B);
  const int nrbg = (int)ceil_div(rows, 128);
  pl.cluster = 0;
  if (g_variant != GEMV_TCGEN05) return pl;
  pl.cluster = Bp == 16 ? cluster_choice<16>(ctx, rows, K) : cluster_choice<32>(ctx, rows, K);
  if (pl.cluster == 0 && nrbg <= ctx->sm_count && nrbg <= kPushMaxCtas) pl.cluster = 1;
  if (nrbg * pl.cluster > kPushMaxCtas) pl.cluster = 0;
  return pl;
}

int gemv_plan_ctas(const GemvPlan& pl, int rows) {
  return pl.cluster >= 1 ? (int)ceil_div(rows, 128) * pl.cluster : pl.grid;
}

// What the chain saves per GEMV is a launch, about 6 us of which its ring covers 3; what it costs is that a row group has four CTAs.  By
// itself a projection runs on clusters of eight while 15 of them hold its row groups, and then streams faster than here, unless it is so
// short that eight, or four, have no unit of k each.  Hence chained up to 3 and from 16 row groups of the residual width on.  Per layer of a
// Llama, one launch per GEMV -> chained, batch 1 | 32: width 256, feed-forward 704 28 -> 26 | 32 -> 30 us; 512, 1408 26.1 -> 27.4 | 29.6 -> 29.8;
// 1024, 2816 30.2 -> 33.2 | 34.8 -> 40.8; 1536, 4224 39.0 -> 41.9 | 50.0 -> 51.7; 2048, 5632 53.2 -> 47.4 | 64.4 -> 58.9; 3072, 8448 69.6 -> 63.2 |
// 85.5 -> 82.2 (1792 and 1920 go either way with the feed-forward's width).  A Gibutar's chains of two GEMVs: the same line, from 24 row groups on
// above 16 sequences, where an exchange moves twice the bytes (eight layers, batch 16 | 32: 2048 458 -> 445 | 577 -> 598 us; four, 3072 351 -> 348 |
// 397 -> 379).  Sublayers normed on their output make chains of six GEMVs, which gain at every width (Kevatar, four layers, batch 16: 512
// 238 -> 216 us, 1024 277 -> 247, 2048 387 -> 330).
constexpr int kChainGroups = 16;
int gemv_chain_clusters(int B, int width, int per_chain, bool output_norms) {
  const char* e = getenv("LMB200_GEMV_CHAIN");                  // 0: one launch per GEMV, 1: chained wherever it can be (A/B runs)
  if ((e && atoi(e) == 0) || g_variant != GEMV_TCGEN05) return 0;
  const int64_t groups = ceil_div(width, 128);
  if (groups * kChainC > kSsqSlots) return 0;                   // a projection leaves 4 sums of squares per row group
  const bool wide_batch = Layout<__nv_bfloat16>::batch_pad(B) > 16;
  if (!e && per_chain < 6 && groups > 3 && groups < (per_chain < 4 && wide_batch ? 24 : kChainGroups)) return 0;
  const int n = wide_batch ? chain_clusters<32>() : chain_clusters<16>();
  return output_norms && groups > n ? 0 : n;                    // an output norm needs every row group resident at once
}
int64_t gemv_chain_scratch_bytes() { return (int64_t)(kChainMaxAttend + 1) * kChainLine * 4; }

// Whether an attention link gains: the keys' time its busiest CTA takes, and what an even spread over the CTAs would take (gemv_chain_attention_plan's comment).
static bool link_pays(int64_t busiest, int64_t even, int B, int G, int D) {
  const int64_t over = busiest - even, kept = std::min<int64_t>(even, 16000);
  if (D == 64) return busiest <= 1050 || (over <= 200 && busiest <= 2300);
  if (G < 4) return over <= (Layout<__nv_bfloat16>::batch_pad(B) == 16 ? 950 : 900 + kept / 20);
  return over <= 1050 + kept * 2 / 25;
}

// One unit per CTA and round; a unit costs about 48 keys' time beside its keys (queries, the four warps' merge), and one of several parts 100 more (partial
// results out, a counter).  The merge at the end takes 4 us, in which a CTA streams some 640 keys (Llama-3-8B shape, one sequence of 1031 keys, nine parts: the
// last one 11.8 us after q/k/v, the others 4.6).  Without the 100 a head was cut into too many parts (28 sequences of 8190 keys: 17 rounds of units; the step
// 1087 us, 954 with two).  The parts' pairs of maximum and sum must fit the receive buffer: at most 64.  The four warps' sums of a unit lie there too: 128 N floats for
// 4 G D.
//   Whether it is worth it: the link saves a launch and its latency, but takes whole units, where the launched kernel's many CTAs even out.  What the busiest CTA
// takes longer than an even spread of the keys tells gains from losses (670 sessions: width 2048 to 8192, head dimension 96 and 128, batch 1 to 32, 64 to 32768 keys;
// up to the line the link gains 0 to 25 us a layer and loses 3 % at worst, above it loses up to 50 us).  Per layer, launched -> link, Llama-3-8B shape: 1031 keys,
// batch 1 (841 keys over) -4.9, batch 17 (1151: 136 heads for 132 CTAs) +2.3; 2050 keys, batch 17 (1872) +10; 8190 keys, batch 32 (596) -16.9, batch 30 (1598) -14.8, batch
// 28 (2450) +4.4, batch 17 (2914) +12.  With a key head per head the launched kernel has a quarter of the parts to merge and is harder to beat: 8190 keys, batch 8 (298) -5.4, 16
// (1193) +13.5, 20 (1491) -9, 26 (3703) +32.  Head dimension 64 is bound by the work per stage, not by its bytes: 1031 keys, batch 1, 16, 17 -2.1, -2.7, +4.1; 4096
// keys, batch 1, 16 +1.2, +3.0; 8190 keys, batch 32 +20.
//   A short context in a large cache leaves most of a head's parts empty, and a CTA still looks at each: from four rounds of parts on that costs more than the
// launch (22 sequences, 100 keys in a cache of 8256: 426 -> 441 us).
//   Narrow models are chained up to three row groups, where an attention between is launched: at width 256 and 384 a link gained 5 % at 64 keys and lost up to
// 12 % at 1031.
bool gemv_chain_attention_plan(int clusters, int width, int B, int KVl, int G, int D, int capacity, int* keys_per_cta, int* nsplit) {
  const char* e = getenv("LMB200_CHAIN_ATTENTION");             // 0: attention as a launch of its own, 1: a link wherever it can be (A/B runs)
  if ((e && atoi(e) == 0) || clusters == 0 || ceil_div(width, 128) < kChainGroups) return false;
  if (!(D == 64 || D == 96 || D == 128) || G < 1 || G > 8 || G * D > 32 * Layout<__nv_bfloat16>::batch_pad(B)) return false;
  const int64_t pairs = (int64_t)B * KVl, ctas = (int64_t)clusters * kChainC, cap = round_up(capacity, 64);
  int64_t best = cap, best_cost = ceil_div(pairs, ctas) * (cap + 48);
  for (int64_t k = 64; k < cap; k += 64) {
    const int64_t ns = ceil_div(cap, k);
    if (ns > 64) continue;
    const int64_t cost = ceil_div(pairs * ns, ctas) * (k + 148) + 640;
    if (cost < best_cost) { best_cost = cost; best = k; }
  }
  *keys_per_cta = (int)best;
  *nsplit = (int)ceil_div(cap, best);
  if (e) return true;
  if (D != 64 && *nsplit > 1 && pairs * *nsplit > 3 * ctas) return false;
  return link_pays(best_cost, pairs * cap / ctas, B, G, D);
}

// The units as chain_unit makes them at these positions, CTA by CTA.  One sequence far longer than the others is a few CTAs' work in the link, while the launched
// kernel cuts it for all: 16 sequences in a cache of 8256, one of 8190 keys and the others of 60, 456 -> 624 us a step (Llama-3-8B shape, four layers), half of them
// long 573 -> 625, all within 40 keys of one another 737 -> 697.
bool gemv_chain_attention_spreads(int clusters, int B, int KVl, int G, int D, int keys_per_cta, int nsplit, const int* pos) {
  const char* e = getenv("LMB200_CHAIN_ATTENTION");
  if (e) return atoi(e) != 0;
  const int64_t pairs = (int64_t)B * KVl, ctas = (int64_t)clusters * kChainC;
  std::vector<int64_t> load(ctas, 0);
  int64_t total = 0;
  bool split = false;
  for (int64_t u = 0; u < pairs * nsplit; ++u) {
    const int T = pos[u % pairs / KVl] + 1, per = (int)std::min<int64_t>(round_up(ceil_div(T, nsplit), 64), keys_per_cta);
    const int64_t begin = u / pairs * per;
    if (begin >= T) continue;
    split = split || T > per;
    total += std::min<int64_t>(T - begin, per);
    load[u % ctas] += std::min<int64_t>(T - begin, per) + (T > per ? 148 : 48);
  }
  return link_pays(*std::max_element(load.begin(), load.end()) + (split ? 640 : 0), total / ctas, B, G, D);
}

int32_t GemvChain::add(const GemvParams& p) {
  if (clusters == 0) return gemv_launch(ctx, LMB200_BF16, p, stream);
  // Every tile costs an exchange inside the cluster, about 2.4 us.  A GEMV of several tiles per cluster whose tiles stream for less than
  // that (a unit is 0.57 us) is better off alone: 51865 x 512 takes 12 us by itself and 31 us here.  Not where a norm follows: its consumer
  // reads the slots that the chain kernel leaves (slots()), a launch of its own leaves as many as its plan has CTAs.
  const bool norm = p.epi == EPI_RESID_NORM || p.epi == EPI_POST_NORM;
  if (!norm && ceil_div(p.rows, 128) > clusters && p.K <= 3 * 128 * kChainC) {
    LMB_TRY(flush());
    return gemv_launch(ctx, LMB200_BF16, p, stream);
  }
  if (n == (attention ? kChainMaxAttend : kChainMax)) LMB_TRY(flush());
  op[n++] = p;
  return LMB200_OK;
}
int32_t GemvChain::add_attention(const AttnParams& a) {
  LMB_REQUIRE(clusters && attention && a.counters && a.pos, "gemv chain: no attention here");
  if (n == kChainMaxAttend) LMB_TRY(flush());
  GemvParams p;
  p.epi = EPI_ATTEND;
  p.B = a.B; p.KVl = a.KVl; p.Hl = a.KVl * a.G; p.D = a.D;
  p.q_out = const_cast<void*>(a.q); p.q_pitch = a.q_pitch;
  p.kv_layer = const_cast<void*>(a.kv_layer); p.kv_batch_stride = a.kv_batch_stride; p.kv_head_stride = a.kv_head_stride;
  p.pos = a.pos; p.qk_scale = a.scale;
  p.ksplit = a.nsplit; p.kc_per_split = a.keys_per_cta;
  p.partials = a.part_o; p.out = a.part_ml; p.counters = a.counters;
  p.act = a.out;
  op[n++] = p;
  return LMB200_OK;
}
int32_t GemvChain::flush() {
  const int count = n;
  n = 0;
  if (count == 0) return LMB200_OK;
  if (count == 1 && op[0].epi != EPI_RESID_NORM && op[0].epi != EPI_POST_NORM && op[0].epi != EPI_ATTEND) return gemv_launch(ctx, LMB200_BF16, op[0], stream);
  int most = 1, D = 0;
  for (int i = 0; i < count; ++i) {
    LMB_REQUIRE(op[i].B >= 1 && op[i].B <= 32 && op[i].push.n <= 1 && !op[i].rn.sum && !op[i].inv.sum, "gemv chain: op %d cannot run here", i);
    LMB_REQUIRE(op[i].epi != EPI_POST_NORM || ceil_div(op[i].rows, 128) <= std::min(clusters, kPushMaxCtas / kChainC),
                "gemv chain: %d rows are more than one wave", op[i].rows);
    if (op[i].epi == EPI_ATTEND) {
      D = op[i].D;
      most = clusters;
    }
    most = std::max(most, (int)ceil_div(op[i].rows, 128));
  }
  LMB_REQUIRE(D > 0 || count <= kChainMax, "gemv chain: %d links", count);
  const int g = std::min(most, clusters);
  return Layout<__nv_bfloat16>::batch_pad(op[0].B) == 16 ? launch_chain<16>(ctx, op, count, done, g, D, stream) : launch_chain<32>(ctx, op, count, done, g, D, stream);
}

// Raise the dynamic shared-memory limit of every instantiation once per device, outside any
// stream capture.
int32_t gemv_configure() {
#define LMB_CFG(KERN, BYTES) \
  LMB_CUDA(cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(BYTES)))
  LMB_CFG((gemv_ring_kernel<float, 1, kMtF32, 3>), kMaxSmem);
  LMB_CFG((gemv_ring_kernel<float, 2, kMtF32, 3>), kMaxSmem);
  LMB_CFG((gemv_ring_kernel<float, 4, kMtF32, 2>), kMaxSmem);
  LMB_CFG((gemv_tc_kernel<16, false>), stream_smem<16>());
  LMB_CFG((gemv_tc_kernel<16, true>), stream_smem<16>());
  LMB_CFG((gemv_tc_kernel<32, false>), stream_smem<32>());
  LMB_CFG((gemv_tc_kernel<32, true>), stream_smem<32>());
  LMB_CFG((gemv_cl_kernel<16, false>), cluster_smem<16>());
  LMB_CFG((gemv_cl_kernel<16, true>), cluster_smem<16>());
  LMB_CFG((gemv_cl_kernel<32, false>), cluster_smem<32>());
  LMB_CFG((gemv_cl_kernel<32, true>), cluster_smem<32>());
  LMB_CFG((gemv_chain_kernel<16, false, 0>), chain_smem<16>());
  LMB_CFG((gemv_chain_kernel<16, true, 0>), chain_smem<16>());
  LMB_CFG((gemv_chain_kernel<32, false, 0>), chain_smem<32>());
  LMB_CFG((gemv_chain_kernel<32, true, 0>), chain_smem<32>());
  LMB_CFG((gemv_chain_kernel<16, false, 64>), chain_smem<16>());
  LMB_CFG((gemv_chain_kernel<32, false, 64>), chain_smem<32>());
  LMB_CFG((gemv_chain_kernel<16, false, 96>), chain_smem<16>());
  LMB_CFG((gemv_chain_kernel<32, false, 96>), chain_smem<32>());
  LMB_CFG((gemv_chain_kernel<16, false, 128>), chain_smem<16>());
  LMB_CFG((gemv_chain_kernel<32, false, 128>), chain_smem<32>());
#undef LMB_CFG
  return LMB200_OK;
}

int32_t gemv_launch(Ctx* ctx, int dtype, GemvParams p, cudaStream_t stream) {
  LMB_REQUIRE(p.B >= 1 && p.B <= 32, "gemv: batch %d outside 1..32", p.B);
  if (dtype == LMB200_BF16) {
    LMB_REQUIRE(p.grid >= 1 && p.partials && p.counters, "gemv: the bf16 kernels need a plan and scratch");
    return Layout<__nv_bfloat16>::batch_pad(p.B) == 16 ? launch_bf16<16>(ctx, p, stream) : launch_bf16<32>(ctx, p, stream);
  }
  LMB_REQUIRE(dtype == LMB200_F32, "gemv: dtype %d", dtype);
  LMB_REQUIRE(p.ksplit >= 1 && p.kc_per_split >= 1 && (int64_t)p.ksplit * p.kc_per_split >= p.KC,
              "gemv: bad k split");
  LMB_REQUIRE(p.ksplit == 1 || (p.partials && p.counters), "gemv: split-K needs scratch");
  switch (Layout<float>::batch_pad(p.B) / 8) {
    case 1: return launch_ring<float, 1, kMtF32, 3>(ctx, p, stream);
    case 2: return launch_ring<float, 2, kMtF32, 3>(ctx, p, stream);
    default: return launch_ring<float, 4, kMtF32, 2>(ctx, p, stream);
  }
}

}  // namespace lmb

#ifdef LMB_GEMV_TRACE
extern "C" int32_t lmb200_debug_gemv_trace(long long* out) {
  return lmb::gemv_trace_copy(out);
}
#endif
