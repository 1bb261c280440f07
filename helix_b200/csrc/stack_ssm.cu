// State-space and matrix-memory layers of layer-list decoders (HB_MIXER_MAMBA2, HB_MIXER_MLSTM), the short causal
// convolutions in front of them (and in front of grouped-query attention with HB_ATTN_QKV_CONV), and the residual step of
// stacks whose two sublayers read the same stream (HB_NORM_PARALLEL).
//
// Both recurrences have one scalar decay per head and token,
//   S_t = a_t S_(t-1) + b_t k_t v_t^T,   o_t = S_t^T q_t            (S [dim][vdim] fp32 per head and sequence)
// and run on the kernels behind lin_recurrence:
//   state-space layer:  a = exp(-exp(A) dt), b = dt, k = B, q = C, v = x, o += D x       (ssm_steps makes a, b)
//   matrix memory:      a = exp(f + m' - m), b = exp(i - m) with the running maximum m = max(f + m', i) of the log gates
//                       (exp_gate_scan: a warp scan over the tokens of an entry, since m -> max(m + f, i) composes
//                       associatively); the normaliser n_t = a n + b k is carried as one more state vector.
// Step entries are runs of tokens [first, first + n) of sequences whose state lives in their slot; an entry that starts at
// position 0 starts from zeros inside the kernels (m from 0), so a slot needs no clearing when it changes hands.
// Everything here is fp32; every sum has a fixed order per output element.
#include <limits.h>
#include <math.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"
#include "stack_common.cuh"

namespace hb {
namespace {

__device__ __forceinline__ float softplus_(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

template <typename WT>
__device__ __forceinline__ void ssm_step(float raw, const WT* __restrict__ a_dt, float* __restrict__ ab, long ldab, int t, int H, int h) {
  const float dt = softplus_(raw + ldf<WT>(a_dt, H + h));
  ab[(size_t)t * ldab + h] = expf(-expf(ldf<WT>(a_dt, h)) * dt);
  ab[(size_t)t * ldab + H + h] = dt;
}

__device__ __forceinline__ void st_pair(float* f, bf16* b, float4 v) {
  if (f) *reinterpret_cast<float4*>(f) = v;
  if (b) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 pk;
    pk.x = *reinterpret_cast<unsigned*>(&lo);
    pk.y = *reinterpret_cast<unsigned*>(&hi);
    *reinterpret_cast<uint2*>(b) = pk;
  }
}

// ------------------------------------------------------------------ short convolutions
template <typename WT>
__global__ void __launch_bounds__(256) short_conv_kernel(ConvArgs a) {
  const int t = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.C) return;
  const int b = a.seq_of[t], t0 = a.cu[b], taps = a.taps;
  const bool fresh = a.first_pos[b] == 0;
  const float* tail = a.state + (size_t)a.slots[b] * a.slot_stride + a.tail_off;  // inputs of positions first - (taps - 1) ..
  const float ib = a.in_bias ? ldf<WT>((const WT*)a.in_bias, a.bias_off + c) : 0.f;
  const WT* w = (const WT*)a.w + (size_t)c * taps;
  float acc = 0.f;
  for (int j = 0; j < taps; ++j) {  // tap j multiplies the input of token t - (taps - 1 - j), oldest first
    const int tau = t - (taps - 1 - j);
    float x;
    if (tau >= t0) x = a.in[(size_t)tau * a.ldi + a.off + c] + ib;
    else x = fresh ? 0.f : tail[(size_t)(tau - t0 + taps - 1) * a.C + c];
    acc = fmaf(ldf<WT>(w, j), x, acc);
  }
  if (a.bias) acc += ldf<WT>((const WT*)a.bias, c);
  if (a.act == 1) acc = acc * sigmoidf_(acc);
  a.out[(size_t)t * a.ldo + c] = acc;
}

// The same for rows whose pieces start on 16-byte boundaries and up to four taps: thread = four neighbouring channels x kConvRun
// consecutive tokens, the last TAPS - 1 inputs in registers, so a row is read once per run instead of once per tap.  A run may
// cross entries: the window is refilled (from the slot or with zeros) wherever an entry starts.
// Steps of a few tokens take runs of one token: a run of eight then was eight dependent chains (entry, slot, tail) in a row, 14 us for 16
// tokens of 16 entries against 5 now; where every entry is a single token the same thread also moves the slot's inputs on.
constexpr int kConvRun = 8;
__device__ __forceinline__ float4 f4add(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
template <typename WT, int TAPS, int RUN>
__global__ void __launch_bounds__(128) short_conv_run_kernel(ConvArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int tb = blockIdx.y * RUN;
  if (a.ab && blockIdx.x == gridDim.x - 1) {  // the last column of blocks makes the run's step sizes
    for (int e = threadIdx.x; e < RUN * a.H; e += blockDim.x)
      if (const int t = tb + e / a.H, col = a.off_dt + e % a.H; t < a.T)
        ssm_step<WT>(RUN == 1 && a.slabs.ws ? slab_sum1(a.slabs, t, col) : a.in[(size_t)t * a.ldi + col], (const WT*)a.a_dt, a.ab, a.ldab, t, a.H, e % a.H);
    return;
  }
  if constexpr (RUN == 1) {
    const int across = (a.C / 4 + 127) / 128;
    if (a.up_out && blockIdx.x >= across) {  // the feed-forward's inner row, which waits for the same launch
      const int e = ((blockIdx.x - across) * 128 + threadIdx.x) * 4;
      if (e >= a.up.N) return;
      const float4 u = slab_sum4(a.up, tb, e);
      const float4 r = make_float4(fmaxf(u.x, 0.f), fmaxf(u.y, 0.f), fmaxf(u.z, 0.f), fmaxf(u.w, 0.f));
      st_pair(nullptr, a.up_out + (size_t)tb * a.up.N + e, make_float4(r.x * r.x, r.y * r.y, r.z * r.z, r.w * r.w));
      return;
    }
  }
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (c >= a.C) return;
  float w[4][TAPS];
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int j = 0; j < TAPS; ++j) w[e][j] = ldf<WT>((const WT*)a.w, (size_t)(c + e) * TAPS + j);
  float4 ib = make_float4(0.f, 0.f, 0.f, 0.f), cb = ib;
  if (a.in_bias) {
    const WT* p = (const WT*)a.in_bias + a.bias_off + c;
    ib = make_float4(ldf<WT>(p, 0), ldf<WT>(p, 1), ldf<WT>(p, 2), ldf<WT>(p, 3));
  }
  if (a.bias) {
    const WT* p = (const WT*)a.bias + c;
    cb = make_float4(ldf<WT>(p, 0), ldf<WT>(p, 1), ldf<WT>(p, 2), ldf<WT>(p, 3));
  }
  if constexpr (RUN > 1) {
    // A run inside one entry, with what it looks back at: all of its rows are read at once (row by row, with the entry's tests in between, left
    // one or two loads in flight: 11k tokens x 6144 channels 175 -> 120 us)
    const int b = a.seq_of[tb];
    if (tb + RUN <= a.cu[b + 1] && tb - (TAPS - 1) >= a.cu[b]) {
      const float* in = a.in + (size_t)(tb - (TAPS - 1)) * a.ldi + a.off + c;
      float4 x[RUN + TAPS - 1];
#pragma unroll
      for (int i = 0; i < RUN + TAPS - 1; ++i) x[i] = *reinterpret_cast<const float4*>(in + (size_t)i * a.ldi);
#pragma unroll
      for (int i = 0; i < RUN + TAPS - 1; ++i) x[i] = f4add(x[i], ib);
#pragma unroll
      for (int tt = 0; tt < RUN; ++tt) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
          acc[0] = fmaf(w[0][j], x[tt + j].x, acc[0]); acc[1] = fmaf(w[1][j], x[tt + j].y, acc[1]);
          acc[2] = fmaf(w[2][j], x[tt + j].z, acc[2]); acc[3] = fmaf(w[3][j], x[tt + j].w, acc[3]);
        }
        if (a.bias) { acc[0] += cb.x; acc[1] += cb.y; acc[2] += cb.z; acc[3] += cb.w; }
        if (a.act == 1) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[e] = acc[e] * sigmoidf_(acc[e]);
        }
        *reinterpret_cast<float4*>(a.out + (size_t)(tb + tt) * a.ldo + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      }
      return;
    }
  }
  float4 win[TAPS > 1 ? TAPS - 1 : 1];
  int t0 = 0, t1 = -1;
  bool fresh = false;
  float* tail = nullptr;
#pragma unroll
  for (int tt = 0; tt < RUN; ++tt) {
    const int t = tb + tt;
    if (t >= a.T) break;
    bool refill = tt == 0;
    if (t >= t1) {
      const int b = a.seq_of[t];
      t0 = a.cu[b]; t1 = a.cu[b + 1];
      fresh = a.first_pos[b] == 0;
      tail = a.state + (size_t)a.slots[b] * a.slot_stride + a.tail_off;
      refill = true;
    }
    if (refill) {
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) {
        const int tau = t - (TAPS - 1 - j);
        if (tau >= t0) win[j] = f4add(*reinterpret_cast<const float4*>(a.in + (size_t)tau * a.ldi + a.off + c), ib);
        else if (!fresh) win[j] = *reinterpret_cast<const float4*>(tail + (size_t)(tau - t0 + TAPS - 1) * a.C + c);
        else win[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    const float4 x = f4add(RUN == 1 && a.slabs.ws ? slab_sum4(a.slabs, t, a.off + c) : *reinterpret_cast<const float4*>(a.in + (size_t)t * a.ldi + a.off + c), ib);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < TAPS - 1; ++j) {  // oldest tap first, as the per-channel kernel
      acc[0] = fmaf(w[0][j], win[j].x, acc[0]); acc[1] = fmaf(w[1][j], win[j].y, acc[1]);
      acc[2] = fmaf(w[2][j], win[j].z, acc[2]); acc[3] = fmaf(w[3][j], win[j].w, acc[3]);
    }
    acc[0] = fmaf(w[0][TAPS - 1], x.x, acc[0]); acc[1] = fmaf(w[1][TAPS - 1], x.y, acc[1]);
    acc[2] = fmaf(w[2][TAPS - 1], x.z, acc[2]); acc[3] = fmaf(w[3][TAPS - 1], x.w, acc[3]);
    if (a.bias) { acc[0] += cb.x; acc[1] += cb.y; acc[2] += cb.z; acc[3] += cb.w; }
    if (a.act == 1) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = acc[e] * sigmoidf_(acc[e]);
    }
    *reinterpret_cast<float4*>(a.out + (size_t)t * a.ldo + c) = make_float4(acc[0], acc[1], acc[2], acc[3]);
#pragma unroll
    for (int j = 0; j + 1 < TAPS - 1; ++j) win[j] = win[j + 1];
    if (TAPS > 1) win[TAPS - 2] = x;
    if (a.single) {  // the entry's only token: the window is what conv_tails would store
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) *reinterpret_cast<float4*>(tail + (size_t)j * a.C + c) = win[j];
    }
  }
}

// Thread = one channel of one entry: the slot's last taps - 1 inputs become those behind the entry's last token.
constexpr int kMaxConvTail = 15;
template <typename WT>
__global__ void __launch_bounds__(256) conv_tails_kernel(ConvArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.y, nt = a.taps - 1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.C || nt <= 0) return;
  const int t0 = a.cu[b], n = a.cu[b + 1] - t0;
  const bool fresh = a.first_pos[b] == 0;
  const float ib = a.in_bias ? ldf<WT>((const WT*)a.in_bias, a.bias_off + c) : 0.f;
  float* tail = a.state + (size_t)a.slots[b] * a.slot_stride + a.tail_off;
  float v[kMaxConvTail];
#pragma unroll
  for (int i = 0; i < kMaxConvTail; ++i) {
    if (i >= nt) break;
    const int e = n + i;  // index into [old tail (nt rows) ; the entry's rows (n)]
    v[i] = e < nt ? (fresh ? 0.f : tail[(size_t)e * a.C + c]) : a.in[(size_t)(t0 + e - nt) * a.ldi + a.off + c] + ib;
  }
#pragma unroll
  for (int i = 0; i < kMaxConvTail; ++i) {
    if (i >= nt) break;
    tail[(size_t)i * a.C + c] = v[i];
  }
}

// ------------------------------------------------------------------ decays and gates
template <typename WT>
__global__ void ssm_steps_kernel(const float* __restrict__ p, long ldp, int off_dt, const WT* __restrict__ a_dt, float* __restrict__ ab,
                                 long ldab, int T, int H) {
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long)T * H) return;
  ssm_step<WT>(p[(size_t)(idx / H) * ldp + off_dt + idx % H], a_dt, ab, ldab, (int)(idx / H), H, (int)(idx % H));
}

// One warp per (entry, head).  The step m -> max(m + f, i) is the pair (f, i); two steps compose to
// (f1 + f2, max(i1 + f2, i2)), so the running maxima of 32 tokens come from one inclusive warp scan.
template <typename WT>
__global__ void __launch_bounds__(32) exp_gate_scan_kernel(GateScanArgs a) {
  const int b = blockIdx.x, h = blockIdx.y, lane = threadIdx.x;
  const int t0 = a.cu[b], t1 = a.cu[b + 1];
  float* ms = a.state + (size_t)a.slots[b] * a.slot_stride + a.m_off + h;
  float m = a.first_pos[b] == 0 ? 0.f : *ms;
  const float bi = a.bias ? ldf<WT>((const WT*)a.bias, a.off_i + h) : 0.f, bf = a.bias ? ldf<WT>((const WT*)a.bias, a.off_f + h) : 0.f;
  const float cap = a.cap, icap = 1.f / cap;
  for (int tc = t0; tc < t1; tc += 32) {
    const int t = tc + lane;
    const bool live = t < t1;
    float gi = -INFINITY, gf = 0.f;
    if (live) {
      const float* pr = a.p + (size_t)t * a.ldp;
      gi = cap * tanhf((pr[a.off_i + h] + bi) * icap);
      const float z = cap * tanhf((pr[a.off_f + h] + bf) * icap);
      gf = fminf(z, 0.f) - log1pf(expf(-fabsf(z)));  // log sigmoid
    }
    float F = gf, I = gi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float Fp = __shfl_up_sync(0xffffffffu, F, o), Ip = __shfl_up_sync(0xffffffffu, I, o);
      if (lane >= o) {
        I = fmaxf(Ip + F, I);
        F = Fp + F;
      }
    }
    const float mt = fmaxf(m + F, I);
    float mp = __shfl_up_sync(0xffffffffu, mt, 1);
    if (lane == 0) mp = m;
    if (live) {
      float* o = a.ab + (size_t)t * a.ldab;
      o[h] = expf(gf + mp - mt);
      o[a.H + h] = expf(gi - mt);
      o[2 * a.H + h] = expf(-mt);
    }
    m = __shfl_sync(0xffffffffu, mt, min(31, t1 - tc - 1));
  }
  if (lane == 0 && t1 > t0) *ms = m;
}

// ------------------------------------------------------------------ the recurrence
__device__ __forceinline__ void cpa4(float* smem_dst, const float* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpa16(float* smem_dst, const float* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Block = (entry, head, 32 NC value columns), DKP / 16 warps: warp w keeps key channels [16 w, 16 w + 16) of the block's
// state columns in registers (lane = NC neighbouring columns; pairs of neighbouring channels as packed f32x2 operands, so one
// instruction serves two state elements, and one 16-byte broadcast read of q or k feeds 4 NC of them).  Tokens are staged
// 16 / NC at a time through a cp.async double buffer (q | k | the block's v columns | a, b); every warp leaves its partial dot
// products (sums of eight channels, added) in shared memory and the block adds them pair by pair once per stage.  The block of the first column slice also
// carries the normaliser vector: lane l of warp w keeps channel 16 w + (l & 15), the 16 lanes' products are added by a
// butterfly.
template <int DKP, int NC>
__global__ void __launch_bounds__(DKP * 2, 512 / DKP) lin_recurrence_kernel(LinRecArgs a) {
  // (64 registers per thread and four 256-thread blocks per SM: a step of 8 sequences x 64 heads x 64 columns is one wave)
  constexpr int kRecTch = 16 / NC;  // tokens per shared-memory stage
  constexpr int KS = DKP / 16, BC = 32 * NC;
  constexpr int per_tok = 2 * DKP + BC + 4, stage_floats = kRecTch * per_tok;
  extern __shared__ __align__(16) float sm[];  // 2 stages | partial outputs [kRecTch][KS][BC] | partial n . q [kRecTch][KS]
  pdl_launch_dependents();
  pdl_wait();
  float* obuf = sm + 2 * stage_floats;
  float* nbuf = obuf + kRecTch * KS * BC;
  const int b = blockIdx.x, h = blockIdx.y, kvh = h / (a.H / a.G);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c0 = blockIdx.z * BC, j0 = c0 + lane * NC;
  const int t0 = a.cu[b], t1 = a.cu[b + 1];
  const int Dk = a.Dk, i0 = w * 16;
  float* slot = a.state + (size_t)a.slots[b] * a.slot_stride;
  float* st = slot + a.s_off + (size_t)h * Dk * a.Dv;
  const bool fresh = a.first_pos[b] == 0;
  const bool hd = a.head_decay != nullptr;
  const float2 hab = make_float2(hd ? a.head_decay[h] : 0.f, 1.f);
  const bool do_n = a.nq != nullptr && blockIdx.z == 0;
  const int nch = i0 + (lane & 15);
  float* nst = slot + a.n_off + (size_t)h * Dk + nch;
  float2 S[NC][8];
#pragma unroll
  for (int e = 0; e < NC; ++e)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      auto ld = [&](int ch) { return (!fresh && j0 + e < a.Dv && ch < Dk) ? st[(size_t)ch * a.Dv + j0 + e] : 0.f; };
      S[e][i] = make_float2(ld(i0 + 2 * i), ld(i0 + 2 * i + 1));
    }
  float nreg = (do_n && !fresh && nch < Dk) ? *nst : 0.f;
  for (int e = threadIdx.x; e < 2 * stage_floats; e += blockDim.x) sm[e] = 0.f;  // padded key channels and columns read zeros
  __syncthreads();
  const bool vec = ((Dk | a.Dv | (int)a.ldq | (int)a.ldk | (int)a.ldv | a.q_off | a.k_off | a.v_off) & 3) == 0 && ((uintptr_t)a.q & 15) == 0 &&
                   ((uintptr_t)a.k & 15) == 0 && ((uintptr_t)a.v & 15) == 0;
  auto issue = [&](int tc, int stage) {  // warp w stages the tokens w, w + KS, ...
    const int nt = min(kRecTch, t1 - tc);
    float* base = sm + stage * stage_floats;
    for (int tt = w; tt < nt; tt += KS) {
      const size_t row = (size_t)(tc + tt);
      const float* sq = a.q + row * a.ldq + a.q_off + (size_t)kvh * Dk;
      const float* sk = a.k + row * a.ldk + a.k_off + (size_t)kvh * Dk;
      const float* sv = a.v + row * a.ldv + a.v_off + (size_t)h * a.Dv + c0;
      float* dst = base + tt * per_tok;
      if (vec) {
        for (int i = lane * 4; i < Dk; i += 128) {
          cpa16(dst + i, sq + i);
          cpa16(dst + DKP + i, sk + i);
        }
        if (lane < 8 * NC && c0 + lane * 4 < a.Dv) cpa16(dst + 2 * DKP + lane * 4, sv + lane * 4);
      } else {
        for (int i = lane; i < Dk; i += 32) {
          cpa4(dst + i, sq + i);
          cpa4(dst + DKP + i, sk + i);
        }
#pragma unroll
        for (int e = 0; e < NC; ++e)
          if (c0 + lane + 32 * e < a.Dv) cpa4(dst + 2 * DKP + lane + 32 * e, sv + lane + 32 * e);
      }
      if (hd) continue;
      if (lane == 8 * NC) cpa4(dst + 2 * DKP + BC, a.ab + row * a.ldab + h);
      if (lane == 8 * NC + 1) cpa4(dst + 2 * DKP + BC + 1, a.ab + row * a.ldab + a.H + h);
    }
    cpa_commit();
  };
  const float skip = a.skip ? (a.f32 ? ((const float*)a.skip)[h] : __bfloat162float(((const bf16*)a.skip)[h])) : 0.f;
  if (t0 < t1) issue(t0, 0);
  int stage = 0;
  for (int tc = t0; tc < t1; tc += kRecTch, stage ^= 1) {
    const int nt = min(kRecTch, t1 - tc);
    if (tc + kRecTch < t1) {
      issue(tc + kRecTch, stage ^ 1);  // the next tokens travel while these are consumed
      cpa_wait<1>();
    } else {
      cpa_wait<0>();
    }
    __syncthreads();
    const float* base = sm + stage * stage_floats;
    if (a.silu) {  // activations of the staged q | k | v, once per stage
      float* raw = sm + stage * stage_floats;
      for (int e = threadIdx.x; e < nt * (2 * DKP + BC); e += blockDim.x) {
        const int at = e / (2 * DKP + BC) * per_tok + e % (2 * DKP + BC);
        const float z = raw[at];
        raw[at] = z * sigmoidf_(z);
      }
      __syncthreads();
    }
    for (int tt = 0; tt < nt; ++tt) {
      const float* tk = base + tt * per_tok;
      const float2 dab = hd ? hab : *reinterpret_cast<const float2*>(tk + 2 * DKP + BC);
      const float da = dab.x, db = dab.y;
      const float2 da2 = make_float2(da, da);
      float2 bv2[NC], oa[NC], ob[NC];  // channels 0 .. 7 and 8 .. 15 of the warp's have a sum each
#pragma unroll
      for (int e = 0; e < NC; ++e) {
        const float bv = db * tk[2 * DKP + lane * NC + e];
        bv2[e] = make_float2(bv, bv);
      }
      const float4* q4 = reinterpret_cast<const float4*>(tk + i0);
      const float4* k4 = reinterpret_cast<const float4*>(tk + DKP + i0);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 q = q4[i], k = k4[i];
        const float2 k01 = make_float2(k.x, k.y), k23 = make_float2(k.z, k.w), q01 = make_float2(q.x, q.y), q23 = make_float2(q.z, q.w);
#pragma unroll
        for (int e = 0; e < NC; ++e) {
          float2& o = i < 2 ? oa[e] : ob[e];
          S[e][2 * i] = __ffma2_rn(da2, S[e][2 * i], __fmul2_rn(k01, bv2[e]));
          o = i % 2 == 0 ? __fmul2_rn(S[e][2 * i], q01) : __ffma2_rn(S[e][2 * i], q01, o);
          S[e][2 * i + 1] = __ffma2_rn(da2, S[e][2 * i + 1], __fmul2_rn(k23, bv2[e]));
          o = __ffma2_rn(S[e][2 * i + 1], q23, o);
        }
      }
#pragma unroll
      for (int e = 0; e < NC; ++e) obuf[(tt * KS + w) * BC + lane * NC + e] = (oa[e].x + oa[e].y) + (ob[e].x + ob[e].y);
      if (do_n) {
        nreg = fmaf(da, nreg, db * tk[DKP + nch]);
        float pn = nreg * tk[nch];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) pn += __shfl_xor_sync(0xffffffffu, pn, o);
        if (lane == 0) nbuf[tt * KS + w] = pn;
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nt * BC; e += blockDim.x) {
      const int tt = e / BC, c = e % BC;
      float part[KS];
#pragma unroll
      for (int ww = 0; ww < KS; ++ww) part[ww] = obuf[(tt * KS + ww) * BC + c];
#pragma unroll
      for (int st = 1; st < KS; st *= 2)
#pragma unroll
        for (int ww = 0; ww < KS; ww += 2 * st) part[ww] += part[ww + st];
      const float o = part[0];
      if (c0 + c < a.Dv) a.out[(size_t)(tc + tt) * a.ldo + (size_t)h * a.Dv + c0 + c] = fmaf(skip, base[tt * per_tok + 2 * DKP + c], o * a.q_scale);
    }
    if (do_n) {
      for (int tt = threadIdx.x; tt < nt; tt += blockDim.x) {
        float o = 0.f;
#pragma unroll
        for (int ww = 0; ww < KS; ++ww) o += nbuf[tt * KS + ww];
        a.nq[(size_t)(tc + tt) * a.ldn + h] = o * a.q_scale;
      }
    }
    __syncthreads();  // the stage and the partial outputs are rewritten in the next iteration
  }
  if (t1 <= t0) return;
#pragma unroll
  for (int e = 0; e < NC; ++e) {
    if (j0 + e >= a.Dv) continue;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i0 + 2 * i < Dk) st[(size_t)(i0 + 2 * i) * a.Dv + j0 + e] = S[e][i].x;
      if (i0 + 2 * i + 1 < Dk) st[(size_t)(i0 + 2 * i + 1) * a.Dv + j0 + e] = S[e][i].y;
    }
  }
  if (do_n && lane < 16 && nch < Dk) *nst = nreg;
}

// Portions without a normaliser: the same arithmetic (state elements, channel sums of eight, their sums pair by pair: the same bits as the
// kernel above and the single-token one) in larger pieces.  A lane keeps CH channels of NC neighbouring columns, LS = DKP / CH lanes
// share the columns.  What bounds it is the FMA pipe (active 68 % of the cycles with four columns, and what warps wait for first), and close behind shared
// memory: a read hands a lane 16 bytes, 512 a warp, at 128 bytes a cycle whoever shares the address, so q and k have to serve many columns each.  Per warp and
// token that is 84 cycles with two columns per lane, as above, 45 with four (16 channels of a 128-channel state), 36 with eight (8 channels: half the
// reads of q and k for twice the sums over lanes), where three blocks fit an SM instead of four.  Tokens go in pairs, so that the sums of a lane fold over the
// LS lanes with all of them useful and one token's products cover the other's shuffles; one barrier per 16 tokens, no partial sums in shared memory.
// Entries are taken longest first.
// Prompts of 700 to 2048 tokens, 8 sequences x 64 heads of 128 x 64 states: two columns 1670, four 1030, eight 1000 us (lin_portion_many);
// one sequence of 2048 723 -> 383 (four columns); 32 heads of 64 x 64, 8 sequences 237 -> 125.
// Sums of r[0 .. CNT) over LS lanes, neighbours first: while a lane has several it gives half of them away, so that lane s ends up with the sum `at`.
template <int CNT, int X, int LS, int M>
__device__ __forceinline__ void fold_lanes(float (&r)[M], int s, int& at) {
  if constexpr (X < LS) {
    if constexpr (CNT > 1) {
      constexpr int half = CNT / 2;
      const bool up = s & X;
      at += up ? half : 0;
#pragma unroll
      for (int e = 0; e < half; ++e) {
        const float give = up ? r[e] : r[e + half], mine = up ? r[e + half] : r[e];
        r[e] = mine + __shfl_xor_sync(0xffffffffu, give, X);
      }
      fold_lanes<half, 2 * X, LS>(r, s, at);
    } else {
      r[0] += __shfl_xor_sync(0xffffffffu, r[0], X);
      fold_lanes<1, 2 * X, LS>(r, s, at);
    }
  }
}
template <int DKP, int CH, int NC, int W, int MB>
__global__ void __launch_bounds__(32 * W, MB) lin_portion_kernel(LinRecArgs a) {
  constexpr int LS = DKP / CH, CW = 32 / LS * NC, BC = W * CW, kTok = 16, NB = CH / 8, NT = 32 * W;
  constexpr int PS = LS + (CH == 8 ? 4 : 2), QS = CH * PS;  // float4 between pieces, floats of a row
  constexpr int per_tok = 2 * QS + BC + 4, stage_floats = kTok * per_tok;
  extern __shared__ __align__(16) float sm[];  // 2 stages
  __shared__ int s_len[128], s_b;
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int per_entry = a.H * ((a.Dv + BC - 1) / BC), rest = blockIdx.x % per_entry, h = rest % a.H, c0 = rest / a.H * BC;
  int b = blockIdx.x / per_entry;
  if (a.B > 1 && a.B <= 128) {
    for (int e = threadIdx.x; e < a.B; e += NT) s_len[e] = a.cu[e + 1] - a.cu[e];
    __syncthreads();
    for (int e = threadIdx.x; e < a.B; e += NT) {
      const int n = s_len[e];
      int rank = 0;
      for (int i = 0; i < a.B; ++i) rank += s_len[i] > n || (s_len[i] == n && i < e);
      if (rank == b) s_b = e;
    }
    __syncthreads();
    b = s_b;
  }
  const int kvh = h / (a.H / a.G), t0 = a.cu[b], t1 = a.cu[b + 1];
  if (t1 <= t0) return;
  const int s = lane % LS, cl = w * CW + lane / LS * NC, j0 = c0 + cl, ch0 = s * CH;
  float* st = a.state + (size_t)a.slots[b] * a.slot_stride + a.s_off + (size_t)h * a.Dk * a.Dv + (size_t)ch0 * a.Dv + j0;
  const bool hd = a.head_decay != nullptr;
  const float2 hab = make_float2(hd ? a.head_decay[h] : 0.f, 1.f);
  if (a.Dk < DKP || a.Dv % BC != 0) {  // padded channels and columns read zeros
    for (int e = threadIdx.x; e < 2 * stage_floats; e += NT) sm[e] = 0.f;
    __syncthreads();
  }
  // Rows of q and k in shared memory: [4-channel piece of a lane's CH][lane of LS], so that a read of 16 bytes covers all banks.  Warp w
  // stages the tokens w, w + W, ...; a lane one piece of q and of k (DKP / 128 of them), and v or the decay
  const float* gq = a.q + (size_t)(t0 + w) * a.ldq + a.q_off + (size_t)kvh * a.Dk + lane * 4;
  const float* gk = a.k + (size_t)(t0 + w) * a.ldk + a.k_off + (size_t)kvh * a.Dk + lane * 4;
  const float* gv = a.v + (size_t)(t0 + w) * a.ldv + a.v_off + (size_t)h * a.Dv + c0 + lane * 4;
  const float* gd = a.ab + (size_t)(t0 + w) * a.ldab + (lane & 1) * a.H + h;
  const long dq = W * a.ldq, dk = W * a.ldk, dv = W * a.ldv, dd = W * a.ldab;
  const bool in_v = lane * 4 < BC && c0 + lane * 4 < a.Dv;
  auto issue = [&](int tc, int stage) {
    const int nt = min(kTok, t1 - tc);
    float* dst = sm + stage * stage_floats + w * per_tok;
#pragma unroll
    for (int r = 0; r < kTok / W; ++r) {
      if (w + r * W < nt) {
#pragma unroll
        for (int p = 0; p < (DKP + 127) / 128; ++p) {
          const int i = lane * 4 + p * 128, at = (i % CH / 4 * PS + i / CH) * 4;
          if (i < a.Dk) {
            cpa16(dst + at, gq + p * 128);
            cpa16(dst + QS + at, gk + p * 128);
          }
        }
        if (in_v) cpa16(dst + 2 * QS + lane * 4, gv);
        if (!hd && lane >= 30) cpa4(dst + 2 * QS + BC + lane - 30, gd);
      }
      gq += dq; gk += dk; gv += dv; gd += dd;
      dst += W * per_tok;
    }
    cpa_commit();
  };
  issue(t0, 0);
  float2 S[NC][CH / 2];
  const bool fresh = a.first_pos[b] == 0;
#pragma unroll
  for (int i = 0; i < CH / 2; ++i)
#pragma unroll
    for (int e = 0; e < NC; e += 4) {
      const bool in = !fresh && ch0 + 2 * i < a.Dk && j0 + e < a.Dv;  // (Dk and Dv are multiples of four)
      const float4 x = in ? *reinterpret_cast<const float4*>(st + (size_t)(2 * i) * a.Dv + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 y = in ? *reinterpret_cast<const float4*>(st + (size_t)(2 * i + 1) * a.Dv + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[e][i] = make_float2(x.x, y.x);
      S[e + 1][i] = make_float2(x.y, y.y);
      S[e + 2][i] = make_float2(x.z, y.z);
      S[e + 3][i] = make_float2(x.w, y.w);
    }
  const float skip = a.skip ? (a.f32 ? ((const float*)a.skip)[h] : __bfloat162float(((const bf16*)a.skip)[h])) : 0.f;
  float* out = a.out + (size_t)h * a.Dv + j0;
  // N neighbouring tokens of a stage
  auto tokens = [&](const float* tk, size_t row, auto count) {
    constexpr int N = decltype(count)::value;
    float r[N * NC];
#pragma unroll
    for (int u = 0; u < N; ++u) {
      const float2 dab = hd ? hab : *reinterpret_cast<const float2*>(tk + u * per_tok + 2 * QS + BC);
      const float2 da2 = make_float2(dab.x, dab.x);
      float2 bv2[NC];
#pragma unroll
      for (int e = 0; e < NC; e += 4) {
        const float4 v = *reinterpret_cast<const float4*>(tk + u * per_tok + 2 * QS + cl + e);
        const float bv[4] = {dab.y * v.x, dab.y * v.y, dab.y * v.z, dab.y * v.w};
#pragma unroll
        for (int f = 0; f < 4; ++f) bv2[e + f] = make_float2(bv[f], bv[f]);
      }
      const float4* q4 = reinterpret_cast<const float4*>(tk + u * per_tok) + s;
      const float4* k4 = reinterpret_cast<const float4*>(tk + u * per_tok + QS) + s;
#pragma unroll
      for (int n = 0; n < NB; ++n) {
        float2 oa[NC];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 q = q4[(2 * n + i) * PS], k = k4[(2 * n + i) * PS];
          const float2 k01 = make_float2(k.x, k.y), k23 = make_float2(k.z, k.w), q01 = make_float2(q.x, q.y), q23 = make_float2(q.z, q.w);
#pragma unroll
          for (int e = 0; e < NC; ++e) {
            float2& sa = S[e][n * 4 + 2 * i];
            float2& sb = S[e][n * 4 + 2 * i + 1];
            sa = __ffma2_rn(da2, sa, __fmul2_rn(k01, bv2[e]));
            oa[e] = i == 0 ? __fmul2_rn(sa, q01) : __ffma2_rn(sa, q01, oa[e]);
            sb = __ffma2_rn(da2, sb, __fmul2_rn(k23, bv2[e]));
            oa[e] = __ffma2_rn(sb, q23, oa[e]);
          }
        }
#pragma unroll
        for (int e = 0; e < NC; ++e) r[u * NC + e] = n == 0 ? oa[e].x + oa[e].y : r[u * NC + e] + (oa[e].x + oa[e].y);
      }
    }
    int at = 0;  // (token, column) of the sum that this lane keeps
    fold_lanes<N * NC, 1, LS>(r, s, at);
    static_assert(N * NC <= LS, "one sum per lane");
    const int u = at / NC, e = at % NC;
    if (s < N * NC && j0 + e < a.Dv) out[(row + u) * a.ldo + e] = fmaf(skip, tk[u * per_tok + 2 * QS + cl + e], r[0] * a.q_scale);
  };
  int stage = 0;
  for (int tc = t0; tc < t1; tc += kTok, stage ^= 1) {
    const int nt = min(kTok, t1 - tc);
    cpa_wait<0>();
    __syncthreads();  // the stage has landed, and everybody is done with the other one
    if (tc + kTok < t1) issue(tc + kTok, stage ^ 1);
    float* base = sm + stage * stage_floats;
    if (a.silu) {  // activations of the staged q | k | v, once per stage
      for (int e = threadIdx.x; e < nt * (2 * QS + BC); e += NT) {
        float& z = base[e / (2 * QS + BC) * per_tok + e % (2 * QS + BC)];
        z = z * sigmoidf_(z);
      }
      __syncthreads();
    }
    int tt = 0;
#pragma unroll 1
    for (; tt + 2 <= nt; tt += 2) tokens(base + tt * per_tok, (size_t)(tc + tt), std::integral_constant<int, 2>());
    if (tt < nt) tokens(base + tt * per_tok, (size_t)(tc + tt), std::integral_constant<int, 1>());
  }
#pragma unroll
  for (int i = 0; i < CH / 2; ++i)
#pragma unroll
    for (int e = 0; e < NC; e += 4) {
      if (ch0 + 2 * i >= a.Dk || j0 + e >= a.Dv) continue;
      *reinterpret_cast<float4*>(st + (size_t)(2 * i) * a.Dv + e) = make_float4(S[e][i].x, S[e + 1][i].x, S[e + 2][i].x, S[e + 3][i].x);
      *reinterpret_cast<float4*>(st + (size_t)(2 * i + 1) * a.Dv + e) = make_float4(S[e][i].y, S[e + 1][i].y, S[e + 2][i].y, S[e + 3][i].y);
    }
}
// Narrower blocks where the wide ones are no more than the SMs (us wide / narrow: one sequence of 2048 tokens x 64 heads of 128 x 64 states
// 492 / 383, four of 500 to 1000 316 / 361; 32 heads of 256 x 40 125 / 92)
bool lin_portion_narrow(const LinRecArgs& a) { return a.Dk <= 64 || (long)a.B * a.H * ((a.Dv + 63) / 64) <= effective_sms(148); }
// Eight columns per lane where there are more blocks than three per SM; fewer are bound by a token's chain, which the sums over twice the lanes lengthen (a step,
// us, four columns | eight: 3 prompts of 1000 to 2048 tokens x 64 heads 1201 | 1217, 8 of 700 to 1500 x 32 heads 1022 | 1045; 8 of 200 to 400 x 64 heads
// 697 | 679, of 700 to 2048 2578 | 2540, 32 of 50 to 100 x 32 heads with two tokens each 912 | 901)
bool lin_portion_many(const LinRecArgs& a) { return (long)a.B * a.H * ((a.Dv + 63) / 64) > 3 * effective_sms(148); }
// Short portions are bound by the state's bytes, which the smaller pieces above have more of in flight: from more than eight tokens on average on narrow blocks, 24 on
// wide ones (us there | here, 32 sequences x 32 heads of 128 x 64 states: of 5 to 10 tokens 31 | 33, of 9 27 | 30, of 12 31 | 33, of 40 70 | 67; 8 sequences of 20
// 19.4 | 20.2; 32 of 9 with 4 heads of 256 x 256 31 | 34; narrow, 8 of 9 with 4 heads of 256 x 256 15.6 | 12.5, 32 heads of 64 x 64 9.5 | 9.6)
bool lin_portion_ok(const LinRecArgs& a) {
  return !a.nq && a.T > (lin_portion_narrow(a) ? 8 : 24) * a.B && a.Dk > 32 && a.Dv > 32 && ((a.Dk | a.Dv | (int)a.ldq | (int)a.ldk | (int)a.ldv | a.q_off | a.k_off | a.v_off) & 3) == 0 &&
         ((a.slot_stride | (long)a.s_off) & 3) == 0 && (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.state) & 15) == 0;
}
template <int DKP, int CH, int NC, int W>
constexpr int portion_cols() { return W * (32 / (DKP / CH)) * NC; }
template <int DKP, int CH, int NC, int W>
constexpr int portion_smem() { return 2 * 16 * (2 * CH * (DKP / CH + (CH == 8 ? 4 : 2)) + portion_cols<DKP, CH, NC, W>() + 4) * 4; }
template <int DKP, int CH, int NC, int W, int MB>
cudaError_t launch_portion(cudaStream_t s, const LinRecArgs& a) {
  constexpr int BC = portion_cols<DKP, CH, NC, W>();
  const long blocks = (long)a.B * a.H * ((a.Dv + BC - 1) / BC);
  if (blocks > INT_MAX) return cudaErrorInvalidValue;
  // Not while the kernel before it drains, as others are: few long blocks, dealt out while that one still fills most SMs, sat three to five to an SM beside
  // empty ones (3 sequences x 32 heads, a step 640 -> 752 us)
  return launch_k(lin_portion_kernel<DKP, CH, NC, W, MB>, dim3((unsigned)blocks), dim3(32 * W), portion_smem<DKP, CH, NC, W>(), s, false, a);
}

// One token on 16 channels of two neighbouring columns (x, y of S): the states move on, o: their products with q; even and odd channels of eight
// have a sum each.  k and q: four channels at a time
template <typename K, typename Q>
__device__ __forceinline__ void step_channels(float2 (&S)[16], float da, float bx, float by, K&& k, Q&& q, float2& o) {
  float2 ox[2], oy[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 k4 = k(i), q4 = q(i);
    const float kk[4] = {k4.x, k4.y, k4.z, k4.w}, qq[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2& s = S[4 * i + e];
      s.x = __fmaf_rn(da, s.x, __fmul_rn(kk[e], bx));
      s.y = __fmaf_rn(da, s.y, __fmul_rn(kk[e], by));
      float& sx = e & 1 ? ox[i / 2].y : ox[i / 2].x;
      float& sy = e & 1 ? oy[i / 2].y : oy[i / 2].x;
      sx = i % 2 == 0 && e < 2 ? __fmul_rn(s.x, qq[e]) : __fmaf_rn(s.x, qq[e], sx);
      sy = i % 2 == 0 && e < 2 ? __fmul_rn(s.y, qq[e]) : __fmaf_rn(s.y, qq[e], sy);
    }
  }
  o = make_float2((ox[0].x + ox[0].y) + (ox[1].x + ox[1].y), (oy[0].x + oy[0].y) + (oy[1].x + oy[1].y));
}
// the warps' shares of a lane's two columns, pair by pair
template <int MAX>
__device__ __forceinline__ float2 step_total(const float (&obuf)[MAX][64], int lane, int warps) {
  float2 part[MAX];
#pragma unroll
  for (int ww = 0; ww < MAX; ++ww) part[ww] = ww < warps ? *reinterpret_cast<const float2*>(&obuf[ww][lane * 2]) : make_float2(0.f, 0.f);
#pragma unroll
  for (int st = 1; st < MAX; st *= 2) {
    if (st >= warps) break;
#pragma unroll
    for (int ww = 0; ww < MAX; ww += 2 * st) {
      part[ww].x += part[ww + st].x;
      part[ww].y += part[ww + st].y;
    }
  }
  return part[0];
}

// The same for entries of one token (decoding): bound by the state's bytes, 32 KB in and out per block of a 128 x 64 state.  Everything a
// block needs is loaded at once (the staging above spent a round trip on the state, one on the token and three barriers): 16
// sequences x 32 heads 12.2 -> 9.1 us.  Warp w has key channels 16 w .. 16 w + 15, a lane two neighbouring columns; the
// arithmetic and its order are those of the kernel above, so both give the same bits.
__global__ void lin_step_kernel(LinRecArgs a) {
  __shared__ __align__(8) float obuf[16][64];
  pdl_launch_dependents();
  if (!a.settled) pdl_wait();
  const int b = blockIdx.x, h = blockIdx.y, c0 = blockIdx.z * 64, kvh = h / (a.H / a.G);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i0 = w * 16, j0 = c0 + lane * 2;
  const int t = a.cu[b];
  const bool fresh = a.first_pos[b] == 0, cols = j0 < a.Dv;
  float* st = a.state + (size_t)a.slots[b] * a.slot_stride + a.s_off + (size_t)h * a.Dk * a.Dv + (size_t)i0 * a.Dv + j0;
  const float* q = a.q + (size_t)t * a.ldq + a.q_off + (size_t)kvh * a.Dk + i0;
  const float* k = a.k + (size_t)t * a.ldk + a.k_off + (size_t)kvh * a.Dk + i0;
  const float* v = a.v + (size_t)t * a.ldv + a.v_off + (size_t)h * a.Dv + j0;
  float2 S[16];
  float4 q4[4], k4[4];
#pragma unroll
  for (int i = 0; i < 16; ++i) S[i] = !fresh && cols && i0 + i < a.Dk ? *reinterpret_cast<const float2*>(st + (size_t)i * a.Dv) : make_float2(0.f, 0.f);
  if (a.settled) pdl_wait();  // (the step's descriptors, read above, were there before its first kernel began)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool in = i0 + 4 * i < a.Dk;  // (Dk is a multiple of four)
    q4[i] = in ? *reinterpret_cast<const float4*>(q + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    k4[i] = in ? *reinterpret_cast<const float4*>(k + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float2 vv = cols ? *reinterpret_cast<const float2*>(v) : make_float2(0.f, 0.f);
  const float da = a.head_decay ? a.head_decay[h] : a.ab[(size_t)t * a.ldab + h], db = a.head_decay ? 1.f : a.ab[(size_t)t * a.ldab + a.H + h];
  if (a.silu) {
    auto act = [](float& z) { z = z * sigmoidf_(z); };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      act(q4[i].x); act(q4[i].y); act(q4[i].z); act(q4[i].w);
      act(k4[i].x); act(k4[i].y); act(k4[i].z); act(k4[i].w);
    }
    act(vv.x);
    act(vv.y);
  }
  float2 o2;
  step_channels(S, da, db * vv.x, db * vv.y, [&](int i) { return k4[i]; }, [&](int i) { return q4[i]; }, o2);
#pragma unroll
  for (int i = 0; i < 16; ++i)
    if (cols && i0 + i < a.Dk) *reinterpret_cast<float2*>(st + (size_t)i * a.Dv) = S[i];
  *reinterpret_cast<float2*>(&obuf[w][lane * 2]) = o2;
  __syncthreads();
  const int warps = blockDim.x >> 5;
  if (w == 0 && cols) {
    const float skip = a.skip ? (a.f32 ? ((const float*)a.skip)[h] : __bfloat162float(((const bf16*)a.skip)[h])) : 0.f;
    const float2 o = step_total<16>(obuf, lane, warps);
    *reinterpret_cast<float2*>(a.out + (size_t)t * a.ldo + (size_t)h * a.Dv + j0) = make_float2(fmaf(skip, vv.x, o.x * a.q_scale), fmaf(skip, vv.y, o.y * a.q_scale));
  }
}
// Heads of up to 32 value columns leave half of a block's lanes idle: beside thousands of others they stay with the kernel above, whose blocks
// are 32 columns wide there (256 sequences x 32 heads of 128 x 24 states 76 us there, 80 here; 64 x 64 heads 37 / 35.5, 16 x 8 6.2 / 3.2).
bool lin_step_ok(const LinRecArgs& a) {
  return a.single && !a.nq && (a.Dv > 32 || (long)a.B * a.H <= 4096) && a.Dk % 4 == 0 && a.Dv % 2 == 0 && ((a.ldq | a.ldk | (long)a.q_off | (long)a.k_off) & 3) == 0 &&
         ((a.ldv | a.ldo | a.slot_stride | (long)a.v_off | (long)a.s_off) & 1) == 0 && (((uintptr_t)a.q | (uintptr_t)a.k) & 15) == 0 &&
         (((uintptr_t)a.v | (uintptr_t)a.out | (uintptr_t)a.state) & 7) == 0;
}

template <int DKP, int NC>
cudaError_t launch_rec(cudaStream_t s, const LinRecArgs& a) {
  constexpr int KS = DKP / 16, BC = 32 * NC, kRecTch = 16 / NC;
  const size_t smem = (size_t)(2 * kRecTch * (2 * DKP + BC + 4) + kRecTch * KS * BC + kRecTch * KS) * 4;
  dim3 grid(a.B, a.H, (a.Dv + BC - 1) / BC);
  return launch_k(lin_recurrence_kernel<DKP, NC>, grid, dim3(DKP * 2), smem, s, false, a);  // (as launch_portion)
}

// ------------------------------------------------------------------ read-outs
// one warp per (token, head)
template <typename WT>
__global__ void memory_readout_kernel(const float* __restrict__ num, long ldnum, const float* __restrict__ nq, long ldn,
                                      const float* __restrict__ ab, long ldab, const float* __restrict__ g, long ldg, const WT* __restrict__ w,
                                      float eps, float scale, float* __restrict__ out, bf16* __restrict__ outb, long ldout, int col0, int T,
                                      int H, int Dv) {
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= T * H) return;
  const int t = item / H, h = item % H, l = threadIdx.x & 31;
  const float den = fmaxf(fabsf(nq[(size_t)t * ldn + h]), ab[(size_t)t * ldab + 2 * H + h]) + 1e-6f;
  const float* src = num + (size_t)t * ldnum + (size_t)h * Dv;
  const float* gs = g + (size_t)t * ldg + (size_t)h * Dv;
  float ss = 0.f;
  for (int i = l; i < Dv; i += 32) {
    const float o = src[i] / den;
    ss = fmaf(o, o, ss);
  }
  ss = warp_sum(ss);
  const float rs = 1.f / sqrtf(ss / (float)Dv + eps);
  for (int i = l; i < Dv; i += 32) {
    const float v = src[i] / den * rs * ldf<WT>(w, (size_t)h * Dv + i) * sigmoidf_(gs[i]) * scale;
    const size_t d = (size_t)t * ldout + col0 + (size_t)h * Dv + i;
    if (out) out[d] = v;
    if (outb) outb[d] = __float2bfloat16(v);
  }
}

template <typename WT>
__device__ __forceinline__ float4 ldf4(const WT* p) {
  if constexpr (sizeof(WT) == 4) return *reinterpret_cast<const float4*>(p);
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float sum_of_squares(float4 v) { return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x))); }
// one block per (part, token)
template <typename WT>
__global__ void __launch_bounds__(256) gated_group_norm_kernel(const float* __restrict__ y, long ldy, const float* __restrict__ z, long ldz,
                                                               const WT* __restrict__ w, float eps, int parts, float* __restrict__ out,
                                                               bf16* __restrict__ outb, int n, int gate_last) {
  __shared__ float red[32];
  const int t = blockIdx.y, part = blockIdx.x, len = n / parts, c0 = part * len;
  const float* ys = y + (size_t)t * ldy + c0;
  const float* zs = z + (size_t)t * ldz + c0;
  constexpr int kKeep = 8;  // gated values a thread keeps between the two passes (parts of up to 2048 entries are read once)
  float keep[kKeep];
  float ss = 0.f;
#pragma unroll
  for (int r = 0; r < kKeep; ++r) {
    const int i = threadIdx.x + r * 256;
    keep[r] = 0.f;
    if (i < len) {
      const float zv = zs[i];
      keep[r] = gate_last ? ys[i] : ys[i] * (zv * sigmoidf_(zv));
    }
    ss = fmaf(keep[r], keep[r], ss);
  }
  for (int i = threadIdx.x + kKeep * 256; i < len; i += blockDim.x) {
    const float zv = zs[i], u = gate_last ? ys[i] : ys[i] * (zv * sigmoidf_(zv));
    ss = fmaf(u, u, ss);
  }
  ss = block_sum(ss, red);
  const float rs = 1.f / sqrtf(ss / (float)len + eps);
#pragma unroll
  for (int r = 0; r < kKeep; ++r) {
    const int i = threadIdx.x + r * 256;
    if (i >= len) break;
    const float v = keep[r] * rs * ldf<WT>(w, c0 + i) * (gate_last ? sigmoidf_(zs[i]) : 1.f);
    const size_t d = (size_t)t * n + c0 + i;
    if (out) out[d] = v;
    if (outb) outb[d] = __float2bfloat16(v);
  }
  for (int i = threadIdx.x + kKeep * 256; i < len; i += blockDim.x) {
    const float zv = zs[i], sg = sigmoidf_(zv), u = gate_last ? ys[i] : ys[i] * (zv * sg);
    const float v = u * rs * ldf<WT>(w, c0 + i) * (gate_last ? sg : 1.f);
    const size_t d = (size_t)t * n + c0 + i;
    if (out) out[d] = v;
    if (outb) outb[d] = __float2bfloat16(v);
  }
}

// (z from slabs is an instance of its own: the branch in the loop kept the rows' loads from being issued together, 114 -> 136 us)
// Many parts of up to 512 entries: a warp each, no barrier, and no idle half of a block (a block per part of 512 entries: 11k tokens x 8 parts 185 -> 83
// us).  The sum is the block's below, where warp c has 128 entries: a sum for each 128, added in the order of block_sum, so the two give the same bits.
template <typename WT, int CH, bool SLABS>
__global__ void __launch_bounds__(256) gated_group_norm_warp_kernel(const float* __restrict__ y, long ldy, const float* __restrict__ z, const bf16* __restrict__ zb, long ldz,
                                                                    const WT* __restrict__ w, float eps, int parts, float* __restrict__ out,
                                                                    bf16* __restrict__ outb, int n, int gate_last, int items, const Slabs zsl, int z_col) {
  pdl_launch_dependents();
  pdl_wait();
  const int item = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= items) return;
  const int t = item / parts, part = item % parts, len = n / parts, c0 = part * len;
  const float* ys = y + (size_t)t * ldy + c0;
  const float* zs = z ? z + (size_t)t * ldz + c0 : nullptr;
  const bf16* zbs = zb ? zb + (size_t)t * ldz + c0 : nullptr;
  static_assert(CH <= 4, "the order of four sums");
  float4 u[CH], g[CH];
  float ss[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (lane + c * 32) * 4;
    u[c] = g[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i >= len) continue;
    u[c] = *reinterpret_cast<const float4*>(ys + i);
    g[c] = SLABS ? slab_sum4(zsl, t, z_col + c0 + i) : zs ? *reinterpret_cast<const float4*>(zs + i) : ldf4<bf16>(zbs + i);
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const float4 s = make_float4(sigmoidf_(g[c].x), sigmoidf_(g[c].y), sigmoidf_(g[c].z), sigmoidf_(g[c].w));
    if (!gate_last) u[c] = make_float4(u[c].x * (g[c].x * s.x), u[c].y * (g[c].y * s.y), u[c].z * (g[c].z * s.z), u[c].w * (g[c].w * s.w));
    g[c] = gate_last ? s : make_float4(1.f, 1.f, 1.f, 1.f);
    ss[c] = warp_sum(sum_of_squares(u[c]));
  }
  const float rs = 1.f / sqrtf(((ss[0] + ss[2]) + (ss[1] + ss[3])) / (float)len + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (lane + c * 32) * 4;
    if (i >= len) continue;
    const size_t d = (size_t)t * n + c0 + i;
    const float4 wv = make_float4(ldf<WT>(w, c0 + i), ldf<WT>(w, c0 + i + 1), ldf<WT>(w, c0 + i + 2), ldf<WT>(w, c0 + i + 3));
    const float4 v = make_float4(u[c].x * rs * wv.x * g[c].x, u[c].y * rs * wv.y * g[c].y, u[c].z * rs * wv.z * g[c].z, u[c].w * rs * wv.w * g[c].w);
    st_pair(out ? out + d : nullptr, outb ? outb + d : nullptr, v);
  }
}

// The same with a part in registers as float4 (parts of a multiple of 4 entries, up to 4 * 256 * CH)
template <typename WT, int CH, bool SLABS>
__global__ void __launch_bounds__(256) gated_group_norm_vec_kernel(const float* __restrict__ y, long ldy, const float* __restrict__ z, const bf16* __restrict__ zb, long ldz,
                                                                   const WT* __restrict__ w, float eps, int parts, float* __restrict__ out,
                                                                   bf16* __restrict__ outb, int n, int gate_last, const Slabs zsl, int z_col) {
  __shared__ float red[32];
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x, part = blockIdx.y, len = n / parts, c0 = part * len;
  const float* ys = y + (size_t)t * ldy + c0;
  const float* zs = z ? z + (size_t)t * ldz + c0 : nullptr;
  const bf16* zbs = zb ? zb + (size_t)t * ldz + c0 : nullptr;
  float4 u[CH], g[CH];
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    u[c] = g[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i >= len) continue;
    u[c] = *reinterpret_cast<const float4*>(ys + i);
    g[c] = SLABS ? slab_sum4(zsl, t, z_col + c0 + i) : zs ? *reinterpret_cast<const float4*>(zs + i) : ldf4<bf16>(zbs + i);
  }
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const float4 s = make_float4(sigmoidf_(g[c].x), sigmoidf_(g[c].y), sigmoidf_(g[c].z), sigmoidf_(g[c].w));
    if (!gate_last) u[c] = make_float4(u[c].x * (g[c].x * s.x), u[c].y * (g[c].y * s.y), u[c].z * (g[c].z * s.z), u[c].w * (g[c].w * s.w));
    g[c] = gate_last ? s : make_float4(1.f, 1.f, 1.f, 1.f);
    ss += sum_of_squares(u[c]);
  }
  const float rs = 1.f / sqrtf(block_sum(ss, red) / (float)len + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    if (i >= len) continue;
    const size_t d = (size_t)t * n + c0 + i;
    float4 v;
    v.x = u[c].x * rs * ldf<WT>(w, c0 + i) * g[c].x; v.y = u[c].y * rs * ldf<WT>(w, c0 + i + 1) * g[c].y;
    v.z = u[c].z * rs * ldf<WT>(w, c0 + i + 2) * g[c].z; v.w = u[c].w * rs * ldf<WT>(w, c0 + i + 3) * g[c].w;
    if (out) *reinterpret_cast<float4*>(out + d) = v;
    if (outb) {
      __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
      uint2 pk;
      pk.x = *reinterpret_cast<unsigned*>(&lo);
      pk.y = *reinterpret_cast<unsigned*>(&hi);
      *reinterpret_cast<uint2*>(outb + d) = pk;
    }
  }
}

__global__ void gate_scale_kernel(const float* __restrict__ in, const bf16* __restrict__ inb, long ldi, const float* __restrict__ g, long ldg,
                                  float scale, float* __restrict__ out, bf16* __restrict__ outb, long ldout, int col0, int n) {
  const int t = blockIdx.y, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const float x = in ? in[(size_t)t * ldi + e] : __bfloat162float(inb[(size_t)t * ldi + e]);
  const float v = x * sigmoidf_(g[(size_t)t * ldg + e]) * scale;
  const size_t d = (size_t)t * ldout + col0 + e;
  if (out) out[d] = v;
  if (outb) outb[d] = __float2bfloat16(v);
}

// ------------------------------------------------------------------ a single-token step between the products
// Block = one head of one token, cluster = the HG heads that share a kv head (and a part of the gated norm).  A block convolves its head's
// value channels and its share of the group's k and q channels, which meet in every block's shared memory; then the recurrence as in
// lin_step_kernel, and the norm's sums of squares meet the same way, added in the order of gated_group_norm_vec_kernel.  The blocks behind the
// tokens' make the feed-forward's inner rows.  What bounds it: the state's bytes (read before the products' launch is over) and a chain of
// two round trips to L2, two cluster barriers and the recurrence; as three launches the same was 15 us of
// a layer's 33 (16 sequences x 32 heads), 8 now; a turn of 2 such layers and 12 tokens 2520 -> 2450.
constexpr int kTokDk = 128, kTokDv = 64, kTokTaps = 4;
template <int HG>
__global__ void __cluster_dims__(HG, 1, 1) __launch_bounds__(256, 4) ssm_token_kernel(const __grid_constant__ SsmTokenArgs a) {
  __shared__ __align__(16) float kq[2 * kTokDk], vs[kTokDv], zs[kTokDv], quads[HG][16];
  __shared__ __align__(16) float obuf[8][64];
  __shared__ float ab[2];
  pdl_launch_dependents();
  const LinRecArgs& r = a.r;
  const ConvArgs& c = a.c;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, heads = r.B * r.H;
  if ((int)blockIdx.x >= heads) {  // (whole clusters of them)
    const int per = (c.up.N / 4 + 255) / 256, at = blockIdx.x - heads, t = at / per, e = (at % per * 256 + tid) * 4;
    pdl_wait();
    if (t >= c.T || e >= c.up.N) return;
    const float4 u = slab_sum4(c.up, t, e);
    const float4 f = make_float4(fmaxf(u.x, 0.f), fmaxf(u.y, 0.f), fmaxf(u.z, 0.f), fmaxf(u.w, 0.f));
    st_pair(nullptr, c.up_out + (size_t)t * c.up.N + e, make_float4(f.x * f.x, f.y * f.y, f.z * f.z, f.w * f.w));
    return;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // (this block runs: the others may write to it)
  const uint32_t rank = cluster_ctarank();
  const int b = blockIdx.x / r.H, h = blockIdx.x % r.H, kvh = h / HG, inner = r.H * kTokDv;
  // what earlier steps and the loading of the model left, before the products are done
  const int t = r.cu[b];
  const bool fresh = r.first_pos[b] == 0;
  float* const slot = r.state + (size_t)r.slots[b] * r.slot_stride;
  const int i0 = w * 16, j0 = lane * 2;
  float* const st = slot + r.s_off + (size_t)h * kTokDk * kTokDv + (size_t)i0 * kTokDv + j0;
  float2 S[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) S[i] = fresh ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(st + (size_t)i * kTokDv);
  // conv threads: four channels each, first the head's values, then this block's share of k | q
  constexpr int kShare = 2 * kTokDk / HG, kConvThreads = (kTokDv + kShare) / 4;
  const int ch = tid * 4 < kTokDv ? h * kTokDv + tid * 4 : 0, shared_at = tid * 4 - kTokDv + (int)rank * kShare;  // place in k | q
  const bool conv = tid < kConvThreads, value = tid * 4 < kTokDv;
  const int cc = value ? ch : inner + (shared_at < kTokDk ? kvh * kTokDk + shared_at : r.G * kTokDk + kvh * kTokDk + shared_at - kTokDk);
  float4 win[kTokTaps - 1];
  uint4 cw[2];  // four taps of the four channels
  uint2 cb = make_uint2(0u, 0u);
  float* const tail = slot + c.tail_off + cc;
  if (conv) {
#pragma unroll
    for (int j = 0; j < kTokTaps - 1; ++j) win[j] = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(tail + (size_t)j * c.C);
    cw[0] = reinterpret_cast<const uint4*>((const bf16*)c.w + (size_t)cc * kTokTaps)[0];
    cw[1] = reinterpret_cast<const uint4*>((const bf16*)c.w + (size_t)cc * kTokTaps)[1];
    if (c.bias) cb = *reinterpret_cast<const uint2*>((const bf16*)c.bias + cc);
  }
  pdl_wait();
  if (tid >= 128 && tid < 144) {
    *reinterpret_cast<float4*>(&zs[(tid - 128) * 4]) = slab_sum4(c.slabs, t, a.z_col + h * kTokDv + (tid - 128) * 4);
  } else if (tid == 160) {
    const bf16* p = (const bf16*)c.a_dt;
    const float dt = softplus_(slab_sum1(c.slabs, t, c.off_dt + h) + ldf<bf16>(p, r.H + h));
    ab[0] = expf(-expf(ldf<bf16>(p, h)) * dt);
    ab[1] = dt;
  }
  float4 made = make_float4(0.f, 0.f, 0.f, 0.f);
  if (conv) {
    const float4 x = slab_sum4(c.slabs, t, c.off + cc);
    const uint32_t wp[8] = {cw[0].x, cw[0].y, cw[0].z, cw[0].w, cw[1].x, cw[1].y, cw[1].z, cw[1].w}, bp[2] = {cb.x, cb.y};
    auto half = [](uint32_t u, int hi) { return __uint_as_float(hi ? u & 0xffff0000u : u << 16); };
    float acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      auto of = [&](const float4& v) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; };
      acc[e] = 0.f;
#pragma unroll
      for (int j = 0; j < kTokTaps; ++j) acc[e] = fmaf(half(wp[2 * e + j / 2], j & 1), of(j < kTokTaps - 1 ? win[j] : x), acc[e]);
      if (c.bias) acc[e] += half(bp[e / 2], e & 1);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = acc[e] * sigmoidf_(acc[e]);
    made = make_float4(acc[0], acc[1], acc[2], acc[3]);
#pragma unroll
    for (int j = 0; j + 1 < kTokTaps - 1; ++j) *reinterpret_cast<float4*>(tail + (size_t)j * c.C) = win[j + 1];
    *reinterpret_cast<float4*>(tail + (size_t)(kTokTaps - 2) * c.C) = x;
    if (value) *reinterpret_cast<float4*>(&vs[tid * 4]) = made;
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (conv && !value) {
#pragma unroll
    for (int o = 0; o < HG; ++o) *cluster_ptr<HG>(reinterpret_cast<float4*>(&kq[shared_at]), o) = made;
  }
  __syncwarp();
  cluster_sync_all();
  const float da = ab[0], db = ab[1];
  const float2 vv = *reinterpret_cast<const float2*>(&vs[j0]);
  float2 o2;
  step_channels(S, da, db * vv.x, db * vv.y, [&](int i) { return *reinterpret_cast<const float4*>(&kq[i0 + 4 * i]); },
                [&](int i) { return *reinterpret_cast<const float4*>(&kq[kTokDk + i0 + 4 * i]); }, o2);
  *reinterpret_cast<float2*>(&obuf[w][j0]) = o2;
  __syncthreads();
  float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
  if (w == 0) {
    const float skip = r.skip ? __bfloat162float(((const bf16*)r.skip)[h]) : 0.f;
    const float2 o = step_total<8>(obuf, lane, 8);
    *reinterpret_cast<float2*>(&vs[j0]) = make_float2(fmaf(skip, vv.x, o.x * r.q_scale), fmaf(skip, vv.y, o.y * r.q_scale));  // (a lane's own columns)
    __syncwarp();
    if (lane < 16) {
      const float4 y = *reinterpret_cast<const float4*>(&vs[lane * 4]), z = *reinterpret_cast<const float4*>(&zs[lane * 4]);
      const float4 s = make_float4(sigmoidf_(z.x), sigmoidf_(z.y), sigmoidf_(z.z), sigmoidf_(z.w));
      u = make_float4(y.x * (z.x * s.x), y.y * (z.y * s.y), y.z * (z.z * s.z), y.w * (z.w * s.w));
      const float ss = sum_of_squares(u);
#pragma unroll
      for (int o2 = 0; o2 < HG; ++o2) *cluster_ptr<HG>(&quads[rank][lane], o2) = ss;
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) *reinterpret_cast<float2*>(st + (size_t)i * kTokDv) = S[i];
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (w == 0) {
    float part[HG / 2];  // a warp of the block kernel has 128 entries, two heads: one's below lane 16, the other's above
#pragma unroll
    for (int p = 0; p < HG / 2; ++p) {
      float s = quads[2 * p][lane & 15] + quads[2 * p + 1][lane & 15];
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      part[p] = s;
    }
#pragma unroll
    for (int o = HG / 4; o > 0; o >>= 1)
#pragma unroll
      for (int p = 0; p < o; ++p) part[p] += part[p + o];
    const float rs = 1.f / sqrtf(part[0] / (float)(HG * kTokDv) + a.eps);
    if (lane < 16) {
      const int col = h * kTokDv + lane * 4;
      const bf16* nw = (const bf16*)a.norm_w + col;
      st_pair(nullptr, a.out + (size_t)t * inner + col, make_float4(u.x * rs * ldf<bf16>(nw, 0), u.y * rs * ldf<bf16>(nw, 1), u.z * rs * ldf<bf16>(nw, 2), u.w * rs * ldf<bf16>(nw, 3)));
    }
  }
}

// ------------------------------------------------------------------ residual step of parallel sublayers
// one block per row; dynamic smem: the summed row [W]
template <typename WT>
__global__ void __launch_bounds__(256) parallel_step_kernel(const float* x, const int32_t* __restrict__ row_index,
                                                            const float* __restrict__ y, const float* __restrict__ y2,
                                                            const WT* __restrict__ bias, float bias_scale, const WT* __restrict__ w1,
                                                            const WT* __restrict__ w2, float eps, float* x_out,
                                                            float* __restrict__ h1, bf16* __restrict__ h1b, float* __restrict__ h2,
                                                            bf16* __restrict__ h2b, int W, const ParScale sc) {
  extern __shared__ __align__(16) float row[];
  __shared__ float red[32];
  const size_t r = blockIdx.x;
  const float* xs = x + (row_index ? (size_t)row_index[r] : r) * W;
  float ss = 0.f;
  for (int i = threadIdx.x; i < W; i += blockDim.x) {
    float v = xs[i];
    if (y) {
      float u = y[r * W + i], u2 = y2 ? y2[r * W + i] : 0.f;
      for (int k = 0; k < sc.top_k; ++k) u2 = fmaf(sc.wts[r * sc.top_k + k], __bfloat162float(sc.rows[(size_t)sc.row_of[r * sc.top_k + k] * W + i]), u2);
      if (sc.s1) u *= ldf<WT>((const WT*)sc.s1, i);
      if (sc.s2) u2 *= ldf<WT>((const WT*)sc.s2, i);
      v = fmaf(sc.m, u + u2, v);
    }
    if (bias) v = fmaf(bias_scale, ldf<WT>(bias, i), v);
    row[i] = v;
    if (x_out) x_out[r * W + i] = v;
    ss = fmaf(v, v, ss);
  }
  if (!w1 && !w2) return;
  ss = block_sum(ss, red);
  const float rs = 1.f / sqrtf(ss / (float)W + eps);
  for (int i = threadIdx.x; i < W; i += blockDim.x) {
    const float u = row[i] * rs;
    if (w1) {
      const float v = u * ldf<WT>(w1, i);
      if (h1) h1[r * W + i] = v;
      if (h1b) h1b[r * W + i] = __float2bfloat16(v);
    }
    if (w2) {
      const float v = u * ldf<WT>(w2, i);
      if (h2) h2[r * W + i] = v;
      if (h2b) h2b[r * W + i] = __float2bfloat16(v);
    }
  }
}

// The same step with the row in registers as float4 (W a multiple of 4, W <= 4 * 256 * kParChunks)
constexpr int kParChunks = 8;
constexpr int kParTop = 8;  // expert rows per token that the in-register form takes
__device__ __forceinline__ float4 fma4(float a, float4 b, float4 c) {
  return make_float4(fmaf(a, b.x, c.x), fmaf(a, b.y, c.y), fmaf(a, b.z, c.z), fmaf(a, b.w, c.w));
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
// What the sublayers' outputs are: rows (or nothing), the slabs of their products, rows of the first and expert rows of the second.  Instances of their own:
// with one for all three a row's loads waited for one another, and for the stores of the piece before (11k tokens x 2048 85 -> 61 us)
enum ParIn : int { PAR_ROWS, PAR_SLABS, PAR_EXPERTS };
template <typename WT, int CH, int IN>
__global__ void __launch_bounds__(256) parallel_step_vec_kernel(const float* x, const int32_t* __restrict__ row_index, const float* __restrict__ y,
                                                                const float* __restrict__ y2, const WT* __restrict__ bias, float bias_scale,
                                                                const WT* __restrict__ w1, const WT* __restrict__ w2, float eps, float* x_out,
                                                                float* __restrict__ h1, bf16* __restrict__ h1b, float* __restrict__ h2,
                                                                bf16* __restrict__ h2b, int W, const ParScale sc) {
  __shared__ float red[32];
  pdl_launch_dependents();
  pdl_wait();
  const size_t r = blockIdx.x;
  const float* xs = x + (row_index ? (size_t)row_index[r] : r) * W;
  constexpr int TOP = IN == PAR_EXPERTS ? kParTop : 0;
  float wk[TOP + 1];
  size_t rk[TOP + 1];
#pragma unroll
  for (int k = 0; k < TOP; ++k) {
    wk[k] = k < sc.top_k ? sc.wts[r * sc.top_k + k] : 0.f;
    rk[k] = k < sc.top_k ? (size_t)sc.row_of[r * sc.top_k + k] * W : 0;
  }
  const bool any = IN != PAR_ROWS || y, second = IN == PAR_ROWS && y2;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 v[CH], u[CH], u2[CH];
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    const bool in = i < W;
    v[c] = in ? *reinterpret_cast<const float4*>(xs + i) : zero;
    if (IN == PAR_SLABS) {
      u[c] = in ? slab_sum4(sc.y_slabs, r, i) : zero;
      u2[c] = in ? slab_sum4(sc.y2_slabs, r, i) : zero;
    } else {
      u[c] = in && any ? *reinterpret_cast<const float4*>(y + r * W + i) : zero;
      u2[c] = in && second ? *reinterpret_cast<const float4*>(y2 + r * W + i) : zero;
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    if (i >= W) continue;
    float4 a = v[c];
    if (any) {
#pragma unroll
      for (int k = 0; k < TOP; ++k)
        if (k < sc.top_k) u2[c] = fma4(wk[k], ldf4<bf16>(sc.rows + rk[k] + i), u2[c]);
      if (sc.s1) u[c] = mul4(u[c], ldf4<WT>((const WT*)sc.s1 + i));
      if (sc.s2) u2[c] = mul4(u2[c], ldf4<WT>((const WT*)sc.s2 + i));
      a = fma4(sc.m, make_float4(u[c].x + u2[c].x, u[c].y + u2[c].y, u[c].z + u2[c].z, u[c].w + u2[c].w), a);
    }
    if (bias) a = fma4(bias_scale, ldf4<WT>(bias + i), a);
    if (x_out) *reinterpret_cast<float4*>(x_out + r * W + i) = a;
    v[c] = a;
    ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
  }
  if (!w1 && !w2) return;
  ss = block_sum(ss, red);
  const float rs = 1.f / sqrtf(ss / (float)W + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    if (i >= W) continue;
    const float4 u = make_float4(v[c].x * rs, v[c].y * rs, v[c].z * rs, v[c].w * rs);
    if (w1) st_pair(h1 ? h1 + r * W + i : nullptr, h1b ? h1b + r * W + i : nullptr, mul4(u, ldf4<WT>(w1 + i)));
    if (w2) st_pair(h2 ? h2 + r * W + i : nullptr, h2b ? h2b + r * W + i : nullptr, mul4(u, ldf4<WT>(w2 + i)));
  }
}

// The embedding, its norm and the first layer's norms with the row in registers: three launches passed it through memory (11k tokens x 2048 in
// 154 us, 47 now), a step of few tokens waited for each of them.  The sums of squares are written out in the order that those three's have,
// so that a row has their bits: sum_of_squares, but for the embedding's norm of fp32 tables, where x^2 is added to y^2's product; the scaled row is
// rounded before a pair's row joins it
template <typename WT, int CH>
__global__ void __launch_bounds__(256) embed_step_kernel(const int32_t* __restrict__ tokens, const WT* __restrict__ table, float scale, BigramArgs bg,
                                                         const WT* __restrict__ w0, float off, const WT* __restrict__ w1, const WT* __restrict__ w2, float eps,
                                                         float* __restrict__ x, float* __restrict__ h1, bf16* __restrict__ h1b, float* __restrict__ h2,
                                                         bf16* __restrict__ h2b, int W) {
  __shared__ float red[32];
  pdl_launch_dependents();
  pdl_wait();
  const size_t r = blockIdx.x;
  const WT* src = table + (size_t)tokens[r] * W;
  const WT* pair = nullptr;
  if (bg.table) {
    const int prev = bg.prev[r];
    const long long row = prev < 0 ? bg.buckets : ((long long)prev * bg.mul_prev + (long long)tokens[r] * bg.mul_cur) % bg.buckets;
    pair = (const WT*)bg.table + (size_t)row * W;
  }
  float4 v[CH];
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    if (i >= W) continue;
    float4 a = ldf4<WT>(src + i);
    a = make_float4(a.x * scale, a.y * scale, a.z * scale, a.w * scale);
    if (pair) {
      const float4 p = ldf4<WT>(pair + i);
      a = make_float4(__fadd_rn(a.x, p.x), __fadd_rn(a.y, p.y), __fadd_rn(a.z, p.z), __fadd_rn(a.w, p.w));
    }
    v[c] = a;
    ss += sizeof(WT) == 4 ? sum_of_squares(make_float4(a.y, a.x, a.z, a.w)) : sum_of_squares(a);
  }
  const float rs0 = 1.f / sqrtf(block_sum(ss, red) / (float)W + eps);
  ss = 0.f;
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    if (i >= W) continue;
    const float4 g = ldf4<WT>(w0 + i);
    const float4 a = make_float4(v[c].x * (rs0 * (off + g.x)), v[c].y * (rs0 * (off + g.y)), v[c].z * (rs0 * (off + g.z)), v[c].w * (rs0 * (off + g.w)));
    *reinterpret_cast<float4*>(x + r * W + i) = a;
    v[c] = a;
    ss += sum_of_squares(a);
  }
  const float rs = 1.f / sqrtf(block_sum(ss, red) / (float)W + eps);
#pragma unroll
  for (int c = 0; c < CH; ++c) {
    const int i = (threadIdx.x + c * 256) * 4;
    if (i >= W) continue;
    const float4 u = make_float4(v[c].x * rs, v[c].y * rs, v[c].z * rs, v[c].w * rs);
    if (w1) st_pair(h1 ? h1 + r * W + i : nullptr, h1b ? h1b + r * W + i : nullptr, mul4(u, ldf4<WT>(w1 + i)));
    if (w2) st_pair(h2 ? h2 + r * W + i : nullptr, h2b ? h2b + r * W + i : nullptr, mul4(u, ldf4<WT>(w2 + i)));
  }
}

__global__ void relu2_kernel(const float* __restrict__ in, long ldi, float* __restrict__ out, bf16* __restrict__ outb, int n) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.y, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const float r = fmaxf(in[(size_t)t * ldi + e], 0.f), v = r * r;
  if (out) out[(size_t)t * n + e] = v;
  if (outb) outb[(size_t)t * n + e] = __float2bfloat16(v);
}
__global__ void relu2_b16_kernel(const bf16* __restrict__ in, long ldi, bf16* __restrict__ out, int n) {
  const int t = blockIdx.y, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const float r = fmaxf(__bfloat162float(in[(size_t)t * ldi + e]), 0.f);
  out[(size_t)t * n + e] = __float2bfloat16(r * r);
}

}  // namespace

cudaError_t stack_ssm_init() {
  cudaError_t e;
#define HB_SMEM(k, n) if ((e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, n)) != cudaSuccess) return e
  HB_SMEM((lin_recurrence_kernel<16, 1>), 64 * 1024);
  HB_SMEM((lin_recurrence_kernel<32, 1>), 64 * 1024);
  HB_SMEM((lin_recurrence_kernel<64, 1>), 64 * 1024);
  HB_SMEM((lin_recurrence_kernel<128, 1>), 96 * 1024);
  HB_SMEM((lin_recurrence_kernel<256, 1>), 160 * 1024);
  HB_SMEM((lin_recurrence_kernel<16, 2>), 64 * 1024);
  HB_SMEM((lin_recurrence_kernel<32, 2>), 64 * 1024);
  HB_SMEM((lin_recurrence_kernel<64, 2>), 96 * 1024);
  HB_SMEM((lin_recurrence_kernel<128, 2>), 128 * 1024);
  HB_SMEM((lin_recurrence_kernel<256, 2>), 200 * 1024);
  HB_SMEM((lin_portion_kernel<64, 8, 4, 4, 5>), (portion_smem<64, 8, 4, 4>()));
  HB_SMEM((lin_portion_kernel<128, 8, 4, 4, 5>), (portion_smem<128, 8, 4, 4>()));
  HB_SMEM((lin_portion_kernel<128, 16, 4, 4, 4>), (portion_smem<128, 16, 4, 4>()));
  HB_SMEM((lin_portion_kernel<128, 8, 8, 4, 3>), (portion_smem<128, 8, 8, 4>()));
  HB_SMEM((lin_portion_kernel<256, 16, 4, 4, 4>), (portion_smem<256, 16, 4, 4>()));
  HB_SMEM((lin_portion_kernel<256, 16, 4, 8, 2>), (portion_smem<256, 16, 4, 8>()));
  HB_SMEM(parallel_step_kernel<float>, 200 * 1024);
  HB_SMEM(parallel_step_kernel<bf16>, 200 * 1024);
#undef HB_SMEM
  return cudaSuccess;
}

// A row pass launched while a product drains finds the SMs set up for the product's shared memory and keeps that little first-level cache to the end, which
// costs one of more than a few million entries more than its launch (11k tokens: convolution of 6144 channels 142 us, 123 behind the product; residual step of
// 2048 columns 62, 49; a step of 8 prompts of 700 to 1500 tokens 1014, 1004; of 16 short ones early is 1.4 % sooner)
static bool launch_early(long entries, long limit_m) { return entries < limit_m << 20; }
bool short_conv_fused(const ConvArgs& a) {
  return a.taps <= 4 && a.T <= 65535 && ((a.C | (int)a.ldi | a.off | (int)a.ldo | (int)a.slot_stride | (int)a.tail_off) & 3) == 0 &&
         ((uintptr_t)a.in & 15) == 0 && ((uintptr_t)a.out & 15) == 0 && ((uintptr_t)a.state & 15) == 0;
}
cudaError_t short_conv(cudaStream_t s, const ConvArgs& a) {
  if (a.T <= 0 || a.C <= 0) return cudaSuccess;
  if (a.taps < 1 || a.taps - 1 > kMaxConvTail) return cudaErrorInvalidValue;
  if (short_conv_fused(a)) {
    const int across = (a.C / 4 + 127) / 128;
    // runs of one token until runs of eight give every SM two blocks (or where the tails ride along)
    const bool one = a.single || (long)across * ((a.T + kConvRun - 1) / kConvRun) < 2 * effective_sms(148);
    if (a.slabs.ws && (!a.single || !a.ab || !a.up_out || (a.up.N & 3) || (a.off_dt & 3))) return cudaErrorInvalidValue;
    const dim3 g(across + (a.up_out ? (a.up.N / 4 + 127) / 128 : 0) + (a.ab ? 1 : 0), one ? a.T : (a.T + kConvRun - 1) / kConvRun);
#define HB_CONV_T(WT, TP) return one ? launch_k(short_conv_run_kernel<WT, TP, 1>, g, dim3(128), 0, s, true, a) : launch_k(short_conv_run_kernel<WT, TP, kConvRun>, g, dim3(128), 0, s, launch_early((long)a.T * a.C, 20), a)
#define HB_CONV(TP) do { if (a.f32) HB_CONV_T(float, TP); else HB_CONV_T(bf16, TP); } while (0)
    if (a.taps == 1) HB_CONV(1);
    if (a.taps == 2) HB_CONV(2);
    if (a.taps == 3) HB_CONV(3);
    HB_CONV(4);
#undef HB_CONV
#undef HB_CONV_T
  }
  if (a.single || a.ab || a.slabs.ws) return cudaErrorInvalidValue;
  dim3 grid((a.C + 255) / 256, a.T);
  if (a.f32) short_conv_kernel<float><<<grid, 256, 0, s>>>(a);
  else short_conv_kernel<bf16><<<grid, 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t conv_tails(cudaStream_t s, const ConvArgs& a) {
  if (a.B <= 0 || a.taps <= 1 || a.C <= 0) return cudaSuccess;
  dim3 grid((a.C + 255) / 256, a.B);
  if (a.f32) return launch_k(conv_tails_kernel<float>, grid, dim3(256), 0, s, true, a);
  return launch_k(conv_tails_kernel<bf16>, grid, dim3(256), 0, s, true, a);
}

cudaError_t ssm_steps(cudaStream_t s, const float* p, long ldp, int off_dt, const void* a_dt, bool f32, float* ab, long ldab, int T, int H) {
  if (T <= 0 || H <= 0) return cudaSuccess;
  const unsigned blocks = (unsigned)(((long)T * H + 255) / 256);
  if (f32) ssm_steps_kernel<float><<<blocks, 256, 0, s>>>(p, ldp, off_dt, (const float*)a_dt, ab, ldab, T, H);
  else ssm_steps_kernel<bf16><<<blocks, 256, 0, s>>>(p, ldp, off_dt, (const bf16*)a_dt, ab, ldab, T, H);
  return cudaGetLastError();
}

cudaError_t exp_gate_scan(cudaStream_t s, const GateScanArgs& a) {
  if (a.B <= 0 || a.H <= 0) return cudaSuccess;
  if (!(a.cap > 0.f)) return cudaErrorInvalidValue;
  if (a.f32) exp_gate_scan_kernel<float><<<dim3(a.B, a.H), 32, 0, s>>>(a);
  else exp_gate_scan_kernel<bf16><<<dim3(a.B, a.H), 32, 0, s>>>(a);
  return cudaGetLastError();
}

bool ssm_token_ok(const SsmTokenArgs& a, int norm_groups) {
  const ConvArgs& c = a.c;
  const LinRecArgs& r = a.r;
  const int hg = r.G > 0 && r.H % r.G == 0 ? r.H / r.G : 0;
  return (hg == 2 || hg == 4 || hg == 8) && norm_groups == r.G && r.Dk == kTokDk && r.Dv == kTokDv && c.taps == kTokTaps && c.act == 1 && !c.f32 && !c.in_bias &&
         r.settled && r.single && c.single && !r.head_decay && !r.silu && !r.nq && c.slabs.ws && c.up_out && c.a_dt &&
         c.C == (r.H * kTokDv + 2 * r.G * kTokDk) && c.T == r.B && r.state == c.state && r.slot_stride == c.slot_stride &&
         (((long)c.off | c.off_dt | a.z_col | c.slot_stride | (long)c.tail_off | (long)r.s_off | c.slabs.N | c.up.N) & 3) == 0 && ((uintptr_t)c.state & 15) == 0 &&
         (((uintptr_t)a.out | (uintptr_t)c.up_out | (uintptr_t)c.bias) & 7) == 0 && ((uintptr_t)c.w & 15) == 0;
}
cudaError_t ssm_token(cudaStream_t s, const SsmTokenArgs& a) {
  if (a.r.B <= 0) return cudaSuccess;
  const int hg = a.r.H / a.r.G, up = a.c.T * ((a.c.up.N / 4 + 255) / 256);
  const dim3 grid(a.r.B * a.r.H + (up + hg - 1) / hg * hg);
  if (hg == 8) return launch_k(ssm_token_kernel<8>, grid, dim3(256), 0, s, true, a);
  if (hg == 4) return launch_k(ssm_token_kernel<4>, grid, dim3(256), 0, s, true, a);
  return hg == 2 ? launch_k(ssm_token_kernel<2>, grid, dim3(256), 0, s, true, a) : cudaErrorInvalidValue;
}

cudaError_t lin_recurrence(cudaStream_t s, const LinRecArgs& a) {
  if (a.B <= 0) return cudaSuccess;
  if (a.G <= 0 || a.H % a.G || a.Dk > 256 || a.Dk <= 0) return cudaErrorInvalidValue;
  if (lin_step_ok(a)) return launch_k(lin_step_kernel, dim3(a.B, a.H, (a.Dv + 63) / 64), dim3((a.Dk + 15) / 16 * 32), 0, s, true, a);
  if (lin_portion_ok(a)) {
    const bool few = lin_portion_narrow(a);
    if (a.Dk <= 64) return launch_portion<64, 8, 4, 4, 5>(s, a);
    if (a.Dk <= 128) return few ? launch_portion<128, 8, 4, 4, 5>(s, a) : lin_portion_many(a) ? launch_portion<128, 8, 8, 4, 3>(s, a) : launch_portion<128, 16, 4, 4, 4>(s, a);
    return few ? launch_portion<256, 16, 4, 4, 4>(s, a) : launch_portion<256, 16, 4, 8, 2>(s, a);
  }
  // two columns per lane (blocks of 64 columns) halve the shared-memory reads per product; heads of up to 32 value columns
  // keep one.  HB_REC_COLS=1 forces the narrow blocks of this kernel (A/B measurements)
  // (the arithmetic per column is the same either way, so the choice never shows in a result; narrow blocks for small grids
  // measured no faster)
  static const bool narrow = [] { const char* e = getenv("HB_REC_COLS"); return e && atoi(e) == 1; }();
  if (a.Dv > 32 && !narrow) {
    if (a.Dk <= 16) return launch_rec<16, 2>(s, a);
    if (a.Dk <= 32) return launch_rec<32, 2>(s, a);
    if (a.Dk <= 64) return launch_rec<64, 2>(s, a);
    if (a.Dk <= 128) return launch_rec<128, 2>(s, a);
    return launch_rec<256, 2>(s, a);
  }
  if (a.Dk <= 16) return launch_rec<16, 1>(s, a);
  if (a.Dk <= 32) return launch_rec<32, 1>(s, a);
  if (a.Dk <= 64) return launch_rec<64, 1>(s, a);
  if (a.Dk <= 128) return launch_rec<128, 1>(s, a);
  return launch_rec<256, 1>(s, a);
}

cudaError_t memory_readout(cudaStream_t s, const float* num, long ldnum, const float* nq, long ldn, const float* ab, long ldab,
                           const float* g, long ldg, const void* w, bool f32, float eps, float scale, float* out, bf16* outb, long ldout,
                           int col0, int T, int H, int Dv) {
  if (T <= 0) return cudaSuccess;
  const unsigned blocks = (unsigned)(((long)T * H + 7) / 8);
  if (f32) memory_readout_kernel<float><<<blocks, 256, 0, s>>>(num, ldnum, nq, ldn, ab, ldab, g, ldg, (const float*)w, eps, scale, out, outb, ldout, col0, T, H, Dv);
  else memory_readout_kernel<bf16><<<blocks, 256, 0, s>>>(num, ldnum, nq, ldn, ab, ldab, g, ldg, (const bf16*)w, eps, scale, out, outb, ldout, col0, T, H, Dv);
  return cudaGetLastError();
}

cudaError_t gated_group_norm(cudaStream_t s, const float* y, long ldy, const float* z, long ldz, const void* w, bool f32, float eps, int parts,
                             float* out, bf16* outb, int T, int n, bool gate_last, const bf16* zb,
                             const Slabs* z_slabs, int z_col) {
  if (T <= 0) return cudaSuccess;
  if (parts < 1 || n % parts) return cudaErrorInvalidValue;
  dim3 grid(parts, T);
  const int len = n / parts;
  const Slabs zsl = z_slabs ? *z_slabs : Slabs();
  if (z_slabs && (f32 || ((z_slabs->N | z_col) & 3))) return cudaErrorInvalidValue;
  if (len % 4 == 0 && len <= 8192 && ((ldy | ldz) & 3) == 0 && (((uintptr_t)y | (uintptr_t)z | (uintptr_t)out) & 15) == 0 && (((uintptr_t)outb | (uintptr_t)zb) & 7) == 0) {
#define HB_GGN(WT, CH, SLABS) \
  return launch_k(gated_group_norm_vec_kernel<WT, CH, SLABS>, dim3(T, parts), dim3(256), 0, s, true, y, ldy, z, zb, ldz, (const WT*)w, eps, parts, out, outb, n, (int)gate_last, zsl, z_col)
#define HB_GGN_T(CH) do { if (f32) HB_GGN(float, CH, false); else if (z_slabs) HB_GGN(bf16, CH, true); else HB_GGN(bf16, CH, false); } while (0)
    // Fewer parts than the blocks that fit the machine are through sooner with a block each (us block | warp: 16 tokens x 8 parts of 512 entries 2.4 | 4.2, of
    // 256 2.4 | 3.0, 64 tokens 3.3 | 4.3 and 3.0 | 3.1, 300 tokens 6.6 | 6.0 and 6.2 | 4.3; of 128 2.7 | 2.4 at 16 tokens), wide parts always (2000 tokens x 4
    // parts of 1024 21 | 24)
    if (len <= 512 && (len <= 128 || (long)T * parts > 8 * effective_sms(148)) && (long)T * parts <= INT_MAX) {
      const int items = T * parts;
#define HB_GGW(WT, CH, SLABS)                                                                                                                                 \
  return launch_k(gated_group_norm_warp_kernel<WT, CH, SLABS>, dim3((items + 7) / 8), dim3(256), 0, s, true, y, ldy, z, zb, ldz, (const WT*)w, eps, parts,    \
                  out, outb, n, (int)gate_last, items, zsl, z_col)
#define HB_GGW_T(CH) do { if (f32) HB_GGW(float, CH, false); else if (z_slabs) HB_GGW(bf16, CH, true); else HB_GGW(bf16, CH, false); } while (0)
      if (len <= 128) HB_GGW_T(1);
      if (len <= 256) HB_GGW_T(2);
      HB_GGW_T(4);
#undef HB_GGW_T
#undef HB_GGW
    }
    if (len <= 1024) HB_GGN_T(1);
    else if (len <= 2048) HB_GGN_T(2);
    else if (len <= 4096) HB_GGN_T(4);
    else HB_GGN_T(8);
#undef HB_GGN_T
#undef HB_GGN
  }
  if (zb || z_slabs) return cudaErrorInvalidValue;
  if (f32) gated_group_norm_kernel<float><<<grid, 256, 0, s>>>(y, ldy, z, ldz, (const float*)w, eps, parts, out, outb, n, gate_last);
  else gated_group_norm_kernel<bf16><<<grid, 256, 0, s>>>(y, ldy, z, ldz, (const bf16*)w, eps, parts, out, outb, n, gate_last);
  return cudaGetLastError();
}

cudaError_t gate_scale_rows(cudaStream_t s, const float* in, const bf16* inb, long ldi, const float* g, long ldg, float scale, float* out,
                            bf16* outb, long ldout, int col0, int T, int n) {
  if (T <= 0 || n <= 0) return cudaSuccess;
  if ((in == nullptr) == (inb == nullptr)) return cudaErrorInvalidValue;
  gate_scale_kernel<<<dim3((n + 255) / 256, T), 256, 0, s>>>(in, inb, ldi, g, ldg, scale, out, outb, ldout, col0, n);
  return cudaGetLastError();
}

cudaError_t parallel_step(cudaStream_t s, const float* x, const int32_t* row_index, const float* y, const float* y2, const void* bias,
                          float bias_scale, const void* w1, const void* w2, bool f32, float eps, float* x_out, float* h1, bf16* h1b, float* h2,
                          bf16* h2b, int rows, int W, const ParScale* scale) {
  if (rows <= 0) return cudaSuccess;
  const ParScale sc = scale ? *scale : ParScale();
  if ((sc.y_slabs.ws != nullptr) != (sc.y2_slabs.ws != nullptr) || (sc.y_slabs.ws && (y || y2 || sc.top_k > 0))) return cudaErrorInvalidValue;
  if (((y2 || sc.top_k > 0) && !y) || (sc.top_k > 0 && (y2 || !sc.rows || !sc.row_of || !sc.wts))) return cudaErrorInvalidValue;
  const uintptr_t al = (uintptr_t)x | (uintptr_t)y | (uintptr_t)y2 | (uintptr_t)bias | (uintptr_t)w1 | (uintptr_t)w2 | (uintptr_t)x_out | (uintptr_t)h1 |
                       (uintptr_t)h1b | (uintptr_t)h2 | (uintptr_t)h2b | (uintptr_t)sc.s1 | (uintptr_t)sc.s2 | (uintptr_t)sc.rows;
  if (W % 4 == 0 && W <= 4 * 256 * kParChunks && (al & 15) == 0 && sc.top_k <= kParTop) {
#define HB_PAR_IN(WT, CH, IN)                                                                                                                  \
  return launch_k(parallel_step_vec_kernel<WT, CH, IN>, dim3(rows), dim3(256), 0, s, launch_early((long)rows * W, 8), x, row_index, y, y2, (const WT*)bias, bias_scale, \
                  (const WT*)w1, (const WT*)w2, eps, x_out, h1, h1b, h2, h2b, W, sc)
#define HB_PAR(WT, CH)                                  \
  do {                                                  \
    if (sc.y_slabs.ws) HB_PAR_IN(WT, CH, PAR_SLABS);    \
    if (sc.top_k > 0) HB_PAR_IN(WT, CH, PAR_EXPERTS);   \
    HB_PAR_IN(WT, CH, PAR_ROWS);                        \
  } while (0)
    if (W <= 1024) { if (f32) HB_PAR(float, 1); else HB_PAR(bf16, 1); }
    else if (W <= 2048) { if (f32) HB_PAR(float, 2); else HB_PAR(bf16, 2); }
    else if (W <= 4096) { if (f32) HB_PAR(float, 4); else HB_PAR(bf16, 4); }
    else { if (f32) HB_PAR(float, 8); else HB_PAR(bf16, 8); }
#undef HB_PAR
#undef HB_PAR_IN
  }
  if ((size_t)W * 4 > 200 * 1024 || sc.y_slabs.ws) return cudaErrorInvalidValue;
  const size_t smem = (size_t)W * 4;
  if (f32)
    parallel_step_kernel<float><<<rows, 256, smem, s>>>(x, row_index, y, y2, (const float*)bias, bias_scale, (const float*)w1, (const float*)w2,
                                                        eps, x_out, h1, h1b, h2, h2b, W, sc);
  else
    parallel_step_kernel<bf16><<<rows, 256, smem, s>>>(x, row_index, y, y2, (const bf16*)bias, bias_scale, (const bf16*)w1, (const bf16*)w2, eps,
                                                       x_out, h1, h1b, h2, h2b, W, sc);
  return cudaGetLastError();
}

bool embed_step_ok(const void* table, const void* w0, const void* w1, const void* w2, const BigramArgs& bg, int W) {
  return W % 8 == 0 && W <= 4 * 256 * kParChunks && (((uintptr_t)table | (uintptr_t)w0 | (uintptr_t)w1 | (uintptr_t)w2 | (uintptr_t)bg.table) & 15) == 0;
}
cudaError_t embed_step(cudaStream_t s, const int32_t* tokens, const void* table, float scale, const BigramArgs& bg, const void* w0, float off, const void* w1,
                       const void* w2, bool f32, float eps, float* x, float* h1, bf16* h1b, float* h2, bf16* h2b, int T, int W) {
  if (T <= 0) return cudaSuccess;
  const uintptr_t al = (uintptr_t)x | (uintptr_t)h1 | (uintptr_t)h1b | (uintptr_t)h2 | (uintptr_t)h2b;
  if (!embed_step_ok(table, w0, w1, w2, bg, W) || (al & 15)) return cudaErrorInvalidValue;
#define HB_EMB(WT, CH)                                                                                                                                  \
  return launch_k(embed_step_kernel<WT, CH>, dim3(T), dim3(256), 0, s, true, tokens, (const WT*)table, scale, bg, (const WT*)w0, off, (const WT*)w1, \
                  (const WT*)w2, eps, x, h1, h1b, h2, h2b, W)
  if (W <= 1024) { if (f32) HB_EMB(float, 1); else HB_EMB(bf16, 1); }
  if (W <= 2048) { if (f32) HB_EMB(float, 2); else HB_EMB(bf16, 2); }
  if (W <= 4096) { if (f32) HB_EMB(float, 4); else HB_EMB(bf16, 4); }
  if (f32) HB_EMB(float, 8); else HB_EMB(bf16, 8);
#undef HB_EMB
}

cudaError_t relu2_rows(cudaStream_t s, const float* in, long ldi, float* out, bf16* outb, int T, int n) {
  if (T <= 0 || n <= 0) return cudaSuccess;
  return launch_k(relu2_kernel, dim3((n + 255) / 256, T), dim3(256), 0, s, true, in, ldi, out, outb, n);
}
cudaError_t relu2_rows_b16(cudaStream_t s, const bf16* in, long ldi, bf16* out, int T, int n) {
  if (T <= 0 || n <= 0) return cudaSuccess;
  relu2_b16_kernel<<<dim3((n + 255) / 256, T), 256, 0, s>>>(in, ldi, out, n);
  return cudaGetLastError();
}

}  // namespace hb
