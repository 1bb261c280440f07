// The scalar-decay recurrence S_t = a_t S_(t-1) + b_t k_t v_t^T, o_t = S_t^T q_t (state-space layers) over long prompt portions, on the
// tensor cores.  With chunks of 128 tokens, i / j counted inside the chunk, n tokens in it, S the state behind the chunk before,
// L_ij = a_(j+1) .. a_i and P_i = a_0 .. a_i:
//
//   A = Q K^T                    o_i = P_i S^T q_i + sum_(j <= i) L_ij b_j A_ij v_j
//   S <- P_(n-1) S + sum_j L_(n-1)j b_j k_j v_j^T
//
// q, k, v, a, b and the state are fp32 and stay so: every operand of a product travels as THREE bf16 terms, x = h + m + l with each the
// rounded rest of the ones before (24 significant bits and fp32's range), and a product is the six term products lh, hl, mm, mh,
// hm, hh with fp32 accumulation, so what is dropped is below 2^-24 of the factors.  The small products come first, and for A the
// second half of hh has an accumulator of its own, because the tensor pipe's accumulators round toward zero: only the last steps
// do so at the sum's full size.  Products of decays are formed in 64 bits; the state and the sum of an output's two parts are
// formed in registers, once per 128 tokens where the token-by-token kernel rounds the state at every token.  Relative errors
// against 64 bits, that kernel / this one: state 7.2e-8 / 6.4e-8, outputs 1.1e-7 / 1.3e-7 at a model's decays, outputs 4.2e-7 /
// 2.3e-7 and state 4.7e-7 / 1.6e-7 over 2048 tokens of slow decays.
//
// Bound by the threads that split operands and by the tensor pipe (six passes).  One CTA per (entry, head, 64 value columns) walks the
// entry's chunks; an entry that starts at position 0 starts from zeros.
//   warp 16   : all products: A | S^T q | W V | U = K^T Vw, in this order
//   warps 0-15: thread (row r = 32 (warp & 3) + lane, quarter qf = warp >> 2).  While the products of a chunk run they split the next
//               chunk's q (into TMEM: the A operand of two products) and v; k, whose tile U's product still reads, comes last.
// TMEM columns: [U (64) | S^T q, then W V (64), both together A's second accumulator | q terms (3 x 64) | A (128), then W terms
// (3 x 64)].  Shared memory: k terms, v terms, one set of tiles that holds S's terms for S^T q and then the weighted v's for U.
// Measured (11k tokens in 8 sequences, 64 heads, 128 x 64 states): 1650 us token by token, 575 us here.
// A NaN or an infinity among the inputs reaches every row of its chunk and head (earlier ones of the same sequence too).
// Waits are bounded: one that runs out marks the launch as failed (the host reads the flag behind the step), and the block runs
// on without products or stores until it has given its TMEM back.
#include <algorithm>

#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"

namespace hb {
namespace {

constexpr int C = 128;             // tokens per chunk
constexpr int NV = 64;             // value columns per CTA
constexpr int kWarps = 16;         // that split operands and finish rows; one more issues the products
constexpr int kThreads = 32 * kWarps + 32;
constexpr int kTile = C * 128;     // 64 bf16 columns of 128 rows
constexpr long long kWaitCycles = 2000000000ll;

struct Sm {
  static constexpr int K = 3 * 2 * kTile, V = 3 * kTile, W = 3 * kTile;
  static constexpr int F = 2 * 8 * C * 4;  // decays of two chunks (below)
  static constexpr int SIZE = 1024 + K + V + W + F + 128;
};
static_assert(Sm::SIZE <= 227 * 1024, "shared memory of one CTA");

__device__ __forceinline__ void split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  h = pack_bf16x2(x0, x1);
  float2 f = unpack_bf16x2(h);
  x0 -= f.x;
  x1 -= f.y;
  m = pack_bf16x2(x0, x1);
  f = unpack_bf16x2(m);
  l = pack_bf16x2(x0 - f.x, x1 - f.y);
}
// eight values as the 16-byte piece `piece` of row r in the three tiles that start at `tile`, `term` bytes apart
__device__ __forceinline__ void put8(uint8_t* tile, int term, int r, int piece, const float (&x)[8]) {
  uint4 t[3];
#pragma unroll
  for (int e = 0; e < 4; ++e) split2(x[2 * e], x[2 * e + 1], (&t[0].x)[e], (&t[1].x)[e], (&t[2].x)[e]);
  uint8_t* d = tile + r * 128 + ((piece ^ (r & 7)) << 4);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(d + i * term) = t[i];
}
// 32 bytes per lane and instruction (a row's quarter in four loads of its own thread, two rows of k in one of a warp)
__device__ __forceinline__ void ld8(const float* p, bool live, float (&x)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) x[e] = 0.f;
  if (live)
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7])
                 : "l"(p));
}
__device__ __forceinline__ void st8(float* p, const float (&x)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "f"(x[4]), "f"(x[5]),
               "f"(x[6]), "f"(x[7])
               : "memory");
}

__global__ void __launch_bounds__(kThreads, 1) rec_chunk_kernel(const __grid_constant__ RecChunkArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;            // [term][64-channel sub-tile][token][128 B]
  uint8_t* sV = sK + Sm::K;      // [term][token][128 B]
  uint8_t* sW = sV + Sm::V;      // [term][key channel or token][128 B]
  float* sF = reinterpret_cast<float*>(sW + Sm::W);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sF + Sm::F / 4);
  uint64_t *k_ready = bars, *s_ready = bars + 1, *a_full = bars + 2, *o1_full = bars + 3, *p_ready = bars + 4, *vw_ready = bars + 5, *o_full = bars + 6,
           *s_done = bars + 7, *d_ready = bars + 8, *a_read = bars + 9;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_ptr + 1);

  const int b = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * NV;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = a.cu[b], n_tok = a.cu[b + 1] - t0;
  if (n_tok <= 0) return;
  const int chunks = (n_tok + C - 1) / C;

  if (threadIdx.x == 0) {
    *dead = 0;
    mbar_init(k_ready, kWarps);
    mbar_init(s_ready, kWarps);
    mbar_init(a_full, 1);
    mbar_init(o1_full, 1);
    mbar_init(p_ready, kWarps);
    mbar_init(vw_ready, kWarps);
    mbar_init(o_full, 1);
    mbar_init(s_done, 1);
    mbar_init(d_ready, 1);
    mbar_init(a_read, kWarps);
    fence_barrier_init();
  }
  if (warp == kWarps) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_ptr, 0);
  const uint32_t tU = tmem, tO = tmem + 64, tQ = tmem + 128, tA = tmem + 320;

  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (*dead || mbar_try_wait(bar, parity)) return;
    const long long c0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
      if (*dead) return;
      if (clock64() - c0 > kWaitCycles) {
        *dead = 1;
        *a.error = 1;
        return;
      }
    }
  };

  if (warp == kWarps) {
    const bool leader = elect_one_sync();
    constexpr uint32_t id_qk = umma_idesc_bf16(C, C, 0, 0), id_mn = umma_idesc_bf16(C, NV, 0, 1), id_upd = umma_idesc_bf16(128, NV, 1, 1);
    const uint64_t kd = umma_desc_kmajor_sw128(smem_u32(sK)), kt = umma_desc_mnmajor_sw128(smem_u32(sK), kTile, 1024);
    const uint64_t vd = umma_desc_mnmajor_sw128(smem_u32(sV), kTile, 1024), wd = umma_desc_mnmajor_sw128(smem_u32(sW), kTile, 1024);
    const int nk = (a.Dk + 15) / 16;  // 16-channel steps of the products over the key channels
    const int k2 = (nk + 1) / 2;      // the first one of the second accumulator
    // Decays of chunk c, made while the products of the one before run: lane = four tokens; tokens behind the entry's end decay nothing
    // and weigh nothing.  [a | b | products of a from token 0, 32, 64, 96 on | b times the product from the next token to the chunk's
    // end | b times the product to the end of the token's 32]
    auto decays = [&](int c) {
      float* f = sF + (c & 1) * 8 * C;
      float av[4], bv[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = c * C + lane * 4 + e;
        const float* ab = a.ab + (size_t)(t0 + i) * a.ldab + h;
        av[e] = i < n_tok ? __ldg(ab) : 1.f;
        bv[e] = i < n_tok ? __ldg(ab + a.H) : 0.f;
        f[lane * 4 + e] = av[e];
        f[C + lane * 4 + e] = bv[e];
      }
      const double all = ((double)av[0] * av[1]) * ((double)av[2] * av[3]);
#pragma unroll
      for (int g = 0; g < 4; ++g) {  // products from token 32 g on (lanes 8 g and above)
        double up = lane >= 8 * g ? all : 1.;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double u = __shfl_up_sync(0xffffffffu, up, o);
          if (lane >= o) up *= u;
        }
        double p = __shfl_up_sync(0xffffffffu, up, 1);
        if (lane <= 8 * g) p = 1.;
#pragma unroll
        for (int e = 0; e < 4; ++e) f[(2 + g) * C + lane * 4 + e] = (float)(p *= av[e]);
      }
      double down = all, part = all;  // products from this lane on, to the chunk's end and to the end of its eight lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double d = __shfl_down_sync(0xffffffffu, down, o), g = __shfl_down_sync(0xffffffffu, part, o);
        if (lane + o < 32) down *= d;
        if ((lane & 7) + o < 8) part *= g;
      }
      double rest = __shfl_down_sync(0xffffffffu, down, 1), near = __shfl_down_sync(0xffffffffu, part, 1);
      if (lane == 31) rest = 1.;
      if ((lane & 7) == 7) near = 1.;
#pragma unroll
      for (int e = 3; e >= 0; --e) {
        f[6 * C + lane * 4 + e] = (float)(rest * bv[e]);
        f[7 * C + lane * 4 + e] = (float)(near * bv[e]);
        rest *= av[e];
        near *= av[e];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(d_ready);
    };
    decays(0);
    constexpr int ti[6] = {2, 0, 1, 1, 0, 0}, tj[6] = {0, 2, 1, 0, 1, 0};  // term pairs, small products first
    for (int c = 0; c < chunks; ++c) {
      const uint32_t ph = c & 1;
      wait(k_ready, ph);
      tc_fence_after();
      if (leader && !*dead) {
#pragma unroll
        for (int p = 0; p < 6; ++p)
          for (int k = 0; k < nk; ++k) {
            const bool second = p == 5 && k >= k2;  // (U's and o's columns are free until S^T q)
            umma_f16_ts(second ? tmem : tA, tQ + ti[p] * 64 + k * 8, kd + ((tj[p] * 2 * kTile + (k >> 2) * kTile + (k & 3) * 32) >> 4), id_qk,
                        second ? k != k2 : p + k != 0);
          }
        umma_commit(a_full);
      }
      wait(s_ready, ph);
      wait(a_read, ph);
      tc_fence_after();
      if (leader && !*dead) {
#pragma unroll
        for (int p = 0; p < 6; ++p)
          for (int k = 0; k < nk; ++k) umma_f16_ts(tO, tQ + ti[p] * 64 + k * 8, wd + ((tj[p] * kTile + k * 16 * 128) >> 4), id_mn, p + k != 0);
        umma_commit(o1_full);
      }
      if (c + 1 < chunks) decays(c + 1);
      wait(p_ready, ph);
      tc_fence_after();
      if (leader && !*dead) {
#pragma unroll
        for (int p = 0; p < 6; ++p)
          for (int k = 0; k < 8; ++k) umma_f16_ts(tO, tA + ti[p] * 64 + k * 8, vd + ((tj[p] * kTile + k * 16 * 128) >> 4), id_mn, p + k != 0);
        umma_commit(o_full);
      }
      wait(vw_ready, ph);
      tc_fence_after();
      if (leader && !*dead) {
#pragma unroll
        for (int p = 0; p < 6; ++p)
          for (int k = 0; k < 8; ++k)
            umma_f16_ss(tU, kt + ((ti[p] * 2 * kTile + k * 16 * 128) >> 4), wd + ((tj[p] * kTile + k * 16 * 128) >> 4), id_upd, p + k != 0);
        umma_commit(s_done);
      }
    }
    wait(s_done, (chunks - 1) & 1);
    if (*dead) {  // products already issued get time to end before the block's memory goes away
      const long long c0 = clock64();
      while (clock64() - c0 < 20000000ll) {}
    }
  } else {
    const int r = (warp & 3) * 32 + lane, qf = warp >> 2;
    const uint32_t lanes = (uint32_t)(warp & 3) << 21;  // this warp's 32 TMEM lanes
    const int kvh = h / (a.H / a.G);
    const float* const q0 = a.q + a.q_off + (size_t)kvh * a.Dk;
    const float* const k0 = a.k + a.k_off + (size_t)kvh * a.Dk;
    const float* const x0 = a.v + a.v_off + (size_t)h * a.Dv + v0;
    float* const st = a.state + (size_t)a.slots[b] * a.slot_stride + a.s_off + (size_t)h * a.Dk * a.Dv + (size_t)r * a.Dv + v0 + qf * 16;
    // (the skip rides on W's diagonal)
    const float skip = a.skip ? (a.f32 ? ((const float*)a.skip)[h] : __bfloat162float(((const bf16*)a.skip)[h])) / a.q_scale : 0.f;
    auto arrive = [&](uint64_t* bar) {
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    // q of chunk c: this thread's row and channel quarter
    auto load_q = [&](int c) {
      const int i = c * C + r;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        float x[2][8];
#pragma unroll
        for (int p = 0; p < 2; ++p) ld8(q0 + (size_t)(t0 + i) * a.ldq + qf * 32 + hh * 16 + p * 8, i < n_tok && qf * 32 + hh * 16 + p * 8 < a.Dk, x[p]);
        uint32_t t[3][8];
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int e = 0; e < 4; ++e) split2(x[p][2 * e], x[p][2 * e + 1], t[0][p * 4 + e], t[1][p * 4 + e], t[2][p * 4 + e]);
#pragma unroll
        for (int i2 = 0; i2 < 3; ++i2) tmem_st_32x32b_x8(tQ + lanes + i2 * 64 + qf * 16 + hh * 8, t[i2]);
      }
    };
    // v of chunk c: row (warp * 4 + lane / 8) + 64 g, eight columns per lane
    const int vr = warp * 4 + (lane >> 3), vp = lane & 7;
    auto read_v = [&](int c, float (&vv)[2][8]) {
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int i = c * C + vr + g * 64;
        ld8(x0 + (size_t)(t0 + i) * a.ldv + vp * 8, i < n_tok && v0 + vp * 8 < a.Dv, vv[g]);
      }
    };
    auto load_v = [&](int c) {
      float vv[2][8];
      read_v(c, vv);
#pragma unroll
      for (int g = 0; g < 2; ++g) put8(sV, kTile, vr + g * 64, vp, vv[g]);
    };
    // k of chunk c: two rows per warp and turn, eight channels per lane
    const int kr = warp * 8 + (lane >> 4), kp = lane & 15;
    auto load_k = [&](int c) {
      float kx[4][8];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int i = c * C + kr + g * 2;
        ld8(k0 + (size_t)(t0 + i) * a.ldk + kp * 8, i < n_tok && kp * 8 < a.Dk, kx[g]);
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) put8(sK + (kp >> 3) * kTile, 2 * kTile, kr + g * 2, kp & 7, kx[g]);
    };
    // lines of chunk c on their way into L2 while the chunk before is worked on: four threads per token
    auto prefetch = [&](int c) {
      const int i = c * C + (threadIdx.x >> 2), e = (threadIdx.x & 3) * 32;
      if (i >= n_tok) return;
      const size_t t = t0 + i;
      if (e < a.Dk) {
        prefetch_l2_line(k0 + t * a.ldk + e);
        prefetch_l2_line(q0 + t * a.ldq + e);
      }
      if (e < NV && v0 + e < a.Dv) prefetch_l2_line(x0 + t * a.ldv + e);
    };

    float S[16];  // the state: key channel r, value columns 16 qf ..
    {
      const bool have = a.first_pos[b] != 0 && r < a.Dk;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        if (have && v0 + qf * 16 + q * 4 < a.Dv) u = *reinterpret_cast<const float4*>(st + q * 4);
        S[4 * q] = u.x; S[4 * q + 1] = u.y; S[4 * q + 2] = u.z; S[4 * q + 3] = u.w;
      }
    }
    float dec = 0.f;  // the chunk's whole decay
    auto read16 = [&](uint32_t col, float (&x)[16]) {
      uint32_t u[16];
      tmem_ld_32x32b_x16(col + lanes + qf * 16, u);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) x[e] = __uint_as_float(u[e]);
    };
    auto advance = [&] {  // S <- dec S + U
      float x[16];
      read16(tU, x);
#pragma unroll
      for (int e = 0; e < 16; ++e) S[e] = fmaf(dec, S[e], x[e]);
    };
    load_q(0);
    load_v(0);
    for (int c = 0; c < chunks; ++c) {
      const uint32_t ph = c & 1;
      const int n = min(C, n_tok - c * C);
      const float* f = sF + ph * 8 * C;
      if (c > 0) {
        wait(s_done, (c - 1) & 1);
        tc_fence_after();
      }
      load_k(c);
      if (c > 0) advance();
      tmem_st_wait();  // q
      fence_proxy_async_smem();
      tc_fence_before();
      arrive(k_ready);
      // ---- the state's operand tiles
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = S[8 * q + e];
        put8(sW, kTile, r, qf * 2 + q, y);
      }
      fence_proxy_async_smem();
      arrive(s_ready);
      if (c + 1 < chunks) prefetch(c + 1);
      wait(d_ready, ph);
      dec = f[2 * C + n - 1];
      // ---- W_ij = L_ij b_j A_ij (zero above the diagonal), j in this thread's quarter of the row, from the right to the left
      wait(a_full, ph);
      tc_fence_after();
      {
        uint32_t x[32], t[3][16];
        tmem_ld_32x32b_x32(tA + lanes + qf * 32, x);
        if (a.Dk > 16) {
          uint32_t y[32];
          tmem_ld_32x32b_x32(tmem + lanes + qf * 32, y);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) x[e] = __float_as_uint(__uint_as_float(x[e]) + __uint_as_float(y[e]));
        } else {
          tmem_ld_wait();
        }
        tc_fence_before();
        arrive(a_read);
        bar_sync(2, 32 * kWarps);  // every quarter of every row has been read: W takes A's columns
        tc_fence_after();
        if ((warp & 3) > qf) {  // a quarter left of the diagonal: one factor per row, one per column
          const float row = f[(3 + qf) * C + r];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float4 g = *reinterpret_cast<const float4*>(f + 7 * C + qf * 32 + 2 * e);
            split2(__uint_as_float(x[2 * e]) * (row * g.x), __uint_as_float(x[2 * e + 1]) * (row * g.y), t[0][e], t[1][e], t[2][e]);
            split2(__uint_as_float(x[2 * e + 2]) * (row * g.z), __uint_as_float(x[2 * e + 3]) * (row * g.w), t[0][e + 1], t[1][e + 1], t[2][e + 1]);
          }
        } else if ((warp & 3) == qf) {  // the diagonal's: products of the decays from the right to the left
          float run = 0.f, next = 1.f;
#pragma unroll
          for (int e = 15; e >= 0; --e) {
            const int j = 2 * e;
            const float2 aj = *reinterpret_cast<const float2*>(f + qf * 32 + j), bj = *reinterpret_cast<const float2*>(f + C + qf * 32 + j);
            run = j + 1 == lane ? 1.f : run * next;
            float w1 = j + 1 <= lane ? __uint_as_float(x[2 * e + 1]) * (run * bj.y) : 0.f;
            if (j + 1 == lane) w1 += skip;
            run = j == lane ? 1.f : run * aj.y;
            float w0 = j <= lane ? __uint_as_float(x[2 * e]) * (run * bj.x) : 0.f;
            if (j == lane) w0 += skip;
            next = aj.x;
            split2(w0, w1, t[0][e], t[1][e], t[2][e]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) t[0][e] = t[1][e] = t[2][e] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) tmem_st_32x32b_x16(tA + lanes + i * 64 + qf * 16, t[i]);
      }
      // ---- P_i S^T q_i
      float vv[2][8];  // (v again, for U's product: the registers were W's)
      read_v(c, vv);
      wait(o1_full, ph);
      tc_fence_after();
      float o1[16];
      {
        const float pi = f[2 * C + r] * a.q_scale;
        read16(tO, o1);
#pragma unroll
        for (int e = 0; e < 16; ++e) o1[e] *= pi;
        tmem_st_wait();  // W
        tc_fence_before();
        arrive(p_ready);
      }
      // ---- the weighted v into the tiles that S^T q has left
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const float w = f[6 * C + vr + g * 64];
        float y[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = vv[g][e] * w;
        put8(sW, kTile, vr + g * 64, vp, y);
      }
      fence_proxy_async_smem();
      arrive(vw_ready);
      if (c + 1 < chunks) load_q(c + 1);  // (both products that read q's terms have ended)
      // ---- output rows
      wait(o_full, ph);
      tc_fence_after();
      {
        float x[16];
        read16(tO, x);
        tc_fence_before();
        if (c + 1 < chunks) load_v(c + 1);  // (W V, the last reader of the v tiles, has ended)
        float* o = a.out + (size_t)(t0 + c * C + r) * a.ldo + (size_t)h * a.Dv + v0 + qf * 16;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] = fmaf(a.q_scale, x[8 * p + e], o1[8 * p + e]);
          if (r < n && v0 + qf * 16 + p * 8 < a.Dv && !*dead) st8(o + p * 8, y);
        }
      }
    }
    wait(s_done, (chunks - 1) & 1);
    tc_fence_after();
    advance();
    if (r < a.Dk && !*dead) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (v0 + qf * 16 + q * 4 < a.Dv) *reinterpret_cast<float4*>(st + q * 4) = make_float4(S[4 * q], S[4 * q + 1], S[4 * q + 2], S[4 * q + 3]);
    }
    tc_fence_before();
  }
  __syncthreads();
  if (warp == kWarps) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace

bool rec_chunk_ok(const RecChunkArgs& a) {
  return a.Dk > 0 && a.Dk <= 128 && a.Dk % 8 == 0 && a.Dv > 0 && a.Dv % 8 == 0 && a.H <= 65535 && a.Dv <= 64 * 65535 && a.q_scale != 0.f &&
         ((a.ldq | a.ldk | a.ldv | a.ldo | (long)a.q_off | (long)a.k_off | (long)a.v_off) & 7) == 0 && ((a.slot_stride | (long)a.s_off) & 3) == 0 &&
         (((uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v | (uintptr_t)a.out) & 31) == 0 && ((uintptr_t)a.state & 15) == 0;
}

cudaError_t stack_chunk_init() {
  return cudaFuncSetAttribute(rec_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Sm::SIZE);
}

cudaError_t rec_chunk(cudaStream_t s, const RecChunkArgs& a) {
  if (a.B <= 0) return cudaSuccess;
  if (!rec_chunk_ok(a) || a.G <= 0 || a.H % a.G || !a.error) return cudaErrorInvalidValue;
  rec_chunk_kernel<<<dim3(a.B, a.H, (a.Dv + NV - 1) / NV), kThreads, Sm::SIZE, s>>>(a);
  return cudaGetLastError();
}

}  // namespace hb
