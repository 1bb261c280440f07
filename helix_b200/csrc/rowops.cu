// K1/K2/K4/K10(sampling)/K11 of SURVEY.md §2.3: HBM-bound row kernels.
// 16-byte vectorised coalesced loads, warp-shuffle + one smem hop for block reductions, fp32 math.
#include <math.h>

#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"

namespace hb {
namespace {

constexpr int kRowThreads = 128;
constexpr int kMaxVec = 4;  // row cached in registers up to 128*4*8 = 4096 elements

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int NT>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();  // protect `red` reuse
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < NT / 32) ? red[l] : 0.f;
  return warp_sum(t);
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

__global__ void embed_gather_kernel(const int32_t* __restrict__ tokens, const bf16* __restrict__ table,
                                    bf16* __restrict__ x, int H) {
  pdl_launch_dependents();
  pdl_wait();
  const int t = blockIdx.x;
  const uint4* src = reinterpret_cast<const uint4*>(table + (size_t)tokens[t] * H);
  uint4* dst = reinterpret_cast<uint4*>(x + (size_t)t * H);
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) dst[i] = __ldg(src + i);
}

__global__ void __launch_bounds__(kRowThreads)
rmsnorm_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ out,
               const int32_t* __restrict__ row_index, int H, float eps) {
  __shared__ float red[kRowThreads / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x;
  const size_t src_row = row_index ? (size_t)row_index[r] : (size_t)r;
  const uint4* src = reinterpret_cast<const uint4*>(x + src_row * H);
  const uint4* wv = reinterpret_cast<const uint4*>(w);
  uint4* dst = reinterpret_cast<uint4*>(out + (size_t)r * H);
  const int nvec = H / 8;
  uint4 cache[kMaxVec];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if (i < nvec) {
      cache[j] = src[i];
      float f[8];
      unpack8(cache[j], f);
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += f[k] * f[k];
    }
  }
  for (int i = threadIdx.x + kMaxVec * kRowThreads; i < nvec; i += kRowThreads) {
    float f[8];
    unpack8(src[i], f);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += f[k] * f[k];
  }
  ss = block_sum<kRowThreads>(ss, red);
  const float inv = rsqrtf(ss / (float)H + eps);
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if (i < nvec) {
      float f[8], g[8];
      unpack8(cache[j], f);
      unpack8(__ldg(wv + i), g);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[k] = f[k] * inv * g[k];
      dst[i] = pack8(f);
    }
  }
  for (int i = threadIdx.x + kMaxVec * kRowThreads; i < nvec; i += kRowThreads) {
    float f[8], g[8];
    unpack8(src[i], f);
    unpack8(__ldg(wv + i), g);
#pragma unroll
    for (int k = 0; k < 8; ++k) f[k] = f[k] * inv * g[k];
    dst[i] = pack8(f);
  }
}

// LayerNorm over rows of up to kMaxVec*128*8 elements held in registers (two-pass mean / variance).
template <bool kEmbed>
__global__ void __launch_bounds__(kRowThreads)
layernorm_kernel(const bf16* __restrict__ x, const bf16* __restrict__ gamma, const bf16* __restrict__ beta,
                 bf16* __restrict__ out, int H, float eps, const int32_t* __restrict__ tokens,
                 const int32_t* __restrict__ positions, const bf16* __restrict__ word, const bf16* __restrict__ pos,
                 const bf16* __restrict__ type0) {
  __shared__ float red[kRowThreads / 32];
  const int r = blockIdx.x;
  const int nvec = H / 8;
  float vals[kMaxVec][8];
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if (i < nvec) {
      if (kEmbed) {
        float a[8], b[8], c[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(word + (size_t)tokens[r] * H) + i), a);
        unpack8(__ldg(reinterpret_cast<const uint4*>(pos + (size_t)positions[r] * H) + i), b);
        unpack8(__ldg(reinterpret_cast<const uint4*>(type0) + i), c);
#pragma unroll
        for (int k = 0; k < 8; ++k) vals[j][k] = a[k] + b[k] + c[k];
      } else {
        unpack8(reinterpret_cast<const uint4*>(x + (size_t)r * H)[i], vals[j]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += vals[j][k];
    }
  }
  const float mean = block_sum<kRowThreads>(sum, red) / (float)H;
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if (i < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = vals[j][k] - mean;
        sq += d * d;
      }
    }
  }
  const float inv = rsqrtf(block_sum<kRowThreads>(sq, red) / (float)H + eps);
#pragma unroll
  for (int j = 0; j < kMaxVec; ++j) {
    const int i = threadIdx.x + j * kRowThreads;
    if (i < nvec) {
      float g[8], b[8], o[8];
      unpack8(__ldg(reinterpret_cast<const uint4*>(gamma) + i), g);
      unpack8(__ldg(reinterpret_cast<const uint4*>(beta) + i), b);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = (vals[j][k] - mean) * inv * g[k] + b[k];
      reinterpret_cast<uint4*>(out + (size_t)r * H)[i] = pack8(o);
    }
  }
}

// Warp-per-row LayerNorm for narrow rows (H <= 1024, e.g. the 768-wide encoder): no shared memory, no block barrier,
// four rows per 128-thread block; the block-per-row kernel above leaves a quarter of its threads idle at H = 768.
template <bool kEmbed>
__global__ void __launch_bounds__(128)
layernorm_warp_kernel(const bf16* __restrict__ x, const bf16* __restrict__ gamma, const bf16* __restrict__ beta,
                      bf16* __restrict__ out, int rows, int H, float eps, const int32_t* __restrict__ tokens,
                      const int32_t* __restrict__ positions, const bf16* __restrict__ word, const bf16* __restrict__ pos,
                      const bf16* __restrict__ type0) {
  pdl_launch_dependents();
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  pdl_wait();
  if (r >= rows) return;
  const int nvec = H / 8;
  float vals[4][8];
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = lane + j * 32;
    if (i < nvec) {
      if (kEmbed) {
        float a[8], b[8], c[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(word + (size_t)tokens[r] * H) + i), a);
        unpack8(__ldg(reinterpret_cast<const uint4*>(pos + (size_t)positions[r] * H) + i), b);
        unpack8(__ldg(reinterpret_cast<const uint4*>(type0) + i), c);
#pragma unroll
        for (int k = 0; k < 8; ++k) vals[j][k] = a[k] + b[k] + c[k];
      } else {
        unpack8(reinterpret_cast<const uint4*>(x + (size_t)r * H)[i], vals[j]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) sum += vals[j][k];
    }
  }
  const float mean = warp_sum(sum) / (float)H;
  float sq = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (lane + j * 32 < nvec) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float d = vals[j][k] - mean;
        sq += d * d;
      }
    }
  }
  const float inv = rsqrtf(warp_sum(sq) / (float)H + eps);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = lane + j * 32;
    if (i < nvec) {
      float g[8], b[8], o[8];
      unpack8(__ldg(reinterpret_cast<const uint4*>(gamma) + i), g);
      unpack8(__ldg(reinterpret_cast<const uint4*>(beta) + i), b);
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = (vals[j][k] - mean) * inv * g[k] + b[k];
      reinterpret_cast<uint4*>(out + (size_t)r * H)[i] = pack8(o);
    }
  }
}

__global__ void rope_table_kernel(const int32_t* __restrict__ positions, const float* __restrict__ inv_freq,
                                  float* __restrict__ cs, int T, int D) {
  const int half = D / 2;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * half) return;
  const int t = i / half, k = i % half;
  float s, c;
  sincosf((float)positions[t] * inv_freq[k], &s, &c);
  cs[(size_t)t * D + k] = c;
  cs[(size_t)t * D + half + k] = s;
}

// One block per token. Pairs (i, i+D/2) of each q/k head are rotated; k,v rows go to the paged cache.
__global__ void __launch_bounds__(256)
rope_kv_write_kernel(bf16* __restrict__ qkv, const int32_t* __restrict__ positions,
                     const int32_t* __restrict__ slot_mapping, const float* __restrict__ inv_freq,
                     bf16* __restrict__ k_cache, bf16* __restrict__ v_cache, int Hq, int Hkv, int D, int page_size) {
  extern __shared__ float cs[];  // cos[D/2], sin[D/2]
  const int t = blockIdx.x;
  const int half = D / 2;
  const float p = (float)positions[t];
  for (int i = threadIdx.x; i < half; i += blockDim.x) {
    float s, c;
    sincosf(p * inv_freq[i], &s, &c);
    cs[i] = c;
    cs[half + i] = s;
  }
  __syncthreads();
  const int row_elems = (Hq + 2 * Hkv) * D;
  bf16* row = qkv + (size_t)t * row_elems;
  // rotate q and k heads: work items = (Hq+Hkv) * half/2 bf16x2 pairs
  const int pairs_per_head = half / 2;
  const int items = (Hq + Hkv) * pairs_per_head;
  for (int it = threadIdx.x; it < items; it += blockDim.x) {
    const int h = it / pairs_per_head, j = (it % pairs_per_head) * 2;
    __nv_bfloat162* lo = reinterpret_cast<__nv_bfloat162*>(row + h * D + j);
    __nv_bfloat162* hi = reinterpret_cast<__nv_bfloat162*>(row + h * D + half + j);
    const float2 a = __bfloat1622float2(*lo), b = __bfloat1622float2(*hi);
    const float c0 = cs[j], c1 = cs[j + 1], s0 = cs[half + j], s1 = cs[half + j + 1];
    *lo = __floats2bfloat162_rn(rope_lo(a.x, b.x, c0, s0), rope_lo(a.y, b.y, c1, s1));
    *hi = __floats2bfloat162_rn(rope_hi(a.x, b.x, c0, s0), rope_hi(a.y, b.y, c1, s1));
  }
  const int slot = slot_mapping ? slot_mapping[t] : -1;
  if (slot < 0) return;
  __syncthreads();  // rotated k visible to the copy below
  const int page = slot / page_size, off = slot % page_size;
  const int vec_per_head = D / 8;
  const uint4* ksrc = reinterpret_cast<const uint4*>(row + Hq * D);
  const uint4* vsrc = reinterpret_cast<const uint4*>(row + (Hq + Hkv) * D);
  for (int it = threadIdx.x; it < Hkv * vec_per_head; it += blockDim.x) {
    const int h = it / vec_per_head, j = it % vec_per_head;
    const size_t dst = (((size_t)page * Hkv + h) * page_size + off) * vec_per_head + j;
    reinterpret_cast<uint4*>(k_cache)[dst] = ksrc[it];
    reinterpret_cast<uint4*>(v_cache)[dst] = vsrc[it];
  }
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {  // splitmix64 finaliser
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ void argmax_merge(float& best, int& bi, float ov, int oi) {
  if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
}
// standard Gumbel noise of (seed, column): -log(-log u) of a uniform u
__device__ __forceinline__ float gumbel_uniform(uint64_t sd, int v) {
  const uint64_t h = mix64(sd ^ (0xD1B54A32D192ED03ull * (uint64_t)(v + 1)));
  // 23 random bits + 0.5: every value is exact in fp32 and u stays strictly inside (0,1) — with 24 bits the
  // "+0.5f" rounds the top half of the range up and u == 1.0 made the noise +inf (a uniformly random token won
  // once per 2^24 draws, ~0.8 % of sampled tokens at a 128k vocabulary).
  return ((float)(h >> 41) + 0.5f) * (1.0f / 8388608.0f);
}
// The inner log is the accurate one: the fast-math log has an absolute error comparable to log(1 - 2^-24).
__device__ __forceinline__ float gumbel_of(float u) { return -__logf(-logf(u)); }
__device__ __forceinline__ float gumbel(uint64_t sd, int v) { return gumbel_of(gumbel_uniform(sd, v)); }
template <int NT>
__device__ __forceinline__ void block_argmax(float& best, int& bi, float* sval, int* sidx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    argmax_merge(best, bi, ov, oi);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) { sval[w] = best; sidx[w] = bi; }
  __syncthreads();
  if (w == 0) {
    best = (l < NT / 32) ? sval[l] : -INFINITY;
    bi = (l < NT / 32) ? sidx[l] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      argmax_merge(best, bi, ov, oi);
    }
  }
}

// ---- sampling without filters: one look at every logit, in two launches ----
// stage 1: grid (chunks, B): per-chunk argmax of logits/T + Gumbel noise -> part[b][chunk]
constexpr int kSampleChunk = 4096;  // vocabulary columns per stage-1 block
__global__ void __launch_bounds__(256)
sample_stage1_kernel(const float* __restrict__ logits, int ldl, const float* __restrict__ temperature,
                     const uint64_t* __restrict__ seed, float* __restrict__ part_val, int* __restrict__ part_idx, int V) {
  __shared__ float sval[8];
  __shared__ int sidx[8];
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.y, chunk = blockIdx.x;
  const float* row = logits + (size_t)b * ldl;
  const float temp = temperature ? temperature[b] : 0.f;
  const bool greedy = !(temp > 0.f);
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const uint64_t sd = seed ? seed[b] : 0;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  const int v_end = min(V, (chunk + 1) * kSampleChunk);
  for (int v = chunk * kSampleChunk + threadIdx.x; v < v_end; v += 256) {
    float x = row[v] * inv_t;
    if (!greedy) x += gumbel(sd, v);
    argmax_merge(best, bi, x, v);
  }
  block_argmax<256>(best, bi, sval, sidx);
  if (threadIdx.x == 0) {
    part_val[b * gridDim.x + chunk] = best;
    part_idx[b * gridDim.x + chunk] = bi;
  }
}
// stage 2: one warp per row merges the chunk winners (lowest index wins ties, as in stage 1)
__global__ void __launch_bounds__(32)
sample_stage2_kernel(const float* __restrict__ part_val, const int* __restrict__ part_idx, int32_t* __restrict__ out,
                     int chunks) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int c = threadIdx.x; c < chunks; c += 32) argmax_merge(best, bi, part_val[b * chunks + c], part_idx[b * chunks + c]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    argmax_merge(best, bi, ov, oi);
  }
  if (threadIdx.x == 0) out[b] = bi < 0x7fffffff ? bi : 0;  // all-NaN row: emit a valid id, never an out-of-range one
}

// float -> unsigned key that orders like the float (and back); NaN is key 0, below every number, and key 0 is a NaN.  (The bits
// change type in asm: the compiler may turn integer operations on a float's sign into float ones, which lose a NaN's bits.)
__device__ __forceinline__ uint32_t fkey(float x) {
  uint32_t u;
  asm("mov.b32 %0, %1;" : "=r"(u) : "f"(x));
  if (x != x) return 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float fkey_inv(uint32_t k) {
  const uint32_t u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float x;
  asm("mov.b32 %0, %1;" : "=f"(x) : "r"(u));
  return x;
}

// ---- rows of the vocabulary, one cluster of NC blocks per row ----
// Both kernels below look at a row many times (bisection passes, arg-max rounds).  Reading 0.5 MB through one SM's L1 per pass left most
// SMs idle; here every block keeps its part of the row in shared memory, passes run on the parts and what they find meets through
// distributed shared memory, one cluster barrier per pass.  Rows whose eighths do not fit (vocabularies above 400k) are read
// from global memory instead (SM = false).
constexpr int kVocThreads = 512, kVocWarps = kVocThreads / 32;
constexpr int kVocSmemFloats = 50000;  // largest part kept on chip (200 KB)
__host__ __device__ inline int voc_slice(int V, int ctas) { return ((V + ctas - 1) / ctas + 3) & ~3; }

template <int NC>
__device__ __forceinline__ void voc_sync() {
  if constexpr (NC == 1) {
    __syncthreads();
  } else {  // (the aligned barrier wants converged warps)
    __syncwarp();
    cluster_sync_all();
  }
}

// f(i, values, how many of them exist) for every group of four columns i .. i + 3 of a slice of n that a thread keeps; eight groups are
// in flight per thread (one at a time left the load at the latency of eight round trips)
template <typename F>
__device__ __forceinline__ void load_slice(const float* __restrict__ src, int n, int tid, F&& f) {
  constexpr int kAhead = 8, kStep = kVocThreads * 4;
  const bool vec = ((uintptr_t)src & 15) == 0;
  for (int i0 = tid * 4; i0 < n; i0 += kStep * kAhead) {
    float v[kAhead][4];
#pragma unroll
    for (int g = 0; g < kAhead; ++g) {
      const int i = i0 + g * kStep;
      if (vec && i + 4 <= n) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(src + i));
        v[g][0] = t.x; v[g][1] = t.y; v[g][2] = t.z; v[g][3] = t.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[g][e] = i + e < n ? __ldg(src + i + e) : 0.f;
      }
    }
#pragma unroll
    for (int g = 0; g < kAhead; ++g) {
      const int i = i0 + g * kStep;
      if (i < n) f(i, v[g], min(4, n - i));
    }
  }
}

// ---- sampling: greedy / temperature (Gumbel-max), optionally from the top-k / top-p survivors ----
// The threshold that separates the survivors is found on the ordered 32-bit keys:
//   top-k : the largest key that keeps >= k tokens (ties at the k-th value are all kept)
//   top-p : among the top-k survivors, the largest key whose tokens' softmax(logits/T) mass reaches p of the survivors' mass
// Probability mass is accumulated in 2^-32 fixed point, so every sum is exact and independent of its order.
// One pass counts the tokens in kBins bins of values and sums the mass.  The counts give top-k's bin, and with each bin's mean weight an
// estimate of where the mass of top-p is reached, good to a few dozen tokens; a second pass sums the mass above a bracket around it exactly
// and hands the bracket's tokens, at most kFin, to block 0, which ranks them and checks that the answer is among them.  Where it is not
// (or the bins are no use: infinite maxima, hundreds of equal logits) the keys are searched by halves.  What is left of the time: the load, these two
// passes and the draw over 32 tokens a thread each, and seven cluster barriers.
// Measured (us, with passes of three keys or 128 bins of masses | now): 32 rows of 128256, kinds of filters mixed 60 | 32, top_p 0.95 68 | 35, top_k 40 25 | 21;
// 1 row 38 | 23; 64 rows of 32768 35 | 23.  The bins cost two barriers before anything is known, so rows whose first pass of keys had left next to
// nothing gain nothing (cold ones, below).
constexpr int kFin = 1024, kBins = 4096, kHeavy = 512;
constexpr float kReach = 80.f;  // tokens on either side of the estimate
struct alignas(16) SampleShared {
  uint32_t hist[kBins];  // tokens per bin: this block's, then the cluster's; afterwards the warps' queues of survivors
  uint32_t heavy[kHeavy];  // mass of the highest bins, in units of 2^-20: this block's, then (a float) the cluster's
  unsigned long long part[2][5];  // this block's totals of a pass: counts (c1 | c2 << 32), c3, masses m1 .. m3
  unsigned long long wred[kVocWarps][5];
  unsigned long long post[2][8];  // the blocks' shares of a sum
  alignas(16) uint32_t list[kFin];
  uint32_t sorted[256];
  float val[kVocWarps], top[8];  // (the blocks' maxima, at the end their best values)
  int idx[kVocWarps], top_idx[8];
  uint32_t warp_c[kVocWarps];
  float warp_m[kVocWarps], reach;
  int bin[2];        // bracket: its lowest and highest bin, the tokens from the lowest up and above the highest
  uint32_t upto[2];
  unsigned long long top_mass;
  uint32_t n_list, result;
};
constexpr int kQueue = kBins / kVocWarps;  // survivors that a warp collects before it draws for 32 of them

template <int NC, bool SM>
__global__ void __cluster_dims__(NC, 1, 1) __launch_bounds__(kVocThreads, 2)
sample_cluster_kernel(const float* __restrict__ logits, int ldl, const float* __restrict__ temperature, const uint64_t* __restrict__ seed,
              const int32_t* __restrict__ top_k, const float* __restrict__ top_p, int32_t* __restrict__ out, int V) {
  extern __shared__ __align__(16) float slice[];
  __shared__ SampleShared sh;
  pdl_launch_dependents();
  pdl_wait();
  typedef unsigned long long u64;
  const int b = blockIdx.x / NC, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = cluster_ctarank();
  const int per = voc_slice(V, NC), start = min(V, (int)rank * per), n = min(V, start + per) - start;
  const float* row = logits + (size_t)b * ldl + start;
  const float temp = temperature ? temperature[b] : 0.f;
  const bool greedy = !(temp > 0.f);
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const int k = top_k ? top_k[b] : 0;
  const float p = top_p ? top_p[b] : 1.f;
  const bool use_k = !greedy && k > 0 && k < V, use_p = !greedy && p > 0.f && p < 1.f, filters = use_k || use_p;

  float best = -INFINITY;
  int bi = 0x7fffffff;
  const uint64_t sd = seed ? seed[b] : 0;
  auto draw = [&](float raw, int i) {
    const int v = start + i;
    float x = raw * inv_t;
    if (!greedy) x += gumbel(sd, v);
    argmax_merge(best, bi, x, v);
  };
  // The same for every token of a part.  -log(-log u) <= -log(1 - u), one fast logarithm: where not even that (and a thousandth, far
  // above the rounding of both) reaches what the warp has found so far, which is soon true of nearly all, the exact noise is not needed.
  float bar = -INFINITY;
  auto draw_over = [&](const float (&raw)[4], int i, int have) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e >= have || raw[e] != raw[e]) continue;  // a NaN is never drawn
      if (greedy) {
        argmax_merge(best, bi, raw[e], start + i + e);
      } else {
        const float u = gumbel_uniform(sd, start + i + e), x = raw[e] * inv_t;
        if (!(x + (1e-3f - __logf(1.f - u)) < bar)) argmax_merge(best, bi, x + gumbel_of(u), start + i + e);
      }
    }
    bar = fmaxf(bar, best);
  };
  auto share_bar = [&] { bar = fkey_inv(__reduce_max_sync(__activemask(), fkey(bar))); };

  if (tid == 0) sh.n_list = 0;
  __syncwarp();  // (the aligned barrier wants converged warps)
  if constexpr (NC > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // (this block runs: others may write to it)
  float mx = -INFINITY;
  if constexpr (SM) {  // (entries behind the slice's end read as NaN)
    load_slice(row, n, tid, [&](int i, const float (&f)[4], int have) {
      if (!filters) {
        draw_over(f, i, have);
        share_bar();
        return;
      }
      const float none = __int_as_float(0x7fffffff);
      const float4 v = make_float4(f[0], have > 1 ? f[1] : none, have > 2 ? f[2] : none, have > 3 ? f[3] : none);
      mx = fmaxf(fmaxf(mx, fmaxf(v.x, v.y)), fmaxf(v.z, v.w));
      *reinterpret_cast<float4*>(slice + i) = v;
    });
  } else if (filters) {
    for (int i = tid; i < n; i += kVocThreads) mx = fmaxf(mx, __ldg(row + i));
  }
  __syncthreads();
  if constexpr (NC > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  auto scan = [&](auto&& f) {  // f(logit)
    if constexpr (SM) {
      for (int i = tid * 4; i < n; i += kVocThreads * 4) {
        const float4 q = *reinterpret_cast<const float4*>(slice + i);
        f(q.x);
        f(q.y);
        f(q.z);
        f(q.w);
      }
    } else {
      for (int i = tid; i < n; i += kVocThreads) f(__ldg(row + i));
    }
  };

  float floor_logit = -INFINITY;
  if (filters) {
    // row maximum (for the softmax weights)
    const uint32_t wm = __reduce_max_sync(0xffffffffu, fkey(mx));
    if (lane == 0) sh.val[warp] = fkey_inv(wm);
    __syncthreads();
    mx = sh.val[lane & (kVocWarps - 1)];
    mx = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(mx)));
    if (tid < NC) cluster_ptr<NC>(sh.top, tid)[rank] = mx;
    voc_sync<NC>();
    mx = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(sh.top[lane & (NC - 1)])));

    auto weight_at = [&](float x) -> u64 {
      const float e = __expf((x - mx) * inv_t) * 4294967296.0f;
      return e >= 0.f ? (u64)__float2uint_rz(e) + (e >= 4294967296.0f) : 0;  // (2^32 at the maximum itself; a NaN logit carries no mass)
    };
    int turn = 0;
    // sums of the cluster's blocks, in every thread of every block
    auto warp_total = [](u64 v) -> u64 {  // (a thread's share is below 2^58: three limbs, one hardware reduction each)
      const u64 a = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0xffffu), c = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 16) & 0x1fffffu),
                d = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 37));
      return a + (c << 16) + (d << 37);
    };
    int at_post = 0;
    auto cluster_add = [&](u64 v) -> u64 {
      v = warp_total(v);
      if (lane == 0) sh.wred[warp][0] = v;
      __syncthreads();
      if (warp == 0) {
        u64 t = lane < kVocWarps ? sh.wred[lane][0] : 0;
#pragma unroll
        for (int o = kVocWarps / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane < NC) cluster_ptr<NC>(sh.post[at_post], lane)[rank] = t;
      }
      voc_sync<NC>();
      u64 t = 0;
#pragma unroll
      for (int c = 0; c < NC; ++c) t += sh.post[at_post][c];
      at_post ^= 1;  // (a slot is written again two sums later, behind the barrier that follows every read of it)
      return t;
    };
    auto cluster_sum = [&](u64 (&v)[5]) {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const u64 t = j == 0 ? (u64)__reduce_add_sync(0xffffffffu, (uint32_t)v[0]) | (u64)__reduce_add_sync(0xffffffffu, (uint32_t)(v[0] >> 32)) << 32
                      : j == 1 ? (u64)__reduce_add_sync(0xffffffffu, (uint32_t)v[1]) : warp_total(v[j]);
        if (lane == 0) sh.wred[warp][j] = t;
      }
      __syncthreads();
      if (warp == 0) {
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          u64 t = lane < kVocWarps ? sh.wred[lane][j] : 0;
#pragma unroll
          for (int o = kVocWarps / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          if (lane == 0) sh.part[turn][j] = t;
        }
      }
      voc_sync<NC>();
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        u64 t = *cluster_ptr<NC>(&sh.part[turn][j], lane & (NC - 1));
#pragma unroll
        for (int o = NC / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        v[j] = t;
      }
      turn ^= 1;  // (a slot is written again two passes later, behind the barrier that follows every read of it)
    };
    // Block 0: the largest key of its list whose tokens, with c_hi tokens of mass m_hi above the list, reach `goal` in number or in mass;
    // `both`: goal in number first, then p of the mass of the tokens that this keeps.  Every block gets the answer (0: there is none).
    // The list is sorted (falling), its masses summed up along the way.
    auto decide = [&](bool by_mass, u64 goal, u64 c_hi, u64 m_hi, bool both) -> uint32_t {
      if (rank == 0) {
        const int nl = (int)sh.n_list, len = nl <= 256 ? 256 : nl <= 512 ? 512 : kFin;
        const uint32_t* list = sh.list;
        for (int i = nl + tid; i < len; i += kVocThreads) sh.list[i] = 0u;
        if (tid < 256) sh.sorted[tid] = 0u;
        if (tid == 0) sh.idx[0] = 0;
        __syncthreads();
        if (len == 256) {  // two threads per entry count the entries before it
          const int at = tid >> 1;
          const uint32_t key = sh.list[at];
          uint32_t before = 0;
#pragma unroll 4
          for (int j = tid & 1; j < (nl + 3) / 4; j += 2) {
            const uint4 q = *reinterpret_cast<const uint4*>(sh.list + 4 * j);
            before += (q.x > key) + (q.y > key) + (q.z > key) + (q.w > key);
            before += (q.x == key && 4 * j < at) + (q.y == key && 4 * j + 1 < at) + (q.z == key && 4 * j + 2 < at) + (q.w == key && 4 * j + 3 < at);
          }
          before += __shfl_xor_sync(0xffffffffu, before, 1);
          if ((tid & 1) == 0 && key != 0) sh.sorted[before] = key;
          list = sh.sorted;
        } else {
          for (int m = 2; m <= len; m *= 2)
            for (int j = m / 2; j > 0; j /= 2) {
              const int i = 2 * tid - (tid & (j - 1));
              if (tid < len / 2) {
                const uint32_t x = sh.list[i], y = sh.list[i + j];
                if ((i & m) == 0 ? x < y : x > y) {
                  sh.list[i] = y;
                  sh.list[i + j] = x;
                }
              }
              if (j > 32 || (j == 1 && m > 32)) __syncthreads();  // (pairs up to 32 apart stay inside a warp's 64 entries)
              else __syncwarp();
            }
        }
        __syncthreads();
        const bool in = tid < len / 2;
        const uint32_t k0 = in ? list[2 * tid] : 0u, k1 = in ? list[2 * tid + 1] : 0u;
        const u64 w0 = k0 ? weight_at(fkey_inv(k0)) : 0, w1 = k1 ? weight_at(fkey_inv(k1)) : 0;
        u64 upto = w0 + w1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const u64 t = __shfl_up_sync(0xffffffffu, upto, o);
          if (lane >= o) upto += t;
        }
        if (lane == 31) sh.wred[warp][0] = upto;
        __syncthreads();
        for (int w = 0; w < warp; ++w) upto += sh.wred[w][0];
        const u64 m1 = upto, m0 = upto - w1, before = m0 - w0;
        auto first = [&](u64 want) {  // the entry at which the mass reaches `want`
          if (k0 && m_hi + m0 >= want && m_hi + before < want) sh.idx[0] = (int)k0;
          if (k1 && m_hi + m1 >= want && m_hi + m0 < want) sh.idx[0] = (int)k1;
          __syncthreads();
        };
        if (by_mass) {
          first(goal);
        } else if (goal > c_hi && goal - c_hi <= (u64)nl) {
          const uint32_t kth = list[goal - c_hi - 1];
          if (!both) {
            if (tid == 0) sh.idx[0] = (int)kth;
            __syncthreads();
          } else {
            const uint32_t k2 = 2 * tid + 2 < len ? list[2 * tid + 2] : 0u;
            if (in && k0 >= kth && k1 < kth) sh.top_mass = m0;
            if (in && k1 >= kth && k2 < kth) sh.top_mass = m1;
            if (tid == 0) sh.idx[0] = (int)kth;  // (no mass at all: all of them)
            __syncthreads();
            first(max((u64)1, (u64)((double)p * (double)sh.top_mass)));
          }
        }
        if (tid < NC) *cluster_ptr<NC>(&sh.result, tid) = (uint32_t)sh.idx[0];
        if (tid == 0) sh.n_list = 0;
      }
      voc_sync<NC>();
      return sh.result;
    };
    auto list_token = [&](uint32_t q) { cluster_ptr<NC>(sh.list, 0)[atomicAdd(cluster_ptr<NC>(&sh.n_list, 0), 1u)] = q; };
    // Without bins: the largest key whose tokens (those with keys >= it) reach `goal`: in number, or in mass (by_mass).  Keeping [lo, ..) is
    // enough (c_lo tokens), keeping [hi, ..) is not (c_hi tokens of mass m_hi).
    auto search = [&](bool by_mass, u64 goal, u64 lo, u64 c_lo) -> u64 {
      u64 hi = (u64)fkey(mx) + 1, c_hi = 0, m_hi = 0;  // (nothing is above the maximum)
      for (int pass = 0; hi - lo > 1 && c_lo - c_hi > 256; ++pass) {
        // Logits are spread more evenly over values than over keys (where half of all keys are exponents nothing has): the first
        // pass looks a few temperatures below the maximum, the next ones divide the values between the bounds; from the eighth
        // on the keys are divided, so at most 8 + 16 passes are needed.
        const u64 d = hi - lo;
        u64 t[3];
        const float flo = fkey_inv((uint32_t)lo), fhi = fkey_inv((uint32_t)(hi - 1));
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float at = pass == 0 ? mx - temp * (j == 0 ? 16.f : j == 1 ? 8.f : 4.f) : flo + (fhi - flo) * (0.25f * (j + 1));
          const u64 by_key = lo + max(1ull, j == 0 ? d / 4 : j == 1 ? d / 2 : d / 4 * 3);
          t[j] = (pass < 8 && at - at == 0.f) ? min(max((u64)fkey(at), lo + 1), hi - 1) : by_key;
        }
        t[1] = max(t[1], t[0]);
        t[2] = max(t[2], t[1]);
        u64 v[5] = {0, 0, 0, 0, 0};
        const uint32_t t1 = (uint32_t)t[0], t2 = (uint32_t)t[1], t3 = (uint32_t)t[2];
        if (by_mass) {
          scan([&](float x) {
            const uint32_t q = fkey(x);
            if (q < t1) return;
            const u64 w = weight_at(x);
            v[0] += q >= t2 ? 0x100000001ull : 1ull;
            v[2] += w;
            if (q >= t2) v[3] += w;
            if (q >= t3) { v[1] += 1; v[4] += w; }
          });
        } else {
          uint32_t c1 = 0, c2 = 0, c3 = 0;
          scan([&](float x) {
            const uint32_t q = fkey(x);
            c1 += q >= t1;
            c2 += q >= t2;
            c3 += q >= t3;
          });
          v[0] = c1 | (u64)c2 << 32;
          v[1] = c3;
        }
        cluster_sum(v);
        const u64 c[3] = {v[0] & 0xffffffffull, v[0] >> 32, v[1]}, m[3] = {v[2], v[3], v[4]};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if ((by_mass ? m[j] : c[j]) >= goal) {
            lo = t[j];
            c_lo = c[j];
          } else {
            hi = t[j];
            c_hi = c[j];
            m_hi = m[j];
            break;
          }
        }
      }
      if (hi - lo <= 1) return lo;
      // few tokens left: block 0 decides
      scan([&](float x) {
        const uint32_t q = fkey(x);
        if (q != 0 && q >= lo && (u64)q < hi) list_token(q);
      });
      voc_sync<NC>();
      return max((u64)decide(by_mass, goal, c_hi, m_hi, false), lo);
    };
    // ---- bins
    // Tokens further below the maximum than 22.2 T weigh nothing and, without a top_k that counts them too, need no bins.  Cold rows' nucleus ends far above that, so
    // they have bins for 10 T only, which spares most of the counting (where it does end below, the keys are searched).  us before the bins | bins for 16
    // at least | now, top_p 0.8 at temperature 0.1: 64 rows of 32768 18.3 | 21.1 | 17.4, 128 of 16384 16.8 | 20.4 | 16.6, 64 of 12000 15.2 | 18.6 | 15.7, 32 of
    // 128256 28 | 26 | 21; top_p 0.9 at 0.3: 18.6 | 21.1 | 19.4, 17.8 | 20.4 | 19.1, 15.4 | 18.6 | 16.7, 28 | 26 | 25.  (At 0.5, 32 of 128256 39 | 27; with 10 T 36.)
    const bool cold = !use_k && temp < 0.45f;
    const float width = use_k ? fmaxf(16.f, 22.5f * temp) : cold ? 10.f * temp : 22.5f * temp;
    const float scale = (float)kBins / width, shift = (width - mx) * scale;
    auto bin_of = [&](float x) { return (int)min(__float2uint_rz(fmaf(x, scale, shift)), (unsigned)kBins - 1); };  // (0, not counted: NaN and what weighs nothing)
    // (the second bound keeps a bin's edge within 1.1 bins of where it should be; below it lies -inf too, and no maximum is a NaN)
    const bool binned = fabsf(mx) * scale < 8388608.f;
    u64 total = 0;
    uint32_t tokens = 0, above[8], c_next = 0;  // tokens in the bins; those in this thread's eight bins and everything above each; above all eight
    float above_m[8], m_next = 0.f;  // and an estimate of their mass
    if (binned) {
      for (int e = tid * 4; e < kBins; e += kVocThreads * 4) *reinterpret_cast<uint4*>(sh.hist + e) = make_uint4(0, 0, 0, 0);
      sh.heavy[tid] = 0;
      __syncthreads();
      u64 m = 0;
      const bool weigh = use_p && !use_k;
      if (cold) {  // (all that weighs something counts in the total)
        const float lowest = mx - 22.5f * temp;
        scan([&](float x) {
          if (!(x >= lowest)) return;
          const u64 w = weight_at(x);
          m += w;
          const int at = bin_of(x);
          if (at == 0) return;
          atomicAdd(&sh.hist[at], 1u);
          if (at >= kBins - kHeavy) atomicAdd(&sh.heavy[at - (kBins - kHeavy)], (uint32_t)(w >> 12));
        });
      } else if (weigh) {
        scan([&](float x) {
          const int at = bin_of(x);
          if (at == 0) return;
          atomicAdd(&sh.hist[at], 1u);
          const u64 w = weight_at(x);
          m += w;
          if (at >= kBins - kHeavy) atomicAdd(&sh.heavy[at - (kBins - kHeavy)], (uint32_t)(w >> 12));
        });
      } else {
        scan([&](float x) {
          const int at = bin_of(x);
          if (at > 0) atomicAdd(&sh.hist[at], 1u);
        });
      }
      total = cluster_add(m);
      if constexpr (NC > 1) {  // block r adds up the r-th part of the bins and hands it to everybody
        for (int e = rank * (kBins / NC) + tid; e < (int)(rank + 1) * (kBins / NC); e += kVocThreads) {
          uint32_t c = 0;
#pragma unroll
          for (int r = 0; r < NC; ++r) c += cluster_ptr<NC>(sh.hist, r)[e];
#pragma unroll
          for (int r = 0; r < NC; ++r) cluster_ptr<NC>(sh.hist, r)[e] = c;
        }
      }
      if (weigh && tid < kHeavy / NC) {
        const int e = rank * (kHeavy / NC) + tid;
        float hm = 0.f;
#pragma unroll
        for (int r = 0; r < NC; ++r) hm += (float)cluster_ptr<NC>(sh.heavy, r)[e];
#pragma unroll
        for (int r = 0; r < NC; ++r) cluster_ptr<NC>(sh.heavy, r)[e] = __float_as_uint(hm * 4096.f);
      }
      voc_sync<NC>();
      static_assert(kBins == 8 * kVocThreads && kHeavy == kVocThreads, "eight bins per thread");
      const bool heavy = tid >= (kBins - kHeavy) / 8;  // (whole warps)
      uint32_t h[8], c = 0;
      float sm = 0.f;
      *reinterpret_cast<uint4*>(h) = *reinterpret_cast<const uint4*>(sh.hist + tid * 8);
      *reinterpret_cast<uint4*>(h + 4) = *reinterpret_cast<const uint4*>(sh.hist + tid * 8 + 4);
#pragma unroll
      for (int e = 7; e >= 0; --e) {
        const int at = tid * 8 + e;
        c += h[e];
        if (heavy && weigh) sm += __uint_as_float(sh.heavy[at - (kBins - kHeavy)]);
        else sm += (float)h[e] * __expf((((float)at + 0.5f) / scale - width) * inv_t) * 4294967296.0f;
        above[e] = c;
        above_m[e] = sm;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t oc = __shfl_down_sync(0xffffffffu, c, o);
        const float om = __shfl_down_sync(0xffffffffu, sm, o);
        if (lane + o < 32) { c += oc; sm += om; }
      }
      if (lane == 0) { sh.warp_c[warp] = c; sh.warp_m[warp] = sm; }
      c_next = __shfl_down_sync(0xffffffffu, c, 1);
      m_next = __shfl_down_sync(0xffffffffu, sm, 1);
      if (lane == 31) { c_next = 0; m_next = 0.f; }
      __syncthreads();
      // the warps above this one; the estimate's bias (values sit anywhere in a bin) goes by what is known: the total, and the heavy bins' share
      uint32_t wc = lane < kVocWarps ? sh.warp_c[lane] : 0;
      const float wm2 = lane < kVocWarps ? sh.warp_m[lane] : 0.f;
      constexpr int kLight = (kBins - kHeavy) / 256;  // warps of the other bins
      float all_heavy = lane >= kLight ? wm2 : 0.f, all_light = lane < kLight ? wm2 : 0.f, later = lane > warp ? wm2 : 0.f;
      uint32_t wc_later = lane > warp ? wc : 0;
      wc_later = __reduce_add_sync(0xffffffffu, wc_later);
      tokens = __reduce_add_sync(0xffffffffu, wc);
      if (!heavy) later = lane > warp && lane < kLight ? wm2 : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        all_heavy += __shfl_xor_sync(0xffffffffu, all_heavy, o);
        all_light += __shfl_xor_sync(0xffffffffu, all_light, o);
        later += __shfl_xor_sync(0xffffffffu, later, o);
      }
      const float bias = weigh && all_light > 0.f ? fmaxf(((float)total - all_heavy) / all_light, 0.f) : 1.f;
      c_next += wc_later;
      m_next += later;
#pragma unroll
      for (int e = 0; e < 8; ++e) { above[e] += c_next; above_m[e] += m_next; }
      if (!heavy) {
#pragma unroll
        for (int e = 0; e < 8; ++e) above_m[e] = fmaf(bias, above_m[e], all_heavy);
        m_next = fmaf(bias, m_next, all_heavy);
      }
    }
    // the bin that reaches `goal` tokens with everything above it -> sh.bin[s], the tokens with or without it -> sh.upto[s]
    auto locate = [&](int s, uint32_t goal, bool with) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t more = e == 7 ? c_next : above[(e + 1) & 7];
        if (above[e] >= goal && more < goal) {
          sh.bin[s] = tid * 8 + e;
          sh.upto[s] = with ? above[e] : more;
        }
      }
    };
    // The bins' answer to `goal`, 0: none.  `both`: the top-k threshold (goal tokens), then top-p's among its survivors.
    auto bracket = [&](bool by_mass, u64 goal, bool both) -> u64 {
      if (tokens == 0 || (!by_mass && goal > tokens)) return 0;
      if (by_mass) {
        if (tid == 0) sh.reach = (float)tokens;
        __syncthreads();
        const float g = (float)goal;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const uint32_t more = e == 7 ? c_next : above[(e + 1) & 7];
          const float more_m = e == 7 ? m_next : above_m[(e + 1) & 7];
          if (above_m[e] >= g && more_m < g) sh.reach = (float)more + (float)(above[e] - more) * ((g - more_m) / (above_m[e] - more_m));
        }
        __syncthreads();
        const float at = sh.reach;
        locate(0, min(tokens, (uint32_t)(at + kReach)), true);
        locate(1, (uint32_t)fmaxf(1.f, at - kReach), false);
      } else {
        locate(0, (uint32_t)goal, true);
        locate(1, both ? 1u : (uint32_t)goal, false);
      }
      __syncthreads();
      const int b_lo = sh.bin[0], b_hi = sh.bin[1];
      const uint32_t c_hi = sh.upto[1];
      const bool many = sh.upto[0] - c_hi > (uint32_t)kFin;
      __syncthreads();  // (the caller may ask again, which writes these four anew)
      if (many) return 0;
      u64 m_hi = 0;
      if (by_mass) {
        scan([&](float x) {
          const int at = bin_of(x);
          if (at < b_lo) return;
          if (at <= b_hi) list_token(fkey(x));
          else m_hi += weight_at(x);
        });
        m_hi = cluster_add(m_hi);
      } else {
        scan([&](float x) {
          const int at = bin_of(x);
          if (at >= b_lo && at <= b_hi) list_token(fkey(x));
        });
        voc_sync<NC>();
      }
      return decide(by_mass, goal, c_hi, m_hi, both);
    };
    u64 lo = 0;
    bool done = false;
    if (use_k) {
      if (binned) {
        lo = bracket(false, (u64)k, use_p);
        done = lo > 0;
        if (lo == 0 && use_p) lo = bracket(false, (u64)k, false);
      }
      if (lo == 0) lo = search(false, (u64)k, 0, (u64)V);
    }
    if (use_p && !done) {
      u64 count = V;
      if (use_k || !binned) {
        u64 v[5] = {0, 0, 0, 0, 0};  // tokens and mass of the top-k survivors (of the whole row without top-k)
        scan([&](float x) {
          if (x == x && fkey(x) >= lo) {
            v[0] += 1;
            v[2] += weight_at(x);
          }
        });
        cluster_sum(v);
        count = v[0];
        total = v[2];
      }
      u64 target = (u64)((double)p * (double)total);
      if (target < 1) target = 1;
      const u64 found = binned ? bracket(true, target, false) : 0;
      lo = found > 0 ? max(found, lo) : search(true, target, lo, count);
    }
    if (lo > 0) floor_logit = fkey_inv((uint32_t)lo);
  }

  if constexpr (SM) {
    if (filters) {
      // Few tokens of a filtered row are drawn for: every warp collects its survivors and draws for 32 at a time
      uint32_t* queue = sh.hist + warp * kQueue;
      int held = 0;
      __syncthreads();  // (the counts are read by every warp)
      for (int i0 = warp * 128; i0 < n; i0 += kVocThreads * 4) {
        const int i = i0 + lane * 4;
        const float none = __int_as_float(0x7fffffff);
        const float4 q4 = i < n ? *reinterpret_cast<const float4*>(slice + i) : make_float4(none, none, none, none);
        const float q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t who = __ballot_sync(0xffffffffu, q[e] >= floor_logit);
          if (q[e] >= floor_logit) queue[held + __popc(who & ((1u << lane) - 1))] = i + e;
          held += __popc(who);
        }
        __syncwarp();
        while (held >= 32) {
          held -= 32;
          const int at = queue[held + lane];
          draw(slice[at], at);
        }
        __syncwarp();
      }
      if (lane < held) {
        const int at = queue[lane];
        draw(slice[at], at);
      }
      __syncwarp();
    }
  } else {
    for (int i = tid; i < n; i += kVocThreads) {
      const float x = __ldg(row + i);
      if (x >= floor_logit) draw(x, i);
    }
    __syncwarp();
  }
  // lowest index wins ties, in whatever order the blocks' winners are merged
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    argmax_merge(best, bi, ov, oi);
  }
  __syncthreads();
  if (lane == 0) { sh.val[warp] = best; sh.idx[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    best = sh.val[lane & (kVocWarps - 1)];
    bi = sh.idx[lane & (kVocWarps - 1)];
#pragma unroll
    for (int o = kVocWarps / 2; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      argmax_merge(best, bi, ov, oi);
    }
    if (lane == 0) {
      cluster_ptr<NC>(sh.top, 0)[rank] = best;
      cluster_ptr<NC>(sh.top_idx, 0)[rank] = bi;
    }
  }
  voc_sync<NC>();
  if (rank == 0 && tid == 0) {
    for (int c = 1; c < NC; ++c) argmax_merge(best, bi, sh.top[c], sh.top_idx[c]);
    out[b] = bi < 0x7fffffff ? bi : 0;  // all-NaN row: emit a valid id, never an out-of-range one
  }
}

// The same for short rows, a block each, whose search by masses and counts of the keys ends within a few passes that cost next to nothing
// (us there | with clusters' bins, 128 rows of 8192: top_k 40 15 | 17, top_p 0.5 17 | 19): a pass compares the row with three keys inside the
// interval that still holds the answer, or sorts it into 128 bins of masses; the last 256 tokens are ranked directly.
constexpr int kRowFin = 256, kRowBins = 128;
struct SampleRowShared {
  uint32_t hist[2][3][kRowBins];  // tokens per value bin, the low 16 bits of their masses, the rest
  unsigned long long tot_c[kRowBins], tot_m[kRowBins];
  unsigned long long part[2][5];  // totals of a pass: counts (c1 | c2 << 32), c3, masses m1 .. m3
  unsigned long long wred[kVocWarps][5];
  uint32_t list[kRowFin];
  unsigned long long mass[kRowFin];
  float val[kVocWarps];
  int idx[kVocWarps];
  uint32_t n_list, result;
};

__global__ void __launch_bounds__(kVocThreads)
sample_row_kernel(const float* __restrict__ logits, int ldl, const float* __restrict__ temperature, const uint64_t* __restrict__ seed,
              const int32_t* __restrict__ top_k, const float* __restrict__ top_p, int32_t* __restrict__ out, int V) {
  extern __shared__ __align__(16) uint32_t keys[];
  __shared__ SampleRowShared sh;
  pdl_launch_dependents();
  pdl_wait();
  typedef unsigned long long u64;
  const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* row = logits + (size_t)b * ldl;
  const float temp = temperature ? temperature[b] : 0.f;
  const bool greedy = !(temp > 0.f);
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const int k = top_k ? top_k[b] : 0;
  const float p = top_p ? top_p[b] : 1.f;
  const bool use_k = !greedy && k > 0 && k < V, use_p = !greedy && p > 0.f && p < 1.f;

  if (tid == 0) sh.n_list = 0;
  float mx = -INFINITY;
  load_slice(row, V, tid, [&](int i, const float (&f)[4], int have) {  // (entries behind the row's end read as key 0, below every float's key)
    uint32_t q[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      mx = fmaxf(mx, e < have ? f[e] : -INFINITY);
      q[e] = e < have ? fkey(f[e]) : 0u;
    }
    *reinterpret_cast<uint4*>(keys + i) = make_uint4(q[0], q[1], q[2], q[3]);
  });
  __syncthreads();
  auto scan = [&](auto&& f) {  // f(key, column)
    for (int i = tid * 4; i < V; i += kVocThreads * 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(keys + i);
      f(q.x, i);
      f(q.y, i + 1);
      f(q.z, i + 2);
      f(q.w, i + 3);
    }
  };

  float floor_logit = -INFINITY;
  if (use_k || use_p) {
    // row maximum (for the softmax weights)
    const uint32_t wm = __reduce_max_sync(0xffffffffu, fkey(mx));
    if (lane == 0) sh.val[warp] = fkey_inv(wm);
    __syncthreads();
    mx = sh.val[lane & (kVocWarps - 1)];
    mx = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(mx)));
    auto weight = [&](uint32_t key) -> u64 {
      const float e = __expf((fkey_inv(key) - mx) * inv_t) * 4294967296.0f;
      return e >= 0.f ? (u64)e : 0;  // a NaN logit carries no mass
    };
    int turn = 0;
    // sums of the block's threads, in every thread
    auto warp_total = [](u64 v) -> u64 {  // (a thread's share is below 2^58: three limbs, one hardware reduction each)
      const u64 a = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0xffffu), c = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 16) & 0x1fffffu),
                d = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 37));
      return a + (c << 16) + (d << 37);
    };
    auto block_sum5 = [&](u64 (&v)[5]) {
#pragma unroll
      for (int j = 0; j < 5; ++j) {
        const u64 t = j == 0 ? (u64)__reduce_add_sync(0xffffffffu, (uint32_t)v[0]) | (u64)__reduce_add_sync(0xffffffffu, (uint32_t)(v[0] >> 32)) << 32
                      : j == 1 ? (u64)__reduce_add_sync(0xffffffffu, (uint32_t)v[1]) : warp_total(v[j]);
        if (lane == 0) sh.wred[warp][j] = t;
      }
      __syncthreads();
      if (warp == 0) {
#pragma unroll
        for (int j = 0; j < 5; ++j) {
          u64 t = lane < kVocWarps ? sh.wred[lane][j] : 0;
#pragma unroll
          for (int o = kVocWarps / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          if (lane == 0) sh.part[turn][j] = t;
        }
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 5; ++j) v[j] = sh.part[turn][j];
      turn ^= 1;  // (a slot is written again two passes later, behind the barrier that follows every read of it)
    };
    // the largest key whose tokens (those with keys >= it) reach `goal`: in number, or in mass (by_mass).  Keeping [lo, ..) is
    // enough (c_lo tokens), keeping [hi, ..) is not (c_hi tokens of mass m_hi).
    auto search = [&](bool by_mass, u64 goal, u64 lo, u64 c_lo) -> u64 {
      u64 hi = (u64)fkey(mx) + 1, c_hi = 0, m_hi = 0;  // (nothing is above the maximum)
      for (int pass = 0; hi - lo > 1 && c_lo - c_hi > (u64)kRowFin; ++pass) {
        // Logits are spread more evenly over values than over keys (where half of all keys are exponents nothing has): the first
        // pass looks a few temperatures below the maximum, the next ones divide the values between the bounds; from the eighth
        // on the keys are divided, so at most 8 + 16 passes are needed.
        const u64 d = hi - lo;
        // A mass between two finite values: the tokens go into kRowBins equal bins of values at once, and the bin that holds the answer is
        // the next interval (a threshold in the bulk of the vocabulary needs two such passes instead of five or six of three keys,
        // which weigh nearly as many tokens each: rows of top_p 0.95 85 -> 70 us; counting is cheap, so top-k stays with the keys).
        // Intervals that no longer split take the keys below.
        {
          const float b_lo = fkey_inv((uint32_t)lo), b_hi = fkey_inv((uint32_t)(hi - 1)), scale = (float)kRowBins / (b_hi - b_lo);
          if (by_mass && pass > 0 && pass < 8 && lo > 0 && scale > 0.f && scale < 1e30f && b_lo - b_lo == 0.f) {
            auto bin_of = [&](uint32_t q) { return min(kRowBins - 1, (int)((fkey_inv(q) - b_lo) * scale)); };
            uint32_t (&hist)[3][kRowBins] = sh.hist[turn];
            for (int e = tid; e < 3 * kRowBins; e += kVocThreads) (&hist[0][0])[e] = 0;
            __syncthreads();
            scan([&](uint32_t q, int) {
              if (q < (uint32_t)lo || (u64)q >= hi) return;
              const int at = bin_of(q);
              atomicAdd(&hist[0][at], 1u);
              const u64 w = weight(q);
              atomicAdd(&hist[1][at], (uint32_t)w & 0xffffu);
              atomicAdd(&hist[2][at], (uint32_t)(w >> 16));
            });
            __syncthreads();
            for (int e = tid; e < kRowBins; e += kVocThreads) {
              sh.tot_c[e] = hist[0][e];
              sh.tot_m[e] = hist[1][e] + ((u64)hist[2][e] << 16);
            }
            __syncthreads();
            turn ^= 1;  // (zeroed again two passes later, behind the barrier that follows every read of it)
            u64 c4[4], m4[4], c_up = 0, m_up = 0;  // a lane's four bins, then everything above them
#pragma unroll
            for (int e = 3; e >= 0; --e) {
              c4[e] = c_up += sh.tot_c[lane * 4 + e];
              m4[e] = m_up += sh.tot_m[lane * 4 + e];
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const u64 c = __shfl_down_sync(0xffffffffu, c_up, o), m = __shfl_down_sync(0xffffffffu, m_up, o);
              if (lane + o < 32) { c_up += c; m_up += m; }
            }
            u64 c_above = __shfl_down_sync(0xffffffffu, c_up, 1), m_above = __shfl_down_sync(0xffffffffu, m_up, 1);
            if (lane == 31) c_above = m_above = 0;
            c_above += c_hi;
            m_above += m_hi;
            int best = -1;  // the highest bin that reaches the goal together with everything above it
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (m4[e] + m_above >= goal) best = lane * 4 + e;
            best = __reduce_max_sync(0xffffffffu, best);
            if (best >= 0) {
              const int src = best >> 2, e = best & 3;
              const u64 c_in = __shfl_sync(0xffffffffu, (e == 0 ? c4[0] : e == 1 ? c4[1] : e == 2 ? c4[2] : c4[3]) + c_above, src);
              const u64 c_out = __shfl_sync(0xffffffffu, (e == 0 ? c4[1] : e == 1 ? c4[2] : e == 2 ? c4[3] : 0ull) + c_above, src);
              const u64 m_out = __shfl_sync(0xffffffffu, (e == 0 ? m4[1] : e == 1 ? m4[2] : e == 2 ? m4[3] : 0ull) + m_above, src);
              auto first_in = [&](int bin) {  // the smallest key of the interval whose bin is at least this one (hi: none)
                u64 a = lo, z = hi;
                while (a < z) {
                  const u64 mid = (a + z) >> 1;
                  if (bin_of((uint32_t)mid) >= bin) z = mid; else a = mid + 1;
                }
                return a;
              };
              const u64 n_lo = best == 0 ? lo : first_in(best), n_hi = best == kRowBins - 1 ? hi : first_in(best + 1);
              if (n_lo > lo || n_hi < hi) {
                lo = n_lo;
                c_lo = c_in;
                hi = n_hi;
                c_hi = c_out;
                m_hi = m_out;
                continue;
              }
            }
          }
        }
        u64 t[3];
        const float flo = fkey_inv((uint32_t)lo), fhi = fkey_inv((uint32_t)(hi - 1));
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const float at = pass == 0 ? mx - temp * (j == 0 ? 16.f : j == 1 ? 8.f : 4.f) : flo + (fhi - flo) * (0.25f * (j + 1));
          const u64 by_key = lo + max(1ull, j == 0 ? d / 4 : j == 1 ? d / 2 : d / 4 * 3);
          t[j] = (pass < 8 && at - at == 0.f) ? min(max((u64)fkey(at), lo + 1), hi - 1) : by_key;
        }
        t[1] = max(t[1], t[0]);
        t[2] = max(t[2], t[1]);
        u64 v[5] = {0, 0, 0, 0, 0};
        const uint32_t t1 = (uint32_t)t[0], t2 = (uint32_t)t[1], t3 = (uint32_t)t[2];
        if (by_mass) {
          scan([&](uint32_t q, int) {
            if (q < t1) return;
            const u64 w = weight(q);
            v[0] += q >= t2 ? 0x100000001ull : 1ull;
            v[2] += w;
            if (q >= t2) v[3] += w;
            if (q >= t3) { v[1] += 1; v[4] += w; }
          });
        } else {
          uint32_t c1 = 0, c2 = 0, c3 = 0;
          scan([&](uint32_t q, int) {
            c1 += q >= t1;
            c2 += q >= t2;
            c3 += q >= t3;
          });
          v[0] = c1 | (u64)c2 << 32;
          v[1] = c3;
        }
        block_sum5(v);
        const u64 c[3] = {v[0] & 0xffffffffull, v[0] >> 32, v[1]}, m[3] = {v[2], v[3], v[4]};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          if ((by_mass ? m[j] : c[j]) >= goal) {
            lo = t[j];
            c_lo = c[j];
          } else {
            hi = t[j];
            c_hi = c[j];
            m_hi = m[j];
            break;
          }
        }
      }
      if (hi - lo <= 1) return lo;
      // few tokens left
      scan([&](uint32_t q, int) {
        if (q < lo || (u64)q >= hi || q == 0) return;
        sh.list[atomicAdd(&sh.n_list, 1u)] = q;
      });
      __syncthreads();
      const int nl = (int)sh.n_list;
      for (int i = tid; i < nl; i += kVocThreads) sh.mass[i] = weight(sh.list[i]);
      __syncthreads();
      const int cand = tid >> 1;
      const uint32_t key = cand < nl ? sh.list[cand] : 0u;
      u64 c = 0, m = 0;
      for (int j = tid & 1; j < nl; j += 2)
        if (sh.list[j] >= key) {
          c += 1;
          m += sh.mass[j];
        }
      c += __shfl_xor_sync(0xffffffffu, c, 1);
      m += __shfl_xor_sync(0xffffffffu, m, 1);
      const bool ok = cand < nl && (by_mass ? m_hi + m : c_hi + c) >= goal;
      const uint32_t wk = __reduce_max_sync(0xffffffffu, ok ? key : 0u);
      if (lane == 0) sh.idx[warp] = (int)wk;
      __syncthreads();
      if (warp == 0) {
        const uint32_t r = __reduce_max_sync(0xffffffffu, (uint32_t)sh.idx[lane & (kVocWarps - 1)]);
        if (lane == 0) {
          sh.result = r;
          sh.n_list = 0;
        }
      }
      __syncthreads();
      return sh.result > lo ? sh.result : lo;
    };
    u64 lo = 0;
    if (use_k) lo = search(false, (u64)k, 0, (u64)V);
    if (use_p) {
      u64 v[5] = {0, 0, 0, 0, 0};  // tokens and mass of the top-k survivors (of the whole row without top-k)
      scan([&](uint32_t q, int i) {
        if (i < V && q >= lo) {
          v[0] += 1;
          v[2] += weight(q);
        }
      });
      block_sum5(v);
      u64 target = (u64)((double)p * (double)v[2]);
      if (target < 1) target = 1;
      lo = search(true, target, lo, v[0]);
    }
    if (lo > 0) floor_logit = fkey_inv((uint32_t)lo);
  }

  float best = -INFINITY;
  int bi = 0x7fffffff;
  const uint64_t sd = seed ? seed[b] : 0;
  scan([&](uint32_t q, int i) {
    if (i >= V) return;
    if (q == 0) return;  // a NaN is never drawn
    const float raw = fkey_inv(q);
    if (raw < floor_logit) return;
    float x = raw * inv_t;
    if (!greedy) x += gumbel(sd, i);
    argmax_merge(best, bi, x, i);
  });
  // lowest index wins ties, in whatever order the blocks' winners are merged
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    argmax_merge(best, bi, ov, oi);
  }
  __syncthreads();
  if (lane == 0) { sh.val[warp] = best; sh.idx[warp] = bi; }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kVocWarps; ++w) argmax_merge(best, bi, sh.val[w], sh.idx[w]);
    out[b] = bi < 0x7fffffff ? bi : 0;  // all-NaN row: emit a valid id, never an out-of-range one
  }
}

// ---- OpenAI presence / frequency penalties: logits[b, tok] -= val for the (tok, val) entries of row b ----
// entries [pen_off[b], pen_off[b+1]) hold the DISTINCT tokens the sequence has generated so far with
// val = presence + frequency * count (computed on the host from the request's exact integer counts)
__global__ void __launch_bounds__(256)
apply_penalties_kernel(float* __restrict__ logits, int ldl, const int32_t* __restrict__ pen_off,
                       const int2* __restrict__ pen, int V) {
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x;
  float* row = logits + (size_t)b * ldl;
  for (int i = pen_off[b] + threadIdx.x; i < pen_off[b + 1]; i += 256) {
    const int2 e = pen[i];
    if (e.x >= 0 && e.x < V) row[e.x] -= __int_as_float(e.y);  // distinct tokens: no two threads touch the same logit
  }
}

// ---- log-probabilities of the sampled token and of the width-1 most likely tokens (descending, lowest id on ties) ----
// One block per row that reads it twice and once more per further pick: for narrow records (logprob_topk below).
constexpr int kLpThreads = 1024;
__global__ void __launch_bounds__(kLpThreads)
logprob_row_kernel(const float* __restrict__ logits, int ldl, int V, const int32_t* __restrict__ sampled,
                    const int32_t* __restrict__ width, int32_t* __restrict__ out_ids, float* __restrict__ out_lp,
                    int max_width) {
  __shared__ float sval[kLpThreads / 32];
  __shared__ int sidx[kLpThreads / 32];
  __shared__ float red[kLpThreads / 32];
  __shared__ float s_bv;
  __shared__ int s_bi;
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x;
  const int w = min(width[b], max_width);
  if (w <= 0) return;
  const float* row = logits + (size_t)b * ldl;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int v = threadIdx.x; v < V; v += kLpThreads) argmax_merge(best, bi, row[v], v);
  block_argmax<kLpThreads>(best, bi, sval, sidx);
  if (threadIdx.x == 0) { s_bv = best; s_bi = bi; }
  __syncthreads();
  const float mx = s_bv;
  float se = 0.f;
  for (int v = threadIdx.x; v < V; v += kLpThreads) se += expf(row[v] - mx);
  se = block_sum<kLpThreads>(se, red);
  const float lse = mx + logf(se);
  int32_t* ids = out_ids + (size_t)b * max_width;
  float* lps = out_lp + (size_t)b * max_width;
  if (threadIdx.x == 0) {
    const int t = sampled[b];
    ids[0] = t;
    lps[0] = (t >= 0 && t < V) ? row[t] - lse : -INFINITY;
  }
  float pv = s_bv;   // the j-th most likely token in the order (value desc, id asc); j = 1 is the argmax found above
  int pi = s_bi;
  for (int j = 1; j < w; ++j) {
    if (threadIdx.x == 0) { ids[j] = pi; lps[j] = pv - lse; }
    if (j + 1 == w) break;
    best = -INFINITY;
    bi = 0x7fffffff;
    for (int v = threadIdx.x; v < V; v += kLpThreads) {
      const float x = row[v];
      if (x < pv || (x == pv && v > pi)) argmax_merge(best, bi, x, v);  // strictly after the previous pick
    }
    __syncthreads();  // sval/sidx reuse
    block_argmax<kLpThreads>(best, bi, sval, sidx);
    if (threadIdx.x == 0) { s_bv = best; s_bi = bi; }
    __syncthreads();
    pv = s_bv;
    pi = s_bi;
    if (pi == 0x7fffffff) {  // fewer than `w` finite logits in the row
      if (threadIdx.x == 0)
        for (int k = j + 1; k < w; ++k) { ids[k] = -1; lps[k] = -INFINITY; }
      break;
    }
  }
}

// The same, a row shared by NC blocks.
// Every block picks the width-1 best of its part (a thread remembers the best of its own entries; after a round only the entries
// of the thread that owned the winner are looked at again, by its whole warp), block 0 merges the short lists by rank.
// Measured (32 rows x 128256, width 6): 69 us with a block per row that read it once per pick, 16 us now.
constexpr int kLpMax = 32;  // picks per merge; wider records take several
template <int NC>
struct LpShared {
  uint32_t wkey[2][kVocWarps];
  int widx[2][kVocWarps];
  uint32_t top_key[kLpMax];
  int top_idx[kLpMax];
  uint32_t all_key[NC * kLpMax];
  int all_idx[NC * kLpMax];
  float red[kVocWarps];
  float part_max, part_sum;
  uint32_t last_key;
  int last_idx;
};
template <int NC, bool SM>
__global__ void __cluster_dims__(NC, 1, 1) __launch_bounds__(kVocThreads)
logprob_topk_kernel(const float* __restrict__ logits, int ldl, int V, const int32_t* __restrict__ sampled,
                    const int32_t* __restrict__ width, int32_t* __restrict__ out_ids, float* __restrict__ out_lp, int max_width) {
  extern __shared__ __align__(16) float slice[];
  __shared__ LpShared<NC> sh;
  pdl_launch_dependents();
  pdl_wait();
  const int b = blockIdx.x / NC, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int w = min(width[b], max_width);
  if (w <= 0) return;  // (the whole cluster)
  const uint32_t rank = cluster_ctarank();
  const int per = voc_slice(V, NC), start = min(V, (int)rank * per), n = min(V, start + per) - start;
  const float* row = logits + (size_t)b * ldl;
  const float* src = row + start;
  constexpr int kStep = kVocThreads * 4;  // a thread's entries: columns 4 tid .. 4 tid + 3 of every kStep
  float mx = -INFINITY;
  uint32_t bk = 0;  // best of this thread's entries in the order (value descending, index ascending); NaN is never picked, zeros tie
  int bi = 0x7fffffff;
  auto as_key = [](float x) -> uint32_t {
    const float y = x + 0.f;
    return y == y ? fkey(y) : 0u;
  };
  load_slice(src, n, tid, [&](int i, const float (&f)[4], int have) {
    float4 v = make_float4(f[0], have > 1 ? f[1] : -INFINITY, have > 2 ? f[2] : -INFINITY, have > 3 ? f[3] : -INFINITY);
    if (SM) *reinterpret_cast<float4*>(slice + i) = v;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e >= have) break;
      mx = fmaxf(mx, f[e]);
      const uint32_t q = as_key(f[e]);
      if (q > bk) { bk = q; bi = start + i + e; }
    }
  });
  // the best entry of thread t0 behind (key, index), found by its whole warp
  auto next_best = [&](int t0, uint32_t after_key, int after_idx, uint32_t& k_out, int& i_out) {
    uint32_t k1 = 0;
    int i1 = 0x7fffffff;
    for (int i = t0 * 4 + (lane & 3) + (lane >> 2) * kStep; i < n; i += 8 * kStep) {
      const uint32_t q = as_key(SM ? slice[i] : __ldg(src + i));
      if (q > after_key || (q == after_key && start + i <= after_idx)) continue;
      if (q > k1) { k1 = q; i1 = start + i; }
    }
    __syncwarp();
    k_out = __reduce_max_sync(0xffffffffu, k1);
    i_out = __reduce_min_sync(0xffffffffu, k1 == k_out ? i1 : 0x7fffffff);
  };
  auto block_max = [&](float v) {
    v = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(v)));
    if (lane == 0) sh.red[warp] = v;
    __syncthreads();
    return fkey_inv(__reduce_max_sync(0xffffffffu, fkey(sh.red[lane & (kVocWarps - 1)])));
  };
  mx = block_max(mx);
  if (tid == 0) sh.part_max = mx;
  voc_sync<NC>();
  mx = fkey_inv(__reduce_max_sync(0xffffffffu, fkey(*cluster_ptr<NC>(&sh.part_max, lane & (NC - 1)))));
  float se = 0.f;
  if constexpr (SM) {
#pragma unroll 4
    for (int i = tid * 4; i < n; i += kStep) {
      const float4 v = *reinterpret_cast<const float4*>(slice + i);
      se += (expf(v.x - mx) + expf(v.y - mx)) + (expf(v.z - mx) + expf(v.w - mx));
    }
  } else {
    for (int i0 = tid * 4; i0 < n; i0 += kStep)
      for (int i = i0; i < min(n, i0 + 4); ++i) se += expf(__ldg(src + i) - mx);
  }
  se = warp_sum(se);
  if (lane == 0) sh.red[warp] = se;
  __syncthreads();
  if (warp == 0) {
    se = warp_sum(lane < kVocWarps ? sh.red[lane] : 0.f);
    if (lane == 0) sh.part_sum = se;
  }
  voc_sync<NC>();
  float sum = 0.f;
  for (int c = 0; c < NC; ++c) sum += *cluster_ptr<NC>(&sh.part_sum, c);
  const float lse = mx + logf(sum);
  int32_t* ids = out_ids + (size_t)b * max_width;
  float* lps = out_lp + (size_t)b * max_width;
  if (rank == 0 && tid == 0) {
    const int t = sampled[b];
    ids[0] = t;
    lps[0] = (t >= 0 && t < V) ? row[t] - lse : -INFINITY;
  }
  for (int base = 0; base < w - 1; base += kLpMax) {
    const int picks = min(w - 1 - base, kLpMax);
    if (base > 0) {  // (a thread's own best may have been picked or lie behind the last pick: look again)
      for (int l = 0; l < 32; ++l) {
        uint32_t k1;
        int i1;
        next_best(warp * 32 + l, sh.last_key, sh.last_idx, k1, i1);
        if (lane == l) { bk = k1; bi = i1; }
      }
    }
    for (int r = 0; r < picks; ++r) {
      const uint32_t wk = __reduce_max_sync(0xffffffffu, bk);
      const int wi = __reduce_min_sync(0xffffffffu, bk == wk ? bi : 0x7fffffff);
      if (lane == 0) { sh.wkey[r & 1][warp] = wk; sh.widx[r & 1][warp] = wi; }
      __syncthreads();
      const uint32_t ck = sh.wkey[r & 1][lane & (kVocWarps - 1)];
      const int ci = sh.widx[r & 1][lane & (kVocWarps - 1)];
      const uint32_t gk = __reduce_max_sync(0xffffffffu, ck);
      const int gi = __reduce_min_sync(0xffffffffu, ck == gk ? ci : 0x7fffffff);
      if (tid == 0) { sh.top_key[r] = gk; sh.top_idx[r] = gi; }
      const uint32_t mine = __ballot_sync(0xffffffffu, bi == gi && gi != 0x7fffffff);
      if (mine) {
        uint32_t k1;
        int i1;
        next_best(warp * 32 + __ffs(mine) - 1, gk, gi, k1, i1);
        if (mine >> lane & 1) { bk = k1; bi = i1; }
      }
    }
    voc_sync<NC>();
    if (rank == 0) {
      const int all = NC * picks;
      for (int e = tid; e < all; e += kVocThreads) {
        sh.all_key[e] = cluster_ptr<NC>(sh.top_key, e / picks)[e % picks];
        sh.all_idx[e] = cluster_ptr<NC>(sh.top_idx, e / picks)[e % picks];
      }
      __syncthreads();
      for (int e = tid; e < all; e += kVocThreads) {
        const uint32_t q = sh.all_key[e];
        const int i = sh.all_idx[e];
        int better = 0;
        for (int j = 0; j < all; ++j) {
          const uint32_t oq = sh.all_key[j];
          const int oi = sh.all_idx[j];
          better += oq > q || (oq == q && (oi < i || (oi == i && j < e)));
        }
        if (better < picks) {
          const int at = base + better;
          const bool none = i == 0x7fffffff;  // fewer than `w` tokens to name
          ids[1 + at] = none && at > 0 ? -1 : i;
          lps[1 + at] = none ? (at > 0 ? -INFINITY : mx - lse) : fkey_inv(q) - lse;
        }
        if (better == picks - 1)
          for (int c = 0; c < NC; ++c) {
            *cluster_ptr<NC>(&sh.last_key, c) = q;
            *cluster_ptr<NC>(&sh.last_idx, c) = i;
          }
      }
    }
    voc_sync<NC>();
  }
  voc_sync<NC>();  // no block's shared memory goes away while another one reads it
}

__global__ void __launch_bounds__(kRowThreads)
cls_pool_l2_kernel(const bf16* __restrict__ x, const int32_t* __restrict__ first_row, float* __restrict__ out, int H) {
  __shared__ float red[kRowThreads / 32];
  const int b = blockIdx.x;
  const bf16* row = x + (size_t)first_row[b] * H;
  float ss = 0.f;
  for (int i = threadIdx.x; i < H; i += kRowThreads) {
    const float v = __bfloat162float(row[i]);
    ss += v * v;
  }
  ss = block_sum<kRowThreads>(ss, red);
  const float inv = 1.0f / fmaxf(sqrtf(ss), 1e-12f);
  for (int i = threadIdx.x; i < H; i += kRowThreads) out[(size_t)b * H + i] = __bfloat162float(row[i]) * inv;
}

}  // namespace

cudaError_t embed_gather(cudaStream_t s, const int32_t* tokens, const bf16* table, bf16* x, int T, int H) {
  if (T <= 0) return cudaSuccess;
  if (H % 8) return cudaErrorInvalidValue;
  return launch_k(embed_gather_kernel, dim3(T), dim3(128), 0, s, true, tokens, table, x, H);
}
cudaError_t rmsnorm(cudaStream_t s, const bf16* x, const bf16* w, bf16* out, const int32_t* row_index, int rows, int H,
                    float eps) {
  if (rows <= 0) return cudaSuccess;
  if (H % 8) return cudaErrorInvalidValue;
  return launch_k(rmsnorm_kernel, dim3(rows), dim3(kRowThreads), 0, s, true, x, w, out, row_index, H, eps);
}
cudaError_t layernorm(cudaStream_t s, const bf16* x, const bf16* gamma, const bf16* beta, bf16* out, int rows, int H,
                      float eps) {
  if (rows <= 0) return cudaSuccess;
  if (H % 8 || H > kMaxVec * kRowThreads * 8) return cudaErrorInvalidValue;
  if (H <= 1024)
    return launch_k(layernorm_warp_kernel<false>, dim3((rows + 3) / 4), dim3(128), 0, s, true, x, gamma, beta, out, rows, H, eps, nullptr, nullptr, nullptr, nullptr,
                    nullptr);
  else
    layernorm_kernel<false><<<rows, kRowThreads, 0, s>>>(x, gamma, beta, out, H, eps, nullptr, nullptr, nullptr, nullptr, nullptr);
  return cudaGetLastError();
}
cudaError_t bert_embed_ln(cudaStream_t s, const int32_t* tokens, const int32_t* positions, const bf16* word,
                          const bf16* pos, const bf16* type0, const bf16* gamma, const bf16* beta, bf16* x, int T, int H,
                          float eps) {
  if (T <= 0) return cudaSuccess;
  if (H % 8 || H > kMaxVec * kRowThreads * 8) return cudaErrorInvalidValue;
  if (H <= 1024)
    return launch_k(layernorm_warp_kernel<true>, dim3((T + 3) / 4), dim3(128), 0, s, true, nullptr, gamma, beta, x, T, H, eps, tokens, positions, word, pos, type0);
  else
    layernorm_kernel<true><<<T, kRowThreads, 0, s>>>(nullptr, gamma, beta, x, H, eps, tokens, positions, word, pos, type0);
  return cudaGetLastError();
}
cudaError_t rope_table(cudaStream_t s, const int32_t* positions, const float* inv_freq, float* cs, int T, int D) {
  if (T <= 0) return cudaSuccess;
  const int n = T * (D / 2);
  rope_table_kernel<<<(n + 255) / 256, 256, 0, s>>>(positions, inv_freq, cs, T, D);
  return cudaGetLastError();
}

cudaError_t rope_kv_write(cudaStream_t s, bf16* qkv, const int32_t* positions, const int32_t* slot_mapping,
                          const float* inv_freq, bf16* k_cache, bf16* v_cache, int T, int Hq, int Hkv, int D,
                          int page_size) {
  if (T <= 0) return cudaSuccess;
  if (D % 8) return cudaErrorInvalidValue;
  rope_kv_write_kernel<<<T, 256, D * sizeof(float), s>>>(qkv, positions, slot_mapping, inv_freq, k_cache, v_cache, Hq,
                                                         Hkv, D, page_size);
  return cudaGetLastError();
}
namespace {
// Dynamic shared memory of the vocabulary kernels: a part of the row when it fits, nothing otherwise.  The opt-in is per device and
// costs well under a microsecond, so it rides with every launch: callers need no initialisation call.
template <typename K, typename... Args>
cudaError_t launch_voc(K* kernel, int ctas, bool on_chip, cudaStream_t s, int B, int V, Args... args) {
  if (on_chip) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kVocSmemFloats * 4);
    if (e != cudaSuccess) return e;
  }
  return launch_k(kernel, dim3(B * ctas), dim3(kVocThreads), on_chip ? (size_t)voc_slice(V, ctas) * 4 : 0, s, true, args...);
}
// Blocks per row: one up to `whole` columns; else as many (at most `most`) as let the machine hold every row's blocks at once (33
// clusters of eight), but enough that two blocks fit an SM (parts of `part` columns).  Every shape gives the same tokens.  Us with 1 / 2 / 4 / 8 blocks per row:
//   top_p 0.95   48 rows of 32768  33 / 28 / 25 / 38     128 of 16384  27 / 24 / 39 / 71     16 of 12000     17 / 18 / 18 / 18
//                32 rows of 128256  - /  - / 38 / 35      96 of 65536   - / 66 / 55 / 71      256 of 128256  - /  - / 281 / 242
//   width 6      48 rows of 50000   - / 14 / 13 / 25     128 of 32768  12 / 13 / 24 / 47     256 of 8192   8.5 / 18 / 38 / 87
// (clusters of eight run 33 at a time whatever their size, which left 256 rows of 1000 to 8192 columns at 20 to 50 % of the speed
// of the block per row that these kernels had replaced).
int voc_ctas(int B, int V, int whole, int most, int part) {
  if (V <= whole) return 1;
  int ctas = most;
  while (ctas > 1 && (long)B * ctas > 264) ctas /= 2;
  while (ctas < 8 && voc_slice(V, ctas) > part) ctas *= 2;
  return ctas;
}
#define HB_VOC(KERNEL, CTAS, ...)                                                             \
  do {                                                                                        \
    const int ctas = (CTAS);                                                                  \
    if (voc_slice(V, ctas) > kVocSmemFloats) return launch_voc(KERNEL<8, false>, 8, false, s, B, V, __VA_ARGS__); \
    if (ctas == 1) return launch_voc(KERNEL<1, true>, 1, true, s, B, V, __VA_ARGS__);         \
    if (ctas == 2) return launch_voc(KERNEL<2, true>, 2, true, s, B, V, __VA_ARGS__);         \
    if (ctas == 4) return launch_voc(KERNEL<4, true>, 4, true, s, B, V, __VA_ARGS__);         \
    return launch_voc(KERNEL<8, true>, 8, true, s, B, V, __VA_ARGS__);                        \
  } while (0)
}  // namespace
// Rows without filters are looked at once, so nothing is gained by keeping them on chip: two launches over chunks of the row, with room
// for the chunks' winners, unless the clusters of few short rows are through sooner.  Us, clusters | two launches: 32 rows of
// 32768, temperature 8.6 | 9.7, 64 rows of 32768 15.8 | 12.4, greedy 10.8 | 7.3, 256 rows of 8192 34 | 12.5, greedy 28 | 7.2, 1 row
// of 128256 12.6 | 7.5, 256 rows of 128256 140 | 93, greedy 71 | 42; 1 row of 65536 7.4 | 7.5, greedy 5.6 | 7.5, 16 rows 12.1 | 8.6.
bool sample_two_stage(int B, int V, bool filtered) { return !filtered && !(B <= 33 && V <= (B <= 4 ? 65536 : 32768)); }
size_t sample_scratch_bytes(int B, int V) { return (size_t)B * ((V + kSampleChunk - 1) / kSampleChunk) * 8; }

cudaError_t sample_tokens(cudaStream_t s, const float* logits, int ldl, const float* temperature, const uint64_t* seed,
                          int32_t* out, int B, int V, void* scratch, const int32_t* top_k, const float* top_p) {
  if (B <= 0) return cudaSuccess;
  if (V <= 0) return cudaErrorInvalidValue;
  const bool filtered = temperature && (top_k || top_p);
  if (sample_two_stage(B, V, filtered)) {
    const int chunks = (V + kSampleChunk - 1) / kSampleChunk;
    float* pv = static_cast<float*>(scratch);
    int* pi = reinterpret_cast<int*>(pv + (size_t)B * chunks);
    const cudaError_t e = launch_k(sample_stage1_kernel, dim3(chunks, B), dim3(256), 0, s, true, logits, ldl, temperature, seed, pv, pi, V);
    if (e != cudaSuccess) return e;
    return launch_k(sample_stage2_kernel, dim3(B), dim3(32), 0, s, true, (const float*)pv, (const int*)pi, out, chunks);
  }
  if (filtered && V <= 8192)
    return launch_k(sample_row_kernel, dim3(B), dim3(kVocThreads), (size_t)voc_slice(V, 1) * 4, s, true, logits, ldl, temperature, seed, top_k, top_p, out, V);
  HB_VOC(sample_cluster_kernel, filtered ? voc_ctas(B, V, 0, 8, 22500) : 8, logits, ldl, temperature, seed, top_k, top_p, out, V);
}
cudaError_t apply_penalties(cudaStream_t s, float* logits, int ldl, const int32_t* pen_off, const void* pen, int B, int V) {
  if (B <= 0) return cudaSuccess;
  return launch_k(apply_penalties_kernel, dim3(B), dim3(256), 0, s, true, logits, ldl, pen_off, (const int2*)pen, V);
}
cudaError_t logprob_topk(cudaStream_t s, const float* logits, int ldl, int V, const int32_t* sampled, const int32_t* width,
                         int32_t* out_ids, float* out_lp, int B, int max_width, int widest) {
  if (B <= 0) return cudaSuccess;
  // Narrow records are two reads of the row (three of width 3) and stay with a block per row, except few long rows, which clusters read
  // sooner.  Us, block per row | clusters: width 2, 64 rows of 128256 19.8 | 23.4, 256 of 128256 47 | 89, 128 of 8192 4.5 | 5.9, 1 of
  // 128256 15.9 | 8.9, 32 of 100000 13.5 | 11.9; width 1, 32 of 65536 9.6 | 8.0, 32 of 32768 6.4 | 7.2.
  const int part = voc_slice(V, 8);
  const bool few = part > kVocSmemFloats || B <= (part <= 25000 ? 33 : 16);
  if ((widest <= 2 && !(few && V > (widest <= 1 ? 32768 : 65536))) || (widest == 3 && B > 128))
    return launch_k(logprob_row_kernel, dim3(B), dim3(kLpThreads), 0, s, true, logits, ldl, V, sampled, width, out_ids, out_lp, max_width);
  HB_VOC(logprob_topk_kernel, voc_ctas(B, V, 32768, V <= 65536 ? 4 : 8, 25000), logits, ldl, V, sampled, width, out_ids, out_lp, max_width);
}
#undef HB_VOC
cudaError_t cls_pool_l2(cudaStream_t s, const bf16* x, const int32_t* first_row, float* out, int B, int H) {
  if (B <= 0) return cudaSuccess;
  cls_pool_l2_kernel<<<B, kRowThreads, 0, s>>>(x, first_row, out, H);
  return cudaGetLastError();
}

}  // namespace hb
