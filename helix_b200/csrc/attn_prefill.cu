// K5: varlen flash attention for prefill (causal, GQA) and for the BERT encoder
// (bidirectional), on tcgen05 tensor cores with S, P and the output accumulator O all resident in TMEM.
// See the kernel comment for the warp roles and the two-q-tile ping-pong schedule.
#include <limits.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>

#include "kernels.h"
#include "launch.h"
#include "ptx.cuh"
#include "tma_host.h"

namespace hb {
namespace {

constexpr int BQ = 128;     // q rows per softmax warpgroup
constexpr int QPAIR = 256;  // q rows per CTA: two q tiles ping-pong on the tensor pipe
constexpr int BKV = 64;     // kv positions per tile (= one KV page)
constexpr int kThreads = 352;  // producer warp, one MMA issuer warp per q tile, two softmax warpgroups
constexpr float kRescaleThreshold = 8.0f;  // log2 units
constexpr int kPolyPairs = 2;  // of eight pairs of exponentials, on the FMA pipe
constexpr int kMaxRows = 512;  // (q pair, sequence) rows of a launch whose order is sorted

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x for two values on the FMA and ALU pipes only: x = n + f with n the nearest whole number, f in [-0.5, 0.5], a degree-3 minimax
// polynomial for 2^f (relative error 7.6e-5, far below the bf16 rounding that P gets), n added into the exponent field: the share of the
// exponentials that FlashAttention-4 takes off the SFU.  Masked scores are -inf, and the clamp keeps the exponent from wrapping: at -127 + 2^-13 the
// polynomial is just above one, so what is left is 0x67 * 2^-149, a bf16 zero (a weight of 2^-126 let large values behind the mask
// through, and its products changed the last bits of sums in the tensor cores).  A NaN passes the clamp (fmaxf would make it a weight of zero); it leaves as
// the largest finite number and makes the row's result infinite or NaN.
__device__ __forceinline__ float clamp_exponent(float x) {
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x) : "f"(-127.f + 1.f / 8192.f));
  return x;
}
__device__ __forceinline__ uint64_t exp2_poly2(uint64_t x2) {
  float x0, x1;
  f2_unpack(x2, x0, x1);
  x2 = f2_pack(clamp_exponent(x0), clamp_exponent(x1));
  const uint64_t magic = f2_pack(12582912.f, 12582912.f);  // 1.5 * 2^23: the sum's low mantissa bits hold round(x)
  const uint64_t t2 = f2_add(x2, magic);
  const uint64_t n2 = f2_add(t2, f2_pack(-12582912.f, -12582912.f));
  const uint64_t f2 = f2_fma(n2, f2_pack(-1.f, -1.f), x2);
  uint64_t p2 = f2_fma(f2_pack(0.05520550534f, 0.05520550534f), f2, f2_pack(0.24261397123f, 0.24261397123f));
  p2 = f2_fma(p2, f2, f2_pack(0.69325476885f, 0.69325476885f));
  p2 = f2_fma(p2, f2, f2_pack(0.99992769957f, 0.99992769957f));
  float t0, t1, p0, p1;
  f2_unpack(t2, t0, t1);
  f2_unpack(p2, p0, p1);
  const uint32_t r0 = __float_as_uint(p0) + (__float_as_uint(t0) << 23);
  const uint32_t r1 = __float_as_uint(p1) + (__float_as_uint(t1) << 23);
  return f2_pack(__uint_as_float(r0), __uint_as_float(r1));
}

// Optional event trace (tools/attn_test -DHB_ATTN_TRACE): CTA 0 stamps clock64() at the hand-off points of q tile 0.
#ifdef HB_ATTN_TRACE
__device__ unsigned long long g_attn_trace[8][4096];
__device__ int g_attn_trace_n[8];
#define HB_TRACE(ev)                                                          \
  do {                                                                        \
    if (blockIdx.x == 0) {                                                    \
      const int i_ = g_attn_trace_n[ev];                                      \
      if (i_ < 4096) { g_attn_trace[ev][i_] = clock64(); g_attn_trace_n[ev] = i_ + 1; } \
    }                                                                         \
  } while (0)
#else
#define HB_TRACE(ev) do {} while (0)
#endif

// The walk of a launch's items: q pair by q pair, the same with its last round as lone q tiles, or sorted by kv tiles (below)
enum Order : int { ORDER_PLAIN = 0, ORDER_SPLIT = 1, ORDER_SORTED = 2 };
// Split walk: the pairs from this one on, those of the last round, are taken as two lone q tiles each, where twice as many of them are no more than
// there are CTAs (elsewhere the answer is `pairs`): a lone q tile takes about 3/4 of a pair's time, and the SMs that would have had nothing take the other
// ones.  us back to back, pages, with the packings that it makes the better ones and the launches as they are now: 32 heads over 8 of 128 columns, 777 x 2 rows
// over 6000 keys 173 -> 170 (64 columns 156 -> 142), 512 over 2500 41 -> 33; 12 heads of their own, 333 x 2 over 4500 68 -> 55
// An instance of its own: the walk's few registers in the plain one cost every other launch 2 % (2048 rows over 7000 191.5 -> 196.5).
__host__ __device__ inline int first_split(int pairs, int ctas) {
  const int full = (pairs - 1) / ctas * ctas;
  return 2 * (pairs - full) <= ctas ? full : pairs;
}

// Where K and V rows come from: the packed activation, the paged planes, or (latent attention) expanded rows — per-head key and
// value parts made from cached latents plus one rotated key part that all heads share.
enum KvSource : int { KV_PACKED = 0, KV_PAGED = 1, KV_EXPANDED = 2 };

template <int DK, int DV, int SRC>
struct ACfg {
  static constexpr int Q_BYTES = BQ * DK * 2;    // one q tile
  static constexpr int K_BYTES = BKV * DK * 2;
  static constexpr int V_BYTES = BKV * DV * 2;
  static constexpr int STAGES = DK * DV >= 128 * 128 && !(SRC == KV_EXPANDED && DK == 128) ? 3 : 4;  // K ring and V ring depth
  // D = 64 (encoder; short sequences, an item's output write-back is a large part of its time) stages O in shared
  // memory and writes it with TMA: one 32-row x 128 B swizzled box per softmax warp.  Expanded rows leave no room for it.
  static constexpr bool STAGE_O = SRC != KV_EXPANDED;
  static constexpr int O_STAGE_BYTES = 32 * DV * 2;  // per softmax warp
  static constexpr int BAR_BYTES = 1024;            // barriers + TMEM pointer, padded so the staging area stays 1024-aligned
  static constexpr int SMEM = 2 * Q_BYTES + STAGES * (K_BYTES + V_BYTES) + 1024 + BAR_BYTES + (STAGE_O ? 8 * O_STAGE_BYTES : 0);
  static constexpr int SMEM_SORTED = SMEM + 2 * kMaxRows;  // the item order behind it
  static_assert(SRC != KV_PACKED || SMEM_SORTED <= 227 * 1024, "shared memory");
  static constexpr int SUBK = DK / 64, SUBV = DV / 64;  // 64-column swizzle sub-tiles per row
  static_assert(SMEM <= 227 * 1024, "shared memory");
};

// PERSISTENT kernel: one CTA per SM walks a static list of (256-row q pair, sequence, q-head) items, heaviest
// (most kv tiles) first and dealt forth and back, so the TMEM allocation, barrier setup and the latency of an
// item's first loads and of its output write-back overlap with the neighbouring items' work.
//
// kv tiles are 64 positions (= one KV page) and every q tile owns TWO S buffers in TMEM:
//   TMEM columns: [S0a S0b S1a S1b] 4 x 64 fp32 | O0 | O1 (D fp32 each, at 256 + t*128).  P_t(j), packed bf16x2,
//   overwrites the first 32 columns of the buffer S_t(j) was read from.
// S_t(j+1) = Q_t·K(j+1)ᵀ is therefore issued BEFORE the softmax of tile j has produced P_t(j): the softmax warps find
// their next S tile waiting when they finish one, and the tensor pipe always has the other buffer's / other q tile's
// work queued.  (With one S buffer per q tile — the previous version — S(j+1) had to wait for PV(j), i.e. for the
// softmax: ncu showed the softmax warps waiting for S 56 % of the time and the tensor pipe 41 % busy.)
//   warp 0 lane 0 : TMA producer (Q pair of the next item as soon as the last S MMA of the current one retired;
//                   K_j / V_j through KST-stage rings that keep running across items)
//   warp 1 lane 0 : MMA issuer, program order  S_t(0) S_t(1) | PV0(j) S0(j+2) PV1(j) S1(j+2) ...  P is consumed straight
//                   from TMEM (tcgen05.mma A-from-TMEM), V straight from its [kv][d] layout (MN-major B).
//   warps 2..5 / 6..9 : softmax warpgroup of q tile 0 / 1, one thread per q row; lazy O rescale; O/l -> global.
//
// KV_PACKED: K/V rows come from the same packed [T, ...] activation as Q (whole-prompt prefill, encoder), kv_len == q_len.
// KV_PAGED: the q rows are the LAST q_len positions of a kv_len-long sequence whose K/V (including the chunk's own,
//                written by the RoPE/KV-write kernel just before) live in the paged pool (chunked prefill, prefix-cache
//                hits): tile j is page_table[b][j].
// KV_EXPANDED: batch entry b is run b of `runs` (q rows [t0, t0 + len) of the packed activation, the last rows of the kv rows
//                [row0, row0 + kv) of the expanded buffers).  A q / k row has DK / 64 sub-tiles: the head's unrotated part in
//                all but the last, the rotated part (shared by all heads on the key side) in the last; parts that are no
//                multiple of 64 wide are zero-filled by the tensor maps.
template <int DK, int DV, int SRC, int ORDER>
__global__ void __launch_bounds__(kThreads, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_o,
                    bf16* __restrict__ out, int ldo,
                    const int32_t* __restrict__ cu_seqlens, int B, int Hq, int group, int causal, float scale_log2,
                    int max_q_pairs, const int32_t* __restrict__ kv_lens, const int32_t* __restrict__ page_table,
                    int max_pages, int Hkv, int chunk, int sink, const float* __restrict__ head_gate, int ldg,
                    int window, float cap_in, float cap_out, const bf16* __restrict__ sink_w,
                    const __grid_constant__ CUtensorMap map_qr, const __grid_constant__ CUtensorMap map_kr,
                    const __grid_constant__ AttnRuns runs, int vdim, int pack) {
  using C = ACfg<DK, DV, SRC>;
  constexpr bool PAGED = SRC == KV_PAGED, EXPANDED = SRC == KV_EXPANDED, SORTED = ORDER == ORDER_SORTED;
  constexpr int KST = C::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                          // [2][Q_BYTES]
  uint8_t* sK = sQ + 2 * C::Q_BYTES;           // [KST][K_BYTES]
  uint8_t* sV = sK + KST * C::K_BYTES;        // [KST][V_BYTES]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + KST * C::V_BYTES);
  uint64_t* q_full = bars + 0;
  uint64_t* q_empty = bars + 1;
  uint64_t* s_full = bars + 2;    // [q tile][S buffer]
  uint64_t* p_full = bars + 6;    // [q tile][S buffer]
  uint64_t* pv_done = bars + 10;  // [q tile][tile parity]: two per q tile, so that a waiter can never be a whole
                                  // phase behind (PV(x-2) is known complete whenever PV(x) is waited for, PV(x-1) is not)
  uint64_t* o_free = bars + 14;   // [2]
  uint64_t* k_full = bars + 16;   // [KST]
  uint64_t* k_empty = k_full + KST;
  uint64_t* v_full = k_empty + KST;
  uint64_t* v_empty = v_full + KST;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(v_empty + KST);
  int* s_rows = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 512);  // rows in the order (-1: none), then warp sums
  uint8_t* sO = reinterpret_cast<uint8_t*>(bars) + C::BAR_BYTES;  // [8 softmax warps][32 rows][DV] (STAGE_O only)
  uint16_t* s_order = reinterpret_cast<uint16_t*>(sO + (C::STAGE_O ? 8 * C::O_STAGE_BYTES : 0));  // [kMaxRows] q pair << 8 | sequence

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  struct Item {
    int b, h, kvh, q0, seq0, len, kv_len, q_off, n0, n1, n;
    int j_lo;  // first kv tile of the item (block mask: the tile that holds the block start of the pair's first row)
    bool valid, act1;
  };
  // A q row is a (token, head) pair: with pack > 0 the 1 << pack neighbouring query heads of an item, which share a kv head, sit side by side
  // in the rows of a tile (row = token << pack | head), so a tile covers 128 >> pack tokens; `it.h` counts such groups of heads.
  // sequence b: its first row in the packed activation, its q rows in this step, its kv positions
  auto set_seq = [&](Item& it, int b) {
    it.b = b;
    if constexpr (EXPANDED) {  // positions below count from the first expanded row of the run
      it.seq0 = runs.t0[b];
      it.len = runs.len[b];
      it.kv_len = runs.kv[b];
    } else {
      it.seq0 = cu_seqlens[b];
      it.len = cu_seqlens[b + 1] - it.seq0;  // q rows of this sequence in the step
      it.kv_len = PAGED ? kv_lens[b] : it.len;
    }
    it.q_off = it.kv_len - it.len;  // position of the first q row (0 unless this is a later chunk of a long prompt)
    if constexpr (!EXPANDED) it.len <<= pack;
  };
  auto set_rows = [&](Item& it, int q0, bool both) {
    it.q0 = q0;
    it.valid = it.q0 < it.len;
    const int kv_tiles = (it.kv_len + BKV - 1) / BKV;
    it.act1 = both && it.q0 + BQ < it.len;
    // causal: q tile t needs kv tiles up to the one holding its last row's own position
    // block mask (chunk > 0, paged only): a row sees its own block of `chunk` positions, counted from position 0, up to
    // itself; tiles before the block of the pair's first row are skipped, n0 / n1 / n count tiles from j_lo
    // sliding window (window > 0, paged only): a row sees the `window` positions that end with itself; tiles before the
    // window of the pair's first row are skipped
    it.j_lo = (PAGED && chunk > 0) ? ((it.q_off + (it.q0 >> pack)) / chunk * chunk) / BKV
              : (SRC != KV_PACKED && window > 0) ? max(0, it.q_off + (it.q0 >> pack) - window + 1) / BKV : 0;
    it.n0 = (causal ? min(kv_tiles, (it.q_off + ((it.q0 + BQ - 1) >> pack)) / BKV + 1) : kv_tiles) - it.j_lo;
    it.n1 = it.act1 ? (causal ? min(kv_tiles, (it.q_off + ((it.q0 + 2 * BQ - 1) >> pack)) / BKV + 1) : kv_tiles) - it.j_lo : 0;
    it.n = max(it.n0, it.n1);
  };
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    if constexpr (C::STAGE_O) tma_prefetch_desc(&map_o);
    if constexpr (EXPANDED) {
      tma_prefetch_desc(&map_qr);
      tma_prefetch_desc(&map_kr);
    }
    mbar_init(q_full, 1);
    mbar_init(q_empty, 2);  // both issuers
    for (int i = 0; i < 4; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&pv_done[i], 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(&o_free[i], 4);
    for (int i = 0; i < KST; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 2);  // released by both issuers
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 2);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  pdl_wait();  // nothing above touches memory that a kernel before this one may write
  // Order of the items (SORTED): rows (q pair, sequence) by falling number of kv tiles, a row's heads side by side (they share keys), dealt
  // to the CTAs forth and back (round r of CTA c is item r G + c, or r G + G - 1 - c in odd rounds).  Every CTA sorts the rows itself
  // (a thread per row, ranks by counting four keys a read; a thread per sequence that walked its rows, and one key a read, cost 2 us more: 6 prompts of 300 to 3000
  // tokens, 64 columns 158.7 -> 156.6).  With sequences of unequal length the plain order, q pair by q pair with a slot
  // for every sequence whether it has that pair or not, left the longest-loaded CTA 24 to 30 % above the mean (6 prompts of 300
  // to 3000 tokens: 231 tile times of a mean of 187, now 191; 64 chunks of 64 to 512: 74 of 57, now 60).  Measured: 250 -> 233 us and 70.8 -> 62.6 us.
  // Everything else runs the kernel with the plain walk: launches whose sequences are short or of about equal lengths (wants_order below), and
  // keys from a page pool or an expanded run (portions of a long context are level already).  The plain order also stands in where a
  // launch turns out to have more rows than kMaxRows.
  if constexpr (SORTED) {
    uint32_t* keys = reinterpret_cast<uint32_t*>(sK);  // scratch over the K ring (nothing has been loaded yet): [kMaxRows] keys, first row of each sequence
    int* starts = reinterpret_cast<int*>(keys + kMaxRows);
    const int b = threadIdx.x;
    Item it;
    int pairs = 0;
    if (b < B) {
      set_seq(it, b);
      pairs = min(max_q_pairs, max(0, (it.len + QPAIR - 1) / QPAIR));
    }
    int upto = pairs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (lane == 31) s_rows[1 + warp] = upto;
    __syncthreads();
    int before = 0, rows = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
      const int v = s_rows[1 + w];
      if (w < warp) before += v;
      rows += v;
    }
    if (rows <= kMaxRows) {
      if (b < B) starts[b] = before + upto - pairs;
      __syncthreads();
      for (int r = threadIdx.x; r < (rows + 3) / 4 * 4; r += kThreads) {
        uint32_t key = 0;  // (no row: nothing is behind it)
        if (r < rows) {
          int q = 0;  // the last sequence that starts at or before row r
          for (int step = 128; step > 0; step >>= 1)
            if (q + step < B && starts[q + step] <= r) q += step;
          set_seq(it, q);
          set_rows(it, (r - starts[q]) * QPAIR, true);
          key = (uint32_t)(3 * it.n + min(it.n0, it.n1) + 6) * kMaxRows + (kMaxRows - 1 - r);  // (a lone q tile takes about 3/4 of a pair's time)
        }
        keys[r] = key;
      }
      __syncthreads();
      for (int r = threadIdx.x; r < rows; r += kThreads) {
        const uint32_t key = keys[r];
        int rank = 0, q = 0;
#pragma unroll 8
        for (int i = 0; i < (rows + 3) / 4; ++i) {
          const uint4 k4 = reinterpret_cast<const uint4*>(keys)[i];
          rank += (k4.x > key) + (k4.y > key) + (k4.z > key) + (k4.w > key);
        }
        for (int step = 128; step > 0; step >>= 1)
          if (q + step < B && starts[q + step] <= r) q += step;
        s_order[rank] = (uint16_t)((r - starts[q]) << 8 | q);
      }
      fence_proxy_async_smem();  // the scratch becomes a target of asynchronous copies
    }
    if (threadIdx.x == 0) s_rows[0] = rows <= kMaxRows ? rows : -1;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // The launch behind may take its places as soon as every block of this one holds its tensor memory (launch.h).  Not behind paged rows with an item a block
  // at most: those launches run for tens of us on fewer SMs than there are, and a next one that sat down early on the free SMs and
  // got the rest as they ended ran 6 % longer than one placed at once (128 items a launch, back to back: 891 rows over 2841 keys
  // 47.4 -> 44.8 us, 700 over 3000 49.8 -> 46.3; with more items than blocks 61.6 both ways).  Packed prompts of that
  // size end within a few us, where the early start is worth more (6.5 -> 6.2 us).
  if (!PAGED || max_q_pairs * B * (Hq >> pack) > (int)gridDim.x) pdl_launch_dependents();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr, 0);  // warp-uniform for the compiler too
  const int rows = SORTED ? s_rows[0] : -1;
  const int groups = Hq >> pack;  // of heads that an item takes together
  const int num_pairs = (SORTED && rows >= 0 ? rows : max_q_pairs * B) * groups;
  const int split_from = ORDER == ORDER_SPLIT ? first_split(num_pairs, gridDim.x) : num_pairs;
  const int num_items = 2 * num_pairs - split_from;
  auto next_item = [&](int idx, int round) {
    if constexpr (SORTED) {
      if (rows >= 0) return round * (int)gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
    }
    return (int)((unsigned)idx + gridDim.x);  // (as a signed sum it took four more registers, spilled, than `idx += gridDim.x` does)
  };
  auto get_item = [&](int idx) {
    Item it;
    if constexpr (SORTED) {
      if (rows >= 0) {
        const int row = idx / groups;
        it.h = idx - row * groups;
        it.kvh = (it.h << pack) / group;
        set_seq(it, s_order[row] & 255);
        set_rows(it, (s_order[row] >> 8) * QPAIR, true);
        return it;
      }
    }
    const bool lone = ORDER == ORDER_SPLIT && idx >= split_from;
    const int second = lone ? (idx - split_from) & 1 : 0;
    if (lone) idx = split_from + ((idx - split_from) >> 1);
    const int per_qp = B * groups;
    const int qp = max_q_pairs - 1 - idx / per_qp;  // latest q rows first, one "round" per q pair index
    const int rem = idx % per_qp;
    const int b = rem / groups;
    it.h = rem % groups;
    it.kvh = (it.h << pack) / group;
    set_seq(it, b);
    set_rows(it, qp * QPAIR + second * BQ, !lone);
    return it;
  };

  // The two single-thread roles run their loops and barrier waits with the WHOLE warp converged and only predicate the
  // TMA / tcgen05 instructions on an elect.sync leader: issuing them under `if (lane == 0)` measured slower (the tensor pipe
  // 33-41 % busy with an issuer that never waited for its inputs).
  if (warp == 0) {
    const bool leader = elect_one_sync();
    {
      int kt = 0, qi = 0;  // running kv-tile / item counters: barrier phases continue across items
      for (int round = 0, idx = blockIdx.x; idx < num_items; idx = next_item(idx, ++round)) {
        const Item it = get_item(idx);
        if (!it.valid) continue;
        mbar_wait(q_empty, (qi & 1) ^ 1);  // every S MMA of the previous item has retired: the Q pair buffer is free
        if (leader) {
          mbar_arrive_expect_tx(q_full, (it.act1 ? 2 : 1) * C::Q_BYTES);
          for (int t = 0; t < (it.act1 ? 2 : 1); ++t)
#pragma unroll
            for (int c = 0; c < C::SUBK; ++c) {
              uint8_t* dst = sQ + t * C::Q_BYTES + c * (BQ * 128);
              const int row = it.seq0 + ((it.q0 + t * BQ) >> pack);
              if constexpr (EXPANDED)
                tma_load_3d(dst, c < C::SUBK - 1 ? &map_q : &map_qr, q_full, c < C::SUBK - 1 ? c * 64 : 0, it.h, row, kEvictFirst);
              else
                tma_load_3d(dst, &map_q, q_full, c * 64, it.h << pack, row, kEvictFirst);
            }
        }
        ++qi;
        for (int j = 0; j < it.n; ++j, ++kt) {
          const int s = kt % KST;
          const uint32_t ph = (kt / KST) & 1;
          int blk = 0;  // PAGED: (page, kv head) block of the tile's page
          if constexpr (EXPANDED) blk = runs.row0[it.b] + (it.j_lo + j) * BKV;  // first expanded row of the tile
          if constexpr (PAGED) blk = page_table[(size_t)it.b * max_pages + it.j_lo + j] * Hkv + it.kvh;
          mbar_wait(&k_empty[s], ph ^ 1);
          if (leader) {
            mbar_arrive_expect_tx(&k_full[s], C::K_BYTES);
#pragma unroll
            for (int c = 0; c < C::SUBK; ++c) {
              uint8_t* dst = sK + s * C::K_BYTES + c * (BKV * 128);
              if constexpr (EXPANDED) {
                if (c < C::SUBK - 1) tma_load_3d(dst, &map_k, &k_full[s], c * 64, it.h, blk, kEvictLast);
                else tma_load_2d(dst, &map_kr, &k_full[s], 0, blk, kEvictLast);
              } else if constexpr (PAGED) {
                tma_load_3d(dst, &map_k, &k_full[s], c * 64, 0, blk, kEvictLast);
              } else {
                tma_load_2d(dst, &map_k, &k_full[s], it.kvh * DK + c * 64, it.seq0 + j * BKV, kEvictLast);
              }
            }
          }
          mbar_wait(&v_empty[s], ph ^ 1);
          if (leader) {
            mbar_arrive_expect_tx(&v_full[s], C::V_BYTES);
#pragma unroll
            for (int c = 0; c < C::SUBV; ++c) {
              uint8_t* dst = sV + s * C::V_BYTES + c * (BKV * 128);
              if constexpr (EXPANDED)
                tma_load_3d(dst, &map_v, &v_full[s], c * 64, it.h, blk, kEvictLast);
              else if constexpr (PAGED)
                tma_load_3d(dst, &map_v, &v_full[s], c * 64, 0, blk, kEvictLast);
              else
                tma_load_2d(dst, &map_v, &v_full[s], it.kvh * DV + c * 64, it.seq0 + j * BKV, kEvictLast);
            }
          }
        }
      }
    }
  } else if (warp == 1 || warp == 2) {
    // One MMA issuer warp PER q tile.  With a single in-order issuer for both tiles (PV0 S0 PV1 S1 ...) the event trace
    // (tools/attn_test -DHB_ATTN_TRACE) showed P0(j) sitting ~900 cycles before the issuer looked at it — it was blocked
    // on the other warpgroup's P — so S0(j+2) was issued only ~600 cycles before the softmax needed it and the second S
    // buffer bought nothing.  The two chains are independent except for the K/V ring slots, which are released by both
    // (empty barriers count 2; a tile one issuer does not need is released by a plain arrive once it has landed).
    // The issuer's own instruction stream is on the critical path (one warp, ~4 cycles per dependent instruction), so:
    // descriptors are a per-kernel base plus a constant (the 14-bit address field never carries), ring slots and phases
    // are running counters, and the steady state is a branch-free instantiation.
    const int t = warp - 1;
    const bool leader = elect_one_sync();
    constexpr uint32_t idesc_qk = umma_idesc_bf16(BQ, BKV, 0, 0);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(BQ, DV, 0, 1);  // A = P from TMEM, B = V is MN-major
    const uint64_t qdesc = umma_desc_kmajor_sw128(smem_u32(sQ + t * C::Q_BYTES));
    const uint64_t kdesc0 = umma_desc_kmajor_sw128(smem_u32(sK));
    const uint64_t vdesc0 = umma_desc_mnmajor_sw128(smem_u32(sV), BKV * 128, 1024);
    const uint32_t tmem_s = tmem_base + t * 128, tmem_o = tmem_base + 256 + t * 128;
    uint64_t* const my_s_full = s_full + t * 2;
    uint64_t* const my_p_full = p_full + t * 2;
    uint64_t* const my_pv_done = pv_done + t * 2;
    int kslot = 0, vslot = 0;  // ring slots of the next K / V tile (this issuer walks ALL tiles of an item)
    uint32_t kphase = 0, vphase = 0;
    int ps = 0;                // absolute index (over the kernel's life) of this q tile's next PV; S buffer = index & 1
    int oi = 0, qi = 0;        // items with work for this q tile (phase of o_free) / items seen (phase of q_full)
    // S(tile x) = Q_t · Kᵀ (K in ring slot kslot) into buffer x & 1
    auto mma_s = [&](int x) {
      const uint32_t d_tmem = tmem_s + (x & 1) * BKV;
      const uint64_t kd = kdesc0 + (uint64_t)(kslot * (C::K_BYTES >> 4));
#pragma unroll
      for (int k = 0; k < DK / 16; ++k)
        umma_f16_ss(d_tmem, qdesc + (((k >> 2) * (BQ * 128) + (k & 3) * 32) >> 4),
                    kd + (((k >> 2) * (BKV * 128) + (k & 3) * 32) >> 4), idesc_qk, k != 0 ? 1u : 0u);
      umma_commit(&my_s_full[x & 1]);
      umma_commit(&k_empty[kslot]);
    };
    // O_t (+)= P(tile x) · V (V in ring slot vslot)
    auto mma_pv = [&](int x, uint32_t acc) {
      const uint32_t p_tmem = tmem_s + (x & 1) * BKV;
      const uint64_t vd = vdesc0 + (uint64_t)(vslot * (C::V_BYTES >> 4));
#pragma unroll
      for (int k = 0; k < BKV / 16; ++k)
        umma_f16_ts(tmem_o, p_tmem + k * 8, vd + ((k * 16 * 128) >> 4), idesc_pv, (acc | k) != 0 ? 1u : 0u);
      umma_commit(&my_pv_done[x & 1]);
      umma_commit(&v_empty[vslot]);
    };
    auto k_advance = [&]() { if (++kslot == KST) { kslot = 0; kphase ^= 1; } };
    auto v_advance = [&]() { if (++vslot == KST) { vslot = 0; vphase ^= 1; } };
    // one kv tile j of the item: PV(j) if this q tile has one, S(j+2) if it has one; slots it does not use are released
    auto step = [&](auto fast_tag, bool has_pv, bool has_k, bool has_s, bool first, bool last_s) {
      constexpr bool FAST = decltype(fast_tag)::value;
      mbar_wait(&v_full[vslot], vphase);
      if (FAST || has_k) mbar_wait(&k_full[kslot], kphase);
      if (FAST || has_pv) {
        if (!FAST && first) mbar_wait(&o_free[t], (oi & 1) ^ 1);  // the previous item's O_t has been read out
        mbar_wait(&my_p_full[ps & 1], (ps >> 1) & 1);
        // P(ps) exists, so S(ps) and — issued before it — PV(ps-2) have completed: observe that pv_done phase here (it
        // costs the issuer nothing) so that no phase of the barrier passes without a wait (compute-sanitizer synccheck);
        // the softmax warps only wait on pv_done when they rescale O and at the end of an item
        if (ps >= 2) mbar_wait(&my_pv_done[ps & 1], ((ps - 2) >> 1) & 1);
        tc_fence_after();
        if (t == 0 && leader) HB_TRACE(0);  // issuer saw P0(j)
        if (leader) {
          mma_pv(ps, FAST ? 1u : (first ? 0u : 1u));
          if (FAST || has_s) mma_s(ps);  // S(j+2) reuses the buffer PV(j) reads: same-thread MMAs retire in order
          if (!FAST && last_s) umma_commit(q_empty);  // that was this q tile's last S MMA of the item
        }
        if (t == 0 && leader) HB_TRACE(1);  // PV0(j), S0(j+2) issued
        ++ps;
      } else if (leader) {
        mbar_arrive(&v_empty[vslot]);
      }
      if (!FAST && has_k && !has_s && leader) mbar_arrive(&k_empty[kslot]);
      v_advance();
      if (FAST || has_k) k_advance();
    };
    for (int round = 0, idx = blockIdx.x; idx < num_items; idx = next_item(idx, ++round)) {
      const Item it = get_item(idx);
      if (!it.valid) continue;
      const int nt = t == 0 ? it.n0 : it.n1, n = it.n;
      mbar_wait(q_full, qi & 1);
      // S(0), S(1): their buffers are free — the PVs that read them were issued earlier by this same thread
      for (int j = 0; j < 2 && j < n; ++j) {
        mbar_wait(&k_full[kslot], kphase);
        tc_fence_after();
        if (leader) {
          if (j < nt) mma_s(ps + j); else mbar_arrive(&k_empty[kslot]);
        }
        k_advance();
      }
      if (leader) {
        if (nt == 0) mbar_arrive(q_empty);
        else if (nt <= 2) umma_commit(q_empty);
      }
      for (int j = 0; j < n; ++j) {
        if (j > 0 && j + 3 < nt)
          step(std::true_type{}, true, true, true, false, false);
        else
          step(std::false_type{}, j < nt, j + 2 < n, j + 2 < nt, j == 0, j + 3 == nt);
      }
      oi += nt > 0;
      ++qi;
    }
  } else {
    const int t = (warp - 3) >> 2;  // q tile of this warpgroup
    const int qd = warp & 3;
    const int r = qd * 32 + lane;  // q row in tile == TMEM lane
    const uint32_t lane_sel = static_cast<uint32_t>(qd * 32) << 16;
    const uint32_t tO = tmem_base + lane_sel + 256 + t * 128;
    int jt = 0;  // kv tiles this warpgroup has processed so far (S buffer and barrier phases)
    const bool follow = !causal && (group & 1);  // rows are rescaled with their warp
    bool passed = false;  // this warp has passed on a turn (the very first one, of tile 0, is not waited for)
    for (int round = 0, idx = blockIdx.x; idx < num_items; idx = next_item(idx, ++round)) {
      const Item it = get_item(idx);
      if (!it.valid) continue;
      const int nt = t == 0 ? it.n0 : it.n1;
      if (nt == 0) continue;
      const int len = it.kv_len;                  // kv positions of the sequence
      const int qt0 = it.q_off + ((it.q0 + t * BQ) >> pack), qt1 = qt0 + ((BQ - 1) >> pack);  // absolute positions of the tile's first and last q row
      const int qpos = qt0 + (r >> pack);
      const bool live = it.q0 + t * BQ + r < it.len;  // the row exists
      const int token = it.seq0 + ((it.q0 + t * BQ + r) >> pack), head = (it.h << pack) + (r & ((1 << pack) - 1));
      const int turns = DK <= 128 ? min(it.n0, it.n1) : 0;  // tiles that both q tiles have
      float m_used = -1e30f, l = 0.f;  // (rows that see nothing yet: far below every score, and finite)
      for (int j = 0; j < nt; ++j) {
        const int tile = jt + j;
        const uint32_t tS = tmem_base + lane_sel + t * 128 + (tile & 1) * BKV;
        if (t == 0 && warp == 3 && lane == 0) HB_TRACE(2);  // softmax 0 starts waiting for S0(j)
        mbar_wait(&s_full[t * 2 + (tile & 1)], (tile >> 1) & 1);
        tc_fence_after();
        if (t == 0 && warp == 3 && lane == 0) HB_TRACE(3);  // got S0(j)
        const int kv0 = (it.j_lo + j) * BKV;
        const int lo = chunk > 0 ? qpos / chunk * chunk : (window > 0 ? qpos - window + 1 : 0);  // first kv position this row sees
        const bool begins = (chunk > 0 && kv0 < qt1 / chunk * chunk) || (window > 0 && kv0 <= qt1 - window);  // some row's block or window, in this tile
        const bool need_mask = (kv0 + BKV > len) || (causal && (kv0 + BKV - 1 > qt0)) || begins;
        const int lim = causal ? min(len - 1, qpos) : len - 1;  // last valid kv position for this row
        // ---- the S row: back-to-back TMEM loads, ONE wait, then max / exp2 / pack entirely in registers
        uint32_t sv[BKV];
#pragma unroll
        for (int c = 0; c < BKV / 32; ++c) {
          uint32_t(&dst)[32] = *reinterpret_cast<uint32_t(*)[32]>(&sv[c * 32]);
          tmem_ld_32x32b_x32(tS + c * 32, dst);
        }
        tmem_ld_wait();
        if (cap_in > 0.f) {
          // capped scores: s <- cap tanh(scale s / cap), left in the exp2 domain (cap_in = scale / cap, cap_out = cap log2 e; the
          // scale below is then one).  tanh(y) = 1 - 2 / (e^2y + 1) keeps the scores at fp32 accuracy, which the one-operation
          // hardware tanh (2^-11 relative) does not; two scores share a reciprocal (1 / a = b / ab), exponents stay below 2^60 so
          // that ab is finite (tanh is 1 there).
          const float k2 = 2.f * 1.4426950408889634f * cap_in, m2 = -2.f * cap_out;
#pragma unroll
          for (int i = 0; i < BKV; i += 2) {
            const float ea = fast_exp2(fminf(__uint_as_float(sv[i]) * k2, 60.f)) + 1.f, eb = fast_exp2(fminf(__uint_as_float(sv[i + 1]) * k2, 60.f)) + 1.f;
            float rc;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(ea * eb));
            rc *= m2;
            sv[i] = __float_as_uint(fmaf(rc, eb, cap_out));
            sv[i + 1] = __float_as_uint(fmaf(rc, ea, cap_out));
          }
        }
        if (need_mask) {  // diagonal / ragged tiles only: knock the invalid columns out once, the hot loops stay branch-free.  One comparison per
          // column and, where a block or a window begins in the tile, another pass (both at once cost 700 cycles, half a tile)
          const int upto = lim - kv0, from = lo - kv0;  // columns that the row sees
#pragma unroll
          for (int i = 0; i < BKV; ++i) sv[i] = i <= upto ? sv[i] : 0xff800000u;  // -inf
          if (begins) {  // (of the whole q tile: a branch on a row's own `from` would part the warp before the aligned operations below)
#pragma unroll
            for (int i = 0; i < BKV; ++i) sv[i] = i >= from ? sv[i] : 0xff800000u;
          }
        }
        float mx8[8];  // eight independent chains instead of one long dependent max chain
#pragma unroll
        for (int i = 0; i < 8; ++i) mx8[i] = __uint_as_float(sv[i]);
#pragma unroll
        for (int i = 8; i < BKV; ++i) mx8[i & 7] = fmaxf(mx8[i & 7], __uint_as_float(sv[i]));
        const float mx = fmaxf(fmaxf(fmaxf(mx8[0], mx8[1]), fmaxf(mx8[2], mx8[3])), fmaxf(fmaxf(mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7])));
        const float sl2 = cap_in > 0.f ? 1.f : scale_log2;
        float m_new = (mx == -INFINITY) ? m_used : mx * sl2;
        if (j == 0) {
          m_used = m_new;
        } else {
          const bool need = m_new > m_used + kRescaleThreshold;
          if (__any_sync(0xffffffffu, need)) {
            mbar_wait(&pv_done[t * 2 + ((tile - 1) & 1)], ((tile - 1) >> 1) & 1);  // PV(j-1), hence every PV so far, is in O_t
            tc_fence_after();
            // (A row that follows its warp has the weight one, without a rounding, at its new maximum.  Where heads can be packed, which depends on the
            // whole launch, and in causal prompts, which may come in portions, only the rows that need it do: a row's bits do not depend on the rows
            // beside it.  The rows of an encoder and expanded rows always stand beside the same ones.  Error against 64 bits with scores of deviation 4,
            // following / not: 1.95e-3 / 2.00e-3; of deviation 1, where hardly any row is rescaled, 1.98e-3 both)
            m_new = EXPANDED || follow ? fmaxf(m_new, m_used) : need ? m_new : m_used;
            const float f = fast_exp2(m_used - m_new);
            m_used = m_new;
            l *= f;
#pragma unroll
            for (int c = 0; c < DV / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(tO + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
              tmem_st_32x32b_x16(tO + c * 32, *reinterpret_cast<uint32_t(*)[16]>(&o[0]));
              tmem_st_32x32b_x16(tO + c * 32 + 16, *reinterpret_cast<uint32_t(*)[16]>(&o[16]));
            }
          }
        }
        // ---- p = exp2(s*scale - m) (masked entries are -inf -> 0), row sum, P (bf16x2) written over the S buffer's head;
        //      scale/subtract and the sum are packed
        if (t == 0 && warp == 3 && lane == 0) HB_TRACE(4);  // loaded, max, rescale decision done
        // The q tiles' warps of a quarter of the SM take turns with the exponentials (barriers 1 + qd: tile 0's turn, 5 + qd: tile 1's).  Left to
        // themselves both worked on their exponentials at the same time and waited for scores, loads and barriers at the same time: a kv
        // tile took 2000 cycles, 1580 now, of which the SFU has 2 x 48 exponentials of 8 cycles.  Two of eight pairs are polynomials (kPolyPairs), which costs a
        // little more than it saves now that there are turns: all on the SFU | so, 6 prompts of 300 to 3000 tokens with 32 heads over 8 184 | 187 us (64
        // columns 154 | 162), 64 chunks of 64 to 512 tokens 62 | 64, 100 rows over 4000 keys, whose q tiles have no partner, 57 | 55.  They stay for the results:
        // the logits of a 16-layer decoder, 5 prompts x 32 steps, have the same rms error (0.02061 | 0.02057), but other single errors, and with the SFU alone
        // the largest ones exceed what the full-size tests allow.
        // Every turn is waited for, the first one of an item too: a warp that passed on its turn twice before the other had taken the first would
        // complete the barrier by itself.  Keys of 192 columns take no turns (with | without: 16 heads, 512 rows over 6000 expanded keys 119 | 99 us, 2048 rows of
        // their own keys 50 | 46); of 128 they do (2 x 1500 rows with a window of 512, before the turns 45.5, with them 43.7).
        if (j < turns && (t == 1 || passed)) bar_sync((t ? 5 : 1) + qd, 64);
        const uint64_t scale2 = f2_pack(sl2, sl2), negm2 = f2_pack(-m_used, -m_used);
        uint64_t sum2a = 0, sum2b = 0;
#pragma unroll
        for (int c = 0; c < BKV / 16; ++c) {
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t x2 = f2_fma(f2_pack(__uint_as_float(sv[c * 16 + 2 * i]), __uint_as_float(sv[c * 16 + 2 * i + 1])),
                                       scale2, negm2);
            uint64_t p2;
            if (i % (8 / kPolyPairs) == 0) {  // evenly between the SFU's
              p2 = exp2_poly2(x2);
            } else {
              float x0, x1;
              f2_unpack(x2, x0, x1);
              p2 = f2_pack(fast_exp2(x0), fast_exp2(x1));
            }
            float p0, p1;
            f2_unpack(p2, p0, p1);
            if (i & 1) sum2b = f2_add(sum2b, p2); else sum2a = f2_add(sum2a, p2);
            pk[i] = pack_bf16x2(p0, p1);
          }
          tmem_st_32x32b_x8(tS + c * 8, pk);
        }
        {
          float s0, s1;
          f2_unpack(f2_add(sum2a, sum2b), s0, s1);
          l += s0 + s1;
        }
        if (t == 0 && warp == 3 && lane == 0) HB_TRACE(5);  // exp loop done, P stores issued
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (j < turns) {  // (before lane 0 goes its own way: bar.arrive wants the whole warp)
          bar_arrive((t ? 1 : 5) + qd, 64);  // the other tile's turn
          passed = true;
        }
        if (lane == 0) mbar_arrive(&p_full[t * 2 + (tile & 1)]);
        if (t == 0 && warp == 3 && lane == 0) HB_TRACE(6);  // P0(j) handed over
      }
      // ---- item epilogue: O / l -> global, then hand O_t back to the MMA issuer
      mbar_wait(&pv_done[t * 2 + ((jt + nt - 1) & 1)], ((jt + nt - 1) >> 1) & 1);
      tc_fence_after();
      if (sink) l += fast_exp2(-m_used);  // one more unit in the denominator: a key of score 0 that carries no value
      if (sink_w != nullptr) l += fast_exp2(__bfloat162float(sink_w[head]) * 1.4426950408889634f - m_used);  // a learned one per head
      float inv_l = l > 0.f ? 1.0f / l : 0.f;
      // optional output gate: the head's rows are scaled by sigmoid(head_gate[token][head]) on their way out
      if (head_gate != nullptr && live) inv_l *= 1.f / (1.f + __expf(-head_gate[(size_t)token * ldg + head]));
      bool staged = false;
      if constexpr (C::STAGE_O) {
        // Every thread writing its own 128-byte row straight to global is 32 distinct lines per store instruction: ncu
        // showed the warps spending about as long draining those stores (LSU queue, then the next TMEM load and even a
        // stack reload stuck behind them) as waiting for the last PV.  Full 32-row chunks go through a swizzled staging
        // buffer and ONE bulk tensor store per warp; the ragged last chunk of a sequence keeps the direct path.
        staged = it.q0 + t * BQ + qd * 32 + 32 <= it.len;  // warp-uniform
        if (staged) {
          uint8_t* stage = sO + (warp - 3) * C::O_STAGE_BYTES;
          if (lane == 0) tma_store_wait_read<0>();  // this warp's previous store has finished reading the buffer
          __syncwarp();
#pragma unroll
          for (int c = 0; c < DV / 32; ++c) {
            uint32_t o[32];
            tmem_ld_32x32b_x32(tO + c * 32, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(o[8 * i + 0]) * inv_l, __uint_as_float(o[8 * i + 1]) * inv_l);
              w.y = pack_bf16x2(__uint_as_float(o[8 * i + 2]) * inv_l, __uint_as_float(o[8 * i + 3]) * inv_l);
              w.z = pack_bf16x2(__uint_as_float(o[8 * i + 4]) * inv_l, __uint_as_float(o[8 * i + 5]) * inv_l);
              w.w = pack_bf16x2(__uint_as_float(o[8 * i + 6]) * inv_l, __uint_as_float(o[8 * i + 7]) * inv_l);
              // 128B swizzle of the box: 16-byte chunk index ^ (row & 7); the box base is 1024-aligned and lane == row
              *reinterpret_cast<uint4*>(stage + (c >> 1) * (32 * 128) + lane * 128 + ((((c & 1) * 4 + i) ^ (lane & 7)) << 4)) = w;
            }
          }
          tc_fence_before();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
#pragma unroll
            for (int c = 0; c < C::SUBV; ++c)
              tma_store_3d(&map_o, stage + c * (32 * 128), c * 64, it.h << pack, it.seq0 + ((it.q0 + t * BQ + qd * 32) >> pack));
            tma_store_commit();
            mbar_arrive(&o_free[t]);
          }
        }
      }
      if (!staged) {
        const int dv = EXPANDED ? vdim : DV;
        bf16* orow = out + (size_t)token * ldo + head * dv;
#pragma unroll
        for (int c = 0; c < DV / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32b_x32(tO + c * 32, o);
          tmem_ld_wait();
          if (live) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (EXPANDED && c * 32 + i * 8 >= dv) break;  // vdim is a multiple of 8
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(o[8 * i + 0]) * inv_l, __uint_as_float(o[8 * i + 1]) * inv_l);
              w.y = pack_bf16x2(__uint_as_float(o[8 * i + 2]) * inv_l, __uint_as_float(o[8 * i + 3]) * inv_l);
              w.z = pack_bf16x2(__uint_as_float(o[8 * i + 4]) * inv_l, __uint_as_float(o[8 * i + 5]) * inv_l);
              w.w = pack_bf16x2(__uint_as_float(o[8 * i + 6]) * inv_l, __uint_as_float(o[8 * i + 7]) * inv_l);
              *reinterpret_cast<uint4*>(orow + c * 32 + i * 8) = w;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&o_free[t]);
      }
      jt += nt;
    }
    if constexpr (C::STAGE_O) {
      if (lane == 0) tma_store_wait_all<0>();  // the bulk stores read this CTA's shared memory: finish them before exit
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

inline int paged_only(int v, bool paged) { return paged ? v : 0; }
int device_sms() {
  static int num_sms = 0;
  if (num_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return num_sms;
}
// Packed launches that sort their items: those whose q pairs differ enough for the order to matter, by what the host knows of the lengths
// (us plain / sorted, 12 heads of 64 or 32 of 128 columns):
//   - sequences of two q pairs and more, of a kv tile and more on average (200 sequences of 25 to 200 tokens 195 / 209, one of 300 beside 199 of
//     50 138 / 149);
//   - empty (sequence, position) slots: a tenth of all, a fifth where the longest has only two or three pairs (16 sequences of 375 to 500
//     62 / 66, of 1125 to 1500 129 / 122);
//   - more items than SMs, twice as many there (3 sequences of 37 to 300 12.4 / 14.5, of 75 to 600 20.3 / 20.5, of 187 to 1500 53 / 31).
// Gains are 20 % on average over such launches.  The indices have to fit the order's entries (order_fits).
int q_pairs(const AttnPrefillArgs& a, int pack) { return (int)((((long long)a.max_seqlen << pack) + QPAIR - 1) / QPAIR); }
bool wants_order(const AttnPrefillArgs& a, int pack, int sms) {
  const int pairs = q_pairs(a, pack);
  if (a.B <= 1 || a.B > 256 || pairs < 2 || ((long long)a.T << pack) < (long long)BKV * a.B) return false;
  const bool short_ones = pairs <= 3;
  return (long long)pairs * a.B * (a.Hq >> pack) > (short_ones ? 2ll : 1ll) * sms && a.T < (short_ones ? 0.8 : 0.9) * (double)a.B * a.max_seqlen;
}
// (for sure: the host knows no more of the rows than that a sequence's last pair may be cut short)
bool order_fits(const AttnPrefillArgs& a, int pack) { return q_pairs(a, pack) <= 255 && ((long long)a.T << pack) / QPAIR + a.B <= kMaxRows; }
template <int D, bool PAGED, int ORDER>
cudaError_t launch(cudaStream_t stream, const AttnPrefillArgs& a, int pack) {
  constexpr int SRC = PAGED ? KV_PAGED : KV_PACKED;
  using C = ACfg<D, D, SRC>;
  CUtensorMap mq, mk, mv, mo;
  const uint64_t hd = (uint64_t)D * 2;
  const uint32_t heads = 1u << pack;
  if (!make_tmap_3d(&mo, a.out, TM_BF16, D, a.Hq, a.T, hd, (uint64_t)a.ldo * 2, 64, heads, 32 >> pack)) return cudaErrorInvalidValue;
  if (!make_tmap_3d(&mq, a.q, TM_BF16, D, a.Hq, a.T, hd, (uint64_t)a.ldq * 2, 64, heads, BQ >> pack)) return cudaErrorInvalidValue;
  if (PAGED) {
    // pool plane = [page][kv head][64 positions][D]: one 3-D block per (page, kv head), as in the decode kernel
    const uint64_t blocks = (uint64_t)a.num_pages * a.Hkv;
    if (!make_tmap_3d(&mk, a.k_cache, TM_BF16, D, 64, blocks, (uint64_t)D * 2, (uint64_t)64 * D * 2, 64, 64, 1)) return cudaErrorInvalidValue;
    if (!make_tmap_3d(&mv, a.v_cache, TM_BF16, D, 64, blocks, (uint64_t)D * 2, (uint64_t)64 * D * 2, 64, 64, 1)) return cudaErrorInvalidValue;
  } else {
    if (!make_tmap_2d(&mk, a.k, TM_BF16, (uint64_t)a.Hkv * D, (uint64_t)a.T, (uint64_t)a.ldk * 2, 64, BKV)) return cudaErrorInvalidValue;
    if (!make_tmap_2d(&mv, a.v, TM_BF16, (uint64_t)a.Hkv * D, (uint64_t)a.T, (uint64_t)a.ldv * 2, 64, BKV)) return cudaErrorInvalidValue;
  }
  auto kern = attn_prefill_kernel<D, D, SRC, ORDER>;
  const int max_q_pairs = q_pairs(a, pack);
  const long long items = (long long)max_q_pairs * a.B * (a.Hq >> pack);
  const int sms = effective_sms(device_sms());  // hb_engine_cfg.sm_budget
  const int grid = (int)std::min<long long>(ORDER == ORDER_SPLIT && 2 * items <= sms ? 2 * items : items, sms);
  const float scale_log2 = a.scale * 1.4426950408889634f;
  return launch_k(kern, dim3(grid), dim3(kThreads), ORDER == ORDER_SORTED ? C::SMEM_SORTED : C::SMEM, stream, true, mq, mk, mv, mo, a.out, a.ldo, a.cu_seqlens, a.B, a.Hq,
                  a.Hq / a.Hkv, a.causal, scale_log2, max_q_pairs, a.kv_lens, a.page_table, a.max_pages, a.Hkv,
                                            paged_only(a.block_mask, PAGED), a.unit_sink, a.head_gate, a.ldg,
                                            paged_only(a.window, PAGED), a.softcap > 0.f ? a.scale / a.softcap : 0.f,
                                            a.softcap > 0.f ? a.softcap * 1.4426950408889634f : 0.f, a.sink, mq, mk, AttnRuns{}, D, pack);
}

// latent attention over expanded rows
template <int DK, int DV>
cudaError_t launch_expanded(cudaStream_t stream, const AttnExpandedArgs& a) {
  using C = ACfg<DK, DV, KV_EXPANDED>;
  CUtensorMap mq, mqr, mk, mkr, mv;
  const uint64_t hd = (uint64_t)(a.nope + a.rot) * 2, H = a.H, T = a.T, rows = a.rows;
  if (!make_tmap_3d(&mq, a.q, TM_BF16, a.nope, H, T, hd, (uint64_t)a.ldq * 2, 64, 1, BQ)) return cudaErrorInvalidValue;
  if (!make_tmap_3d(&mqr, a.q + a.nope, TM_BF16, a.rot, H, T, hd, (uint64_t)a.ldq * 2, 64, 1, BQ)) return cudaErrorInvalidValue;
  if (!make_tmap_3d(&mk, a.k, TM_BF16, a.nope, H, rows, (uint64_t)a.nope * 2, (uint64_t)a.ldkv * 2, 64, 1, BKV)) return cudaErrorInvalidValue;
  if (!make_tmap_3d(&mv, a.v, TM_BF16, a.vdim, H, rows, (uint64_t)a.vdim * 2, (uint64_t)a.ldkv * 2, 64, 1, BKV)) return cudaErrorInvalidValue;
  if (!make_tmap_2d(&mkr, a.k_rot, TM_BF16, a.rot, rows, (uint64_t)a.ldkr * 2, 64, BKV)) return cudaErrorInvalidValue;
  auto kern = attn_prefill_kernel<DK, DV, KV_EXPANDED, ORDER_PLAIN>;
  int longest = 0;
  for (int i = 0; i < a.runs.n; ++i) longest = std::max(longest, a.runs.len[i]);
  const int max_q_pairs = (longest + QPAIR - 1) / QPAIR;
  const long long items = (long long)max_q_pairs * a.runs.n * a.H;
  int dev = 0, num_sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = (int)std::min<long long>(items, effective_sms(num_sms));
  return launch_k(kern, dim3(grid), dim3(kThreads), C::SMEM, stream, true, mq, mk, mv, mq, a.out, a.ldo, nullptr, a.runs.n, a.H, 1, 1,
                  a.scale * 1.4426950408889634f, max_q_pairs, nullptr, nullptr, 0, a.H, 0, 0, a.head_gate, a.ldg, a.window, 0.f, 0.f, a.sink, mqr, mkr,
                  a.runs, a.vdim, 0);
}

// ---------------------------------------------------------------- test-only on-device checker
__global__ void attn_naive_kernel(const bf16* q, int ldq, const bf16* k, int ldk, const bf16* v, int ldv, float* out,
                                  int ldo, const int32_t* cu, int Hq, int group, int D, int causal, float scale) {
  const int b = blockIdx.z, h = blockIdx.y;
  const int seq0 = cu[b], len = cu[b + 1] - seq0;
  const int qi = blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= len) return;
  const int kvh = h / group;
  const bf16* qr = q + (size_t)(seq0 + qi) * ldq + h * D;
  float m = -INFINITY, l = 0.f;
  float acc[128];
  for (int d = 0; d < D; ++d) acc[d] = 0.f;
  const int last = causal ? qi : len - 1;
  for (int j = 0; j <= last; ++j) {
    const bf16* kr = k + (size_t)(seq0 + j) * ldk + kvh * D;
    float s = 0.f;
    for (int d = 0; d < D; ++d) s += __bfloat162float(qr[d]) * __bfloat162float(kr[d]);
    s *= scale;
    const float mn = fmaxf(m, s);
    const float f = expf(m - mn), p = expf(s - mn);
    const bf16* vr = v + (size_t)(seq0 + j) * ldv + kvh * D;
    for (int d = 0; d < D; ++d) acc[d] = acc[d] * f + p * __bfloat162float(vr[d]);
    l = l * f + p;
    m = mn;
  }
  for (int d = 0; d < D; ++d) out[(size_t)(seq0 + qi) * ldo + h * D + d] = acc[d] / l;
}

}  // namespace

cudaError_t attn_prefill_init() {
  cudaError_t e;
#define HB_ATTR(D_, P_, S_)                                                                                      \
  if ((e = cudaFuncSetAttribute(attn_prefill_kernel<D_, D_, P_, S_>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                S_ == ORDER_SORTED ? ACfg<D_, D_, P_>::SMEM_SORTED : ACfg<D_, D_, P_>::SMEM)) != cudaSuccess)     \
    return e;
#define HB_ATTRD(D_)                                                                                                        \
  HB_ATTR(D_, KV_PACKED, ORDER_PLAIN) HB_ATTR(D_, KV_PACKED, ORDER_SPLIT) HB_ATTR(D_, KV_PACKED, ORDER_SORTED)               \
  HB_ATTR(D_, KV_PAGED, ORDER_PLAIN) HB_ATTR(D_, KV_PAGED, ORDER_SPLIT)
  HB_ATTRD(128) HB_ATTRD(64)
#undef HB_ATTRD
#undef HB_ATTR
#define HB_ATTRX(K_, V_)                                                                                                  \
  if ((e = cudaFuncSetAttribute(attn_prefill_kernel<K_, V_, KV_EXPANDED, ORDER_PLAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                ACfg<K_, V_, KV_EXPANDED>::SMEM)) != cudaSuccess)                                        \
    return e;
  HB_ATTRX(128, 64) HB_ATTRX(128, 128) HB_ATTRX(192, 64) HB_ATTRX(192, 128)
#undef HB_ATTRX
  return cudaSuccess;
}

// Query heads (a power of two, given as its logarithm) that share a kv head and the rows of a tile.  Packed tiles span fewer tokens, so less
// of their diagonal is masked and less of a last tile is empty: 6 prompts of 300 to 3000 tokens, 32 heads over 8: 173 kv tiles per SM -> 148, 223 ->
// 193 us; 8 of about 1000 97 -> 87.  They are also fewer: the packing that leaves the SMs the least to do one after the other is taken (a lone q
// tile takes about 4/5 of a pair's time; 100 rows over 4000 keys 53 us unpacked, 61 by four; one prompt of 128 tokens, 128 columns 8.7 | 10.4).
// A wide packing has more q pairs, and where they are more than the order holds, the order is worth more than the packing.  us with 1 | 2 | 4 | .. heads
// per tile, [ ] in plain order: 32 heads over 8, 16 prompts of 500 to 4500 tokens 1037 | 978 | [1045], 6 of 2000 to 11300 2732 | 2669 | [3165], 30 of 500
// to 6200 3844 | [3827] | [4048], 20 of 500 to 5000 1971 | 1875 | [1840]; 32 over 1, 8 of 200 to 1800 157 | 134 | 128 | 126 | 122 | [165], 10 of
// 500 to 3500 476 | 433 | 394 | [417] | [480] | [431].
static bool splits(long long pairs, int sms) { return pairs <= INT_MAX / 2 && first_split((int)pairs, (int)std::min<long long>(2 * pairs, sms)) < pairs; }
AttnPrefillPlan attn_prefill_plan(const AttnPrefillArgs& a, int sms) {
  const int group = a.Hq / a.Hkv;
  const bool paged = a.k_cache != nullptr;
  int best = 0;
  long long least = 0;
  for (int p = 0; p <= 5 && group % (1 << p) == 0; ++p) {
    if (!paged && p > 0 && wants_order(a, p, sms) && !order_fits(a, p) && order_fits(a, 0)) break;
    const long long rows = (long long)a.max_seqlen << p, items = (rows + QPAIR - 1) / QPAIR * a.B * (a.Hq >> p);
    const bool halves = rows > BQ && (paged || !wants_order(a, p, sms)) && splits(items, sms);
    const long long cost = (items + sms - 1) / sms * (rows <= BQ ? 40 : 50) - (halves ? 9 : 0);  // (a last round of lone q tiles, after those that are lone anyway)
    if (p == 0 || cost <= least) {
      best = p;
      least = cost;
    }
  }
  // (launches that may or may not fit: the kernel counts)
  return {best, !paged && wants_order(a, best, sms) && q_pairs(a, best) <= 255};
}

cudaError_t attn_prefill(cudaStream_t stream, const AttnPrefillArgs& a) {
  if (a.B <= 0 || a.T <= 0) return cudaSuccess;
  if (a.Hq % a.Hkv) return cudaErrorInvalidValue;
  const bool paged = a.k_cache != nullptr;
  if ((a.ldq % 8) || (a.ldo % 8) || (!paged && ((a.ldk % 8) || (a.ldv % 8)))) return cudaErrorInvalidValue;
  if (a.block_mask < 0 || (a.block_mask > 0 && (!paged || !a.causal))) return cudaErrorInvalidValue;
  if (a.window < 0 || (a.window > 0 && (!paged || !a.causal || a.block_mask > 0))) return cudaErrorInvalidValue;
  const int sms = effective_sms(device_sms());
  if (sms <= 0) return cudaErrorNoDevice;
  if (paged) {
    if (!a.v_cache || !a.page_table || !a.kv_lens || a.max_pages <= 0 || a.num_pages <= 0 || a.page_size != 64) return cudaErrorInvalidValue;
  }
  const auto [pack, sorted] = attn_prefill_plan(a, sms);
  // (sequences of one lone q tile have nothing to split)
  const bool split = ((long long)a.max_seqlen << pack) > BQ && splits((long long)q_pairs(a, pack) * a.B * (a.Hq >> pack), sms);
#define HB_LAUNCH(D_)                                                                                                                              \
  if (paged) return split ? launch<D_, true, ORDER_SPLIT>(stream, a, pack) : launch<D_, true, ORDER_PLAIN>(stream, a, pack);                       \
  return sorted ? launch<D_, false, ORDER_SORTED>(stream, a, pack)                                                                                 \
         : split ? launch<D_, false, ORDER_SPLIT>(stream, a, pack) : launch<D_, false, ORDER_PLAIN>(stream, a, pack)
  if (a.D == 128) { HB_LAUNCH(128); }
  if (a.D == 64) { HB_LAUNCH(64); }
#undef HB_LAUNCH
  return cudaErrorInvalidValue;
}

bool attn_expanded_ok(int nope, int rot, int vdim) {
  return nope > 0 && rot > 0 && vdim > 0 && nope % 8 == 0 && rot % 8 == 0 && vdim % 8 == 0 && nope <= 128 && rot <= 64 && vdim <= 128;
}
cudaError_t attn_expanded(cudaStream_t stream, const AttnExpandedArgs& a) {
  if (a.runs.n <= 0) return cudaSuccess;
  if (!attn_expanded_ok(a.nope, a.rot, a.vdim) || a.H <= 0 || a.T <= 0 || a.rows <= 0 || a.runs.n > AttnRuns::kMax || a.window < 0) return cudaErrorInvalidValue;
  if (a.ldq % 8 || a.ldkv % 8 || a.ldkr % 8 || a.ldo % 8) return cudaErrorInvalidValue;
  const bool wide = a.nope > 64;
  if (a.vdim <= 64) return wide ? launch_expanded<192, 64>(stream, a) : launch_expanded<128, 64>(stream, a);
  return wide ? launch_expanded<192, 128>(stream, a) : launch_expanded<128, 128>(stream, a);
}

#ifdef HB_ATTN_TRACE
void attn_trace_dump() {
  static unsigned long long h[8][4096];
  int n[8];
  cudaMemcpyFromSymbol(h, g_attn_trace, sizeof(h));
  cudaMemcpyFromSymbol(n, g_attn_trace_n, sizeof(n));
  for (int e = 0; e < 7; ++e) {
    printf("TRACE %d %d:", e, n[e]);
    for (int i = 0; i < n[e] && i < 400; ++i) printf(" %llu", h[e][i] - h[2][0]);
    printf("\n");
  }
}
#endif

cudaError_t attn_naive_check(cudaStream_t stream, const AttnPrefillArgs& a, float* out_f32) {
  dim3 grid((a.max_seqlen + 63) / 64, a.Hq, a.B);
  attn_naive_kernel<<<grid, 64, 0, stream>>>(a.q, a.ldq, a.k, a.ldk, a.v, a.ldv, out_f32, a.ldo, a.cu_seqlens, a.Hq,
                                             a.Hq / a.Hkv, a.D, a.causal, a.scale);
  return cudaGetLastError();
}

}  // namespace hb
