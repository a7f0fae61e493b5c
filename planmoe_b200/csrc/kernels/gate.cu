// Fused gate kernels (sm_100a): softmax + top-k + slot-location scan + slot map + GShard loss.
//
// One pass over the logits replaces the reference's chain of ~20 ATen launches plus its
// Blelloch-scan kernel (PlanMoE/impls/fast_dispatch.py:143-190, impls/losses.py:12-19,
// custom/custom_kernel.cpp:338-383).  Slot ordering is the reference's: within an expert, every
// k-th pick ranks after all (k-1)-th picks, and picks of equal k rank by token index.
//
//   gate_stats   per token: softmax (or scores taken as they are), top-k (ties -> lower expert id, NaN before every
//                number), raw gate scores; per block: (k, expert) histograms, in-block ranks, per-expert score sums;
//                marks every slot of the map as empty.
//   gate_assign  per block: base offsets from the histograms of preceding blocks / lower k,
//                locations, normalised gates, slot map; block 0 also reduces the loss.
//   gate_bwd     per token: d(logits) from d(gates) and d(l_aux) (softmax recomputed).
//   cumsum_sub_one  stand-alone column-wise inclusive cumsum minus one of an int32 [S, E] mask.
//
// Everything is reduced in a fixed order: results are bit-reproducible run to run.

#include "planmoe.h"
#include "kernels/common.cuh"
#include "kernels/launch.cuh"

namespace planmoe {

// Threads (= tokens) per block.  The assign kernel of every block sums the histograms of the blocks before it, so half as
// many blocks is a quarter of that work: with 64 threads it took 14 us for 16384 tokens and 8 experts.
constexpr int kGateThreads = 128;
constexpr int kGateWarps = kGateThreads / 32;
constexpr int kMaxE = 64;   // experts handled by the fused gate (per-thread register row)
constexpr int kMaxK = 4;

template <class T, int ME>
__device__ __forceinline__ void load_row(const T* row, int E, float* v) {
#pragma unroll
  for (int e = 0; e < ME; ++e) v[e] = (e < E) ? to_f32(row[e]) : -INFINITY;
}

template <int ME>
__device__ __forceinline__ void softmax_row(float* p, int E) {
  float mx = -INFINITY;
#pragma unroll
  for (int e = 0; e < ME; ++e) mx = fmaxf(mx, p[e]);
  float sum = 0.f;
#pragma unroll
  for (int e = 0; e < ME; ++e) { p[e] = (e < E) ? expf(p[e] - mx) : 0.f; sum += p[e]; }
  const float inv = 1.f / sum;
#pragma unroll
  for (int e = 0; e < ME; ++e) p[e] *= inv;
}

template <class T, int ME, bool SCORES>
__global__ void __launch_bounds__(kGateThreads)
gate_stats_kernel(const T* __restrict__ logits, int S, int E, int K, int nblk,
                  int* __restrict__ idx,          // [K][S]
                  float* __restrict__ raw_gate,   // [K][S] un-normalised softmax score of pick k
                  int* __restrict__ rank_in_blk,  // [K][S]
                  int* __restrict__ blk_count,    // [K][E][nblk]
                  float* __restrict__ blk_score,  // [E][nblk]  sum of softmax scores
                  int* __restrict__ slot_map, long long slots,
                  const int* __restrict__ perm)   // token at each position of the slot order, or null: token order
{
  chain_begin();
  __shared__ int warp_cnt[kGateWarps][kMaxK][kMaxE];
  __shared__ float score_sum[kGateWarps][kMaxE];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pos = blockIdx.x * kGateThreads + tid;
  const bool live = pos < S;
  const int t = live && perm != nullptr ? perm[pos] : pos;

  for (int i = tid; i < kGateWarps * kMaxK * kMaxE; i += kGateThreads) (&warp_cnt[0][0][0])[i] = 0;
  for (long long i = pos; i < slots; i += (long long)gridDim.x * kGateThreads) slot_map[i] = -1;
  __syncthreads();

  float p[ME];
  int pick[kMaxK];
  if (live) {
    load_row<T, ME>(logits + (size_t)t * E, E, p);
    if constexpr (!SCORES) softmax_row<ME>(p, E);
  } else {
#pragma unroll
    for (int e = 0; e < ME; ++e) p[e] = 0.f;
  }

  // per-expert score sums: warp shuffle reduce, fixed order
#pragma unroll
  for (int e = 0; e < ME; ++e) {
    if (e < E) {
      float s = warp_sum(p[e]);
      if (lane == 0) score_sum[warp][e] = s;
    }
  }

  unsigned long long taken = 0ull;
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K) break;                           // unrolled: the picks stay in registers
    int best = -1;                               // K <= E: one expert is always left
    float bv = 0.f;
#pragma unroll
    for (int e = 0; e < ME; ++e) {
      if (e < E && !((taken >> e) & 1ull) && (best < 0 || p[e] > bv || (isnan(p[e]) && !isnan(bv)))) { bv = p[e]; best = e; }
    }
    pick[k] = live ? best : -1;
    taken |= 1ull << best;
    if (live) {
      idx[(size_t)k * S + t] = best;
      raw_gate[(size_t)k * S + t] = bv;
    }
    // rank among the lanes of this warp that picked the same expert for this k
    const unsigned peers = __match_any_sync(0xffffffffu, pick[k]);
    const int r = __popc(peers & ((1u << lane) - 1u));
    if (live && r == 0) warp_cnt[warp][k][best] = __popc(peers);
    pick[k] = live ? (best | (r << 8)) : -1;    // stash the in-warp rank
  }
  __syncthreads();

#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K) break;                           // unrolled: the picks stay in registers
    if (!live) break;
    const int e = pick[k] & 0xff, r = pick[k] >> 8;
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_cnt[w][k][e];
    rank_in_blk[(size_t)k * S + t] = before + r;
  }
  for (int i = tid; i < K * E; i += kGateThreads) {
    const int k = i / E, e = i - k * E;
    int c = 0;
    for (int w = 0; w < kGateWarps; ++w) c += warp_cnt[w][k][e];
    blk_count[(size_t)i * nblk + blockIdx.x] = c;
  }
  for (int e = tid; e < E; e += kGateThreads) {
    float s = 0.f;
    for (int w = 0; w < kGateWarps; ++w) s += score_sum[w][e];
    blk_score[(size_t)e * nblk + blockIdx.x] = s;
  }
}

__global__ void __launch_bounds__(kGateThreads)
gate_assign_kernel(int S, int E, int K, int C, int normalize, float eps,
                   const int* __restrict__ idx, const float* __restrict__ raw_gate,
                   const int* __restrict__ rank_in_blk, const int* __restrict__ blk_count,
                   const float* __restrict__ blk_score, int nblk,
                   int* __restrict__ loc, GatePtrs gates, int* __restrict__ slot_map,
                   int* __restrict__ top1_count,  // [E] tokens whose first pick is e
                   int* __restrict__ used,        // [E] slots of expert e that hold a token, or null
                   float* __restrict__ l_aux,     // [1]
                   __nv_bfloat16* __restrict__ l_aux_bf16,   // [1] or null
                   const int* __restrict__ perm,
                   int* __restrict__ copies)      // [3][K][S]: idx, loc and gates (fp32) once more, or null
{
  chain_begin();
  __shared__ int base[kMaxK][kMaxE];
  __shared__ float red[kMaxE];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.x;
  // the token's own values are on their way while the histograms are summed
  const int pos = b * kGateThreads + tid;
  const int t = pos < S ? (perm != nullptr ? perm[pos] : pos) : 0;
  int pick[kMaxK], rank[kMaxK];
  float g[kMaxK];
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K || pos >= S) break;
    pick[k] = idx[(size_t)k * S + t];
    rank[k] = rank_in_blk[(size_t)k * S + t];
    g[k] = raw_gate[(size_t)k * S + t];
  }
  // base[k][e] = picks of expert e that rank before this block's k-th picks: every block's picks of a lower k,
  // then the k-th picks of the blocks before this one.  One warp per (k, e), lanes strided over that list.
  for (int i = warp; i < K * E; i += kGateWarps) {
    const int k = i / E, e = i - k * E;
    int acc = 0;
    for (int kk = 0; kk <= k; ++kk) {
      const int* row = blk_count + (size_t)(kk * E + e) * nblk;
      const int n = kk < k ? nblk : b;
      for (int bb = lane; bb < n; bb += 32) acc += row[bb];
    }
    acc = __reduce_add_sync(0xffffffffu, acc);
    if (lane == 0) base[k][e] = acc;
  }
  __syncthreads();

  if (pos < S) {
    const bool norm = normalize && K > 1;
    float denom = 0.f;
#pragma unroll
    for (int k = 0; k < kMaxK; ++k) denom += k < K ? g[k] : 0.f;
    denom = denom < eps ? eps : denom;             // like torch.clamp: a NaN stays one
#pragma unroll
    for (int k = 0; k < kMaxK; ++k) {
      if (k >= K) break;
      const int l = base[k][pick[k]] + rank[k];
      loc[(size_t)k * S + t] = l;
      const float gate = norm ? g[k] / denom : g[k];
      gates.p[k][t] = gate;
      if (copies != nullptr) {
        copies[(size_t)k * S + t] = pick[k];
        copies[(size_t)(K + k) * S + t] = l;
        copies[(size_t)(2 * K + k) * S + t] = __float_as_int(gate);
      }
      if (slot_map != nullptr && l < C) slot_map[(size_t)pick[k] * C + l] = t * K + k;
    }
  }

  if (b == 0) {
    // l_aux = E / S^2 * sum_e (sum_t score[t][e]) * (#tokens with top-1 == e); one warp per expert, lanes strided
    // over the blocks, lane sums combined by a shuffle tree: a fixed order
    for (int e = warp; e < E; e += kGateWarps) {
      float s = 0.f;
      int c = 0;
      for (int bb = lane; bb < nblk; bb += 32) {
        s += blk_score[(size_t)e * nblk + bb];
        c += blk_count[(size_t)e * nblk + bb];
      }
      s = warp_sum(s);
      c = __reduce_add_sync(0xffffffffu, c);
      if (used != nullptr) {
        int n = 0;
        for (int kk = 1; kk < K; ++kk)
          for (int bb = lane; bb < nblk; bb += 32) n += blk_count[(size_t)(kk * E + e) * nblk + bb];
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) used[e] = min(C, c + n);
      }
      if (lane == 0) {
        top1_count[e] = c;
        red[e] = s * (float)c;
      }
    }
    __syncthreads();
    if (tid == 0) {
      float acc = 0.f;
      for (int e = 0; e < E; ++e) acc += red[e];
      acc = acc * (float)E / ((float)S * (float)S);
      l_aux[0] = acc;
      if (l_aux_bf16 != nullptr) l_aux_bf16[0] = __float2bfloat16_rn(acc);
    }
  }
}

// No histograms here, so that blocks may be small, which spreads few tokens with many experts over more SMs: 128 threads take
// 4.6, 6.0 and 20.9 us for 8192 tokens with 8, 16 and 64 experts (top-2, 2, 4), 32 threads 4.5, 5.6 and 17.1; from 16384 tokens
// on the two differ by less than 4 % either way.
constexpr int kGateBwdThreads = 32;
template <class T, int ME, bool SCORES>
__global__ void __launch_bounds__(kGateBwdThreads)
gate_bwd_kernel(const T* __restrict__ logits, int S, int E, int K, int normalize, float eps,
                const int* __restrict__ idx, GatePtrs dgates,                     // K rows of S, null = zeros
                const float* __restrict__ dl_aux,                                 // [1] or null
                const __nv_bfloat16* __restrict__ dl_aux_bf16,                    // [1] or null
                const int* __restrict__ top1_count, T* __restrict__ dlogits) {
  chain_begin();
  const int t = blockIdx.x * kGateBwdThreads + threadIdx.x;
  if (t >= S) return;
  float p[ME];
  if (SCORES && K == 0) {                         // the loss alone: its gradient does not depend on the scores
#pragma unroll
    for (int e = 0; e < ME; ++e) p[e] = 0.f;
  } else {
    load_row<T, ME>(logits + (size_t)t * E, E, p);
    if constexpr (!SCORES) softmax_row<ME>(p, E);
  }

  // d(score): loss part for every expert, gate part for the picked ones
  const float dl = dl_aux ? dl_aux[0] : dl_aux_bf16 ? __bfloat162float(dl_aux_bf16[0]) : 0.f;
  const float lw = dl * (float)E / ((float)S * (float)S);
  int pk[kMaxK];
  float ds_pick[kMaxK];
  float denom = 0.f, dot = 0.f;
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K) break;                           // unrolled: the picks stay in registers
    pk[k] = idx[(size_t)k * S + t];
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < ME; ++e) s = (e == pk[k]) ? p[e] : s;
    ds_pick[k] = s;    // temporarily the score
    denom += s;
  }
  const bool norm = normalize && K > 1;
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K) break;                           // unrolled: the picks stay in registers
    const float dg = dgates.p[k] ? dgates.p[k][t] : 0.f;
    dot += dg * ds_pick[k];
  }
#pragma unroll
  for (int k = 0; k < kMaxK; ++k) {
    if (k >= K) break;                           // unrolled: the picks stay in registers
    const float dg = dgates.p[k] ? dgates.p[k][t] : 0.f;
    if (norm) {
      if (denom < eps) ds_pick[k] = dg / eps;
      else ds_pick[k] = dg / denom - dot / (denom * denom);
    } else {
      ds_pick[k] = dg;
    }
  }
  float ds[ME];
  float inner = 0.f;
#pragma unroll
  for (int e = 0; e < ME; ++e) {
    float d = 0.f;
    if (e < E) {
      d = lw * (float)top1_count[e];
#pragma unroll
      for (int k = 0; k < kMaxK; ++k) d += (k < K && pk[k] == e) ? ds_pick[k] : 0.f;
    }
    ds[e] = d;
    inner += d * p[e];
  }
  T* out = dlogits + (size_t)t * E;
#pragma unroll
  for (int e = 0; e < ME; ++e)
    if (e < E) out[e] = from_f32<T>(SCORES ? ds[e] : p[e] * (ds[e] - inner));
}

template <class T, bool SCORES>
void launch_gate_forward(const T* logits, int S, int E, int K, int C, bool normalize, float eps,
                         int* idx, int* loc, GatePtrs gates, float* raw_gate, int* slot_map,
                         int* top1_count, int* used, float* l_aux, int* ws_rank, int* ws_blk_count,
                         float* ws_blk_score, cudaStream_t stream, const int* perm, void* l_aux_bf16, int* copies) {
  const int nblk = (S + kGateThreads - 1) / kGateThreads;
  auto stats = E <= 8 ? gate_stats_kernel<T, 8, SCORES> : E <= 16 ? gate_stats_kernel<T, 16, SCORES>
             : E <= 32 ? gate_stats_kernel<T, 32, SCORES> : gate_stats_kernel<T, 64, SCORES>;
  launch_chained(stats, nblk, kGateThreads, 0, stream, logits, S, E, K, nblk, idx, raw_gate, ws_rank, ws_blk_count, ws_blk_score,
                                           slot_map, slot_map != nullptr ? (long long)E * C : 0, perm);
  launch_chained(gate_assign_kernel, nblk, kGateThreads, 0, stream, S, E, K, C, normalize ? 1 : 0, eps, idx,
                                                      raw_gate, ws_rank, ws_blk_count, ws_blk_score,
                                                      nblk, loc, gates, slot_map, top1_count, used, l_aux,
                                                      reinterpret_cast<__nv_bfloat16*>(l_aux_bf16), perm, copies);
}

template <class T, bool SCORES>
void launch_gate_backward(const T* logits, int S, int E, int K, bool normalize, float eps,
                          const int* idx, GatePtrs dgates, const float* dl_aux,
                          const int* top1_count, T* dlogits, cudaStream_t stream, const void* dl_aux_bf16) {
  const int nblk = (S + kGateBwdThreads - 1) / kGateBwdThreads;
  auto bwd = E <= 8 ? gate_bwd_kernel<T, 8, SCORES> : E <= 16 ? gate_bwd_kernel<T, 16, SCORES>
           : E <= 32 ? gate_bwd_kernel<T, 32, SCORES> : gate_bwd_kernel<T, 64, SCORES>;
  launch_chained(bwd, nblk, kGateBwdThreads, 0, stream, logits, S, E, K, normalize ? 1 : 0, eps, idx, dgates, dl_aux,
                                         reinterpret_cast<const __nv_bfloat16*>(dl_aux_bf16), top1_count, dlogits);
}

int gate_workspace_blocks(int S) { return (S + kGateThreads - 1) / kGateThreads; }

// ---- batch-prioritised routing: the order in which tokens claim slots -------------------------------
// The reference sorts tokens by the score of their best expert, highest first (importance = -max softmax
// score, PlanMoE/impls/fast_dispatch.py:135-138,153-154), and scans locations in that order.  Here the order
// comes from a rank: key[t] = max_e softmax(logits[t])[e] = 1 / sum_e exp(l[t][e] - max_e l[t]);
// rank[t] = number of tokens that go before t (larger key, or the same key and a lower index), perm = rank^-1.
// Few tokens: S^2 comparisons on fp32 keys staged through shared memory.  Many: sorted tiles.  Both are exact, stable and the same
// work whatever the keys are.  (us for 4096, 16384 and 65536 tokens: counting 14 - 16, 46 - 48, 500; tiles 12 - 20, 27 - 35, 95 - 128,
// for two and sixteen experts.)
constexpr int kSortTokens = 8192;

template <class T>
__global__ void __launch_bounds__(256)
importance_key_kernel(const T* __restrict__ logits, int S, int E, float* __restrict__ key) {
  chain_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= S) return;
  const T* row = logits + (size_t)t * E;
  float mx = -INFINITY;
  for (int e = 0; e < E; ++e) mx = fmaxf(mx, to_f32(row[e]));
  float sum = 0.f;
  for (int e = 0; e < E; ++e) sum += expf(to_f32(row[e]) - mx);
  const float k = 1.f / sum;
  key[t] = k > 0.f ? k : 0.f;                     // NaN scores go last: ranks stay a permutation
}

// 32 tokens per CTA, eight threads per token: each thread counts over an eighth of every key tile, the eight
// counts are added by shuffles.  Ties need the index only in the tile that holds the token: every key of an earlier tile
// goes before it from equality on, every key of a later one only when it is larger, so that a comparison is one test and
// one add, on four keys per load.  A tile of 4096 keys leaves few barriers.
constexpr int kCountTile = 4096;
__global__ void __launch_bounds__(256)
importance_count_kernel(const float* __restrict__ key, int S, int* __restrict__ rank, int* __restrict__ perm) {
  chain_begin();
  __shared__ __align__(16) float tile[kCountTile];
  const int part = threadIdx.x & 7;
  const int t0 = blockIdx.x * 32, t = t0 + (threadIdx.x >> 3);   // a CTA's tokens lie in one tile
  const float mine = t < S ? key[t] : 0.f;
  int before = 0;
  for (int base = 0; base < S; base += kCountTile) {
    __syncthreads();
    for (int i = threadIdx.x; i < kCountTile; i += blockDim.x) tile[i] = base + i < S ? key[base + i] : -INFINITY;
    __syncthreads();
    const int own = t0 - base;
    const int n = min(kCountTile, S - base);      // keys are positive: the padding behind the last one never counts
    if (own >= 0 && own < kCountTile) {
      for (int i = part; i < n; i += 8) before += (tile[i] > mine || (tile[i] == mine && base + i < t)) ? 1 : 0;
    } else if (own > 0) {
#pragma unroll 4
      for (int i = part * 4; i < n; i += 32) {    // an earlier tile is full
        const float4 k = *reinterpret_cast<const float4*>(tile + i);
        before += (k.x >= mine) + (k.y >= mine) + (k.z >= mine) + (k.w >= mine);
      }
    } else {
#pragma unroll 4
      for (int i = part * 4; i < n; i += 32) {
        const float4 k = *reinterpret_cast<const float4*>(tile + i);
        before += (k.x > mine) + (k.y > mine) + (k.z > mine) + (k.w > mine);
      }
    }
  }
  before += __shfl_xor_sync(0xffffffffu, before, 1);
  before += __shfl_xor_sync(0xffffffffu, before, 2);
  before += __shfl_xor_sync(0xffffffffu, before, 4);
  if (part == 0 && t < S) { rank[t] = before; perm[before] = t; }
}

// Key and index make one 64-bit word, so that no two are equal and smaller goes first.  Blocks sort tiles of 1024 words; a
// token's rank is then its place in its own tile plus, by binary search, how many words of every other tile are smaller.
constexpr int kSortTile = 1024;
constexpr int kSortThreads = kSortTile / 2;

template <class T>
__global__ void __launch_bounds__(kSortThreads)
importance_sort_kernel(const T* __restrict__ logits, int S, int E, unsigned long long* __restrict__ sorted) {
  chain_begin();
  __shared__ unsigned long long w[2][kSortTile];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t0 = blockIdx.x * kSortTile;
  // Two words a thread, 32 places apart: distances below 32 by shuffle, 32 in the thread, the ten larger ones in shared memory.
  const int i0 = warp * 64 + lane;
  unsigned long long x[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int t = t0 + i0 + 32 * h;
    x[h] = ~0ull;                                 // behind the last token: behind every token
    if (t < S) {
      const T* row = logits + (size_t)t * E;
      float mx = -INFINITY;
#pragma unroll 8
      for (int e = 0; e < E; ++e) mx = fmaxf(mx, to_f32(row[e]));
      float sum = 0.f;
#pragma unroll 8
      for (int e = 0; e < E; ++e) sum += expf(to_f32(row[e]) - mx);
      float k = 1.f / sum;
      k = k > 0.f ? k : 0.f;                      // NaN scores go last
      x[h] = ((unsigned long long)~__float_as_uint(k) << 32) | (unsigned)t;    // positive floats compare as their bits
    }
  }
  int buf = 0;
#pragma unroll
  for (int k = 2; k <= kSortTile; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      unsigned long long y[2];
      if (j == 32) {
        y[0] = x[1]; y[1] = x[0];
      } else if (j < 32) {
        y[0] = __shfl_xor_sync(0xffffffffu, x[0], j); y[1] = __shfl_xor_sync(0xffffffffu, x[1], j);
      } else {                                    // two buffers: one barrier a stage
        w[buf][i0] = x[0]; w[buf][i0 + 32] = x[1];
        __syncthreads();
        y[0] = w[buf][i0 ^ j]; y[1] = w[buf][(i0 + 32) ^ j];
        buf ^= 1;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + 32 * h;
        const bool smaller = ((i & j) == 0) == ((i & k) == 0);
        x[h] = (x[h] < y[h]) == smaller ? x[h] : y[h];
      }
    }
  }
  sorted[t0 + i0] = x[0];
  sorted[t0 + i0 + 32] = x[1];
}

constexpr int kRankThreads = 128;
__global__ void __launch_bounds__(kRankThreads)
importance_rank_kernel(const unsigned long long* __restrict__ sorted, int S, int* __restrict__ rank, int* __restrict__ perm) {
  chain_begin();
  const int i = blockIdx.x * kRankThreads + threadIdx.x;        // a place in a sorted tile: neighbours search alike
  const int tiles = (S + kSortTile - 1) / kSortTile, own = i / kSortTile;
  const unsigned long long word = sorted[i];
  if (word == ~0ull) return;
  int before = i - own * kSortTile;
#pragma unroll 8
  for (int tile = 0; tile < tiles; ++tile) {
    const unsigned long long* s = sorted + (size_t)tile * kSortTile;
    int n = 0;                                    // words of the tile that are smaller
#pragma unroll
    for (int step = kSortTile / 2; step > 0; step >>= 1) n += s[n + step - 1] < word ? step : 0;
    n += s[n] < word ? 1 : 0;
    before += tile == own ? 0 : n;
  }
  const int t = (int)(unsigned)word;
  rank[t] = before;
  perm[before] = t;
}

long long importance_workspace(int S) { return (long long)((S + kSortTile - 1) / kSortTile) * kSortTile; }

template <class T>
void launch_importance_order(const T* logits, int S, int E, unsigned long long* ws, int* rank, int* perm, cudaStream_t stream) {
  if (S <= 0) return;
  if (S < kSortTokens) {
    float* key = reinterpret_cast<float*>(ws);
    launch_chained(importance_key_kernel<T>, (S + 255) / 256, 256, 0, stream, logits, S, E, key);
    launch_chained(importance_count_kernel, (S + 31) / 32, 256, 0, stream, key, S, rank, perm);
    return;
  }
  const int tiles = (S + kSortTile - 1) / kSortTile;
  launch_chained(importance_sort_kernel<T>, tiles, kSortThreads, 0, stream, logits, S, E, ws);
  launch_chained(importance_rank_kernel, tiles * (kSortTile / kRankThreads), kRankThreads, 0, stream, ws, S, rank, perm);
}
template void launch_importance_order<float>(const float*, int, int, unsigned long long*, int*, int*, cudaStream_t);
template void launch_importance_order<__nv_bfloat16>(const __nv_bfloat16*, int, int, unsigned long long*, int*, int*, cudaStream_t);
template void launch_importance_order<__half>(const __half*, int, int, unsigned long long*, int*, int*, cudaStream_t);

// slot map of a permuted token order back to token ids: owner = position * K + k -> perm[position] * K + k
__global__ void remap_slot_map_kernel(int* __restrict__ slot_map, long long n, const int* __restrict__ perm, int K) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int o = slot_map[i];
  if (o >= 0) slot_map[i] = perm[o / K] * K + o % K;
}
void launch_remap_slot_map(int* slot_map, long long n, const int* perm, int K, cudaStream_t stream) {
  if (n > 0) remap_slot_map_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(slot_map, n, perm, K);
}

#define INSTANTIATE(T, SCORES)                                                                    \
  template void launch_gate_forward<T, SCORES>(const T*, int, int, int, int, bool, float, int*, int*,     \
                                               GatePtrs, float*, int*, int*, int*, float*, int*, int*, float*, \
                                               cudaStream_t, const int*, void*, int*);                    \
  template void launch_gate_backward<T, SCORES>(const T*, int, int, int, bool, float, const int*, GatePtrs, \
                                                const float*, const int*, T*, cudaStream_t, const void*);
INSTANTIATE(float, false)
INSTANTIATE(__nv_bfloat16, false)
INSTANTIATE(__half, false)
INSTANTIATE(float, true)

// ---- stand-alone cumsum - 1 -----------------------------------------------------------------
// Two passes over [S, E] int32: per-tile column sums, then each tile scans with the carried base.
constexpr int kScanRows = 128;

__global__ void cumsum_tile_sums_kernel(const int* __restrict__ x, int S, int E, int* __restrict__ tile_sum) {
  const int e = blockIdx.y * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int r0 = blockIdx.x * kScanRows;
  int acc = 0;
  for (int r = r0; r < min(r0 + kScanRows, S); ++r) acc += x[(size_t)r * E + e];
  tile_sum[(size_t)blockIdx.x * E + e] = acc;
}

__global__ void cumsum_apply_kernel(const int* __restrict__ x, int S, int E,
                                    const int* __restrict__ tile_sum, int* __restrict__ out) {
  const int e = blockIdx.y * blockDim.x + threadIdx.x;
  if (e >= E) return;
  int acc = -1;
  for (int b = 0; b < (int)blockIdx.x; ++b) acc += tile_sum[(size_t)b * E + e];
  const int r0 = blockIdx.x * kScanRows;
  for (int r = r0; r < min(r0 + kScanRows, S); ++r) {
    acc += x[(size_t)r * E + e];
    out[(size_t)r * E + e] = acc;
  }
}

void launch_cumsum_sub_one(const int* x, int* out, int* tile_sum, int S, int E, cudaStream_t stream) {
  const int tiles = (S + kScanRows - 1) / kScanRows;
  const int threads = E < 128 ? ((E + 31) / 32) * 32 : 128;
  dim3 grid(tiles, (E + threads - 1) / threads);
  cumsum_tile_sums_kernel<<<grid, threads, 0, stream>>>(x, S, E, tile_sum);
  cumsum_apply_kernel<<<grid, threads, 0, stream>>>(x, S, E, tile_sum, out);
}
int cumsum_tiles(int S) { return (S + kScanRows - 1) / kScanRows; }

}  // namespace planmoe
