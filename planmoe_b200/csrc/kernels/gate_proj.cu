// The linear gate's projection and its gradients (sm_100a), on bf16 tokens as they are.
//
//   gate_project   logits[t][e] = <x[t], w[e]>
//   gate_wgrad     dw[e][m] = sum_t dlogits[t][e] * x[t][m], as partial sums over chunks of tokens
//   gather_gate    dx[t] = sum_k (gate *) slot row of pick k + sum_e dlogits[t][e] * w[e]: the two parts of a token's
//                  gradient in one pass, rounded once
//
// The composition that they take the place of (x.float(), an fp32 library GEMM, its two gradient GEMMs, a cast and an
// add) read and wrote the [tokens, model_dim] matrix nine times, six of them in fp32: 728 us of a training step of 16384
// tokens of 4096 with 8 experts.  Every one of these kernels reads it once.
//
// All products and sums are at fp32 precision: tokens are exact in bf16, and fp32 weights enter the tensor cores as the sum
// of three bf16 terms of eight bits each, which is exact.

#include "planmoe.h"
#include "kernels/common.cuh"
#include "kernels/launch.cuh"

#include <type_traits>

namespace planmoe {

namespace {

constexpr int kProjWarps = 8;

__device__ __forceinline__ void mma_16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// upper halves of two fp32 words = their leading eight significant bits as bf16 (towards zero)
__device__ __forceinline__ uint32_t upper_halves(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ float below_upper(float a) { return a - __uint_as_float(__float_as_uint(a) & 0xffff0000u); }

// One block per 16 * MT tokens; its warps share the contraction, 32 columns at a time (chunk w, w + 8, ...), and their
// sums are added in warp order.  A lane's 16-byte pieces of two token rows and of one weight row are the fragments of two
// m16n8k16 steps: which column a fragment register stands for is free as long as both operands agree.  Bound by the token
// rows (DRAM) and, with many experts, by the weights that every block reads again from L2: with more than eight experts,
// 32 tokens a block halve the latter once there are blocks enough (8192 x 4096, 16 experts: 24 us against 34 with 16
// tokens; 4096 tokens: the same).  With fewer experts 16 tokens a block are better at every size (16384 x 4096, 8 experts:
// 34 us against 42).
constexpr int kProjWide = 4096;                   // tokens from which on a block takes 32, with more than eight experts

template <int NT, int MT, bool W_BF16>
__global__ void __launch_bounds__(kProjWarps * 32)
gate_project_kernel(const __nv_bfloat16* __restrict__ x, const void* __restrict__ w_, float* __restrict__ logits, int S, int E,
                    int M, int round_bf16) {
  chain_begin();
  __shared__ float part[kProjWarps][16 * MT][NT * 8 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  const int t0 = blockIdx.x * 16 * MT;
  const uint4* xr[MT][2];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h)                   // rows past the end repeat the last one (not stored)
      xr[m][h] = reinterpret_cast<const uint4*>(x + (long long)min(t0 + m * 16 + h * 8 + g, S - 1) * M) + c;
  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[m][n][i] = 0.f;
  // The rows and weights of a warp's next chunk are on their way while it works on this one: without that the kernel took
  // 48 us for 16384 x 4096, 20 of them for the bytes.
  const int chunks = M / 32;
  uint4 a[2][MT][2], wr[2][NT][W_BF16 ? 1 : 2];
  auto fetch = [&](int buf, int ch) {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      a[buf][m][0] = __ldg(xr[m][0] + ch * 4);
      a[buf][m][1] = __ldg(xr[m][1] + ch * 4);
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const long long at = (long long)min(n * 8 + g, E - 1) * M + ch * 32 + c * 8;
      const uint4* src = W_BF16 ? reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(w_) + at)
                                : reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(w_) + at);
#pragma unroll
      for (int i = 0; i < (W_BF16 ? 1 : 2); ++i) wr[buf][n][i] = __ldg(src + i);
    }
  };
  auto multiply = [&](int buf) {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      uint4 b[W_BF16 ? 1 : 3];
      if constexpr (W_BF16) {
        b[0] = wr[buf][n][0];
      } else {
        const uint4 lo = wr[buf][n][0], hi = wr[buf][n][W_BF16 ? 0 : 1];
        float f[8] = {__uint_as_float(lo.x), __uint_as_float(lo.y), __uint_as_float(lo.z), __uint_as_float(lo.w),
                      __uint_as_float(hi.x), __uint_as_float(hi.y), __uint_as_float(hi.z), __uint_as_float(hi.w)};
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          b[s] = make_uint4(upper_halves(f[0], f[1]), upper_halves(f[2], f[3]), upper_halves(f[4], f[5]), upper_halves(f[6], f[7]));
          if (s < 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = below_upper(f[i]);
          }
        }
      }
#pragma unroll
      for (int s = (W_BF16 ? 1 : 3) - 1; s >= 0; --s) {          // the small terms first
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          mma_16816(acc[m][n], a[buf][m][0].x, a[buf][m][1].x, a[buf][m][0].y, a[buf][m][1].y, b[s].x, b[s].y);
          mma_16816(acc[m][n], a[buf][m][0].z, a[buf][m][1].z, a[buf][m][0].w, a[buf][m][1].w, b[s].z, b[s].w);
        }
      }
    }
  };
  if (warp < chunks) fetch(0, warp);
  for (int ch = warp; ch < chunks; ch += 2 * kProjWarps) {
    const int c1 = ch + kProjWarps, c2 = c1 + kProjWarps;
    if (c1 < chunks) fetch(1, c1);
    multiply(0);
    if (c2 < chunks) fetch(0, c2);
    if (c1 < chunks) multiply(1);
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      part[warp][m * 16 + g][n * 8 + 2 * c] = acc[m][n][0];
      part[warp][m * 16 + g][n * 8 + 2 * c + 1] = acc[m][n][1];
      part[warp][m * 16 + g + 8][n * 8 + 2 * c] = acc[m][n][2];
      part[warp][m * 16 + g + 8][n * 8 + 2 * c + 1] = acc[m][n][3];
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * MT * E; i += kProjWarps * 32) {
    const int r = i / E, e = i - r * E;
    if (t0 + r >= S) break;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kProjWarps; ++w) s += part[w][r][e];
    logits[(long long)(t0 + r) * E + e] = round_bf16 ? __bfloat162float(__float2bfloat16_rn(s)) : s;
  }
}

__device__ __forceinline__ void bf16_pairs(const uint4& raw, unsigned long long* p) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = pair_of(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}

// Block (column slab of 256, chunk of tokens): a lane holds 8 columns of EB experts, the 8 warps take the chunk's tokens in
// turn; their sums are added in warp order through shared memory, one expert after the other.  The gradients of the logits
// wait in shared memory as pairs {d, d}; a warp's eight rows of a stage are requested together, before the barriers around
// those (one row at a time: 104 us for 16384 x 4096, 20 of them for the bytes).
constexpr int kWgradTokens = 64;                  // tokens whose logit gradients are staged at a time

template <int EB>
__global__ void __launch_bounds__(256)
gate_wgrad_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ dl, float* __restrict__ partial, int S, int E,
                  int M, int chunk_tokens) {
  chain_begin();
  __shared__ float2 d_s[kWgradTokens][EB];
  __shared__ float red[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  const bool in = col < M;                        // M is a multiple of 8
  const int c0 = blockIdx.y * chunk_tokens, c1 = min(S, c0 + chunk_tokens);
  unsigned long long acc[EB][4];
#pragma unroll
  for (int e = 0; e < EB; ++e)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[e][i] = 0ull;
  constexpr int kRows = kWgradTokens / 8;
  for (int b0 = c0; b0 < c1; b0 += kWgradTokens) {
    const int n = min(kWgradTokens, c1 - b0);
    uint4 raw[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int t = warp + 8 * r;
      raw[r] = make_uint4(0, 0, 0, 0);
      if (in && t < n) raw[r] = __ldg(reinterpret_cast<const uint4*>(x + (long long)(b0 + t) * M + col));
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kWgradTokens * EB; i += 256) {
      const int t = i / EB, e = i - t * EB;
      const float v = t < n && e < E ? dl[(long long)(b0 + t) * E + e] : 0.f;
      d_s[t][e] = make_float2(v, v);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      unsigned long long p[4];
      bf16_pairs(raw[r], p);
#pragma unroll
      for (int e = 0; e < EB; ++e) {
        const unsigned long long d = *reinterpret_cast<const unsigned long long*>(&d_s[warp + 8 * r][e]);
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[e][i] = fma_pair(p[i], d, acc[e][i]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < EB; ++e) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = unpair(acc[e][i]);
      red[warp][lane * 8 + 2 * i] = f.x;
      red[warp][lane * 8 + 2 * i + 1] = f.y;
    }
    __syncthreads();
    const int m = blockIdx.x * 256 + threadIdx.x;
    if (e < E && m < M) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
      partial[((long long)blockIdx.y * E + e) * M + m] = s;
    }
  }
}

// One block per (32 tokens, 256 columns), 4 tokens a warp.  The slab of the weights is staged once per block, and a warp's
// slots are looked up by one load per lane, so that all its rows are requested together.  (With the weights read by every
// warp and the slots looked up token by token: 128 us for 16384 x 4096, top-2, 8 experts; 61 of them for the bytes.)
constexpr int kGatherTokens = 4;                    // 8: 110 us, two blocks per SM

enum GatherForm { kGatherPlain, kGatherGated, kGatherInt8 };

template <int MAXK, bool W_BF16, int FORM>
__global__ void __launch_bounds__(256, MAXK <= 2 ? 4 : 2)
gather_gate_kernel(const void* __restrict__ slots_, const float2* __restrict__ scales, const int* __restrict__ idx, const int* __restrict__ loc,
                   const float* __restrict__ gates, const float* __restrict__ dl, const void* __restrict__ w_,
                   __nv_bfloat16* __restrict__ dx, int K, int S, int M, int E, int C) {
  chain_begin();
  constexpr bool GATED = FORM == kGatherGated, Q8 = FORM == kGatherInt8;
  extern __shared__ __align__(16) float gather_smem[];
  float* w_s = gather_smem;        // [E][first four, last four of eight columns][32 lanes][4]: no bank conflicts
  float2* dl_s = reinterpret_cast<float2*>(gather_smem + E * 256);                // [32 tokens][E], pairs {d, d}
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slabs = (M + 255) / 256;              // neighbouring blocks take neighbouring columns of the same tokens
  const int tb = (int)(blockIdx.x / slabs) * 8 * kGatherTokens, c0 = (int)(blockIdx.x % slabs) * 256;
  const int col = c0 + lane * 8, t0 = tb + warp * kGatherTokens;
  // lane (token, pick): its slot, -1 without one
  static_assert(kGatherTokens * MAXK <= 32, "one lane per token and pick");
  long long at = -1;
  float gv = 0.f;
  {
    const int tok = t0 + lane / MAXK, k = lane % MAXK;
    if (lane < kGatherTokens * MAXK && k < K && tok < S) {
      const int e = idx[(size_t)k * S + tok], l = loc[(size_t)k * S + tok];
      if (e >= 0 && l >= 0 && l < C) at = (long long)e * C + l;
      if constexpr (GATED) gv = gates[(size_t)k * S + tok];
    }
  }
  uint4 raw[kGatherTokens][MAXK];                 // int8: eight bytes and the pair
#pragma unroll
  for (int t = 0; t < kGatherTokens; ++t)
#pragma unroll
    for (int k = 0; k < MAXK; ++k) {
      const long long row = __shfl_sync(0xffffffffu, at, t * MAXK + k);
      raw[t][k] = make_uint4(0, 0, 0, 0);
      if (row >= 0 && col < M) {
        if constexpr (Q8) {
          const uint2 q = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const unsigned char*>(slots_) + row * M + col));
          const float2 sl = __ldg(scales + (size_t)(col >> 7) * ((size_t)E * C) + row);
          raw[t][k] = make_uint4(q.x, q.y, __float_as_uint(sl.x), __float_as_uint(sl.y));
        } else {
          raw[t][k] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(slots_) + row * M + col));
        }
      }
    }
  for (int i = threadIdx.x; i < E * 256; i += 256) {
    const int m = c0 + (i & 255);
    float v = 0.f;
    if (m < M) {
      const long long o = (long long)(i >> 8) * M + m;
      v = W_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(w_)[o]) : reinterpret_cast<const float*>(w_)[o];
    }
    w_s[(i & ~255) + ((i & 4) ? 128 : 0) + ((i & 255) >> 3) * 4 + (i & 3)] = v;
  }
  for (int i = threadIdx.x; i < 8 * kGatherTokens * E; i += 256) {
    const int t = tb + i / E;
    const float v = t < S ? dl[(long long)tb * E + i] : 0.f;
    dl_s[i] = make_float2(v, v);
  }
  __syncthreads();
  unsigned long long acc[kGatherTokens][4];
#pragma unroll
  for (int t = 0; t < kGatherTokens; ++t) {
#pragma unroll
    for (int k = 0; k < MAXK; ++k) {
      unsigned long long p[4];
      if constexpr (Q8) {                         // a pick without a slot has scale and low zero
        const unsigned long long sc = pair_const(__uint_as_float(raw[t][k].z)), low = pair_const(__uint_as_float(raw[t][k].w));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint32_t w = (i < 2 ? raw[t][k].x : raw[t][k].y) >> (16 * (i & 1));
          p[i] = fma_pair(pair_of((float)(w & 0xffu), (float)((w >> 8) & 0xffu)), sc, low);
        }
      } else {
        bf16_pairs(raw[t][k], p);
      }
      if constexpr (GATED) {
        const unsigned long long gp = pair_const(__shfl_sync(0xffffffffu, gv, t * MAXK + k));
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = k == 0 ? mul_pair(p[i], gp) : fma_pair(p[i], gp, acc[t][i]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[t][i] = k == 0 ? p[i] : add_pair(acc[t][i], p[i]);
      }
    }
  }
  const float2* mine = dl_s + warp * kGatherTokens * E;
#pragma unroll 2
  for (int e = 0; e < E; ++e) {
    const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(w_s + e * 256 + lane * 4);
    const ulonglong2 hi = *reinterpret_cast<const ulonglong2*>(w_s + e * 256 + 128 + lane * 4);
    const unsigned long long w[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
    for (int t = 0; t < kGatherTokens; ++t) {
      const unsigned long long d = *reinterpret_cast<const unsigned long long*>(&mine[t * E + e]);
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[t][i] = fma_pair(w[i], d, acc[t][i]);
    }
  }
  if (col >= M) return;
#pragma unroll
  for (int t = 0; t < kGatherTokens; ++t) {
    if (t0 + t >= S) break;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = unpair(acc[t][i]);
      const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
      o[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(dx + (long long)(t0 + t) * M + col) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int NT, bool W_BF16>
void project_nt(const void* x, const void* w, float* logits, int S, int E, int M, bool round_bf16, cudaStream_t stream) {
  const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(x);
  if constexpr (NT > 1) {
    if (S >= kProjWide) {
      launch_chained(gate_project_kernel<NT, 2, W_BF16>, (S + 31) / 32, kProjWarps * 32, 0, stream, xb, w, logits, S, E, M, round_bf16);
      return;
    }
  }
  launch_chained(gate_project_kernel<NT, 1, W_BF16>, (S + 15) / 16, kProjWarps * 32, 0, stream, xb, w, logits, S, E, M, round_bf16);
}

}  // namespace

void launch_gate_project(const void* x, const void* w, bool w_bf16, float* logits, int S, int E, int M, bool round_bf16,
                         cudaStream_t stream) {
  if (E <= 8) {
    if (w_bf16) project_nt<1, true>(x, w, logits, S, E, M, round_bf16, stream);
    else project_nt<1, false>(x, w, logits, S, E, M, round_bf16, stream);
  } else {
    if (w_bf16) project_nt<2, true>(x, w, logits, S, E, M, round_bf16, stream);
    else project_nt<2, false>(x, w, logits, S, E, M, round_bf16, stream);
  }
}

// Chunks of tokens: two blocks per SM over all column slabs (what is resident with eight experts), at least 32 tokens each.
// Twice as many chunks were a second, half empty wave and twice the partial sums to add up.
int gate_wgrad_chunks(int S, int M) {
  const int slabs = (M + 255) / 256;
  int n = 2 * 148 / slabs;
  if (n > S / 32) n = S / 32;
  return n < 1 ? 1 : n;
}

void launch_gate_wgrad(const void* x, const float* dl, float* partial, int S, int E, int M, cudaStream_t stream) {
  const int n = gate_wgrad_chunks(S, M), tokens = (S + n - 1) / n;
  const dim3 grid((M + 255) / 256, n);
  const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(x);
  if (E <= 2) launch_chained(gate_wgrad_kernel<2>, grid, 256, 0, stream, xb, dl, partial, S, E, M, tokens);
  else if (E <= 4) launch_chained(gate_wgrad_kernel<4>, grid, 256, 0, stream, xb, dl, partial, S, E, M, tokens);
  else if (E <= 8) launch_chained(gate_wgrad_kernel<8>, grid, 256, 0, stream, xb, dl, partial, S, E, M, tokens);
  else launch_chained(gate_wgrad_kernel<16>, grid, 256, 0, stream, xb, dl, partial, S, E, M, tokens);
}

void launch_gather_gate(const void* slots, const float* scales, const int* idx, const int* loc, const float* gates,
                        const float* dl, const void* w, bool w_bf16, void* dx, int K, int S, int M, int E, int C,
                        cudaStream_t stream) {
  const unsigned grid = (unsigned)((S + 8 * kGatherTokens - 1) / (8 * kGatherTokens)) * (unsigned)((M + 255) / 256);
  const int smem = E * 256 * (int)sizeof(float) + 8 * kGatherTokens * E * (int)sizeof(float2);      // at most 20 KiB
  __nv_bfloat16* db = reinterpret_cast<__nv_bfloat16*>(dx);
  auto pick = [&](auto form) {
    constexpr int F = decltype(form)::value;
    return K <= 1 ? (w_bf16 ? gather_gate_kernel<1, true, F> : gather_gate_kernel<1, false, F>)
         : K <= 2 ? (w_bf16 ? gather_gate_kernel<2, true, F> : gather_gate_kernel<2, false, F>)
                  : (w_bf16 ? gather_gate_kernel<4, true, F> : gather_gate_kernel<4, false, F>);
  };
  auto kern = scales != nullptr ? pick(std::integral_constant<int, kGatherInt8>{})
            : gates != nullptr  ? pick(std::integral_constant<int, kGatherGated>{})
                                : pick(std::integral_constant<int, kGatherPlain>{});
  launch_chained(kern, grid, 256, smem, stream, slots, reinterpret_cast<const float2*>(scales), idx, loc, gates, dl, w, db, K, S, M, E, C);
}

}  // namespace planmoe
