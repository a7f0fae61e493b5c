// ZFP fixed-rate 2-D and LZ codec kernels (sm_100a) plus their CPU twins.
//
// ZFP: one thread per 4x4 block; a thread reads four 4-element row segments (neighbouring threads
// read neighbouring segments, so rows are read coalesced) and writes its 2*rate-byte code word.  LZ: one warp per 2 KiB block for both directions, then a per-slice scan and a
// compaction copy pack the blocks back to back.  Both reuse the host/device block coders of
// codec_core.h, so the CUDA streams are bit-identical to the CPU oracle.
//
// Counterparts in the reference: libzfp calls of PlanMoE/custom/compressor/zfpc.cpp:31-51,66-85 and
// the GPULZ kernels + CUB scans of PlanMoE/custom/compressor/gpulz.cu:16-313,418-536.

#include "codec/codecs.h"
#include "codec/codec_core.h"
#include <cstddef>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstring>
#include <vector>

namespace planmoe {

using namespace codec;

namespace {

__host__ __device__ inline float load_elem(const void* base, int elem, long long i) {
  if (elem == 0) return reinterpret_cast<const float*>(base)[i];
#if defined(__CUDA_ARCH__)
  if (elem == 1) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[i]);
  return __half2float(reinterpret_cast<const __half*>(base)[i]);
#else
  const uint16_t h = reinterpret_cast<const uint16_t*>(base)[i];
  if (elem == 1) {
    union { uint32_t u; float f; } v;
    v.u = (uint32_t)h << 16;
    return v.f;
  }
  return __half2float(*reinterpret_cast<const __half*>(&h));
#endif
}
__host__ __device__ inline void store_elem(void* base, int elem, long long i, float f) {
  if (elem == 0) { reinterpret_cast<float*>(base)[i] = f; return; }
  if (elem == 1) { reinterpret_cast<__nv_bfloat16*>(base)[i] = __float2bfloat16_rn(f); return; }
  reinterpret_cast<__half*>(base)[i] = __float2half_rn(f);
}

// One block of the CPU twins.
inline void zfp_block_io(bool encode, const void* x_in, void* x_out, int elem, uint8_t* stream,
                                             long long b, long long rows, long long M, int rate) {
  const long long bx = M / 4, by = (rows + 3) / 4;
  const long long per_slice = bx * by;
  const long long slice = b / per_slice, bb = b - slice * per_slice;
  const long long yb = bb / bx, xb = bb - yb * bx;
  const int words_n = rate / 2;                         // 16 * rate / 32
  uint32_t words[kZfpMaxWords];
  float f[16];
  uint32_t* dst = reinterpret_cast<uint32_t*>(stream + b * (long long)(2 * rate));
  if (encode) {
    for (int r = 0; r < 4; ++r) {
      const long long row = yb * 4 + r;
      for (int c = 0; c < 4; ++c)
        f[r * 4 + c] = row < rows ? load_elem(x_in, elem, (slice * rows + row) * M + xb * 4 + c) : 0.f;
    }
    for (int i = 0; i < words_n; ++i) words[i] = 0;
    zfp_encode_block(f, words, 16 * rate);
    for (int i = 0; i < words_n; ++i) dst[i] = words[i];
  } else {
    for (int i = 0; i < words_n; ++i) words[i] = dst[i];
    zfp_decode_block(words, f, 16 * rate);
    for (int r = 0; r < 4; ++r) {
      const long long row = yb * 4 + r;
      if (row >= rows) break;
      for (int c = 0; c < 4; ++c) store_elem(x_out, elem, (slice * rows + row) * M + xb * 4 + c, f[r * 4 + c]);
    }
  }
}

// One thread per block, the bit planes of its 16 coefficients and its code words in its own column of shared memory.
// Bound by integer issue: the serial bit-plane coder took 4685 warp instructions per 32 blocks (318 us to encode 8192 x
// 4096 bf16, 84 % of the issue slots), its group tests one by one 2070 (140 us); see zfp_encode_block_planes.  VEC: rows of a block are
// moved as one 4-element vector, which needs the tensor's base to lie on such a vector (rows are multiples of four
// elements); other bases take the element loop.
constexpr int kZfpThreads = 128;
__device__ const DoubledOnes kDoubledOnes;          // half a KiB: it stays in L1

template <int ELEM> struct ZfpElem { using type = float; };
template <> struct ZfpElem<1> { using type = __nv_bfloat16; };
template <> struct ZfpElem<2> { using type = __half; };

template <int ELEM, bool VEC>
__device__ __forceinline__ void zfp_load_row(const void* x, long long at, float* f) {
  if constexpr (!VEC) {
    for (int c = 0; c < 4; ++c) f[c] = load_elem(x, ELEM, at + c);
  } else if constexpr (ELEM == 0) {
    const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + at);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  } else {
    using T = typename ZfpElem<ELEM>::type;
    const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(x) + at);
    T v[4];
    *reinterpret_cast<uint2*>(v) = raw;
#pragma unroll
    for (int c = 0; c < 4; ++c) f[c] = (float)v[c];
  }
}
template <int ELEM, bool VEC>
__device__ __forceinline__ void zfp_store_row(void* x, long long at, const float* f) {
  if constexpr (!VEC) {
    for (int c = 0; c < 4; ++c) store_elem(x, ELEM, at + c, f[c]);
  } else if constexpr (ELEM == 0) {
    *reinterpret_cast<float4*>(reinterpret_cast<float*>(x) + at) = make_float4(f[0], f[1], f[2], f[3]);
  } else {
    using T = typename ZfpElem<ELEM>::type;
    T v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] = (T)f[c];
    *reinterpret_cast<uint2*>(reinterpret_cast<T*>(x) + at) = *reinterpret_cast<const uint2*>(v);
  }
}

// Slice, block row and block column of block b (32-bit divisions wherever the block numbers fit).
__device__ __forceinline__ void zfp_block_at(long long b, long long nblocks, long long rows, long long M, long long& slice,
                                             long long& yb, long long& xb) {
  const long long bx = M / 4, per_slice = bx * ((rows + 3) / 4);
  if (nblocks <= 0xffffffffll) {
    const uint32_t s = (uint32_t)b / (uint32_t)per_slice, bb = (uint32_t)b - s * (uint32_t)per_slice;
    const uint32_t y = bb / (uint32_t)bx;
    slice = s; yb = y; xb = bb - y * (uint32_t)bx;
  } else {
    slice = b / per_slice;
    const long long bb = b - slice * per_slice;
    yb = bb / bx;
    xb = bb - yb * bx;
  }
}

template <int ELEM, bool VEC>
__global__ void __launch_bounds__(kZfpThreads)
zfp_encode_kernel(const void* __restrict__ x, uint8_t* __restrict__ stream, long long nblocks, long long rows, long long M,
                  int rate) {
  __shared__ uint32_t planes[16 * kZfpThreads];
  __shared__ uint32_t words[kZfpMaxWords * kZfpThreads];
  const long long b = (long long)blockIdx.x * kZfpThreads + threadIdx.x;
  if (b >= nblocks) return;                       // no barrier below: every thread uses its own column only
  long long slice, yb, xb;
  zfp_block_at(b, nblocks, rows, M, slice, yb, xb);
  float f[16];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const long long row = yb * 4 + r;
    if (row < rows) {
      zfp_load_row<ELEM, VEC>(x, (slice * rows + row) * M + xb * 4, f + r * 4);
    } else {
      f[r * 4] = f[r * 4 + 1] = f[r * 4 + 2] = f[r * 4 + 3] = 0.f;
    }
  }
  uint32_t* w = words + threadIdx.x;
  zfp_encode_block_planes(f, planes + threadIdx.x, w, kDoubledOnes.v, kZfpThreads, 16 * rate);
  uint8_t* dst = stream + b * (2 * rate);         // the stream is a fresh allocation: 8-byte stores are aligned
  for (int i = 0; i < rate / 2; i += 2)
    *reinterpret_cast<uint2*>(dst + 4 * i) = make_uint2(w[i * kZfpThreads], w[(i + 1) * kZfpThreads]);
}

template <int ELEM, bool VEC, bool WIDE>
__global__ void __launch_bounds__(kZfpThreads)
zfp_decode_kernel(const uint8_t* __restrict__ stream, void* __restrict__ x, long long nblocks, long long rows, long long M,
                  int rate) {
  __shared__ uint32_t planes[16 * kZfpThreads];
  __shared__ uint32_t words[kZfpMaxWords * kZfpThreads];
  const long long b = (long long)blockIdx.x * kZfpThreads + threadIdx.x;
  if (b >= nblocks) return;
  uint32_t* w = words + threadIdx.x;
  const uint8_t* src = stream + b * (2 * rate);
  for (int i = 0; i < rate / 2; i += 2) {
    if constexpr (WIDE) {                         // the stream starts on an 8-byte boundary
      const uint2 v = *reinterpret_cast<const uint2*>(src + 4 * i);
      w[i * kZfpThreads] = v.x;
      w[(i + 1) * kZfpThreads] = v.y;
    } else {
      w[i * kZfpThreads] = reinterpret_cast<const uint32_t*>(src)[i];
      w[(i + 1) * kZfpThreads] = reinterpret_cast<const uint32_t*>(src)[i + 1];
    }
  }
  float f[16];
  zfp_decode_block_planes(w, f, planes + threadIdx.x, kZfpThreads, 16 * rate);
  long long slice, yb, xb;
  zfp_block_at(b, nblocks, rows, M, slice, yb, xb);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const long long row = yb * 4 + r;
    if (row < rows) zfp_store_row<ELEM, VEC>(x, (slice * rows + row) * M + xb * 4, f + r * 4);
  }
}

template <int ELEM>
void zfp_launch(bool encode, const void* x_in, void* x_out, uint8_t* stream, long long nblocks, long long rows, long long M,
                int rate, cudaStream_t s) {
  const unsigned grid = (unsigned)((nblocks + kZfpThreads - 1) / kZfpThreads);
  const uintptr_t base = reinterpret_cast<uintptr_t>(encode ? x_in : x_out);
  const bool vec = base % (4 * sizeof(typename ZfpElem<ELEM>::type)) == 0;
  const bool wide = reinterpret_cast<uintptr_t>(stream) % 8 == 0;
  if (encode) {
    if (vec) zfp_encode_kernel<ELEM, true><<<grid, kZfpThreads, 0, s>>>(x_in, stream, nblocks, rows, M, rate);
    else zfp_encode_kernel<ELEM, false><<<grid, kZfpThreads, 0, s>>>(x_in, stream, nblocks, rows, M, rate);
  } else {
    if (vec && wide) zfp_decode_kernel<ELEM, true, true><<<grid, kZfpThreads, 0, s>>>(stream, x_out, nblocks, rows, M, rate);
    else zfp_decode_kernel<ELEM, false, false><<<grid, kZfpThreads, 0, s>>>(stream, x_out, nblocks, rows, M, rate);
  }
}
void zfp_launch_elem(bool encode, const void* x_in, void* x_out, int elem, uint8_t* stream, long long n, long long rows,
                     long long M, int rate, cudaStream_t s) {
  if (n <= 0) return;
  if (elem == 0) zfp_launch<0>(encode, x_in, x_out, stream, n, rows, M, rate, s);
  else if (elem == 1) zfp_launch<1>(encode, x_in, x_out, stream, n, rows, M, rate, s);
  else zfp_launch<2>(encode, x_in, x_out, stream, n, rows, M, rate, s);
}

}  // namespace

size_t zfp_stream_bytes(long long rows, long long M, int rate) {
  return (size_t)(((rows + 3) / 4) * (M / 4) * 2 * rate);
}

void zfp_encode_cpu(const void* x, int elem, uint8_t* stream, long long lead, long long rows, long long M, int rate) {
  const long long n = lead * ((rows + 3) / 4) * (M / 4);
  for (long long b = 0; b < n; ++b) zfp_block_io(true, x, nullptr, elem, stream, b, rows, M, rate);
}
void zfp_decode_cpu(const uint8_t* stream, void* x, int elem, long long lead, long long rows, long long M, int rate) {
  const long long n = lead * ((rows + 3) / 4) * (M / 4);
  for (long long b = 0; b < n; ++b)
    zfp_block_io(false, nullptr, x, elem, const_cast<uint8_t*>(stream), b, rows, M, rate);
}
void launch_zfp_encode(const void* x, int elem, uint8_t* stream, long long lead, long long rows, long long M, int rate,
                       cudaStream_t s) {
  zfp_launch_elem(true, x, nullptr, elem, stream, lead * ((rows + 3) / 4) * (M / 4), rows, M, rate, s);
}
void launch_zfp_decode(const uint8_t* stream, void* x, int elem, long long lead, long long rows, long long M, int rate,
                       cudaStream_t s) {
  zfp_launch_elem(false, nullptr, x, elem, const_cast<uint8_t*>(stream), lead * ((rows + 3) / 4) * (M / 4), rows, M, rate, s);
}

// ------------------------------------------------------------------------------------------------
// LZ
// ------------------------------------------------------------------------------------------------
namespace {

__host__ __device__ inline long long lz_blocks(long long raw_bytes) { return (raw_bytes + kLzBlockBytes - 1) / kLzBlockBytes; }
__host__ __device__ inline long long lz_header_bytes(long long nb) { return ((4 + 4 * (nb + 1)) + 15) / 16 * 16; }

// Bytes of block b's code by its slice's header, 0 if they cannot be a code or do not lie inside the slice.
__host__ __device__ inline int lz_code_bytes(const uint32_t* hdr, long long b, long long nb, long long slice_bytes) {
  const long long from = hdr[1 + b], to = hdr[2 + b];
  return to - from < 2 || to - from > kLzSlotBytes || lz_header_bytes(nb) + to > slice_bytes ? 0 : (int)(to - from);
}

__host__ __device__ inline int lz_encode_one(const uint8_t* raw, long long raw_bytes, long long blk, int sym, uint8_t* slot) {
  const long long off = blk * kLzBlockBytes;
  const int bytes = (int)(raw_bytes - off < kLzBlockBytes ? raw_bytes - off : kLzBlockBytes);
  if (sym == 2) return lz_encode_block<uint16_t>(reinterpret_cast<const uint16_t*>(raw + off), bytes / 2, slot);
  return lz_encode_block<uint32_t>(reinterpret_cast<const uint32_t*>(raw + off), bytes / 4, slot);
}
__host__ __device__ inline void lz_decode_one(const uint8_t* packed, uint8_t* raw, long long raw_bytes, long long blk, int sym) {
  const long long off = blk * kLzBlockBytes;
  const int bytes = (int)(raw_bytes - off < kLzBlockBytes ? raw_bytes - off : kLzBlockBytes);
  if (sym == 2) lz_decode_block<uint16_t>(packed, reinterpret_cast<uint16_t*>(raw + off), bytes / 2);
  else lz_decode_block<uint32_t>(packed, reinterpret_cast<uint32_t*>(raw + off), bytes / 4);
}

// Warp-parallel block coder.  One warp codes one 2 KiB block, 32 positions ("a row") at a time, and produces exactly
// the bytes of the serial coder lz_encode_block (the CPU twin, which the tests compare against).  A row's symbols are
// held bit-sliced: B[b] is bit b of all 32 symbols, from a bit transpose over the warp (of two rows at once with 16-bit
// symbols), read back from shared memory by every lane.
//   1. lane d compares the row with the symbols d + 1 positions back: all 32 positions at once, by and-ing, over the
//      symbol's bits, B[b] with itself shifted across the row boundary.  A 32 x 32 bit transpose over the warp turns
//      that into one mask of candidate distances per position (bit d set: in[p] == in[p - d - 1]).
//   2. a candidate at distance d matches L symbols from p exactly when the masks of p .. p + L - 1 all have bit d, so
//      the longest match comes from and-ing masks until nothing survives, and the first candidate of maximal length
//      (the serial coder's choice) is the largest surviving distance.  Matches are at most 32 long: the masks of this
//      row and the next are enough.
//   3. token starts are the positions reachable from 0 by p + (match ? length : 1).  Every lane gets, by pointer doubling
//      over the row, the set of starts a walk from it visits and where that walk enters the next row; the row's own
//      entry picks one of them.
//   4. the row's tokens are written at their ordinals; their flags are compressed by one or-reduction.
// Bound by the integer pipe.  8192 x 4096 bf16: 537 us when candidates were compared through shared memory and tokens
// walked serially per lane; 432 us with a ballot per bit and the match length counted symbol by symbol (10.4 k warp
// instructions a block).
//
// scratch layout: [slices][nb] slots of kLzScratchSlot bytes {token data, flag words, token count}, then int sizes
// [slices][nb] (bytes of the block's code)
constexpr int kLzWarps = 4;                       // blocks coded per CTA
constexpr int kLzScratchFlags = kLzBlockBytes;
constexpr int kLzScratchCount = kLzScratchFlags + 128;
constexpr int kLzScratchSlot = kLzScratchCount + 16;
static_assert(kLzWindow == 32 && kLzMaxMatch == 32 && kLzScratchSlot % 16 == 0, "lz encoder: rows of 32, distance masks");

// Bit c of lane r becomes bit r of lane c.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    const uint32_t m = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t keep = (lane & s) ? ~m : m;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    const uint32_t rot = __funnelshift_l(y, y, (lane & s) ? 32 - s : s);
    x = (x & keep) | (rot & ~keep);
  }
  return x;
}

template <class Sym>
__device__ __forceinline__ void lz_encode_block_warp(const Sym* __restrict__ in, int nsym, uint8_t* __restrict__ slot,
                                                     int* __restrict__ out_size, uint32_t* sm, int lane) {
  constexpr int kBits = 8 * (int)sizeof(Sym);
  constexpr int kRowsAtOnce = 32 / kBits;         // rows whose symbols fill one word per lane
  constexpr int min_match = sizeof(Sym) == 2 ? 2 : 1;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t* masks = sm;                           // candidate masks of the row in work and of the next one
  uint32_t* bits = sm + 64;                       // B of the newest kRowsAtOnce rows
  uint16_t* data = reinterpret_cast<uint16_t*>(slot);
  uint32_t* flag_words = reinterpret_cast<uint32_t*>(slot + kLzScratchFlags);
  uint32_t prev[kBits];                           // B of the row before
#pragma unroll
  for (int b = 0; b < kBits; ++b) prev[b] = 0u;
  const int rows = (nsym + 31) >> 5;
  auto row_mask = [&](int k) { const int left = nsym - k * 32; return left >= 32 ? 0xffffffffu : left <= 0 ? 0u : (1u << left) - 1u; };
  auto load = [&](int k) { const int p = k * 32 + lane; return p < nsym ? in[p] : (Sym)0; };
  // B of rows k .. k + kRowsAtOnce - 1, symbols v (and u): lane b gets the word of bit b
  auto slice = [&](Sym v, Sym u) {
    const uint32_t w = warp_transpose32(kBits == 32 ? (uint32_t)v : (uint32_t)v | ((uint32_t)u << (kBits & 31)), lane);
    __syncwarp();                                 // the last readers of `bits` are done
    bits[lane] = w;
    __syncwarp();
  };
  auto candidates = [&](int k) {
    uint32_t acc = row_mask(k);
    if (k == 0) acc &= ~((2u << lane) - 1u);      // nothing lies before position 0
    const uint4* words = reinterpret_cast<const uint4*>(bits + (k % kRowsAtOnce) * kBits);
#pragma unroll
    for (int b4 = 0; b4 < kBits / 4; ++b4) {
      const uint4 q = words[b4];
      const uint32_t cur[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc &= ~(cur[j] ^ __funnelshift_lc(prev[b4 * 4 + j], cur[j], lane + 1));
        prev[b4 * 4 + j] = cur[j];
      }
    }
    return warp_transpose32(acc, lane);
  };

  // symbols are loaded kRowsAtOnce rows ahead of their slicing
  Sym v = load(0), v_next = load(1), a0 = load(2), a1 = load(3);
  slice(v, v_next);
  uint32_t eq = candidates(0);                    // this lane's mask of row k
  int entry = 0, ntok = 0, dbytes = 0;
  uint64_t facc = 0;                              // flags not yet written, first token lowest
  int fbits = 0;
  for (int k = 0; k < rows; ++k) {
    uint32_t eq_next = 0u;
    if (k + 1 < rows) {
      if ((k + 1) % kRowsAtOnce == 0) slice(v_next, a0);
      eq_next = candidates(k + 1);
    }
    masks[lane] = eq;
    masks[32 + lane] = eq_next;
    __syncwarp();

    // 2. longest match: up to seven symbols without a branch.  m_i: distances that match i + 1 symbols.
    const uint32_t* at = masks + lane;
    const uint32_t m1 = eq & at[1], m2 = m1 & at[2], m3 = m2 & at[3], m4 = m3 & at[4], m5 = m4 & at[5], m6 = m5 & at[6];
    const bool four = m3 != 0u;
    uint32_t m = four ? m3 : eq;
    int best = four ? 4 : eq != 0u ? 1 : 0;
    const uint32_t two = four ? m5 : m1;          // two (four: six) symbols
    if (two != 0u) { m = two; best = four ? 6 : 2; }
    const uint32_t odd = four ? (two != 0u ? m6 : m4) : (two != 0u ? m2 : 0u);
    if (odd != 0u) { m = odd; ++best; }
    if (m6 != 0u) {
      while (best < kLzMaxMatch) {
        const uint32_t t = m & at[best];
        if (t == 0u) break;
        m = t;
        ++best;
      }
    }
    const bool match = best >= min_match;
    __syncwarp();                                 // the masks of row k are overwritten in the next round

    // 3. starts of this row and the entry into the next
    uint32_t visits = 1u << lane;
    int to = lane + (match ? best : 1);           // 32 and above: a position of the next row
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      const uint32_t vo = __shfl_sync(0xffffffffu, visits, to & 31);
      const int too = __shfl_sync(0xffffffffu, to, to & 31);
      if (to < 32) { visits |= vo; to = too; }
    }
    const uint32_t starts = __shfl_sync(0xffffffffu, visits, entry) & row_mask(k);
    entry = __shfl_sync(0xffffffffu, to, entry) & 31;

    // 4. tokens
    const bool is = (starts >> lane) & 1u;
    const int r = __popc(starts & lt), cnt = __popc(starts);
    const uint32_t flags = __reduce_or_sync(0xffffffffu, is && match ? 1u << r : 0u);
    const uint32_t pair = (uint32_t)best | ((uint32_t)(32 - __clz(m)) << 8);
    if constexpr (sizeof(Sym) == 2) {
      if (is) data[ntok + r] = match ? (uint16_t)pair : (uint16_t)v;
      dbytes += 2 * cnt;
    } else {
      const uint32_t matches = __ballot_sync(0xffffffffu, is && match);
      if (is) {
        uint16_t* d = data + dbytes / 2 + 2 * r - __popc(matches & lt);
        d[0] = match ? (uint16_t)pair : (uint16_t)v;
        if (!match) d[1] = (uint16_t)(v >> 16);
      }
      dbytes += 4 * cnt - 2 * __popc(matches);
    }
    ntok += cnt;
    facc |= (uint64_t)flags << fbits;
    fbits += cnt;
    if (fbits >= 32) {
      if (lane == 0) *flag_words = (uint32_t)facc;
      ++flag_words;
      facc >>= 32;
      fbits -= 32;
    }
    v = v_next;
    v_next = a0;
    a0 = a1;
    a1 = load(k + 4);
    eq = eq_next;
  }
  if (lane == 0) {
    if (fbits > 0) *flag_words = (uint32_t)facc;
    *reinterpret_cast<uint32_t*>(slot + kLzScratchCount) = (uint32_t)ntok;
    *out_size = 2 + ((ntok + 7) >> 3) + dbytes;
  }
}

template <class Sym>
__global__ void __launch_bounds__(kLzWarps * 32)
lz_encode_blocks_kernel(const uint8_t* __restrict__ raw, uint8_t* __restrict__ slots, int* __restrict__ blk_sizes,
                        long long slices, long long raw_bytes) {
  __shared__ __align__(16) uint32_t sm[kLzWarps][96];     // see lz_encode_block_warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long nb = lz_blocks(raw_bytes);
  const long long i = (long long)blockIdx.x * kLzWarps + warp;
  if (i >= slices * nb) return;
  const long long s = i / nb, b = i - s * nb;
  const long long off = b * kLzBlockBytes;
  const int bytes = (int)(raw_bytes - off < kLzBlockBytes ? raw_bytes - off : kLzBlockBytes);
  lz_encode_block_warp<Sym>(reinterpret_cast<const Sym*>(raw + s * raw_bytes + off), bytes / (int)sizeof(Sym),
                            slots + i * kLzScratchSlot, blk_sizes + i, sm[warp], lane);
}

// One CTA per slice: exclusive scan of the block sizes -> header of the slice payload.  Four sizes a thread, so that a
// slice of 8 MiB (4096 blocks) is one round.
constexpr int kLzScanThreads = 1024;
__global__ void __launch_bounds__(kLzScanThreads)
lz_scan_kernel(const int* __restrict__ blk_sizes, uint8_t* __restrict__ payload, int* __restrict__ sizes, long long raw_bytes,
               long long payload_stride) {
  __shared__ unsigned warp_tot[32];
  const long long nb = lz_blocks(raw_bytes);
  const long long s = blockIdx.x;
  uint32_t* hdr = reinterpret_cast<uint32_t*>(payload + s * payload_stride);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned carry = 0;
  for (long long base = 0; base < nb; base += 4 * kLzScanThreads) {
    const long long i = base + 4 * threadIdx.x;
    unsigned v[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) { v[j] = i + j < nb ? (unsigned)blk_sizes[s * nb + i + j] : 0u; sum += v[j]; }
    unsigned incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    unsigned tot = warp_tot[lane], wincl = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, wincl, o);
      if (lane >= o) wincl += t;
    }
    const unsigned before_warp = __shfl_sync(0xffffffffu, wincl - tot, warp);
    unsigned at = carry + before_warp + incl - sum;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i + j < nb) hdr[1 + i + j] = at;
      at += v[j];
    }
    carry += __shfl_sync(0xffffffffu, wincl, 31);
    __syncthreads();                              // warp_tot is written again in the next round
  }
  if (threadIdx.x == 0) {
    hdr[0] = (uint32_t)nb;
    hdr[1 + nb] = carry;
    for (long long w = 2 + nb; w < lz_header_bytes(nb) / 4; ++w) hdr[w] = 0;   // header padding
    sizes[s] = (int)(lz_header_bytes(nb) + carry);
  }
}

// n bytes from a 4-byte aligned source to any address: byte stores up to the destination's next word, then whole words
// put together from two source words (the word behind the last one that is copied may be read, not used).
__device__ __forceinline__ void warp_copy_to_bytes(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, int n, int lane) {
  const int head = min(n, (int)((4 - (reinterpret_cast<uintptr_t>(dst) & 3)) & 3));
  if (lane < head) dst[lane] = src[lane];
  const int words = (n - head) >> 2;
  const uint32_t* s32 = reinterpret_cast<const uint32_t*>(src);
  uint32_t* d32 = reinterpret_cast<uint32_t*>(dst + head);
  for (int i = lane; i < words; i += 32) d32[i] = __funnelshift_r(s32[i], s32[i + 1], 8 * head);
  const int done = head + 4 * words;
  if (lane < n - done) dst[done + lane] = src[done + lane];
}

// One warp per block: {token count, flags, data} of its scratch slot to its place in the payload.  Word copies: byte
// copies took 61 us for 8192 x 4096 bf16.
__global__ void __launch_bounds__(128)
lz_compact_kernel(const uint8_t* __restrict__ slots, const int* __restrict__ blk_sizes, uint8_t* __restrict__ payload,
                  long long raw_bytes, long long payload_stride) {
  const long long nb = lz_blocks(raw_bytes);
  const long long i = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const long long s = blockIdx.y;
  const int lane = threadIdx.x & 31;
  if (i >= nb) return;
  const uint32_t* hdr = reinterpret_cast<const uint32_t*>(payload + s * payload_stride);
  uint8_t* dst = payload + s * payload_stride + lz_header_bytes(nb) + hdr[1 + i];
  const uint8_t* src = slots + (s * nb + i) * kLzScratchSlot;
  const int n = blk_sizes[s * nb + i];
  const int ntok = (int)*reinterpret_cast<const uint32_t*>(src + kLzScratchCount);
  const int flag_bytes = (ntok + 7) >> 3;
  if (lane < 2) dst[lane] = (uint8_t)(ntok >> (8 * lane));
  warp_copy_to_bytes(dst + 2, src + kLzScratchFlags, flag_bytes, lane);
  warp_copy_to_bytes(dst + 2 + flag_bytes, src, n - 2 - flag_bytes, lane);
}

// Warp-parallel block decoder (same output as lz_decode_block).  Tokens are laid out first, 32 at a time: a scan of
// their lengths gives each its position, where it leaves one word {start mark, literal or distance}.  Positions are then
// resolved a row of 32 at a time: a position belongs to the last start at or before it; a source in an earlier row is
// already known, a source in the same row (matches may copy what an earlier or the same match produced) is reached by
// five rounds of pointer doubling in registers.  The former decoder doubled pointers ten times over the whole block
// in shared memory (285 us for 8192 x 4096 bf16).
constexpr int kLzCodeWords = (3 + kLzSlotBytes + 3) / 4;
constexpr int kLzMaxSym = kLzBlockBytes / 2;
struct LzDecSmem {
  uint32_t code[kLzCodeWords + 1];                // the block's code, as it lies in global words
  uint32_t info[kLzMaxSym];                       // token words, then the decoded symbols
};

template <class Sym>
__device__ __forceinline__ void lz_decode_block_warp(const uint8_t* __restrict__ g_code, int code_bytes,
                                                     Sym* __restrict__ g_out, int nsym, LzDecSmem& sm, int lane) {
  const int mis = (int)(reinterpret_cast<uintptr_t>(g_code) & 3);
  const uint32_t* g_words = reinterpret_cast<const uint32_t*>(g_code - mis);
  const int whole = (mis + code_bytes) >> 2, tail = (mis + code_bytes) & 3;
  for (int i = lane; i < whole; i += 32) sm.code[i] = g_words[i];
  uint8_t* code = reinterpret_cast<uint8_t*>(sm.code) + mis;
  if (lane < tail) reinterpret_cast<uint8_t*>(sm.code + whole)[lane] = reinterpret_cast<const uint8_t*>(g_words + whole)[lane];
  const int rows = (nsym + 31) >> 5;
  for (int k = 0; k < rows; ++k) sm.info[k * 32 + lane] = 0u;
  __syncwarp();
  const uint32_t lt = (1u << lane) - 1u;
  const int ntok = min((int)code[0] | ((int)code[1] << 8), nsym);
  const int flag_bytes = (ntok + 7) >> 3;
  const int data_at = 2 + flag_bytes;
  const int last = code_bytes - 1;                // reads of a damaged code stay inside it

  int total = 0, lits = 0;
  for (int t0 = 0; t0 < ntok; t0 += 32) {
    const int t = t0 + lane;
    const bool live = t < ntok;
    const bool match = live && ((code[min(2 + (t >> 3), last)] >> (t & 7)) & 1u);
    int off = data_at + 2 * t;
    if constexpr (sizeof(Sym) == 4) {
      const uint32_t lit = __ballot_sync(0xffffffffu, live && !match);
      off += 2 * (lits + __popc(lit & lt));
      lits += __popc(lit);
    }
    const uint32_t b0 = code[min(off, last)], b1 = code[min(off + 1, last)];
    const int len = !live ? 0 : match ? (int)b0 : 1;
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    const int p = total + incl - len;
    if (live && p < nsym)
      sm.info[p] = match ? 0xc0000000u | b1 : 0x80000000u | (sizeof(Sym) == 2 ? b0 | (b1 << 8) : (uint32_t)off);
    total += __shfl_sync(0xffffffffu, incl, 31);
  }
  __syncwarp();
  uint32_t carry = 0u;                            // the last token that starts before the row
  for (int k = 0; k < rows; ++k) {
    const int p = k * 32 + lane;
    const uint32_t w = sm.info[p];
    const uint32_t starts = __ballot_sync(0xffffffffu, w >> 31);
    const uint32_t upto = starts & (lt | (1u << lane));
    uint32_t own = __shfl_sync(0xffffffffu, w, upto ? 31 - __clz(upto) : 0);
    if (upto == 0u) own = carry;
    if (starts != 0u) carry = __shfl_sync(0xffffffffu, w, 31 - __clz(starts));
    uint32_t val = 0u;
    int from = lane;
    if (p < total) {
      if (own & 0x40000000u) {
        const int src = max(p - (int)(own & 0xffu), 0);
        if (src < k * 32) val = sm.info[src];
        else from = src & 31;
      } else if (w >> 31) {
        if constexpr (sizeof(Sym) == 2) {
          val = w & 0xffffu;
        } else {
          const int off = (int)(w & 0xffffu);
#pragma unroll
          for (int b = 0; b < 4; ++b) val |= (uint32_t)code[min(off + b, last)] << (8 * b);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) from = __shfl_sync(0xffffffffu, from, from);
    val = __shfl_sync(0xffffffffu, val, from);
    sm.info[p] = val;
    if (p < nsym) g_out[p] = (Sym)val;
    __syncwarp();
  }
}

template <class Sym>
__global__ void __launch_bounds__(kLzWarps * 32)
lz_decode_blocks_kernel(const uint8_t* __restrict__ payload, uint8_t* __restrict__ raw, long long slices, long long raw_bytes,
                        long long payload_stride) {
  __shared__ LzDecSmem smem[kLzWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long nb = lz_blocks(raw_bytes);
  const long long i = (long long)blockIdx.x * kLzWarps + warp;
  if (i >= slices * nb) return;
  const long long s = i / nb, b = i - s * nb;
  const uint8_t* base = payload + s * payload_stride;
  const uint32_t* hdr = reinterpret_cast<const uint32_t*>(base);
  const long long off = b * kLzBlockBytes;
  const int bytes = (int)(raw_bytes - off < kLzBlockBytes ? raw_bytes - off : kLzBlockBytes);
  const long long code_at = lz_header_bytes(nb) + (long long)hdr[1 + b];
  const int code_bytes = lz_code_bytes(hdr, b, nb, payload_stride);
  if (code_bytes < 2) return;                     // corrupt header: leave the block untouched
  lz_decode_block_warp<Sym>(base + code_at, code_bytes,
                            reinterpret_cast<Sym*>(raw + s * raw_bytes + off), bytes / (int)sizeof(Sym), smem[warp], lane);
}

}  // namespace

size_t lz_payload_capacity(long long raw_bytes) {
  const long long nb = lz_blocks(raw_bytes);
  return (size_t)((lz_header_bytes(nb) + nb * kLzSlotBytes + 15) / 16 * 16);
}
void lz_slice_layout(long long raw_bytes, long long* len_off, long long* header_bytes) {
  const long long nb = lz_blocks(raw_bytes);
  *len_off = 4 * (1 + nb);
  *header_bytes = lz_header_bytes(nb);
}
size_t lz_scratch_bytes(long long slices, long long raw_bytes) {
  const long long nb = lz_blocks(raw_bytes);
  return (size_t)(slices * nb * (kLzScratchSlot + 4));
}

void lz_encode_cpu(const uint8_t* raw, uint8_t* payload, int* sizes, long long slices, long long raw_bytes,
                   long long payload_stride, int sym) {
  const long long nb = lz_blocks(raw_bytes);
  std::vector<uint8_t> slot(kLzSlotBytes);
  for (long long s = 0; s < slices; ++s) {
    uint8_t* base = payload + s * payload_stride;
    uint32_t* hdr = reinterpret_cast<uint32_t*>(base);
    hdr[0] = (uint32_t)nb;
    uint32_t off = 0;
    for (long long b = 0; b < nb; ++b) {
      const int n = lz_encode_one(raw + s * raw_bytes, raw_bytes, b, sym, slot.data());
      hdr[1 + b] = off;
      std::memcpy(base + lz_header_bytes(nb) + off, slot.data(), n);
      off += (uint32_t)n;
    }
    hdr[1 + nb] = off;
    for (long long w = 2 + nb; w < lz_header_bytes(nb) / 4; ++w) hdr[w] = 0;   // header padding
    sizes[s] = (int)(lz_header_bytes(nb) + off);
  }
}
void lz_decode_cpu(const uint8_t* payload, uint8_t* raw, long long slices, long long raw_bytes, long long payload_stride,
                   int sym) {
  const long long nb = lz_blocks(raw_bytes);
  for (long long s = 0; s < slices; ++s) {
    const uint8_t* base = payload + s * payload_stride;
    const uint32_t* hdr = reinterpret_cast<const uint32_t*>(base);
    for (long long b = 0; b < nb; ++b)
      if (lz_code_bytes(hdr, b, nb, payload_stride) > 0)
        lz_decode_one(base + lz_header_bytes(nb) + hdr[1 + b], raw + s * raw_bytes, raw_bytes, b, sym);
  }
}

void launch_lz_encode(const uint8_t* raw, uint8_t* payload, int* sizes, uint8_t* scratch, long long slices,
                      long long raw_bytes, long long payload_stride, int sym, cudaStream_t stream) {
  const long long nb = lz_blocks(raw_bytes);
  const long long total = slices * nb;
  if (total <= 0) return;
  uint8_t* slots = scratch;
  int* blk_sizes = reinterpret_cast<int*>(scratch + total * kLzScratchSlot);
  const unsigned ctas = (unsigned)((total + kLzWarps - 1) / kLzWarps);
  if (sym == 2)
    lz_encode_blocks_kernel<uint16_t><<<ctas, kLzWarps * 32, 0, stream>>>(raw, slots, blk_sizes, slices, raw_bytes);
  else
    lz_encode_blocks_kernel<uint32_t><<<ctas, kLzWarps * 32, 0, stream>>>(raw, slots, blk_sizes, slices, raw_bytes);
  lz_scan_kernel<<<(unsigned)slices, kLzScanThreads, 0, stream>>>(blk_sizes, payload, sizes, raw_bytes, payload_stride);
  dim3 grid((unsigned)((nb + 3) / 4), (unsigned)slices);
  lz_compact_kernel<<<grid, 128, 0, stream>>>(slots, blk_sizes, payload, raw_bytes, payload_stride);
}
void launch_lz_decode(const uint8_t* payload, uint8_t* raw, long long slices, long long raw_bytes,
                      long long payload_stride, int sym, cudaStream_t stream) {
  const long long total = slices * lz_blocks(raw_bytes);
  if (total <= 0) return;
  const unsigned ctas = (unsigned)((total + kLzWarps - 1) / kLzWarps);
  if (sym == 2)
    lz_decode_blocks_kernel<uint16_t><<<ctas, kLzWarps * 32, 0, stream>>>(payload, raw, slices, raw_bytes, payload_stride);
  else
    lz_decode_blocks_kernel<uint32_t><<<ctas, kLzWarps * 32, 0, stream>>>(payload, raw, slices, raw_bytes, payload_stride);
}

}  // namespace planmoe
