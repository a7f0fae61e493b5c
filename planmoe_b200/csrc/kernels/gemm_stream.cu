// Grouped bf16 GEMM for a handful of rows a group: y[g] = act(x[g] . w[g] + b[g]) with at most 32 rows, w [K, N] with N
// contiguous.  A decoding step or a small batch meets every expert's weights; reading them is all the work there is.
//
// Tiles of 128 x 256 (gemm_tcgen05.cu) leave SMs without loads in flight where there are few of them: 8 experts of 4096 x 1024 are 32
// CTAs.  Here a tile is 64 columns wide, the narrowest that the weights' swizzled layout has, and its CTA goes through the whole
// contraction: four times the CTAs, no sum that is shared between them, and outputs whose products are added up in the same order
// as there, bit for bit.  (The contraction of a wide tile split over a cluster rounds differently; it took 17.0 us where this takes
// 15.7, 8 x 4096 x 1024, 19.7 for 11.0, 5 x 2048 x 2048, and 12.4 for 14.8, 1 x 4096 x 4096.)  Two CTAs fit on an SM.  Groups without a
// token read no weights: their rows are zeros, so that the bias is all there is.  For which launches: stream_gemm_pays.
//
//   warp 0      TMA producer; then the accumulators, TMEM to shared memory
//   warp 1      MMA issuer (tcgen05.mma.cta_group::1, 128 x 64 x 16; rows behind the tile's are whatever lies behind them in
//               shared memory and are never read back)
//   all warps   bias, activation and stores, eight columns a thread
// No cluster multicast of loads.  Every wait is bounded.

#include "planmoe.h"
#include "kernels/gemm_local.h"
#include "kernels/gemm_tc.cuh"
#include "kernels/launch.cuh"

namespace planmoe {

namespace {

constexpr int kStreamThreads = 128;
constexpr int kStreamCols = 64;
constexpr int kAccRow = kStreamCols + 4;           // floats between rows of the accumulators in shared memory: lanes on different banks

// Two K blocks a stage: what bounds a CTA is the round of waiting, issuing and committing, not the bytes in flight (6, 8 or 9 stages
// of one block take the same time).  us for stages x blocks of 8 x 1, 4 x 2, 2 x 4: 8 x 4096 x 1024 18.3, 15.7, 17.1; 1 x 4096 x 4096
// 18.2, 14.8, 15.9; 12 x 2048 x 1024 12.1, 11.9, 13.2.
constexpr int kPer = 2, kStages = 4;
constexpr uint32_t kABytes = kStreamRows * BK * 2, kBBytes = kStreamCols * BK * 2, kBlockBytes = kABytes + kBBytes;
constexpr uint32_t kStage = kPer * kBlockBytes;
constexpr uint32_t kRing = kStages * kStage, kMmaRows = BM * BK * 2;
constexpr uint32_t kPad = kMmaRows - kBlockBytes;  // the MMA reads 128 rows from the last block's start, too
constexpr uint32_t kSmemTotal = kRing + kPad + 256;
static_assert(kMmaRows > kBlockBytes && kStage % 1024 == 0, "ring");
static_assert(kStreamRows == 32 && kStreamRows * kAccRow * 4 <= kRing, "one warp's TMEM lanes; they take the ring's place");
static_assert(2 * (kSmemTotal + 1024) <= 233472, "two CTAs fit on an SM");

struct StreamCtl {
  uint64_t full[kStages], empty[kStages], acc_full;
  uint32_t tmem_base;
  volatile int abort;
};
static_assert(sizeof(StreamCtl) <= 256, "control block");

template <int ACT>
__device__ __forceinline__ void act8(const pair_t* x, uint4& out, uint4& deriv) {
  pair_t f[4], d[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) act_both<ACT>(x[i], f[i], d[i]);
  out = make_uint4(pack_pair(f[0]), pack_pair(f[1]), pack_pair(f[2]), pack_pair(f[3]));
  deriv = make_uint4(pack_pair(d[0]), pack_pair(d[1]), pack_pair(d[2]), pack_pair(d[3]));
}

__global__ void __launch_bounds__(kStreamThreads)
stream_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const StreamGemm p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0u) {            // swizzled tiles need 1024-byte aligned stages
    if (threadIdx.x == 0) report_status(p.status, kStatusBadArgument, 1024, (int)(smem_u32(smem) & 1023u), 0);
    return;                                        // same address in every CTA: the whole grid returns
  }
  StreamCtl* const ctl = reinterpret_cast<StreamCtl*>(smem + kRing + kPad);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nt_count = (p.N + kStreamCols - 1) / kStreamCols;
  const int g = (int)blockIdx.x / nt_count, n0 = ((int)blockIdx.x - g * nt_count) * kStreamCols;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(smem_u32(&ctl->full[s]), 1); mbar_init(smem_u32(&ctl->empty[s]), 1); }
    mbar_init(smem_u32(&ctl->acc_full), 1);
    ctl->abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc<1>(smem_u32(&ctl->tmem_base), kStreamCols);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  chain_begin();
  const bool live = p.rows_used == nullptr || p.rows_used[g] > 0;
  const int kbs = live ? (p.K + BK - 1) / BK : 0;  // none where the group holds no token
  float* const acc = reinterpret_cast<float*>(smem);

  if (warp == 0) {
    const bool leader = elect_one();
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int kb = 0; kb < kbs; kb += kPer) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1u, &ctl->abort, p.budget_ns, p.status, 0, stage));
      if (!ok) break;
      if (leader) {
        const uint32_t full = smem_u32(&ctl->full[stage]), sa = smem_u32(smem) + stage * kStage;
        const int n = min(kPer, kbs - kb);
        mbar_expect_tx(full, n * kBlockBytes);
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          if (j < n) {
            tma_load_4d<1>(sa + j * kBlockBytes, &tmA, full, (kb + j) * BK, 0, g, 0);
            tma_load_4d<1>(sa + j * kBlockBytes + kABytes, &tmB, full, n0, (kb + j) * BK, g, 0);
          }
        }
      }
      __syncwarp();
      if (++stage == kStages) { stage = 0; phase ^= 1u; }
    }
    if (!ok) __nanosleep(200000);                  // let copies already in flight land before teardown
    __syncwarp();
    // The accumulators of row `lane`, laid over the ring: every load has been read by an MMA that has completed.
    if (ok && kbs > 0)
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->acc_full), 0, &ctl->abort, p.budget_ns, p.status, 2, 0));
    if (ok) {
      uint32_t v[kStreamCols];
      if (kbs > 0) {
        tc_fence_after();
        tmem_ld32(tmem, v);
        tmem_ld32(tmem + 32, v + 32);
        tmem_ld_wait();
        tmem_ld_ready(v);
        tmem_ld_ready(v + 32);
      } else {
#pragma unroll
        for (int i = 0; i < kStreamCols; ++i) v[i] = 0u;
      }
      if (lane < p.M) {
#pragma unroll
        for (int i = 0; i < kStreamCols; i += 4) *reinterpret_cast<uint4*>(acc + lane * kAccRow + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(false, true, BM, kStreamCols);
    const bool leader = elect_one();
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int kb = 0; kb < kbs; kb += kPer) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->full[stage]), phase, &ctl->abort, p.budget_ns, p.status, 1, stage));
      if (!ok) break;
      tc_fence_after();
      if (leader) {
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          const uint32_t sa = smem_u32(smem) + stage * kStage + j * kBlockBytes, sb = sa + kABytes;
          if (j < kbs - kb) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16<1>(tmem, make_desc(sa + k * (UMMA_K * 2), 16, 1024), make_desc(sb + k * (UMMA_K * 128), 64 * BK * 2, 1024), idesc,
                           (kb | j | k) != 0 ? 1u : 0u);
          }
        }
        umma_commit<1>(smem_u32(&ctl->empty[stage]));
      }
      __syncwarp();
      if (++stage == kStages) { stage = 0; phase ^= 1u; }
    }
    if (ok && kbs > 0 && leader) umma_commit<1>(smem_u32(&ctl->acc_full));
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, kStreamCols);
  }

  if (ctl->abort) return;
  constexpr int kVecs = kStreamCols / 8;
  for (int i = threadIdx.x; i < p.M * kVecs; i += kStreamThreads) {
    const int r = i / kVecs, c = (i % kVecs) * 8, n = n0 + c;
    if (n >= p.N) continue;                        // N is a multiple of 8
    const float4 a = *reinterpret_cast<const float4*>(acc + r * kAccRow + c), b = *reinterpret_cast<const float4*>(acc + r * kAccRow + c + 4);
    pair_t x[4] = {pair_of(a.x, a.y), pair_of(a.z, a.w), pair_of(b.x, b.y), pair_of(b.z, b.w)};
    if (p.bias != nullptr) {
      const uint4 bv = __ldg(reinterpret_cast<const uint4*>(p.bias + (long long)g * p.N + n));
      const uint32_t w[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = add_pair(x[j], pair_of(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u)));
    }
    uint4 out, deriv;
    switch (p.activation) {
      case kActRelu: act8<kActRelu>(x, out, deriv); break;
      case kActGelu: act8<kActGelu>(x, out, deriv); break;
      case kActSilu: act8<kActSilu>(x, out, deriv); break;
      default: act8<kActIdentity>(x, out, deriv); break;
    }
    *reinterpret_cast<uint4*>(p.D + (long long)g * p.d_group_stride + (long long)r * p.d_row_stride + n) = out;
    if (p.aux != nullptr)
      *reinterpret_cast<uint4*>(p.aux + (long long)g * p.aux_group_stride + (long long)r * p.aux_row_stride + n) = deriv;
  }
}

}  // namespace

// Few rows, and at most a third of the SMs have a wide tile.  us with 8 rows a group and weights from HBM, tiles of 256 and of 64
// columns (wide tiles, groups x contraction x columns): 8 (4 x 2048 x 512) 19.1 and 9.0, 16 (1 x 4096 x 4096) 34.6 and 14.8, 32 (8 x 4096
// x 1024) 34.5 and 15.7, 40 (5 x 2048 x 2048) 20.1 and 11.0, 48 (48 x 512 x 256) 8.8 and 7.2.  With one K block a stage 64 wide tiles
// would gain, too (8 x 2048 x 2048: 21.0 and 13.6), 128 lose (8 x 1024 x 4096: 15.3 and 17.3): there the wide ones are loads enough
// for the chip.
bool stream_gemm_pays(int groups, int M, int N, int sms) {
  return M <= kStreamRows && 3ll * groups * ((N + BN - 1) / BN) <= sms;
}

cudaError_t launch_stream_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const StreamGemm& p, cudaStream_t stream) {
  static std::atomic<unsigned long long> told{0};
  if (const cudaError_t e = allow_smem(stream_gemm_kernel, (int)kSmemTotal, told); e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.groups * ((p.N + kStreamCols - 1) / kStreamCols)), 1, 1);      // few, see stream_gemm_pays
  cfg.blockDim = dim3(kStreamThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;     // see launch.cuh
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, stream_gemm_kernel, ta, tb, p);
}

}  // namespace planmoe
