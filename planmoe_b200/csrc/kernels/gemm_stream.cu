// Grouped bf16 GEMM for a handful of rows a group: y[g] = act(x[g] . w[g] + b[g]) with at most 32 rows, w [K, N] with N
// contiguous.  A decoding step or a small batch meets every expert's weights; reading them is all the work there is.
//
// One CTA per 128 x 256 tile over the whole contraction (gemm_tcgen05.cu) leaves SMs without loads in flight where there are few
// tiles: 8 experts of 4096 x 1024 are 32 CTAs.  Here a cluster of up to eight CTAs shares a tile and splits its contraction; each
// keeps a partial sum in TMEM, lays it out in shared memory, and adds up a share of the columns over the cluster's shared
// memories in CTA order, so that results do not depend on timing.  Two CTAs fit on an SM.  Groups without a token read no
// weights: their rows are zeros, so that the bias is all there is.  For which launches: stream_gemm_pays.
//
//   warp 0      TMA producer       warp 1   MMA issuer (tcgen05.mma.cta_group::1, 128 x 256 x 16; rows behind the tile's are
//                                           whatever lies behind them in shared memory and are never read back)
//   warps 2..5  partial sums to shared memory; then all warps add up and store
// No cluster multicast of loads.  Every wait is bounded.

#include "planmoe.h"
#include "kernels/gemm_local.h"
#include "kernels/gemm_tc.cuh"

namespace planmoe {

namespace {

constexpr int kStreamThreads = 192;
constexpr int kMaxSplit = 8;
constexpr uint32_t kBBytes = BN * BK * 2;          // 32 KiB
constexpr int kPartRow = BN + 4;                   // floats between rows of a partial sum: lanes on different banks

constexpr uint32_t kABytes = kStreamRows * BK * 2, kStage = kABytes + kBBytes;
constexpr int kStages = 3;
constexpr uint32_t kRing = kStages * kStage, kSmemTotal = kRing + 256;
static_assert(kStreamRows * kPartRow * 4 <= kRing, "the partial sum takes the ring's place");
static_assert(kABytes + 128 * 128 <= kStage, "the MMA reads 128 rows from the stage's start");

struct StreamCtl {
  uint64_t full[kStages], empty[kStages], acc_full;
  uint32_t tmem_base;
  volatile int abort;
};
static_assert(sizeof(StreamCtl) <= 256, "control block");

__device__ __forceinline__ float4 ld_cluster(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

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
  StreamCtl* const ctl = reinterpret_cast<StreamCtl*>(smem + kRing);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int nt_count = (p.N + BN - 1) / BN, tile = (int)blockIdx.x / p.split;
  const int g = tile / nt_count, n0 = (tile - g * nt_count) * BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(smem_u32(&ctl->full[s]), 1); mbar_init(smem_u32(&ctl->empty[s]), 1); }
    mbar_init(smem_u32(&ctl->acc_full), 1);
    ctl->abort = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc<1>(smem_u32(&ctl->tmem_base), BN);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl->tmem_base;

  chain_begin();
  // this CTA's K blocks; none where the group holds no token
  const int kb_total = (p.K + BK - 1) / BK, per = (kb_total + p.split - 1) / p.split;
  const int kb0 = rank * per;
  const bool live = p.rows_used == nullptr || p.rows_used[g] > 0;
  const int kbs = live ? max(0, min(per, kb_total - kb0)) : 0;

  if (warp == 0) {
    const bool leader = elect_one();
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int kb = 0; kb < kbs; ++kb) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->empty[stage]), phase ^ 1u, &ctl->abort, p.budget_ns, p.status, 0, stage));
      if (!ok) break;
      if (leader) {
        const uint32_t full = smem_u32(&ctl->full[stage]), sa = smem_u32(smem) + stage * kStage, sb = sa + kABytes;
        const int k0 = (kb0 + kb) * BK;
        mbar_expect_tx(full, kStage);
        tma_load_4d<1>(sa, &tmA, full, k0, 0, g, 0);
#pragma unroll
        for (int h = 0; h < BN / 64; ++h) tma_load_4d<1>(sb + h * (64 * BK * 2), &tmB, full, n0 + h * 64, k0, g, 0);
      }
      __syncwarp();
      if (++stage == kStages) { stage = 0; phase ^= 1u; }
    }
    if (!ok) __nanosleep(200000);                  // let copies already in flight land before teardown
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(false, true, BM);
    const bool leader = elect_one();
    uint32_t stage = 0, phase = 0;
    bool ok = true;
    for (int kb = 0; kb < kbs; ++kb) {
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->full[stage]), phase, &ctl->abort, p.budget_ns, p.status, 1, stage));
      if (!ok) break;
      tc_fence_after();
      if (leader) {
        const uint32_t sa = smem_u32(smem) + stage * kStage, sb = sa + kABytes;
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_bf16<1>(tmem, make_desc(sa + k * (UMMA_K * 2), 16, 1024), make_desc(sb + k * (UMMA_K * 128), 64 * BK * 2, 1024), idesc,
                       (kb | k) != 0 ? 1u : 0u);
        umma_commit<1>(smem_u32(&ctl->empty[stage]));
      }
      __syncwarp();
      if (++stage == kStages) { stage = 0; phase ^= 1u; }
    }
    if (ok && kbs > 0 && leader) umma_commit<1>(smem_u32(&ctl->acc_full));
    __syncwarp();
  } else {
    // The partial sum of row q * 32 + lane, laid over the ring: every load has been read by an MMA that has completed.
    const int q = warp & 3, row = q * 32 + lane;
    if (q * 32 < p.M) {
      bool ok = true;
      if (kbs > 0)
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&ctl->acc_full), 0, &ctl->abort, p.budget_ns, p.status, 2, 0));
      if (ok) {
        tc_fence_after();
        float* const out = reinterpret_cast<float*>(smem) + row * kPartRow;
#pragma unroll 1
        for (int c = 0; c < BN; c += 64) {
          uint32_t v[64];
          if (kbs > 0) {
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + c, v);
            tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + c + 32, v + 32);
            tmem_ld_wait();
            tmem_ld_ready(v);
            tmem_ld_ready(v + 32);
          } else {
#pragma unroll
            for (int i = 0; i < 64; ++i) v[i] = 0u;
          }
          if (row < p.M) {
#pragma unroll
            for (int i = 0; i < 64; i += 4) *reinterpret_cast<uint4*>(out + c + i) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                              // every CTA's partial sum is in place
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<1>(tmem, BN);
  }

  // columns [rank, rank + 1) * BN / split of the tile, eight at a time, over the cluster's partial sums in CTA order
  if (!ctl->abort) {
    const int width = BN / p.split, vecs = width / 8;
    for (int i = threadIdx.x; i < p.M * vecs; i += kStreamThreads) {
      const int r = i / vecs, c = rank * width + (i - r * vecs) * 8, n = n0 + c;
      if (n >= p.N) continue;                      // N is a multiple of 8
      const uint32_t at = smem_u32(smem) + (uint32_t)(r * kPartRow + c) * 4u;
      pair_t x[4] = {0ull, 0ull, 0ull, 0ull};
      for (int s = 0; s < p.split; ++s) {
        const uint32_t src = map_to_cta(at, (uint32_t)s);
        const float4 a = ld_cluster(src), b = ld_cluster(src + 16);
        x[0] = add_pair(x[0], pair_of(a.x, a.y)); x[1] = add_pair(x[1], pair_of(a.z, a.w));
        x[2] = add_pair(x[2], pair_of(b.x, b.y)); x[3] = add_pair(x[3], pair_of(b.z, b.w));
      }
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
  cluster_sync_all();                              // nobody leaves while its partial sum may still be read
}

}  // namespace

// Few rows and tiles for at most a third of the SMs.  us with 8 rows a group, one CTA a tile and split: 32 tiles (8 x 4096 x 1024) 34
// and 16, 16 tiles (1 x 4096 x 4096) 34 and 16, 8 tiles (4 x 2048 x 512) 19 and 8; 64 tiles 21 and 25 (8 x 2048 x 2048) or 37 and 31 (32 x
// 4096 x 512); 128 tiles (8 x 1024 x 4096) 15 and 21.  With 64 rows the partial sums cost more than the split gives (8 x 4096 x 1024: 35
// and 43).
bool stream_gemm_pays(int groups, int M, int N, int sms) {
  return M <= kStreamRows && 3ll * groups * ((N + BN - 1) / BN) <= sms;
}

// Splits until there are two CTAs for every SM, with at least four K blocks each: what a split adds is the exchange of its
// partial sum.
cudaError_t launch_stream_gemm(const CUtensorMap& ta, const CUtensorMap& tb, StreamGemm p, int sms, cudaStream_t stream) {
  const int tiles = p.groups * ((p.N + BN - 1) / BN), kbs = (p.K + BK - 1) / BK;       // few, see stream_gemm_pays
  p.split = 1;
  while (p.split < kMaxSplit && tiles * p.split < 2 * sms && kbs >= 8 * p.split) p.split *= 2;
  static const cudaError_t configured = cudaFuncSetAttribute(stream_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemTotal);
  if (configured != cudaSuccess) return configured;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles * p.split), 1, 1);
  cfg.blockDim = dim3(kStreamThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;     // see launch.cuh
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, stream_gemm_kernel, ta, tb, p);
}

}  // namespace planmoe
