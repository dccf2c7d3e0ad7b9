// gemm_split.cu — the contraction kernel for launches that cannot fill the GPU with 128 x 256 tiles (gemm_sm100.cu): a few rows,
// short sequences, one sample's low-resolution convolution.  Same operands, same products, same results as launch_gemm's form
//
//   Y[m, n] = act( sum_k A[m, k] * W[n, k] + bias[n] ) (+ residual[m, n])          (LayerOps.hpp:24-111)
//
// What bounds such a launch is not the tensor pipe but how many SMs take part and how long the chain of one tile is.  So:
//   * the weights are the M side of the MMA (TMEM lane = output feature) and `bn` activation rows (16 ... 128) its N side: a tile
//     of 40 rows costs a 48-column instruction, not a 256-column one, and each k-step still consumes 128 rows of weights;
//   * K is cut into `splits` ranges that the CTAs of one thread-block cluster take; their partial tiles meet through distributed
//     shared memory (CTA j sums column slice j of all partials, in split order: deterministic) and each CTA finishes its slice;
//   * one tile per CTA, no persistent loop; the accumulators leave through shared memory, so that row-major results are stored
//     with a lane per output feature and channel-major ones with a lane per pixel, both coalesced;
//   * launched with programmatic stream serialization: barriers, tensor memory and the first stages of WEIGHTS are set up while
//     the producing kernel still runs; only the activation loads and everything after wait for it.
// The tile width and the split count come from a small cost model (plan_split) whose constants were fitted to measurements.
#include "common.h"
#include "planes.cuh"
#include "sm100_ptx.cuh"
#include "epilogue.cuh"
#include "launch.cuh"
#include "tensor_map.h"

#include <cstdlib>

namespace mb {
namespace {

constexpr int SG_THREADS = 256;
constexpr int SG_M = 128;            // weight rows of a tile
constexpr int SG_MAX_BN = 128;
constexpr int SG_MAX_STAGES = 8;
constexpr int SG_RING_LIMIT = 212992;  // 208 KB of operand stages; the partial tiles reuse them
constexpr int SG_RING_TWO = 106496;    // 104 KB: two CTAs to an SM
constexpr int SG_MAX_SPLITS = 16;      // (above eight: the non-portable cluster size)

// Cost model (SM cycles): constants fitted to 20 shapes x 30 (width, split) pairs on B200, cold L2 (K = 256 ... 32768, 24 ... 5120 rows);
// over those the chosen launch is within 1 % of the best one in the geometric mean.
constexpr double SG_PER_BLOCK = 175.0;     // issue of a k-block beyond its MMAs
constexpr double SG_FIXED = 10600.0;       // launch, barriers, first loads, drain
constexpr double SG_TAIL_PER_COL = 70.0;   // accumulators -> shared memory -> output, per column of the tile
constexpr double SG_SPLIT = 970.0, SG_SPLIT_PER_COL = 30.0;  // cluster barriers and the partial tiles through distributed shared memory
constexpr double SG_LOAD_ALL = 51.6, SG_LOAD_MAX = 68.8;     // operand bytes per cycle an SM gets with all / few SMs loading

constexpr float SHRINK_PER_MMA = 3.1e-8f;

struct SplitGemmParams {
  int m, n, kblocks;
  int tiles_o, bn, splits;
  const float* bias;
  const float* residual;
  int activation;
  float* out_f32;
  long long ldo;
  __nv_bfloat16* out_split;
  long long np;
  int ohw;
  int conv_ks, conv_cblocks, conv_pad, conv_hp, conv_wp, conv_h, conv_w;
  float acc_scale;
  float shrink;  // what a partial sum would have lost per k-block that follows its range (see split_weight)
  int f16, stages, stage_bytes, w_ready;
  int* err_word;
};

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// Weight of split s's partial sum.  The tensor core adds with truncation, so in ONE accumulator over all of K the contribution of an
// early range would have shrunk a little with every MMA that came after it.  The weights apply that shrinkage to the ranges that
// were summed apart, and the result is then scaled as the unsplit kernel's is: a row gives the same answer in a small batch
// (here) and in a large one (gemm_sm100.cu).  Relative difference of the two kernels' results, 40 x 1024 outputs, eight splits,
// three MMAs per product: K = 32768 1.0e-4 unweighted, 1e-5 weighted (each is 5.3e-5 from the fp64 product); K = 2048 6.5e-6 and
// 9e-7.  Fitted: 3e-8 ... 3.2e-8 per MMA at every K and product count.
__device__ __forceinline__ float split_weight(const SplitGemmParams& p, int s) {
  const int end = static_cast<int>(static_cast<long long>(p.kblocks) * (s + 1) / p.splits);
  return 1.0f - p.shrink * static_cast<float>(p.kblocks - end);
}

template <int BK, int AP, int WP>  // AP, WP: operand planes of the activations and the weights
__global__ void __launch_bounds__(SG_THREADS, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const SplitGemmParams p) {
  constexpr int SWZ = BK * 2;
  constexpr int W_TILE = SG_M * BK * 2;
  const int A_TILE = p.bn * BK * 2;
  extern __shared__ __align__(1024) uint8_t sg_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sg_smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[SG_MAX_STAGES], empty_bar[SG_MAX_STAGES], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ long long col_off[SG_MAX_BN];  // where a column (activation row) lands in the output; -1 = nowhere

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int split = static_cast<int>(blockIdx.x) % p.splits;
  const int tile = static_cast<int>(blockIdx.x) / p.splits;
  const int to = tile % p.tiles_o, tr = tile / p.tiles_o;
  const int kb0 = static_cast<int>(static_cast<long long>(p.kblocks) * split / p.splits);
  const int kb1 = static_cast<int>(static_cast<long long>(p.kblocks) * (split + 1) / p.splits);
  const uint32_t tmem_cols = p.bn <= 32 ? 32u : (p.bn <= 64 ? 64u : 128u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, tmem_cols);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  // (behind the allocation: a kernel that starts now may take all of an SM's tensor memory and then wait for this one)
  pdl_launch_dependents();
  const uint32_t tmem = tmem_slot;
  const bool conv = p.conv_ks > 0;

  if (warp == 0) {
    const bool one = elect_one();
    const uint32_t tx = static_cast<uint32_t>(WP * W_TILE + AP * A_TILE);
    auto load_w = [&](int kb, int stage) {
      if (!one) return;
      mbar_expect_tx(&full_bar[stage], tx);
      uint8_t* s = smem + stage * p.stage_bytes;
      tma_load_3d(s, &map_w, &full_bar[stage], kb * BK, to * SG_M, 0);
      if (WP == 2) tma_load_3d(s + W_TILE, &map_w, &full_bar[stage], kb * BK, to * SG_M, 1);
    };
    auto load_a = [&](int kb, int stage) {
      uint8_t* s = smem + stage * p.stage_bytes + WP * W_TILE;
      int col = kb * BK, row = tr * p.bn;
      if (conv) {
        const int t = kb / p.conv_cblocks, kh = t / p.conv_ks, kw = t - kh * p.conv_ks;
        row += (kh - p.conv_pad) * p.conv_wp + (kw - p.conv_pad);  // may be negative: TMA zero-fills
        col = (kb - t * p.conv_cblocks) * BK;
      }
      if (!one) return;
      tma_load_3d(s, &map_a, &full_bar[stage], col, row, 0);
      if (AP == 2) tma_load_3d(s + A_TILE, &map_a, &full_bar[stage], col, row, 1);
    };
    // the weights of the first stages do not depend on the kernel before this one
    const int pre = min(p.stages, kb1 - kb0);
    if (!p.w_ready) pdl_wait();
    for (int i = 0; i < pre; ++i) load_w(kb0 + i, i);
    pdl_wait();
    for (int i = 0; i < pre; ++i) load_a(kb0 + i, i);
    int stage = pre == p.stages ? 0 : pre;
    uint32_t phase = pre == p.stages ? 1 : 0;
    for (int kb = kb0 + pre; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, &abort_flag, p.err_word, 41)) break;
      load_w(kb, stage);
      load_a(kb, stage);
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    __syncwarp();
  } else if (warp == 1) {
    const bool one = elect_one();
    const uint32_t idesc = make_idesc(SG_M, p.bn, p.f16);
    int stage = 0;
    uint32_t phase = 0;
    bool ready = false;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(&full_bar[stage], phase, &abort_flag, p.err_word, 42)) break;
      tcgen05_fence_after();
      const uint32_t sw = smem_u32(smem + stage * p.stage_bytes), sa = sw + WP * W_TILE;
      const uint64_t dw = make_smem_desc(sw, SWZ), da = make_smem_desc(sa, SWZ);
      const uint64_t dw_lo = dw + (W_TILE >> 4), da_lo = da + (A_TILE >> 4);
      uint64_t* done = &empty_bar[stage];
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
      ready = mbar_test(&full_bar[stage], phase);
      if (one) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {  // 32 bytes further along K = 2 in the descriptor's address field
          umma_bf16(tmem, dw + 2 * k, da + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          if (AP == 2) umma_bf16(tmem, dw + 2 * k, da_lo + 2 * k, idesc, 1u);
          if (WP == 2) umma_bf16(tmem, dw_lo + 2 * k, da + 2 * k, idesc, 1u);
        }
        umma_commit(done);
      }
      __syncwarp();
    }
    if (one) umma_commit(&acc_bar);
    __syncwarp();
  }

  // every thread below reads or writes memory that the previous kernels of the stream may still be using
  pdl_wait();
  const bool chan_major = conv || p.ohw > 0;
  if (threadIdx.x < p.bn) {
    const int row = tr * p.bn + static_cast<int>(threadIdx.x);
    long long off = -1;
    if (row < p.m) {
      if (conv) {
        const int per = p.conv_hp * p.conv_wp, smp = row / per, rem = row - smp * per, yq = rem / p.conv_wp;
        const int yy = yq - p.conv_pad, xx = rem - yq * p.conv_wp - p.conv_pad;
        if (yy >= 0 && yy < p.conv_h && xx >= 0 && xx < p.conv_w)
          off = (static_cast<long long>(smp) * p.n * p.conv_h + yy) * p.conv_w + xx;
      } else if (p.ohw > 0) {
        const int smp = row / p.ohw;
        off = static_cast<long long>(smp) * p.n * p.ohw + (row - smp * p.ohw);
      } else {
        off = row;
      }
    }
    col_off[threadIdx.x] = off;
  }
  {
    int ok = 1;
    if (lane == 0) ok = mbar_wait(&acc_bar, 0, &abort_flag, p.err_word, 43) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) while (!mbar_try_wait(&acc_bar, 0)) {}  // completes at once: lane 0 saw the phase
  }
  tcgen05_fence_after();
  // The ring is free now (all MMAs have read it); with several CTAs to a tile, in every one of them.
  if (p.splits > 1) cluster_sync_all(); else __syncthreads();

  // accumulators -> staging tile of the CTA that finishes their columns: [split][column of the slice][pitch] floats
  float* stg = reinterpret_cast<float*>(smem);
  const int slice = p.bn / p.splits;
  const int pitch = chan_major ? SG_M + 1 : SG_M;  // channel-major tiles are read with a lane per column
  const int quad = warp & 3;
  const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
  for (int c0 = (warp >> 2) * 16; c0 < p.bn; c0 += 32) {
    float v[16];
    tmem_ld_32x16(taddr + c0, v);
    if (p.splits == 1) {
#pragma unroll
      for (int j = 0; j < 16; ++j) stg[(c0 + j) * pitch + quad * 32 + lane] = v[j];
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int owner = (c0 + j) / slice, cl = c0 + j - owner * slice;
        st_cluster_f32(mapa_shared(smem_u32(stg + (split * slice + cl) * pitch + quad * 32 + lane), owner), v[j]);
      }
    }
  }
  tcgen05_fence_before();
  if (p.splits > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }

  const int oc0 = to * SG_M, col_base = split * slice;
  if (!chan_major) {
    // a warp takes a row, a lane four consecutive output features
    const int oc = oc0 + lane * 4;
    const bool vec = ((p.ldo & 3) == 0) && oc + 4 <= p.n &&
                     ((reinterpret_cast<uintptr_t>(p.out_f32) | reinterpret_cast<uintptr_t>(p.residual)) & 15) == 0;
    float b[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias != nullptr) {
#pragma unroll
      for (int e = 0; e < 4; ++e) if (oc + e < p.n) b[e] = __ldg(p.bias + oc + e);
    }
    for (int cl = warp; cl < slice; cl += SG_THREADS / 32) {
      const long long row = col_off[col_base + cl];
      if (row < 0) continue;  // warp-uniform
      const float* src = stg + cl * pitch + lane * 4;
      float4 a = *reinterpret_cast<const float4*>(src + (p.splits - 1) * slice * pitch);  // (the last range's weight is 1)
      for (int s = p.splits - 2; s >= 0; --s) {
        const float4 q = *reinterpret_cast<const float4*>(src + s * slice * pitch);
        const float w = split_weight(p, s);
        a.x = fmaf(q.x, w, a.x); a.y = fmaf(q.y, w, a.y); a.z = fmaf(q.z, w, a.z); a.w = fmaf(q.w, w, a.w);
      }
      float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = apply_act(__fmaf_rn(v[e], p.acc_scale, b[e]), p.activation);
      const long long o = row * p.ldo + oc;
      if (p.residual != nullptr) {
        if (vec) {
          const float4 r = __ldg(reinterpret_cast<const float4*>(p.residual + o));
          v[0] += r.x; v[1] += r.y; v[2] += r.z; v[3] += r.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) if (oc + e < p.n) v[e] += __ldg(p.residual + o + e);
        }
      }
      if (p.out_f32 != nullptr) {
        if (vec) *reinterpret_cast<float4*>(p.out_f32 + o) = make_float4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
          for (int e = 0; e < 4; ++e) if (oc + e < p.n) p.out_f32[o + e] = v[e];
        }
      }
      if (p.out_split != nullptr && oc < p.np) {
        // columns n .. np - 1 are written as zero (the consumer's padded K)
        uint32_t h[2], l[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = oc + e < p.n ? v[e] : 0.0f;
        split_pair(v[0], v[1], p.f16, h[0], l[0]);
        split_pair(v[2], v[3], p.f16, h[1], l[1]);
        __nv_bfloat16* oh = p.out_split + row * p.np + oc;
        *reinterpret_cast<uint2*>(oh) = make_uint2(h[0], h[1]);
        *reinterpret_cast<uint2*>(oh + static_cast<long long>(p.m) * p.np) = make_uint2(l[0], l[1]);
      }
    }
  } else {
    // a lane takes a pixel; consecutive lanes run over the slice's pixels first
    const long long hw = conv ? static_cast<long long>(p.conv_h) * p.conv_w : static_cast<long long>(p.ohw);
    const int nch = min(SG_M, p.n - oc0);
    for (int i = threadIdx.x; i < slice * nch; i += SG_THREADS) {
      const int ch = i / slice, cl = i - ch * slice;
      const long long off = col_off[col_base + cl];
      if (off < 0) continue;
      const float* src = stg + cl * pitch + ch;
      float a = src[(p.splits - 1) * slice * pitch];
      for (int s = p.splits - 2; s >= 0; --s) a = fmaf(src[s * slice * pitch], split_weight(p, s), a);
      a = __fmaf_rn(a, p.acc_scale, p.bias != nullptr ? __ldg(p.bias + oc0 + ch) : 0.0f);
      a = apply_act(a, p.activation);
      const long long o = off + static_cast<long long>(oc0 + ch) * hw;
      if (p.residual != nullptr) a += __ldg(p.residual + o);
      p.out_f32[o] = a;
    }
  }
}

// Tile width and split count of one launch and its estimated time in SM cycles.
struct SplitPlan { int bn = 0, splits = 0; double cycles = 1e30; };

SplitPlan plan_split(const GemmArgs& g, int bk, int kblocks) {
  const int sms = ctx().sm_count;
  const int products = 1 + (g.a_planes == 2) + (g.w_planes == 2);
  const int tiles_o = (g.n + SG_M - 1) / SG_M;
  SplitPlan best;
  static const int widths[] = {16, 32, 48, 64, 96, 128};
  for (int bn : widths) {
    if (bn > 16 && bn >= g.m + 32) break;
    const long long tiles = static_cast<long long>(tiles_o) * ((g.m + bn - 1) / bn);
    const int stage = (g.w_planes * SG_M + g.a_planes * bn) * bk * 2;
    for (int splits = 1; splits <= SG_MAX_SPLITS; splits *= 2) {
      // (clusters of sixteen: one GPC each, and not every GPC has sixteen SMs free - eight of them took 57 us where sixteen-SM
      // work in clusters of eight took 46)
      if (bn % splits != 0 || splits > kblocks || (splits > 8 && tiles > 4)) break;
      const long long ctas = tiles * splits;
      // CTAs that share an SM overlap one's loads and stores with the other's MMAs: whole rounds of two per SM
      const bool two = ctas > sms && 2 * stage <= SG_RING_TWO && bn * (SG_M + 1) * 4 <= SG_RING_TWO;
      const long long rounds = two ? (ctas + 2 * sms - 1) / (2 * sms) : (ctas + sms - 1) / sms;
      const int kb = (kblocks + splits - 1) / splits;
      const double share = two ? static_cast<double>(ctas < 2 * sms ? (ctas + sms - 1) / sms : 2) : 1.0;
      const double mma = share * kb * ((bk / 16) * products * (bn > 92 ? bn * 0.5 : 46.0) + SG_PER_BLOCK);
      const double busy = static_cast<double>(ctas < sms ? ctas : sms) / sms;
      const double load = share * kb * stage / (SG_LOAD_MAX - (SG_LOAD_MAX - SG_LOAD_ALL) * busy);
      const double tail = SG_FIXED + bn * SG_TAIL_PER_COL + (splits > 1 ? SG_SPLIT + bn * SG_SPLIT_PER_COL : 0.0);
      const double t = static_cast<double>(rounds) * ((mma > load ? mma : load) + tail);
      if (t < best.cycles) { best.bn = bn; best.splits = splits; best.cycles = t; }
    }
  }
  return best;
}

template <int BK, int AP, int WP>
int launch_split_t(const GemmArgs& g, const SplitPlan& plan, cudaStream_t st) {
  const bool conv = g.conv_ks > 0;
  const int kp = round_up(g.k, 64);
  CUtensorMap map_a, map_w;
  MB_TRY(make_plane_map(&map_a, g.a, g.a_planes, g.m, conv ? g.conv_c : kp, BK, plan.bn));
  MB_TRY(make_plane_map(&map_w, g.w, g.w_planes, g.n, kp, BK, SG_M));
  SplitGemmParams p;
  p.m = g.m; p.n = g.n;
  p.kblocks = conv ? g.conv_ks * g.conv_ks * (g.conv_c / BK) : kp / BK;
  p.tiles_o = (g.n + SG_M - 1) / SG_M;
  p.bn = plan.bn; p.splits = plan.splits;
  p.bias = g.bias; p.residual = g.residual; p.activation = g.activation;
  p.out_f32 = g.out_f32; p.ldo = g.ldo; p.out_split = g.out_split; p.np = round_up(g.n, 64); p.ohw = g.out_nchw_hw;
  p.conv_ks = g.conv_ks; p.conv_cblocks = conv ? g.conv_c / BK : 1; p.conv_pad = g.conv_pad;
  p.conv_hp = g.conv_h + 2 * g.conv_pad; p.conv_wp = g.conv_w + 2 * g.conv_pad; p.conv_h = g.conv_h; p.conv_w = g.conv_w;
  p.acc_scale = gemm_acc_scale(g);
  p.shrink = SHRINK_PER_MMA * (BK / 16) * (AP + WP - 1);
  p.f16 = plane_format() == PLANES_F16 ? 1 : 0;
  p.w_ready = g.w_ready ? 1 : 0;
  p.err_word = ctx().dev_error_word;
  p.stage_bytes = (WP * SG_M + AP * p.bn) * BK * 2;
  const int per_split = (p.kblocks + p.splits - 1) / p.splits;
  const long long ctas = static_cast<long long>(p.tiles_o) * ((g.m + p.bn - 1) / p.bn) * p.splits;
  const bool two = ctas > ctx().sm_count && 2 * p.stage_bytes <= SG_RING_TWO && p.bn * (SG_M + 1) * 4 <= SG_RING_TWO;
  p.stages = (two ? SG_RING_TWO : SG_RING_LIMIT) / p.stage_bytes;
  if (p.stages > SG_MAX_STAGES) p.stages = SG_MAX_STAGES;
  if (p.stages > per_split) p.stages = per_split;
  const int staging = p.bn * (SG_M + 1) * 4, ring = p.stages * p.stage_bytes;
  const int smem = (ring > staging ? ring : staging) + 1024;
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BK, AP, WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_RING_LIMIT + 1024));
    MB_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BK, AP, WP>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return MIMIR_B200_OK;
  }));
  GemmProfile prof(st);
  MB_TRY(prof.begin());
  MB_TRY(launch_pdl(gemm_split_kernel<BK, AP, WP>, dim3(static_cast<unsigned>(ctas)), dim3(SG_THREADS), static_cast<size_t>(smem), st, p.splits, map_a, map_w, p));
  MB_TRY(prof.end());
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace

double gemm_split_cycles(const GemmArgs& g, int bk, int* bn, int* splits) {
  constexpr double never = 1e30;
  if (g.a_group_rows > 0 || g.gn_part != nullptr) return never;
  const int kblocks = g.conv_ks > 0 ? g.conv_ks * g.conv_ks * (g.conv_c / bk) : round_up(g.k, 64) / bk;
  const char* e = getenv("MIMIR_B200_GEMM_SPLIT");  // "0": never; "<bn>,<splits>": always, in that shape
  if (e && e[0] == '0' && e[1] == '\0') return never;
  int fb = 0, fs = 0;
  if (e && sscanf(e, "%d,%d", &fb, &fs) == 2) {
    *bn = fb; *splits = fs;
    return fb >= 16 && fb <= SG_MAX_BN && fb % 16 == 0 && fs >= 1 && fs <= SG_MAX_SPLITS && fb % fs == 0 && fs <= kblocks ? 0.0 : never;
  }
  const SplitPlan plan = plan_split(g, bk, kblocks);
  *bn = plan.bn; *splits = plan.splits;
  // (convolutions: shifted row blocks and channel-major stores, 1.3 to 1.4 times the estimate in 25 shapes)
  return plan.cycles * (g.conv_ks > 0 || g.out_nchw_hw > 0 ? 1.35 : 1.0);
}

int launch_gemm_split(const GemmArgs& g, int bk, int bn, int splits, cudaStream_t st) {
  SplitPlan plan;
  plan.bn = bn; plan.splits = splits;
  if (g.a_planes == 2 && g.w_planes == 2) return bk == 64 ? launch_split_t<64, 2, 2>(g, plan, st) : launch_split_t<32, 2, 2>(g, plan, st);
  if (g.a_planes == 2 && g.w_planes == 1) return bk == 64 ? launch_split_t<64, 2, 1>(g, plan, st) : launch_split_t<32, 2, 1>(g, plan, st);
  if (g.a_planes == 1 && g.w_planes == 1) return bk == 64 ? launch_split_t<64, 1, 1>(g, plan, st) : launch_split_t<32, 1, 1>(g, plan, st);
  return fail(MIMIR_B200_E_INVALID, "gemm: %d activation and %d weight planes", g.a_planes, g.w_planes);
}

}  // namespace mb
