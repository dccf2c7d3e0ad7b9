// gemm_split.cu — the contraction kernel for launches that cannot fill the GPU with 128 x 256 tiles (gemm_sm100.cu): a few rows,
// short sequences, one sample's low-resolution convolution.  Same operands, same products as launch_gemm's form, and results that differ
// from its by the order of their sums only (split_weights)
//
//   Y[m, n] = act( sum_k A[m, k] * W[n, k] + bias[n] ) (+ residual[m, n])          (LayerOps.hpp:24-111)
//
// What bounds such a launch is not the tensor pipe but how many SMs take part and how long the chain of one tile is.  So:
//   * the weights are the M side of the MMA (TMEM lane = output feature) and `bn` activation rows (16 ... 128) its N side, their two
//     planes behind one another as ONE operand of 2 bn columns: an instruction of up to 92 columns costs the same 46 cycles, so
//     hi and lo together cost little more than hi alone, and the sums of the small products get columns of their own;
//   * K is cut into `splits` ranges that the CTAs of one thread-block cluster take; their partial tiles meet through distributed
//     shared memory (CTA j sums column slice j of all partials, in split order: deterministic) and each CTA finishes its slice;
//   * one tile per CTA, no persistent loop.  Row-major results leave from the registers that read tensor memory (a lane per output
//     feature, swapped with its neighbour for 8-byte accesses), channel-major ones through shared memory with a lane per pixel;
//   * sixteen warps finish a tile.  The tail was half of such a launch: eight warps took 0.5 to 1 us for each eight columns, a chain
//     of dependent instructions (index divisions, a branch per element, a residual load waited for on the spot) at two warps
//     to an issue slot.  333 x 1000 x 1000 by CTA stamps, from the input's arrival to the last store: 9.5 -> 5.9 us (accumulators
//     4.4 -> 3.6, exchange 2.2 -> 1.5, stores 2.9 -> 0.8); 1000 x 2304 x 768 10.6 -> 8, 1000 x 768 x 768 with a residual 9.5 -> 4.7;
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

constexpr int SG_THREADS = 512;
constexpr int SG_GROUPS = SG_THREADS / 128;  // column groups of the epilogue: four warps, one per tensor-memory lane quadrant, to a group
constexpr int SG_M = 128;            // weight rows of a tile
constexpr int SG_MAX_BN = 128;
constexpr int SG_MAX_STAGES = 8;
constexpr int SG_RING_LIMIT = 212992;  // 208 KB: operand stages and, where three stages remain, the partial tiles behind them (else in their place)
constexpr int SG_RING_TWO = 106496;    // 104 KB: two CTAs to an SM
constexpr int SG_MAX_SPLITS = 16;      // (above eight: the non-portable cluster size)

// Cost model (SM cycles): constants fitted to 25 shapes x 20 to 35 (width, split) pairs on B200, weights of 160 MB walked through
// (K = 256 ... 32768, 17 ... 5120 rows); over those the chosen launch is within 1 % of the best one in the geometric mean, 9 % at worst.
// A k-block costs what its operands take to arrive, or its MMAs where those are more; issuing them costs nothing beside that.
constexpr double SG_FIXED = 5100.0;        // launch, barriers, first loads, drain
constexpr double SG_TAIL_PER_COL = 36.0;   // accumulators -> output, per column that a CTA finishes
constexpr double SG_SPLIT = 1550.0, SG_SPLIT_PER_COL = 60.0;  // cluster barriers and the partial tiles through distributed shared memory
constexpr double SG_LOAD_ALL = 56.9, SG_LOAD_MAX = 62.9;      // operand bytes per cycle an SM gets with all / few SMs loading
// Channel-major results (30 convolutions, 32 ... 512 channels on 7^2 ... 112^2 pixels: within 1 % of the best of every form and the spatial
// tiles): taps find their operands in L2, scattered stores cost more.
constexpr double SG_CM_BLOCK = 0.9, SG_CM_FIXED = 7700.0, SG_CM_TAIL_PER_COL = 181.0;
constexpr double SG_TWO_TAIL = 1.27;       // a tail beside another CTA's main loop on the same SM

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
  const unsigned* w_amax;  // see GemmArgs
  int f16, stages, stage_bytes, w_ready;
  float weight[SG_MAX_SPLITS];  // of the ranges' partial sums (split_weights)
  int stg_off;  // the staging tile: behind the operand ring, or in its place (0)
  int* err_word;
};

__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Accesses under a predicate and not behind a branch, so that those of a chunk interleave.
__device__ __forceinline__ float2 ld_if(bool on, const float* p) {
  float2 v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t@q ld.global.nc.v2.f32 {%0, %1}, [%3];\n\t}"
               : "=&f"(v.x), "=&f"(v.y) : "r"(static_cast<int>(on)), "l"(p));
  return v;
}
__device__ __forceinline__ void st_if(bool on, float* p, float2 v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %0, 0;\n\t@q st.global.v2.f32 [%1], {%2, %3};\n\t}" ::"r"(static_cast<int>(on)), "l"(p), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void st_if(bool on, __nv_bfloat16* p, uint32_t v) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %0, 0;\n\t@q st.global.b32 [%1], %2;\n\t}" ::"r"(static_cast<int>(on)), "l"(p), "r"(v) : "memory");
}

// N accumulator columns of this lane's output feature; with two activation planes the products of the lo plane (and of the weights'
// lo plane) are in columns of their own, `bn` further on: far smaller sums, which the tensor core's truncating adds cannot cost
// what they cost the main one.
template <int N, int AP>
__device__ __forceinline__ void load_acc(uint32_t taddr, int bn, float (&v)[N]) {
  if (N == 16) {
    tmem_ld_32x16(taddr, *reinterpret_cast<float (*)[16]>(v));
    if (AP == 2) {
      float w[16];
      tmem_ld_32x16(taddr + bn, w);
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] += w[j];
    }
  } else {
    tmem_ld_32x8(taddr, *reinterpret_cast<float (*)[8]>(v));
    if (AP == 2) {
      float w[8];
      tmem_ld_32x8(taddr + bn, w);
#pragma unroll
      for (int j = 0; j < N; ++j) v[j] += w[j];
    }
  }
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
  const uint32_t tmem_cols = AP * p.bn <= 32 ? 32u : (AP * p.bn <= 64 ? 64u : (AP * p.bn <= 128 ? 128u : 256u));

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
  if (p.splits > 1 && p.stg_off > 0) cluster_arrive();  // (waited for ahead of the first store into another CTA)
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
    if (one) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&map_a)) : "memory");
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
    const uint32_t idesc = make_idesc(SG_M, AP * p.bn, p.f16), idesc_lo = make_idesc(SG_M, p.bn, p.f16);
    int stage = 0;
    uint32_t phase = 0;
    bool ready = false;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(&full_bar[stage], phase, &abort_flag, p.err_word, 42)) break;
      tcgen05_fence_after();
      const uint32_t sw = smem_u32(smem + stage * p.stage_bytes), sa = sw + WP * W_TILE;
      const uint64_t dw = make_smem_desc(sw, SWZ), da = make_smem_desc(sa, SWZ);
      const uint64_t dw_lo = dw + (W_TILE >> 4);
      uint64_t* done = &empty_bar[stage];
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
      ready = mbar_test(&full_bar[stage], phase);
      if (one) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {  // 32 bytes further along K = 2 in the descriptor's address field
          // (the lo plane of the activations lies behind the hi plane: one instruction covers both)
          umma_bf16(tmem, dw + 2 * k, da + 2 * k, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          if (WP == 2) umma_bf16(tmem + (AP == 2 ? p.bn : 0), dw_lo + 2 * k, da + 2 * k, idesc_lo, 1u);
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
  const float acc_scale = p.w_amax == nullptr ? p.acc_scale : p.acc_scale * plane_unscale(__ldg(p.w_amax));
  const int slice = (p.bn + p.splits - 1) / p.splits;  // columns a CTA finishes; the last ones fewer, or none
  const int oc0 = to * SG_M, row0 = tr * p.bn + split * slice;
  const int quad = warp & 3, group = warp >> 2;
  // Row-major results: a lane holds one output feature of eight columns (rows of Y) and swaps with its neighbour, so that it ends
  // with two consecutive features of four columns, c0 + 2 i + (lane & 1): 8-byte accesses, two rows to a warp instruction.
  const int odd = lane & 1, fe = oc0 + quad * 32 + (lane & ~1), first_row = row0 + odd;
  const int ldo = static_cast<int>(p.ldo), mine = min(slice, p.bn - split * slice), live = min(mine, p.m - row0) - odd;  // (column c0 + 2 i is written where c0 + 2 i < live)
  const bool vec = ((ldo & 1) == 0) && fe + 2 <= p.n && ((reinterpret_cast<uintptr_t>(p.out_f32) | reinterpret_cast<uintptr_t>(p.residual)) & 7) == 0;
  const bool one_by_one = !vec && fe < p.n;
  const bool has_res = p.residual != nullptr;
  float2 b2 = make_float2(0.f, 0.f), res[4];
  auto load_res = [&](int c0) {  // the residual of chunk c0: asked for one chunk ahead of its use
    const float* src = p.residual + static_cast<long long>(first_row + c0) * ldo + fe;
#pragma unroll
    for (int i = 0; i < 4; ++i) res[i] = ld_if(vec && c0 + 2 * i < live, src + static_cast<long long>(2 * i) * ldo);
    if (one_by_one) {
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        if (c0 + 2 * i >= live) break;
        const float x = __ldg(src + static_cast<long long>(2 * i) * ldo), y = fe + 1 < p.n ? __ldg(src + static_cast<long long>(2 * i) * ldo + 1) : 0.0f;
        if (i == 0) res[0] = make_float2(x, y); else if (i == 1) res[1] = make_float2(x, y); else if (i == 2) res[2] = make_float2(x, y); else res[3] = make_float2(x, y);
      }
    }
  };
  if (chan_major) {
    if (threadIdx.x < p.bn) {
      const int row = tr * p.bn + static_cast<int>(threadIdx.x);
      long long off = -1;
      if (row < p.m) {
        if (conv) {
          const int per = p.conv_hp * p.conv_wp, smp = row / per, rem = row - smp * per, yq = rem / p.conv_wp;
          const int yy = yq - p.conv_pad, xx = rem - yq * p.conv_wp - p.conv_pad;
          if (yy >= 0 && yy < p.conv_h && xx >= 0 && xx < p.conv_w)
            off = (static_cast<long long>(smp) * p.n * p.conv_h + yy) * p.conv_w + xx;
        } else {
          const int smp = row / p.ohw;
          off = static_cast<long long>(smp) * p.n * p.ohw + (row - smp * p.ohw);
        }
      }
      col_off[threadIdx.x] = off;
    }
  } else {
    if (p.bias != nullptr) {
      if (fe < p.n) b2.x = __ldg(p.bias + fe);
      if (fe + 1 < p.n) b2.y = __ldg(p.bias + fe + 1);
    }
    if (has_res) load_res(group * 8);
  }
  {
    int ok = 1;
    if (lane == 0) ok = mbar_wait(&acc_bar, 0, &abort_flag, p.err_word, 43) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok) while (!mbar_try_wait(&acc_bar, 0)) {}  // completes at once: lane 0 saw the phase
  }
  tcgen05_fence_after();
  const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
  float* stg = reinterpret_cast<float*>(smem + p.stg_off);
  const int pitch = chan_major ? SG_M + 1 : SG_M;  // channel-major tiles are read with a lane per column
  if (p.splits > 1 || chan_major) {
    // accumulators -> staging tile of the CTA that finishes their columns: [split][column of the slice][pitch] floats.  Where
    // it has the ring's place, every CTA of the cluster must have read its operands; else they need only have started.
    if (p.splits > 1) {
      if (p.stg_off == 0) cluster_sync_all(); else cluster_wait();
    }
    for (int c0 = group * 16; c0 < p.bn; c0 += 16 * SG_GROUPS) {
      float v[16];
      load_acc<16, AP>(taddr + c0, p.bn, v);
      int owner = p.splits > 1 ? c0 / slice : 0, cl = c0 - owner * slice;
      if (p.splits == 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j) stg[(c0 + j) * pitch + quad * 32 + lane] = v[j];
      } else {
        const uint32_t own = smem_u32(stg + split * slice * pitch + quad * 32 + lane);
        uint32_t at = mapa_shared(own, owner) + cl * pitch * 4;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          st_cluster_f32(at, v[j]);
          at += pitch * 4;
          if (++cl == slice && j < 15) { cl = 0; at = mapa_shared(own, ++owner); }
        }
      }
    }
    tcgen05_fence_before();
    if (p.splits > 1) cluster_sync_all(); else __syncthreads();
  }

  if (!chan_major) {
    for (int c0 = group * 8; c0 < mine; c0 += 8 * SG_GROUPS) {  // (warp-uniform)
      float v[8];
      if (p.splits == 1) {
        load_acc<8, AP>(taddr + c0, p.bn, v);
      } else {
        const float* src = stg + c0 * pitch + quad * 32 + lane;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.0f;
        for (int s = 0; s < p.splits; ++s) {  // in split order
          const float w = p.weight[s];
#pragma unroll
          for (int j = 0; j < 8; ++j) if (c0 + j < slice) v[j] = fmaf(src[j * pitch], w, v[j]);
          src += slice * pitch;
        }
      }
      float2 u[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * i] : v[2 * i + 1], 1);
        u[i] = odd ? make_float2(other, v[2 * i + 1]) : make_float2(v[2 * i], other);
        u[i].x = __fmaf_rn(u[i].x, acc_scale, b2.x);
        u[i].y = __fmaf_rn(u[i].y, acc_scale, b2.y);
      }
      if (p.activation == MIMIR_B200_ELT_GELU) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { u[i].x = gelu_ref(u[i].x); u[i].y = gelu_ref(u[i].y); }
      } else if (p.activation >= 0) {
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          float2 t = i == 0 ? u[0] : i == 1 ? u[1] : i == 2 ? u[2] : u[3];
          t.x = apply_act(t.x, p.activation); t.y = apply_act(t.y, p.activation);
          if (i == 0) u[0] = t; else if (i == 1) u[1] = t; else if (i == 2) u[2] = t; else u[3] = t;
        }
      }
      if (has_res) {
#pragma unroll
        for (int i = 0; i < 4; ++i) { u[i].x += res[i].x; u[i].y += res[i].y; }
        load_res(c0 + 8 * SG_GROUPS);
      }
      if (p.out_f32 != nullptr) {
        float* dst = p.out_f32 + static_cast<long long>(first_row + c0) * ldo + fe;
#pragma unroll
        for (int i = 0; i < 4; ++i) st_if(vec && c0 + 2 * i < live, dst + static_cast<long long>(2 * i) * ldo, u[i]);
        if (one_by_one) {
#pragma unroll 1
          for (int i = 0; i < 4; ++i) {
            if (c0 + 2 * i >= live) break;
            const float2 t = i == 0 ? u[0] : i == 1 ? u[1] : i == 2 ? u[2] : u[3];
            dst[static_cast<long long>(2 * i) * ldo] = t.x;
            if (fe + 1 < p.n) dst[static_cast<long long>(2 * i) * ldo + 1] = t.y;
          }
        }
      }
      if (p.out_split != nullptr) {
        // columns n .. np - 1 are written as zero (the consumer's padded K)
        const int np = static_cast<int>(p.np);
        __nv_bfloat16* dst = p.out_split + static_cast<long long>(first_row + c0) * np + fe;
        const long long plane = static_cast<long long>(p.m) * np;
        uint32_t h[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split_pair(fe < p.n ? u[i].x : 0.0f, fe + 1 < p.n ? u[i].y : 0.0f, p.f16, h[i], l[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          __nv_bfloat16* at = dst + static_cast<long long>(2 * i) * np;
          const bool in = fe < np && c0 + 2 * i < live;
          st_if(in, at, h[i]);
          st_if(in, at + plane, l[i]);
        }
      }
    }
  } else {
    // a lane takes a pixel; consecutive lanes run over the slice's pixels first
    const long long hw = conv ? static_cast<long long>(p.conv_h) * p.conv_w : static_cast<long long>(p.ohw);
    const int nch = min(SG_M, p.n - oc0), total = max(mine, 0) * nch, width = max(mine, 1);
    const int step_ch = SG_THREADS / width, step_cl = SG_THREADS - step_ch * width;
    int ch = static_cast<int>(threadIdx.x) / width, cl = static_cast<int>(threadIdx.x) - ch * width;
    for (int i = threadIdx.x; i < total; i += 4 * SG_THREADS) {
      float a[4], r[4];
      long long o[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = i + u * SG_THREADS < total;
        const long long off = in ? col_off[split * slice + cl] : -1;
        o[u] = off < 0 ? -1 : off + static_cast<long long>(oc0 + ch) * hw;
        r[u] = has_res && o[u] >= 0 ? __ldg(p.residual + o[u]) : 0.0f;
        a[u] = 0.0f;
        if (in) {
          const float* src = stg + cl * pitch + ch;
          for (int s = 0; s < p.splits; ++s) a[u] = fmaf(src[s * slice * pitch], p.weight[s], a[u]);
          a[u] = __fmaf_rn(a[u], acc_scale, p.bias != nullptr ? __ldg(p.bias + oc0 + ch) : 0.0f);
        }
        ch += step_ch;
        cl += step_cl;
        if (cl >= width) { cl -= width; ++ch; }
      }
      if (p.activation >= 0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = apply_act(a[u], p.activation);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) if (o[u] >= 0) p.out_f32[o[u]] = has_res ? a[u] + r[u] : a[u];
    }
  }
  tcgen05_fence_before();
  __syncthreads();  // every warp has read the accumulators
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
}

template <int BK, int AP, int WP>
int prepare_split_kernel() {
  static PerDeviceOnce attr_once;
  return attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BK, AP, WP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_RING_LIMIT + 1024));
    MB_CUDA(cudaFuncSetAttribute(gemm_split_kernel<BK, AP, WP>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return MIMIR_B200_OK;
  });
}

// Stands for the kernel where the runtime is asked how many clusters fit: for kernels that allocate tensor memory it says one CTA per SM
// whatever they take of it.
__global__ void __launch_bounds__(SG_THREADS, 2) split_footprint_kernel() {}

// (any number of CTAs may share a tile; seven and nine fit the GPCs no better than eight and ten: 40 x 1024 x 32768 in ten 31.1 us, nine 33.4,
// eight 35.1, as more SMs have weights on the way)
constexpr int SG_SPLITS[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16};

// n[two][i]: clusters of SG_SPLITS[i] CTAs that run at the same time, one or two CTAs to an SM.  A cluster lives in one GPC, whose SM count is no
// multiple of it: of the 148 SMs clusters of four use 132, of eight 120, of sixteen 112 (128 CTAs in clusters of eight: 12.9 us, two
// rounds, where 64 in clusters of four take 8.0).
struct ClusterTable { int n[2][sizeof(SG_SPLITS) / sizeof(int)]; };
const ClusterTable* active_clusters() {
  static PerDeviceOnce once;
  static ClusterTable table[64];  // (PerDeviceOnce counts as many devices)
  ClusterTable& t = table[ctx().device];
  const int rc = once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(split_footprint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SG_RING_LIMIT + 4096));
    MB_CUDA(cudaFuncSetAttribute(split_footprint_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (int j = 0; j < static_cast<int>(sizeof(SG_SPLITS) / sizeof(int)); ++j)
      for (int w = 0; w < 2; ++w) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(SG_SPLITS[j] * 512));
        cfg.blockDim = dim3(SG_THREADS);
        cfg.dynamicSmemBytes = (w ? SG_RING_TWO : SG_RING_LIMIT) + 4096;  // (with the kernel's static part)
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(SG_SPLITS[j]);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        MB_CUDA(cudaOccupancyMaxActiveClusters(&n, split_footprint_kernel, &cfg));
        t.n[w][j] = n;
      }
    return MIMIR_B200_OK;
  });
  return rc == MIMIR_B200_OK ? &t : nullptr;
}

// Tile width and split count of one launch and its estimated time in SM cycles.
struct SplitPlan { int bn = 0, splits = 0; double cycles = 1e30; };

SplitPlan plan_split(const GemmArgs& g, int bk, int kblocks) {
  const int sms = ctx().sm_count;
  const int tiles_o = (g.n + SG_M - 1) / SG_M;
  const bool cm = g.conv_ks > 0 || g.out_nchw_hw > 0;
  auto mma = [](int n) { return n > 92 ? n * 0.5 : 46.0; };  // an instruction of 128 x n x 16
  SplitPlan best;
  const ClusterTable* clusters = active_clusters();
  if (clusters == nullptr) return best;
  static const int widths[] = {16, 32, 48, 64, 96, 128};
  for (int bn : widths) {
    if (bn > 16 && bn >= g.m + 32) break;
    const long long tiles = static_cast<long long>(tiles_o) * ((g.m + bn - 1) / bn);
    const int stage = (g.w_planes * SG_M + g.a_planes * bn) * bk * 2;
    for (int i = 0; i < static_cast<int>(sizeof(SG_SPLITS) / sizeof(int)); ++i) {
      const int splits = SG_SPLITS[i];
      if (splits > kblocks || splits > bn) break;
      const long long ctas = tiles * splits;
      // CTAs that share an SM overlap one's loads and stores with the other's MMAs: whole rounds of two per SM
      const bool two = ctas > sms && 2 * stage <= SG_RING_TWO && (bn + splits - 1) * (SG_M + 1) * 4 <= SG_RING_TWO;
      const int active = clusters->n[two ? 1 : 0][i];
      if (active <= 0) continue;
      const long long rounds = (tiles + active - 1) / active;
      const double busy = static_cast<double>(ctas < sms ? ctas : sms) / sms;
      const double load = stage / (SG_LOAD_MAX - (SG_LOAD_MAX - SG_LOAD_ALL) * busy);
      const double block = (bk / 16) * (mma(g.a_planes * bn) + (g.w_planes == 2 ? mma(bn) : 0.0));
      const double main = (two ? 2.0 : 1.0) * ((kblocks + splits - 1) / splits) * (block > load ? block : load) * (cm ? SG_CM_BLOCK : 1.0);
      const double tail = (cm ? SG_CM_FIXED : SG_FIXED) + bn * (cm ? SG_CM_TAIL_PER_COL : SG_TAIL_PER_COL) / splits + (splits > 1 ? SG_SPLIT + bn * SG_SPLIT_PER_COL : 0.0);
      const double t = static_cast<double>(rounds) * (main + (two ? SG_TWO_TAIL : 1.0) * tail);
      if (t < best.cycles) { best.bn = bn; best.splits = splits; best.cycles = t; }
    }
  }
  return best;
}

// The tensor core adds with truncation, so in ONE accumulator over all of K (gemm_sm100.cu: `products` instructions per 16 of K) the
// contribution of an early range shrinks a little with every instruction that comes after it, 3.1e-8 of its value (fitted: 3e-8 ... 3.2e-8
// at every K and product count), and half as much for those of its own range.  The ranges summed apart here do not lose that, and in
// one instruction per 16 of K less than they would have.  The weights put it back, and the result is then scaled as the unsplit
// kernel's is: a row gives the same answer in a small batch and in a large one.  Relative difference of the two, 40 x 1024 outputs,
// K = 32768, three MMAs per product: 1e-4 without the weights, 1e-5 with them.  What the weights put back is the mean loss, not what each
// sum lost; the fewer ranges, the more of that differs.  162 x 130 outputs in one / three / eight ranges: K = 4608 5.6e-6 / 2.4e-6 / 1.7e-6,
// K = 9216 1.1e-5 / 4.4e-6 / 3.0e-6, K = 32768 3.9e-5 / 1.5e-5 / 9.5e-6; one range is the nearest to the products in 64 bits (K = 9216:
// 5.5e-6 against 1.5e-5 in three).
void split_weights(SplitGemmParams& p, long long ksteps, int steps_per_block, int products) {
  auto at = [&](int s) {  // (zero-padded K adds exact zeros and loses nothing)
    const long long step = static_cast<long long>(p.kblocks) * s / p.splits * steps_per_block;
    return step < ksteps ? step : ksteps;
  };
  for (int s = 0; s < p.splits; ++s) {
    const double after = p.splits > 1 ? 3.1e-8 * products * static_cast<double>(ksteps - at(s + 1)) : 0.0;
    p.weight[s] = static_cast<float>(1.0 - after - 1.5e-8 * (products - 1) * static_cast<double>(at(s + 1) - at(s)));
  }
  if (p.splits == 1) {  // (a factor of the result: row-major tiles then leave tensor memory without another multiplication)
    p.acc_scale *= p.weight[0];
    p.weight[0] = 1.0f;
  }
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
  p.w_amax = g.w_amax;
  split_weights(p, conv ? static_cast<long long>(p.kblocks) * (BK / 16) : (g.k + 15) / 16, BK / 16, AP + WP - 1);
  p.f16 = plane_format() == PLANES_F16 ? 1 : 0;
  p.w_ready = g.w_ready ? 1 : 0;
  p.err_word = ctx().dev_error_word;
  p.stage_bytes = (WP * SG_M + AP * p.bn) * BK * 2;
  const int per_split = (p.kblocks + p.splits - 1) / p.splits;
  const long long ctas = static_cast<long long>(p.tiles_o) * ((g.m + p.bn - 1) / p.bn) * p.splits;
  const bool two = ctas > ctx().sm_count && 2 * p.stage_bytes <= SG_RING_TWO && (p.bn + p.splits - 1) * (SG_M + 1) * 4 <= SG_RING_TWO;
  p.stages = (two ? SG_RING_TWO : SG_RING_LIMIT) / p.stage_bytes;
  if (p.stages > SG_MAX_STAGES) p.stages = SG_MAX_STAGES;
  if (p.stages > per_split) p.stages = per_split;
  // the staging tile gets a place of its own where that leaves three stages (or all there are)
  const int staging = p.splits * ((p.bn + p.splits - 1) / p.splits) * (SG_M + 1) * 4, limit = two ? SG_RING_TWO : SG_RING_LIMIT;
  const int fit = (limit - staging) / p.stage_bytes;
  p.stg_off = 0;
  if (p.splits > 1 && (fit >= p.stages || fit >= 3)) {
    if (p.stages > fit) p.stages = fit;
    p.stg_off = p.stages * p.stage_bytes;
  }
  const int ring = p.stages * p.stage_bytes;
  const int smem = (p.stg_off > 0 ? ring + staging : ring > staging ? ring : staging) + 1024;
  MB_TRY((prepare_split_kernel<BK, AP, WP>()));
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
  if (g.a_group_rows > 0) return never;
  const int kblocks = g.conv_ks > 0 ? g.conv_ks * g.conv_ks * (g.conv_c / bk) : round_up(g.k, 64) / bk;
  const char* e = getenv("MIMIR_B200_GEMM_SPLIT");  // "0": never; "<bn>,<splits>": always, in that shape
  if (e && e[0] == '0' && e[1] == '\0') return never;
  int fb = 0, fs = 0;
  if (e && sscanf(e, "%d,%d", &fb, &fs) == 2) {
    *bn = fb; *splits = fs;
    return fb >= 16 && fb <= SG_MAX_BN && fb % 16 == 0 && fs >= 1 && fs <= SG_MAX_SPLITS && fs <= fb && fs <= kblocks ? 0.0 : never;
  }
  const SplitPlan plan = plan_split(g, bk, kblocks);
  *bn = plan.bn; *splits = plan.splits;
  return plan.cycles;
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
