// skinny_cluster.cu — Linear for at most 16 rows and a weight matrix that fits the GPU's registers in one wave: what a decode step
// and a small encoder run by the dozen.  Same arithmetic as skinny.cu (exact fp32 FMA, LayerOps.hpp:81-110):
//
//   y[r, o] = act( sum_k n(x)[r, k] * W[o, k] + b[o] ) (+ residual[r, o]),   n = identity or a token-wise LayerNorm of x
//
// Such a layer reads 2 to 10 MB of weights: 1 to 2 us at the memory rate, but the streaming kernel and its finishing kernel took
// 6.5 + 3 us each, almost all of it latency.  Here
//   * a CTA takes tiles of 32 output features and a K range; every warp streams its four weight rows through a ring of its own in
//     shared memory (a lane reads only what it copied itself: no barriers).  The copies start before anything else and, under
//     programmatic stream serialization, while the kernel that produces x still runs;
//   * where one K range per tile would leave SMs idle, the CTAs of a cluster take the ranges; their sums meet in the first CTA's
//     shared memory, in K order (deterministic), which applies bias, activation and residual: no scratch, no second kernel;
//   * with many tiles (a vocabulary projection) one CTA per SM keeps its x in shared memory and walks its tiles;
//   * a LayerNorm that feeds only this layer is applied while x is staged: every CTA takes the row statistics itself (16 rows of
//     768 values are 48 KB from L2), which saves a launch of 4 us;
//   * (weights that are bfloat16 values take skinny_mma.cu, with 16-bit copies of them: launch_pack_bf16);
//   * the step loop is rolled and small.  With weights held in registers and every step unrolled, instruction fetch was the top
//     stall (no_instruction 1.7 per issue on the vocabulary projection, 38 us).
#include "common.h"
#include "epilogue.cuh"
#include "launch.cuh"

namespace mb {
namespace {

constexpr int SC_THREADS = 256, SC_WARPS = 8;
constexpr int SC_WR = 4;                    // weight rows of a warp
constexpr int SC_ROWS = SC_WARPS * SC_WR;   // output features of a tile
constexpr int SC_STEP = 128;                // k of a warp step: 32 lanes x 4

struct SkinnyClusterParams {
  const float* x; const float* w; const float* bias; const float* residual; float* y;
  const float* gamma; const float* beta;  // LayerNorm (ln != 0), either may be null
  float eps;
  int ln, m, k, n, kc, act, w_ready;
};

// Four consecutive weights of a row.
__device__ __forceinline__ void copy_quad(uint32_t dst, const float* w, long long i, bool valid) {
  const float* src = w + (valid ? i : 0);
  const int n = valid ? 16 : 0;  // source size 0: zero-fill
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

// gamma and beta of the k range into shared memory (weights: ahead of the dependency wait)
__device__ __forceinline__ void stage_affine(const SkinnyClusterParams& p, float* gb, int k0, int klen, int kc) {
  if (!p.ln) return;
  for (int c = threadIdx.x; c < klen; c += SC_THREADS) {
    gb[c] = p.gamma ? __ldg(p.gamma + k0 + c) : 1.0f;
    gb[kc + c] = p.beta ? __ldg(p.beta + k0 + c) : 0.0f;
  }
}

// xs[MT][kc] = (normalised) x[.., k0 .. k0 + klen), zero past m and klen.  A warp takes whole rows and has all its loads in flight
// before it uses the first: with one load per loop iteration this took 4 us of the 9 that such a launch lasted.
template <int MT>
__device__ __forceinline__ void stage_rows(const SkinnyClusterParams& p, float* xs, const float* gb, int k0, int klen, int kc, int warp, int lane) {
  constexpr int ROWS = MT > SC_WARPS ? MT / SC_WARPS : 1;  // rows of a warp
  if (p.ln && p.k <= 1024) {
    if (MT < SC_WARPS && warp >= MT) { __syncthreads(); return; }
    // mean and variance of each row (LayerOps.hpp:264-319) from registers; the k range leaves them normalised
    float4 v[ROWS][8];
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = warp + i * SC_WARPS, c = (lane + 32 * j) * 4;
        v[i][j] = (r < p.m && c < p.k) ? *reinterpret_cast<const float4*>(p.x + static_cast<long long>(r) * p.k + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    __syncthreads();  // gamma and beta are in shared memory
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int r = warp + i * SC_WARPS;
      float s = 0.0f, q = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) s += (v[i][j].x + v[i][j].y) + (v[i][j].z + v[i][j].w);
      const float mean = warp_total(s) / static_cast<float>(p.k);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if ((lane + 32 * j) * 4 < p.k) {
          const float a = v[i][j].x - mean, b = v[i][j].y - mean, e = v[i][j].z - mean, f = v[i][j].w - mean;
          q += (a * a + b * b) + (e * e + f * f);
        }
      const float rstd = 1.0f / sqrtf(warp_total(q) / static_cast<float>(p.k) + p.eps);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = (lane + 32 * j) * 4 - k0;
        if (c < 0 || c >= kc) continue;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < klen && r < p.m) {
          const float4 g = *reinterpret_cast<const float4*>(gb + c), b = *reinterpret_cast<const float4*>(gb + kc + c);
          o = make_float4((v[i][j].x - mean) * rstd * g.x + b.x, (v[i][j].y - mean) * rstd * g.y + b.y, (v[i][j].z - mean) * rstd * g.z + b.z,
                          (v[i][j].w - mean) * rstd * g.w + b.w);
        }
        *reinterpret_cast<float4*>(xs + r * kc + c) = o;
      }
      for (int c = p.k - k0 + lane * 4; c < kc; c += 128) *reinterpret_cast<float4*>(xs + r * kc + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  if (p.ln) {  // long rows: statistics first, then the common copy below applies them
    for (int r = warp; r < p.m; r += SC_WARPS) {
      const float* row = p.x + static_cast<long long>(r) * p.k;
      float s = 0.0f, q = 0.0f;
#pragma unroll 8
      for (int c = lane * 4; c < p.k; c += 128) {
        const float4 v = *reinterpret_cast<const float4*>(row + c);
        s += (v.x + v.y) + (v.z + v.w);
      }
      const float mean = warp_total(s) / static_cast<float>(p.k);
#pragma unroll 8
      for (int c = lane * 4; c < p.k; c += 128) {
        const float4 v = *reinterpret_cast<const float4*>(row + c);
        const float a = v.x - mean, b = v.y - mean, e = v.z - mean, f = v.w - mean;
        q += (a * a + b * b) + (e * e + f * f);
      }
      const float rstd = 1.0f / sqrtf(warp_total(q) / static_cast<float>(p.k) + p.eps);
      for (int c = lane * 4; c < kc; c += 128) {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < klen) {
          const float4 v = *reinterpret_cast<const float4*>(row + k0 + c);
          o = make_float4((v.x - mean) * rstd, (v.y - mean) * rstd, (v.z - mean) * rstd, (v.w - mean) * rstd);
        }
        *reinterpret_cast<float4*>(xs + r * kc + c) = o;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < MT * klen; i += SC_THREADS) {
      const int r = i / klen, c = i - r * klen;
      xs[r * kc + c] = r < p.m ? xs[r * kc + c] * gb[c] + gb[kc + c] : 0.0f;
    }
    for (int i = threadIdx.x; i < (MT - p.m) * kc; i += SC_THREADS) xs[p.m * kc + i] = 0.0f;
    return;
  }
  // batches of eight loads per thread
  const int total = MT * (kc / 4);
  for (int i0 = threadIdx.x; i0 < total; i0 += 8 * SC_THREADS) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u * SC_THREADS, r = i / (kc / 4), c = (i - r * (kc / 4)) * 4;
      v[u] = (i < total && r < p.m && c < klen) ? *reinterpret_cast<const float4*>(p.x + static_cast<long long>(r) * p.k + k0 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (i0 + u * SC_THREADS < total) *reinterpret_cast<float4*>(xs + (i0 + u * SC_THREADS) * 4) = v[u];
  }
}

__device__ __forceinline__ void finish(const SkinnyClusterParams& p, int r, int o, float v) {
  if (p.bias) v += __ldg(p.bias + o);
  v = sk_act(v, p.act);
  const long long at = static_cast<long long>(r) * p.n + o;
  if (p.residual) v += p.residual[at];
  p.y[at] = v;
}

// Sums over the warp's lanes of N values each: R rounds of recursive halving (skinny.cu), then the lanes that hold the same values
// add them up.  A lane ends with the sums of indices (lane >> (5 - R)) * (N >> R) + t.
template <int N, int R>
__device__ __forceinline__ void lane_exchange(float (&acc)[N], int lane) {
  constexpr int PER = N >> R;
#pragma unroll
  for (int round = 0; round < 5; ++round) {
    const int mask = 16 >> round, half = N >> (round + 1);
    if (round < R) {
      const bool upper = (lane & mask) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float send = upper ? acc[i] : acc[i + half];
        const float keep = upper ? acc[i + half] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
      }
    } else {
#pragma unroll
      for (int i = 0; i < PER; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], mask);
    }
  }
}

// MT rows of x.  grid = tiles * cluster size, or (cluster size 1) any number of CTAs that walk the tiles.
template <int MT>
__global__ void __launch_bounds__(SC_THREADS, 2) skinny_cluster_kernel(const SkinnyClusterParams p) {
  constexpr int N = MT * SC_WR;
  constexpr int R = N % 32 == 0 ? 5 : 4, PER = N >> R;  // halving rounds of the exchange, values left
  constexpr int QB = 16;                                // bytes of a lane's four weights
  constexpr int STAGE = SC_WR * 32 * QB, STAGES = 6;
  extern __shared__ __align__(16) float sc_smem[];
  float* xs = sc_smem;                       // [MT][kc]
  float* gb = sc_smem + MT * p.kc;           // [2][kc]: the LayerNorm's gamma and beta
  float* part = gb + 2 * p.kc;               // rank 0: [cluster size][MT][SC_ROWS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank, size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  uint8_t* ring = reinterpret_cast<uint8_t*>(part + (size > 1 ? size * MT * SC_ROWS : 0)) + warp * (STAGES * STAGE) + lane * QB;
  const uint32_t ring_addr = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
  const int k0 = static_cast<int>(rank) * p.kc, klen = min(p.kc, p.k - k0), nsteps = (klen + SC_STEP - 1) / SC_STEP;
  const int tile0 = static_cast<int>(blockIdx.x / size), tile_step = static_cast<int>(gridDim.x / size);
  const int tiles = (p.n + SC_ROWS - 1) / SC_ROWS;
  const int total = ((tiles - tile0 + tile_step - 1) / tile_step) * nsteps;

  if (size > 1) cluster_arrive();  // (waited for before the first write into another CTA)
  if (!p.w_ready) pdl_wait();
  int f_o = tile0 * SC_ROWS + warp * SC_WR, f_ks = 0, f_slot = 0, f_left = total;  // the next step to fetch
  auto fetch = [&]() {
    if (f_left > 0) {
      const int c = f_ks * SC_STEP + lane * 4;
      const uint32_t dst = ring_addr + f_slot * STAGE;
      const long long at = static_cast<long long>(f_o) * p.k + k0 + c;
#pragma unroll
      for (int j = 0; j < SC_WR; ++j) copy_quad(dst + j * 32 * QB, p.w, at + static_cast<long long>(j) * p.k, c < klen && f_o + j < p.n);
      if (++f_ks == nsteps) { f_ks = 0; f_o += tile_step * SC_ROWS; }
      if (++f_slot == STAGES) f_slot = 0;
      --f_left;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // one group per step, empty past the end
  };
#pragma unroll 1
  for (int u = 0; u < STAGES - 1; ++u) fetch();
  stage_affine(p, gb, k0, klen, p.kc);
  pdl_launch_dependents();
  pdl_wait();
  stage_rows<MT>(p, xs, gb, k0, klen, p.kc, warp, lane);
  __syncthreads();

  float acc[N];
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0.0f;
  int o = tile0 * SC_ROWS + warp * SC_WR, ks = 0, slot = 0;
#pragma unroll 1
  for (int g = 0; g < total; ++g) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    float4 w[SC_WR];
#pragma unroll
    for (int j = 0; j < SC_WR; ++j) w[j] = *reinterpret_cast<const float4*>(ring + slot * STAGE + j * 32 * QB);
    fetch();  // (into the slot read one step ago)
    const float* xr = xs + ks * SC_STEP + lane * 4;
#pragma unroll
    for (int r = 0; r < MT; ++r) {
      const float4 xv = *reinterpret_cast<const float4*>(xr + r * p.kc);
#pragma unroll
      for (int j = 0; j < SC_WR; ++j) {
        float a = acc[j * MT + r];
        a = fmaf(w[j].x, xv.x, a);
        a = fmaf(w[j].y, xv.y, a);
        a = fmaf(w[j].z, xv.z, a);
        a = fmaf(w[j].w, xv.w, a);
        acc[j * MT + r] = a;
      }
    }
    if (++slot == STAGES) slot = 0;
    if (++ks < nsteps) continue;
    ks = 0;
    lane_exchange<N, R>(acc, lane);  // index = row-of-W * MT + row-of-x
    const bool writer = (lane & ((1 << (5 - R)) - 1)) == 0;
    if (size > 1) {
      cluster_wait();  // every CTA of the cluster runs: rank 0's shared memory may be written
      uint32_t base;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(base) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(part))));
      base += rank * (MT * SC_ROWS) * 4;
#pragma unroll
      for (int t = 0; t < PER; ++t) {
        const int idx = (lane >> (5 - R)) * PER + t, j = idx / MT, r = idx - j * MT;
        if (writer) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(base + static_cast<uint32_t>((r * SC_ROWS + warp * SC_WR + j) * 4)), "f"(acc[t]) : "memory");
      }
    } else {
#pragma unroll
      for (int t = 0; t < PER; ++t) {
        const int idx = (lane >> (5 - R)) * PER + t, j = idx / MT, r = idx - j * MT;
        if (writer && r < p.m && o + j < p.n) finish(p, r, o + j, acc[t]);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] = 0.0f;
    o += tile_step * SC_ROWS;
  }
  if (size == 1) return;
  cluster_arrive();
  cluster_wait();
  if (rank != 0) return;
  for (int i = threadIdx.x; i < p.m * SC_ROWS; i += SC_THREADS) {
    const int r = i / SC_ROWS, oo = tile0 * SC_ROWS + i % SC_ROWS;
    if (oo >= p.n) continue;
    float v = part[i];
    for (uint32_t s = 1; s < size; ++s) v += part[s * (MT * SC_ROWS) + i];
    finish(p, r, oo, v);
  }
}

constexpr size_t SC_SMEM_MAX = size_t(220) << 10;
constexpr int SC_MAX_K = 4096;

struct ClusterShape { int splits = 0, kc = 0, ctas = 0; size_t smem = 0; };
// K ranges and CTAs of a launch.  After its input is ready such a launch takes the x reads from shared memory of the busiest SM
// (8 warps x steps x MT x 4 cycles; the FMAs are no more) plus a latency chain: few CTAs per SM (one where possible - the
// previous kernel's CTAs still hold resources when this one's should start loading), little work in each, a cluster only where
// K ranges are needed to occupy the SMs.  Chosen for 16 rows whatever m is: a sample gives the same bits in every batch size.
ClusterShape cluster_shape(int k, int n) {
  constexpr int mt = 16;
  const int sms = ctx().sm_count, tiles = (n + SC_ROWS - 1) / SC_ROWS;
  const int all = (k + SC_STEP - 1) / SC_STEP;
  const size_t ring = static_cast<size_t>(SC_WARPS) * (6 * 16) * SC_WR * 32;
  ClusterShape best;
  long long best_cost = 0;
  for (int splits = 1; splits <= 8; ++splits) {
    const int steps = (all + splits - 1) / splits;
    if (splits > 1 && (steps * (splits - 1) >= all || static_cast<long long>(tiles) * splits > 2 * sms)) continue;
    const size_t smem = static_cast<size_t>(mt + 2) * steps * SC_STEP * 4 + (splits > 1 ? static_cast<size_t>(splits) * mt * SC_ROWS * 4 : 0) + ring;
    if (smem > SC_SMEM_MAX) continue;
    const long long waves = (static_cast<long long>(tiles) * splits + sms - 1) / sms;
    const long long cost = waves * (steps * mt * 32 + 600) + (splits > 1 ? 300 + 60 * splits : 0);
    if (best.splits == 0 || cost < best_cost) {
      best.splits = splits; best.kc = steps * SC_STEP; best.smem = smem;
      best.ctas = splits > 1 || tiles < sms ? tiles * splits : sms;
      best_cost = cost;
    }
  }
  return best;
}

template <int MT>
int launch_mt(const SkinnyClusterParams& p, const ClusterShape& c, cudaStream_t st) {
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(skinny_cluster_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SC_SMEM_MAX)));
    return MIMIR_B200_OK;
  }));
  return launch_pdl(skinny_cluster_kernel<MT>, dim3(static_cast<unsigned>(c.ctas)), dim3(SC_THREADS), c.smem, st, c.splits, p);
}

// dst = the upper halves of src's bit patterns; *inexact becomes 1 when some lower half is not zero or a value is not finite (cut
// into planes, x would meet an infinite weight with zeros)
__global__ void pack_bf16_kernel(const float* __restrict__ src, uint16_t* __restrict__ dst, size_t n, int* __restrict__ inexact) {
  bool bad = false;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t u = __float_as_uint(__ldg(src + i));
    dst[i] = static_cast<uint16_t>(u >> 16);
    bad = bad || (u & 0xffffu) != 0 || (u & 0x7f800000u) == 0x7f800000u;
  }
  if (bad) *inexact = 1;
}

}  // namespace

bool skinny_cluster_supported(int m, int k, int n) {
  return m >= 1 && m <= 16 && k % 4 == 0 && k <= SC_MAX_K && cluster_shape(k, n).splits > 0;
}

int launch_pack_bf16(const float* src, uint16_t* dst, size_t n, int* inexact, cudaStream_t st) {
  size_t blocks = (n + 1023) / 1024;
  if (blocks > static_cast<size_t>(ctx().sm_count) * 8) blocks = static_cast<size_t>(ctx().sm_count) * 8;
  pack_bf16_kernel<<<static_cast<unsigned>(blocks), 256, 0, st>>>(src, dst, n, inexact);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

int launch_skinny_cluster(const SkinnyClusterArgs& a, cudaStream_t st) {
  if (a.w_bf16 != nullptr) return launch_skinny_mma(a, st);
  if (!skinny_cluster_supported(a.m, a.k, a.n)) return fail(MIMIR_B200_E_INVALID, "skinny linear: not a shape of the cluster kernel");
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta);
  if (bits & 15) return fail(MIMIR_B200_E_INVALID, "skinny linear: operands not 16-byte aligned");
  const ClusterShape c = cluster_shape(a.k, a.n);
  SkinnyClusterParams p;
  p.x = a.x; p.w = a.w; p.bias = a.bias; p.residual = a.residual; p.y = a.y;
  p.gamma = a.gamma; p.beta = a.beta; p.eps = a.eps; p.ln = a.ln ? 1 : 0;
  p.m = a.m; p.k = a.k; p.n = a.n; p.kc = c.kc; p.act = a.activation; p.w_ready = a.w_ready ? 1 : 0;
  if (a.m <= 4) MB_TRY(launch_mt<4>(p, c, st));
  else if (a.m <= 8) MB_TRY(launch_mt<8>(p, c, st));
  else MB_TRY(launch_mt<16>(p, c, st));
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb
