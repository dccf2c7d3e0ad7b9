// skinny_cluster.cu — Linear for at most 16 rows and a weight matrix that fits the GPU's registers in one wave: what a decode step
// and a small encoder run by the dozen.  Same arithmetic as skinny.cu (exact fp32 FMA, LayerOps.hpp:81-110):
//
//   y[r, o] = act( sum_k n(x)[r, k] * W[o, k] + b[o] ) (+ residual[r, o]),   n = identity or a token-wise LayerNorm of x
//
// Such a layer reads 2 to 10 MB of weights: 1 to 2 us at the memory rate, but the streaming kernel and its finishing kernel took
// 6.5 + 3 us each, almost all of it latency.  Here
//   * a CTA takes 32 output features and a K range of at most 384, and holds its weights in registers: the loads are issued before
//     anything else and, under programmatic stream serialization, while the kernel that produces x still runs;
//   * the CTAs of a cluster hold the K ranges of one tile; their sums meet in the first CTA's shared memory, in K order
//     (deterministic), which applies bias, activation and residual: no scratch, no second kernel;
//   * a LayerNorm that feeds only this layer is applied while x is staged: every CTA takes the row statistics itself (16 rows of
//     768 values are 48 KB from L2), which saves a launch of 4 us.
#include "common.h"
#include "epilogue.cuh"
#include "launch.cuh"

namespace mb {
namespace {

constexpr int SC_THREADS = 256, SC_WARPS = 8;
constexpr int SC_WR = 4;                    // weight rows of a warp
constexpr int SC_ROWS = SC_WARPS * SC_WR;   // output features of a CTA
constexpr int SC_STEP = 128;                // k of a warp step: 32 lanes x 4

struct SkinnyClusterParams {
  const float* x; const float* w; const float* bias; const float* residual; float* y;
  const float* gamma; const float* beta;  // LayerNorm (ln != 0), either may be null
  float eps;
  int ln, m, k, n, kc, act, w_ready;
};

__device__ __forceinline__ float4 ld_weights(const float* p) {  // read once; volatile: stays ahead of the dependency wait
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}

template <int MT, int STEPS>
__global__ void __launch_bounds__(SC_THREADS, 2) skinny_cluster_kernel(const SkinnyClusterParams p) {
  constexpr int N = MT * SC_WR, PER = N / 32;
  constexpr int KC = STEPS * SC_STEP;
  extern __shared__ __align__(16) float sc_smem[];
  float* xs = sc_smem;                       // [MT][KC]
  float* part = sc_smem + MT * KC;           // rank 0: [cluster size][MT][SC_ROWS]
  __shared__ float mean_s[MT], rstd_s[MT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank, size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  const int tile = static_cast<int>(blockIdx.x / size);
  const int k0 = static_cast<int>(rank) * p.kc, klen = min(p.kc, p.k - k0);
  const int o0 = tile * SC_ROWS + warp * SC_WR;

  cluster_arrive();  // (waited for before the first write into another CTA)
  if (!p.w_ready) pdl_wait();
  float4 wv[STEPS][SC_WR];
#pragma unroll
  for (int s = 0; s < STEPS; ++s)
#pragma unroll
    for (int j = 0; j < SC_WR; ++j) {
      const int c = s * SC_STEP + lane * 4;
      wv[s][j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < klen && o0 + j < p.n) wv[s][j] = ld_weights(p.w + static_cast<long long>(o0 + j) * p.k + k0 + c);
    }
  pdl_launch_dependents();
  pdl_wait();

  if (p.ln) {
    // mean and variance of each row (LayerOps.hpp:264-319), two passes; rows of up to 1024 values stay in registers in between
    for (int r = warp; r < p.m; r += SC_WARPS) {
      const float* row = p.x + static_cast<long long>(r) * p.k;
      float s = 0.0f, q = 0.0f, mean;
      if (p.k <= 1024) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (lane + 32 * j) * 4 < p.k ? *reinterpret_cast<const float4*>(row + (lane + 32 * j) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
        mean = warp_total(s) / static_cast<float>(p.k);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if ((lane + 32 * j) * 4 < p.k) {
            const float a = v[j].x - mean, b = v[j].y - mean, e = v[j].z - mean, f = v[j].w - mean;
            q += (a * a + b * b) + (e * e + f * f);
          }
      } else {
        for (int c = lane * 4; c < p.k; c += 128) {
          const float4 v = *reinterpret_cast<const float4*>(row + c);
          s += (v.x + v.y) + (v.z + v.w);
        }
        mean = warp_total(s) / static_cast<float>(p.k);
        for (int c = lane * 4; c < p.k; c += 128) {
          const float4 v = *reinterpret_cast<const float4*>(row + c);
          const float a = v.x - mean, b = v.y - mean, e = v.z - mean, f = v.w - mean;
          q += (a * a + b * b) + (e * e + f * f);
        }
      }
      q = warp_total(q);
      if (lane == 0) {
        mean_s[r] = mean;
        rstd_s[r] = 1.0f / sqrtf(q / static_cast<float>(p.k) + p.eps);
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < MT * (KC / 4); i += SC_THREADS) {
    const int r = i / (KC / 4), c = (i - r * (KC / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < p.m && c < klen) {
      v = *reinterpret_cast<const float4*>(p.x + static_cast<long long>(r) * p.k + k0 + c);
      if (p.ln) {
        const float mu = mean_s[r], rs = rstd_s[r];
        float4 g = make_float4(1.f, 1.f, 1.f, 1.f), b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.gamma) g = __ldg(reinterpret_cast<const float4*>(p.gamma + k0 + c));
        if (p.beta) b = __ldg(reinterpret_cast<const float4*>(p.beta + k0 + c));
        v.x = (v.x - mu) * rs * g.x + b.x; v.y = (v.y - mu) * rs * g.y + b.y;
        v.z = (v.z - mu) * rs * g.z + b.z; v.w = (v.w - mu) * rs * g.w + b.w;
      }
    }
    *reinterpret_cast<float4*>(xs + r * KC + c) = v;
  }
  __syncthreads();

  float acc[N];
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0.0f;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
#pragma unroll
    for (int r = 0; r < MT; ++r) {
      const float4 xv = *reinterpret_cast<const float4*>(xs + r * KC + s * SC_STEP + lane * 4);
#pragma unroll
      for (int j = 0; j < SC_WR; ++j) {
        float a = acc[j * MT + r];
        a = fmaf(wv[s][j].x, xv.x, a);
        a = fmaf(wv[s][j].y, xv.y, a);
        a = fmaf(wv[s][j].z, xv.z, a);
        a = fmaf(wv[s][j].w, xv.w, a);
        acc[j * MT + r] = a;
      }
    }
  }
  // recursive halving (skinny.cu): a lane ends with the sums of indices lane * PER + t, index = row-of-W * MT + row-of-x
#pragma unroll
  for (int half = N / 2, mask = 16; mask >= 1; half >>= 1, mask >>= 1) {
    const bool upper = (lane & mask) != 0;
    if (half >= 1) {
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float send = upper ? acc[i] : acc[i + half];
        const float keep = upper ? acc[i + half] : acc[i];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
      }
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], mask);  // fewer values than lanes: the holders of one value add up
    }
  }
  cluster_wait();  // every CTA of the cluster runs: rank 0's shared memory may be written
  uint32_t base;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(base) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(part))));
  base += static_cast<uint32_t>(rank * (MT * SC_ROWS) * 4);
  auto put = [&](int idx, float v) {
    const int j = idx / MT, r = idx - j * MT;
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(base + static_cast<uint32_t>((r * SC_ROWS + warp * SC_WR + j) * 4)), "f"(v) : "memory");
  };
  if (PER >= 1) {
#pragma unroll
    for (int t = 0; t < (PER >= 1 ? PER : 1); ++t) put(lane * PER + t, acc[t]);
  } else if ((lane & 1) == 0) {
    put(lane >> 1, acc[0]);  // N = 16: two lanes hold each value
  }
  cluster_arrive();
  cluster_wait();
  if (rank != 0) return;
  for (int i = threadIdx.x; i < p.m * SC_ROWS; i += SC_THREADS) {
    const int r = i / SC_ROWS, o = tile * SC_ROWS + (i & (SC_ROWS - 1));
    if (o >= p.n) continue;
    float v = part[i];
    for (uint32_t s = 1; s < size; ++s) v += part[s * (MT * SC_ROWS) + i];
    if (p.bias) v += __ldg(p.bias + o);
    v = sk_act(v, p.act);
    const long long at = static_cast<long long>(r) * p.n + o;
    if (p.residual) v += p.residual[at];
    p.y[at] = v;
  }
}

struct ClusterShape { int steps = 0, splits = 0; };
// The fewest k steps per CTA with which the K ranges fit a cluster and all CTAs are resident at once (two per SM).
ClusterShape cluster_shape(int k, int n) {
  const int tiles = (n + SC_ROWS - 1) / SC_ROWS;
  for (int steps = 1; steps <= 3; ++steps) {
    const int splits = (k + steps * SC_STEP - 1) / (steps * SC_STEP);
    if (splits <= 8 && static_cast<long long>(tiles) * splits <= 2 * ctx().sm_count) return {steps, splits};
  }
  return {};
}

template <int MT>
int launch_mt(const SkinnyClusterParams& p, const ClusterShape& c, cudaStream_t st) {
  const dim3 grid(static_cast<unsigned>((p.n + SC_ROWS - 1) / SC_ROWS * c.splits)), block(SC_THREADS);
  const size_t smem = (static_cast<size_t>(MT) * p.kc + static_cast<size_t>(c.splits) * MT * SC_ROWS) * sizeof(float);
  if (c.steps == 1) return launch_pdl(skinny_cluster_kernel<MT, 1>, grid, block, smem, st, c.splits, p);
  if (c.steps == 2) return launch_pdl(skinny_cluster_kernel<MT, 2>, grid, block, smem, st, c.splits, p);
  return launch_pdl(skinny_cluster_kernel<MT, 3>, grid, block, smem, st, c.splits, p);
}

}  // namespace

bool skinny_cluster_supported(int m, int k, int n) {
  return m >= 1 && m <= 16 && k % 4 == 0 && cluster_shape(k, n).steps > 0;
}

int launch_skinny_cluster(const SkinnyClusterArgs& a, cudaStream_t st) {
  if (!skinny_cluster_supported(a.m, a.k, a.n)) return fail(MIMIR_B200_E_INVALID, "skinny linear: not a shape of the cluster kernel");
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w) | reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta);
  if (bits & 15) return fail(MIMIR_B200_E_INVALID, "skinny linear: operands not 16-byte aligned");
  const ClusterShape c = cluster_shape(a.k, a.n);
  SkinnyClusterParams p;
  p.x = a.x; p.w = a.w; p.bias = a.bias; p.residual = a.residual; p.y = a.y;
  p.gamma = a.gamma; p.beta = a.beta; p.eps = a.eps; p.ln = a.ln ? 1 : 0;
  p.m = a.m; p.k = a.k; p.n = a.n; p.kc = c.steps * SC_STEP; p.act = a.activation; p.w_ready = a.w_ready ? 1 : 0;
  if (a.m <= 4) MB_TRY(launch_mt<4>(p, c, st));
  else if (a.m <= 8) MB_TRY(launch_mt<8>(p, c, st));
  else MB_TRY(launch_mt<16>(p, c, st));
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb
