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
constexpr int SC_STEP = 128;                // k of a warp step: 32 lanes x 4

struct SkinnyClusterParams {
  const float* x; const void* w; const float* bias; const float* residual; float* y;
  const float* gamma; const float* beta;  // LayerNorm (ln != 0), either may be null
  float eps;
  int ln, m, k, n, kc, act, w_ready;
};

// Four consecutive weights of a row, as fp32 or as bfloat16 (where every weight is one exactly: half the bytes, the same values).
// Read once; volatile: the loads stay ahead of the dependency wait.
template <int BF16> struct Quad;
template <> struct Quad<0> {
  float4 v;
  __device__ void zero() { v = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ void load(const void* w, long long i) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(static_cast<const float*>(w) + i));
  }
  __device__ float4 get() const { return v; }
};
template <> struct Quad<1> {
  uint2 v;
  __device__ void zero() { v = make_uint2(0u, 0u); }
  __device__ void load(const void* w, long long i) {
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(static_cast<const uint16_t*>(w) + i));
  }
  __device__ float4 get() const {
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
  }
};
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

// MT rows of x, WR weight rows of a warp, STEPS 128-wide k steps of a CTA.
template <int MT, int WR, int STEPS, int BF16>
__global__ void __launch_bounds__(SC_THREADS, 2) skinny_cluster_kernel(const SkinnyClusterParams p) {
  constexpr int SC_WR = WR, SC_ROWS = SC_WARPS * WR;  // output features of a CTA
  constexpr int N = MT * WR;
  constexpr int R = N % 32 == 0 ? 5 : N % 16 == 0 ? 4 : N % 8 == 0 ? 3 : 2, PER = N >> R;  // halving rounds of the exchange, values left
  constexpr int KC = STEPS * SC_STEP;
  extern __shared__ __align__(16) float sc_smem[];
  float* xs = sc_smem;                       // [MT][KC]
  float* gb = sc_smem + MT * KC;             // [2][KC]: the LayerNorm's gamma and beta
  float* part = gb + 2 * KC;                 // rank 0: [cluster size][MT][SC_ROWS]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank, size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  const int tile = static_cast<int>(blockIdx.x / size);
  const int k0 = static_cast<int>(rank) * p.kc, klen = min(p.kc, p.k - k0);
  const int o0 = tile * SC_ROWS + warp * SC_WR;

  cluster_arrive();  // (waited for before the first write into another CTA)
  if (!p.w_ready) pdl_wait();
  Quad<BF16> wv[STEPS][SC_WR];
#pragma unroll
  for (int s = 0; s < STEPS; ++s)
#pragma unroll
    for (int j = 0; j < SC_WR; ++j) {
      const int c = s * SC_STEP + lane * 4;
      wv[s][j].zero();
      if (c < klen && o0 + j < p.n) wv[s][j].load(p.w, static_cast<long long>(o0 + j) * p.k + k0 + c);
    }
  stage_affine(p, gb, k0, klen, KC);
  pdl_launch_dependents();
  pdl_wait();

  stage_rows<MT>(p, xs, gb, k0, klen, KC, warp, lane);
  __syncthreads();

  float acc[N];
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0.0f;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    float4 w[SC_WR];
#pragma unroll
    for (int j = 0; j < SC_WR; ++j) w[j] = wv[s][j].get();
#pragma unroll
    for (int r = 0; r < MT; ++r) {
      const float4 xv = *reinterpret_cast<const float4*>(xs + r * KC + s * SC_STEP + lane * 4);
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
  }
  // index = row-of-W * MT + row-of-x
  lane_exchange<N, R>(acc, lane);
  cluster_wait();  // every CTA of the cluster runs: rank 0's shared memory may be written
  uint32_t base;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(base) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(part))));
  base += static_cast<uint32_t>(rank * (MT * SC_ROWS) * 4);
  auto put = [&](int idx, float v) {
    const int j = idx / MT, r = idx - j * MT;
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(base + static_cast<uint32_t>((r * SC_ROWS + warp * SC_WR + j) * 4)), "f"(v) : "memory");
  };
  if ((lane & ((1 << (5 - R)) - 1)) == 0) {
#pragma unroll
    for (int t = 0; t < PER; ++t) put((lane >> (5 - R)) * PER + t, acc[t]);
  }
  cluster_arrive();
  cluster_wait();
  if (rank != 0) return;
  for (int i = threadIdx.x; i < p.m * SC_ROWS; i += SC_THREADS) {
    const int r = i / SC_ROWS, o = tile * SC_ROWS + i % SC_ROWS;
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

// The same for weight matrices of any number of rows (a decoder's vocabulary projection): one CTA per SM keeps all of x in shared
// memory and every warp walks groups of four weight rows on its own, with RING k steps of weights in flight in registers across
// group borders.  No partial sums leave the warp.  16 samples x 768 -> 32000 (bfloat16 copies): the streaming kernel with its
// staged x slices and finishing kernel took 54 us; the x reads from shared memory alone are 11 us, the weights 7.5 us.
template <int MT, int BF16>
__global__ void __launch_bounds__(SC_THREADS, 1) skinny_rows_kernel(const SkinnyClusterParams p) {
  constexpr int WR = 4, N = MT * WR, RING = BF16 ? 6 : 3;
  constexpr int R = N % 32 == 0 ? 5 : 4, PER = N >> R;
  extern __shared__ __align__(16) float sc_smem[];
  const int kp = p.kc, nsteps = kp / SC_STEP;
  float* xs = sc_smem;
  float* gb = sc_smem + MT * kp;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (p.n + WR - 1) / WR, stride = static_cast<int>(gridDim.x) * SC_WARPS;
  const int first = static_cast<int>(blockIdx.x) * SC_WARPS + warp;
  const int mine = first < groups ? (groups - first + stride - 1) / stride : 0;
  Quad<BF16> wv[RING][WR];
  int f_o = first * WR, f_ks = 0;  // the next step to fetch
  auto fetch = [&](Quad<BF16> (&q)[WR]) {
    const int c = f_ks * SC_STEP + lane * 4;
#pragma unroll
    for (int j = 0; j < WR; ++j) {
      q[j].zero();
      if (c < p.k && f_o + j < p.n) q[j].load(p.w, static_cast<long long>(f_o + j) * p.k + c);
    }
    if (++f_ks == nsteps) { f_ks = 0; f_o += stride * WR; }
  };
  if (!p.w_ready) pdl_wait();
#pragma unroll
  for (int u = 0; u < RING; ++u) fetch(wv[u]);
  stage_affine(p, gb, 0, p.k, kp);
  pdl_launch_dependents();
  pdl_wait();
  stage_rows<MT>(p, xs, gb, 0, p.k, kp, warp, lane);
  __syncthreads();

  float acc[N];
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0.0f;
  int o = first * WR, ks = 0;
  const int total = mine * nsteps;
  for (int g = 0; g < total; g += RING) {
#pragma unroll
    for (int u = 0; u < RING; ++u) {
      if (g + u >= total) break;
      float4 w[WR];
#pragma unroll
      for (int j = 0; j < WR; ++j) w[j] = wv[u][j].get();
      fetch(wv[u]);
#pragma unroll
      for (int r = 0; r < MT; ++r) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + r * kp + ks * SC_STEP + lane * 4);
#pragma unroll
        for (int j = 0; j < WR; ++j) {
          float a = acc[j * MT + r];
          a = fmaf(w[j].x, xv.x, a);
          a = fmaf(w[j].y, xv.y, a);
          a = fmaf(w[j].z, xv.z, a);
          a = fmaf(w[j].w, xv.w, a);
          acc[j * MT + r] = a;
        }
      }
      if (++ks == nsteps) {
        ks = 0;
        lane_exchange<N, R>(acc, lane);
        if ((lane & ((1 << (5 - R)) - 1)) == 0) {
#pragma unroll
          for (int t = 0; t < PER; ++t) {
            const int idx = (lane >> (5 - R)) * PER + t, j = idx / MT, r = idx - j * MT;
            if (r < p.m && o + j < p.n) {
              float v = acc[t];
              if (p.bias) v += __ldg(p.bias + o + j);
              v = sk_act(v, p.act);
              const long long at = static_cast<long long>(r) * p.n + o + j;
              if (p.residual) v += p.residual[at];
              p.y[at] = v;
            }
          }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = 0.0f;
        o += stride * WR;
      }
    }
  }
}

struct ClusterShape { int wr = 0, steps = 0, splits = 0; };
// Rows per warp, k steps per CTA and K ranges of a launch.  The time of such a launch after its input is ready is the x reads
// from shared memory of the busiest SM (8 warps x steps x MT x 4 cycles; the FMAs are no more) plus a latency chain, so: few CTAs per SM (one where possible - the previous kernel's CTAs still hold registers
// when this one's should start loading), little work in each, a cluster only where K needs it.
ClusterShape cluster_shape(int m, int k, int n, bool bf16) {
  const int mt = m <= 4 ? 4 : m <= 8 ? 8 : 16, sms = ctx().sm_count;
  ClusterShape best;
  long long best_cost = 0;
  for (int wr = 2; wr <= 4; ++wr)
    for (int steps = 2; steps <= 6; ++steps) {
      if (steps == 5 || (!bf16 && (steps > 3 || wr == 3))) continue;
      const int splits = (k + steps * SC_STEP - 1) / (steps * SC_STEP);
      const long long ctas = static_cast<long long>((n + SC_WARPS * wr - 1) / (SC_WARPS * wr)) * splits;
      if (splits > 8 || ctas > 2 * sms) continue;
      const long long cost = (ctas + sms - 1) / sms * (steps * mt * 32 + 600) + (splits > 1 ? 300 + 60 * splits : 0);
      if (best.wr == 0 || cost < best_cost) { best = {wr, steps, splits}; best_cost = cost; }
    }
  return best;
}

template <int MT, int WR, int STEPS, int BF16>
int launch_shape(const SkinnyClusterParams& p, const ClusterShape& c, cudaStream_t st) {
  constexpr int ROWS = SC_WARPS * WR;
  const size_t smem = (static_cast<size_t>(MT + 2) * p.kc + static_cast<size_t>(c.splits) * MT * ROWS) * sizeof(float);
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(skinny_cluster_kernel<MT, WR, STEPS, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 ((MT + 2) * STEPS * SC_STEP + 8 * MT * ROWS) * static_cast<int>(sizeof(float))));
    return MIMIR_B200_OK;
  }));
  return launch_pdl(skinny_cluster_kernel<MT, WR, STEPS, BF16>, dim3(static_cast<unsigned>((p.n + ROWS - 1) / ROWS * c.splits)), dim3(SC_THREADS), smem, st,
                    c.splits, p);
}
template <int MT, int WR>
int launch_rows(const SkinnyClusterParams& p, const ClusterShape& c, bool bf16, cudaStream_t st) {
  if (bf16) return c.steps == 2 ? launch_shape<MT, WR, 2, 1>(p, c, st) : c.steps == 3 ? launch_shape<MT, WR, 3, 1>(p, c, st) : c.steps == 4 ? launch_shape<MT, WR, 4, 1>(p, c, st) : launch_shape<MT, WR, 6, 1>(p, c, st);
  return c.steps == 2 ? launch_shape<MT, WR, 2, 0>(p, c, st) : launch_shape<MT, WR, 3, 0>(p, c, st);
}
template <int MT>
int launch_mt(const SkinnyClusterParams& p, const ClusterShape& c, bool bf16, cudaStream_t st) {
  if (c.wr == 2) return launch_rows<MT, 2>(p, c, bf16, st);
  if (c.wr == 3) return launch_rows<MT, 3>(p, c, true, st);
  return launch_rows<MT, 4>(p, c, bf16, st);
}

constexpr size_t ROWS_SMEM = size_t(200) << 10;

template <int MT>
int launch_rows_kernel(SkinnyClusterParams p, bool bf16, cudaStream_t st) {
  p.kc = round_up(p.k, SC_STEP);
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(skinny_rows_kernel<MT, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ROWS_SMEM)));
    MB_CUDA(cudaFuncSetAttribute(skinny_rows_kernel<MT, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ROWS_SMEM)));
    return MIMIR_B200_OK;
  }));
  const int want = (p.n + 4 * SC_WARPS - 1) / (4 * SC_WARPS), sms = ctx().sm_count;
  return launch_pdl(bf16 ? skinny_rows_kernel<MT, 1> : skinny_rows_kernel<MT, 0>, dim3(static_cast<unsigned>(want < sms ? want : sms)), dim3(SC_THREADS),
                    static_cast<size_t>(MT + 2) * p.kc * sizeof(float), st, 1, p);
}

// dst = the upper halves of src's bit patterns; *inexact becomes 1 when some lower half is not zero
__global__ void pack_bf16_kernel(const float* __restrict__ src, uint16_t* __restrict__ dst, size_t n, int* __restrict__ inexact) {
  bool bad = false;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t u = __float_as_uint(__ldg(src + i));
    dst[i] = static_cast<uint16_t>(u >> 16);
    bad = bad || (u & 0xffffu) != 0;
  }
  if (bad) *inexact = 1;
}

}  // namespace

bool skinny_cluster_supported(int m, int k, int n) {
  // (with bfloat16 weights every shape that fits as fp32 fits too: the choice of a fused LayerNorm does not depend on them)
  return m >= 1 && m <= 16 && k % 4 == 0 && cluster_shape(m, k, n, false).wr > 0;
}

bool skinny_rows_supported(int m, int k, int n) {
  const int mt = m <= 4 ? 4 : m <= 8 ? 8 : 16;
  return m >= 1 && m <= 16 && k % 4 == 0 && n >= 2048 && static_cast<size_t>(mt + 2) * round_up(k, SC_STEP) * sizeof(float) <= ROWS_SMEM;
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
  const bool cluster = skinny_cluster_supported(a.m, a.k, a.n);
  if (!cluster && !skinny_rows_supported(a.m, a.k, a.n)) return fail(MIMIR_B200_E_INVALID, "skinny linear: not a shape of these kernels");
  const bool bf16 = a.w_bf16 != nullptr;
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(bf16 ? static_cast<const void*>(a.w_bf16) : a.w) |
                         reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta);
  if (bits & 15) return fail(MIMIR_B200_E_INVALID, "skinny linear: operands not 16-byte aligned");
  const ClusterShape c = cluster ? cluster_shape(a.m, a.k, a.n, bf16) : ClusterShape();
  SkinnyClusterParams p;
  p.x = a.x; p.w = bf16 ? static_cast<const void*>(a.w_bf16) : a.w; p.bias = a.bias; p.residual = a.residual; p.y = a.y;
  p.gamma = a.gamma; p.beta = a.beta; p.eps = a.eps; p.ln = a.ln ? 1 : 0;
  p.m = a.m; p.k = a.k; p.n = a.n; p.kc = c.steps * SC_STEP; p.act = a.activation; p.w_ready = a.w_ready ? 1 : 0;
  if (!cluster) MB_TRY(a.m <= 4 ? launch_rows_kernel<4>(p, bf16, st) : a.m <= 8 ? launch_rows_kernel<8>(p, bf16, st) : launch_rows_kernel<16>(p, bf16, st));
  else if (a.m <= 4) MB_TRY(launch_mt<4>(p, c, bf16, st));
  else if (a.m <= 8) MB_TRY(launch_mt<8>(p, c, bf16, st));
  else MB_TRY(launch_mt<16>(p, c, bf16, st));
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb
