// skinny_mma.cu — Linear for at most 16 rows whose weights are bfloat16 values (a decode step of a checkpoint rounded to bf16):
//
//   y[r, o] = act( sum_k n(x)[r, k] * W[o, k] + b[o] ) (+ residual[r, o]),   n = identity or a token-wise LayerNorm of x
//
// (LayerOps.hpp:81-110.)  Such a layer is 1 to 5 MB of weights, under a microsecond of memory traffic; what it costs is the chain
// from its input's arrival to its last store.  With fp32 FMAs out of shared memory (skinny_cluster.cu) that chain was 2.8 us for the LayerNorm
// and the staging of x and 3 to 4 us for the products, at 16 FMAs and a 128-bit shared read per four weights.  Here
//   * the products run on the warp-level tensor instruction (m16n8k16: 16 output features x 8 rows).  x is cut into THREE bfloat16
//     planes that hold it exactly (8 + 8 + 8 significant bits), each with accumulators of its own; a product of bfloat16 values is
//     exact, so what is rounded is what fp32 FMAs round too: the sums.  The instruction cuts sums off instead of rounding them, so the hi
//     plane's leave it after 16 of K and are added up in fp32 (left in the accumulator, the error was 1.2 times that of the FMAs);
//   * a CTA takes 16 output features and all of K (a cluster of up to four where K > 1024), its eight warps a range of K each.  A lane
//     loads the weights of its fragments (16 bytes a row) straight into registers, before the kernel ahead has finished; x likewise, once,
//     with no staging in between;
//   * the LayerNorm's statistics are the warps' means and squared deviations, merged after one exchange;
//   * with more tiles than CTAs that fit (a vocabulary projection), the planes of x stay in registers and a CTA walks its tiles, the
//     next tile's weights on the way.
// Within a step of 16 samples (12 layers of 768, vocabulary 32000), by CTA stamps from the input's arrival to the last store:
// 768 -> 2304 with LayerNorm 8.0 -> 5.0 us, 768 -> 768 5.4 -> 2.9, 768 -> 3072 with LayerNorm 7.3 -> 5.6, 3072 -> 768 8.5 -> 4.2.  What is left of a
// LayerNorm form: x 0.6, statistics and planes 2.3, products 1.5 (the instruction issues every 32 cycles), sums and store 0.6.  (The forms
// without one are half a microsecond shorter since a warp looks for infinities once.)
// Whole steps, FMAs / now: 16 samples, 12 layers of 768, 814 / 610 us; of 1024 with ffn 4096 892 / 793; 9 samples, six such layers, 326 / 261, of
// 896 with ffn 3584 (14 samples) 375 / 278.  From K = 769 to a CTA on, 9 to 16 rows take more registers than two CTAs to an SM leave
// (skinny_mma_kernel<4, 2, false>: 128, and 300 bytes of spills); the gain there is the smaller one.
#include <type_traits>

#include "common.h"
#include "epilogue.cuh"
#include "launch.cuh"

namespace mb {
namespace {

constexpr int SM_THREADS = 256, SM_WARPS = 8;
constexpr int SM_FEATURES = 16;     // output features of a tile
constexpr int SM_UNIT = 32;         // k of a unit: a lane holds eight consecutive weights of a row
constexpr int SM_MAX_UNITS = 4;     // units of a warp
constexpr int SM_MAX_CLUSTER = 4;
constexpr int SM_PITCH = 20;        // floats from row to row of a warp's sums: conflict-free writes

struct SkinnyMmaParams {
  const float* x; const uint16_t* w; const float* bias; const float* residual; float* y;
  const float* gamma; const float* beta;  // LayerNorm (ln != 0), either may be null
  float eps;
  int ln, m, k, n, act, w_ready;
};

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// x0, x1 as pairs of bfloat16: hi + mid + lo is x exactly (each cut off after eight significant bits); INF: infinities stay in hi, with
// nothing in the other planes (inf - inf there would make NaN of them).
template <bool INF>
__device__ __forceinline__ void planes3(float x0, float x1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
  hi = __byte_perm(u0, u1, 0x7632);
  float r0 = x0 - __uint_as_float(u0 & 0xffff0000u), r1 = x1 - __uint_as_float(u1 & 0xffff0000u);
  if (INF) {
    r0 = fabsf(x0) == INFINITY ? 0.0f : r0;
    r1 = fabsf(x1) == INFINITY ? 0.0f : r1;
  }
  const uint32_t v0 = __float_as_uint(r0), v1 = __float_as_uint(r1);
  mid = __byte_perm(v0, v1, 0x7632);
  lo = __byte_perm(__float_as_uint(r0 - __uint_as_float(v0 & 0xffff0000u)), __float_as_uint(r1 - __uint_as_float(v1 & 0xffff0000u)), 0x7632);
}
__device__ __forceinline__ float quad_total(float v) {  // over the four lanes of a row
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// U: units of a warp at most; NT: groups of eight rows; LOOP: a CTA walks tiles (cluster size 1).
template <int U, int NT, bool LOOP>
__global__ void __launch_bounds__(SM_THREADS, LOOP ? 1 : 2) skinny_mma_kernel(const SkinnyMmaParams p) {
  __shared__ float sums[LOOP ? 2 : 1][SM_WARPS][16 * SM_PITCH];
  __shared__ float gather[SM_MAX_CLUSTER][SM_THREADS];  // rank 0: the sums of every CTA of the cluster
  __shared__ float2 stats[SM_WARPS][16];                // a warp's mean and squared deviations of each row
  __shared__ __align__(16) float gb[2][SM_WARPS * U * SM_UNIT];  // gamma and beta of this CTA's K
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  uint32_t rank = 0, size = 1;
  if (!LOOP) {
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    if (size > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  const int units = (p.k + SM_UNIT - 1) / SM_UNIT;
  const int c0 = units * static_cast<int>(rank) / static_cast<int>(size), c1 = units * (static_cast<int>(rank) + 1) / static_cast<int>(size);
  const int u0 = c0 + (c1 - c0) * warp / SM_WARPS, nu = c0 + (c1 - c0) * (warp + 1) / SM_WARPS - u0;  // this warp's units
  const int kw = u0 * SM_UNIT + t * 8;                                                                // this lane's first k
  const int tiles = (p.n + SM_FEATURES - 1) / SM_FEATURES;
  int tile = LOOP ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x / size);

  auto load_w = [&](int tl, uint4 (&w)[U][2]) {
    const uint16_t* row = p.w + static_cast<long long>(tl * SM_FEATURES + g) * p.k + kw;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        w[u][h] = make_uint4(0u, 0u, 0u, 0u);
        if (u < nu && kw + u * SM_UNIT < p.k && tl < tiles && tl * SM_FEATURES + g + 8 * h < p.n)  // (k is a multiple of eight)
          w[u][h] = __ldg(reinterpret_cast<const uint4*>(row + static_cast<long long>(8 * h) * p.k + u * SM_UNIT));
      }
  };
  if (!p.w_ready) pdl_wait();
  uint4 w[U][2];
  load_w(tile, w);
  if (p.ln) {  // (weights too)
    const int n = min(c1 * SM_UNIT, p.k) - c0 * SM_UNIT;
    for (int i = tid; i < n; i += SM_THREADS) {
      gb[0][i] = p.gamma ? __ldg(p.gamma + c0 * SM_UNIT + i) : 1.0f;
      gb[1][i] = p.beta ? __ldg(p.beta + c0 * SM_UNIT + i) : 0.0f;
    }
  }
  const int fr = tid >> 4, ff = tid & 15;  // the row and the feature whose sums this thread finishes
  pdl_launch_dependents();
  pdl_wait();

  // x: NT rows of eight values a unit
  float4 v[U][NT][2];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const float* row = p.x + static_cast<long long>(g + 8 * j) * p.k + kw;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = u < nu && kw + u * SM_UNIT < p.k && g + 8 * j < p.m;
      v[u][j][0] = in ? *reinterpret_cast<const float4*>(row + u * SM_UNIT) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[u][j][1] = in ? *reinterpret_cast<const float4*>(row + u * SM_UNIT + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  if (p.ln) {
    // mean and variance of each row (LayerOps.hpp:264-319)
    const float inv_k = 1.0f / static_cast<float>(p.k);
    if (LOOP || size == 1) {
      const int kn = min(nu * SM_UNIT, p.k - u0 * SM_UNIT);  // (elements of a row in this warp; none: no weight below)
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        float s = 0.0f, q = 0.0f, e = 0.0f;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h) s += (v[u][j][h].x + v[u][j][h].y) + (v[u][j][h].z + v[u][j][h].w);
        const float inv_n = kn > 0 ? 1.0f / static_cast<float>(kn) : 0.0f;
        const float mean = quad_total(s) * inv_n;
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u < nu && kw + u * SM_UNIT < p.k)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const float a = v[u][j][h].x - mean, b = v[u][j][h].y - mean, c = v[u][j][h].z - mean, d = v[u][j][h].w - mean;
              q += (a * a + b * b) + (c * c + d * d);
              e += (a + b) + (c + d);  // what the mean missed
            }
        q = quad_total(q);
        e = quad_total(e) * inv_n;
        if (t == 0) stats[warp][g + 8 * j] = make_float2(mean + e, q);
      }
    } else {  // K over a cluster: every CTA reads its rows whole
      for (int r = warp; r < p.m; r += SM_WARPS) {
        const float* row = p.x + static_cast<long long>(r) * p.k;
        float s = 0.0f, q = 0.0f;
#pragma unroll 8
        for (int c = lane * 4; c < p.k; c += 128) {
          const float4 a = *reinterpret_cast<const float4*>(row + c);
          s += (a.x + a.y) + (a.z + a.w);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        const float mean = s * inv_k;
#pragma unroll 8
        for (int c = lane * 4; c < p.k; c += 128) {
          const float4 b = *reinterpret_cast<const float4*>(row + c);
          const float a0 = b.x - mean, a1 = b.y - mean, a2 = b.z - mean, a3 = b.w - mean;
          q += (a0 * a0 + a1 * a1) + (a2 * a2 + a3 * a3);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) q += __shfl_xor_sync(0xffffffffu, q, d);
        if (lane == 0) stats[0][r] = make_float2(mean, q);
      }
    }
    __syncthreads();
    float n_w[SM_WARPS];  // elements of a row in each warp
#pragma unroll
    for (int i = 0; i < SM_WARPS; ++i) {
      const int a = c0 + (c1 - c0) * i / SM_WARPS, b = c0 + (c1 - c0) * (i + 1) / SM_WARPS;
      n_w[i] = static_cast<float>(max(min(b * SM_UNIT, p.k) - a * SM_UNIT, 0));
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      float mean = 0.0f, q = 0.0f;
      if (LOOP || size == 1) {
        const float ref = stats[SM_WARPS - 1][g + 8 * j].x;  // (the last warp always has a unit)
        float2 s[SM_WARPS];
#pragma unroll
        for (int i = 0; i < SM_WARPS; ++i) {
          s[i] = stats[i][g + 8 * j];
          mean = fmaf(n_w[i], s[i].x - ref, mean);
        }
        mean = fmaf(mean, inv_k, ref);
#pragma unroll
        for (int i = 0; i < SM_WARPS; ++i) q += fmaf(n_w[i] * (s[i].x - mean), s[i].x - mean, s[i].y);
      } else if (g + 8 * j < p.m) {
        mean = stats[0][g + 8 * j].x;
        q = stats[0][g + 8 * j].y;
      }
      const float rstd = 1.0f / sqrtf(q * inv_k + p.eps);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!(u < nu && kw + u * SM_UNIT < p.k)) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = kw - c0 * SM_UNIT + u * SM_UNIT + 4 * h;
          const float4 ga = *reinterpret_cast<const float4*>(&gb[0][c]), be = *reinterpret_cast<const float4*>(&gb[1][c]);
          float4& a = v[u][j][h];
          a = make_float4((a.x - mean) * rstd * ga.x + be.x, (a.y - mean) * rstd * ga.y + be.y, (a.z - mean) * rstd * ga.z + be.z, (a.w - mean) * rstd * ga.w + be.w);
        }
      }
    }
  }
  // (rows past m hold what the LayerNorm makes of zeros: their products are never written)
  uint32_t hi[U][NT][4], mid[U][NT][4], lo[U][NT][4];
  auto cut = [&](auto inf) {
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          planes3<decltype(inf)::value>(v[u][j][h].x, v[u][j][h].y, hi[u][j][2 * h], mid[u][j][2 * h], lo[u][j][2 * h]);
          planes3<decltype(inf)::value>(v[u][j][h].z, v[u][j][h].w, hi[u][j][2 * h + 1], mid[u][j][2 * h + 1], lo[u][j][2 * h + 1]);
        }
  };
  // The warp looks once whether it has an infinity (in x, or where gamma or beta make one): a maximum per value in place of a comparison and
  // a selection at each of them (a step of 16 samples 624 -> 610 us).  NaN is in no maximum; its planes are NaN either way.
  float top = 0.0f;
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        top = fmaxf(fmaxf(fmaxf(top, fabsf(v[u][j][h].x)), fmaxf(fabsf(v[u][j][h].y), fabsf(v[u][j][h].z))), fabsf(v[u][j][h].w));
  if (__any_sync(0xffffffffu, top == INFINITY)) cut(std::true_type{}); else cut(std::false_type{});

  int buf = 0;
#pragma unroll 1
  do {
    const int o = tile * SM_FEATURES + ff;
    const bool mine = fr < p.m && o < p.n && fr < 8 * NT && (LOOP || rank == 0);
    const long long at = static_cast<long long>(fr) * p.n + o;
    float bias = 0.0f, res = 0.0f;  // asked for ahead of the products
    if (mine && p.bias != nullptr) bias = __ldg(p.bias + o);
    if (mine && p.residual != nullptr) res = p.residual[at];
    float acc[3][NT][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;  // (warp-uniform)
#pragma unroll
      for (int s = 0; s < 2; ++s) {  // 16 of K: any order of K will do that is the same on both sides
        const uint32_t a[4] = {s ? w[u][0].z : w[u][0].x, s ? w[u][1].z : w[u][1].x, s ? w[u][0].w : w[u][0].y, s ? w[u][1].w : w[u][1].y};
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // (the instruction cuts its sum off: added up here, rounded to nearest)
          mma_16816(d, a, hi[u][j][2 * s], hi[u][j][2 * s + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[0][j][e] += d[e];
          mma_16816(acc[1][j], a, mid[u][j][2 * s], mid[u][j][2 * s + 1]);
          mma_16816(acc[2][j], a, lo[u][j][2 * s], lo[u][j][2 * s + 1]);
        }
      }
    }
    if (LOOP) load_w(tile + static_cast<int>(gridDim.x), w);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)  // element e: feature g + 8 (e / 2), row 8 j + 2 t + (e & 1)
        sums[LOOP ? buf : 0][warp][(8 * j + 2 * t + (e & 1)) * SM_PITCH + g + 8 * (e >> 1)] = acc[0][j][e] + (acc[1][j][e] + acc[2][j][e]);
    __syncthreads();
    float y = 0.0f;
    if (fr < 8 * NT) {
#pragma unroll
      for (int i = 0; i < SM_WARPS; ++i) y += sums[LOOP ? buf : 0][i][fr * SM_PITCH + ff];  // in K order
    }
    if (!LOOP && size > 1) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA of the cluster runs
      uint32_t dst;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&gather[rank][tid]))));
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(y) : "memory");
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      y = gather[0][tid];
      for (uint32_t c = 1; c < size; ++c) y += gather[c][tid];
    }
    if (mine) {
      y = sk_act(y + bias, p.act);
      if (p.residual != nullptr) y += res;
      p.y[at] = y;
    }
    buf ^= 1;
    tile += static_cast<int>(gridDim.x);
  } while (LOOP && tile < tiles);
}

template <int U, int NT>
int launch_nt(const SkinnyMmaParams& p, int cluster, cudaStream_t st) {
  const int tiles = (p.n + SM_FEATURES - 1) / SM_FEATURES;
  // From two tiles to an SM on, x's planes are worth keeping.  A one-layer step of 16 samples with CTAs that walk tiles / a CTA to a tile:
  // 300 tiles 101.6 / 103.1 us, 500 tiles 111 / 119, 1000 tiles 144 / 159, 2000 tiles 180 / 219.
  if (cluster == 1 && tiles > 2 * ctx().sm_count)
    return launch_pdl(skinny_mma_kernel<U, NT, true>, dim3(static_cast<unsigned>(ctx().sm_count)), dim3(SM_THREADS), 0, st, 1, p);
  return launch_pdl(skinny_mma_kernel<U, NT, false>, dim3(static_cast<unsigned>(tiles * cluster)), dim3(SM_THREADS), 0, st, cluster, p);
}
template <int U>
int launch_u(const SkinnyMmaParams& p, int cluster, cudaStream_t st) {
  return p.m <= 8 ? launch_nt<U, 1>(p, cluster, st) : launch_nt<U, 2>(p, cluster, st);
}

}  // namespace

bool skinny_mma_supported(int m, int k, int n) {
  return m >= 1 && m <= 16 && n >= 1 && k >= 8 && k % 8 == 0 && k <= SM_MAX_CLUSTER * SM_WARPS * SM_MAX_UNITS * SM_UNIT;
}

int launch_skinny_mma(const SkinnyClusterArgs& a, cudaStream_t st) {
  if (!skinny_mma_supported(a.m, a.k, a.n) || a.w_bf16 == nullptr) return fail(MIMIR_B200_E_INVALID, "skinny linear: not a shape of the tensor-core kernel");
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w_bf16) | reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta);
  if (bits & 15) return fail(MIMIR_B200_E_INVALID, "skinny linear: operands not 16-byte aligned");
  SkinnyMmaParams p;
  p.x = a.x; p.w = a.w_bf16; p.bias = a.bias; p.residual = a.residual; p.y = a.y; p.gamma = a.gamma; p.beta = a.beta; p.eps = a.eps; p.ln = a.ln ? 1 : 0;
  p.m = a.m; p.k = a.k; p.n = a.n; p.act = a.activation; p.w_ready = a.w_ready ? 1 : 0;
  // as few CTAs to a tile as the warps' registers allow: the same for every m, so that a sample gives the same bits in every batch size
  const int units = (a.k + SM_UNIT - 1) / SM_UNIT;
  int cluster = 1;
  while ((units + cluster - 1) / cluster > SM_WARPS * SM_MAX_UNITS) cluster *= 2;
  const int u = ((units + cluster - 1) / cluster + SM_WARPS - 1) / SM_WARPS;
  if (u == 1) MB_TRY(launch_u<1>(p, cluster, st));
  else if (u == 2) MB_TRY(launch_u<2>(p, cluster, st));
  else if (u == 3) MB_TRY(launch_u<3>(p, cluster, st));
  else MB_TRY(launch_u<4>(p, cluster, st));
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb
