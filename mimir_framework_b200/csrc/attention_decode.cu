// attention_decode.cu — the attention core of a decode step: one query row per (sample, head) against the key / value cache
// (LayerOps.hpp:1044-1090 for the last row of a causal forward).  One launch appends the token's K and V to the cache and attends.
//
// The work is reading the cache once: 16 samples x 992 positions x 768 values x 2 are 98 MB a layer, 15 us at the memory rate.
// The three launches this replaces (cache write, 128-key chunks, merge over a scratch) took 34 us.  Here
//   * a cluster of up to eight CTAs shares the keys of one (sample, head); a warp takes groups of keys, LPK lanes to a key with
//     16 bytes each, and has the K and the V rows of a group in flight together (16 loads of 16 bytes a lane);
//   * scores meet by recursive halving, so that a lane exponentiates one score and not all of them; online softmax per warp;
//   * warps meet in shared memory, CTAs in rank 0's through distributed shared memory, in key order;
//   * under programmatic stream serialization the first groups of old keys are fetched while the QKV projection still runs.
#include "common.h"
#include "launch.cuh"

#include <cmath>

namespace mb {
namespace {

constexpr int AD_THREADS = 128, AD_WARPS = 4;
constexpr int AD_OCC = 3;  // CTAs per SM
constexpr int AD_U = 8;  // K rows (and V rows) a lane has in flight

struct AttnDecodeParams {
  const float* qkv;  // [batch][3 * embed]
  float* kcache;     // [batch][max_seq][embed]
  float* vcache;
  float* out;        // [batch][embed]
  const int* pos_dev;
  int pos, heads, embed, max_seq, cached_ready;
  float scale;
};

template <int LPK>
__global__ void __launch_bounds__(AD_THREADS, AD_OCC) attn_decode_fused_kernel(const AttnDecodeParams p) {
  constexpr int HD = LPK * 4, KPW = 32 / LPK;  // head size; keys a warp covers with one load
  constexpr int GROUP = KPW * AD_U;
  __shared__ float s_m[AD_WARPS], s_l[AD_WARPS];
  __shared__ __align__(16) float s_o[AD_WARPS * KPW][HD];
  __shared__ __align__(16) float gather[8][HD + 4];  // rank 0: every CTA's (max, sum, unnormalised O)
  uint32_t rank, size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const int bh = static_cast<int>(blockIdx.x / size), b = bh / p.heads, h = bh - b * p.heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPK, q4 = lane % LPK;  // key of a load, 16-byte column of the head
  const int pos = p.pos_dev ? *p.pos_dev : p.pos, nkeys = pos + 1;
  // contiguous ranges of whole groups, per CTA and then per warp
  const int groups = (nkeys + GROUP - 1) / GROUP;
  const int parts = static_cast<int>(size) * AD_WARPS, me = static_cast<int>(rank) * AD_WARPS + warp;
  const int g0 = static_cast<int>(static_cast<long long>(groups) * me / parts), g1 = static_cast<int>(static_cast<long long>(groups) * (me + 1) / parts);
  const long long head_off = static_cast<long long>(b) * p.max_seq * p.embed + h * HD + q4 * 4;
  const float* kc = p.kcache + head_off;
  const float* vc = p.vcache + head_off;
  const float* qrow = p.qkv + static_cast<long long>(b) * 3 * p.embed + h * HD + q4 * 4;

  float4 kv[AD_U], vv[AD_U];
  int off[AD_U];  // of a lane's rows within a group
#pragma unroll
  for (int u = 0; u < AD_U; ++u) off[u] = (u * KPW + sub) * p.embed;
  auto load_rows = [&](float4 (&r)[AD_U], const float* base, int g) {  // the cached rows of group g (the new one comes from the projection)
    const float* at = base + static_cast<long long>(g) * (GROUP * p.embed);
    if ((g + 1) * GROUP <= pos) {  // (warp-uniform) all cached: no predicates
#pragma unroll
      for (int u = 0; u < AD_U; ++u)
        asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r[u].x), "=f"(r[u].y), "=f"(r[u].z), "=f"(r[u].w) : "l"(at + off[u]));
    } else {
#pragma unroll
      for (int u = 0; u < AD_U; ++u) {
        r[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g * GROUP + u * KPW + sub < pos)
          asm volatile("ld.global.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(r[u].x), "=f"(r[u].y), "=f"(r[u].z), "=f"(r[u].w) : "l"(at + off[u]));
      }
    }
  };
  if (!p.cached_ready) pdl_wait();
  if (g0 < g1) {
    load_rows(kv, kc, g0);
    load_rows(vv, vc, g0);
  }
  pdl_launch_dependents();
  pdl_wait();
  const float4 q = *reinterpret_cast<const float4*>(qrow);

  float m = -1e30f, l = 0.0f;  // the reference's initial maximum (LayerOps.hpp:1052)
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int g = g0; g < g1; ++g) {
    if (pos >= g * GROUP && pos < (g + 1) * GROUP) {  // (warp-uniform) the new key is in this group: use it and store it
#pragma unroll
      for (int u = 0; u < AD_U; ++u)
        if (g * GROUP + u * KPW + sub == pos) {
          kv[u] = *reinterpret_cast<const float4*>(qrow + p.embed);
          vv[u] = *reinterpret_cast<const float4*>(qrow + 2 * p.embed);
          const long long o = head_off + static_cast<long long>(pos) * p.embed;
          *reinterpret_cast<float4*>(p.kcache + o) = kv[u];
          *reinterpret_cast<float4*>(p.vcache + o) = vv[u];
        }
    }
    float d[AD_U];
#pragma unroll
    for (int u = 0; u < AD_U; ++u) d[u] = fmaf(q.w, kv[u].w, fmaf(q.z, kv[u].z, fmaf(q.y, kv[u].y, q.x * kv[u].x)));
    if (g + 1 < g1) load_rows(kv, kc, g + 1);  // in flight while this group's softmax and P V run
    // sum over the LPK lanes of a key: three rounds halve the eight values, the rest add one value up; the lane's bits LPK/2,
    // LPK/4, LPK/8 name the key of the load it ends with
#pragma unroll
    for (int half = AD_U / 2, mask = LPK / 2; half >= 1; half >>= 1, mask >>= 1) {
      const bool upper = (lane & mask) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float send = upper ? d[i] : d[i + half];
        const float keep = upper ? d[i + half] : d[i];
        d[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
      }
    }
#pragma unroll
    for (int mask = LPK / (2 * AD_U); mask >= 1; mask >>= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], mask);
    const int mine = (q4 * AD_U) / LPK;  // which of the AD_U
    const bool in = g * GROUP + mine * KPW + sub < nkeys;
    const float s = in ? d[0] * p.scale : -INFINITY;
    float mx = s;
#pragma unroll
    for (int mask = 16; mask >= LPK / AD_U; mask >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, mask));
    const float mn = fmaxf(m, mx), corr = expf(m - mn);
    m = mn;
    const float pr = expf(s - mn);  // exp(-inf) = 0 past the last key
    l = fmaf(l, corr, pr);
    acc.x *= corr; acc.y *= corr; acc.z *= corr; acc.w *= corr;
#pragma unroll
    for (int u = 0; u < AD_U; ++u) {
      const float w = __shfl_sync(0xffffffffu, pr, sub * LPK + u * (LPK / AD_U));
      acc.x = fmaf(w, vv[u].x, acc.x); acc.y = fmaf(w, vv[u].y, acc.y); acc.z = fmaf(w, vv[u].z, acc.z); acc.w = fmaf(w, vv[u].w, acc.w);
    }
    if (g + 1 < g1) load_rows(vv, vc, g + 1);
  }
  // l: LPK / 8 lanes hold the same probabilities; the sum over the warp counts each that often (a power of two, exact)
#pragma unroll
  for (int mask = 16; mask >= 1; mask >>= 1) l += __shfl_xor_sync(0xffffffffu, l, mask);
  l *= static_cast<float>(AD_U) / LPK;
  *reinterpret_cast<float4*>(&s_o[warp * KPW + sub][q4 * 4]) = acc;
  if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA of the cluster runs
  float cm = s_m[0];
#pragma unroll
  for (int w = 1; w < AD_WARPS; ++w) cm = fmaxf(cm, s_m[w]);
  uint32_t dst;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&gather[rank][0]))));
  auto put = [&](int i, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + i * 4), "f"(v) : "memory"); };
  for (int d = threadIdx.x; d < HD; d += AD_THREADS) {
    float o = 0.0f;
#pragma unroll
    for (int w = 0; w < AD_WARPS; ++w) {
      float t = s_o[w * KPW][d];
#pragma unroll
      for (int k = 1; k < KPW; ++k) t += s_o[w * KPW + k][d];
      o = fmaf(t, expf(s_m[w] - cm), o);
    }
    put(4 + d, o);
  }
  if (threadIdx.x == 0) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < AD_WARPS; ++w) t = fmaf(s_l[w], expf(s_m[w] - cm), t);
    put(0, cm);
    put(1, t);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (rank != 0) return;
  float gm = -1e30f;
  for (uint32_t c = 0; c < size; ++c) gm = fmaxf(gm, gather[c][0]);
  float gl = 0.0f;
  for (uint32_t c = 0; c < size; ++c) gl = fmaf(gather[c][1], expf(gather[c][0] - gm), gl);
  const float inv = 1.0f / (gl + 1e-9f);  // LayerOps.hpp:1076
  for (int d = threadIdx.x; d < HD; d += AD_THREADS) {
    float o = 0.0f;
    for (uint32_t c = 0; c < size; ++c) o = fmaf(gather[c][4 + d], expf(gather[c][0] - gm), o);
    p.out[static_cast<long long>(b) * p.embed + h * HD + d] = o * inv;
  }
}

}  // namespace

bool attention_decode_fused_supported(int batch, int embed, int heads) {
  const int hd = heads > 0 ? embed / heads : 0;
  return heads > 0 && embed % heads == 0 && (hd == 32 || hd == 64 || hd == 128) && static_cast<long long>(batch) * heads <= (1 << 24);
}

int launch_attention_decode_fused(const float* qkv, float* kcache, float* vcache, float* out, int batch, int embed, int heads, int max_seq,
                                  int pos, const int* pos_dev, bool cached_ready, cudaStream_t st) {
  if (!attention_decode_fused_supported(batch, embed, heads)) return fail(MIMIR_B200_E_UNSUPPORTED, "attention: not a head layout of the fused decode kernel");
  const int hd = embed / heads, bh = batch * heads;
  AttnDecodeParams p;
  p.qkv = qkv; p.kcache = kcache; p.vcache = vcache; p.out = out; p.pos_dev = pos_dev; p.pos = pos; p.heads = heads; p.embed = embed;
  p.max_seq = max_seq; p.cached_ready = cached_ready ? 1 : 0;
  p.scale = 1.0f / sqrtf(static_cast<float>(hd));
  // as many CTAs per (sample, head) as keep the launch within one wave, in powers of two (clusters of three left SMs empty:
  // 16 samples x 12 heads, 992 keys: 25 us; of two, 17.3 us = 5.6 TB/s)
  const int fit = AD_OCC * ctx().sm_count / bh;
  const int c = fit >= 8 ? 8 : fit >= 4 ? 4 : fit >= 2 ? 2 : 1;
  const dim3 grid(static_cast<unsigned>(bh) * static_cast<unsigned>(c)), block(AD_THREADS);
  if (hd == 32) MB_TRY(launch_pdl(attn_decode_fused_kernel<8>, grid, block, 0, st, c, p));
  else if (hd == 64) MB_TRY(launch_pdl(attn_decode_fused_kernel<16>, grid, block, 0, st, c, p));
  else MB_TRY(launch_pdl(attn_decode_fused_kernel<32>, grid, block, 0, st, c, p));
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb
