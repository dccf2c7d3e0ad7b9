// norm_rows.cu — LayerNorm, GroupNorm (+ SiLU, + residual), RMSNorm and softmax of rows that fit the registers of the threads that
// share them (LayerOps.hpp:264-361, 488-550; LayerOpsExt.hpp:345-378): one read and one write of every element, nothing staged.
//
// What bounds it: HBM for many rows, latency for few.  A row belongs to a warp, to a CTA of 64 ... 512 threads or to a cluster of two,
// four or eight such CTAs, chosen so that a thread holds 4 ... 32 values: enough loads in flight to stream, few enough rows per SM
// to leave none idle.  The two reductions of a row (mean and centred second moment; maximum and sum of exponentials) take one
// barrier each: warp sums through shared memory, CTA sums pushed into every peer's shared memory before a cluster barrier.  Rows
// whose length is no multiple of four are read and written element by element, still in whole lines.
// ROWS_FIGURES
#include "common.h"
#include "launch.cuh"

namespace mb {
namespace {

constexpr int NR_MAX_THREADS = 512;

__device__ __forceinline__ void nr_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void nr_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

template <bool MAX>
__device__ __forceinline__ float combine(float a, float b) { return MAX ? fmaxf(a, b) : a + b; }

struct RowShared {
  float warp[3][NR_MAX_THREADS / 32];
  float cta[3][8];
};

// Over the threads that share the row, NR values at once; the row's first reduction has step 0, its second step 1.
template <bool MAX, bool WARP, int NR>
__device__ __forceinline__ void row_reduce(float (&v)[NR], int step, RowShared& sh, uint32_t rank, uint32_t size) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
#pragma unroll
    for (int k = 0; k < NR; ++k) v[k] = combine<MAX>(v[k], __shfl_xor_sync(0xffffffffu, v[k], d));
  if (WARP) return;
  const int nw = static_cast<int>(blockDim.x) >> 5;
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < NR; ++k) sh.warp[step + k][threadIdx.x >> 5] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NR; ++k) {
    v[k] = sh.warp[step + k][0];
    for (int w = 1; w < nw; ++w) v[k] = combine<MAX>(v[k], sh.warp[step + k][w]);
  }
  if (size > 1) {
    if (step == 0) nr_cluster_wait();  // every CTA of the cluster runs (the arrive is at the kernel's start)
    if (threadIdx.x < size) {
#pragma unroll
      for (int k = 0; k < NR; ++k) {
        uint32_t a;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&sh.cta[step + k][rank]))), "r"(threadIdx.x));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v[k]) : "memory");
      }
    }
    nr_cluster_arrive();
    nr_cluster_wait();
#pragma unroll
    for (int k = 0; k < NR; ++k) {
      v[k] = sh.cta[step + k][0];
      for (uint32_t c = 1; c < size; ++c) v[k] = combine<MAX>(v[k], sh.cta[step + k][c]);
    }
  }
}
template <bool MAX, bool WARP>
__device__ __forceinline__ float row_reduce1(float v, int step, RowShared& sh, uint32_t rank, uint32_t size) {
  float a[1] = {v};
  row_reduce<MAX, WARP, 1>(a, step, sh, rank, size);
  return a[0];
}

// NV: vectors (VEC: of four floats) of a thread; WARP: a row per warp, else a row per CTA or cluster.
template <int FAM, bool VEC, int NV, bool WARP>
__global__ void __launch_bounds__(WARP ? 128 : NR_MAX_THREADS) norm_rows_kernel(const RowNormArgs p, const int slice) {
  constexpr int W = VEC ? 4 : 1;
  __shared__ RowShared sh;
  uint32_t rank = 0, size = 1;
  if (!WARP) {
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    if (size > 1) nr_cluster_arrive();
  }
  pdl_launch_dependents();
  pdl_wait();
  const int T = WARP ? 32 : static_cast<int>(blockDim.x), t = WARP ? static_cast<int>(threadIdx.x & 31) : static_cast<int>(threadIdx.x);
  const long long row = WARP ? static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : static_cast<long long>(blockIdx.x / size);
  if (WARP && row >= p.rows) return;
  const int off = static_cast<int>(rank) * slice, n = min(slice, static_cast<int>(p.len) - off);  // this CTA's part of the row
  const long long base = row * p.len + off;
  const float* g = p.x + base;

  float v[NV][W];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (t + j * T) * W;
    if (VEC) {
      const float4 q = i < n ? __ldcs(reinterpret_cast<const float4*>(g + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[j][0] = q.x; v[j][W > 1 ? 1 : 0] = W > 1 ? q.y : q.x;
      if (W > 1) { v[j][W - 2] = q.z; v[j][W - 1] = q.w; }
    } else {
      v[j][0] = i < n ? __ldcs(g + i) : 0.0f;
    }
  }
  float mul = 1.0f, sub = 0.0f;  // meanvar and rms: (x - sub) * mul; softmax: maximum and 1 / sum (log: log of the sum)
  const float fn = static_cast<float>(p.len);
  if (FAM == ROWS_MEANVAR) {
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int e = 0; e < W; ++e) s += v[j][e];
    sub = row_reduce1<false, WARP>(s, 0, sh, rank, size) / fn;
    // second moment about that mean, and what the mean is off by: a large common offset costs the first sum its low bits
    float c[2] = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if ((t + j * T) * W < n) {
#pragma unroll
        for (int e = 0; e < W; ++e) { const float d = v[j][e] - sub; c[0] += d; c[1] = fmaf(d, d, c[1]); }
      }
    row_reduce<false, WARP, 2>(c, 1, sh, rank, size);
    const float dm = c[0] / fn;
    sub += dm;
    mul = 1.0f / sqrtf(fmaxf(c[1] - c[0] * dm, 0.0f) / fn + p.eps);
  } else if (FAM == ROWS_RMS) {
    float q = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int e = 0; e < W; ++e) q = fmaf(v[j][e], v[j][e], q);
    mul = 1.0f / sqrtf(row_reduce1<false, WARP>(q, 0, sh, rank, size) / fn + p.eps);
  } else {
    float m = -INFINITY, s = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if ((t + j * T) * W < n) {
#pragma unroll
        for (int e = 0; e < W; ++e) m = fmaxf(m, v[j][e]);
      }
    sub = row_reduce1<true, WARP>(m, 0, sh, rank, size);
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if ((t + j * T) * W < n) {
#pragma unroll
        for (int e = 0; e < W; ++e) {
          const float ex = __expf(v[j][e] - sub);
          s += ex;
          if (!p.log_softmax) v[j][e] = ex;
        }
      }
    s = row_reduce1<false, WARP>(s, 1, sh, rank, size);
    mul = p.log_softmax ? logf(s) : 1.0f / s;
  }

  float* o = p.y + base;
  // GroupNorm: the channel of this thread's elements, advanced without divisions
  unsigned ch = 0, rem = 0, ch_step = 0, rem_step = 0;
  const unsigned hw = static_cast<unsigned>(p.hw);
  if (FAM == ROWS_MEANVAR && p.per_channel) {
    const unsigned first = static_cast<unsigned>(off + t * W), step = static_cast<unsigned>(T * W);
    ch = static_cast<unsigned>(static_cast<int>(row % p.groups) * p.cpg) + first / hw;
    rem = first % hw;
    ch_step = step / hw;
    rem_step = step % hw;
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (t + j * T) * W;
    if (i >= n) break;
    float r[W];
#pragma unroll
    for (int e = 0; e < W; ++e) r[e] = v[j][e];
    if (FAM == ROWS_SOFTMAX) {
#pragma unroll
      for (int e = 0; e < W; ++e) r[e] = p.log_softmax ? (r[e] - sub) - mul : r[e] * mul;
    } else {
#pragma unroll
      for (int e = 0; e < W; ++e) r[e] = (r[e] - sub) * mul;
    }
    if (FAM == ROWS_RMS && p.gamma != nullptr) {
      if (VEC && off + i + W <= p.n_gamma) {
        const float4 w = __ldg(reinterpret_cast<const float4*>(p.gamma + off + i));
        r[0] *= w.x; r[W > 1 ? 1 : 0] *= W > 1 ? w.y : 1.0f;
        if (W > 1) { r[W - 2] *= w.z; r[W - 1] *= w.w; }
      } else {
#pragma unroll
        for (int e = 0; e < W; ++e) if (off + i + e < p.n_gamma) r[e] *= __ldg(p.gamma + off + i + e);
      }
    }
    if (FAM == ROWS_MEANVAR) {
      if (p.gamma != nullptr) {
        if (p.per_channel) {  // (vectors never cross a channel: hw is a multiple of four there)
          const float w = __ldg(p.gamma + ch), b = p.beta != nullptr ? __ldg(p.beta + ch) : 0.0f;
#pragma unroll
          for (int e = 0; e < W; ++e) r[e] = r[e] * w + b;
        } else if (VEC) {
          const float4 w = __ldg(reinterpret_cast<const float4*>(p.gamma + off + i));
          float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
          if (p.beta != nullptr) b = __ldg(reinterpret_cast<const float4*>(p.beta + off + i));
          r[0] = r[0] * w.x + b.x;
          if (W > 1) { r[1 % W] = r[1 % W] * w.y + b.y; r[W - 2] = r[W - 2] * w.z + b.z; r[W - 1] = r[W - 1] * w.w + b.w; }
        } else {
          r[0] = r[0] * __ldg(p.gamma + off + i) + (p.beta != nullptr ? __ldg(p.beta + off + i) : 0.0f);
        }
      }
      if (p.act == MIMIR_B200_ELT_SILU) {
#pragma unroll
        for (int e = 0; e < W; ++e) r[e] = r[e] * (1.0f / (1.0f + expf(-r[e])));
      }
      if (p.residual != nullptr) {
        if (VEC) {
          const float4 q = __ldg(reinterpret_cast<const float4*>(p.residual + base + i));
          r[0] += q.x;
          if (W > 1) { r[1 % W] += q.y; r[W - 2] += q.z; r[W - 1] += q.w; }
        } else {
          r[0] += __ldg(p.residual + base + i);
        }
      }
      if (p.per_channel) {
        ch += ch_step;
        rem += rem_step;
        if (rem >= hw) { rem -= hw; ++ch; }
      }
    }
    if (VEC) __stcs(reinterpret_cast<float4*>(o + i), make_float4(r[0], r[1 % W], r[2 % W], r[3 % W]));
    else __stcs(o + i, r[0]);
  }
}

// Threads and CTAs that share a row.
struct RowShape { int threads = 0, ctas = 1; };  // threads = 32: a warp
RowShape row_shape(long long rows, long long len) {
  const long long sms = ctx().sm_count;
  RowShape s;
  s.threads = len <= 1024 ? 32 : 64;
  while (s.threads < NR_MAX_THREADS && len > s.threads * 16LL && s.threads > 32) s.threads *= 2;
  // few rows: more threads to a row, down to four values each
  while (s.threads < NR_MAX_THREADS && rows * s.threads < sms * 512 && len > s.threads * 8LL) s.threads *= 2;
  while (s.ctas < 8 && len > static_cast<long long>(s.ctas) * NR_MAX_THREADS * 32) s.ctas *= 2;
  while (s.ctas < 8 && s.threads == NR_MAX_THREADS && rows * s.ctas * 2 <= sms * 2 && len > static_cast<long long>(s.ctas) * NR_MAX_THREADS * 8) s.ctas *= 2;
  return s;
}

template <int FAM, bool VEC, int NV>
int launch_nv(const RowNormArgs& a, const RowShape& s, int slice, cudaStream_t st) {
  if (s.threads == 32) return launch_pdl(norm_rows_kernel<FAM, VEC, NV, true>, dim3(static_cast<unsigned>((a.rows + 3) / 4)), dim3(128), 0, st, 1, a, slice);
  return launch_pdl(norm_rows_kernel<FAM, VEC, NV, false>, dim3(static_cast<unsigned>(a.rows * s.ctas)), dim3(static_cast<unsigned>(s.threads)), 0, st, s.ctas, a, slice);
}
template <int FAM>
int launch_fam(const RowNormArgs& a, const RowShape& s, bool vec, cudaStream_t st) {
  const int slice = static_cast<int>((((a.len + s.ctas - 1) / s.ctas) + 3) & ~3LL);
  const int per = (slice + s.threads - 1) / s.threads;  // values of a thread
  if (vec) {
    const int nv = (slice / 4 + s.threads - 1) / s.threads;
    if (nv <= 1) return launch_nv<FAM, true, 1>(a, s, slice, st);
    if (nv <= 2) return launch_nv<FAM, true, 2>(a, s, slice, st);
    if (nv <= 4) return launch_nv<FAM, true, 4>(a, s, slice, st);
    if (nv <= 6) return launch_nv<FAM, true, 6>(a, s, slice, st);
    return launch_nv<FAM, true, 8>(a, s, slice, st);
  }
  if (per <= 8) return launch_nv<FAM, false, 8>(a, s, slice, st);
  if (per <= 16) return launch_nv<FAM, false, 16>(a, s, slice, st);
  return launch_nv<FAM, false, 32>(a, s, slice, st);
}

}  // namespace

bool norm_rows_supported(long long rows, long long len) {
  // Longer rows: with a row for every SM the two-sweep kernel (second read from L2) keeps more rows in flight than clusters do.
  return rows >= 1 && rows * 8 < 0x7fffffffLL && (len <= NR_MAX_THREADS * 32 || (len <= 8LL * NR_MAX_THREADS * 32 && rows < ctx().sm_count));
}

int launch_norm_rows(const RowNormArgs& a, cudaStream_t st) {
  const RowShape s = row_shape(a.rows, a.len);
  const bool affine16 = a.per_channel ? (a.hw & 3) == 0
                                      : ((reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta)) & 15) == 0;
  const bool vec = (a.len & 3) == 0 && affine16 &&
                   ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.residual)) & 15) == 0;
  int r;
  if (a.family == ROWS_MEANVAR) r = launch_fam<ROWS_MEANVAR>(a, s, vec, st);
  else if (a.family == ROWS_RMS) r = launch_fam<ROWS_RMS>(a, s, vec, st);
  else r = launch_fam<ROWS_SOFTMAX>(a, s, vec, st);
  if (r == MIMIR_B200_OK) count_launch();
  return r;
}

}  // namespace mb
