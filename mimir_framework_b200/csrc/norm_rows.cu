// norm_rows.cu — LayerNorm, GroupNorm (+ SiLU, + residual), RMSNorm and softmax of rows that fit the registers of the threads that
// share them (LayerOps.hpp:264-361, 488-550; LayerOpsExt.hpp:345-378): one read and one write of every element, nothing staged.
//
// What bounds it: HBM for many rows, latency for few.  A row belongs to a warp, to a CTA of 64 ... 512 threads or to a cluster of two,
// four or eight such CTAs, chosen so that a thread holds 4 ... 32 values: enough loads in flight to stream, few enough rows per SM
// to leave none idle.  The two reductions of a row (mean and centred second moment; maximum and sum of exponentials) take one
// barrier each: warp sums through shared memory; over a cluster, CTA results pushed into every peer's shared memory before a cluster barrier.  Rows
// whose length is no multiple of four keep vector accesses: they lie on the tensor's 16-byte boundaries (SHIFT below).
// LayerNorm 32768 x 768: 41.2 -> 32.8 us (6.1 TB/s); 49840 x 674: 165 -> 72; softmax 2339 x 206: 8.2 -> 4.1, 114 x 4255: 13.3 -> 4.4;
// GroupNorm + SiLU 576 rows of 41 334 (odd image): 141 -> 87 us.  Eight rows of 32 768 in clusters of eight, one exchange instead of two and gamma
// asked for ahead of the wait: the registry transformer at batch 8 192.0 -> 189.9 us (four norms), at batch 1 from host arrays 235 -> 228 us.
#include "common.h"
#include "epilogue.cuh"
#include "launch.cuh"
#include "planes.cuh"

namespace mb {
namespace {

constexpr int NR_MAX_THREADS = 512;
constexpr long long NR_FEW_ROWS = 64;

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

// NV: vectors of four floats of a thread; WARP: a row per warp, else a row per CTA or cluster.  SHIFT: rows may start anywhere; vectors
// lie on 16-byte boundaries of the tensor all the same, those at a row's ends are moved element by element, and gamma / beta (or
// the channel of a GroupNorm) are looked up per element.  `slice`: elements of a CTA, counted from the boundary before the row.
// PLANES: a LayerNorm that only a contraction reads writes that contraction's operand planes, and the fp32 result and the pass that would
// cut it never exist (a pass of its own wrote and read them again: 1 to 3 us of a chain of launches; 40 samples x 128 tokens x 256, two
// layers: 255.6 -> 249.1 us).  Rows of k elements, a multiple of 64: the planes have no padding and the layout of the fp32 result.
template <int FAM, bool SHIFT, int NV, bool WARP, bool PLANES>
__global__ void __launch_bounds__(WARP ? 128 : NR_MAX_THREADS, WARP ? 8 : 2) norm_rows_kernel(const RowNormArgs p, const int slice) {
  __shared__ RowShared sh;
  uint32_t rank = 0, size = 1;
  if (!WARP) {
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    if (size > 1) nr_cluster_arrive();
  }
  pdl_launch_dependents();
  if (!WARP && FAM == ROWS_MEANVAR && !p.per_channel && p.gamma != nullptr && p.rows <= NR_FEW_ROWS) {
    // few long rows: gamma and beta, as long as the row, come from memory where a streaming layer has passed since (weights: no wait)
    for (int i = static_cast<int>(rank) * slice + static_cast<int>(threadIdx.x) * 32; i < min(static_cast<int>(p.len), (static_cast<int>(rank) + 1) * slice); i += static_cast<int>(blockDim.x) * 32) {
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gamma + i));
      if (p.beta != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.beta + i));
    }
  }
  pdl_wait();
  const int T = WARP ? 32 : static_cast<int>(blockDim.x), t = WARP ? static_cast<int>(threadIdx.x & 31) : static_cast<int>(threadIdx.x);
  const long long row = WARP ? static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : static_cast<long long>(blockIdx.x / size);
  if (WARP && row >= p.rows) return;
  const long long base = row * p.len;
  const int len = static_cast<int>(p.len), lead = SHIFT ? static_cast<int>(base & 3) : 0;
  const int first = static_cast<int>(rank) * slice + t * 4 - lead;  // the row's element where this thread's first vector starts
  auto el = [&](int j) { return first + j * T * 4; };
  auto mine = [&](int j) { return (t + j * T) * 4 < slice && el(j) < len; };
  auto whole = [&](int j) { return !SHIFT || (el(j) >= 0 && el(j) + 4 <= len); };  // (of a vector that is mine)
  auto in = [&](int j, int e) { return !SHIFT || static_cast<unsigned>(el(j) + e) < static_cast<unsigned>(len); };

  float v[NV][4];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const float* g = p.x + base + el(j);
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mine(j)) {
      if (whole(j)) {
        q = __ldcs(reinterpret_cast<const float4*>(g));
      } else {
        if (in(j, 0)) q.x = __ldcs(g);
        if (in(j, 1)) q.y = __ldcs(g + 1);
        if (in(j, 2)) q.z = __ldcs(g + 2);
        if (in(j, 3)) q.w = __ldcs(g + 3);
      }
    }
    v[j][0] = q.x; v[j][1] = q.y; v[j][2] = q.z; v[j][3] = q.w;
  }
  float mul = 1.0f, sub = 0.0f;  // meanvar and rms: (x - sub) * mul; softmax: maximum and 1 / sum (log: log of the sum)
  const float fn = static_cast<float>(p.len);
  if (FAM == ROWS_MEANVAR) {
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; ++j) s += (v[j][0] + v[j][1]) + (v[j][2] + v[j][3]);
    // (over a cluster: each CTA's own mean and second moment first, which then meet in ONE exchange - T. F. Chan, G. H. Golub, R. J. LeVeque
    // 1979 - with a cluster barrier fewer than exchanging the mean before the second moment)
    const bool parts = !WARP && size > 1;
    auto count = [&](int r) { return max(min((r + 1) * slice - lead, len) - max(r * slice - lead, 0), 0); };  // a CTA's elements of the row
    const float n_own = parts ? static_cast<float>(max(count(static_cast<int>(rank)), 1)) : fn;
    sub = row_reduce1<false, WARP>(s, 0, sh, 0, 1) / n_own;
    // second moment about that mean, and what the mean is off by: a large common offset costs the first sum its low bits
    float c[2] = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (mine(j)) {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (in(j, e)) { const float d = v[j][e] - sub; c[0] += d; c[1] = fmaf(d, d, c[1]); }
      }
    row_reduce<false, WARP, 2>(c, 1, sh, 0, 1);
    const float dm = c[0] / n_own;
    sub += dm;
    // (a second moment beyond fp32 makes the row zero, as the reference's does; c[0] * dm may then be infinite as well)
    float m2 = c[1] < INFINITY ? fmaxf(c[1] - c[0] * dm, 0.0f) : c[1];
    if (parts) {
      nr_cluster_wait();  // every CTA of the cluster runs (the arrive is at the kernel's start)
      if (threadIdx.x < size) {
        uint32_t at;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(&sh.cta[0][rank]))), "r"(threadIdx.x));
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(sub) : "memory");
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at + static_cast<uint32_t>(sizeof(sh.cta[0]))), "f"(m2) : "memory");
      }
      nr_cluster_arrive();
      nr_cluster_wait();
      const float ref = sh.cta[0][0];
      float off = 0.0f;
      for (int r = 1; r < static_cast<int>(size); ++r) off = fmaf(static_cast<float>(count(r)), sh.cta[0][r] - ref, off);
      sub = ref + off / fn;
      m2 = 0.0f;
      for (int r = 0; r < static_cast<int>(size); ++r) {
        const float d = sh.cta[0][r] - sub;
        if (count(r) > 0) m2 += fmaf(static_cast<float>(count(r)) * d, d, sh.cta[1][r]);
      }
    }
    mul = 1.0f / sqrtf(m2 / fn + p.eps);
  } else if (FAM == ROWS_RMS) {
    float q = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) q = fmaf(v[j][e], v[j][e], q);
    mul = 1.0f / sqrtf(row_reduce1<false, WARP>(q, 0, sh, rank, size) / fn + p.eps);
  } else {
    float m = -INFINITY, s = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (mine(j)) {
#pragma unroll
        for (int e = 0; e < 4; ++e) if (in(j, e)) m = fmaxf(m, v[j][e]);
      }
    sub = row_reduce1<true, WARP>(m, 0, sh, rank, size);
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (mine(j)) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float ex = in(j, e) ? __expf(v[j][e] - sub) : 0.0f;
          s += ex;
          if (!p.log_softmax) v[j][e] = ex;
        }
      }
    s = row_reduce1<false, WARP>(s, 1, sh, rank, size);
    mul = p.log_softmax ? logf(s) : 1.0f / s;
  }

  // GroupNorm: the channel of a vector's first element, advanced without divisions (a row's first vector may start before it)
  int ch = 0, rem = 0, ch_step = 0, rem_step = 0;
  if (FAM == ROWS_MEANVAR && p.per_channel) {
    const int f = first + p.hw;
    ch = static_cast<int>(row % p.groups) * p.cpg - 1 + f / p.hw;
    rem = f % p.hw;
    ch_step = T * 4 / p.hw;
    rem_step = T * 4 % p.hw;
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    if (!mine(j)) break;
    const int i = el(j);
    float r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (FAM == ROWS_SOFTMAX) r[e] = p.log_softmax ? (v[j][e] - sub) - mul : v[j][e] * mul;
      else r[e] = (v[j][e] - sub) * mul;
    }
    if (FAM == ROWS_RMS && p.gamma != nullptr) {
      if (!SHIFT && i + 4 <= p.n_gamma) {
        const float4 w = __ldg(reinterpret_cast<const float4*>(p.gamma + i));
        r[0] *= w.x; r[1] *= w.y; r[2] *= w.z; r[3] *= w.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) if (in(j, e) && i + e < p.n_gamma) r[e] *= __ldg(p.gamma + i + e);
      }
    }
    if (FAM == ROWS_MEANVAR) {
      if (p.gamma != nullptr) {
        float4 w, b = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.per_channel && (!SHIFT || rem + 3 < p.hw) && ch >= 0) {
          w.x = w.y = w.z = w.w = __ldg(p.gamma + ch);
          if (p.beta != nullptr) b.x = b.y = b.z = b.w = __ldg(p.beta + ch);
        } else if (!SHIFT) {
          w = __ldg(reinterpret_cast<const float4*>(p.gamma + i));
          if (p.beta != nullptr) b = __ldg(reinterpret_cast<const float4*>(p.beta + i));
        } else {
          float ww[4] = {1.f, 1.f, 1.f, 1.f}, bb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (in(j, e)) {
              const int k = p.per_channel ? ch + (rem + e) / p.hw : i + e;
              ww[e] = __ldg(p.gamma + k);
              if (p.beta != nullptr) bb[e] = __ldg(p.beta + k);
            }
          w = make_float4(ww[0], ww[1], ww[2], ww[3]);
          b = make_float4(bb[0], bb[1], bb[2], bb[3]);
        }
        r[0] = r[0] * w.x + b.x; r[1] = r[1] * w.y + b.y; r[2] = r[2] * w.z + b.z; r[3] = r[3] * w.w + b.w;
      }
      if (p.act == MIMIR_B200_ELT_SILU) {
#pragma unroll
        for (int e = 0; e < 4; e += 2) silu2(r[e], r[e + 1]);
      }
      if (p.residual != nullptr) {
        const float* q = p.residual + base + i;
        if (whole(j)) {
          const float4 a = __ldg(reinterpret_cast<const float4*>(q));
          r[0] += a.x; r[1] += a.y; r[2] += a.z; r[3] += a.w;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) if (in(j, e)) r[e] += __ldg(q + e);
        }
      }
      if (p.per_channel) {
        ch += ch_step;
        rem += rem_step;
        if (rem >= p.hw) { rem -= p.hw; ++ch; }
      }
    }
    if (PLANES) {
      uint2 h, l;
      split_pair(r[0], r[1], p.f16, h.x, l.x);
      split_pair(r[2], r[3], p.f16, h.y, l.y);
      *reinterpret_cast<uint2*>(p.y_split + base + i) = h;
      if (p.split_planes == 2) *reinterpret_cast<uint2*>(p.y_split + p.rows * p.len + base + i) = l;
      continue;
    }
    float* o = p.y + base + i;
    if (whole(j)) {
      __stcs(reinterpret_cast<float4*>(o), make_float4(r[0], r[1], r[2], r[3]));
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) if (in(j, e)) __stcs(o + e, r[e]);
    }
  }
}

// Threads and CTAs that share a row.
struct RowShape { int threads = 0, ctas = 1; };  // threads = 32: a warp
RowShape row_shape(long long rows, long long len) {
  const long long sms = ctx().sm_count;
  RowShape s;
  s.threads = len <= 1027 ? 32 : 64;  // (+ 3: see launch_norm_rows)
  while (s.threads < NR_MAX_THREADS && len > s.threads * 16LL && s.threads > 32) s.threads *= 2;
  // few rows: more threads to a row, down to four values each
  while (s.threads < NR_MAX_THREADS && rows * s.threads < sms * 512 && len > s.threads * 8LL) s.threads *= 2;
  // As few CTAs as hold the row: cluster barriers cost more than the occupancy that fewer values a thread would give (128 rows of
  // 46 656 values, GroupNorm: four CTAs 20 us, eight 31 us).
  while (s.ctas < 8 && len > static_cast<long long>(s.ctas) * NR_MAX_THREADS * 32) s.ctas *= 2;
  while (s.ctas < 8 && s.threads == NR_MAX_THREADS && rows * s.ctas * 2 <= sms * 2 && len > static_cast<long long>(s.ctas) * NR_MAX_THREADS * 8) s.ctas *= 2;
  return s;
}

template <int FAM, bool SHIFT, int NV, bool PLANES>
int launch_nv(const RowNormArgs& a, const RowShape& s, int slice, cudaStream_t st) {
  if (s.threads == 32) return launch_pdl(norm_rows_kernel<FAM, SHIFT, NV, true, PLANES>, dim3(static_cast<unsigned>((a.rows + 3) / 4)), dim3(128), 0, st, 1, a, slice);
  return launch_pdl(norm_rows_kernel<FAM, SHIFT, NV, false, PLANES>, dim3(static_cast<unsigned>(a.rows * s.ctas)), dim3(static_cast<unsigned>(s.threads)), 0, st, s.ctas, a,
                    slice);
}
template <int FAM, bool SHIFT, bool PLANES = false>
int launch_shift(const RowNormArgs& a, const RowShape& s, cudaStream_t st) {
  const long long span = a.len + (SHIFT ? 3 : 0);  // with what may lie between the boundary before the row and its start
  const int slice = static_cast<int>((((span + s.ctas - 1) / s.ctas) + 3) & ~3LL);
  const int nv = (slice / 4 + s.threads - 1) / s.threads;
  if (nv <= 1) return launch_nv<FAM, SHIFT, 1, PLANES>(a, s, slice, st);
  if (nv <= 2) return launch_nv<FAM, SHIFT, 2, PLANES>(a, s, slice, st);
  if (nv <= 3) return launch_nv<FAM, SHIFT, 3, PLANES>(a, s, slice, st);
  if (nv <= 4) return launch_nv<FAM, SHIFT, 4, PLANES>(a, s, slice, st);
  if (nv <= 5) return launch_nv<FAM, SHIFT, 5, PLANES>(a, s, slice, st);
  if (nv <= 6) return launch_nv<FAM, SHIFT, 6, PLANES>(a, s, slice, st);
  if (nv <= 7) return launch_nv<FAM, SHIFT, 7, PLANES>(a, s, slice, st);
  return launch_nv<FAM, SHIFT, 8, PLANES>(a, s, slice, st);
}
template <int FAM>
int launch_fam(const RowNormArgs& a, const RowShape& s, bool shift, cudaStream_t st) {
  return shift ? launch_shift<FAM, true>(a, s, st) : launch_shift<FAM, false>(a, s, st);
}

}  // namespace

bool norm_rows_supported(const RowNormArgs& a) {
  // (tensors that do not start on 16 bytes go to the sweep and chunk kernels)
  if (((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.y) | reinterpret_cast<uintptr_t>(a.residual)) & 15) != 0) return false;
  if (a.rows < 1 || a.rows * 8 >= 0x7fffffffLL) return false;
  const long long len = a.len + 3;
  // Longer rows: with a row for every SM the two-sweep kernel (second read from L2) keeps more rows in flight than clusters do -
  // unless it would have to move them element by element.
  return len <= NR_MAX_THREADS * 32 || (len <= 8LL * NR_MAX_THREADS * 24 && a.rows < ctx().sm_count) ||
         (len <= 8LL * NR_MAX_THREADS * 32 && (a.len & 3) != 0);
}

bool norm_rows_planes_ok(long long rows, long long len, int k) {
  RowNormArgs a;
  a.rows = rows; a.len = len;
  return k > 0 && k % 64 == 0 && len % k == 0 && norm_rows_supported(a);
}

int launch_norm_rows(const RowNormArgs& a, cudaStream_t st) {
  const RowShape s = row_shape(a.rows, a.len + 3);
  const bool affine = a.per_channel ? (a.hw & 3) == 0
                                    : ((reinterpret_cast<uintptr_t>(a.gamma) | reinterpret_cast<uintptr_t>(a.beta)) & 15) == 0;
  const bool shift = (a.len & 3) != 0 || !affine;
  int r;
  if (a.y_split != nullptr) {
    if (a.family != ROWS_MEANVAR || shift) return fail(MIMIR_B200_E_UNSUPPORTED, "norm: operand planes need aligned rows and parameters");
    r = launch_shift<ROWS_MEANVAR, false, true>(a, s, st);
  } else if (a.family == ROWS_MEANVAR) r = launch_fam<ROWS_MEANVAR>(a, s, shift, st);
  else if (a.family == ROWS_RMS) r = launch_fam<ROWS_RMS>(a, s, shift, st);
  else r = launch_fam<ROWS_SOFTMAX>(a, s, shift, st);
  if (r == MIMIR_B200_OK) count_launch();
  return r;
}

}  // namespace mb
