// conv2d.cu — Conv2d lowered to the tensor-core GEMM.  Replaces the inline Conv2d case of the
// layer switch (Model.cpp:4897-5089): CHW activations, OIHW weights, square kernel, zero padding,
// no bias.  The reference itself computes im2col rows ordered (ic, kh, kw) (Model.cpp:5005-5029)
// times the transposed weights (Model.cpp:5032); here the im2col rows are produced directly as the
// bf16 hi/lo planes the GEMM consumes (one pass over the input, no fp32 column matrix), the OIHW
// weight block already is the K-major [oc][ic*k*k] operand, and the GEMM epilogue writes NCHW.
#include "common.h"
#include "epilogue.cuh"
#include "planes.cuh"

namespace mb {
namespace {

__device__ __forceinline__ void cp_async16_zfill(void* smem_dst, const void* gmem_src, bool valid) {
  // 16 bytes, or 16 zero bytes when !valid (source size 0: nothing is read)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gmem_src), "r"(valid ? 16 : 0)
               : "memory");
}

__device__ __forceinline__ void cp_async4_zfill(void* smem_dst, const void* gmem_src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
               "l"(gmem_src), "r"(valid ? 4 : 0)
               : "memory");
}

// One thread produces 8 consecutive K entries of one output pixel.
__global__ void im2col_split_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ dst, long long rows, int ic, int h,
                                    int w, int ks, int stride, int pad, int oh, int ow, int k, int kp, int planes, int f16) {
  const int chunks = kp >> 3;
  const long long total = rows * chunks;
  const long long plane_stride = rows * static_cast<long long>(kp);
  const int ohw = oh * ow, kk = ks * ks;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    // consecutive threads write consecutive 16-byte chunks of one im2col row (coalesced stores, the
    // larger stream); the input, 1/k^2 of the size, is re-read through L1/L2
    const long long r = i / chunks;
    const int c = static_cast<int>(i - r * chunks);
    const long long smp = r / ohw;
    const int pix = static_cast<int>(r - smp * ohw);
    const int oy = pix / ow, ox = pix - oy * ow;
    const float* xs = x + smp * ic * h * w;
    __align__(16) uint16_t hi[8];
    __align__(16) uint16_t lo[8];
    // (ci, ky, kx) of the chunk's first entry by division, of the other seven by stepping
    int ci = (c * 8) / kk, t = c * 8 - ci * kk;
    int ky = t / ks, kx = t - ky * ks;
    const int iy0 = oy * stride - pad, ix0 = ox * stride - pad;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v = 0.0f;
      if (c * 8 + j < k) {
        const int iy = iy0 + ky, ix = ix0 + kx;
        if (iy >= 0 && iy < h && ix >= 0 && ix < w) v = __ldg(xs + (static_cast<long long>(ci) * h + iy) * w + ix);
      }
      split_one(v, f16, hi[j], lo[j]);
      if (++kx == ks) {
        kx = 0;
        if (++ky == ks) { ky = 0; ++ci; }
      }
    }
    __nv_bfloat16* d = dst + r * kp + c * 8;
    *reinterpret_cast<uint4*>(d) = *reinterpret_cast<const uint4*>(hi);
    if (planes == 2) *reinterpret_cast<uint4*>(d + plane_stride) = *reinterpret_cast<const uint4*>(lo);
  }
}

// The same rows from a staged input patch: a CTA owns `tpx` consecutive output pixels of one output row and a block of `cb` input
// channels (a multiple of 8, or all of them), loads the patch those pixels read - cb x ks rows of (tpx - 1) * stride + ks input
// pixels, coalesced, a warp per row - into shared memory once, and assembles the 16-byte chunks of its K range from there.  A thread
// keeps one chunk of the K range and walks the pixels, so the eight places of the patch a chunk reads are worked out once; consecutive
// threads hold consecutive chunks of one pixel, i.e. contiguous stores.
// (With the index arithmetic done per chunk and pixel the kernel was bound by it: 16 x 512 x 64^2, 3 x 3 stride 2: 208 us for 302 MB
// written; now 118 us.  64 x 3 x 224^2, 7 x 7 stride 2: 310 us, now 129 us.)
// KS: the kernel size, 0 = any (then `ks_any`).
template <int KS>
__global__ void __launch_bounds__(256) im2col_tile_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ dst, long long rows,
                                                          int ic, int h, int w, int ks_any, int stride, int pad, int oh, int ow, int kp,
                                                          int planes, int f16, int cb, int nblocks, int tpx) {
  extern __shared__ float patch[];  // [cbn][ks][pw], then one zero
  const int ks = KS ? KS : ks_any, kk = ks * ks;
  const int ox0 = blockIdx.x * tpx, oy = blockIdx.y;
  const int smp = blockIdx.z / nblocks, blk = blockIdx.z - smp * nblocks;
  const int c0 = blk * cb, cbn = min(cb, ic - c0);
  const int pw = (tpx - 1) * stride + ks;
  const int iy0 = oy * stride - pad, ix0 = ox0 * stride - pad;
  const float* xs = x + (static_cast<long long>(smp) * ic + c0) * h * w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < cbn * ks; r += 8) {
    const int c = r / ks, iy = iy0 + r - c * ks;
    const float* line = xs + (static_cast<long long>(c) * h + iy) * w;
    const bool row_in = iy >= 0 && iy < h;
    for (int px = lane; px < pw; px += 32) {
      const int ix = ix0 + px;
      const bool ok = row_in && ix >= 0 && ix < w;  // (asynchronous: a warp's rows are all in flight at once)
      cp_async4_zfill(&patch[r * pw + px], ok ? line + ix : x, ok);
    }
  }
  if (threadIdx.x == 0) patch[cbn * ks * pw] = 0.0f;
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // this block's chunks of a row: its channels' K range; the last block also writes the zero padding up to kp
  const int ch_lo = (c0 * kk) >> 3, ch_hi = (blk == nblocks - 1) ? (kp >> 3) : (((c0 + cbn) * kk) >> 3);
  const int nch = ch_hi - ch_lo, npx = min(tpx, ow - ox0);
  const int groups = nch < 256 ? 256 / nch : 1;  // pixels the CTA works on at once
  const int g = nch < 256 ? static_cast<int>(threadIdx.x) / nch : 0;
  const long long plane_stride = rows * static_cast<long long>(kp);
  const long long row0 = (static_cast<long long>(smp) * oh + oy) * ow + ox0;
  if (g >= groups) return;
  for (int chunk = static_cast<int>(threadIdx.x) - g * nch; chunk < nch; chunk += 256) {
    int off[8], step[8];  // where the chunk's elements of pixel 0 are, and how far the next pixel's (0: the zero past the last channel)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int kidx = (ch_lo + chunk) * 8 + j - c0 * kk, ci = kidx / kk, t = kidx - ci * kk, ky = t / ks;
      off[j] = ci < cbn ? (ci * ks + ky) * pw + t - ky * ks : cbn * ks * pw;
      step[j] = ci < cbn ? stride : 0;
    }
    for (int p = g; p < npx; p += groups) {
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int j = 0; j < 8; j += 2) split_pair(patch[off[j] + p * step[j]], patch[off[j + 1] + p * step[j + 1]], f16, hi[j >> 1], lo[j >> 1]);
      __nv_bfloat16* d = dst + (row0 + p) * kp + (ch_lo + chunk) * 8;
      *reinterpret_cast<uint4*>(d) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      if (planes == 2) *reinterpret_cast<uint4*>(d + plane_stride) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

}  // namespace

int launch_im2col_split(const float* x, __nv_bfloat16* dst, int batch, int ic, int h, int w, int ks, int stride, int pad,
                        int oh, int ow, int planes, cudaStream_t st) {
  if (batch <= 0 || ic <= 0 || oh <= 0 || ow <= 0 || ks <= 0 || stride <= 0)
    return fail(MIMIR_B200_E_INVALID, "Conv2d: in_channels and out_channels must be set");
  const int k = ic * ks * ks, kp = round_up(k, 64);
  const long long rows = static_cast<long long>(batch) * oh * ow;
  {
    // the staged form: channel blocks of a multiple of 8 (so that every block starts on a chunk boundary) within 48 KB
    static const bool off = [] { const char* e = getenv("MIMIR_B200_IM2COL_TILED"); return e && e[0] == '0'; }();
    // about 64 pixels of a row, evenly cut; patches of 28 KB: several CTAs to an SM, one's loads beside another's stores
    const int cuts = (ow + 63) / 64, tpx = (ow + cuts - 1) / cuts;
    const int pw = (tpx - 1) * stride + ks;
    const long long per_ch = static_cast<long long>(ks) * pw * 4;
    int cb = static_cast<int>(std::min<long long>(ic, (28 * 1024) / per_ch));
    if (cb < ic) cb &= ~7;
    if (cb == 0) cb = static_cast<int>(std::min<long long>(ic, (47 * 1024) / per_ch));
    if (cb < ic) cb &= ~7;
    const int nblocks = cb > 0 ? (ic + cb - 1) / cb : 0;
    if (!off && cb > 0 && static_cast<long long>(batch) * nblocks <= 65535 && oh <= 65535) {
      const dim3 grid(cuts, oh, batch * nblocks);
      auto kern = ks == 3 ? im2col_tile_kernel<3> : ks == 7 ? im2col_tile_kernel<7> : im2col_tile_kernel<0>;
      kern<<<grid, 256, static_cast<size_t>(cb) * per_ch + 4, st>>>(x, dst, rows, ic, h, w, ks, stride, pad, oh, ow, kp, planes, plane_format() == PLANES_F16, cb,
                                                                    nblocks, tpx);
      MB_CUDA(cudaGetLastError());
      count_launch();
      return MIMIR_B200_OK;
    }
  }
  const long long total = rows * (kp >> 3);
  long long blocks = (total + 255) / 256;
  const long long cap = static_cast<long long>(ctx().sm_count) * 32;
  if (blocks > cap) blocks = cap;
  im2col_split_kernel<<<static_cast<int>(blocks), 256, 0, st>>>(x, dst, rows, ic, h, w, ks, stride, pad, oh, ow, k, kp, planes, plane_format() == PLANES_F16);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb

// ---------------------------------------------------------------------------------------------
// Stride-1 "same" convolutions without a materialised im2col: the GEMM kernel sums one shifted
// GEMM per filter tap over the zero-padded NHWC activation matrix (see GemmParams::conv_*).  The
// two kernels below produce its operands.
// ---------------------------------------------------------------------------------------------
namespace mb {
namespace {

constexpr int TP_C = 64, TP_X = 64;

// NCHW fp32 -> zero-padded NHWC planes.  A channel plane is read as one line of h * w pixels, so that no tile (64 channels x 64
// pixels) is cut short at the end of an image row; a CTA owns `tiles_per_cta` consecutive tiles of one sample and 64 channels, and the
// source of tile t + 1 is on its way into the second shared-memory buffer while tile t is normalised, split and stored: the loads of a
// CTA never stop for its stores.  A thread stores eight channels of a pixel as one 16-byte word per plane.  The tile is kept with its
// 16-byte column groups XOR-ed with the channel's octet: the eight lanes that write one pixel's 64 channels then read eight
// different bank groups.
//   VEC = 1: planes start on 16-byte boundaries (h * w a multiple of 4): 16-byte copies.  VEC = 0: 4-byte copies.
//   UP = 1: x is the half-size image of a 2 x 2 nearest upsample: each source pixel is normalised and split once and stored four times.
// The padding ring is shared out evenly among a sample's CTAs.
// Measured (17 samples, 70 x 70, 64 ... 256 channels, six passes): 382 -> 93 us against the element-wise form this replaces, which took every
// width that is no multiple of four; UNet 256 x 256 upsampled pass 152 -> 110 us.
constexpr int LR_TS = TP_X + 4;
template <int UP, int VEC>
__global__ void __launch_bounds__(256, 5) nchw_to_padded_nhwc_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ dst, int c, int h, int w, int pad,
                                                                     int planes, long long plane_stride, const PreNorm pre, int f16, int tiles_per_cta) {
  __shared__ __align__(16) float tile[2][TP_C][LR_TS];
  const int hp = h + 2 * pad, wp = w + 2 * pad;
  const int cb = blockIdx.x * TP_C, n = blockIdx.z;
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  const long long sample = static_cast<long long>(n) * hp * wp;
  auto store8 = [&](long long pixel, int ch, const uint4& hi, const uint4& lo) {
    __nv_bfloat16* o = dst + (sample + pixel) * c + ch;
    *reinterpret_cast<uint4*>(o) = hi;
    if (planes == 2) *reinterpret_cast<uint4*>(o + plane_stride) = lo;
  };
  const int sw_ = UP ? w >> 1 : w, src_pixels = (UP ? h >> 1 : h) * sw_;
  const float* src = x + (static_cast<long long>(n) * c + cb) * src_pixels;
  const int t0 = blockIdx.y * tiles_per_cta, t1 = min(t0 + tiles_per_cta, (src_pixels + TP_X - 1) / TP_X);
  auto issue = [&](int t) {
    const int p0 = t * TP_X;
    float(*buf)[LR_TS] = tile[t & 1];
    constexpr int PER = VEC ? TP_X / 4 : TP_X;  // copies of one channel
#pragma unroll
    for (int i = 0; i < TP_C * PER / 256; ++i) {
      const int idx = threadIdx.x + 256 * i, cc = idx / PER, q = idx - cc * PER, oct = (cc >> 3) & 7;
      const int p = p0 + (VEC ? 4 * q : q);
      const bool ok = p < src_pixels && cb + cc < c;
      const float* from = ok ? src + static_cast<long long>(cc) * src_pixels + p : x;
      if (VEC) cp_async16_zfill(&buf[cc][4 * (q ^ oct)], from, ok);
      else cp_async4_zfill(&buf[cc][4 * ((q >> 2) ^ oct) + (q & 3)], from, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  issue(t0);
  // this CTA's share of the padding ring: whole rows above and below, then the sides
  {
    const int ring = hp * wp - h * w, r0 = static_cast<int>(static_cast<long long>(ring) * blockIdx.y / gridDim.y),
              r1 = static_cast<int>(static_cast<long long>(ring) * (blockIdx.y + 1) / gridDim.y);
    for (int i = r0 * 8 + threadIdx.x; i < r1 * 8; i += 256) {
      int r = i >> 3, pixel;
      const int ch = cb + 8 * (i & 7);
      if (r < pad * wp) {
        pixel = r;
      } else if ((r -= pad * wp) < pad * wp) {
        pixel = (h + pad) * wp + r;
      } else {
        r -= pad * wp;
        const int y = r / (2 * pad), q = r - y * 2 * pad;
        pixel = (y + pad) * wp + (q < pad ? q : w + q);
      }
      if (ch < c) store8(pixel, ch, zero4, zero4);
    }
  }
  // this thread's eight channels on the way out, and their GroupNorm scale / shift
  const int ch8 = 8 * (threadIdx.x & 7), oct = threadIdx.x & 7;
  float sc[8], sf[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) { sc[k] = 1.0f; sf[k] = 0.0f; }
  if (pre.stats != nullptr) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int ch = cb + ch8 + k;
      if (ch < c) {
        const float* st = pre.stats + (static_cast<long long>(n) * pre.groups + ch / (c / pre.groups)) * 2;
        const float mean = __ldg(st), inv = __ldg(st + 1);
        const float g = pre.gamma != nullptr ? __ldg(pre.gamma + ch) : 1.0f;
        const float b = (pre.gamma != nullptr && pre.beta != nullptr) ? __ldg(pre.beta + ch) : 0.0f;
        sc[k] = inv * g;
        sf[k] = b - mean * inv * g;
      }
    }
  }
  for (int t = t0; t < t1; ++t) {
    if (t + 1 < t1) issue(t + 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const float(*buf)[LR_TS] = tile[t & 1];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int sx = (threadIdx.x + 256 * i) >> 3, p = t * TP_X + sx;
      if (p < src_pixels && cb + ch8 < c) {
        const int col = 4 * ((sx >> 2) ^ oct) + (sx & 3);  // (ch8 + k) >> 3 = oct for every k
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = buf[ch8 + k][col];
        if (pre.stats != nullptr) {  // GroupNorm (+ SiLU) of the producer applied here
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            float r = fmaf(v[k], sc[k], sf[k]);
            if (pre.act == MIMIR_B200_ELT_SILU) r = r * __fdividef(1.0f, 1.0f + __expf(-r));
            v[k] = r;
          }
        }
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_pair(v[2 * j], v[2 * j + 1], f16, hi[j], lo[j]);
        const uint4 h4 = make_uint4(hi[0], hi[1], hi[2], hi[3]), l4 = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        const int y = p / sw_, px = p - y * sw_;
        if (UP) {
          const int o = (2 * y + pad) * wp + 2 * px + pad;
          store8(o, cb + ch8, h4, l4);
          store8(o + 1, cb + ch8, h4, l4);
          store8(o + wp, cb + ch8, h4, l4);
          store8(o + wp + 1, cb + ch8, h4, l4);
        } else {
          store8((y + pad) * wp + px + pad, cb + ch8, h4, l4);
        }
      }
    }
    __syncthreads();  // the buffer is refilled by the copy issued at the top of the next iteration
  }
}

// dst[pl][o][(kh*ks + kw)*ic + i] = split(w[o][i][kh][kw]); the padded tail of K is zero
__global__ void conv_weight_planes_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ dst, int oc, int ic, int ks,
                                          int kp, int planes, int f16, float scale) {
  const int k = ks * ks * ic;
  const long long total = static_cast<long long>(oc) * kp;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int o = static_cast<int>(i / kp), kk = static_cast<int>(i - static_cast<long long>(o) * kp);
    float v = 0.0f;
    if (kk < k) {
      const int t = kk / ic, ci = kk - t * ic;
      v = __ldg(w + (static_cast<long long>(o) * ic + ci) * ks * ks + t);
    }
    uint16_t hi, lo;
    split_one(v * scale, f16, hi, lo);
    uint16_t* d16 = reinterpret_cast<uint16_t*>(dst);
    d16[i] = hi;
    if (planes == 2) d16[i + total] = lo;
  }
}

}  // namespace

int launch_nchw_to_padded_nhwc_split(const float* x, __nv_bfloat16* dst, int batch, int c, int h, int w, int pad, int planes,
                                     cudaStream_t st, const PreNorm& pre, int up) {
  if (batch <= 0 || c <= 0 || h <= 0 || w <= 0 || pad < 0) return fail(MIMIR_B200_E_INVALID, "Conv2d: bad activation shape");
  if (up && ((h | w) & 1)) return fail(MIMIR_B200_E_INVALID, "Conv2d: an upsampled input needs even dimensions");
  const int hp = h + 2 * pad, wp = w + 2 * pad, sms = ctx().sm_count;
  if (batch > 65535 || static_cast<long long>(hp) * wp >= (1LL << 27)) return fail(MIMIR_B200_E_UNSUPPORTED, "Conv2d: image too large for the layout kernel");
  if ((c & 7) != 0 || (reinterpret_cast<uintptr_t>(dst) & 15) != 0) return fail(MIMIR_B200_E_INVALID, "Conv2d: bad operand plane layout");
  if (pre.stats != nullptr && (pre.groups <= 0 || c % pre.groups != 0)) return fail(MIMIR_B200_E_INVALID, "Conv2d: bad fused GroupNorm");
  const long long plane_stride = static_cast<long long>(batch) * hp * wp * c;
  const int src_pixels = up ? (h >> 1) * (w >> 1) : h * w, tiles = (src_pixels + TP_X - 1) / TP_X, cblocks = (c + TP_C - 1) / TP_C;
  // eight tiles to a CTA (long enough to stream), fewer while that leaves SMs without one
  int per = 8;
  while (per > 1 && static_cast<long long>((tiles + per - 1) / per) * cblocks * batch < 4LL * sms) per >>= 1;
  while ((tiles + per - 1) / per > 65535) per *= 2;
  const bool vec = (src_pixels & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  const int f16 = plane_format() == PLANES_F16;
  const dim3 grid(cblocks, (tiles + per - 1) / per, batch);
  auto kern = up ? (vec ? nchw_to_padded_nhwc_kernel<1, 1> : nchw_to_padded_nhwc_kernel<1, 0>)
                 : (vec ? nchw_to_padded_nhwc_kernel<0, 1> : nchw_to_padded_nhwc_kernel<0, 0>);
  kern<<<grid, 256, 0, st>>>(x, dst, c, h, w, pad, planes, plane_stride, pre, f16, per);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

int launch_conv_weight_planes(const float* w, __nv_bfloat16* dst, int oc, int ic, int ks, int planes, cudaStream_t st, float scale) {
  const int kp = round_up(ks * ks * ic, 64);
  const long long total = static_cast<long long>(oc) * kp;
  long long blocks = (total + 255) / 256;
  if (blocks > ctx().sm_count * 16) blocks = ctx().sm_count * 16;
  conv_weight_planes_kernel<<<static_cast<int>(blocks), 256, 0, st>>>(w, dst, oc, ic, ks, kp, planes, plane_format() == PLANES_F16, scale);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace mb

// ---------------------------------------------------------------------------------------------
// Convolutions with very few output channels (an RGB head: 128 -> 3): on the tensor core a 128-row weight tile would be
// all padding, and the layer is bound by reading its input once.  Direct fp32 convolution instead: a CTA owns a
// 128 x 8 pixel tile of one sample, stages the input tile (with its halo) for four channels at a time in shared memory,
// and every thread accumulates all output channels of its four pixels in the reference's order (ic, kh, kw ascending,
// Model.cpp:5005-5032) with FMAs.  No operand planes, no layout pass.
// ---------------------------------------------------------------------------------------------
namespace mb {
namespace {

constexpr int SO_TX = 32, SO_TY = 8, SO_PX = 4, SO_CC = 2, SO_NBUF = 2, SO_MAX_OC = 8, SO_MAX_KS = 7;
constexpr int so_rows(int oc) { return oc <= 4 ? 2 : 1; }  // output rows per thread: as many as the accumulators leave registers for

// A thread owns SO_PX consecutive pixels of R consecutive rows.  Every input row segment it reads from shared memory
// feeds all taps of up to R output rows, and the weights of one (channel, kernel row) come as broadcast 16-byte loads,
// so the FMA pipe and not the shared-memory pipe sets the pace.  The input tile and the weights of the next SO_CC
// channels arrive through cp.async (4-byte copies, plain zero stores for the padding ring) into the next slot of a
// ring of SO_NBUF buffers while the current channels are being consumed: one barrier per chunk, no registers spent on staging.
// Each output element accumulates over (ic, kh, kw) ascending: the reference's order (Model.cpp:5005-5032).
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))), "l"(gmem_src)
               : "memory");
}


// VEC = 0: tile rows of TW = 128 + KS - 1 pixels copied element by element, a pad word after every SO_PX pixels (the lanes of a
//          warp then read their segments SO_PX + 1 words apart: no bank conflicts).  Any image width and alignment.
// VEC = 1: image rows that are whole 16-byte chunks (width a multiple of 4, aligned base): a tile row is the 136 pixels from
//          x0 - 4, copied as 34 aligned 16-byte chunks (zero-filled outside the image); a lane reads its four pixels with one
//          128-bit load and takes the halo from its neighbours' registers.
template <int KS, int R, int VEC>
struct SmallOcGeom {
  static constexpr int PAD = KS / 2, TW = SO_TX * SO_PX + KS - 1, TH = SO_TY * R + KS - 1, SEG = SO_PX + KS - 1;
  static constexpr int TWV = SO_TX * SO_PX + 8, CHUNKS = TWV / 4;
  static constexpr int TWP = VEC ? TWV : TW + TW / SO_PX + 1;  // row stride in shared memory
  static constexpr int TILE = SO_CC * TH * TWP, WOFF = (SO_NBUF * TILE + 3) & ~3;
};

// CTAs of an SM that the compiler makes room for in registers (0: it chooses).  Four, in 64 registers, for forms of one to three channels with few
// spills, or none: the plain 1 x 1 to 3 channels on 16 x 128 of 256^2 298 us against 340, the normalising ones to 1 and 3 channels, with the
// statistics, 460 and 510 against 512 and 525 in 80 registers.  The 3 x 3 to 3 channels loses by it: normalising, 16 x 128 of 256^2 669 us against
// 644 with three, plain, 16 x 64 of 128^2 82 against 77 with one and one image of 256^2 64 against 59.  Element by element the
// compiler's own choice is better for 1 x 1 (17 x 64 of 361^2 to 8 channels 443 us against 493, 3 x 32 of 513^2 to one 94 against 97), 3 x 3 to 1, 2
// and 5 (17 x 64 of 361^2 473, 526 and 738 against 477, 557 and 786), 5 x 5 to one (601 against 613) and 7 x 7 to 3, 6 and 7 (16 x 64 of 128 x 126: 203, 305 and 348 against 206, 321 and 356), and one for the rest (3 x 3 and
// 7 x 7 to 8 channels 133 and 385 against 142 and 411, 5 x 5 234 against 244).
constexpr int so_ctas(int oc, int ks, int vec, int norm) {
  if (!vec) return ks == 1 || (ks == 3 && (oc <= 2 || oc == 5)) || (ks == 5 && oc == 1) || (ks == 7 && (oc == 3 || oc == 6 || oc == 7)) ? 0 : 1;
  if (oc == 3 && ks == 3) return norm ? 3 : 1;
  return oc <= 3 && ks <= 3 ? 4 : 1;
}

// NORM: x is the input of a GroupNorm (+ SiLU), which every thread applies to the chunks it has copied itself, between their arrival and the barrier
// that lets the others read them; the padding ring stays zero.  A tensor less written and read (conv_small_oc_pays_norm has the figures).
template <int OC, int KS, int R, int VEC, int NORM>
__global__ void __launch_bounds__(SO_TX * SO_TY, so_ctas(OC, KS, VEC, NORM)) conv_small_oc_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                       float* __restrict__ y, const float* __restrict__ residual, int ic,
                                                                       int h, int wd, int act, const float4* __restrict__ coef, int pre_silu) {
  static_assert(VEC || !NORM, "whole chunks");
  using G = SmallOcGeom<KS, R, VEC>;
  constexpr int PAD = G::PAD, TW = G::TW, TH = G::TH, TWP = G::TWP, TILE = G::TILE, SEG = G::SEG, KK = KS * KS;
  constexpr int WROW = (KS * OC + 3) & ~3;  // the weights of one (channel, kernel row) as [kw][o], padded to whole float4s
  constexpr int WCH = SO_CC * KS * WROW;
  extern __shared__ __align__(16) float so_smem[];  // [SO_NBUF][TILE] input tiles, then (16-byte aligned) [SO_NBUF][WCH] weights
  const int n = blockIdx.z;
  const int x0 = blockIdx.x * (SO_TX * SO_PX), y0 = blockIdx.y * (SO_TY * R);
  const int tx = threadIdx.x & (SO_TX - 1), ty = threadIdx.x / SO_TX;
  const float* xs = x + static_cast<long long>(n) * ic * h * wd;
  float acc[OC][R][SO_PX];
#pragma unroll
  for (int o = 0; o < OC; ++o)
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int q = 0; q < SO_PX; ++q) acc[o][j][q] = 0.0f;
  for (int i = threadIdx.x; i < SO_NBUF * WCH; i += SO_TX * SO_TY) so_smem[G::WOFF + i] = 0.0f;  // the float4 padding is read, never used
  __syncthreads();
  // a lane copies the same columns of every tile row: their offsets and bounds once per thread
  constexpr int NX = (TW + SO_TX - 1) / SO_TX;
  int xsrc[NX], xdst[NX];  // xsrc < 0: outside the image (or past the tile): a zero is stored, or nothing
#pragma unroll
  for (int k = 0; k < NX; ++k) {
    const int xx = tx + k * SO_TX, gx = x0 - PAD + xx;
    xdst[k] = xx < TW ? xx + xx / SO_PX : -1;
    xsrc[k] = (xx < TW && gx >= 0 && gx < wd) ? gx : -1;
  }
  // a thread copies the same chunks of every tile: their places once per thread (VEC)
  constexpr int CELLS = SO_CC * TH * G::CHUNKS, NC = VEC ? (CELLS + SO_TX * SO_TY - 1) / (SO_TX * SO_TY) : 1;
  int csrc[NC];  // within the first SO_CC channels; < 0: outside the image (a chunk is wholly inside or wholly outside)
  auto cell = [&](int k) { return static_cast<int>(threadIdx.x) + k * (SO_TX * SO_TY); };  // chunk `cell` of the tile, which has no padding
  static_assert(!VEC || TWP == 4 * G::CHUNKS, "chunks side by side");
  if (VEC) {
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const int idx = cell(k), row = idx / G::CHUNKS, ch = idx - row * G::CHUNKS;
      const int c = row / TH, yy = row - c * TH, gy = y0 + yy - PAD, gx = x0 - 4 + 4 * ch;
      csrc[k] = idx < CELLS && gy >= 0 && gy < h && gx >= 0 && gx < wd ? (c * h + gy) * wd + gx : -1;
    }
  }
  const int second = h * wd;  // csrc from here on: the second channel of a chunk of two
  static_assert(SO_CC == 2, "two channels at a time");
  auto fetch = [&](int c0, int buf) {
    const int cc = min(SO_CC, ic - c0);
    float* tile = so_smem + buf * TILE;
    if (VEC) {
      const float* src = xs + static_cast<long long>(c0) * second;
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        if (cell(k) >= CELLS) continue;
        const bool ok = csrc[k] >= 0 && (cc == SO_CC || csrc[k] < second);
        cp_async16_zfill(tile + 4 * cell(k), ok ? src + csrc[k] : xs, ok);
      }
    } else
    for (int row = ty; row < SO_CC * TH; row += SO_TY) {  // one warp per tile row
      const int c = row / TH, yy = row - c * TH, gy = y0 + yy - PAD;
      const bool row_ok = c < cc && gy >= 0 && gy < h;
      const float* src = xs + (static_cast<long long>(c0 + c) * h + gy) * wd;
      float* dst = tile + row * TWP;
#pragma unroll
      for (int k = 0; k < NX; ++k) {
        if (xdst[k] < 0) continue;
        if (row_ok && xsrc[k] >= 0) cp_async4(dst + xdst[k], src + xsrc[k]);
        else dst[xdst[k]] = 0.0f;
      }
    }
    float* wch = so_smem + G::WOFF + buf * WCH;
    for (int i = threadIdx.x; i < OC * cc * KK; i += SO_TX * SO_TY) {
      const int o = i / (cc * KK), r = i - o * cc * KK;  // OIHW: (c, kh, kw) of the chunk are contiguous per o
      const int c = r / KK, t = r - c * KK, kh = t / KS, kw = t - kh * KS;
      cp_async4(wch + (c * KS + kh) * WROW + kw * OC + o, w + (static_cast<long long>(o) * ic + c0) * KK + r);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto normalise = [&](int c0, int buf) {
    float* tile = so_smem + buf * TILE;
    const float4 k0 = __ldg(coef + static_cast<long long>(n) * ic + c0), k1 = __ldg(coef + static_cast<long long>(n) * ic + min(c0 + 1, ic - 1));
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      if (csrc[k] < 0) continue;
      const bool b = csrc[k] >= second;
      const float m = b ? k1.x : k0.x, a = b ? k1.y : k0.y, o = b ? k1.z : k0.z;
      float4 v = *reinterpret_cast<const float4*>(tile + 4 * cell(k));
      const unsigned long long m2 = pack2(-m, -m), a2 = pack2(a, a), o2 = pack2(o, o);
      unpack2(fma2(add2(pack2(v.x, v.y), m2), a2, o2), v.x, v.y);
      unpack2(fma2(add2(pack2(v.z, v.w), m2), a2, o2), v.z, v.w);
      if (pre_silu) { silu2(v.x, v.y); silu2(v.z, v.w); }
      *reinterpret_cast<float4*>(tile + 4 * cell(k)) = v;
    }
  };
  // SO_NBUF - 1 chunks in flight; one commit per iteration (an empty group past the end) keeps the wait count uniform
#pragma unroll
  for (int b = 0; b < SO_NBUF - 1; ++b) {
    if (b * SO_CC < ic) fetch(b * SO_CC, b);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int cur = 0;
  for (int c0 = 0; c0 < ic; c0 += SO_CC, cur = cur + 1 == SO_NBUF ? 0 : cur + 1) {
    const int cc = min(SO_CC, ic - c0);
    asm volatile("cp.async.wait_group %0;" ::"n"(SO_NBUF - 2) : "memory");
    if (NORM) normalise(c0, cur);
    __syncthreads();  // this chunk has landed for every thread, and everyone is done with the buffer refilled next
    if (c0 + (SO_NBUF - 1) * SO_CC < ic) fetch(c0 + (SO_NBUF - 1) * SO_CC, cur == 0 ? SO_NBUF - 1 : cur - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const float* tile = so_smem + cur * TILE;
    const float* wch = so_smem + G::WOFF + cur * WCH;
    for (int c = 0; c < cc; ++c) {
#pragma unroll
      for (int r = 0; r < R + KS - 1; ++r) {  // input rows ascending = kernel rows ascending for every output row
        float seg[SEG];
        if (VEC) {
          // pixels x0 + 4 tx .. + 3 sit at tile columns 4 tx + 4 .. 4 tx + 7; the PAD values either side come from the neighbour
          // lanes' vectors (from shared memory at the two ends of the warp)
          const float* rowp = tile + (c * TH + ty * R + r) * TWP + 4 * tx;
          const float4 m = *reinterpret_cast<const float4*>(rowp + 4);
          const float mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
          for (int i = 0; i < SO_PX; ++i) seg[PAD + i] = mv[i];
#pragma unroll
          for (int i = 0; i < PAD; ++i) {
            const float lft = __shfl_up_sync(0xffffffffu, mv[SO_PX - PAD + i], 1);
            const float rgt = __shfl_down_sync(0xffffffffu, mv[i], 1);
            seg[i] = tx == 0 ? rowp[4 - PAD + i] : lft;
            seg[PAD + SO_PX + i] = tx == SO_TX - 1 ? rowp[8 + i] : rgt;
          }
        } else {
          const float* row = tile + (c * TH + ty * R + r) * TWP + tx * (SO_PX + 1);
#pragma unroll
          for (int i = 0; i < SEG; ++i) seg[i] = row[i + i / SO_PX];
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int kh = r - j;
          if (kh < 0 || kh >= KS) continue;
          float wv[WROW];
          const float4* w4 = reinterpret_cast<const float4*>(wch + (c * KS + kh) * WROW);
#pragma unroll
          for (int v = 0; v < WROW / 4; ++v) {
            const float4 t = w4[v];
            wv[4 * v] = t.x, wv[4 * v + 1] = t.y, wv[4 * v + 2] = t.z, wv[4 * v + 3] = t.w;
          }
#pragma unroll
          for (int kw = 0; kw < KS; ++kw)
#pragma unroll
            for (int o = 0; o < OC; ++o)
#pragma unroll
              for (int q = 0; q < SO_PX; ++q) acc[o][j][q] = fmaf(seg[kw + q], wv[kw * OC + o], acc[o][j][q]);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int gy = y0 + ty * R + j;
    if (gy >= h) continue;
#pragma unroll
    for (int o = 0; o < OC; ++o) {
#pragma unroll
      for (int q = 0; q < SO_PX; ++q) {
        const int gx = x0 + tx * SO_PX + q;
        if (gx < wd) {
          const long long oi = ((static_cast<long long>(n) * OC + o) * h + gy) * wd + gx;
          float v = acc[o][j][q];
          if (act == MIMIR_B200_ELT_RELU) v = fmaxf(v, 0.0f);
          else if (act == MIMIR_B200_ELT_SILU) v = v * (1.0f / (1.0f + expf(-v)));
          if (residual != nullptr) v += __ldg(residual + oi);
          y[oi] = v;
        }
      }
    }
  }
}

template <int OC, int KS, int VEC, int NORM>
int launch_small_oc_v(const float* x, const float* w, float* y, const float* residual, int batch, int ic, int h, int wd, int act,
                      cudaStream_t st, const float4* coef, int pre_silu) {
  constexpr int R = so_rows(OC);
  using G = SmallOcGeom<KS, R, VEC>;
  constexpr int SMEM = (G::WOFF + SO_NBUF * SO_CC * KS * ((KS * OC + 3) & ~3)) * static_cast<int>(sizeof(float));
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(conv_small_oc_kernel<OC, KS, R, VEC, NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    return MIMIR_B200_OK;
  }));
  dim3 grid((wd + SO_TX * SO_PX - 1) / (SO_TX * SO_PX), (h + SO_TY * R - 1) / (SO_TY * R), batch);
  conv_small_oc_kernel<OC, KS, R, VEC, NORM><<<grid, SO_TX * SO_TY, SMEM, st>>>(x, w, y, residual, ic, h, wd, act, coef, pre_silu);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

bool small_oc_vec(int h, int wd) {
  static const bool off = [] { const char* e = getenv("MIMIR_B200_CONV_SMALL_OC_VEC"); return e && e[0] == '0'; }();
  return !off && (wd & 3) == 0 && static_cast<long long>(h) * wd * SO_CC <= 0x7fffffffLL;
}

template <int OC, int KS>
int launch_small_oc_k(const float* x, const float* w, float* y, const float* residual, int batch, int ic, int h, int wd, int act,
                      cudaStream_t st, const float4* coef, int pre_silu) {
  // whole 16-byte chunks per image row and an aligned base: the vector form (MIMIR_B200_CONV_SMALL_OC_VEC=0 turns it off)
  const bool vec = small_oc_vec(h, wd) && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  if (coef != nullptr) {
    if (!vec) return fail(MIMIR_B200_E_INVALID, "conv_small_oc: a normalised input comes in whole aligned chunks");
    return launch_small_oc_v<OC, KS, 1, 1>(x, w, y, residual, batch, ic, h, wd, act, st, coef, pre_silu);
  }
  if (vec) return launch_small_oc_v<OC, KS, 1, 0>(x, w, y, residual, batch, ic, h, wd, act, st, nullptr, 0);
  return launch_small_oc_v<OC, KS, 0, 0>(x, w, y, residual, batch, ic, h, wd, act, st, nullptr, 0);
}

template <int OC>
int launch_small_oc_t(const float* x, const float* w, float* y, const float* residual, int batch, int ic, int h, int wd, int ks, int pad,
                      int act, cudaStream_t st, const float4* coef, int pre_silu) {
  (void)pad;
  switch (ks) {
    case 1: return launch_small_oc_k<OC, 1>(x, w, y, residual, batch, ic, h, wd, act, st, coef, pre_silu);
    case 3: return launch_small_oc_k<OC, 3>(x, w, y, residual, batch, ic, h, wd, act, st, coef, pre_silu);
    case 5: return launch_small_oc_k<OC, 5>(x, w, y, residual, batch, ic, h, wd, act, st, coef, pre_silu);
    case 7: return launch_small_oc_k<OC, 7>(x, w, y, residual, batch, ic, h, wd, act, st, coef, pre_silu);
    default: return fail(MIMIR_B200_E_INVALID, "conv_small_oc: kernel size %d", ks);
  }
}

}  // namespace

bool conv_small_oc_supported(int oc, int ks, int stride, int pad, int h, int wd, int batch, int act) {
  static const bool off = [] { const char* e = getenv("MIMIR_B200_CONV_SMALL_OC"); return e && e[0] == '0'; }();
  return !off && oc >= 1 && oc <= SO_MAX_OC && stride == 1 && ks >= 1 && ks <= SO_MAX_KS && (ks & 1) == 1 && pad == ks / 2 && batch <= 65535 &&
         (h + SO_TY - 1) / SO_TY <= 65535 && (act == -1 || act == MIMIR_B200_ELT_RELU || act == MIMIR_B200_ELT_SILU) &&
         static_cast<long long>(h) * wd >= 4096;  // small images keep the tensor-core path (too few tiles to fill the SMs)
}

bool conv_small_oc_takes_norm(int h, int wd) { return small_oc_vec(h, wd); }

// Where that is the faster one.  The normalised tensor is not written and read again, but the convolution, which waits for its own instructions, takes
// longer: the tensor has to be several times L2 (384 MB), its statistics long rows (a CTA sweeps each), its kernel small.  To 3 channels,
// 3 x 3, GroupNorm apart and in here: 16 x 128 of 256^2 with 32 groups 703 and 660 us, 8 of them 369 and 363; but 16 x 128 of 128^2 208 and 228,
// 96 x 64 of 128^2 in rows of two channels 475 and 491, and to 8 channels with 7 x 7 2276 and 2337; to one
// channel with 1 x 1 256 MB are enough (21 x 96 of 192^2, 297 MB, 657 and 581).  With fewer rows than SMs, longer
// than registers, the GroupNorm that reads and writes is the slower one by far, and 96 MB or rows of 900 K values are enough: 3 x 128 of 256^2 (96 MB)
// 198 and 195 us, 4 x 64 of 364^2 237 and 192, 2 x 128 of 512^2 669 and 350, 1 x 128 of 256^2 in eight groups (1 M values) 163 and 155, in one
// 454 and 159; in 16 141 and 155.
bool conv_small_oc_pays_norm(int batch, int ic, int oc, int h, int wd, int ks, int groups) {
  if (!conv_small_oc_takes_norm(h, wd) || groups <= 0) return false;
  RowNormArgs r;
  r.rows = static_cast<long long>(batch) * groups; r.len = static_cast<long long>(ic / groups) * h * wd;
  const long long bytes = static_cast<long long>(batch) * ic * h * wd * 4;
  if (r.rows < ctx().sm_count) return bytes >= (32ll << 20) && !norm_rows_supported(r) && (bytes >= (96ll << 20) || r.len >= 900000);
  return bytes >= ((oc * ks * ks <= 8 ? 256ll : 384ll) << 20) && r.len >= 65536 && oc * ks * ks <= 80;
}

int launch_conv_small_oc(const float* x, const float* w, float* y, const float* residual, int batch, int ic, int oc, int h, int wd, int ks,
                         int pad, int act, cudaStream_t st, const float4* coef, int pre_silu) {
  switch (oc) {
    case 1: return launch_small_oc_t<1>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 2: return launch_small_oc_t<2>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 3: return launch_small_oc_t<3>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 4: return launch_small_oc_t<4>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 5: return launch_small_oc_t<5>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 6: return launch_small_oc_t<6>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 7: return launch_small_oc_t<7>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    case 8: return launch_small_oc_t<8>(x, w, y, residual, batch, ic, h, wd, ks, pad, act, st, coef, pre_silu);
    default: return fail(MIMIR_B200_E_INVALID, "conv_small_oc: %d output channels", oc);
  }
}

}  // namespace mb
