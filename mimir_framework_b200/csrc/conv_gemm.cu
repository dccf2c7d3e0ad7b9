// conv_gemm.cu — stride-1 "same" convolutions with ks >= 3 on large images, as an implicit GEMM over spatial tiles
// (the inline Conv2d case, Model.cpp:4897-5089).  Same operands (zero-padded NHWC planes, (tap, channel) weight planes), same
// products and epilogue as the shifted-GEMM form of gemm_sm100.cu.
//
// That form is bound by what an SM can take from L2: a tile of 256 pixels reads its activation block once per tap, nine times for
// a 3 x 3 kernel (80 bytes per cycle and SM on a 128 -> 128 layer in the two-MMA mode, where about 50 arrive; the tensor pipe
// was 48 to 54 % busy).  Here a tile is 16 x 16 pixels of one sample, and a K block of 32 or 64 channels brings the tile with its rows of
// halo, 16 x (16 + ks - 1) pixels, ONCE per kernel column: a vertical shift by one row is 16 pixels further into the same
// shared-memory tile, 16 x 64 or 128 bytes, a whole number of swizzle atoms, so the ks taps of a column are the same copy under ks
// descriptors.  Activation bytes from L2 fall to (16 + ks - 1) / (16 ks) of before (0.375 for 3 x 3).
//
//   warp 0     : TMA producer of activation tiles   (ring of A_STAGES, one per (BK channels, kernel column))
//   warp 1     : MMA issuer: weights are the M side (128 output channels), 256 pixels (or 128) the N side; two accumulators in TMEM
//   warps 2..9 : epilogue: 32 x 32 chunks turned around in shared memory so that a lane owns a pixel; NCHW stores
//   warp 10    : TMA producer of weight tiles       (ring of W_STAGES, one per tap and plane)
// Where a GroupNorm reads the result the epilogue leaves its moments behind (GN): a sweep over a tensor larger than L2 less, and the
// warps that take them have the time, as the MMAs of a K of 576 and more outlast the stores: 2 to 3 us of 110 to 450 on a launch, for
// sweeps of 7 to 89 us (UNet of 16 samples: 4167 -> 3945 us, conv stack 7159 -> 7055).
// Every wait is bounded, as in gemm_sm100.cu.
#include "common.h"
#include "epilogue.cuh"
#include "launch.cuh"
#include "planes.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

#include <cstdlib>

namespace mb {
namespace {

constexpr int CG_THREADS = 352;
constexpr int CG_N = 256;                      // pixels of a tile: 16 x 16 or, for 1 x 1 kernels, 256 of the flattened image; or half of that
constexpr int CG_M = 128;                      // output channels of a tile
constexpr int CG_EPI = 8 * 32 * 33 * 4;
constexpr int CG_COEF = 8 * 128 * 4;
constexpr int CG_MAX_RING = 16;
constexpr int CG_SMEM_MAX = 232448;

struct ConvGemmParams {
  int batch, oc, h, w, ks, cblocks;            // cblocks = channels / BK
  int px, tw_log, tiles_x, tiles_y, tiles_o, num_tiles;  // a tile has px pixels (256 or 128) and is 1 << tw_log of them wide
  int a_stages, a_stage_bytes, w_stages;
  const float* residual;
  int res_up;                                  // 1: the residual is [oc][h/2][w/2], a value for 2 x 2 pixels
  float* out;
  int activation;
  float acc_scale;
  int f16;
  float4* gn_part;                             // [sample][four channels][spatial tile x 2 halves] (mean, second moment about it, values, -)
  int* err_word;
};

// Sums over the warp of eight values a lane (recursive halving): lanes 4 g ... 4 g + 3 end with that of value g.
__device__ __forceinline__ float sum8(float (&a)[8], int lane) {
  int mask = 16;
#pragma unroll
  for (int half = 4; half >= 1; half >>= 1, mask >>= 1) {
    const bool upper = (lane & mask) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = upper ? a[i] : a[i + half], keep = upper ? a[i + half] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
    }
  }
  a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
  return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

// What only some forms need: an argument of its own (with these among ConvGemmParams the compiler took 168 registers for every form and the
// plain one lost 10 % of a 1 x 1 convolution)
struct ConvFormParams {
  int flat_pad, flat_w, flat_iw, flat_ih;      // CG_FLAT: the line of padded images flat_w wide, whose inside is flat_ih x flat_iw
  const float4* res_coef;                      // CG_RN: see GemmArgs
  int res_silu;
};

struct ConvTile { int oc0, n, y0, x0; };
__device__ __forceinline__ ConvTile conv_tile(const ConvGemmParams& p, int t) {  // output-channel tiles fastest: they share activations in L2
  ConvTile c;
  c.oc0 = (t % p.tiles_o) * CG_M;
  int s = t / p.tiles_o;
  c.x0 = (s % p.tiles_x) << p.tw_log;
  s /= p.tiles_x;
  c.y0 = (s % p.tiles_y) * (p.px >> p.tw_log);
  c.n = s / p.tiles_y;
  return c;
}

// BK: channels of a K block, 32 (64-byte swizzle rows) or 64 (128-byte rows)
// FORM: what the epilogue does beside, each in a form of its own (the plain one runs in 128 registers, which the others leave)
enum : int { CG_PLAIN = 0, CG_GN = 1 /* moments of the result for the GroupNorm that reads it */, CG_RN = 2 /* the residual is a GroupNorm's input */,
             CG_FLAT = 4 /* the line of a padded image */ };
template <int AP, int WP, int BK, int FORM>
__global__ void __launch_bounds__(CG_THREADS, 1)
conv_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const ConvGemmParams p,
                 const ConvFormParams f) {
  constexpr int W_TILE = CG_M * BK * 2;
  constexpr bool GN = (FORM & CG_GN) != 0, RN = (FORM & CG_RN) != 0, FLAT = (FORM & CG_FLAT) != 0;
  extern __shared__ __align__(1024) uint8_t cg_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(cg_smem_raw) + 1023) & ~uintptr_t(1023));
  const int a_plane = p.a_stage_bytes / AP;                                   // halo tile of one plane
  uint8_t* a_ring = smem;
  uint8_t* w_ring = smem + p.a_stages * p.a_stage_bytes;
  float* epi = reinterpret_cast<float*>(w_ring + p.w_stages * W_TILE);
  __shared__ uint64_t a_full[CG_MAX_RING], a_empty[CG_MAX_RING], w_full[CG_MAX_RING], w_empty[CG_MAX_RING], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int warp = warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.a_stages; ++s) { mbar_init(&a_full[s], 1); mbar_init(&a_empty[s], 1); }
    for (int s = 0; s < p.w_stages; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 8); }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_wait();

  if (warp == 0) {
    const bool one = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = static_cast<int>(blockIdx.x); t < p.num_tiles && ok; t += static_cast<int>(gridDim.x)) {
      const ConvTile c = conv_tile(p, t);
      for (int cb = 0; cb < p.cblocks && ok; ++cb)
        for (int kw = 0; kw < p.ks; ++kw) {
          if (!mbar_wait_warp(&a_empty[stage], phase ^ 1, &abort_flag, p.err_word, 51)) { ok = false; break; }
          if (one) {
            uint8_t* dst = a_ring + stage * p.a_stage_bytes;
            mbar_expect_tx(&a_full[stage], static_cast<uint32_t>(p.a_stage_bytes));
            tma_load_5d(dst, &map_a, &a_full[stage], cb * BK, c.x0 + kw, c.y0, c.n, 0);  // (padded coordinates: the halo starts at y0)
            if (AP == 2) tma_load_5d(dst + a_plane, &map_a, &a_full[stage], cb * BK, c.x0 + kw, c.y0, c.n, 1);
          }
          __syncwarp();
          if (++stage == p.a_stages) { stage = 0; phase ^= 1; }
        }
    }
    for (int s = 0; s < p.a_stages; ++s) {  // drain: no copy may be in flight when the CTA exits
      if (!mbar_wait_warp(&a_empty[stage], phase ^ 1, &abort_flag, p.err_word, 52)) break;
      if (++stage == p.a_stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 10) {
    const bool one = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = static_cast<int>(blockIdx.x); t < p.num_tiles && ok; t += static_cast<int>(gridDim.x)) {
      const int oc0 = (t % p.tiles_o) * CG_M;
      for (int cb = 0; cb < p.cblocks && ok; ++cb)
        for (int kw = 0; kw < p.ks && ok; ++kw)
          for (int kh = 0; kh < p.ks; ++kh) {
            const int col = ((kh * p.ks + kw) * p.cblocks + cb) * BK;
            for (int plane = 0; plane < WP && ok; ++plane) {  // a ring slot per plane
              if (!mbar_wait_warp(&w_empty[stage], phase ^ 1, &abort_flag, p.err_word, 53)) { ok = false; break; }
              if (one) {
                mbar_expect_tx(&w_full[stage], W_TILE);
                tma_load_3d(w_ring + stage * W_TILE, &map_w, &w_full[stage], col, oc0, plane);
              }
              __syncwarp();
              if (++stage == p.w_stages) { stage = 0; phase ^= 1; }
            }
            if (!ok) break;
          }
    }
    for (int s = 0; s < p.w_stages; ++s) {
      if (!mbar_wait_warp(&w_empty[stage], phase ^ 1, &abort_flag, p.err_word, 54)) break;
      if (++stage == p.w_stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    const bool one = elect_one();
    const uint32_t idesc = make_idesc(CG_M, p.px, p.f16);
    int as = 0, ws = 0, acc = 0;
    uint32_t aph = 0, wph = 0, acc_phase = 0;
    bool ok = true, w_ready = false;
    for (int t = static_cast<int>(blockIdx.x); t < p.num_tiles && ok; t += static_cast<int>(gridDim.x)) {
      if (!mbar_wait_warp(&acc_empty[acc], acc_phase ^ 1, &abort_flag, p.err_word, 55)) break;
      tcgen05_fence_after();
      const uint32_t d = tmem + static_cast<uint32_t>(acc * CG_N);
      bool first = true;
      for (int b = 0; b < p.cblocks * p.ks && ok; ++b) {  // (BK channels, kernel column)
        if (!mbar_wait_warp(&a_full[as], aph, &abort_flag, p.err_word, 56)) { ok = false; break; }
        const uint64_t da0 = make_smem_desc(smem_u32(a_ring + as * p.a_stage_bytes), BK * 2);
        for (int kh = 0; kh < p.ks && ok; ++kh) {
          // kh rows further down: tile width x 2 BK bytes, in the descriptor's address field (16 bytes)
          const uint64_t da = da0 + static_cast<uint64_t>((kh << p.tw_log) * (BK / 8)), da_lo = da + static_cast<uint64_t>(a_plane >> 4);
#pragma unroll
          for (int plane = 0; plane < WP; ++plane) {  // of the weights; their lo plane meets the activations' hi plane only
            if (!__all_sync(0xffffffffu, w_ready) && !mbar_wait_warp(&w_full[ws], wph, &abort_flag, p.err_word, 57)) { ok = false; break; }
            tcgen05_fence_after();
            const uint64_t dw = make_smem_desc(smem_u32(w_ring + ws * W_TILE), BK * 2);
            uint64_t* w_done = &w_empty[ws];
            if (++ws == p.w_stages) { ws = 0; wph ^= 1; }
            w_ready = mbar_test(&w_full[ws], wph);
            if (one) {
#pragma unroll
              for (int k = 0; k < BK / 16; ++k) {
                umma_bf16(d, dw + 2 * k, da + 2 * k, idesc, (first && k == 0) ? 0u : 1u);
                if (AP == 2 && plane == 0) umma_bf16(d, dw + 2 * k, da_lo + 2 * k, idesc, 1u);
              }
              umma_commit(w_done);
              if (kh + 1 == p.ks && plane + 1 == WP) umma_commit(&a_empty[as]);
            }
            first = false;
            __syncwarp();
          }
        }
        if (++as == p.a_stages) { as = 0; aph ^= 1; }
      }
      if (!ok) break;
      if (one) umma_commit(&acc_full[acc]);
      __syncwarp();
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  } else {
    // epilogue: TMEM lane = output channel, column = pixel (16 to a row)
    const int ew = warp - 2, quad = warp & 3, half = ew >> 2;
    float* tbuf = epi + ew * (32 * 33);
    float* coef = epi + CG_EPI / 4 + ew * 128;  // RN: -mean, gamma / std and beta of this warp's 32 channels, each in a row, for pairs of channels
    const int chunks = p.px / 64;  // of 32 pixels, in each half of the tile
    const long long hw = FLAT ? static_cast<long long>(f.flat_ih) * f.flat_iw : static_cast<long long>(p.h) * p.w;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = static_cast<int>(blockIdx.x); t < p.num_tiles; t += static_cast<int>(gridDim.x)) {
      const ConvTile c = conv_tile(p, t);
      const int oc0 = c.oc0 + quad * 32, nch = p.oc - oc0;
      // chunk ci of this warp: 32 consecutive pixels of the tile
      auto place = [&](int ci, bool& in, long long& o0) {
        const int px = (half * chunks + ci) * 32 + lane, y = c.y0 + (px >> p.tw_log), x = c.x0 + (px & ((1 << p.tw_log) - 1));
        in = y < p.h && x < p.w;
        o0 = (static_cast<long long>(c.n) * p.oc + oc0) * hw + static_cast<long long>(y) * p.w + x;
        if (FLAT) {
          const int iy = x / f.flat_w - f.flat_pad, ix = x % f.flat_w - f.flat_pad;
          in = static_cast<unsigned>(iy) < static_cast<unsigned>(f.flat_ih) && static_cast<unsigned>(ix) < static_cast<unsigned>(f.flat_iw);
          o0 = (static_cast<long long>(c.n) * p.oc + oc0) * hw + static_cast<long long>(iy) * f.flat_iw + ix;
        }
      };
      // The residual of a chunk is requested one chunk ahead, the first one's before the accumulators are waited for: a 1 x 1 skip
      // layer reads and writes more than it multiplies, and its loads would each wait a full memory latency.
      float q[32];
      auto request = [&](int ci) {
        bool in;
        long long o0, step = hw;
        place(ci, in, o0);
        // an upsampled residual: the two rows of a chunk read eight neighbours each, one sector, of the half-size image
        if (p.res_up) {
          const int px = (half * chunks + ci) * 32 + lane, y = c.y0 + (px >> p.tw_log), x = c.x0 + (px & ((1 << p.tw_log) - 1));
          step = hw >> 2;
          o0 = (static_cast<long long>(c.n) * p.oc + oc0) * step + static_cast<long long>(y >> 1) * (p.w >> 1) + (x >> 1);
        }
        if (in) {
#pragma unroll
          for (int j = 0; j < 32; ++j) q[j] = j < nch ? __ldg(p.residual + o0 + j * step) : 0.0f;
        }
      };
      if (p.residual != nullptr && nch > 0) request(0);
      if (RN && nch > 0) {
        const float4 k = __ldg(f.res_coef + static_cast<long long>(c.n) * p.oc + oc0 + lane);
        __syncwarp();
        coef[lane] = -k.x;
        coef[32 + lane] = k.y;
        coef[64 + lane] = k.z;
        __syncwarp();
      }
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&acc_full[acc], acc_phase, &abort_flag, p.err_word, 58) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      while (!mbar_try_wait(&acc_full[acc], acc_phase)) {}  // completes at once: lane 0 saw the phase
      tcgen05_fence_after();
      const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(acc * CG_N);
      // A lane's own moments of each four channels: sums about the first value it met, so that a large mean costs nothing
      float ref[8], s1[8], s2[8];
      int pixels = 0;
      if (GN) {
#pragma unroll
        for (int g = 0; g < 8; ++g) ref[g] = s1[g] = s2[g] = 0.0f;
      }
      if (nch > 0) {
#pragma unroll 1
        for (int ci = 0; ci < chunks; ++ci) {
          if (c.y0 + (((half * chunks + ci) * 32) >> p.tw_log) >= p.h) break;  // warp-uniform
          bool in;
          long long o0;
          place(ci, in, o0);
          float v[32];
          tmem_ld_32x32(taddr + (half * chunks + ci) * 32, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) tbuf[j * 33 + lane] = __fmul_rn(v[j], p.acc_scale);  // [pixel][channel]
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = tbuf[lane * 33 + j];
          __syncwarp();
          if (p.activation != -1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], p.activation);
          }
          if (p.residual != nullptr) {
            if (RN) {
#pragma unroll
              for (int j = 0; j < 32; j += 4) {  // (the same for every lane)
                const float4 m = *reinterpret_cast<const float4*>(coef + j), a = *reinterpret_cast<const float4*>(coef + 32 + j),
                             o = *reinterpret_cast<const float4*>(coef + 64 + j);
                unpack2(fma2(add2(pack2(q[j], q[j + 1]), pack2(m.x, m.y)), pack2(a.x, a.y), pack2(o.x, o.y)), q[j], q[j + 1]);
                unpack2(fma2(add2(pack2(q[j + 2], q[j + 3]), pack2(m.z, m.w)), pack2(a.z, a.w), pack2(o.z, o.w)), q[j + 2], q[j + 3]);
              }
              if (f.res_silu) {
#pragma unroll
                for (int j = 0; j < 32; j += 2) silu2(q[j], q[j + 1]);
              }
#pragma unroll
              for (int j = 0; j < 32; j += 2) unpack2(add2(pack2(v[j], v[j + 1]), pack2(q[j], q[j + 1])), v[j], v[j + 1]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += q[j];
            }
            if (ci + 1 < chunks) request(ci + 1);
          }
          if (in) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < nch) p.out[o0 + j * hw] = v[j];
          }
          if (GN && in) {
            if (pixels++ == 0) {
#pragma unroll
              for (int g = 0; g < 8; ++g) ref[g] = v[4 * g];
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float e = v[j] - ref[j >> 2];
              s1[j >> 2] += e;
              s2[j >> 2] = fmaf(e, e, s2[j >> 2]);
            }
          }
        }
        if (GN) {
          // the lanes' moments meet (T. F. Chan, G. H. Golub, R. J. LeVeque 1979); a second moment beyond fp32 stays infinite
          const float n = 4.0f * pixels, inv = pixels > 0 ? 1.0f / n : 0.0f;
          const float total = 4.0f * __reduce_add_sync(0xffffffffu, pixels), inv_total = total > 0.0f ? 1.0f / total : 0.0f;
          float a[8];
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float d = s1[g] * inv;
            s2[g] = s2[g] < INFINITY ? fmaxf(s2[g] - s1[g] * d, 0.0f) : s2[g];
            ref[g] += d;  // the lane's mean
            a[g] = n * ref[g];
          }
          const float mean = sum8(a, lane) * inv_total;
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const float d = ref[g] - __shfl_sync(0xffffffffu, mean, 4 * g);
            a[g] = fmaf(n * d, d, s2[g]);
          }
          const float m2 = sum8(a, lane);
          if ((lane & 3) == 0) {
            const int spatial = p.tiles_x * p.tiles_y, place = (t / p.tiles_o) % spatial * 2 + half;
            p.gn_part[(static_cast<long long>(c.n) * (p.oc >> 2) + (oc0 >> 2) + (lane >> 2)) * (2 * spatial) + place] = make_float4(mean, m2, total, 0.0f);
          }
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Image and tile shape of a launch.  A 1 x 1 kernel sees the image as one line (tiles of 256 consecutive pixels, whole 128-byte
// lines in every channel plane; the line of the padded image where that is what the planes hold: with 16-pixel rows its scattered 64-byte stores held DRAM at 4 TB/s).  Otherwise 16 x 16 (32 x 8 where
// the width allows whole lines measured the same: there the MMAs, not the stores, set the pace).
struct ConvShape { int h, w, tw_log, tiles_x, tiles_y; };
ConvShape conv_shape(const GemmArgs& g, int px) {
  ConvShape s{g.conv_h, g.conv_w, 4, 0, 0};
  if (g.conv_ks == 1) { s.w = (g.conv_h + 2 * g.conv_src_pad) * (g.conv_w + 2 * g.conv_src_pad); s.h = 1; s.tw_log = px == CG_N ? 8 : 7; }
  const int tw = 1 << s.tw_log, th = px >> s.tw_log;
  s.tiles_x = (s.w + tw - 1) / tw;
  s.tiles_y = (s.h + th - 1) / th;
  return s;
}

long long tiles_of(const GemmArgs& g, int px) {
  const ConvShape sh = conv_shape(g, px);
  const long long per = static_cast<long long>(g.conv_h + 2 * g.conv_pad) * (g.conv_w + 2 * g.conv_pad);
  return g.m / per * sh.tiles_y * sh.tiles_x * ((g.n + CG_M - 1) / CG_M);
}

// Blocks of 64 channels where two activation tiles and three weight planes of them fit the ring: a 128-byte row costs the copy engine
// little more than a 64-byte one, and with 448 rows to a tap and 32 channels (3 x 3, four planes) those set the pace: a tile of 128 pixels
// took 676 cycles for 384 of MMAs.  16 x 512 -> 512 on 16^2: 62.8 -> 53.0 us, with two products 52.2 -> 42.4; 3 x 256 -> 256 on 56^2, tiles
// of 256 pixels: 45.2 -> 44.3.  A normalised residual's coefficients leave the 3 x 3 form of 256 pixels and four planes a slot short, which then takes
// blocks of 32: 16 x 256 -> 256 on 64^2 with its producer 427 -> 388 us (405 with the GroupNorm apart), 512 -> 256 830 -> 747 (763).
bool conv_wide_blocks(const GemmArgs& g, int px) {
  const char* e = getenv("MIMIR_B200_CONV_BK");  // "32": never
  if (g.conv_c % 64 != 0 || (e && atoi(e) == 32)) return false;
  const ConvShape sh = conv_shape(g, px);
  const int tw = 1 << sh.tw_log, rows = (px >> sh.tw_log) + g.conv_ks - 1;
  return 2 * g.a_planes * tw * rows * 128 + 3 * CG_M * 128 <= CG_SMEM_MAX - CG_EPI - (g.res_coef != nullptr ? CG_COEF : 0) - 2048;
}

// Estimated SM cycles of a launch and the tile it takes: within 5 % of 50 measured launches, K = 64 ... 4608.  Tiles of 128 pixels (half of
// the accumulator's columns: the same sums in the same order, bit for bit) where 256 leave SMs without one: they load the weights whole, so
// that one takes 0.64 of a tile's MMA time with three MMAs per product and 0.68 with two (0.83 and 0.94 in blocks of 32 channels), and 2800
// cycles less beside it.  16 x 512 -> 512 on 16^2, 64 tiles: 78.1 -> 53.0 us; 4 x 128 -> 128 on 63^2, 64 tiles: 30.9 -> 23.2; 8 x 64 -> 64
// on 58^2, 128 tiles: stays (19.0, 22.4 in 256).
double conv_cycles(const GemmArgs& g, int* px) {
  const int sms = ctx().sm_count, products = g.a_planes + g.w_planes - 1;
  const bool wide = conv_wide_blocks(g, CG_N / 2);
  const double mma = 1.15 * g.k / 16.0 * products * 128.0;
  const double part = (products == 3 ? (wide ? 0.64 : 0.83) : products == 2 ? (wide ? 0.68 : 0.94) : (wide ? 0.8 : 1.0)) * mma;
  const double whole = 17400.0 + static_cast<double>((tiles_of(g, CG_N) + sms - 1) / sms) * (mma > 4500.0 ? mma : 4500.0);
  const double half = 14600.0 + static_cast<double>((tiles_of(g, CG_N / 2) + sms - 1) / sms) * (part > 2800.0 ? part : 2800.0);
  const char* force = getenv("MIMIR_B200_CONV_PX");  // "128", "256": always
  *px = force && (atoi(force) == CG_N || atoi(force) == CG_N / 2) ? atoi(force) : half < whole ? CG_N / 2 : CG_N;
  return *px == CG_N ? whole : half;
}

// (mean, 1 / std) of one (sample, group) from the tiles' moments, a CTA each, in double and in an order that does not change.  (A warp each took
// 14 us for the 512 x 512 entries of 16 images of 256^2.)
__global__ void __launch_bounds__(128) conv_gn_stats_kernel(const float4* __restrict__ part, float* __restrict__ stats, int entries, float eps) {
  __shared__ double sh[4][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double n = 0.0, mean = 0.0, m2 = 0.0;
  auto merge = [&](double nb, double mb, double m2b) {
    if (nb <= 0.0) return;
    const double nt = n + nb, d = mb - mean, f = nb / nt;
    mean += d * f;
    m2 += m2b + d * d * n * f;
    n = nt;
  };
  const float4* e = part + static_cast<long long>(blockIdx.x) * entries;
  for (int i = threadIdx.x; i < entries; i += 128) {
    const float4 q = __ldg(e + i);
    merge(q.z, q.x, q.y);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const double nb = __shfl_down_sync(0xffffffffu, n, d), mb = __shfl_down_sync(0xffffffffu, mean, d), m2b = __shfl_down_sync(0xffffffffu, m2, d);
    merge(nb, mb, m2b);  // (lanes past the end merge what nobody reads)
  }
  if (lane == 0) { sh[warp][0] = n; sh[warp][1] = mean; sh[warp][2] = m2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w) merge(sh[w][0], sh[w][1], sh[w][2]);
    stats[2 * blockIdx.x] = static_cast<float>(mean);
    stats[2 * blockIdx.x + 1] = 1.0f / sqrtf(static_cast<float>(n > 0.0 ? m2 / n : 0.0) + eps);
  }
}

template <int AP, int WP, int BK, int FORM>
int launch_conv_t(const GemmArgs& g, cudaStream_t st) {
  const int ks = g.conv_ks, pad = g.conv_pad;
  ConvGemmParams p;
  p.batch = g.m / ((g.conv_h + 2 * pad) * (g.conv_w + 2 * pad));
  conv_cycles(g, &p.px);
  const ConvShape sh = conv_shape(g, p.px);
  const int hp = sh.h + 2 * pad, wp = sh.w + 2 * pad, tw = 1 << sh.tw_log, th = p.px >> sh.tw_log;
  p.oc = g.n; p.h = sh.h; p.w = sh.w; p.ks = ks; p.cblocks = g.conv_c / BK;
  p.tw_log = sh.tw_log;
  p.tiles_x = sh.tiles_x; p.tiles_y = sh.tiles_y;
  p.tiles_o = (p.oc + CG_M - 1) / CG_M;
  p.num_tiles = p.batch * p.tiles_y * p.tiles_x * p.tiles_o;
  const int rows = th + ks - 1;
  p.a_stage_bytes = AP * tw * rows * BK * 2;
  const int ring = CG_SMEM_MAX - CG_EPI - (FORM & CG_RN ? CG_COEF : 0) - 1024 - 1024;  // (less the barriers)
  p.a_stages = 3;
  p.w_stages = (ring - p.a_stages * p.a_stage_bytes) / (CG_M * BK * 2);
  if (p.w_stages < 3 * WP) {
    p.a_stages = 2;
    p.w_stages = (ring - p.a_stages * p.a_stage_bytes) / (CG_M * BK * 2);
  }
  if (p.w_stages > CG_MAX_RING) p.w_stages = CG_MAX_RING;
  p.residual = g.residual; p.res_up = g.residual != nullptr && g.residual_up ? 1 : 0; p.out = g.out_f32; p.activation = g.activation;
  p.acc_scale = gemm_acc_scale(g);
  p.f16 = plane_format() == PLANES_F16 ? 1 : 0;
  p.gn_part = g.gn_part;
  const ConvFormParams f{g.conv_src_pad, g.conv_w + 2 * g.conv_src_pad, g.conv_w, g.conv_h, g.res_coef, g.res_act == MIMIR_B200_ELT_SILU ? 1 : 0};
  p.err_word = ctx().dev_error_word;
  CUtensorMap map_a, map_w;
  MB_TRY(make_image_map(&map_a, g.a, AP, p.batch, hp, wp, g.conv_c, BK, tw, rows));
  MB_TRY(make_plane_map(&map_w, g.w, WP, g.n, round_up(g.k, 64), BK, CG_M));
  const size_t smem = static_cast<size_t>(p.a_stages) * p.a_stage_bytes + static_cast<size_t>(p.w_stages) * (CG_M * BK * 2) + CG_EPI + (FORM & CG_RN ? CG_COEF : 0) + 1024;
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(conv_gemm_kernel<AP, WP, BK, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, CG_SMEM_MAX - 1024));
    return MIMIR_B200_OK;
  }));
  const int sms = ctx().sm_count;
  GemmProfile prof(st);
  MB_TRY(prof.begin());
  MB_TRY(launch_pdl(conv_gemm_kernel<AP, WP, BK, FORM>, dim3(static_cast<unsigned>(p.num_tiles < sms ? p.num_tiles : sms)), dim3(CG_THREADS), smem, st, 1, map_a, map_w, p, f));
  MB_TRY(prof.end());
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace

long long conv_gemm_tiles(const GemmArgs& g) { return tiles_of(g, CG_N); }

double conv_gemm_cycles(const GemmArgs& g) {
  constexpr double never = 1e30;
  const char* e = getenv("MIMIR_B200_CONV_SPATIAL");  // "0": never, "1": wherever the form allows
  if (e && e[0] == '0') return never;
  if (g.conv_ks < 1 || g.conv_ks > 7 || g.conv_c % 32 != 0 || g.bias != nullptr || g.out_f32 == nullptr || g.out_split != nullptr)
    return never;
  if (!(g.a_planes == 2 || g.w_planes == 1)) return never;
  if (e && e[0] == '1') return 0.0;
  // 1 x 1 (and im2col rows): nothing to share between taps; long K is better off in CTA pairs (K = 4608, 512 channels: 170 against
  // 111 us), short K is bound by its stores (K = 192, 64 channels: 139 against 247 us)
  if (g.conv_ks == 1 && g.conv_c > 1024) return never;
  int px;
  return conv_cycles(g, &px);
}

// A 1 x 1 convolution on planes that have a ring of `ring` pixels: the layout pass that it saves grows with the input, what the ring costs (tiles
// of it, stores that cross lines) with the output and the ring.  Two convolutions of one tensor, planes laid out twice and once: 64 x 64 -> 64
// of 64^2 245 and 231 us, 128 -> 256 of 56^2 627 and 618, 256 -> 256 572 and 548, 12 x 256 -> 256 of 78^2 372 and 356; but 64 -> 256 of 64^2 555 and
// 562, 512 -> 1024 of 32^2 (a ring of 13 %) 1809 and 1827, 256 -> 512 of 48^2 (9 %) 322 and 327 (64 -> 64 of 40^2, 10 %, 128 and 125), 64 -> 256 of
// 64^2 with a ring of two (13 %) 802 and 827, and, where the ring is a third
// wave of half tiles to two, 4 x 64 -> 128 of 96^2 61.0 and 67.3, a fifth to four 6 x 64 -> 64 of 112^2 84.6 and 86.7 (with half as many
// outputs as inputs a third more waves pay: 10 x 256 -> 64 of 104^2 542 and 516, 19 x 256 -> 96 of 54^2 200 and 180).  An epilogue that normalises
// the residual hides both (6 x 128 -> 128 of 112^2 128 and 118, 4 x 64 -> 128 of 96^2 63.0 and 63.5, 64 x 64 -> 256 of 64^2 398 and 399), and where
// the image's channel planes do not start on lines the stores cross them in any case and the layout pass is the slower one (64 x 64 -> 256 of 63^2 640
// and 616, 51 x 256 -> 256 of 33^2, 13 %, 368 and 332, 64 x 128 -> 64 of 37^2 with a ring of two, 23 %, 281 and 265; of 33^2, 25 %, 197 and 203).
bool conv_gemm_ring_pays(const GemmArgs& g, int ring, bool normed_residual) {
  const long long pixels = static_cast<long long>(g.conv_h) * g.conv_w;
  const bool crossing = pixels % 32 != 0;
  const long long widest = crossing ? 123 : normed_residual || g.n <= 256 ? 111 : 108;  // per cent
  if (100ll * (g.conv_h + 2 * ring) * (g.conv_w + 2 * ring) > widest * pixels) return false;
  if (normed_residual) return true;
  GemmArgs q = g;
  q.conv_src_pad = ring;
  auto waves = [](const GemmArgs& a) {
    int px;
    conv_cycles(a, &px);
    return (tiles_of(a, px) + ctx().sm_count - 1) / ctx().sm_count * (px == CG_N ? 2 : 1);  // of half tiles
  };
  const long long before = waves(g), after = waves(q);
  if (2 * g.n <= g.conv_c) return 3 * after <= 4 * before;
  return crossing ? 4 * after <= 5 * before : g.n <= 2 * g.conv_c && 6 * after <= 7 * before;
}

size_t conv_gemm_gn_bytes(const GemmArgs& g) {
  const ConvShape a = conv_shape(g, CG_N), b = conv_shape(g, CG_N / 2);
  const long long per = static_cast<long long>(g.conv_h + 2 * g.conv_pad) * (g.conv_w + 2 * g.conv_pad);
  const long long tiles = static_cast<long long>(a.tiles_x) * a.tiles_y, halves = static_cast<long long>(b.tiles_x) * b.tiles_y;
  return static_cast<size_t>(g.m / per * (g.n / 4) * 2 * (tiles > halves ? tiles : halves)) * sizeof(float4);
}

int launch_conv_gn_stats(const GemmArgs& g, float* stats, int groups, float eps, cudaStream_t st) {
  int px;
  conv_cycles(g, &px);
  const ConvShape sh = conv_shape(g, px);
  const int batch = g.m / ((g.conv_h + 2 * g.conv_pad) * (g.conv_w + 2 * g.conv_pad)), slabs = batch * groups;
  return launch_merge_moments(g.gn_part, stats, slabs, g.n / groups / 4 * 2 * sh.tiles_x * sh.tiles_y, eps, st);
}

int launch_merge_moments(const float4* part, float* stats, int rows, int entries, float eps, cudaStream_t st) {
  conv_gn_stats_kernel<<<rows, 128, 0, st>>>(part, stats, entries, eps);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

template <int AP, int WP>
int launch_conv_planes(const GemmArgs& g, bool wide, cudaStream_t st) {
  const int form = (g.gn_part != nullptr ? CG_GN : 0) | (g.res_coef != nullptr ? CG_RN : 0) | (g.conv_src_pad > 0 ? CG_FLAT : 0);
  if ((form & (CG_GN | CG_RN)) != 0 && g.n % 32 != 0) return fail(MIMIR_B200_E_INVALID, "conv: this form needs output channels in whole chunks of 32");
  switch (form) {
    case CG_PLAIN: return wide ? launch_conv_t<AP, WP, 64, CG_PLAIN>(g, st) : launch_conv_t<AP, WP, 32, CG_PLAIN>(g, st);
    case CG_GN: return wide ? launch_conv_t<AP, WP, 64, CG_GN>(g, st) : launch_conv_t<AP, WP, 32, CG_GN>(g, st);
    case CG_RN: return wide ? launch_conv_t<AP, WP, 64, CG_RN>(g, st) : launch_conv_t<AP, WP, 32, CG_RN>(g, st);
    case CG_FLAT: return wide ? launch_conv_t<AP, WP, 64, CG_FLAT>(g, st) : launch_conv_t<AP, WP, 32, CG_FLAT>(g, st);
    case CG_RN | CG_FLAT: return wide ? launch_conv_t<AP, WP, 64, CG_RN | CG_FLAT>(g, st) : launch_conv_t<AP, WP, 32, CG_RN | CG_FLAT>(g, st);
    default: return fail(MIMIR_B200_E_INVALID, "conv: no such form of the epilogue");
  }
}

int launch_conv_gemm(const GemmArgs& g, cudaStream_t st) {
  int px;
  conv_cycles(g, &px);
  const bool wide = conv_wide_blocks(g, px);
  if (g.a_planes == 2 && g.w_planes == 2) return launch_conv_planes<2, 2>(g, wide, st);
  if (g.a_planes == 2 && g.w_planes == 1) return launch_conv_planes<2, 1>(g, wide, st);
  if (g.a_planes == 1 && g.w_planes == 1) return launch_conv_planes<1, 1>(g, wide, st);
  return fail(MIMIR_B200_E_INVALID, "conv: %d activation and %d weight planes", g.a_planes, g.w_planes);
}

}  // namespace mb
