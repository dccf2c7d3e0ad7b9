// gemm_sm100.cu — the contraction kernel every dense layer funnels into (Linear, the attention
// projections, Conv2d lowered to GEMM).  Replaces LayerOps::linear_forward (LayerOps.hpp:24-111)
// and HardwareOpt::matmul_fma_saturated (HardwareOpt.hpp:95-149).
//
//   Y[m, n] = act( sum_k A[m, k] * W[n, k] + bias[n] ) (+ residual[m, n])
//
// Both operands are K-major ("TN"), which is the reference's Linear layout (W is [out][in]).
// fp32 operands are carried as bf16 planes: x = hi + lo with hi = bf16(x), lo = bf16(x - hi).
// The kernel issues hi*hi + lo*hi + hi*lo (the lo*lo term, ~2^-18 relative, is dropped) with fp32
// accumulation in tensor memory, which keeps the result within ~2^-16 per product of the fp32
// CPU path while running on the bf16 tensor pipe.
//
// sm_100a structure (one CTA per SM, persistent over output tiles):
//   warp 0      : TMA producer  — cp.async.bulk.tensor (no multicast) into a ring of smem stages
//   warp 1      : MMA issuer    — one thread issues tcgen05.mma, operands from smem descriptors,
//                                 accumulators in TMEM (2 x 256 columns, double buffered)
//   warps 2..9  : epilogue      — tcgen05.ld TMEM -> registers, bias / activation / residual, 256-bit
//                                 stores of fp32 rows and/or the bf16 hi/lo planes of the next layer
//                                 (or channel-major NCHW for convs)
// Every mbarrier wait is bounded: after ~2 s it sets the device error word and the CTA drains.
#include "common.h"
#include "planes.cuh"
#include "sm100_ptx.cuh"
#include "epilogue.cuh"
#include "launch.cuh"
#include "tensor_map.h"

#include <climits>
#include <cmath>
#include <cstring>

namespace mb {

namespace {

constexpr int BM = 128;        // rows of the output tile (TMEM lanes)
constexpr int BN = 256;        // columns of the output tile (one MMA, N = 256)
constexpr int UMMA_K = 16;     // bf16 K per tcgen05.mma
constexpr int NUM_ACC = 2;     // TMEM accumulator buffers
constexpr int TMEM_COLS = 512;
constexpr int NUM_THREADS = 320;  // 10 warps: TMA, MMA, 8 epilogue
constexpr int EPI_WARPS = 8;
constexpr float ACC_TRUNC_PER_MMA = 1.5e-8f;  // mean relative loss of the fp32 accumulator per tcgen05.mma (truncating adds)

struct GemmParams {
  int m, n, kblocks;         // kblocks = kp / BK
  int a_planes, w_planes;
  int tiles_m, tiles_n, group_n;
  const float* bias;
  const float* residual;
  int activation;
  float* out_f32;
  long long ldo;
  __nv_bfloat16* out_split;  // [2][m][np]
  long long np;              // round_up(n, 64)
  int ohw;                   // > 0: fp32 output (and residual) are NCHW, row = sample * ohw + pixel
  int bn;                    // columns of an output tile = N of one MMA: BN, or 192 on request (plain row-major form only)
  // Convolution as a sum of shifted GEMMs (conv_ks > 0): A is the zero-padded NHWC activation matrix
  // [samples * hp * wp, C]; k-block kb belongs to tap t = kb / conv_cblocks and reads A rows shifted by
  // (kh - pad) * wp + (kw - pad); output rows live on the padded grid, border rows are dropped.
  int conv_ks, conv_cblocks, conv_pad, conv_hp, conv_wp, conv_h, conv_w;
  // swap != 0 (channel-major outputs with at most 128 output channels): the weights are the M side of the
  // MMA (TMEM lane = output channel) and 256 activation rows are its N side.  A tcgen05.mma with M = 128 costs
  // the same whatever its N, so a narrow layer computed the usual way (N = its few channels, padded to the
  // tile) pays for 256 columns it does not have; swapped, every instruction does full work.
  int swap;
  int tma_store;  // fp32 row-major output leaves through TMA stores (map_o) instead of per-lane stores
  // Every accumulator is multiplied by this before bias / activation: 1 + ACC_TRUNC_PER_MMA * (MMAs per output).
  // The tensor core adds each MMA's products to the fp32 accumulator with truncation, not round-to-nearest, which
  // shrinks every result by a little less than 2^-26 of its value per instruction (see launch_gemm_t).
  float acc_scale;
  const unsigned* w_amax;  // see GemmArgs
  int f16;        // operand planes (and out_split) hold IEEE half instead of bfloat16
  // The operand ring: a stage holds only the planes the precision mode uses (32 KB with two activation planes and one
  // weight plane at BK = 32), so the same shared memory gives six stages instead of four - the K = 768 layers were
  // starved of operands with four (the MMA thread spent a quarter of every tile waiting on a full barrier).
  int stages, stage_bytes;
  // Tiles from this one on run as two of 128 columns each: the last wave's, where it would leave half of the CTAs idle.
  int full_tiles;
  int* err_word;
  // grouped form: W rows of tile (tm, tn) start at (tm * BM / a_group_rows) * w_group_rows + tn * bn (0 = one group)
  int a_group_rows, w_group_rows;
};

// Tile order: groups of `group_n` column tiles; inside a group the row tile runs fastest, so the
// CTAs resident at one time share a few W column tiles (kept in L2) while A streams through.
__device__ __forceinline__ void tile_coords(int t, const GemmParams& p, int& tm, int& tn) {
  const int per_group = p.group_n * p.tiles_m;
  const int g = t / per_group;
  const int r = t - g * per_group;
  const int gn0 = g * p.group_n;
  const int gw = min(p.group_n, p.tiles_n - gn0);
  tn = gn0 + r % gw;
  tm = r / gw;
}

// The tile of work item t and, of a tile that is cut in two, which half of its columns (else -1).
__device__ __forceinline__ int work_coords(int t, const GemmParams& p, int& tm, int& tn) {
  int half = -1;
  if (t >= p.full_tiles) {
    half = (t - p.full_tiles) & 1;
    t = p.full_tiles + ((t - p.full_tiles) >> 1);
  }
  tile_coords(t, p, tm, tn);
  return half;
}

template <int BK>
struct SmemLayout {
  static constexpr int kATile = BM * BK * 2;
  static constexpr int kWTile = BN * BK * 2;
};

constexpr int MAX_STAGES = 8;

// The MMA role: MP planes on the M side, NP on the N side.  The whole warp runs it and one elected lane issues (elect_one); the
// next stage's barrier is polled before the current stage's MMAs are issued, so that a K block costs its MMAs and not the
// latency of a wait on top (see gemm_split.cu).  Measured per 64-wide K block of one MMA per product: 1 100 cycles as a
// branch on lane 0, about 300 in this form; with two and three MMAs per product the tensor pipe is the limit again.
template <int BK, int PAIR, int MP, int NP>
__device__ __forceinline__ void mma_role(const GemmParams& p, uint8_t* smem, uint64_t* full_bar, uint64_t* empty_bar, uint64_t* acc_full,
                                         uint64_t* acc_empty, volatile int* abort_flag, uint32_t tmem_base, int t_first, int t_step,
                                         int num_tiles) {
  constexpr int SWZ = BK * 2, A_TILE = BM * BK * 2, W_TILE = (PAIR ? BN / 2 : BN) * BK * 2;
  const bool one = elect_one();
  const uint32_t idesc_full = make_idesc(PAIR ? 2 * BM : BM, p.bn, p.f16), idesc_half = make_idesc(PAIR ? 2 * BM : BM, BN / 2, p.f16);
  const int stages = p.stages, stage_bytes = p.stage_bytes, kblocks = p.kblocks;
  int stage = 0, acc = 0;
  uint32_t phase = 0, acc_phase = 0;
  bool ready = false;
  for (int t = t_first; t < num_tiles; t += t_step) {
    if (!mbar_wait_warp(&acc_empty[acc], acc_phase ^ 1, abort_flag, p.err_word, 3)) return;
    tcgen05_fence_after();
    const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
    const uint32_t idesc = t >= p.full_tiles ? idesc_half : idesc_full;
    for (int kb = 0; kb < kblocks; ++kb) {
      if (!__all_sync(0xffffffffu, ready) && !mbar_wait_warp(&full_bar[stage], phase, abort_flag, p.err_word, 4)) return;
      tcgen05_fence_after();
      const uint32_t sa = smem_u32(smem + stage * stage_bytes);
      const uint64_t da = make_smem_desc(sa, SWZ), dw = make_smem_desc(sa + MP * A_TILE, SWZ);
      const uint64_t da_lo = da + (A_TILE >> 4), dw_lo = dw + (W_TILE >> 4);
      uint64_t* done = &empty_bar[stage];
      if (++stage == stages) { stage = 0; phase ^= 1; }
      ready = mbar_test(&full_bar[stage], phase);
      if (one) {
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k) {  // 32 bytes further along K = 2 in a descriptor's address field
          const uint32_t add = (kb | k) != 0 ? 1u : 0u;
          if (PAIR) {
            umma_bf16_pair(d_tmem, da + 2 * k, dw + 2 * k, idesc, add);
            if (MP == 2) umma_bf16_pair(d_tmem, da_lo + 2 * k, dw + 2 * k, idesc, 1u);
            if (NP == 2) umma_bf16_pair(d_tmem, da + 2 * k, dw_lo + 2 * k, idesc, 1u);
          } else {
            umma_bf16(d_tmem, da + 2 * k, dw + 2 * k, idesc, add);
            if (MP == 2) umma_bf16(d_tmem, da_lo + 2 * k, dw + 2 * k, idesc, 1u);
            if (NP == 2) umma_bf16(d_tmem, da + 2 * k, dw_lo + 2 * k, idesc, 1u);
          }
        }
        if (PAIR) {  // frees the stage in both CTAs when these MMAs have read it
          umma_commit_pair(mapa_shared(smem_u32(done), 0));
          umma_commit_pair(mapa_shared(smem_u32(done), 1));
        } else {
          umma_commit(done);
        }
      }
      __syncwarp();
    }
    if (one) {
      if (PAIR) {
        umma_commit_pair(mapa_shared(smem_u32(&acc_full[acc]), 0));
        umma_commit_pair(mapa_shared(smem_u32(&acc_full[acc]), 1));
      } else {
        umma_commit(&acc_full[acc]);
      }
    }
    __syncwarp();
    if (++acc == NUM_ACC) { acc = 0; acc_phase ^= 1; }
  }
}

// CM = 1 compiles the channel-major forms in (NCHW output, convolution as shifted GEMMs, swapped operands); the plain
// row-major form (CM = 0: every Linear and attention projection) is built without them, so that the two families
// neither share a register budget nor slow each other's epilogue down.
// PAIR = 1 (not with swapped operands): the kernel runs as clusters of two CTAs on neighbouring SMs that share one 256-row x 256-column
// tile (tcgen05 with cta_group::2).  Each CTA loads its own 128 rows of A and only HALF of the W tile; the even-ranked
// CTA issues the MMAs for both, each CTA reads its 128 accumulator rows out of its own tensor memory.  The operand
// bytes an SM pulls from L2 per MMA cycle drop by a quarter to a third, which is what the short-K layers are short of.
template <int BK, int RING_BYTES, int CM, int PAIR>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tn_bf16split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                         const __grid_constant__ CUtensorMap map_o, const GemmParams p) {
  constexpr int SWZ = BK * 2;                      // bytes per smem row = swizzle span
  constexpr int A_TILE = BM * BK * 2;
  constexpr int W_TILE = (PAIR ? BN / 2 : BN) * BK * 2;  // a CTA of a pair holds half of the N side
  const int STAGES = p.stages, STAGE_BYTES = p.stage_bytes;
  const uint32_t crank = PAIR ? cluster_ctarank() : 0u;  // 0 = the pair's leader
  const int t_first = PAIR ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x);
  const int t_step = PAIR ? static_cast<int>(gridDim.x >> 1) : static_cast<int>(gridDim.x);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 1024-byte alignment is required by the 128-byte swizzle atoms
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // behind the stages: one staging tile per epilogue warp (32 x 33 floats for the swapped form's transposition, or a
  // dense 128-byte-swizzled 32 x 32 tile, 1024-byte aligned, as the source of a TMA store), then the barriers
  uint8_t* epi_tiles = smem + RING_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi_tiles + EPI_WARPS * 32 * 33 * 4);
  uint64_t* empty_bar = full_bar + MAX_STAGES;
  uint64_t* acc_full = empty_bar + MAX_STAGES;
  uint64_t* acc_empty = acc_full + NUM_ACC;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + NUM_ACC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int all_tiles = p.tiles_m * p.tiles_n;
  const int num_tiles = CM == 0 && p.full_tiles < all_tiles ? 2 * all_tiles - p.full_tiles : all_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < NUM_ACC; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], PAIR ? 2 * EPI_WARPS : EPI_WARPS);  // the leader's collects both CTAs' epilogue warps
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(tmem_slot, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // planes on the M side (128-row tiles) and on the N side (256-row tiles) of the MMA
  const bool swapped = CM && p.swap;
  const bool conv = CM && p.conv_ks > 0;
  const int m_planes = swapped ? p.w_planes : p.a_planes, n_planes = swapped ? p.a_planes : p.w_planes;
  const uint32_t tx_bytes = PAIR ? static_cast<uint32_t>(2 * (m_planes * A_TILE + n_planes * W_TILE))  // both CTAs' loads land on the leader's barrier
                                 : static_cast<uint32_t>(m_planes * A_TILE + n_planes * (p.bn * BK * 2));

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------------------
    // (the whole warp runs the loop, one elected lane issues: see elect_one)
    const bool one = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = t_first; t < num_tiles && ok; t += t_step) {
      int tm, tn, cut = -1;
      if (CM == 0) cut = work_coords(t, p, tm, tn); else tile_coords(t, p, tm, tn);
      if (PAIR) tm = tm * 2 + static_cast<int>(crank);  // p.tiles_m counts row PAIRS
      // (of a tile that is cut in two: 128 columns, 64 of them in each CTA of a pair)
      const CUtensorMap* const wmap = cut >= 0 ? &map_o : &map_w;
      const uint32_t tx = cut >= 0 ? static_cast<uint32_t>((PAIR ? 2 : 1) * (m_planes * A_TILE + n_planes * (W_TILE / 2))) : tx_bytes;
      const int w_row = swapped ? tm * BM
                        : cut >= 0 ? tn * BN + cut * (BN / 2) + (PAIR ? static_cast<int>(crank) * (BN / 4) : 0)
                        : PAIR ? tn * BN + static_cast<int>(crank) * (BN / 2)
                               : tn * p.bn + (p.a_group_rows > 0 ? (tm * BM / p.a_group_rows) * p.w_group_rows : 0);
      const int a_row0 = swapped ? tn * BN : tm * BM;  // swapped: 256 activation rows (tile tn) are the N side
      for (int kb = 0; kb < p.kblocks; ++kb) {
        if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag, p.err_word, 1)) { ok = false; break; }
        uint8_t* m_base = smem + stage * STAGE_BYTES;
        uint8_t* n_base = m_base + m_planes * A_TILE;
        int a_col = kb * BK, a_row = a_row0;
        if (conv) {
          const int tap = kb / p.conv_cblocks, cb = kb - tap * p.conv_cblocks;
          const int kh = tap / p.conv_ks, kw = tap - kh * p.conv_ks;
          a_row += (kh - p.conv_pad) * p.conv_wp + (kw - p.conv_pad);  // may be negative: TMA zero-fills
          a_col = cb * BK;
        }
        if (one) {
          if (PAIR) {
            // the leader arms its barrier for the bytes of both CTAs; this CTA's bytes are counted there whichever
            // of the two arrives first (the phase cannot complete before the leader's arrive)
            if (crank == 0) mbar_expect_tx(&full_bar[stage], tx);
            const uint32_t fb = mapa_shared(smem_u32(&full_bar[stage]), 0);
            tma_load_3d_pair(m_base, &map_a, fb, a_col, a_row, 0);
            if (m_planes == 2) tma_load_3d_pair(m_base + A_TILE, &map_a, fb, a_col, a_row, 1);
            tma_load_3d_pair(n_base, wmap, fb, kb * BK, w_row, 0);
            if (n_planes == 2) tma_load_3d_pair(n_base + W_TILE, wmap, fb, kb * BK, w_row, 1);
          } else {
            mbar_expect_tx(&full_bar[stage], tx);
            uint8_t* ab = swapped ? n_base : m_base;
            uint8_t* wb = swapped ? m_base : n_base;
            tma_load_3d(ab, &map_a, &full_bar[stage], a_col, a_row, 0);
            if (p.a_planes == 2) tma_load_3d(ab + (swapped ? W_TILE : A_TILE), &map_a, &full_bar[stage], a_col, a_row, 1);
            tma_load_3d(wb, wmap, &full_bar[stage], kb * BK, w_row, 0);
            if (p.w_planes == 2) tma_load_3d(wb + (swapped ? A_TILE : W_TILE), wmap, &full_bar[stage], kb * BK, w_row, 1);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    // Drain: every stage this warp filled must have landed and been consumed (or the abort
    // flag is up) before the CTA may exit with copies in flight.
    for (int s = 0; s < STAGES; ++s) {
      if (!mbar_wait_warp(&empty_bar[stage], phase ^ 1, abort_flag, p.err_word, 2)) break;
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------------------
    if (crank == 0) {  // (of a pair: the leader)
      if (m_planes == 2 && n_planes == 2) mma_role<BK, PAIR, 2, 2>(p, smem, full_bar, empty_bar, acc_full, acc_empty, abort_flag, tmem_base, t_first, t_step, num_tiles);
      else if (m_planes == 2) mma_role<BK, PAIR, 2, 1>(p, smem, full_bar, empty_bar, acc_full, acc_empty, abort_flag, tmem_base, t_first, t_step, num_tiles);
      else if (n_planes == 2) mma_role<BK, PAIR, 1, 2>(p, smem, full_bar, empty_bar, acc_full, acc_empty, abort_flag, tmem_base, t_first, t_step, num_tiles);
      else mma_role<BK, PAIR, 1, 1>(p, smem, full_bar, empty_bar, acc_full, acc_empty, abort_flag, tmem_base, t_first, t_step, num_tiles);
    }
  } else {
    // ------------------------------ epilogue (warps 2..9) ---------------------------------
    // Two warps per TMEM lane quadrant, each owning half of the tile's columns.  A lane holds 32 consecutive
    // columns of its row: row-major outputs leave as whole 128-byte lines through 256-bit stores;
    // channel-major (NCHW) outputs are coalesced across lanes (lane <-> pixel).
    const int ew = warp - 2;
    const int quad = warp & 3;   // TMEM lane quadrant this warp may read
    const int half = ew >> 2;    // which half of the columns
    const bool chan_major = CM && (p.ohw > 0 || p.conv_ks > 0);
    const float acc_scale = p.w_amax == nullptr ? p.acc_scale : p.acc_scale * plane_unscale(__ldg(p.w_amax));
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = t_first; t < num_tiles; t += t_step) {
      int tm, tn, cut = -1;
      if (CM == 0) cut = work_coords(t, p, tm, tn); else tile_coords(t, p, tm, tn);
      if (PAIR) tm = tm * 2 + static_cast<int>(crank);
      // lane 0 does the bounded wait; the verdict is made warp-uniform because tcgen05.ld below
      // is a warp-collective instruction
      int ok = 1;
      if (lane == 0) ok = mbar_wait(&acc_full[acc], acc_phase, abort_flag, p.err_word, 5) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      while (!mbar_try_wait(&acc_full[acc], acc_phase)) {}  // completes at once: lane 0 saw the phase
      tcgen05_fence_after();
      const int row0 = tm * BM + quad * 32;
      const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(acc * BN);
      if (swapped) {
        // TMEM lane = output channel, column = activation row (pixel).  Each 32 x 32 chunk is turned around
        // through a padded shared-memory tile so that a lane owns a pixel again and the NCHW stores (and
        // residual loads) of a warp are 128 contiguous bytes per channel, as in the unswapped form.
        float* tbuf = reinterpret_cast<float*>(epi_tiles) + ew * (32 * 33);
        const int oc0 = row0;  // first output channel of this warp's 32 lanes
        const long long hw = conv ? static_cast<long long>(p.conv_h) * p.conv_w : static_cast<long long>(p.ohw);
        // where this lane's pixel of chunk ci lands in the NCHW output; false = the chunk is past the matrix (warp-uniform)
        auto geom = [&](int ci, int& c0, bool& pv, long long& o0) -> bool {
          c0 = (half * (BN / 64) + ci) * 32;
          const int r0 = tn * BN + c0;
          if (r0 >= p.m || oc0 >= p.n) return false;
          const int prow = r0 + lane;
          pv = prow < p.m;
          long long pbase = 0;
          if (conv) {
            const int per = p.conv_hp * p.conv_wp;
            const int smp = prow / per, rem = prow - smp * per;
            const int yq = rem / p.conv_wp;
            const int yy = yq - p.conv_pad, xx = rem - yq * p.conv_wp - p.conv_pad;
            pv = pv && yy >= 0 && yy < p.conv_h && xx >= 0 && xx < p.conv_w;
            pbase = static_cast<long long>(smp) * p.n * hw + static_cast<long long>(yy) * p.conv_w + xx;
          } else {
            const long long smp = prow / p.ohw;
            pbase = smp * p.n * hw + (prow - smp * p.ohw);
          }
          o0 = pbase + static_cast<long long>(oc0) * hw;
          return true;
        };
        const bool full = oc0 + 32 <= p.n;
        // With a short K the epilogue, not the MMA, sets the pace.  The residual of a chunk is requested before the chunk
        // is read out of tensor memory and turned around, and the lines of the next chunk are pulled into L2 meanwhile, so
        // that the loads do not each wait a full memory latency.
        constexpr int NCH = (BN / 32) / 2;
#pragma unroll 1
        for (int ci = 0; ci < NCH; ++ci) {
          int c0; bool pv; long long o0;
          if (!geom(ci, c0, pv, o0)) break;
          float q[32];
          if (p.residual != nullptr) {
            if (pv) {
#pragma unroll
              for (int j = 0; j < 32; ++j) q[j] = (full || oc0 + j < p.n) ? __ldg(p.residual + o0 + j * hw) : 0.0f;
            }
            int c1; bool pv1; long long o1;
            if (ci + 1 < NCH && geom(ci + 1, c1, pv1, o1) && pv1) {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (full || oc0 + j < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.residual + o1 + j * hw));
            }
          }
          float v[32];
          tmem_ld_32x32(taddr0 + c0, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) tbuf[j * 33 + lane] = __fmul_rn(v[j], acc_scale);  // [pixel][channel]
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = tbuf[lane * 33 + j];  // lane = pixel r0 + lane, j = channel oc0 + j
          __syncwarp();
          if (p.activation != -1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], p.activation);
          }
          if (pv) {
            if (p.residual != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += q[j];
            }
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (full || oc0 + j < p.n) p.out_f32[o0 + j * hw] = v[j];
          }
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
        if (++acc == NUM_ACC) { acc = 0; acc_phase ^= 1; }
        continue;
      }
      const int col_limit = (p.out_split != nullptr) ? static_cast<int>(p.np) : p.n;
      // channel-major addressing of this lane's row
      bool cm_ok = false;
      long long cm_o0 = 0, cm_stride = 0;
      if (chan_major) {
        const int row = row0 + lane;
        cm_ok = row < p.m;
        if (conv) {
          const int per = p.conv_hp * p.conv_wp;
          const int smp = row / per, rem = row - smp * per;
          const int yq = rem / p.conv_wp;
          const int yy = yq - p.conv_pad, xx = rem - yq * p.conv_wp - p.conv_pad;
          cm_ok = cm_ok && yy >= 0 && yy < p.conv_h && xx >= 0 && xx < p.conv_w;
          cm_stride = static_cast<long long>(p.conv_h) * p.conv_w;
          cm_o0 = static_cast<long long>(smp) * p.n * cm_stride + static_cast<long long>(yy) * p.conv_w + xx;
        } else {
          const long long smp = row / p.ohw;
          cm_stride = p.ohw;
          cm_o0 = smp * p.n * cm_stride + (row - smp * p.ohw);
        }
      }
      // one 32-column chunk of this lane's row: scale, bias, activation, residual, stores
      auto process = [&](const int c0, const int col0, float (&v)[32]) {
        (void)c0;
        const bool full_cols = (col0 + 32 <= p.n);
        // scale and bias (the same 32 values for every lane: broadcast loads) in one rounding, as in gemm_split.cu: both kernels
        // give the same bits where they add up K in the same order
        if (p.bias != nullptr && full_cols && ((reinterpret_cast<uintptr_t>(p.bias + col0) & 15) == 0)) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 b4 = __ldg(reinterpret_cast<const float4*>(p.bias + col0 + j));
            v[j] = __fmaf_rn(v[j], acc_scale, b4.x); v[j + 1] = __fmaf_rn(v[j + 1], acc_scale, b4.y);
            v[j + 2] = __fmaf_rn(v[j + 2], acc_scale, b4.z); v[j + 3] = __fmaf_rn(v[j + 3], acc_scale, b4.w);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __fmaf_rn(v[j], acc_scale, (p.bias != nullptr && col0 + j < p.n) ? __ldg(p.bias + col0 + j) : 0.0f);
        }
        switch (p.activation) {  // hoisted out of the element loop
          case MIMIR_B200_ELT_GELU:
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = gelu_ref(v[j]);
            break;
          case -1:
            break;
          default:
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], p.activation);
            break;
        }
        if (chan_major) {
          if (cm_ok) {
            const long long o0 = cm_o0 + static_cast<long long>(col0) * cm_stride;
            if (p.residual != nullptr) {
              // all loads first: the output may alias nothing here, but the compiler cannot know, and
              // load -> store -> load chains would serialise on memory latency
              float q[32];
#pragma unroll
              for (int j = 0; j < 32; ++j) q[j] = (full_cols || col0 + j < p.n) ? __ldg(p.residual + o0 + j * cm_stride) : 0.0f;
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += q[j];
            }
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (full_cols || col0 + j < p.n) p.out_f32[o0 + j * cm_stride] = v[j];
          }
        } else {
          // row-major: this lane owns 32 consecutive columns of its row = one 128-byte line, moved with
          // 256-bit loads / stores (full 32-byte sectors, no transposition needed)
          const int row = row0 + lane;
          if (row < p.m) {
            const long long ro = static_cast<long long>(row) * p.ldo + col0;
            if (p.residual != nullptr) {
              const float* rr = p.residual + ro;
              if (full_cols && ((reinterpret_cast<uintptr_t>(rr) & 31) == 0)) {
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                  float q[8];
                  ld_global_v8(rr + j, q);
#pragma unroll
                  for (int e = 0; e < 8; ++e) v[j + e] += q[e];
                }
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < p.n) v[j] += __ldg(rr + j);
              }
            }
            if (p.out_f32 != nullptr && !p.tma_store) {
              float* o = p.out_f32 + ro;
              if (full_cols && ((reinterpret_cast<uintptr_t>(o) & 31) == 0)) {
#pragma unroll
                for (int j = 0; j < 32; j += 8) st_global_v8(o + j, &v[j]);
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < p.n) o[j] = v[j];
              }
            }
            if (p.out_split != nullptr) {
              // hi/lo planes for the next GEMM; columns n..np-1 are written as zero so that the padded
              // K of the consumer stays zero (np is a multiple of 64, so the chunk is always whole)
              uint32_t hi[16], lo[16];
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                const float x0 = (full_cols || col0 + j < p.n) ? v[j] : 0.0f;
                const float x1 = (full_cols || col0 + j + 1 < p.n) ? v[j + 1] : 0.0f;
                split_pair(x0, x1, p.f16, hi[j >> 1], lo[j >> 1]);
              }
              __nv_bfloat16* oh = p.out_split + static_cast<long long>(row) * p.np + col0;
              __nv_bfloat16* ol = oh + static_cast<long long>(p.m) * p.np;
              st_global_v8_b32(oh, &hi[0]);
              st_global_v8_b32(oh + 16, &hi[8]);
              st_global_v8_b32(ol, &lo[0]);
              st_global_v8_b32(ol + 16, &lo[8]);
            }
          }
          if (p.tma_store) {
            // fp32 rows through a TMA store: staged in shared memory (128-byte swizzle, conflict-free 128-bit writes)
            // the 32 x 32 chunk is one copy, clipped at the edges of the output by the tensor map.
            float* tile = reinterpret_cast<float*>(epi_tiles + ew * 4096);
            if (lane == 0) bulk_wait_read0();  // the previous chunk's copy has read the tile
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 8; ++c)
              *reinterpret_cast<float4*>(tile + lane * 32 + ((c ^ (lane & 7)) << 2)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&map_o, tile, col0, row0);
              bulk_commit();
            }
          }
        }
      };
      // (Tried: the next chunk's tensor-memory load in flight while this one is processed - two register sets, the
      // plain form has the room.  Measured neutral to 7 % slower on the K = 768 layers: the load's latency is not what
      // the short-K tiles wait for; operand and store bytes per MMA cycle are.)
      const int bn = cut >= 0 ? BN / 2 : p.bn, nch = (bn / 32) / 2;
#pragma unroll 1
      for (int ci = 0; ci < nch; ++ci) {
        const int c0 = (half * (bn / 64) + ci) * 32;
        const int col0 = tn * p.bn + (cut > 0 ? BN / 2 : 0) + c0;
        if (col0 >= col_limit) break;  // warp-uniform
        float v[32];
        tmem_ld_32x32(taddr0 + c0, v);
        process(c0, col0, v);
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&acc_empty[acc]), 0));  // the leader's MMA thread waits for both CTAs
        else mbar_arrive(&acc_empty[acc]);
      }
      if (++acc == NUM_ACC) { acc = 0; acc_phase ^= 1; }
    }
    if (lane == 0) bulk_wait_read0();  // no copy may still be reading shared memory when the CTA exits
  }

  tcgen05_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the other may still signal it
  if (warp == 1) {
    tcgen05_fence_after();
    if (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

}  // namespace

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}
}  // namespace

// 3-D map over bf16 planes [planes][rows][kp]; box = {bk, box_rows, 1}; swizzle span = bk * 2 bytes.
int make_plane_map(CUtensorMap* map, const void* base, int planes, long long rows, int kp, int bk, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(MIMIR_B200_E_CUDA, "cuTensorMapEncodeTiled entry point not available");
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return fail(MIMIR_B200_E_INVALID, "GEMM operand not 16-byte aligned");
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(kp), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(planes)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(kp) * 2, static_cast<cuuint64_t>(rows) * kp * 2};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(bk), static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUtensorMapSwizzle sw = (bk == 64) ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MIMIR_B200_E_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
  return MIMIR_B200_OK;
}

// 5-D map over zero-padded NHWC planes [planes][n][hp][wp][c]; box = {bc, bx, by, 1, 1}; swizzle span = bc * 2 bytes.
int make_image_map(CUtensorMap* map, const void* base, int planes, int n, int hp, int wp, int c, int bc, int bx, int by) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(MIMIR_B200_E_CUDA, "cuTensorMapEncodeTiled entry point not available");
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (bc != 32 && bc != 64) || c % bc != 0) return fail(MIMIR_B200_E_INVALID, "conv operand layout");
  const cuuint64_t row = static_cast<cuuint64_t>(c) * 2, line = row * wp, image = line * hp;
  cuuint64_t dims[5] = {static_cast<cuuint64_t>(c), static_cast<cuuint64_t>(wp), static_cast<cuuint64_t>(hp), static_cast<cuuint64_t>(n), static_cast<cuuint64_t>(planes)};
  cuuint64_t strides[4] = {row, line, image, image * n};
  cuuint32_t box[5] = {static_cast<cuuint32_t>(bc), static_cast<cuuint32_t>(bx), static_cast<cuuint32_t>(by), 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  const CUtensorMapSwizzle sw = (bc == 64) ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MIMIR_B200_E_CUDA, "cuTensorMapEncodeTiled (image) failed (%d)", static_cast<int>(r));
  return MIMIR_B200_OK;
}

// What an accumulator is multiplied by before bias / activation: the mean loss of the tensor core's truncating adds undone, the
// weight scale divided out.  Measured on B200 against fp64 products of the same operand planes (random normal operands, K = 256 ...
// 4096, two and three MMAs per 16-wide K step): the accumulated result is low by 1.47e-8 ... 1.58e-8 of its value per MMA
// instruction that added into it; all-positive operands lose 2.1e-8 ... 3.6e-8.  Zero-padded K adds exact zeros and loses nothing,
// so only the real K counts.  Undoing the mean loss halves the accumulation error.
float gemm_acc_scale(const GemmArgs& g) {
  const long long ksteps = g.conv_ks > 1 ? static_cast<long long>(g.conv_ks) * g.conv_ks * ((g.conv_c + UMMA_K - 1) / UMMA_K)
                                         : (g.k + UMMA_K - 1) / UMMA_K;
  const int products = 1 + (g.a_planes == 2 ? 1 : 0) + (g.w_planes == 2 ? 1 : 0);
  static const bool comp = [] { const char* e = getenv("MIMIR_B200_ACC_COMP"); return !(e && e[0] == '0'); }();
  return (comp ? 1.0f + ACC_TRUNC_PER_MMA * static_cast<float>(ksteps * products) : 1.0f) / g.w_scale;
}

int GemmProfile::begin() {
  if (!ctx().prof_gemm) return MIMIR_B200_OK;
  MB_CUDA(cudaEventCreate(&e0));
  MB_CUDA(cudaEventCreate(&e1));
  MB_CUDA(cudaEventRecord(e0, st));
  return MIMIR_B200_OK;
}
int GemmProfile::end() {
  if (!e0) return MIMIR_B200_OK;
  MB_CUDA(cudaEventRecord(e1, st));
  ctx().prof_events.push_back(e0);
  ctx().prof_events.push_back(e1);
  return MIMIR_B200_OK;
}

// ------------------------------------------------------------------------------------------
// fp32 -> bf16 hi/lo planes
// ------------------------------------------------------------------------------------------
namespace {

// One thread per 8 consecutive K elements of one row; the padded tail kp > k is written as zero.
__global__ void split_rows_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long rows, int k,
                                  int kp, int planes, int f16, float scale, const unsigned* __restrict__ amax) {
  pdl_launch_dependents();
  pdl_wait();
  if (amax != nullptr) scale = plane_scale(__ldg(amax));
  const int chunks = kp >> 3;
  const long long total = rows * chunks;
  const long long plane_stride = rows * static_cast<long long>(kp);
  const bool vec_ok = ((k & 3) == 0) && ((reinterpret_cast<uintptr_t>(src) & 15) == 0);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / chunks;
    const int c = static_cast<int>(i - r * chunks) << 3;
    float v[8];
    const float* s = src + r * k + c;
    if (vec_ok && c + 8 <= k) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(s));
      const float4 b = __ldg(reinterpret_cast<const float4*>(s + 4));
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = (c + j < k) ? __ldg(s + j) : 0.0f;
    }
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) split_pair(v[j] * scale, v[j + 1] * scale, f16, h[j >> 1], l[j >> 1]);
    __nv_bfloat16* d = dst + r * kp + c;
    *reinterpret_cast<uint4*>(d) = make_uint4(h[0], h[1], h[2], h[3]);
    if (planes == 2) *reinterpret_cast<uint4*>(d + plane_stride) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// src fp32 [k, n] row-major -> planes of the transpose [n, kp].  32x32 tiles through shared memory.
__global__ void split_transposed_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int k, int n,
                                        int kp, int planes, int f16, float scale) {
  __shared__ float tile[32][33];
  const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int kk = k0 + i, nn = n0 + threadIdx.x;
    tile[i][threadIdx.x] = (kk < k && nn < n) ? __ldg(src + static_cast<long long>(kk) * n + nn) : 0.0f;
  }
  __syncthreads();
  const long long plane_stride = static_cast<long long>(n) * kp;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int nn = n0 + i, kk = k0 + threadIdx.x;
    if (nn < n && kk < kp) {
      uint16_t h, l;
      split_one(tile[threadIdx.x][i] * scale, f16, h, l);
      uint16_t* d16 = reinterpret_cast<uint16_t*>(dst);
      d16[static_cast<long long>(nn) * kp + kk] = h;
      if (planes == 2) d16[plane_stride + static_cast<long long>(nn) * kp + kk] = l;
    }
  }
}

// 2-D map over the fp32 row-major output [rows][ld]; box = 32 x 32, 128-byte swizzle (the epilogue's staging tile)
int make_out_map(CUtensorMap* map, const float* base, long long rows, int cols, long long ld) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(MIMIR_B200_E_CUDA, "cuTensorMapEncodeTiled entry point not available");
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MIMIR_B200_E_CUDA, "cuTensorMapEncodeTiled (output) failed (%d)", static_cast<int>(r));
  return MIMIR_B200_OK;
}

int env_int(const char* name, int dflt) {
  const char* v = getenv(name);
  return (v && *v) ? atoi(v) : dflt;
}

// The form of a launch, the same for its choice (big_tile_cycles, the K block in launch_gemm) and for the launch itself.

// narrow channel-major layers run with the operands swapped (see GemmParams::swap); short K keeps the usual
// form, whose epilogue writes NCHW with coalesced stores
bool swaps_operands(const GemmArgs& g) {
  const char* noswap = getenv("MIMIR_B200_GEMM_NOSWAP");
  const int k = g.conv_ks > 0 ? g.conv_ks * g.conv_ks * g.conv_c : round_up(g.k, 64);
  return (g.conv_ks > 0 || g.out_nchw_hw > 0) && g.n <= BM && g.bias == nullptr && g.out_split == nullptr && g.out_f32 != nullptr &&
         g.m >= 4 * BN && k >= 256 && !(noswap && noswap[0] == '1');
}

// Optional (MIMIR_B200_GEMM_TMA_STORE=1): row-major fp32 outputs leave through TMA stores.  Measured neutral on the
// decoder's K = 768 layers (1 078 vs 1 100 TFLOP/s issued): what slows those layers is not the shape of the stores but
// their bytes - the operand loads alone run at ~62 B per cycle and SM, next to what an SM can take from L2, and the
// same kernel without any output store reaches 1 315.
bool stores_by_tma(const GemmArgs& g) {
  static const bool on = [] { const char* e = getenv("MIMIR_B200_GEMM_TMA_STORE"); return e && e[0] == '1'; }();
  return on && g.conv_ks <= 0 && g.out_nchw_hw <= 0 && g.out_f32 != nullptr && g.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(g.out_f32) & 15) == 0;
}

// MIMIR_B200_GEMM_BN=192: 192-column tiles.  On paper they shorten launches whose last wave is mostly empty (N = 768
// over 256 row tiles: 7 waves of 192 columns instead of 6 of 256, 12.5 % less work per SM); measured, the
// 32768 x 768 x 768 projection takes 0.076 ms either way and the K = 3072 one 0.243 against 0.251: an N = 192
// instruction costs the tensor pipe about what an N = 256 one does.  Kept as a switch, off by default.
int tile_columns(const GemmArgs& g) {
  static const int force = env_int("MIMIR_B200_GEMM_BN", 0);
  return force == 192 && g.conv_ks <= 0 && !swaps_operands(g) && !stores_by_tma(g) ? 192 : BN;
}

// CTA pairs: every form but the swapped one, full-width tiles.  Taken by default where they were measured to pay: launches of at least one
// full wave of tiles in the modes with two or three MMAs per product (same-run A/B: the K = N = 4096 layer 14.9-15.0
// -> 14.5 ms per three-layer step = 0.333 of the sustained peak, the whole ceiling of the three-MMA scheme; the decoder
// step 18.51 -> 18.2 ms).  The one-MMA mode (14.78 -> 14.88 ms) and launches of a few tiles (the registry
// transformer's 1024-row layers: 0.290 -> 0.295 ms per step) are better off alone.  MIMIR_B200_GEMM_PAIR=0 turns pairs
// off, =1 takes them wherever the form allows.
bool takes_pairs(const GemmArgs& g) {
  static const int pair_env = env_int("MIMIR_B200_GEMM_PAIR", -1);
  const long long tiles_m = (g.m + BM - 1) / BM, tiles = tiles_m * ((g.n + BN - 1) / BN);
  return !swaps_operands(g) && !stores_by_tma(g) && tile_columns(g) == BN && tiles_m >= 2 && g.a_group_rows <= 0 &&
         (pair_env == 1 || (pair_env != 0 && g.a_planes + g.w_planes >= 3 && tiles >= ctx().sm_count));
}

// The last wave's tiles as halves where it has at most half as many tiles as there are CTAs (pairs): the same sums in the same order, bit
// for bit.  A half takes 0.53 of a tile with three MMAs per product, 0.67 with two (the activations are loaded whole).
bool halves_last_wave(const GemmArgs& g) {
  static const bool on = env_int("MIMIR_B200_GEMM_HALVES", 1) != 0;
  return on && g.conv_ks <= 0 && g.out_nchw_hw <= 0 && !stores_by_tma(g) && tile_columns(g) == BN && g.a_group_rows <= 0 && g.a_planes + g.w_planes >= 3;
}

template <int BK>
int launch_gemm_t(const GemmArgs& g, cudaStream_t st) {
  const int kp = round_up(g.k, 64);
  const bool conv = g.conv_ks > 0;
  CUtensorMap map_a, map_w;
  // conv: A rows are `conv_c` channels long and K = taps * conv_c runs over (tap, channel)
  const bool swap = swaps_operands(g);
  MB_TRY(make_plane_map(&map_a, g.a, g.a_planes, g.m, conv ? g.conv_c : kp, BK, swap ? BN : BM));
  const bool tma_store = stores_by_tma(g);
  CUtensorMap map_o = map_a;  // (a valid map when unused)
  if (tma_store) MB_TRY(make_out_map(&map_o, g.out_f32, g.m, g.n, g.ldo));
  GemmParams p;
  p.tma_store = tma_store ? 1 : 0;
  p.swap = swap ? 1 : 0;
  p.tiles_m = swap ? (g.n + BM - 1) / BM : (g.m + BM - 1) / BM;
  p.bn = tile_columns(g);
  const bool pair = takes_pairs(g);
  if (g.a_group_rows > 0 && (swap || conv || g.out_nchw_hw > 0 || g.a_group_rows % BM != 0 || g.w_group_rows <= 0 ||
                             g.w_rows_total < static_cast<long long>((g.m + g.a_group_rows - 1) / g.a_group_rows - 1) * g.w_group_rows + g.n))
    return fail(MIMIR_B200_E_INVALID, "gemm: bad grouped-form arguments");
  MB_TRY(make_plane_map(&map_w, g.w, g.w_planes, g.a_group_rows > 0 ? g.w_rows_total : g.n, kp, BK, swap ? BM : (pair ? BN / 2 : p.bn)));
  p.m = g.m;
  p.n = g.n;
  p.kblocks = conv ? g.conv_ks * g.conv_ks * (g.conv_c / BK) : kp / BK;
  p.conv_ks = g.conv_ks;
  p.conv_cblocks = conv ? g.conv_c / BK : 1;
  p.conv_pad = g.conv_pad;
  p.conv_hp = g.conv_h + 2 * g.conv_pad;
  p.conv_wp = g.conv_w + 2 * g.conv_pad;
  p.conv_h = g.conv_h;
  p.conv_w = g.conv_w;
  p.a_planes = g.a_planes;
  p.w_planes = g.w_planes;
  p.tiles_n = swap ? (g.m + BN - 1) / BN : (g.n + p.bn - 1) / p.bn;
  if (pair) p.tiles_m = (p.tiles_m + 1) / 2;  // row PAIRS: the CTA of rank r takes row tile 2 * pair + r
  p.group_n = env_int("MIMIR_B200_GEMM_GROUP_N", 8);
  if (p.group_n < 1) p.group_n = 1;
  if (p.group_n > p.tiles_n) p.group_n = p.tiles_n;
  p.bias = g.bias;
  p.residual = g.residual;
  p.activation = g.activation;
  p.out_f32 = g.out_f32;
  p.ldo = g.ldo;
  p.out_split = g.out_split;
  p.np = round_up(g.n, 64);
  p.ohw = g.out_nchw_hw;
  p.err_word = ctx().dev_error_word;
  p.a_group_rows = g.a_group_rows;
  p.w_group_rows = g.w_group_rows;
  p.acc_scale = gemm_acc_scale(g);
  p.w_amax = g.w_amax;
  p.f16 = plane_format() == PLANES_F16 ? 1 : 0;
  constexpr int RING_BYTES = 196608;  // 192 KB of operand stages, cut into as many stages as the planes in use allow
  constexpr int SMEM = RING_BYTES + 1024 /*align slack*/ + 512 /*barriers*/ + EPI_WARPS * 32 * 33 * 4 /*swapped-epilogue tiles*/;
  static_assert(SMEM <= 232448, "exceeds the 227 KB of shared memory a CTA may use");
  {
    const int m_pl = swap ? g.w_planes : g.a_planes, n_pl = swap ? g.a_planes : g.w_planes;
    p.stage_bytes = m_pl * BM * BK * 2 + n_pl * (pair ? BN / 2 : BN) * BK * 2;
    p.stages = RING_BYTES / p.stage_bytes;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    const int want = env_int("MIMIR_B200_GEMM_STAGES", 0);
    if (want >= 2 && want < p.stages) p.stages = want;
  }
  const bool cm = swap || conv || g.out_nchw_hw > 0;
  auto kern = cm ? (pair ? gemm_tn_bf16split_kernel<BK, RING_BYTES, 1, 1> : gemm_tn_bf16split_kernel<BK, RING_BYTES, 1, 0>)
                 : (pair ? gemm_tn_bf16split_kernel<BK, RING_BYTES, 0, 1> : gemm_tn_bf16split_kernel<BK, RING_BYTES, 0, 0>);
  static PerDeviceOnce attr_once;
  MB_TRY(attr_once.run([&]() -> int {
    MB_CUDA(cudaFuncSetAttribute(gemm_tn_bf16split_kernel<BK, RING_BYTES, 0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    MB_CUDA(cudaFuncSetAttribute(gemm_tn_bf16split_kernel<BK, RING_BYTES, 1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    MB_CUDA(cudaFuncSetAttribute(gemm_tn_bf16split_kernel<BK, RING_BYTES, 0, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    MB_CUDA(cudaFuncSetAttribute(gemm_tn_bf16split_kernel<BK, RING_BYTES, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    return MIMIR_B200_OK;
  }));
  const int tiles = p.tiles_m * p.tiles_n;
  int grid = tiles < ctx().sm_count ? tiles : ctx().sm_count;
  if (pair) {
    const int pairs = ctx().sm_count / 2;
    grid = 2 * (tiles < pairs ? tiles : pairs);
  }
  p.full_tiles = INT_MAX;
  const int workers = pair ? ctx().sm_count / 2 : ctx().sm_count, rest = tiles % workers;
  if (halves_last_wave(g) && rest > 0 && 2 * rest <= workers) {
    p.full_tiles = tiles - rest;
    MB_TRY(make_plane_map(&map_o, g.w, g.w_planes, g.n, kp, BK, pair ? BN / 4 : BN / 2));
    if (tiles < workers) grid = (pair ? 2 : 1) * 2 * rest;
  }
  GemmProfile prof(st);
  MB_TRY(prof.begin());
  if (pair) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MB_CUDA(cudaLaunchKernelEx(&cfg, kern, map_a, map_w, map_o, p));
  } else {
    kern<<<grid, NUM_THREADS, SMEM, st>>>(map_a, map_w, map_o, p);
  }
  MB_CUDA(cudaGetLastError());
  MB_TRY(prof.end());
  count_launch();
  return MIMIR_B200_OK;
}

}  // namespace

int plane_format() {
  static const int fmt = [] {
    const char* e = getenv("MIMIR_B200_PLANES");
    return (e && (e[0] == 'b' || e[0] == 'B')) ? PLANES_BF16 : PLANES_F16;
  }();
  return fmt;
}

namespace {
// largest finite |w| as its bit pattern (non-negative floats order like unsigned integers)
__global__ void absmax_kernel(const float* __restrict__ w, size_t n, unsigned* __restrict__ out) {
  unsigned m = 0;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const unsigned u = __float_as_uint(__ldg(w + i)) & 0x7fffffffu;
    if (u < 0x7f800000u && u > m) m = u;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
  if ((threadIdx.x & 31) == 0 && m != 0) atomicMax(out, m);
}
}  // namespace

int launch_absmax(const float* w_dev, size_t n, unsigned* word, cudaStream_t st) {
  MB_CUDA(cudaMemsetAsync(word, 0, sizeof(unsigned), st));
  const size_t want = (n + 255) / 256;
  const int blocks = static_cast<int>(want < static_cast<size_t>(ctx().sm_count) * 8 ? want : static_cast<size_t>(ctx().sm_count) * 8);
  absmax_kernel<<<blocks, 256, 0, st>>>(w_dev, n, word);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

int weight_plane_scale(const float* w_dev, size_t n, cudaStream_t st, float* scale) {
  *scale = 1.0f;
  if (plane_format() != PLANES_F16 || n == 0 || w_dev == nullptr) return MIMIR_B200_OK;
  static std::mutex mu;  // one spare device word is shared by every caller
  std::lock_guard<std::mutex> lk(mu);
  unsigned* word = reinterpret_cast<unsigned*>(ctx().dev_error_word) + 8;  // a spare word of the 256-byte error block
  MB_TRY(launch_absmax(w_dev, n, word, st));
  unsigned bits = 0;
  MB_CUDA(cudaMemcpyAsync(&bits, word, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
  MB_CUDA(cudaStreamSynchronize(st));
  *scale = ldexpf(1.0f, plane_scale_exponent(bits));
  return MIMIR_B200_OK;
}

int launch_split(const float* src, __nv_bfloat16* dst, int64_t rows, int k, int planes, cudaStream_t st, float scale, const unsigned* amax) {
  if (rows <= 0 || k <= 0) return MIMIR_B200_OK;
  const int kp = round_up(k, 64);
  const long long total = rows * (kp >> 3);
  const int threads = 256;
  long long blocks = (total + threads - 1) / threads;
  const long long cap = static_cast<long long>(ctx().sm_count) * 16;
  if (blocks > cap) blocks = cap;
  MB_TRY(launch_pdl(split_rows_kernel, dim3(static_cast<int>(blocks)), dim3(threads), 0, st, 1, src, dst, rows, k, kp, planes, plane_format() == PLANES_F16, scale, amax));
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

int launch_split_transposed(const float* src, __nv_bfloat16* dst, int k, int n, int planes, cudaStream_t st, float scale) {
  if (n <= 0 || k <= 0) return MIMIR_B200_OK;
  const int kp = round_up(k, 64);
  dim3 grid((n + 31) / 32, kp / 32), block(32, 8);
  split_transposed_kernel<<<grid, block, 0, st>>>(src, dst, k, n, kp, planes, plane_format() == PLANES_F16, scale);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

namespace {
// One CTA that waits on an mbarrier nobody arrives on, with the kernels' own bounded wait and a caller-given limit:
// the wait runs out, the error word and the abort flag are set, the roles leave, the TMEM columns are freed and the
// kernel returns - the give-up path of the tensor-core kernels, run on purpose.
__global__ void __launch_bounds__(64) wait_timeout_selftest_kernel(unsigned long long limit_ns, int* err_word) {
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 32);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_slot;
  if (warp == 0) {
    // the same whole-warp form the epilogue and softmax warps use: lane 0 waits, the verdict is made warp-uniform
    int ok = 1;
    if (lane == 0) ok = mbar_wait_limit(&bar, 0, &abort_flag, err_word, 90, limit_ns, 0xF) ? 1 : 0;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    (void)ok;
  } else if (lane == 0) {
    // a second role that sees the first one's abort flag and leaves (or runs out itself)
    mbar_wait_limit(&bar, 0, &abort_flag, err_word, 91, 4 * limit_ns, 0xF);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, 32);
  }
}
}  // namespace

int launch_wait_timeout_selftest(unsigned long long limit_ns, cudaStream_t st) {
  if (limit_ns == 0 || limit_ns > 100000000ull) return fail(MIMIR_B200_E_INVALID, "selftest: the limit must be within (0, 100 ms]");
  wait_timeout_selftest_kernel<<<1, 64, 0, st>>>(limit_ns, ctx().dev_error_word);
  MB_CUDA(cudaGetLastError());
  count_launch();
  return MIMIR_B200_OK;
}

namespace {
// Estimated SM cycles of a launch in 128 x 256 tiles (the same model as gemm_split.cu's plan_split: the larger of MMA time and
// operand loads per tile, whole waves, one exposed epilogue).
double big_tile_cycles(const GemmArgs& g) {
  const int products = 1 + (g.a_planes == 2) + (g.w_planes == 2);
  const double k = g.conv_ks > 0 ? static_cast<double>(g.k) : static_cast<double>(round_up(g.k, 64));
  const double mma = k / UMMA_K * products * 128.0, load = k * 2.0 * (g.a_planes * BM + g.w_planes * BN) / 51.6;
  if (g.conv_ks > 0 || g.out_nchw_hw > 0) {  // 256 pixels x 128 channels either way round; the epilogue's scattered stores bound short K
    const long long tiles = static_cast<long long>((g.m + BN - 1) / BN) * ((g.n + BM - 1) / BM), waves = (tiles + ctx().sm_count - 1) / ctx().sm_count;
    return 19000.0 + waves * (1.2 * mma > 12000.0 ? 1.2 * mma : 12000.0);
  }
  const long long tiles = static_cast<long long>((g.m + BM - 1) / BM) * ((g.n + BN - 1) / BN);
  const long long waves = (tiles + ctx().sm_count - 1) / ctx().sm_count;
  const double tile = mma > load ? mma : load;
  const double even = 15100.0 + waves * (tile > 12000.0 ? tile : 12000.0);  // (a tile's epilogue takes about 12 000 cycles beside the next main loop)
  // One tile to an SM starts cold: 1.25 tiles where the loop is short, and a long one has that behind it (measured, three MMAs per product,
  // 128 tiles, K = 1024 / 2048 / 4096: 26.4 / 42.5 / 77 us; this gives 26.5 / 42.4 / 74; 1.25 tiles for any K would give 85, which narrow
  // tiles beat on paper and miss by 15 % live).  Last waves in halves (launch_gemm_t): 1536 x 4096 x 4096 takes 110 us, here 106.
  if (waves == 1) {
    const double brief = 15100.0 + (1.25 * tile > 12000.0 ? 1.25 * tile : 12000.0), lengthy = 21000.0 + 1.02 * tile;
    return brief < lengthy ? brief : lengthy;
  }
  const bool pair = takes_pairs(g);
  const long long units = pair ? static_cast<long long>((g.m + 2 * BM - 1) / (2 * BM)) * ((g.n + BN - 1) / BN) : tiles;
  const int workers = pair ? ctx().sm_count / 2 : ctx().sm_count;
  const long long rest = units % workers;
  if (!halves_last_wave(g) || rest == 0 || 2 * rest > workers) return even;
  const double cut = 21000.0 + (static_cast<double>(units / workers) + (products == 3 ? 0.53 : 0.67)) * tile;
  return cut < even ? cut : even;
}
// The form of a launch.  128 x 256 tiles, narrow tiles with split K (only where the big tiles fill the GPU less than one and a half times:
// beyond that re-reading the operands costs more than an even last wave gives), and for convolutions tiles of 256 pixels.
enum class GemmForm { big, split, spatial };
struct GemmChoice { GemmForm form = GemmForm::big; int sbk = 64, bn = 0, splits = 0; };
// the arguments of the spatial-tile kernel: im2col rows are the pixels of an image with round_up(k, 64) channels
GemmArgs spatial_args(const GemmArgs& g) {
  GemmArgs c = g;
  if (g.conv_ks == 0 && g.out_nchw_hw > 0) {
    c.conv_ks = 1; c.conv_c = round_up(g.k, 64); c.conv_pad = 0; c.conv_h = 1; c.conv_w = g.out_nchw_hw;
    c.out_nchw_hw = 0;
  }
  return c;
}
GemmChoice choose_form(const GemmArgs& g) {
  GemmChoice r;
  r.sbk = (g.conv_ks == 0 || g.conv_c % 64 == 0) ? 64 : 32;
  const long long big_tiles = static_cast<long long>((g.m + BM - 1) / BM) * ((g.n + BN - 1) / BN);
  static const bool force_pairs = env_int("MIMIR_B200_GEMM_PAIR", -1) == 1;  // pairs wherever the form allows
  if (force_pairs) return r;
  const double big = big_tile_cycles(g);
  const double split = big_tiles < ctx().sm_count + ctx().sm_count / 2 ? gemm_split_cycles(g, r.sbk, &r.bn, &r.splits) : 1e30;
  const GemmArgs c = spatial_args(g);
  const double spatial = c.conv_ks > 0 ? conv_gemm_cycles(c) : 1e30;
  if (spatial < 1e30 && spatial <= split && spatial <= big) {
    r.form = GemmForm::spatial;
    return r;
  }
  // (4096 rows and more may come in micro-batches, which should then give the bits of a single pass: from 64 big tiles on those give
  // way only to a launch of half the cost - 4096 x 512 x 512 stays, at 0.55)
  const bool whole = g.conv_ks == 0 && g.out_nchw_hw == 0 && g.m >= 4096 && big_tiles >= 64;
  if (split < (whole ? 0.5 : 1.0) * big) r.form = GemmForm::split;
  return r;
}
}  // namespace

bool gemm_takes_spatial(const GemmArgs& g) { return choose_form(g).form == GemmForm::spatial; }

int launch_gemm(const GemmArgs& g, cudaStream_t st) {
  if (g.m <= 0 || g.n <= 0 || g.k <= 0) return fail(MIMIR_B200_E_INVALID, "gemm: empty dimension");
  if (!g.a || !g.w) return fail(MIMIR_B200_E_INVALID, "gemm: null operand");
  if (!g.out_f32 && !g.out_split) return fail(MIMIR_B200_E_INVALID, "gemm: no output");
  if (g.residual && !g.out_f32 && g.ldo < g.n) return fail(MIMIR_B200_E_INVALID, "gemm: residual needs the fp32 output stride");
  // K block per stage.  With at most three planes in play (one of the operands single-plane) a 64-wide block still leaves
  // three 64 KB stages, halves the barrier round trips per MMA and uses 128-byte swizzle rows: measured on the decoder's
  // K = 768 layers 0.77 -> 0.90 of the sustained cuBLAS rate.  With four planes (both operands split) 64-wide blocks leave a CTA on its
  // own two 96 KB stages, which measured slower than four 48 KB stages of 32, but a CTA of a pair three of 64 KB: the copy engine takes
  // half as many rows, 4096 x 4096 x 4096 three times 962 -> 939 us, 20000 x 1100 twice 355 -> 333, a 15 x 721 decoder 5.89 -> 5.78 ms.
  if (g.conv_ks > 0) {
    if (g.conv_c <= 0 || g.conv_c % 32 != 0 || g.k != g.conv_ks * g.conv_ks * g.conv_c || g.out_split || !g.out_f32)
      return fail(MIMIR_B200_E_INVALID, "gemm: bad shifted-convolution arguments");
  }
  const bool pairs = g.conv_ks == 0 && g.out_nchw_hw <= 0 && takes_pairs(g);
  const int bk = env_int("MIMIR_B200_GEMM_BK", (g.a_planes + g.w_planes <= 3 || pairs) ? 64 : 32);
  // planned for the spatial-tile kernel (conv_takes_residual_up, conv_can_emit_gn, conv_takes_normed_residual, conv_takes_padded_planes): the
  // others add a residual of the output's own shape as it is, leave no statistics and read planes of their own
  if (g.residual_up || g.gn_part != nullptr || g.res_coef != nullptr || g.conv_src_pad > 0) {
    if (conv_gemm_cycles(g) >= 1e30) return fail(MIMIR_B200_E_INVALID, "gemm: this residual, GroupNorm statistics or planes with a ring need the spatial-tile kernel");
    return launch_conv_gemm(g, st);
  }
  const GemmChoice c = choose_form(g);
  if (c.form == GemmForm::spatial) return launch_conv_gemm(spatial_args(g), st);
  if (c.form == GemmForm::split) return launch_gemm_split(g, c.sbk, c.bn, c.splits, st);
  if (bk == 64 && (g.conv_ks == 0 || g.conv_c % 64 == 0)) return launch_gemm_t<64>(g, st);
  return launch_gemm_t<32>(g, st);
}

}  // namespace mb
