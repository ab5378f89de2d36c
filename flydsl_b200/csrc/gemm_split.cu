// Grouped GEMM with the K range of every tile shared by a cluster of CTAs (few tiles, long K).
//
// The one-CTA-per-tile kernel (gemm_sm100.cu) leaves most SMs idle when a launch has fewer tiles than the
// GPU has SMs: a decode step's down projection over two experts is 32 tiles of 112 K blocks, a 64-row dense
// GEMM 9 tiles of 56.  Here a cluster of 2, 4 or 8 CTAs takes one tile together: rank r runs K blocks
// [KB*r/S, KB*(r+1)/S) with the same roles and ring as the other kernel, parks its fp32 partial sums in its
// own shared memory, and after an exchange over distributed shared memory each rank adds up, scales and
// stores every S-th row.  The partial sums are added in rank order, in fp32 (int32 for int8 operands), so the
// result does not depend on timing and nothing is rounded to 16 bits before the last step.
//
// What bounds it is latency: the serial K blocks of a tile (about 0.6 us each) before, the fill and the exchange
// now.  Measured on one B200, whole calls: dense M=64 N=2112 K=7168 43.0 -> 18.4 us (8 CTAs per tile), one token
// through a layer of 8 experts, 4096 x 14336, top-2: 136 -> 99 us (4 CTAs per tile in the down projection).
//
// Row blocks of 16, 32 or 64 rows (the launches that have few tiles); no per-row destinations.
// Every wait is bounded, as in the other kernel; all CTAs of a cluster meet once more before they exit, so
// that no shared memory goes away while a peer may still read it.
#include <cuda.h>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "gemm_args.cuh"
#include "gemm_ptx.cuh"

namespace flymoe {

constexpr int kSplitMaxRows = 64;
constexpr int kSplitStages = 4;
// A slots hold 64 rows; the MMA's rows 64-127 read on into the weight tile and land in TMEM lanes nobody reads.
constexpr int kSplitAStage = kSplitMaxRows * BK;
constexpr int kSplitStageBytes = kSplitAStage + kBTileBytes;
// Exchange row: 256 fp32 partial sums; 16 bytes of skew keep the row-per-lane float4 stores conflict-free.
constexpr int kExchPitch = BN * 4 + 16;

struct __align__(16) SplitCtrl {
  unsigned long long full[kSplitStages];
  unsigned long long empty[kSplitStages];
  unsigned long long tmem_full[kAccStages];
  unsigned long long tmem_empty[kAccStages];
  unsigned long long exch_full;                 // every rank's partial sums of the tile are in place
  unsigned long long exch_free;                 // every rank has read this rank's partial sums
  uint32_t tmem_base;
  int abort_flag;
};
constexpr size_t kSplitSmem = size_t(kSplitStages) * kSplitStageBytes + size_t(kSplitMaxRows) * kExchPitch +
                              sizeof(SplitCtrl) + 1024;
static_assert(kSplitSmem <= 232448, "shared memory budget of one SM exceeded");

__device__ __forceinline__ void red_add_2x16(void* p, uint32_t lo, uint32_t hi, bool bf) {
  if (bf) asm volatile("red.global.add.noftz.v2.bf16x2 [%0], {%1, %2};" ::"l"(p), "r"(lo), "r"(hi) : "memory");
  else asm volatile("red.global.add.noftz.v2.f16x2 [%0], {%1, %2};" ::"l"(p), "r"(lo), "r"(hi) : "memory");
}

template <int STAGE, int SCALING>
__global__ void __launch_bounds__(kNumThreads, 1)
moe_gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const GemmArgs a, const int group_m, const int split) {
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  uint8_t* exch = smem + size_t(kSplitStages) * kSplitStageBytes;
  SplitCtrl* ctrl = reinterpret_cast<SplitCtrl*>(exch + size_t(kSplitMaxRows) * kExchPitch);
  volatile int* abort_flag = &ctrl->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int KB = a.k_dim / BK;
  const int rank = int(cluster_rank());
  const int kb0 = int((long long)KB * rank / split), kb1 = int((long long)KB * (rank + 1) / split);
  const int first_tile = int(blockIdx.x) / split, tile_step = int(gridDim.x) / split;

  const int valid_rows = routed_rows(a);
  TileSched sched;
  sched.num_mblocks = (valid_rows + a.tile_m - 1) / a.tile_m;
  sched.num_ntiles = STAGE == 1 ? a.n_dim / 128 : (a.n_dim + BN - 1) / BN;
  sched.total = sched.num_mblocks * sched.num_ntiles;
  sched.group_m = group_m;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSplitStages; ++i) {
      mbar_init(smem_u32(&ctrl->full[i]), 1);
      mbar_init(smem_u32(&ctrl->empty[i]), 1);
    }
    for (int i = 0; i < kAccStages; ++i) {
      mbar_init(smem_u32(&ctrl->tmem_full[i]), 1);
      mbar_init(smem_u32(&ctrl->tmem_empty[i]), kEpilogueWarps);
    }
    mbar_init(smem_u32(&ctrl->exch_full), uint32_t(split) * kEpilogueWarps);
    mbar_init(smem_u32(&ctrl->exch_free), uint32_t(split) * kEpilogueWarps);
    ctrl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&ctrl->tmem_base)), "r"(uint32_t(kTmemCols)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  cluster_sync_all();                            // the barriers of every rank exist before anyone arrives remotely
  tcgen05_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;

  // Register re-split as in the one-CTA kernel: 128*40 + 256*232 = 384*168 exactly.
  static_assert(128 * 40 + 256 * 232 <= kNumThreads * 168, "setmaxnreg split exceeds the launch allocation");
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    const bool gather = a.a_layout != FLYMOE_ROWS_SORTED;
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      int stage = 0;
      uint32_t phase = 0;
      const uint32_t tx_bytes = uint32_t(a.tile_m) * BK + kBTileBytes;
      bool ok = true;
      for (int t = first_tile; t < sched.total && ok; t += tile_step) {
        int mb, n;
        sched.decode(t, mb, n);
        const int e = block_expert(a, mb);
        if (e < 0 || e >= a.experts) continue;
        int rows[4];
        if (gather) gather_rows4(a, mb * a.tile_m + lane * 4, min((mb + 1) * a.tile_m, valid_rows), rows);
        for (int kb = kb0; kb < kb1; ++kb) {
          ok = warp_wait(smem_u32(&ctrl->empty[stage]), phase ^ 1, abort_flag, a.status, 1, 64);
          if (!ok) break;
          const uint32_t full = smem_u32(&ctrl->full[stage]);
          const uint32_t sa = smem_u32(smem + size_t(stage) * kSplitStageBytes);
          const uint32_t sb = sa + kSplitAStage;
          if (elect_one()) {
            mbar_expect_tx(full, tx_bytes);
            if (!gather) tma_load_2d(sa, &tmap_a, full, kb * BK, mb * a.tile_m);
            if (STAGE == 1) {
              tma_load_3d(sb, &tmap_b, full, kb * BK, n * 128, e);
              tma_load_3d(sb + 128 * BK, &tmap_b, full, kb * BK, a.n_dim + n * 128, e);
            } else {
              tma_load_3d(sb, &tmap_b, full, kb * BK, n * BN, e);
            }
          }
          if (gather) {
            __syncwarp();                        // the expected byte count is set before any of it can arrive
            if (lane * 4 < a.tile_m) tma_gather4(sa + uint32_t(lane) * 512u, &tmap_a, full, kb * BK, rows);
          }
          if (++stage == kSplitStages) { stage = 0; phase ^= 1; }
        }
      }
    } else if (warp == 1) {
      // ---------------------------------------------------------------- MMA issuer
      auto issue = [&](auto kind_c, uint32_t idesc) {
        constexpr int KIND = decltype(kind_c)::value;
        int stage = 0, acc = 0;
        uint32_t phase = 0, acc_phase = 0;
        int mb = 0, n = 0, e_next = -1;                    // expert id: loaded a whole tile early
        if (int(first_tile) < sched.total) {
          sched.decode(first_tile, mb, n);
          e_next = block_expert(a, mb);
        }
        for (int t = first_tile; t < sched.total; t += tile_step) {
          const int e = e_next;
          if (t + int(tile_step) < sched.total) {
            sched.decode(t + tile_step, mb, n);
            e_next = block_expert(a, mb);
          }
          if (e < 0 || e >= a.experts) continue;
          for (int kb = kb0; kb < kb1; ++kb) {
            // per-token scaling: one accumulator stage per tile; block scaling: one per K block, started from zero
            if (SCALING == kScaleBlock128 || kb == kb0) {
              if (!warp_wait(smem_u32(&ctrl->tmem_empty[acc]), acc_phase ^ 1, abort_flag, a.status, 2)) return;
            }
            if (!warp_wait(smem_u32(&ctrl->full[stage]), phase, abort_flag, a.status, 3)) return;
            tcgen05_fence_after();
            const uint32_t sa = smem_u32(smem + size_t(stage) * kSplitStageBytes);
            const uint64_t adesc = make_smem_desc(sa);
            const uint64_t bdesc = make_smem_desc(sa + kSplitAStage);
            const uint32_t d_tmem = tmem_base + uint32_t(acc) * BN;
            const bool last = SCALING == kScaleBlock128 || kb + 1 == kb1;
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < BK / 32; ++k)
                umma<KIND>(d_tmem, adesc + uint64_t(k * 2), bdesc + uint64_t(k * 2), idesc,
                           (k > 0 || (SCALING == kScalePerToken && kb > kb0)) ? 1u : 0u);
              umma_commit(smem_u32(&ctrl->empty[stage]));
              if (last) umma_commit(smem_u32(&ctrl->tmem_full[acc]));
            }
            __syncwarp();
            if (last && ++acc == kAccStages) { acc = 0; acc_phase ^= 1; }
            if (++stage == kSplitStages) { stage = 0; phase ^= 1; }
          }
        }
      };
      if (SCALING == kScaleBlock128 || a.in_dtype == FLYMOE_E4M3) issue(std::integral_constant<int, 0>{}, kInstrDescF8);
      else if (a.in_dtype == FLYMOE_I8) issue(std::integral_constant<int, 1>{}, kInstrDescI8);
      else issue(std::integral_constant<int, 2>{}, a.in_dtype == FLYMOE_BF16 ? kInstrDescBF16 : kInstrDescF16);
    }
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    // ------------------------------------------------------------------ epilogue
    const int wg = (warp - 4) >> 2;
    const int q = warp & 3;
    const int row_in_tile = q * 32 + lane;
    const bool warp_active = q * 32 < a.tile_m;
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    int acc = 0;
    uint32_t acc_phase = 0, tile_iter = 0;
    bool ok = true;
    const uint32_t full_bar0 = smem_u32(&ctrl->tmem_full[0]);
    const uint32_t empty_bar0 = smem_u32(&ctrl->tmem_empty[0]);
    const uint32_t exch_full = smem_u32(&ctrl->exch_full), exch_free = smem_u32(&ctrl->exch_free);
    const int pad_id = (a.topk << 24) | a.num_tokens;
    const bool i8 = SCALING == kScalePerToken && a.in_dtype == FLYMOE_I8;
    const bool bf = a.out_dtype == FLYMOE_BF16;
    for (int t = first_tile; t < sched.total && ok; t += tile_step) {
      int mb, n;
      sched.decode(t, mb, n);
      const int e = block_expert(a, mb);
      if (e < 0 || e >= a.experts) continue;
      // index of a row's activation scale, -1 for pad rows
      auto scale_row = [&](int r, int id) -> long long {
        const int tok = id_token(id), slot = id_slot(id);
        if (tok >= a.num_tokens || slot >= a.topk) return -1;
        if (a.a_scale_layout == FLYMOE_ROWS_BY_TOKEN) return tok;
        if (a.a_scale_layout == FLYMOE_ROWS_BY_PAIR) return (long long)tok * a.topk + slot;
        if (SCALING == kScalePerToken && a.a_scale_layout == FLYMOE_ROWS_BY_SLOT) return (long long)slot * a.num_tokens + tok;
        return r;
      };
      auto row_id = [&](int row) {
        const int r = mb * a.tile_m + row;
        return (row < a.tile_m && r < valid_rows) ? sorted_id(a, r) : pad_id;
      };
      // ---- this rank's K blocks --------------------------------------------------------
      const bool half_ok = STAGE == 1 ? true : (n * BN + wg * 128 < a.n_dim);
      const bool work = warp_active && half_ok;
      const uint32_t tcol0 = tmem_base + lane_base + (STAGE == 1 ? uint32_t(wg * 64) : uint32_t(wg * 128));
      const uint32_t tcol1 = tmem_base + lane_base + (STAGE == 1 ? uint32_t(128 + wg * 64) : uint32_t(wg * 128 + 64));
      uint32_t part[128];                        // fp32 (int8 operands: int32) partial sums
      if (SCALING == kScaleBlock128) {
        const long long sidx = scale_row(mb * a.tile_m + row_in_tile, row_id(row_in_tile));
        const bool valid = sidx >= 0;
        const float* sa_run = a.scale_a + (valid ? sidx : 0) * a.sa_row_stride + (long long)kb0 * a.sa_stride;
        const int wblk_per_expert = (STAGE == 1 ? 2 * a.n_dim : a.n_dim + 127) / 128;
        const int blk0 = STAGE == 1 ? n : n * 2 + wg;
        const int blk1 = STAGE == 1 ? a.n_dim / 128 + n : blk0;
        const float* sw0_ptr = a.scale_w + ((long long)e * wblk_per_expert + (half_ok ? blk0 : 0)) * KB;
        const int sw1_off = (blk1 - (half_ok ? blk0 : 0)) * KB;
        unsigned long long acc2[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) acc2[j] = 0ull;
        float sa_next = valid ? __ldg(sa_run) : 0.f;
        float s0_next = __ldg(sw0_ptr + kb0);
        float s1_next = STAGE == 1 ? __ldg(sw0_ptr + kb0 + sw1_off) : 0.f;
        uint32_t v0[32], v1[32];
        for (int kb = kb0; kb < kb1; ++kb) {
          const uint32_t stage_off = uint32_t(acc) * BN;
          if (!mbar_wait(full_bar0 + uint32_t(acc) * 8u, acc_phase, abort_flag, a.status, 4)) { ok = false; break; }
          tcgen05_fence_after();
          if (work) {
            tmem_ld_x32(tcol0 + stage_off, v0);
            tmem_ld_x32(tcol0 + stage_off + 32, v1);
          }
          const unsigned long long c0 = pack_f32x2(sa_next * s0_next);
          const unsigned long long c1 = STAGE == 1 ? pack_f32x2(sa_next * s1_next) : c0;
          if (work) tmem_ld_wait();
          if (kb + 1 < kb1) {
            sa_run += a.sa_stride;
            sa_next = valid ? __ldg(sa_run) : 0.f;
            s0_next = __ldg(sw0_ptr + kb + 1);
            if (STAGE == 1) s1_next = __ldg(sw0_ptr + kb + 1 + sw1_off);
          }
          if (work) {
#pragma unroll
            for (int j = 0; j < 16; ++j) ffma2(acc2[j], v0[2 * j], v0[2 * j + 1], c0);
            tmem_ld_x32(tcol1 + stage_off, v0);
#pragma unroll
            for (int j = 0; j < 16; ++j) ffma2(acc2[16 + j], v1[2 * j], v1[2 * j + 1], c0);
            tmem_ld_x32(tcol1 + stage_off + 32, v1);
            tmem_ld_wait();
          }
          if (!work) __syncwarp();
          if (lane == 0) mbar_arrive_relaxed(empty_bar0 + uint32_t(acc) * 8u);
          if (work) {
#pragma unroll
            for (int j = 0; j < 16; ++j) ffma2(acc2[32 + j], v0[2 * j], v0[2 * j + 1], c1);
#pragma unroll
            for (int j = 0; j < 16; ++j) ffma2(acc2[48 + j], v1[2 * j], v1[2 * j + 1], c1);
          }
          acc_phase ^= uint32_t(acc);
          acc ^= 1;
        }
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          float lo, hi;
          unpack_f32x2(acc2[j], lo, hi);
          part[2 * j] = __float_as_uint(lo);
          part[2 * j + 1] = __float_as_uint(hi);
        }
      } else {
        const uint32_t stage_off = uint32_t(acc) * BN;
        if (!mbar_wait(full_bar0 + uint32_t(acc) * 8u, acc_phase, abort_flag, a.status, 4)) { ok = false; break; }
        tcgen05_fence_after();
        if (work) {
          tmem_ld_x32(tcol0 + stage_off, part);
          tmem_ld_x32(tcol0 + stage_off + 32, part + 32);
          tmem_ld_x32(tcol1 + stage_off, part + 64);
          tmem_ld_x32(tcol1 + stage_off + 32, part + 96);
          tmem_ld_wait();
        } else {
          __syncwarp();
        }
        if (lane == 0) mbar_arrive_relaxed(empty_bar0 + uint32_t(acc) * 8u);
        acc_phase ^= uint32_t(acc);
        acc ^= 1;
      }
      // ---- exchange ----------------------------------------------------------------------
      if (!mbar_wait_cluster(exch_free, (tile_iter & 1) ^ 1, abort_flag, a.status, 7)) { ok = false; break; }
      if (work && row_in_tile < a.tile_m) {
        uint8_t* row = exch + size_t(row_in_tile) * kExchPitch;
        const int col0 = STAGE == 1 ? wg * 64 : wg * 128, col1 = STAGE == 1 ? 128 + wg * 64 : wg * 128 + 64;
#pragma unroll
        for (int j = 0; j < 64; j += 4) {
          *reinterpret_cast<uint4*>(row + (col0 + j) * 4) = make_uint4(part[j], part[j + 1], part[j + 2], part[j + 3]);
          *reinterpret_cast<uint4*>(row + (col1 + j) * 4) =
              make_uint4(part[64 + j], part[64 + j + 1], part[64 + j + 2], part[64 + j + 3]);
        }
      }
      __syncwarp();
      if (lane < split) mbar_arrive_rank(exch_full, uint32_t(lane));
      if (!mbar_wait_cluster(exch_full, tile_iter & 1, abort_flag, a.status, 5)) { ok = false; break; }
      // ---- rows rank, rank + S, ... : one warp per row, lane l owns columns 4l..4l+3 of both halves ----
      for (int row = rank + split * (warp - 4); row < a.tile_m; row += split * kEpilogueWarps) {
        const int r = mb * a.tile_m + row;
        const int id = row_id(row);
        const int tok = id_token(id), slot = id_slot(id);
        const bool valid = tok < a.num_tokens && slot < a.topk;
        float f[8];                              // first half (stage 1: gate), second half (up)
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = 0.f;
        if (valid) {
          const uint32_t at = smem_u32(exch + size_t(row) * kExchPitch) + uint32_t(lane) * 16u;
          int isum[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) isum[j] = 0;
#pragma unroll 4
          for (int s = 0; s < split; ++s) {
            const uint32_t ra = map_to_rank(at, uint32_t(s));
            const uint4 x = ld_cluster_v4(ra), y = ld_cluster_v4(ra + 512u);
            const uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (SCALING == kScalePerToken && i8) isum[j] += int(w[j]);
              else f[j] += __uint_as_float(w[j]);
            }
          }
          if (SCALING == kScalePerToken) {
            if (i8) {
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = __int2float_rn(isum[j]);
            }
            const float sa = row_scale(a.scale_a, scale_row(r, id));
            const long long wrows = STAGE == 1 ? 2LL * a.n_dim : (long long)a.n_dim;
            const float* sw = a.scale_w + (long long)e * wrows + (STAGE == 1 ? n * 128 : n * BN) + lane * 4;
            const bool second = STAGE == 1 || n * BN + 128 + lane * 4 < a.n_dim;
            const float4 s0 = col_scales4(a.scale_w, sw);
            const float4 s1 = second ? col_scales4(a.scale_w, sw + (STAGE == 1 ? a.n_dim : 128)) : s0;
            const float c[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] *= sa * c[j];
          }
        }
        const float wgt = (a.doweight && valid) ? __ldg(a.sorted_weights + r) : 1.f;
        if (STAGE == 1 && SCALING == kScalePerToken && a.out_dtype == FLYMOE_F32) {
          if (valid) {
            float* og = static_cast<float*>(a.out) + ((long long)tok * a.topk + slot) * (2LL * a.n_dim) +
                        (long long)n * 128 + lane * 4;
            red_add_v4_f32(og, f[0], f[1], f[2], f[3]);
            red_add_v4_f32(og + a.n_dim, f[4], f[5], f[6], f[7]);
          }
        } else if (STAGE == 1) {
          float h[4], amax = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            h[j] = f[j] * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * f[j])) * (f[4 + j] * wgt);
            amax = fmaxf(amax, fabsf(h[j]));
          }
          const long long orow = a.out_layout == FLYMOE_ROWS_SORTED ? (long long)r : (long long)tok * a.topk + slot;
          const long long ocol = (long long)n * 128 + lane * 4;
          if (a.out_dtype == FLYMOE_E4M3) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            if (valid || (r < valid_rows && a.out_layout == FLYMOE_ROWS_SORTED)) {
              float sc = __fdiv_rn(valid ? amax : 0.f, 448.0f);
              if (sc == 0.f) sc = 1.f;
              const float inv = __fdiv_rn(1.0f, sc);
              const uint32_t pk = valid ? float4_to_e4m3x4(h[0] * inv, h[1] * inv, h[2] * inv, h[3] * inv) : 0u;
              *reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(a.out) + orow * a.n_dim + ocol) = pk;
              if (lane == 0) a.out_scale[(long long)n * a.out_scale_stride + orow] = sc;
            }
          } else if (valid) {
            uint2 pk;
            pk.x = bf ? pack_bf16x2(h[0], h[1]) : pack_f16x2(h[0], h[1]);
            pk.y = bf ? pack_bf16x2(h[2], h[3]) : pack_f16x2(h[2], h[3]);
            *reinterpret_cast<uint2*>(static_cast<uint8_t*>(a.out) + (orow * a.n_dim + ocol) * 2) = pk;
          }
        } else if (valid) {
          const long long orow = a.accumulate ? (long long)tok : (long long)tok * a.topk + slot;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int col = n * BN + h * 128 + lane * 4;
            if (col >= a.n_dim) continue;
            const float x0 = f[h * 4] * wgt, x1 = f[h * 4 + 1] * wgt, x2 = f[h * 4 + 2] * wgt, x3 = f[h * 4 + 3] * wgt;
            if (a.out_dtype == FLYMOE_F32) {
              red_add_v4_f32(static_cast<float*>(a.out) + orow * a.n_dim + col, x0, x1, x2, x3);
              continue;
            }
            uint8_t* op = static_cast<uint8_t*>(a.out) + (orow * a.n_dim + col) * 2;
            const uint32_t lo = bf ? pack_bf16x2(x0, x1) : pack_f16x2(x0, x1);
            const uint32_t hi = bf ? pack_bf16x2(x2, x3) : pack_f16x2(x2, x3);
            if (a.accumulate) red_add_2x16(op, lo, hi, bf);
            else *reinterpret_cast<uint2*>(op) = make_uint2(lo, hi);
          }
        }
      }
      __syncwarp();
      if (lane < split) mbar_arrive_rank(exch_free, uint32_t(lane));
      ++tile_iter;
    }
    __syncwarp();
  }

  tcgen05_fence_before();
  cluster_sync_all();                            // no rank leaves while its partial sums may still be read
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemCols))
                 : "memory");
  }
}

// ------------------------------------------------------------------------------ host
template <int STAGE, int SCALING>
static cudaLaunchConfig_t split_config(int split, cudaLaunchAttribute* attr) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = unsigned(split);
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kNumThreads);
  cfg.gridDim = dim3(unsigned(split));
  cfg.dynamicSmemBytes = kSplitSmem;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Clusters of `split` CTAs that fit on the GPU at once (asked for once per device and cluster size); 0 where such a
// cluster cannot be scheduled at all, as in a context limited to part of the GPU.
template <int STAGE, int SCALING>
static int resident_clusters(int dev, int split) {
  static std::atomic<int> known[64][9];                    // answer + 1
  int n = known[dev][split].load(std::memory_order_relaxed) - 1;
  if (n >= 0) return n;
  auto* kernel = moe_gemm_split_kernel<STAGE, SCALING>;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = split_config<STAGE, SCALING>(split, &attr);
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSplitSmem)) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  known[dev][split].store(n + 1, std::memory_order_relaxed);
  return n;
}

template <int STAGE, int SCALING>
static int launch_split(const GemmArgs& a, const CUtensorMap& map_a, const CUtensorMap& map_b, int group_m, int split,
                        cudaStream_t stream) {
  auto* kernel = moe_gemm_split_kernel<STAGE, SCALING>;
  FLYMOE_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSplitSmem)));
  const int ntiles = STAGE == 1 ? a.n_dim / 128 : ceil_div(a.n_dim, BN);
  const long long tiles = (long long)a.size_expert_ids * ntiles;
  int dev = 0;
  FLYMOE_CUDA_CHECK(cudaGetDevice(&dev));
  const int resident = resident_clusters<STAGE, SCALING>(dev, split);    // at least one, or the plan would not say `split`
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = split_config<STAGE, SCALING>(split, &attr);
  cfg.gridDim = dim3(unsigned((tiles < resident ? int(tiles) : resident) * split));
  cfg.stream = stream;
  FLYMOE_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, a, group_m, split));
  return FLYMOE_OK;
}

int launch_gemm_split(int stage, const GemmArgs& a, const CUtensorMap& map_a, const CUtensorMap& map_b, int group_m,
                      int split, cudaStream_t stream) {
  if (a.scaling == FLYMOE_SCALE_PER_TOKEN)
    return stage == 1 ? launch_split<1, kScalePerToken>(a, map_a, map_b, group_m, split, stream)
                      : launch_split<2, kScalePerToken>(a, map_a, map_b, group_m, split, stream);
  return stage == 1 ? launch_split<1, kScaleBlock128>(a, map_a, map_b, group_m, split, stream)
                    : launch_split<2, kScaleBlock128>(a, map_a, map_b, group_m, split, stream);
}

void split_residency(int stage, int scaling, int* clusters) {
  int dev = 0;
  const bool known = cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64;
  for (int i = 1, s = 2; i < kClusterSizes; ++i, s *= 2)
    clusters[i] = !known ? 0
                : scaling == FLYMOE_SCALE_PER_TOKEN
                    ? (stage == 1 ? resident_clusters<1, kScalePerToken>(dev, s) : resident_clusters<2, kScalePerToken>(dev, s))
                    : (stage == 1 ? resident_clusters<1, kScaleBlock128>(dev, s) : resident_clusters<2, kScaleBlock128>(dev, s));
}

int plan_ksplit(int stage, const GemmArgs& a, const int* clusters) {
  if (a.tile_m > kSplitMaxRows || a.row_dst != nullptr) return 1;
  const int KB = a.k_dim / BK;
  const long long pairs = (long long)a.num_tokens * a.topk;
  // most row blocks the routing can produce: every block holds at least one (token, slot) pair
  const long long blocks = pairs < a.size_expert_ids ? pairs : a.size_expert_ids;
  const long long tiles = blocks * (stage == 1 ? a.n_dim / 128 : ceil_div(a.n_dim, BN));
  // Rounds of tiles times the K blocks of one round, plus the fixed part of a round (pipeline fill, tile end,
  // exchange) in K blocks.  A larger cluster has to win by a tenth, so that launches that fill the GPU anyway
  // stay with the kernel that has no exchange.
  int best = 1;
  double best_cost = 1e30;
  for (int i = 0, s = 1; i < kClusterSizes && s <= KB; ++i, s *= 2) {
    // Clusters do not cross GPCs: 148 SMs ran 74 of 2, 33 of 4 and 15 of 8 at once.  Counting SMs / 8 = 18 instead, the
    // 18 tiles of a dense M=64 N=4608 K=7168 were planned as one round of 8 and ran as two: 26.1 us, 18.4 as one of 4.
    const long long slots = clusters[i];
    if (slots < 1) continue;
    const double rounds = double((tiles + slots - 1) / slots);
    const double cost = rounds * (double((KB + s - 1) / s) + (s == 1 ? 3.0 : 5.0));
    if (cost < 0.9 * best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

}  // namespace flymoe
