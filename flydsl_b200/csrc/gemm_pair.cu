// Grouped GEMM on CTA pairs (tcgen05 cta_group::2) for per-token scaling and experts with many rows.
//
// Two CTAs of one cluster share a tile of 256 sorted rows x 256 weight rows: each brings its own 128 rows of
// activations and HALF of the weight tile into shared memory (32 KB per 128-byte-wide K block instead of 48 KB), and
// the pair's leader issues M=256 N=256 MMAs that read both halves.  With one scale per row and column the MMAs
// accumulate over the whole K range, so the tensor cores are the bound once the operands arrive: 48 KB per K block
// are 768 cycles at the 64 bytes a cycle an SM takes from L2, 32 KB are the 512 the MMAs need.
//   warp 0      TMA producer: this CTA's A rows (one or two boxes of a row block x 128 B) and 128 weight rows x 128 B
//               per K block.  The loads of both CTAs complete on the leader's full barrier.
//   warp 1      (leader) MMA issuer: four M=256 N=256 MMAs per K block into one of two TMEM stages.
//   warp 2      store warp: one bulk store / bulk reduction per finished output row.
//   warps 4-19  epilogue: four warpgroups; each thread owns one row and 2 x 32 of the tile's columns.
// Measured on one B200 (bench.py --tokens 2048 --experts 8 --scaling pertoken --tile-m 128 [--in-dtype bf16]; 16384 rows,
// 4096 x 7168 and 7168 x 2048): fp8 333 us (2887 TFLOP/s) and 212 us (2273) against 355 and 315 for the one-CTA kernel,
// bf16 654 us (1470 TFLOP/s) and 352 us (1367) against 702 and 422.  Block scaling stays with the one-CTA kernel: there the
// epilogue is the bound (a 16-warp variant of this kernel took 245 us against 242, and the T=4096 layer, whose 256-row
// tiles are half empty, 4.5 ms against 3.4).
//
// Column order.  The leader's 128 weight rows are the tile's first block (stage 1: gate; stage 2: columns 0-127),
// the other CTA's are its second block (up; columns 128-255); a thread owns the same 32 columns of both, so gate and
// up of an output column meet in one thread.
//
// An expert's row blocks (of 64 or 128 rows) are contiguous in sorted order, so its rows are cut into tiles of 256
// whatever the block size; the table of tiles is derived from sorted_expert_ids at kernel start.  A last tile of at
// most 128 rows runs without the second CTA's rows.
//
// Every wait is bounded as in gemm_sm100.cu; both CTAs meet once more before they exit.
#include <cuda.h>
#include <type_traits>

#include "common.cuh"
#include "gemm_args.cuh"
#include "gemm_ptx.cuh"

namespace flymoe {

constexpr int kPairThreads = 640;
constexpr int kPairEpiWarps = 16;
constexpr int kPairStageBytes = kATileBytes + kBTileBytes / 2;      // 32 KB per CTA and K block
template <int STAGE> struct PairCfg {
  static constexpr int ring = STAGE == 1 ? 6 : 4;
  // stage 2: finished output rows, 256 16-bit results; 16 bytes of skew against bank conflicts
  static constexpr int pitch = STAGE == 1 ? 0 : 528;
};

struct __align__(16) PairCtrl {
  unsigned long long full[6];                   // leader's: both CTAs' operands of a K block have landed
  unsigned long long empty[6];
  unsigned long long acc_full[2];               // [TMEM stage]
  unsigned long long acc_empty[2];              // leader's: the epilogue warps of both CTAs have read the stage
  unsigned long long stg_full;
  unsigned long long stg_free;
  unsigned long long stg_dst[BM];
  uint32_t tmem_base;
  int abort_flag;
  int scan[2][32];
  uint16_t table[kTileTable];                   // see build_tile_table
};
template <int STAGE> constexpr size_t pair_smem() {
  return size_t(PairCfg<STAGE>::ring) * kPairStageBytes + size_t(BM) * PairCfg<STAGE>::pitch + sizeof(PairCtrl) + 1024;
}
static_assert(pair_smem<1>() <= 232448 && pair_smem<2>() <= 232448, "shared memory budget of one SM exceeded");

__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1,
                                                 int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void mbar_arrive_relaxed_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// KIND: 0 = f8f6f4, 1 = i8, 2 = f16
template <int KIND>
__device__ __forceinline__ void umma_pair(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  if (KIND == 0)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(acc) : "memory");
  else if (KIND == 1)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(acc) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(ad), "l"(bd), "r"(idesc), "r"(acc) : "memory");
}
// Arrives on the barrier at this shared-memory offset in both CTAs once the MMAs issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(uint16_t(3)) : "memory");
}

template <int STAGE>
__global__ void __launch_bounds__(kPairThreads, 1)
moe_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const GemmArgs a, const int group_m) {
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  constexpr int kRing = PairCfg<STAGE>::ring;
  constexpr int kPitch = PairCfg<STAGE>::pitch;
  uint8_t* staging = smem + size_t(kRing) * kPairStageBytes;
  PairCtrl* ctrl = reinterpret_cast<PairCtrl*>(staging + size_t(BM) * kPitch);
  volatile int* abort_flag = &ctrl->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int KB = a.k_dim / BK;
  const int rank = int(cluster_rank());
  const int valid_rows = min(__ldg(a.num_valid_ids), a.size_expert_ids * a.tile_m);
  const bool uses_staging = STAGE == 2 && a.out_dtype != FLYMOE_F32;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(smem_u32(&ctrl->full[i]), 1);                    // the leader's producer
      mbar_init(smem_u32(&ctrl->empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&ctrl->acc_full[i]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[i]), 2 * kPairEpiWarps);
    }
    mbar_init(smem_u32(&ctrl->stg_full), kPairEpiWarps);
    mbar_init(smem_u32(&ctrl->stg_free), 1);
    ctrl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&ctrl->tmem_base)), "r"(uint32_t(kTmemCols)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  const int num_tiles = build_tile_table<kPairThreads>(a, valid_rows, 2 * BM / a.tile_m, ctrl->table, ctrl->scan);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();                            // both CTAs' barriers and TMEM exist
  tcgen05_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;

  TileSched sched;
  sched.num_mblocks = num_tiles;
  sched.num_ntiles = STAGE == 1 ? a.n_dim / 128 : (a.n_dim + BN - 1) / BN;
  sched.total = sched.num_mblocks * sched.num_ntiles;
  sched.group_m = group_m;
  const int first_tile = int(blockIdx.x) >> 1, tile_step = int(gridDim.x) >> 1;
  // tile -> N tile, expert, this CTA's first sorted row and how many rows it has
  auto tile_at = [&](int t, int& n, int& e, int& rows, int* other_rows = nullptr) -> int {
    int p;
    sched.decode(t, p, n);
    const uint32_t entry = ctrl->table[p];
    const int b = int(entry & 0xfff);
    e = __ldg(a.sorted_expert_ids + b);
    rows = pair_rows(int(entry >> 12) + 1, a.tile_m, rank);
    if (other_rows) *other_rows = pair_rows(int(entry >> 12) + 1, a.tile_m, 1 - rank);
    return b * a.tile_m + rank * BM;
  };

  // Register re-split: 640 threads x 96 registers are allocated at launch; 128 x 32 + 512 x 112 fit in them
  // (a larger request would wait forever for registers that are never released).
  static_assert(128 * 32 + 512 * 112 <= kPairThreads * 96, "setmaxnreg split exceeds the launch allocation");
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
    if (warp == 0) {
      // ---------------------------------------------------------------- TMA producer
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = first_tile; t < sched.total && ok; t += tile_step) {
        int n, e, rows, other_rows;
        const int row0 = tile_at(t, n, e, rows, &other_rows);
        const int wrow = STAGE == 1 ? rank * a.n_dim + n * 128 : n * BN + rank * 128;
        // The leader announces the bytes of both CTAs on its barrier (an arrival from the other CTA that names its own
        // share needs release or relaxed semantics at cluster scope; the release alone took ~1500 cycles a K block).
        // The other CTA's bytes may land before the announcement: the phase still waits for the leader's arrival.
        // The activations come in boxes of one row block: a 128-row box would read up to 64 rows past the last block.
        const uint32_t tx_bytes = uint32_t(kBTileBytes) + uint32_t(rows + other_rows) * BK;
        for (int kb = 0; kb < KB; ++kb) {
          ok = warp_wait(smem_u32(&ctrl->empty[stage]), phase ^ 1, abort_flag, a.status, 1, 32);
          if (!ok) break;
          const uint32_t full = map_to_rank(smem_u32(&ctrl->full[stage]), 0);
          const uint32_t sa = smem_u32(smem + size_t(stage) * kPairStageBytes);
          if (elect_one()) {
            if (rank == 0) mbar_expect_tx(smem_u32(&ctrl->full[stage]), tx_bytes);
            if (rows > 0) tma_load_2d_pair(sa, &tmap_a, full, kb * BK, row0);
            if (rows > a.tile_m) tma_load_2d_pair(sa + uint32_t(a.tile_m) * BK, &tmap_a, full, kb * BK, row0 + a.tile_m);
            tma_load_3d_pair(sa + kATileBytes, &tmap_b, full, kb * BK, wrow, e);
          }
          __syncwarp();
          if (++stage == kRing) { stage = 0; phase ^= 1; }
        }
      }
      // Nothing else waits for the last releases of the ring, which are the leader's MMAs arriving in BOTH CTAs: they have
      // to land before this CTA's shared memory goes away.
      for (int i = 0; i < kRing && ok; ++i) {
        ok = warp_wait(smem_u32(&ctrl->empty[stage]), phase ^ 1, abort_flag, a.status, 1, 32);
        if (++stage == kRing) { stage = 0; phase ^= 1; }
      }
    } else if (warp == 1 && rank == 0) {
      // ---------------------------------------------------------------- MMA issuer
      auto issue = [&](auto kind_c, uint32_t dtype_bits) {
        constexpr int KIND = decltype(kind_c)::value;
        const uint32_t idesc = dtype_bits | uint32_t(BN >> 3) << 17 | uint32_t(256 >> 4) << 24;
        int stage = 0, acc = 0;
        uint32_t phase = 0, acc_phase = 0;
        for (int t = first_tile; t < sched.total; t += tile_step) {
          for (int kb = 0; kb < KB; ++kb) {
            if (kb == 0 && !warp_wait(smem_u32(&ctrl->acc_empty[acc]), acc_phase ^ 1, abort_flag, a.status, 2)) return;
            if (!__all_sync(0xffffffffu, mbar_wait_cluster(smem_u32(&ctrl->full[stage]), phase, abort_flag, a.status, 3))) return;
            const uint32_t sa = smem_u32(smem + size_t(stage) * kPairStageBytes);
            const uint64_t adesc = make_smem_desc(sa);
            const uint64_t bdesc = make_smem_desc(sa + kATileBytes);
            const uint32_t d_tmem = tmem_base + uint32_t(acc) * BN;
            tcgen05_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < BK / 32; ++k)
                umma_pair<KIND>(d_tmem, adesc + uint64_t(k * 2), bdesc + uint64_t(k * 2), idesc, (k > 0 || kb > 0) ? 1u : 0u);
              umma_commit_pair(smem_u32(&ctrl->empty[stage]));
              if (kb + 1 == KB) umma_commit_pair(smem_u32(&ctrl->acc_full[acc]));
            }
            __syncwarp();
            if (kb + 1 == KB && ++acc == 2) { acc = 0; acc_phase ^= 1; }
            if (++stage == kRing) { stage = 0; phase ^= 1; }
          }
        }
      };
      if (a.in_dtype == FLYMOE_E4M3) issue(std::integral_constant<int, 0>{}, kInstrDescF8 - kInstrDescShape);
      else if (a.in_dtype == FLYMOE_I8) issue(std::integral_constant<int, 1>{}, kInstrDescI8 - kInstrDescShape);
      else issue(std::integral_constant<int, 2>{}, (a.in_dtype == FLYMOE_BF16 ? kInstrDescBF16 : kInstrDescF16) - kInstrDescShape);
    } else if (warp == 2 && uses_staging) {
      // ---------------------------------------------------------------- store warp
      bool ok = true;
      uint32_t it = 0;
      const bool bf = a.out_dtype == FLYMOE_BF16;
      for (int t = first_tile; t < sched.total && ok; t += tile_step) {
        int n, e, rows;
        tile_at(t, n, e, rows);
        if (rows <= 0) continue;
        if (!mbar_wait(smem_u32(&ctrl->stg_full), it & 1, abort_flag, a.status, 6, 64)) { ok = false; break; }
        const uint32_t bytes = uint32_t(min(BN, a.n_dim - n * BN)) * 2u;
#pragma unroll
        for (int i = 0; i < BM / 32; ++i) {
          const int row = i * 32 + lane;
          const unsigned long long dst = ctrl->stg_dst[row];
          if (dst != 0ull) {
            const uint32_t sp = smem_u32(staging + size_t(row) * kPitch);
            void* gp = reinterpret_cast<void*>(dst);
            if (!a.accumulate) bulk_store(gp, sp, bytes);
            else if (bf) bulk_reduce_add_bf16(gp, sp, bytes);
            else bulk_reduce_add_f16(gp, sp, bytes);
          }
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        bulk_wait_read_all();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->stg_free));
        ++it;
      }
      bulk_wait_all();
    }
    __syncwarp();
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    // ------------------------------------------------------------------ epilogue
    const int wg = (warp - 4) >> 2;              // 0..3
    const int row = (warp & 3) * 32 + lane;      // TMEM lane = row of this CTA's block
    int acc = 0;
    uint32_t acc_phase = 0, tile_iter = 0;
    bool ok = true;
    const uint32_t tcol = tmem_base + (uint32_t((warp & 3) * 32) << 16) + uint32_t(wg * 32);
    const uint32_t full_bar = smem_u32(&ctrl->acc_full[0]);                      // the other stage's: + 8 bytes
    const uint32_t empty_bar = map_to_rank(smem_u32(&ctrl->acc_empty[0]), 0);
    const int pad_id = (a.topk << 24) | a.num_tokens;
    for (int t = first_tile; t < sched.total && ok; t += tile_step) {
      int n, e, rows;
      const int row0 = tile_at(t, n, e, rows);
      const bool work = rows > 0;
      float v1[32], v2[32];                      // results: first block, second block
      if (!mbar_wait(full_bar + uint32_t(acc) * 8u, acc_phase, abort_flag, a.status, 4)) { ok = false; break; }
      tcgen05_fence_after();
      const uint32_t tc = tcol + uint32_t(acc) * BN;
      if (work) {
        tmem_ld_x32(tc, reinterpret_cast<uint32_t*>(v1));
        tmem_ld_x32(tc + 128, reinterpret_cast<uint32_t*>(v2));
        tmem_ld_wait();
      } else {
        __syncwarp();
      }
      if (lane == 0) mbar_arrive_relaxed_cluster(empty_bar + uint32_t(acc) * 8u);
      acc_phase ^= uint32_t(acc);
      acc ^= 1;
      if (!work) continue;

      // ---- tile epilogue -----------------------------------------------------------
      const int r = row0 + row;
      const bool in_tile = row < rows && r < valid_rows;
      const int id = in_tile ? __ldg(a.sorted_ids + r) : pad_id;
      const int tok = id_token(id), slot = id_slot(id);
      const bool valid = tok < a.num_tokens && slot < a.topk;
      const int col1 = wg * 32;                  // column of v1[0] within the first block, of v2[0] within the second
      {
        const bool i8 = a.in_dtype == FLYMOE_I8;
        float sa = 0.f;
        if (valid) {
          const long long sidx = a.a_scale_layout == FLYMOE_ROWS_BY_TOKEN ? (long long)tok
                               : a.a_scale_layout == FLYMOE_ROWS_BY_PAIR ? (long long)tok * a.topk + slot
                               : a.a_scale_layout == FLYMOE_ROWS_BY_SLOT ? (long long)slot * a.num_tokens + tok : (long long)r;
          sa = row_scale(a.scale_a, sidx);
        }
        const long long wrows = STAGE == 1 ? 2LL * a.n_dim : (long long)a.n_dim;
        const float* sw1 = a.scale_w + (long long)e * wrows + (STAGE == 1 ? n * 128 : n * BN) + col1;
        const float* sw2 = sw1 + (STAGE == 1 ? a.n_dim : 128);
        const bool has2 = STAGE == 1 || n * BN + 128 < a.n_dim;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 s4 = col_scales4(a.scale_w, sw1 + j);
          const float4 u4 = has2 ? col_scales4(a.scale_w, sw2 + j) : s4;
          const float c[4] = {s4.x, s4.y, s4.z, s4.w}, d[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float p = i8 ? __int2float_rn(__float_as_int(v1[j + u])) : v1[j + u];
            const float w = i8 ? __int2float_rn(__float_as_int(v2[j + u])) : v2[j + u];
            v1[j + u] = valid ? p * (sa * c[u]) : 0.f;
            v2[j + u] = valid ? w * (sa * d[u]) : 0.f;
          }
          asm volatile("" ::: "memory");         // keeps the scale loads from being hoisted in front of the math
        }
      }
      const float wgt = (a.doweight && valid) ? __ldg(a.sorted_weights + r) : 1.f;
      const bool bf = a.out_dtype == FLYMOE_BF16;
      if (STAGE == 1 && a.out_dtype == FLYMOE_F32) {
        // the split-K output contract: raw gate and up sums, added to out[t*topk+s][0:I | I:2I]
        if (valid) {
          float* og = static_cast<float*>(a.out) + ((long long)tok * a.topk + slot) * (2LL * a.n_dim) + (long long)n * 128 + col1;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            red_add_v4_f32(og + j, v1[j], v1[j + 1], v1[j + 2], v1[j + 3]);
            red_add_v4_f32(og + a.n_dim + j, v2[j], v2[j + 1], v2[j + 2], v2[j + 3]);
          }
        }
      } else if (STAGE == 1) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          v1[j] = v1[j] * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * v1[j])) * (v2[j] * wgt);
        const long long orow = a.out_layout == FLYMOE_ROWS_SORTED ? (long long)r : (long long)tok * a.topk + slot;
        const long long ocol = (long long)n * 128 + col1;
        if (valid) {
          uint8_t* op = static_cast<uint8_t*>(a.out) + (orow * a.n_dim + ocol) * 2;
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint4 pk;
            pk.x = bf ? pack_bf16x2(v1[j + 0], v1[j + 1]) : pack_f16x2(v1[j + 0], v1[j + 1]);
            pk.y = bf ? pack_bf16x2(v1[j + 2], v1[j + 3]) : pack_f16x2(v1[j + 2], v1[j + 3]);
            pk.z = bf ? pack_bf16x2(v1[j + 4], v1[j + 5]) : pack_f16x2(v1[j + 4], v1[j + 5]);
            pk.w = bf ? pack_bf16x2(v1[j + 6], v1[j + 7]) : pack_f16x2(v1[j + 6], v1[j + 7]);
            *reinterpret_cast<uint4*>(op + j * 2) = pk;
          }
        }
      } else if (a.out_dtype == FLYMOE_F32) {
        if (valid) {
          float* op = static_cast<float*>(a.out) + (long long)tok * a.n_dim + (long long)n * BN + col1;
          const bool has2 = n * BN + 128 < a.n_dim;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            red_add_v4_f32(op + j, v1[j] * wgt, v1[j + 1] * wgt, v1[j + 2] * wgt, v1[j + 3] * wgt);
            if (has2) red_add_v4_f32(op + 128 + j, v2[j] * wgt, v2[j + 1] * wgt, v2[j + 2] * wgt, v2[j + 3] * wgt);
          }
        }
      } else {
        // 16-bit output: the row's 256 results meet in its staging slot and leave as ONE bulk reduce-add or store
        if (!mbar_wait(smem_u32(&ctrl->stg_free), (tile_iter & 1) ^ 1, abort_flag, a.status, 7)) { ok = false; break; }
        if (valid) {
          uint8_t* op = staging + size_t(row) * kPitch + col1 * 2;
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            uint4 pk, p2;
            pk.x = bf ? pack_bf16x2(v1[j] * wgt, v1[j + 1] * wgt) : pack_f16x2(v1[j] * wgt, v1[j + 1] * wgt);
            pk.y = bf ? pack_bf16x2(v1[j + 2] * wgt, v1[j + 3] * wgt) : pack_f16x2(v1[j + 2] * wgt, v1[j + 3] * wgt);
            pk.z = bf ? pack_bf16x2(v1[j + 4] * wgt, v1[j + 5] * wgt) : pack_f16x2(v1[j + 4] * wgt, v1[j + 5] * wgt);
            pk.w = bf ? pack_bf16x2(v1[j + 6] * wgt, v1[j + 7] * wgt) : pack_f16x2(v1[j + 6] * wgt, v1[j + 7] * wgt);
            p2.x = bf ? pack_bf16x2(v2[j] * wgt, v2[j + 1] * wgt) : pack_f16x2(v2[j] * wgt, v2[j + 1] * wgt);
            p2.y = bf ? pack_bf16x2(v2[j + 2] * wgt, v2[j + 3] * wgt) : pack_f16x2(v2[j + 2] * wgt, v2[j + 3] * wgt);
            p2.z = bf ? pack_bf16x2(v2[j + 4] * wgt, v2[j + 5] * wgt) : pack_f16x2(v2[j + 4] * wgt, v2[j + 5] * wgt);
            p2.w = bf ? pack_bf16x2(v2[j + 6] * wgt, v2[j + 7] * wgt) : pack_f16x2(v2[j + 6] * wgt, v2[j + 7] * wgt);
            *reinterpret_cast<uint4*>(op + j * 2) = pk;
            *reinterpret_cast<uint4*>(op + 256 + j * 2) = p2;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        if (wg == 0) {
          const long long orow = a.accumulate ? (long long)tok : (long long)tok * a.topk + slot;
          ctrl->stg_dst[row] = valid ? reinterpret_cast<unsigned long long>(static_cast<uint8_t*>(a.out) +
                                                                            (orow * a.n_dim + (long long)n * BN) * 2)
                                     : 0ull;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->stg_full));
      }
      ++tile_iter;
    }
    __syncwarp();
  }

  tcgen05_fence_before();
  cluster_sync_all();                            // no remote arrival or MMA is outstanding when a CTA leaves
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemCols))
                 : "memory");
  }
}

// ------------------------------------------------------------------------------ host
template <int STAGE>
static int launch_pair(const GemmArgs& a, const CUtensorMap& map_a, const CUtensorMap& map_b, int group_m, int clusters,
                       cudaStream_t stream) {
  auto* kernel = moe_gemm_pair_kernel<STAGE>;
  FLYMOE_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(pair_smem<STAGE>())));
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kPairThreads);
  cfg.gridDim = dim3(unsigned(clusters) * 2);
  cfg.dynamicSmemBytes = pair_smem<STAGE>();
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  FLYMOE_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, map_a, map_b, a, group_m));
  return FLYMOE_OK;
}

// Per-token scaling, rows in sorted order, and experts that nearly fill a 128-row half on average: below that the second
// CTA of most pairs idles, above it the one-CTA kernel needs a second tile.  Both stages with their gathers against the
// one-CTA kernel, even routing, experts of 4096 x 2048, 7168 x 2048, 4096 x 14336 and 2048 x 1024, fp8 and bf16, 64- and
// 128-row blocks: 96 and 112 rows per expert 0.96-1.19 of its time (384 tokens, 8 experts of 4096 x 14336: 329 us there,
// 390 here), 120 rows 0.90-1.04, 128 rows 0.84-1.00, 136 rows 0.80-0.89, 512 rows 0.80-0.95.
bool use_pair_kernel(const GemmArgs& a) {
  if (a.scaling != FLYMOE_SCALE_PER_TOKEN || a.tile_m < 64 || a.a_layout != FLYMOE_ROWS_SORTED) return false;
  if (a.size_expert_ids > kTileTable) return false;
  return (long long)a.num_tokens * a.topk >= 120LL * a.experts;
}

int launch_gemm_pair(int stage, const GemmArgs& a, int ctas, cudaStream_t stream) {
  CUtensorMap map_a, map_b;
  const int rc = make_gemm_maps(stage, a, a.tile_m, 128, &map_a, &map_b);
  if (rc != FLYMOE_OK) return rc;
  // consecutive tiles (running at the same time) share one expert's weight tile
  const long long g = ((long long)a.num_tokens * a.topk + 2LL * BM * a.experts - 1) / (2LL * BM * a.experts);
  // at least 2: an expert with a few rows beyond its first tile would otherwise stream its weights (more than L2 holds)
  // once per tile.  1024 tokens, 8 experts of 4096 x 14336, top-2, bf16: 1143 -> 1078 us; 4 is no better than 2.
  const int group_m = int(g < 2 ? 2 : (g > 8 ? 8 : g));
  const int ntiles = stage == 1 ? a.n_dim / 128 : ceil_div(a.n_dim, BN);
  const long long max_tiles = (long long)a.size_expert_ids * ntiles;
  int clusters = ctas / 2;
  if (max_tiles < clusters) clusters = int(max_tiles);
  return stage == 1 ? launch_pair<1>(a, map_a, map_b, group_m, clusters, stream)
                    : launch_pair<2>(a, map_a, map_b, group_m, clusters, stream);
}

}  // namespace flymoe
