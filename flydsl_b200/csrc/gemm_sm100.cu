// Grouped FP8 (e4m3) GEMM for both MoE stages on sm_100a.
//
// One persistent CTA per SM walks a static sequence of (sorted row block, N tile)
// tiles.  Warp roles (384 threads):
//   warp 0      TMA producer: per 128-wide K block one A box (tile_m sorted rows x 128 B)
//               and 256 weight rows x 128 B into a 4-deep (stage 2: 3-deep) shared-memory
//               ring (128-byte swizzle, K-major).
//   warp 1      MMA issuer: four tcgen05.mma (M=128, N=256, K=32) per K block into one of
//               two 256-column TMEM accumulator stages; tcgen05.commit releases the smem
//               stage and publishes the TMEM stage.
//   warp 2      store warp: sends the finished rows that the epilogue threads parked in
//               shared-memory slots to global memory as bulk stores / bulk reductions
//               (one per slot), so their issue cost is off the epilogue's path.
//   warp 3      row gather (only when the activations are not in sorted-row order): copies the
//               tile's A rows, picked through the sorted-id list, into the ring with cp.async
//               (16 bytes per request, the 128-byte swizzle applied by hand), two K blocks in
//               flight; the TMA producer then fetches the weights only.  Row blocks of 16 or
//               32 rows (merged ones included); larger blocks are gathered ahead of the launch.
//   warps 4-11  epilogue, two warpgroups.  Each thread owns one sorted row (its TMEM lane)
//               and 128 of the tile's 256 accumulator columns.
//
// Two scaling modes (template parameter SCALING):
//   kScaleBlock128   activation scales per (row, 128 K), weight scales per 128x128 block.
//               The scales are arbitrary fp32, so they cannot ride inside the MMA: every
//               K block starts its TMEM stage from zero, and the epilogue folds the K
//               block's partial sums into register accumulators with the product of the
//               row's activation scale and the weight block's scale (packed fma.rn.f32x2).
//   kScalePerToken   one scale per activation row and one per weight row (output
//               column): the MMA accumulates over the whole K range in TMEM and the
//               epilogue drains each tile once.  fp8 e4m3 or int8 operands.
//
// Stage 1 tile: 128 gate rows + 128 up rows of W1 (one quantisation group of the
// output); each warpgroup takes 64 gate + 64 up columns, computes silu(gate)*up and
// either stores f16/bf16 or requantises to e4m3 with the per-row 1x128 scale (row amax
// exchanged between the two warpgroups through shared memory).
// Stage 2 tile: 256 rows of W2; each warpgroup takes 128 columns; every thread multiplies
// its row by the routing weight, parks the 256 bytes in a private shared-memory slot and
// the store warp adds them into out[token] with one bulk reduce (cp.reduce.async.bulk),
// bulk-stores per-pair rows for a later top-k reduce, or (ROW_DST instantiation) stores
// each row to a caller-given address, which may be in a peer GPU's memory.  The same
// kernel with one expert and identity routing is the dense block-scaled GEMM.
//
// MERGE instantiations run an expert's consecutive row blocks of 16, 32 or 64 rows as one tile of up to 128.
//
// Two other kernels take what this one is not good at: gemm_split.cu launches with few tiles (a
// cluster of CTAs shares K), gemm_pair.cu per-token scaling with many rows per expert (CTA pairs).
//
// Every wait is bounded: when one gives up it raises the CTA's abort flag and the
// device status word, every role drains out, TMEM is released and the kernel returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math.h>
#include <stdio.h>
#include <type_traits>

#include "common.cuh"
#include "gemm_args.cuh"
#include "gemm_ptx.cuh"

namespace flymoe {

// Upper bound on the persistent grid (0 = one CTA per SM).  A caller that overlaps the GEMMs with
// communication kernels leaves those kernels some SMs: a persistent CTA that cannot become resident
// at launch would otherwise run its whole tile list after the others have finished.
static int g_cta_limit = 0;

constexpr int kMaxStages = 4;
// Depth of the shared-memory operand ring.  Stage 2 gives one slot up for a staging area from
// which finished output rows leave by bulk reduce/store (measured: a 3-deep ring is as fast as 4).
template <int STAGE> struct RingDepth { static constexpr int value = STAGE == 1 ? 4 : 3; };
// Per-epilogue-thread staging slot for finished output: stage 2 holds 256 B of 16-bit results,
// stage 1 holds 64 e4m3 codes; 16 B of skew keep 16-byte shared-memory stores conflict-free.
template <int STAGE> struct Staging {
  static constexpr int stride = STAGE == 1 ? 80 : 272;
  static constexpr int bytes = 256 * stride;
};
constexpr int kStageBytes = kATileBytes + kBTileBytes;

struct __align__(16) SmemCtrl {
  unsigned long long full[kMaxStages];
  unsigned long long empty[kMaxStages];
  unsigned long long tmem_full[kAccStages];
  unsigned long long tmem_empty[kAccStages];
  unsigned long long amax_bar[2];
  unsigned long long stg_full;                  // epilogue warps -> store warp: slots and destinations written
  unsigned long long stg_free;                  // store warp -> epilogue warps: slots have been read
  unsigned long long stg_dst[256];              // per epilogue thread: global address of its row segment, 0 = none
  uint32_t tmem_base;
  int abort_flag;
  float amax[2][2][BM];
};
template <int STAGE> constexpr size_t smem_bytes() {
  return size_t(RingDepth<STAGE>::value) * kStageBytes + Staging<STAGE>::bytes + sizeof(SmemCtrl) + 1024;
}
// Table of merged row tiles (MERGE instantiations), behind the control block.
struct MergeTable {
  int scan[2][32];
  uint16_t table[kTileTable];
};
static_assert(smem_bytes<1>() + sizeof(MergeTable) <= 232448 && smem_bytes<2>() + sizeof(MergeTable) <= 232448,
              "shared memory budget of one SM exceeded");

// Optional whole-kernel wait accounting (build with -DFLYMOE_PROF, `python -m flydsl_b200.build
// --prof`): every CTA's producer thread, MMA thread and first epilogue thread add up the cycles they
// spend in each wait and write the sums once at the end; flymoe_prof_read() copies them out as
// [CTA][role][8] int64 (`python bench.py --wait-accounting` prints the means).
#ifdef FLYMOE_PROF
__device__ long long g_prof[256][3][8];
#define PROF_DECL long long prof_t0 = clock64(), prof_s = 0, prof_w[6] = {0, 0, 0, 0, 0, 0};
#define PROF_START prof_s = clock64();
#define PROF_STOP(i) prof_w[i] += clock64() - prof_s;
#define PROF_COUNT(i) prof_w[i] += 1;
#define PROF_WRITE(role)                                                         \
  do {                                                                           \
    if (blockIdx.x < 256) {                                                      \
      g_prof[blockIdx.x][role][0] = clock64() - prof_t0;                         \
      for (int pi = 0; pi < 6; ++pi) g_prof[blockIdx.x][role][1 + pi] = prof_w[pi]; \
    }                                                                            \
  } while (0)
#else
#define PROF_DECL
#define PROF_START
#define PROF_STOP(i)
#define PROF_COUNT(i)
#define PROF_WRITE(role) do {} while (0)
#endif

// ROW_DST (stage 2 only): every output row goes to a caller-given address instead of out[t*k+s].  A
// separate instantiation, so that the common kernel's register allocation is not touched.
// GATHER: a separate instantiation, so that the kernels reading sorted rows keep their register allocation.
// MERGE: consecutive row blocks of one expert (16, 32 or 64 rows each) run as one tile of up to 128 rows, so that the
// expert's weights are fetched and multiplied once for all of them instead of once per block.
template <int STAGE, bool ROW_DST, int SCALING, bool GATHER, bool MERGE>
__global__ void __launch_bounds__(kNumThreads, 1)
moe_gemm_sm100_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                      const GemmArgs a, const int group_m) {
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  constexpr int kStages = RingDepth<STAGE>::value;
  uint8_t* staging = smem + size_t(kStages) * kStageBytes;
  SmemCtrl* ctrl = reinterpret_cast<SmemCtrl*>(staging + Staging<STAGE>::bytes);
  volatile int* abort_flag = &ctrl->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int KB = a.k_dim / BK;

  const int valid_rows = min(__ldg(a.num_valid_ids), a.size_expert_ids * a.tile_m);
  // A rows are fetched by index (row = token, or token*topk+slot) instead of by one TMA box per K block
  constexpr bool gather = GATHER;
  // Outputs that leave through the staging slots (everything except 16-bit stage-1 and fp32 stage-2 output)
  const bool uses_staging = STAGE == 1 ? a.out_dtype == FLYMOE_E4M3 : a.out_dtype != FLYMOE_F32;
  MergeTable* merge = reinterpret_cast<MergeTable*>(ctrl + 1);
  TileSched sched;
  sched.num_mblocks = MERGE ? build_tile_table<kNumThreads>(a, valid_rows, BM / a.tile_m, merge->table, merge->scan)
                            : (valid_rows + a.tile_m - 1) / a.tile_m;
  // row tile -> its first row block and its rows
  auto tile_block = [&](int m) -> int { return MERGE ? int(merge->table[m] & 0xfff) : m; };
  auto tile_rows = [&](int m) -> int { return MERGE ? (int(merge->table[m] >> 12) + 1) * a.tile_m : a.tile_m; };
  sched.num_ntiles = STAGE == 1 ? a.n_dim / 128 : (a.n_dim + BN - 1) / BN;
  sched.total = sched.num_mblocks * sched.num_ntiles;
  sched.group_m = group_m;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&ctrl->full[i]), gather ? 2 : 1);     // TMA thread (+ the gather warp)
      mbar_init(smem_u32(&ctrl->empty[i]), 1);
    }
    for (int i = 0; i < kAccStages; ++i) {
      mbar_init(smem_u32(&ctrl->tmem_full[i]), 1);
      mbar_init(smem_u32(&ctrl->tmem_empty[i]), kEpilogueWarps);
    }
    mbar_init(smem_u32(&ctrl->amax_bar[0]), kEpilogueWarps);
    mbar_init(smem_u32(&ctrl->amax_bar[1]), kEpilogueWarps);
    mbar_init(smem_u32(&ctrl->stg_full), kEpilogueWarps);
    mbar_init(smem_u32(&ctrl->stg_free), 1);
    ctrl->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&ctrl->tmem_base)), "r"(uint32_t(kTmemCols)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = ctrl->tmem_base;

  // Register re-split: 384 threads x 168 registers are allocated at launch; the producer warpgroup
  // drops to 40 and the two epilogue warpgroups rise to 232 (128*40 + 256*232 = 384*168 exactly --
  // a larger request would wait forever for registers that are never released).
  static_assert(128 * 40 + 256 * 232 <= kNumThreads * 168, "setmaxnreg split exceeds the launch allocation");
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    // The single-thread roles run under elect.sync when the tensor cores are what bounds the kernel (per-token
    // scaling): descriptors then stay in uniform registers and an MMA costs its 128 cycles instead of ~165-250.
    // Measured, 4096 x 7168 x 7168: fp8 230 -> 191 us, bf16 255 -> 187 us.  With block scaling the epilogue is the
    // bound and the same change is even to slightly slower (T=4096 layer 3.43 against 3.44-3.50 ms), so that
    // instantiation keeps the plain predicate.
    const bool one_thread = SCALING == kScalePerToken ? elect_one() : lane == 0;
    if (warp == 0 && one_thread) {
      // ---------------------------------------------------------------- TMA producer
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      PROF_DECL
      int mb_next = 0, n_next = 0, e_next = -1;
      if (int(blockIdx.x) < sched.total) {
        sched.decode(blockIdx.x, mb_next, n_next);
        e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
      }
      for (int t = blockIdx.x; t < sched.total && ok; t += gridDim.x) {
        const int mb = mb_next, n = n_next, e = e_next;
        if (t + int(gridDim.x) < sched.total) {          // next tile's expert id: loaded a whole tile early
          sched.decode(t + gridDim.x, mb_next, n_next);
          e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
        }
        if (e < 0 || e >= a.experts) continue;
        const int row0 = tile_block(mb) * a.tile_m, rows = tile_rows(mb);
        const uint32_t tx_bytes = (gather ? 0u : uint32_t(rows) * BK) + kBTileBytes;
        for (int kb = 0; kb < KB; ++kb) {
          PROF_START
          if (!mbar_wait(smem_u32(&ctrl->empty[stage]), phase ^ 1, abort_flag, a.status, 1, 64)) { ok = false; break; }
          PROF_STOP(0) PROF_COUNT(5)
          const uint32_t full = smem_u32(&ctrl->full[stage]);
          const uint32_t sa = smem_u32(smem + size_t(stage) * kStageBytes);
          const uint32_t sb = sa + kATileBytes;
          mbar_expect_tx(full, tx_bytes);
          if (!gather) tma_load_2d(sa, &tmap_a, full, kb * BK, row0);
          if (MERGE && !gather)
            for (int m = a.tile_m; m < rows; m += a.tile_m)
              tma_load_2d(sa + uint32_t(m) * BK, &tmap_a, full, kb * BK, row0 + m);
          if (STAGE == 1) {
            tma_load_3d(sb, &tmap_b, full, kb * BK, n * 128, e);
            tma_load_3d(sb + 128 * BK, &tmap_b, full, kb * BK, a.n_dim + n * 128, e);
          } else {
            tma_load_3d(sb, &tmap_b, full, kb * BK, n * BN, e);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1; }
        }
      }
      PROF_WRITE(0);
    } else if (warp == 1 && one_thread) {
      // ---------------------------------------------------------------- MMA issuer
      PROF_DECL
      auto issue = [&](auto kind_c, const uint32_t idesc) {
        constexpr int KIND = decltype(kind_c)::value;
        int stage = 0, acc = 0;
        uint32_t phase = 0, acc_phase = 0;
        int mb_next = 0, n_next = 0, e_next = -1;
        if (int(blockIdx.x) < sched.total) {
          sched.decode(blockIdx.x, mb_next, n_next);
          e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
        }
        for (int t = blockIdx.x; t < sched.total; t += gridDim.x) {
          const int e = e_next;
          if (t + int(gridDim.x) < sched.total) {
            sched.decode(t + gridDim.x, mb_next, n_next);
            e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
          }
          if (e < 0 || e >= a.experts) continue;
          for (int kb = 0; kb < KB; ++kb) {
            // per-token scaling: one accumulator stage per tile; block scaling: one per K block, started from zero
            if (SCALING == kScaleBlock128 || kb == 0) {
              PROF_START
              if (!mbar_wait(smem_u32(&ctrl->tmem_empty[acc]), acc_phase ^ 1, abort_flag, a.status, 2)) return;
              PROF_STOP(0)
            }
            PROF_START
            if (!mbar_wait(smem_u32(&ctrl->full[stage]), phase, abort_flag, a.status, 3)) return;
            PROF_STOP(1)
            PROF_COUNT(5) PROF_START
            tcgen05_fence_after();
            const uint32_t sa = smem_u32(smem + size_t(stage) * kStageBytes);
            const uint64_t adesc = make_smem_desc(sa);
            const uint64_t bdesc = make_smem_desc(sa + kATileBytes);
            const uint32_t d_tmem = tmem_base + uint32_t(acc) * BN;
#pragma unroll
            for (int k = 0; k < BK / 32; ++k)
              umma<KIND>(d_tmem, adesc + uint64_t(k * 2), bdesc + uint64_t(k * 2), idesc,
                         (k > 0 || (SCALING == kScalePerToken && kb > 0)) ? 1u : 0u);
            umma_commit(smem_u32(&ctrl->empty[stage]));
            if (SCALING == kScaleBlock128 || kb + 1 == KB) {
              umma_commit(smem_u32(&ctrl->tmem_full[acc]));
              if (++acc == kAccStages) { acc = 0; acc_phase ^= 1; }
            }
            PROF_STOP(3)
            if (++stage == kStages) { stage = 0; phase ^= 1; }
          }
        }
      };
      if (SCALING == kScaleBlock128 || a.in_dtype == FLYMOE_E4M3) issue(std::integral_constant<int, 0>{}, kInstrDescF8);
      else if (a.in_dtype == FLYMOE_I8) issue(std::integral_constant<int, 1>{}, kInstrDescI8);
      else issue(std::integral_constant<int, 2>{}, a.in_dtype == FLYMOE_BF16 ? kInstrDescBF16 : kInstrDescF16);
      PROF_WRITE(1);
    } else if (warp == 2 && uses_staging) {
      // ---------------------------------------------------------------- store warp
      // Issues the bulk store / bulk reduce of every epilogue thread's staging slot, eight slots per
      // lane, so that the ~10 cycles each of those 256 operations takes to be accepted are spent here
      // and not by the epilogue warps between two tiles.
      bool ok = true;
      uint32_t it = 0;
      int mb_next = 0, n_next = 0, e_next = -1;
      if (int(blockIdx.x) < sched.total) {
        sched.decode(blockIdx.x, mb_next, n_next);
        e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
      }
      constexpr uint32_t kSlotBytes = STAGE == 1 ? 64u : 256u;
      const bool bf = a.out_dtype == FLYMOE_BF16;
      for (int t = blockIdx.x; t < sched.total && ok; t += gridDim.x) {
        const int e = e_next, n = n_next;
        if (t + int(gridDim.x) < sched.total) {
          sched.decode(t + gridDim.x, mb_next, n_next);
          e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
        }
        if (e < 0 || e >= a.experts) continue;
        if (!mbar_wait(smem_u32(&ctrl->stg_full), it & 1, abort_flag, a.status, 6, 64)) { ok = false; break; }
        // stage 2 with n_dim = 64 mod 128 (dense GEMM only): the tile's last segment holds 64 columns
        const int cols_left = STAGE == 2 ? a.n_dim - n * BN : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int sl = i * 32 + lane;
          const unsigned long long dst = ctrl->stg_dst[sl];
          if (dst != 0ull) {
            const uint32_t sp = smem_u32(staging + size_t(sl) * Staging<STAGE>::stride);
            void* gp = reinterpret_cast<void*>(dst);
            const uint32_t bytes = (STAGE == 2 && cols_left - (sl >> 7) * 128 < 128) ? kSlotBytes / 2 : kSlotBytes;
            if (STAGE == 1 || !a.accumulate) bulk_store(gp, sp, bytes);
            else if (bf) bulk_reduce_add_bf16(gp, sp, bytes);
            else bulk_reduce_add_f16(gp, sp, bytes);
          }
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        bulk_wait_read_all();                      // the slots may be overwritten from here on
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->stg_free));
        ++it;
      }
      bulk_wait_all();                             // every row segment has landed before the CTA retires
    } else if (warp == 3 && gather) {
      // ---------------------------------------------------------------- row gather
      // Lane l serves rows l, l+32, l+64, l+96 of the tile: eight 16-byte cp.async per row and K block,
      // written where the 128-byte swizzle puts them (chunk c of row r at r*128 + ((c ^ (r & 7)) << 4)).
      // A K block's copies are completed two K blocks later (cp.async.wait_group), made visible to the
      // tensor cores' proxy (fence.proxy.async) and then signalled on the stage's full barrier, next to
      // the TMA thread's arrival for the weights.  Pad rows are zero-filled (source size 0).
      // One warp issues every request, which keeps up with row blocks of 16 or 32 rows (decode); with
      // 64 and 128 rows a K block takes longer here than in the tensor cores, so the host wrappers gather
      // such blocks ahead of the launch (stage 1 of the T=4096 layer 2.5 ms against 1.9 + 0.08 ms).  Merged
      // blocks of 16 or 32 rows still come through here, up to 1024 requests per K block: slower per tile
      // (merge_blocks counts it), but instead of the weights once per block (333 tokens over 256 experts of
      // 7168 x 2048, 16-row blocks, Zipf: 1332 us one by one, 500 merged).
      constexpr int kInFlight = 2;
      int stage = 0, pending = 0;
      uint32_t phase = 0;
      bool ok = true;
      const int pad_id = (a.topk << 24) | a.num_tokens;
      auto complete_oldest = [&]() {             // the oldest pending K block's rows have landed
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        const int s_old = (stage - pending + 2 * kStages) % kStages;
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->full[s_old]));
        --pending;
      };
      for (int t = blockIdx.x; t < sched.total && ok; t += gridDim.x) {
        int mb, n;
        sched.decode(t, mb, n);
        const int e = __ldg(a.sorted_expert_ids + tile_block(mb));
        if (e < 0 || e >= a.experts) continue;
        const int row0 = tile_block(mb) * a.tile_m, rows = tile_rows(mb);
        const uint8_t* src[4];
        uint32_t nbytes[4];                      // 16 = copy, 0 = zero-fill (pad row)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int row = j * 32 + lane;
          const int r = row0 + row;
          const int id = (row < rows && r < valid_rows) ? __ldg(a.sorted_ids + r) : pad_id;
          const int tok = id_token(id), slot = id_slot(id);
          const bool valid = tok < a.num_tokens && slot < a.topk;
          const long long srow = a.a_layout == FLYMOE_ROWS_BY_TOKEN ? (long long)tok
                               : a.a_layout == FLYMOE_ROWS_BY_SLOT ? (long long)slot * a.num_tokens + tok
                                                                   : (long long)tok * a.topk + slot;
          src[j] = a.a + (valid ? srow : 0) * a.k_dim;
          nbytes[j] = valid ? 16u : 0u;
        }
        for (int kb = 0; kb < KB; ++kb) {
          if (!mbar_wait(smem_u32(&ctrl->empty[stage]), phase ^ 1, abort_flag, a.status, 10, 32)) { ok = false; break; }
          const uint32_t sa = smem_u32(smem + size_t(stage) * kStageBytes);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int row = j * 32 + lane;
            if (row < rows) {
              const uint8_t* g = src[j] + kb * BK;
              const uint32_t d = sa + uint32_t(row) * 128u;
#pragma unroll
              for (int c = 0; c < 8; ++c)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                             ::"r"(d + (uint32_t(c ^ (row & 7)) << 4)), "l"(g + c * 16), "r"(nbytes[j]) : "memory");
            }
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
          if (++stage == kStages) { stage = 0; phase ^= 1; }
          if (++pending > kInFlight) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kInFlight) : "memory");
            complete_oldest();
          }
        }
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      while (pending > 0) complete_oldest();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    // ------------------------------------------------------------------ epilogue
    const int wg = (warp - 4) >> 2;          // 0 or 1
    const int q = warp & 3;                  // TMEM lane quadrant of this warp
    const int row_in_tile = q * 32 + lane;
    const uint32_t lane_base = uint32_t(q * 32) << 16;
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t tile_iter = 0;
    bool ok = true;
    PROF_DECL
    static_assert(kAccStages == 2, "the epilogue's stage/phase stepping assumes two accumulator stages");
    const uint32_t full_bar0 = smem_u32(&ctrl->tmem_full[0]);     // stage 1's barrier is 8 bytes further
    const uint32_t empty_bar0 = smem_u32(&ctrl->tmem_empty[0]);
    constexpr int NACC = 128;                // fp32 accumulators per thread
    // Routing of a tile (expert id, this thread's packed row id) is loaded one tile ahead.
    const int pad_id = (a.topk << 24) | a.num_tokens;
    int mb_next = 0, n_next = 0, e_next = -1, id_next = pad_id;
    auto load_routing = [&](int tt) {
      sched.decode(tt, mb_next, n_next);
      e_next = __ldg(a.sorted_expert_ids + tile_block(mb_next));
      const int rr = tile_block(mb_next) * a.tile_m + row_in_tile;
      id_next = (row_in_tile < tile_rows(mb_next) && rr < valid_rows) ? __ldg(a.sorted_ids + rr) : pad_id;
    };
    if (int(blockIdx.x) < sched.total) load_routing(blockIdx.x);
    for (int t = blockIdx.x; t < sched.total && ok; t += gridDim.x) {
      const int mb = mb_next, n = n_next, e = e_next, id = id_next;
      if (t + int(gridDim.x) < sched.total) load_routing(t + gridDim.x);
      if (e < 0 || e >= a.experts) continue;

      const int rows = tile_rows(mb);
      const bool warp_active = q * 32 < rows;
      const int r = tile_block(mb) * a.tile_m + row_in_tile;
      const bool in_tile = row_in_tile < rows && r < valid_rows;
      const int tok = id_token(id), slot = id_slot(id);
      const bool valid = in_tile && tok < a.num_tokens && slot < a.topk;
      long long sidx = 0;
      if (valid) {
        sidx = a.a_scale_layout == FLYMOE_ROWS_BY_TOKEN ? (long long)tok
             : a.a_scale_layout == FLYMOE_ROWS_BY_PAIR ? (long long)tok * a.topk + slot : (long long)r;
        if (SCALING == kScalePerToken && a.a_scale_layout == FLYMOE_ROWS_BY_SLOT) sidx = (long long)slot * a.num_tokens + tok;
      }
      // stage 2: a warpgroup whose 128 columns lie beyond n_dim (last tile of a row) has nothing to do
      const bool half_ok = STAGE == 1 ? true : (n * BN + wg * 128 < a.n_dim);
      // routing weight of this row, used after the K loop.  The loop runs at the register limit, and where
      // this value is requested decides whether ptxas spills inside it: stage 2 asks here (its latency
      // hides behind the loop), stage 1 after the loop (measured: no spills either way, `-Xptxas -v`).
      float wgt = 1.f;
      if (STAGE == 2 && a.doweight && valid) wgt = __ldg(a.sorted_weights + r);
      // a warp whose 32 rows are all padding has nothing to fold in (4096 tokens over 256 experts, whose second row blocks
      // hold a dozen rows: within the spread of two runs, 0.5 %; it leaves the FMA pipe to the other warps)
      const bool work = warp_active && half_ok && __any_sync(0xffffffffu, valid);
      // stage 1: first half = gate columns, second half = up columns; stage 2: two halves of 128 columns
      const uint32_t tcol0 = tmem_base + lane_base + (STAGE == 1 ? uint32_t(wg * 64) : uint32_t(wg * 128));
      const uint32_t tcol1 = tmem_base + lane_base + (STAGE == 1 ? uint32_t(128 + wg * 64) : uint32_t(wg * 128 + 64));
      float accv[NACC];
      if (SCALING == kScaleBlock128) {
      const float* sa_ptr = a.scale_a + sidx * a.sa_row_stride;
      // weight block scales of this tile
      const int wblk_per_expert = (STAGE == 1 ? 2 * a.n_dim : a.n_dim) / 128;
      const int blk0 = STAGE == 1 ? n : n * 2 + wg;
      const int blk1 = STAGE == 1 ? a.n_dim / 128 + n : blk0;
      const float* sw0_ptr = a.scale_w + ((long long)e * wblk_per_expert + (half_ok ? blk0 : 0)) * KB;
      const int sw1_off = (blk1 - (half_ok ? blk0 : 0)) * KB;      // up-projection scales, relative to sw0_ptr

      // fp32 accumulators held as packed pairs so the scale-FMA runs as fma.rn.f32x2
      unsigned long long acc2[NACC / 2];
#pragma unroll
      for (int j = 0; j < NACC / 2; ++j) acc2[j] = 0ull;

      float sa_next = valid ? __ldg(sa_ptr) : 0.f;
      float s0_next = __ldg(sw0_ptr);
      float s1_next = STAGE == 1 ? __ldg(sw0_ptr + sw1_off) : 0.f;
      const float* sa_run = sa_ptr;            // running pointer: one add per K block, no multiply
      // One K block = four 32-column chunks through two register buffers, two tcgen05.ld in flight at
      // a time: the thread waits twice per K block, not once per chunk.
      uint32_t v0[32], v1[32];
      // measured: two K blocks per loop trip help stage 1 (~1.5 %) and cost stage 2 about as much
#pragma unroll (STAGE == 1 ? 2 : 1)
      for (int kb = 0; kb < KB; ++kb) {
        const uint32_t stage_off = uint32_t(acc) * BN;
        PROF_START
        if (!mbar_wait(full_bar0 + uint32_t(acc) * 8u, acc_phase, abort_flag, a.status, 4)) { ok = false; break; }
        PROF_STOP(0) PROF_COUNT(5)
        tcgen05_fence_after();
        if (work) {                            // both chunks of the first half on their way at once
          tmem_ld_x32(tcol0 + stage_off, v0);
          tmem_ld_x32(tcol0 + stage_off + 32, v1);
        }
        const unsigned long long c0 = pack_f32x2(sa_next * s0_next);
        const unsigned long long c1 = STAGE == 1 ? pack_f32x2(sa_next * s1_next) : c0;
        if (work) tmem_ld_wait();
        if (kb + 1 < KB) {                     // next K block's scales: in flight during this block's math
          sa_run += a.sa_stride;
          sa_next = valid ? __ldg(sa_run) : 0.f;
          s0_next = __ldg(sw0_ptr + kb + 1);
          if (STAGE == 1) s1_next = __ldg(sw0_ptr + kb + 1 + sw1_off);
        }
        if (work) {
          // each buffer is refilled with its chunk of the second half as soon as it has been folded in
#pragma unroll
          for (int j = 0; j < 16; ++j) ffma2(acc2[j], v0[2 * j], v0[2 * j + 1], c0);
          tmem_ld_x32(tcol1 + stage_off, v0);
#pragma unroll
          for (int j = 0; j < 16; ++j) ffma2(acc2[16 + j], v1[2 * j], v1[2 * j + 1], c0);
          tmem_ld_x32(tcol1 + stage_off + 32, v1);
          tmem_ld_wait();
        }
        // The K block's partial sums are in registers now (tcgen05.wait::ld has returned, so the loads
        // have completed and need no further ordering): hand the TMEM stage back before the last
        // chunk's FMAs.  The arrive publishes no memory, hence relaxed; tcgen05.wait::ld is warp-wide
        // (.sync.aligned), so when lane 0 is past it every lane's loads have landed.
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
      for (int j = 0; j < NACC / 2; ++j) unpack_f32x2(acc2[j], accv[2 * j], accv[2 * j + 1]);
      } else {
        // One scale per activation row, one per weight row: the whole K range has been accumulated in
        // TMEM; drain the tile once and scale it here.
        const uint32_t stage_off = uint32_t(acc) * BN;
        PROF_START
        if (!mbar_wait(full_bar0 + uint32_t(acc) * 8u, acc_phase, abort_flag, a.status, 4)) { ok = false; break; }
        PROF_STOP(0) PROF_COUNT(5)
        tcgen05_fence_after();
        // the raw accumulators land in the registers of accv and are scaled in place
        uint32_t* v = reinterpret_cast<uint32_t*>(accv);
        if (work) {
          tmem_ld_x32(tcol0 + stage_off, v);
          tmem_ld_x32(tcol0 + stage_off + 32, v + 32);
          tmem_ld_x32(tcol1 + stage_off, v + 64);
          tmem_ld_x32(tcol1 + stage_off + 32, v + 96);
          tmem_ld_wait();
        } else {
          __syncwarp();
        }
        if (lane == 0) mbar_arrive_relaxed(empty_bar0 + uint32_t(acc) * 8u);
        acc_phase ^= uint32_t(acc);
        acc ^= 1;
        if (work) {
          // 16-bit operands come without scales (null pointers): every factor is 1
          const float sa = valid ? row_scale(a.scale_a, sidx) : 0.f;
          const long long wrows = STAGE == 1 ? 2LL * a.n_dim : (long long)a.n_dim;
          // weight-row scales of this thread's two 64-column halves (the same addresses in every lane)
          const float* sw0 = a.scale_w + (long long)e * wrows + (STAGE == 1 ? n * 128 + wg * 64 : n * BN + wg * 128);
          const float* sw1 = STAGE == 1 ? sw0 + a.n_dim : sw0 + 64;
          const bool i8 = a.in_dtype == FLYMOE_I8;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float* sw = h == 0 ? sw0 : sw1;
#pragma unroll
            for (int j = 0; j < 64; j += 4) {
              const float4 s4 = col_scales4(a.scale_w, sw + j);
              const float c[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int idx = h * 64 + j + u;
                const float p = i8 ? __int2float_rn(int(v[idx])) : accv[idx];
                accv[idx] = p * (sa * c[u]);
              }
              asm volatile("" ::: "memory");       // keeps the 32 scale loads from being hoisted in front of the math
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < NACC; ++j) accv[j] = 0.f;
        }
      }
      // Destination of this row when the caller gave per-row addresses: requested after the K loop (the
      // loop runs at the register limit) and needed only once the row has been packed.
      unsigned long long row_dst_base = 0ull;
      if (STAGE == 2 && ROW_DST && valid)
        row_dst_base = __ldg(a.row_dst + ((long long)tok * a.topk + slot));
      if (STAGE == 1 && a.doweight && valid) wgt = __ldg(a.sorted_weights + r);

      // ---- tile epilogue -----------------------------------------------------------
      // Kept short on purpose: this code runs once per tile between two main loops, and a long
      // straight-line tail (IEEE division, accurate exp) costs more in instruction fetch than in math.
      PROF_START
      if (STAGE == 1 && SCALING == kScalePerToken && a.out_dtype == FLYMOE_F32) {
        // The reference's split-K output contract (kernels/moe_gemm_2stage.py:121-122, :1345): the scaled gate
        // and up sums are ADDED to out[t*topk+s][0:I | I:2I] (fp32, zeroed by the caller) -- no activation,
        // no routing weight.  The whole K range is summed here, so every element receives one addition.
        if (warp_active && valid) {
          float* og = static_cast<float*>(a.out) + ((long long)tok * a.topk + slot) * (2LL * a.n_dim) +
                      (long long)n * 128 + wg * 64;
          float* ou = og + a.n_dim;
#pragma unroll
          for (int j = 0; j < 64; j += 4) red_add_v4_f32(og + j, accv[j], accv[j + 1], accv[j + 2], accv[j + 3]);
#pragma unroll
          for (int j = 0; j < 64; j += 4)
            red_add_v4_f32(ou + j, accv[64 + j], accv[64 + j + 1], accv[64 + j + 2], accv[64 + j + 3]);
        }
      } else if (STAGE == 1) {
        // accv[0..63] = gate, accv[64..127] = up, columns n*128 + wg*64 + j
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const float g = accv[j];
          const float hval = g * fast_rcp(1.0f + fast_exp2(-1.4426950408889634f * g)) * (accv[64 + j] * wgt);
          accv[j] = hval;
          amax = fmaxf(amax, fabsf(hval));
        }
        const long long orow = a.out_layout == FLYMOE_ROWS_SORTED ? (long long)r : (long long)tok * a.topk + slot;
        const long long ocol = (long long)n * 128 + wg * 64;
        if (a.out_dtype == FLYMOE_E4M3) {
          const int buf = tile_iter & 1;
          const uint32_t bar = smem_u32(&ctrl->amax_bar[buf]);
          if (warp_active) ctrl->amax[buf][wg][row_in_tile] = valid ? amax : 0.f;
          __syncwarp();
          if (lane == 0) mbar_arrive(bar);
          if (!mbar_wait(bar, (tile_iter >> 1) & 1, abort_flag, a.status, 5)) { ok = false; break; }
          // the store warp has finished reading the previous tile's slots
          if (!mbar_wait(smem_u32(&ctrl->stg_free), (tile_iter & 1) ^ 1, abort_flag, a.status, 7)) { ok = false; break; }
          unsigned long long dst_addr = 0ull;
          const bool wr = warp_active && (valid || (in_tile && a.out_layout == FLYMOE_ROWS_SORTED));
          if (wr) {
            const float m = fmaxf(ctrl->amax[buf][0][row_in_tile], ctrl->amax[buf][1][row_in_tile]);
            float sc = __fdiv_rn(m, 448.0f);
            if (sc == 0.f) sc = 1.f;
            const float inv = valid ? __fdiv_rn(1.0f, sc) : 0.f;     // pad rows: every code becomes 0
            // 64 codes go through this thread's staging slot and leave as one 64-byte bulk store
            uint8_t* op = staging + size_t(threadIdx.x - 128) * Staging<STAGE>::stride;
#pragma unroll
            for (int j = 0; j < 64; j += 16) {
              uint4 pk;
              pk.x = float4_to_e4m3x4(accv[j + 0] * inv, accv[j + 1] * inv, accv[j + 2] * inv, accv[j + 3] * inv);
              pk.y = float4_to_e4m3x4(accv[j + 4] * inv, accv[j + 5] * inv, accv[j + 6] * inv, accv[j + 7] * inv);
              pk.z = float4_to_e4m3x4(accv[j + 8] * inv, accv[j + 9] * inv, accv[j + 10] * inv, accv[j + 11] * inv);
              pk.w = float4_to_e4m3x4(accv[j + 12] * inv, accv[j + 13] * inv, accv[j + 14] * inv, accv[j + 15] * inv);
              if (!valid) pk = make_uint4(0, 0, 0, 0);
              *reinterpret_cast<uint4*>(op + j) = pk;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            dst_addr = reinterpret_cast<unsigned long long>(static_cast<uint8_t*>(a.out) + orow * a.n_dim + ocol);
            if (wg == 0) a.out_scale[(long long)n * a.out_scale_stride + orow] = sc;
          }
          ctrl->stg_dst[threadIdx.x - 128] = dst_addr;
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctrl->stg_full));
        } else if (warp_active && valid) {
          uint8_t* op = static_cast<uint8_t*>(a.out) + (orow * a.n_dim + ocol) * 2;
          const bool bf = a.out_dtype == FLYMOE_BF16;
#pragma unroll
          for (int j = 0; j < 64; j += 8) {
            uint4 pk;
            pk.x = bf ? pack_bf16x2(accv[j + 0], accv[j + 1]) : pack_f16x2(accv[j + 0], accv[j + 1]);
            pk.y = bf ? pack_bf16x2(accv[j + 2], accv[j + 3]) : pack_f16x2(accv[j + 2], accv[j + 3]);
            pk.z = bf ? pack_bf16x2(accv[j + 4], accv[j + 5]) : pack_f16x2(accv[j + 4], accv[j + 5]);
            pk.w = bf ? pack_bf16x2(accv[j + 6], accv[j + 7]) : pack_f16x2(accv[j + 6], accv[j + 7]);
            *reinterpret_cast<uint4*>(op + j * 2) = pk;
          }
        }
      } else if (a.out_dtype == FLYMOE_F32) {
        if (warp_active && valid && half_ok) {
          // fp32 output: vector reductions straight from registers (accumulate mode only)
          float* op = static_cast<float*>(a.out) + (long long)tok * a.n_dim + (long long)n * BN + wg * 128;
#pragma unroll
          for (int j = 0; j < 128; j += 4)
            red_add_v4_f32(op + j, accv[j] * wgt, accv[j + 1] * wgt, accv[j + 2] * wgt, accv[j + 3] * wgt);
        }
      } else {
        // 16-bit output: each thread parks its 128 results (256 B) in its own slot of the staging area
        // together with the global address of its row segment; the store warp sends every slot off as
        // ONE bulk reduce-add (or bulk store), instead of 16 scattered 16-byte atomics per thread.
        uint8_t* slot_ptr = staging + size_t(threadIdx.x - 128) * Staging<STAGE>::stride;
        if (!mbar_wait(smem_u32(&ctrl->stg_free), (tile_iter & 1) ^ 1, abort_flag, a.status, 7)) { ok = false; break; }
        unsigned long long dst_addr = 0ull;
        if (warp_active && valid && half_ok) {
          const bool bf = a.out_dtype == FLYMOE_BF16;
#pragma unroll
          for (int j = 0; j < 128; j += 8) {
            uint4 pk;
            pk.x = bf ? pack_bf16x2(accv[j] * wgt, accv[j + 1] * wgt) : pack_f16x2(accv[j] * wgt, accv[j + 1] * wgt);
            pk.y = bf ? pack_bf16x2(accv[j + 2] * wgt, accv[j + 3] * wgt) : pack_f16x2(accv[j + 2] * wgt, accv[j + 3] * wgt);
            pk.z = bf ? pack_bf16x2(accv[j + 4] * wgt, accv[j + 5] * wgt) : pack_f16x2(accv[j + 4] * wgt, accv[j + 5] * wgt);
            pk.w = bf ? pack_bf16x2(accv[j + 6] * wgt, accv[j + 7] * wgt) : pack_f16x2(accv[j + 6] * wgt, accv[j + 7] * wgt);
            *reinterpret_cast<uint4*>(slot_ptr + j * 2) = pk;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          const long long orow = a.accumulate ? (long long)tok : (long long)tok * a.topk + slot;
          const long long col_bytes = ((long long)n * BN + wg * 128) * 2;
          if (ROW_DST) {
            // rows leave for caller-given addresses (another GPU's buffer included): the bulk store
            // carries the row segment there while the next tile is in the tensor cores
            // a misaligned address would fault the bulk store: drop the row and report instead
            const unsigned long long base = row_dst_base;
            if ((base & 15ull) != 0ull) atomicCAS(a.status, 0, FLYMOE_STATUS_ROW_DST_MISALIGNED);
            else dst_addr = base != 0ull ? base + (unsigned long long)col_bytes : 0ull;
          } else {
            dst_addr = reinterpret_cast<unsigned long long>(static_cast<uint8_t*>(a.out) + orow * a.n_dim * 2 + col_bytes);
          }
        }
        ctrl->stg_dst[threadIdx.x - 128] = dst_addr;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->stg_full));
      }
      PROF_STOP(1) PROF_COUNT(4)
      ++tile_iter;
    }
    if (threadIdx.x == 128) PROF_WRITE(2);
  }

  tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemCols))
                 : "memory");
  }
}

// One thread waits, with the kernels' own bounded wait, on a barrier that nobody arrives at.
__global__ void bounded_wait_selftest_kernel(int* status, unsigned long long limit_ns, int code) {
  __shared__ unsigned long long bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait(smem_u32(&bar), 0, &abort_flag, status, code, 64, limit_ns);
}

}  // namespace flymoe

extern "C" int flymoe_set_gemm_cta_limit(int max_ctas) {
  if (max_ctas < 0) {
    flymoe::set_last_error_msg("set_gemm_cta_limit: max_ctas must be >= 0");
    return FLYMOE_ERR_INVALID_ARGUMENT;
  }
  flymoe::g_cta_limit = max_ctas;
  return FLYMOE_OK;
}

extern "C" int flymoe_selftest_bounded_wait(int64_t limit_ns, void* stream) {
  using namespace flymoe;
  FLYMOE_REQUIRE(limit_ns > 0 && limit_ns <= 100000000, "selftest_bounded_wait: limit_ns must be in (0, 1e8]");
  int* status = device_status_ptr();
  FLYMOE_REQUIRE(status != nullptr, "selftest_bounded_wait: no CUDA device");
  bounded_wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(
      status, static_cast<unsigned long long>(limit_ns), FLYMOE_STATUS_SELFTEST_TIMEOUT);
  FLYMOE_CUDA_CHECK(cudaGetLastError());
  return FLYMOE_OK;
}

#ifdef FLYMOE_PROF
extern "C" int flymoe_prof_read(long long* host_out) {
  FLYMOE_CUDA_CHECK(cudaDeviceSynchronize());
  FLYMOE_CUDA_CHECK(cudaMemcpyFromSymbol(host_out, flymoe::g_prof, sizeof(flymoe::g_prof)));
  return FLYMOE_OK;
}
#endif

namespace flymoe {

// ------------------------------------------------------------------------------ host
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

static int make_map(CUtensorMap* map, const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides,
                    const cuuint32_t* box) {
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
  if (fn == nullptr) {
    set_last_error_msg("cuTensorMapEncodeTiled is not available from this driver");
    return FLYMOE_ERR_CUDA;
  }
  cuuint32_t elem_strides[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, rank, const_cast<void*>(base), dims, strides, box, elem_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[128];
    snprintf(buf, sizeof(buf), "cuTensorMapEncodeTiled failed with CUresult %d", int(r));
    set_last_error_msg(buf);
    return FLYMOE_ERR_CUDA;
  }
  return FLYMOE_OK;
}

int make_gemm_maps(int stage, const GemmArgs& a, int a_box_rows, int b_box_rows, CUtensorMap* map_a, CUtensorMap* map_b) {
  const long long wrows = stage == 1 ? 2LL * a.n_dim : a.n_dim;
  cuuint64_t adims[2] = {cuuint64_t(a.k_dim), cuuint64_t(a.a_rows)};
  cuuint64_t astrides[1] = {cuuint64_t(a.k_dim)};
  cuuint32_t abox[2] = {cuuint32_t(BK), cuuint32_t(a_box_rows)};
  const int rc = make_map(map_a, a.a, 2, adims, astrides, abox);
  if (rc != FLYMOE_OK) return rc;
  cuuint64_t bdims[3] = {cuuint64_t(a.k_dim), cuuint64_t(wrows), cuuint64_t(a.experts)};
  cuuint64_t bstrides[2] = {cuuint64_t(a.k_dim), cuuint64_t(wrows) * cuuint64_t(a.k_dim)};
  cuuint32_t bbox[3] = {cuuint32_t(BK), cuuint32_t(b_box_rows), 1};
  return make_map(map_b, a.w, 3, bdims, bstrides, bbox);
}

template <int STAGE, bool ROW_DST, int SCALING, bool GATHER, bool MERGE>
static int launch_kernel(int grid, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_b,
                         const GemmArgs& a, int group_m) {
  auto* kernel = moe_gemm_sm100_kernel<STAGE, ROW_DST, SCALING, GATHER, MERGE>;
  constexpr size_t smem = smem_bytes<STAGE>() + (MERGE ? sizeof(MergeTable) : 0);
  FLYMOE_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  kernel<<<grid, kNumThreads, smem, stream>>>(map_a, map_b, a, group_m);
  FLYMOE_CUDA_CHECK(cudaGetLastError());
  return FLYMOE_OK;
}

template <int STAGE, bool ROW_DST, int SCALING, bool MERGE>
static int launch_one(int grid, cudaStream_t stream, const CUtensorMap& map_a, const CUtensorMap& map_b,
                      const GemmArgs& a, int group_m) {
  if (a.a_layout != FLYMOE_ROWS_SORTED)
    return launch_kernel<STAGE, ROW_DST, SCALING, true, MERGE>(grid, stream, map_a, map_b, a, group_m);
  return launch_kernel<STAGE, ROW_DST, SCALING, false, MERGE>(grid, stream, map_a, map_b, a, group_m);
}

// Expected row tiles of an expert that receives `mean` rows on average, spread as under even routing (Poisson, tails by
// the normal distribution).
static double row_tiles(double mean, int unit) {
  if (mean >= 4.0 * unit) return mean / unit + 0.5;
  double n = 1.0 - exp(-mean);
  for (int j = 1; j <= 8; ++j) {
    const double p = 0.5 * erfc((j * unit + 0.5 - mean) / sqrt(2.0 * mean));
    if (p < 1e-3) break;
    n += p;
  }
  return n;
}

// Microseconds of a launch whose row tiles hold `rows` rows: rounds of tiles times (fill, tile end and K blocks).  One
// warp fetches rows by index, so a gathered K block costs with its rows what 16 bytes per request cost.  Fitted to layers
// of 8 experts of 1024 x 512 (1 and 2 rounds of 4 to 8 K blocks) and of 16 of 4096 x 1536 (2 to 50 rounds of 12 to 32).
static double tile_rounds_us(double tiles, double rows, bool gather, int KB, int ctas) {
  const double kblock = gather ? 0.6 + 0.008 * (rows - 16.0) : 0.6 + 0.0012 * rows;
  return ceil(tiles / ctas) * (1.5 + 0.0375 * rows + KB * kblock);
}

// Row blocks of an expert are merged where fewer rounds of longer tiles are expected to take less time than the blocks
// one by one, the table at kernel start (1.5 us) included.  Layers on one B200, whole calls in a CUDA graph, us one by
// one -> merged, even routing:
//   8 experts of 1024 x 512, top-2, 16-row blocks: 192 tokens 31 -> 39, 512 tokens 43 -> 51 (both left alone: the blocks
//   fit one or two rounds, the merged tiles are one long one), 1024 tokens 69 -> 57, 2048 tokens 117 -> 66;
//   16 experts of 4096 x 1536, top-2, 32-row blocks: 205 tokens 92 -> 100 (left alone), 384 tokens 123 -> 108, 2048 398 -> 235;
//   64 experts of 2048 x 1024, top-6, 32-row blocks: 273 tokens 115 -> 123 (left alone), 341 tokens 143 -> 130;
//   8 experts of 4096 x 14336, top-2, 128 tokens, 32-row blocks: 421 -> 302.
// From 0.8 of a block per expert on, a launch that this expects to lose less than 3 % is merged all the same: skewed
// routing has the busy experts' second blocks there already (205 tokens through that layer in 64-row blocks, Zipf:
// 405 -> 303 merged; even 321 -> 323).
// Launches that stream 512 MB of weights or more are merged from a quarter of a block per expert on.  Under even routing
// no expert has a second block there, and the merging kernel is even to 6 % slower (42 to 102 tokens through the
// 4096 x 14336 layer: 281 -> 292, 290 -> 301 us); under skewed routing the busy experts have many (the same 102 tokens,
// Zipf, its first stage merged: 390 -> 323; 128 tokens over 256 experts of 7168 x 2048, 16-row blocks: 691 -> 315).
static bool merge_blocks(int stage, const GemmArgs& a, int ctas) {
  if (a.tile_m >= BM || a.row_dst != nullptr || a.size_expert_ids > kTileTable || a.experts < 2) return false;
  const int ntiles = stage == 1 ? a.n_dim / 128 : ceil_div(a.n_dim, BN);
  if ((long long)a.size_expert_ids * ntiles <= ctas) return false;      // one round, however the rows fall
  const long long rows = (long long)a.num_tokens * a.topk;
  const long long weight_bytes = (stage == 1 ? 2LL : 1LL) * a.n_dim * a.k_dim * a.experts;
  if (weight_bytes >= (512LL << 20) && 4 * rows >= (long long)a.tile_m * a.experts) return true;
  const double mean = double(rows) / a.experts;
  const double blocks = row_tiles(mean, a.tile_m), tiles = row_tiles(mean, BM);
  const bool gather = a.a_layout != FLYMOE_ROWS_SORTED;
  const double apart = tile_rounds_us(blocks * a.experts * ntiles, a.tile_m, gather, a.k_dim / BK, ctas);
  // a tile holds its share of the blocks on average; a launch of one round takes as long as its longest tile
  double tile_rows = a.tile_m * blocks / tiles;
  if (tiles * a.experts * ntiles <= ctas) tile_rows = ceil((mean + sqrt(mean)) / a.tile_m) * a.tile_m;
  if (tile_rows > BM) tile_rows = BM;
  const double merged = tile_rounds_us(tiles * a.experts * ntiles, tile_rows, gather, a.k_dim / BK, ctas) + 1.5;
  return merged < (mean >= 0.8 * a.tile_m ? 1.03 : 1.0) * apart;
}

int choose_ksplit(int stage, const GemmArgs& a) {
  // a caller that leaves other kernels some SMs gets no clusters
  if (g_cta_limit > 0 && g_cta_limit < sm_count()) return 1;
  // no more than SMs / s clusters of s run at once: where they would not pay, the real numbers need not be asked for
  const int sms = sm_count();
  int clusters[kClusterSizes] = {sms, sms / 2, sms / 4, sms / 8};
  if (plan_ksplit(stage, a, clusters) == 1) return 1;
  split_residency(stage, a.scaling, clusters);
  return plan_ksplit(stage, a, clusters);
}

int launch_gemm_sm100(int stage, const GemmArgs& a, cudaStream_t stream) {
  if (a.tile_m != 16 && a.tile_m != 32 && a.tile_m != 64 && a.tile_m != 128) {
    set_last_error_msg("tcgen05 GEMM: tile_m must be 16, 32, 64 or 128");
    return FLYMOE_ERR_UNSUPPORTED;
  }
  if (a.a_layout != FLYMOE_ROWS_SORTED && a.a_layout != FLYMOE_ROWS_BY_TOKEN && a.a_layout != FLYMOE_ROWS_BY_PAIR &&
      a.a_layout != FLYMOE_ROWS_BY_SLOT) {
    set_last_error_msg("tcgen05 GEMM: unknown activation row layout");
    return FLYMOE_ERR_UNSUPPORTED;
  }
  const bool per_token = a.scaling == FLYMOE_SCALE_PER_TOKEN;
  if (per_token && (a.row_dst != nullptr || a.out_dtype == FLYMOE_E4M3)) {
    set_last_error_msg("tcgen05 GEMM: per-token scaling supports neither per-row destinations nor e4m3 output");
    return FLYMOE_ERR_UNSUPPORTED;
  }
  const int ctas = g_cta_limit > 0 && g_cta_limit < sm_count() ? g_cta_limit : sm_count();
  if (ctas >= 2 && use_pair_kernel(a)) return launch_gemm_pair(stage, a, ctas, stream);
  CUtensorMap map_a, map_b;
  // rows fetched by index come in boxes of one row; stage 1 fetches gate and up rows apart
  const int rc = make_gemm_maps(stage, a, a.a_layout == FLYMOE_ROWS_SORTED ? a.tile_m : 1, stage == 1 ? 128 : BN,
                                &map_a, &map_b);
  if (rc != FLYMOE_OK) return rc;
  const long long pairs = (long long)a.num_tokens * a.topk;
  const int split = a.ksplit > 0 ? a.ksplit : choose_ksplit(stage, a);
  const bool merge = split == 1 && merge_blocks(stage, a, ctas);
  const long long per_tile = (long long)a.experts * (merge ? BM : a.tile_m);
  long long g = (pairs + per_tile - 1) / per_tile;
  const int group_m = int(g < 1 ? 1 : (g > 16 ? 16 : g));
  if (split > 1) return launch_gemm_split(stage, a, map_a, map_b, group_m, split, stream);
  const int ntiles = stage == 1 ? a.n_dim / 128 : ceil_div(a.n_dim, BN);
  const long long max_tiles = (long long)a.size_expert_ids * ntiles;
  const int grid = int(max_tiles < ctas ? max_tiles : ctas);
  if (grid <= 0) return FLYMOE_OK;
  if (merge) {
    if (per_token)
      return stage == 1 ? launch_one<1, false, kScalePerToken, true>(grid, stream, map_a, map_b, a, group_m)
                        : launch_one<2, false, kScalePerToken, true>(grid, stream, map_a, map_b, a, group_m);
    return stage == 1 ? launch_one<1, false, kScaleBlock128, true>(grid, stream, map_a, map_b, a, group_m)
                      : launch_one<2, false, kScaleBlock128, true>(grid, stream, map_a, map_b, a, group_m);
  }
  if (per_token)
    return stage == 1 ? launch_one<1, false, kScalePerToken, false>(grid, stream, map_a, map_b, a, group_m)
                      : launch_one<2, false, kScalePerToken, false>(grid, stream, map_a, map_b, a, group_m);
  if (stage == 1) return launch_one<1, false, kScaleBlock128, false>(grid, stream, map_a, map_b, a, group_m);
  if (a.row_dst != nullptr) return launch_one<2, true, kScaleBlock128, false>(grid, stream, map_a, map_b, a, group_m);
  return launch_one<2, false, kScaleBlock128, false>(grid, stream, map_a, map_b, a, group_m);
}

}  // namespace flymoe

extern "C" int flymoe_gemm_merges_blocks(int stage, int num_tokens, int topk, int experts, int n_dim, int k_bytes,
                                         int size_expert_ids, int tile_m, int x_layout, int ctas) {
  flymoe::GemmArgs a{};
  a.num_tokens = num_tokens;
  a.topk = topk;
  a.experts = experts;
  a.n_dim = n_dim;
  a.k_dim = k_bytes;
  a.size_expert_ids = size_expert_ids;
  a.tile_m = tile_m;
  a.a_layout = x_layout;
  return flymoe::merge_blocks(stage, a, ctas > 0 ? ctas : flymoe::sm_count()) ? 1 : 0;
}
